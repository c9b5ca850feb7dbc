"""The order of waiting and releasing in kernels that are chained with programmatic dependent launch."""
import re
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parent.parent / "commbench_b200" / "csrc"
# calls that wait for another rank (prim/ptx.cuh, prim/barrier.cuh)
PEER_WAIT = re.compile(r"\b(wait_flag_ge_sys\w*|rank_wait_block|\w+_barrier_(?:block|warp))\(")


def _kernels():
    """(file, name, body without comments) of every __global__ function."""
    for f in sorted(CSRC.rglob("*.cu*")):
        text = re.sub(r"//[^\n]*", "", f.read_text())
        for m in re.finditer(r"__global__", text):
            brace, semicolon = text.find("{", m.end()), text.find(";", m.end())
            if brace < 0 or 0 <= semicolon < brace:
                continue                                  # a declaration
            depth, i = 1, brace + 1
            while depth:
                depth += {"{": 1, "}": -1}.get(text[i], 0)
                i += 1
            name = re.findall(r"(\w+)\s*\(", re.sub(r"__launch_bounds__\([^)]*\)", "", text[m.end():brace]))[0]
            yield f.name, name, text[brace:i]


RELEASING = [k for k in _kernels() if "pdl_launch_dependents(" in k[2]]


def test_the_scan_sees_the_kernels():
    names = {k[1] for k in RELEASING}
    assert {"moe_recv_dequant_kernel", "moe_combine_reduce_kernel", "moe_plan_kernel", "fa_split_kernel",
            "gemm_small_kernel"} <= names
    assert {k[1] for k in RELEASING if PEER_WAIT.search(k[2])} >= {"moe_recv_dequant_kernel",
                                                                   "moe_combine_reduce_kernel"}


@pytest.mark.parametrize("kernel", RELEASING, ids=lambda k: k[1])
def test_a_kernel_releases_after_it_has_waited_for_other_ranks(kernel):
    """A kernel that it releases may take every SM's shared memory.  Started before this wait ends, it would
    keep from running what another rank waits for."""
    body = kernel[2]
    released = body.index("pdl_launch_dependents(")
    assert all(w.start() < released for w in PEER_WAIT.finditer(body))


@pytest.mark.parametrize("kernel", [k for k in RELEASING if k[0].startswith("moe_")], ids=lambda k: k[1])
def test_kernels_in_front_of_the_expert_products_wait_first(kernel):
    """The products read the plan before their own wait."""
    body = kernel[2]
    assert 0 <= body.find("pdl_wait(") < body.index("pdl_launch_dependents(")
