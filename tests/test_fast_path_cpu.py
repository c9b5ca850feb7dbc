"""Without its extension the short call path takes no call, and the operators go on as before."""
import shutil

import pytest
import torch

from commbench_b200 import _native as N


@pytest.fixture(params=["missing", "unreadable", "another PyTorch"])
def no_extension(native_lib, monkeypatch, tmp_path, request):
    path = tmp_path / "_fast_ops.so"
    if request.param == "unreadable":
        path.write_bytes(b"no shared object")
    elif request.param == "another PyTorch":
        shutil.copy(N._FAST_PATH, path)
        monkeypatch.setattr(torch, "__version__", "0.0.0")
    monkeypatch.setattr(N, "_FAST_PATH", path)
    monkeypatch.setattr(N, "_fast", None)


def test_calls_go_to_the_general_path(no_extension):
    from commbench_b200.ops.cp import flash_attention
    from commbench_b200.ops.gemm import GemmError, gemm, quantize_blockscaled_pow2
    from commbench_b200.runtime.context import CommError

    x = torch.zeros(16, 128, dtype=torch.bfloat16)
    with pytest.warns(RuntimeWarning, match="short call path off"):
        f = N.fast()
    assert f.gemm(x, x, None, 1.0, 0, 0, 0) is None
    # the general path's own refusal of a CPU tensor
    with pytest.raises(GemmError, match="CUDA tensor"):
        gemm(x, x)
    with pytest.raises(GemmError, match="CUDA tensor"):
        quantize_blockscaled_pow2(x)
    with pytest.raises(CommError, match="CUDA tensor"):
        flash_attention(x.view(1, 16, 1, 128), x.view(1, 16, 1, 128), x.view(1, 16, 1, 128))


def test_the_extension_that_was_built_here_is_used(native_lib, monkeypatch):
    monkeypatch.setattr(N, "_fast", None)
    assert not isinstance(N.fast(), N._NoFast)
