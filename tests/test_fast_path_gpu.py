"""The short call path of the small operators: what it takes gives the general path's bits, what it does
not take falls back to it, errors stay what they were."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _general(monkeypatch):
    """N.fast() whose functions take nothing."""
    from commbench_b200 import _native as N

    class Nothing:
        def __getattr__(self, name):
            return lambda *a: None

    monkeypatch.setattr(N, "_fast", Nothing())


def _inputs(m=37, n=200, k=256):
    g = torch.Generator(device="cuda").manual_seed(m + n)
    x = torch.randn(m, k, device="cuda", generator=g).bfloat16()
    w = (torch.randn(n, k, device="cuda", generator=g) * 0.02).bfloat16()
    return x, w


def _calls():
    from commbench_b200.ops import gemm as G
    from commbench_b200.ops.cp import flash_attention
    from commbench_b200.ops.tp_fp8 import MxWeight, quantize_act_mx

    x, w = _inputs()
    f8 = [t.to(torch.float8_e4m3fn) for t in (x, w)]
    mx = MxWeight.from_bf16(w)
    xq, xsf = quantize_act_mx(x)
    bq, bs = G.quantize_blockscaled(x, 1)
    wq, ws = G.quantize_blockscaled(w, 128)
    q = torch.randn(2, 3, 8, 128, device="cuda").bfloat16()
    kv = torch.randn(2, 700, 2, 128, device="cuda").bfloat16()
    long = torch.randn(1, 1300, 8, 128, device="cuda").bfloat16()
    return [lambda: G.gemm(x, w), lambda: G.gemm(x, w, alpha=0.5, bn=64), lambda: G.gemm(*f8, alpha=0.25),
            lambda: G.quantize_blockscaled(x, 1), lambda: G.quantize_blockscaled_pow2(x, 1),
            lambda: G.gemm_fp8_mx(xq, xsf, mx.q, mx.sf), lambda: G.gemm_fp8_mx(xq, xsf, mx.q, mx.sf, pair=False),
            lambda: G.gemm_fp8_blockscaled(bq, bs, wq, ws),
            lambda: flash_attention(q, kv, kv, q_offset=697), lambda: flash_attention(long, long, long, causal=False),
            lambda: flash_attention(q, kv, kv, q_offset=697, kv_offset=3, scale=0.1)]


def _same(a, b):
    a, b = (x if isinstance(x, tuple) else (x,) for x in (a, b))
    assert len(a) == len(b)
    for s, t in zip(a, b):
        assert s.dtype == t.dtype and s.shape == t.shape and s.device == t.device
        assert torch.equal(s.view(torch.uint8), t.view(torch.uint8))


@pytest.mark.parametrize("i", range(11))
def test_short_path_gives_the_same_bits(native_lib, monkeypatch, i):
    call = _calls()[i]
    fast = call()
    _general(monkeypatch)
    _same(fast, call())


def test_short_path_takes_the_plain_call(native_lib):
    from commbench_b200 import _native as N

    x, w = _inputs()
    f = N.fast()
    out = torch.empty(x.shape[0], w.shape[0], device="cuda", dtype=torch.bfloat16)
    assert f.gemm(x, w, out, 1.0, 0, 0, 0) is out
    assert f.gemm(x, torch.nn.Parameter(w), None, 1.0, 0, 0, 0) is not None
    assert f.quantize_rows(x, True) is not None


def test_short_path_leaves_the_rest(native_lib):
    """Layouts, types, views and modes that it does not know."""
    from commbench_b200 import _native as N
    from torch.utils._python_dispatch import TorchDispatchMode

    class Sub(torch.Tensor):
        pass

    class Mode(TorchDispatchMode):
        def __torch_dispatch__(self, func, types, args=(), kwargs=None):
            return func(*args, **(kwargs or {}))

    x, w = _inputs()
    f = N.fast()
    args = (None, 1.0, 0, 0, 0)
    wide = torch.randn(37, 264, device="cuda").bfloat16()
    for a, b in [(x.cpu(), w), (x.float(), w), (x, w[:, :128]), (x.t(), w), (wide[:, 1:257], w),
                 (wide.view(-1)[4:4 + 37 * 256].view(37, 256), w), (x[0], w), (x.as_subclass(Sub), w),
                 (x.half(), w.half()), (x[:0], w), (None, w), (1, w)]:
        assert f.gemm(a, b, *args) is None
    assert f.gemm(x, w, x, 1.0, 0, 0, 0) is None                    # a result of another shape
    assert f.gemm(x, w, None, 1, 0, 0, 0) is None                   # alpha is no float
    assert f.gemm(x, w, None, 1.0, 77, 0, 0) is None                # a refused tile
    assert f.gemm(x, w) is None
    with Mode():
        assert f.gemm(x, w, *args) is None
    assert f.quantize_rows(x[:, :200].contiguous(), False) is None  # no multiple of 128
    q = torch.randn(1, 4, 3, 128, device="cuda").bfloat16()
    kv = torch.randn(1, 9, 2, 128, device="cuda").bfloat16()
    assert f.attention(q, kv, kv, True, 0, 0, None, 0) is None      # 3 heads over 2
    assert f.attention(q[..., :64].contiguous(), kv, kv, True, 0, 0, None, 0) is None


def test_errors_are_those_of_the_general_path(native_lib):
    from commbench_b200.ops.gemm import GemmError, gemm
    from commbench_b200.ops.cp import flash_attention
    from commbench_b200.runtime.context import CommError

    x, w = _inputs()
    with pytest.raises(GemmError, match="contiguous"):
        gemm(x.t(), w)
    with pytest.raises(GemmError, match="inner dimensions"):
        gemm(x, w[:, :128].contiguous())
    with pytest.raises(GemmError, match="bn must be"):
        gemm(x, w, bn=77)
    q = torch.randn(1, 4, 3, 128, device="cuda").bfloat16()
    kv = torch.randn(1, 9, 2, 128, device="cuda").bfloat16()
    with pytest.raises(CommError):
        flash_attention(q, kv, kv)


def test_short_path_follows_the_current_stream_and_is_captured(native_lib):
    from commbench_b200.ops.gemm import gemm

    x, w = _inputs(64, 512, 512)
    ref = gemm(x, w)
    side = torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(side):
        busy = torch.zeros(1 << 26, device="cuda")
        y = x + 0.0 * busy[0].bfloat16()          # ready on this stream only
        out = gemm(y, w)
    torch.cuda.current_stream().wait_stream(side)
    assert torch.equal(out, ref)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        cap = gemm(x, w)
    cap.zero_()
    graph.replay()
    assert torch.equal(cap, ref)


@pytest.mark.parametrize("i", range(11))
def test_short_path_is_asked_and_answers(native_lib, monkeypatch, i):
    """Every call that is compared with the general path above is one that the extension takes."""
    from commbench_b200 import _native as N

    ext, answers = N.fast(), []

    class Spy:
        def __getattr__(self, name):
            def call(*args):
                answers.append(getattr(ext, name)(*args))
                return answers[-1]
            return call

    call = _calls()[i]
    monkeypatch.setattr(N, "_fast", Spy())
    call()
    assert len(answers) == 1 and answers[0] is not None


@pytest.mark.parametrize("rows,k", [(1, 128), (37, 256), (129, 640), (1000, 3584)])
def test_row_quantiser_of_the_short_path(native_lib, monkeypatch, rows, k):
    """Scales in fp32, at one row, ragged rows, K groups that are not whole, and rows of zeros."""
    from commbench_b200.ops.gemm import quantize_blockscaled

    g = torch.Generator(device="cuda").manual_seed(rows)
    x = torch.randn(rows, k, device="cuda", generator=g).bfloat16()
    x[rows // 2] = 0
    fast = quantize_blockscaled(x, 1)
    _general(monkeypatch)
    _same(fast, quantize_blockscaled(x, 1))
