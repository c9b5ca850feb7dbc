"""tcgen05 GEMM vs a plain PyTorch fp32 reference of the same op."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _ref(a, b, alpha=1.0):
    return alpha * (a.float() @ b.float().t())


def _check(out, ref, tol):
    err = (out.float() - ref).abs().max().item()
    scale = ref.abs().max().item() + 1e-6
    assert err / scale < tol, f"max abs err {err} vs scale {scale}"


# bn 512 / 384 = a CTA pair (cluster of two, `tcgen05.mma.cta_group::2`) per 256 x 256 /
# 256 x 128 tile; the others one CTA per 128 x bn tile.
@pytest.mark.parametrize("bn", [512, 384, 256, 128, 64])
@pytest.mark.parametrize("shape", [(128, 256, 64), (256, 512, 256), (384, 768, 1024),
                                   (1000, 1304, 520), (16, 8192, 1024)])
def test_gemm_bf16_matches_fp32_reference(native_lib, shape, bn):
    from commbench_b200.ops.gemm import gemm

    M, N, K = shape
    g = torch.Generator(device="cuda").manual_seed(1234 + M + N + K)
    a = torch.randn(M, K, device="cuda", generator=g).mul_(0.5).bfloat16()
    b = torch.randn(N, K, device="cuda", generator=g).mul_(0.5).bfloat16()
    status = torch.zeros(4, dtype=torch.int32, device="cuda")
    out = gemm(a, b, bn=bn, status_ptr=status.data_ptr())
    torch.cuda.synchronize()
    assert int(status[0].item()) == 0, hex(int(status[0].item()) & 0xffffffff)
    _check(out, _ref(a, b), 1e-2)


def test_gemm_pair_every_element_exact_on_small_ints(native_lib):
    """CTA-pair tiles: integer-valued inputs make fp32 accumulation exact, so a row or column
    half that lands in the wrong place shows up as a mismatch, not as noise."""
    from commbench_b200.ops.gemm import gemm

    M, N, K = 768, 1024, 320
    g = torch.Generator(device="cuda").manual_seed(11)
    a = torch.randint(-3, 4, (M, K), device="cuda", generator=g).bfloat16()
    b = torch.randint(-3, 4, (N, K), device="cuda", generator=g).bfloat16()
    for bn in (512, 384):
        out = gemm(a, b, bn=bn)
        assert torch.equal(out.float(), _ref(a, b).bfloat16().float()), bn


def test_gemm_bf16_full_tensor_exact_on_small_ints(native_lib):
    """Integer-valued inputs make the fp32 accumulation exact: every element must match."""
    from commbench_b200.ops.gemm import gemm

    M, N, K = 256, 512, 192
    g = torch.Generator(device="cuda").manual_seed(7)
    a = torch.randint(-3, 4, (M, K), device="cuda", generator=g).bfloat16()
    b = torch.randint(-3, 4, (N, K), device="cuda", generator=g).bfloat16()
    out = gemm(a, b, bn=128)
    ref = _ref(a, b)
    assert torch.equal(out.float(), ref.bfloat16().float())


def test_gemm_bf16_large_auto_tile(native_lib):
    from commbench_b200.ops.gemm import gemm

    M, N, K = 4096, 4096, 2048
    g = torch.Generator(device="cuda").manual_seed(3)
    a = torch.randn(M, K, device="cuda", generator=g).mul_(0.1).bfloat16()
    b = torch.randn(N, K, device="cuda", generator=g).mul_(0.1).bfloat16()
    out = gemm(a, b, alpha=0.5)
    _check(out, _ref(a, b, 0.5), 1e-2)


@pytest.mark.parametrize("shape", [(128, 256, 128), (512, 1024, 512), (300, 520, 1024)])
def test_gemm_fp8_matches_fp32_reference(native_lib, shape):
    from commbench_b200.ops.gemm import gemm

    M, N, K = shape
    g = torch.Generator(device="cuda").manual_seed(99)
    a = torch.randn(M, K, device="cuda", generator=g).to(torch.float8_e4m3fn)
    b = torch.randn(N, K, device="cuda", generator=g).to(torch.float8_e4m3fn)
    out = gemm(a, b, alpha=0.25, bn=128)
    _check(out, _ref(a, b, 0.25), 1e-2)
    out2 = gemm(a, b, alpha=0.25, bn=512)  # CTA pair
    _check(out2, _ref(a, b, 0.25), 1e-2)


def test_blockscaled_fp8_roundtrip_and_gemm(native_lib):
    """1x128 activation scales and 128x128 weight scales: quantise, check against a PyTorch
    emulation of the same scheme, then run the GEMM on the expanded operands."""
    from commbench_b200.ops.gemm import (dequantize_blockscaled, quantize_blockscaled)
    from commbench_b200.ops.gemm import gemm_fp8_blockscaled_expanded as gemm_fp8_blockscaled

    M, N, K = 256, 384, 512
    g = torch.Generator(device="cuda").manual_seed(21)
    a = torch.randn(M, K, device="cuda", generator=g).bfloat16()
    b = (torch.randn(N, K, device="cuda", generator=g) * 0.02).bfloat16()
    aq, as_ = quantize_blockscaled(a, 1)
    bq, bs = quantize_blockscaled(b, 128)
    # reference quantisation
    af = a.float().view(M, K // 128, 128)
    ref_s = af.abs().amax(-1) / 448.0
    assert torch.allclose(as_, ref_s, rtol=1e-6)
    bf = b.float().view(N // 128, 128, K // 128, 128)
    ref_bs = bf.abs().amax(dim=(1, 3)) / 448.0
    assert torch.allclose(bs, ref_bs, rtol=1e-6)
    ad = dequantize_blockscaled(aq, as_, 1)
    bd = dequantize_blockscaled(bq, bs, 128)
    assert (ad.float() - a.float()).abs().max() <= 0.07 * a.float().abs().max()
    out = gemm_fp8_blockscaled(aq, as_, bq, bs)
    ref = ad.float() @ bd.float().t()
    _check(out, ref, 1e-2)
    _check(out, a.float() @ b.float().t(), 6e-2)


def _bs_reference(aq, as_, bq, bs):
    """fp32 product of the SAME quantised operands with their block scales applied."""
    M, K = aq.shape
    N = bq.shape[0]
    a = aq.float().view(M, K // 128, 128) * as_[:, :, None]
    bsr = bs.repeat_interleave(128, dim=0)[:N]
    b = bq.float().view(N, K // 128, 128) * bsr[:, :, None]
    return a.view(M, K) @ b.view(N, K).t()


@pytest.mark.parametrize("shape", [(128, 256, 128), (256, 256, 256), (512, 768, 1024),
                                   (1000, 1304, 640), (256, 512, 4096)])
def test_blockscaled_fp8_gemm_in_kernel_scales(native_lib, shape):
    """Block-scaled fp8 contraction with the scales applied inside the kernel (per K block,
    fp32 promotion): against the fp32 product of the same quantised operands.  `pair` is accepted and
    changes nothing."""
    from commbench_b200.ops.gemm import gemm_fp8_blockscaled, quantize_blockscaled

    M, N, K = shape
    g = torch.Generator(device="cuda").manual_seed(5 + M + N + K)
    # magnitudes that differ per block, so that a wrong or missing scale shows
    a = torch.randn(M, K, device="cuda", generator=g) * \
        (1.0 + torch.arange(K // 128, device="cuda").float().repeat_interleave(128))[None, :]
    b = torch.randn(N, K, device="cuda", generator=g) * 0.02 * \
        (1.0 + (torch.arange(N, device="cuda") // 128).float())[:, None]
    aq, as_ = quantize_blockscaled(a.bfloat16().contiguous(), 1)
    bq, bs = quantize_blockscaled(b.bfloat16().contiguous(), 128)
    status = torch.zeros(4, dtype=torch.int32, device="cuda")
    out = gemm_fp8_blockscaled(aq, as_, bq, bs, pair=True, status_ptr=status.data_ptr())
    assert torch.equal(out, gemm_fp8_blockscaled(aq, as_, bq, bs, pair=False))
    torch.cuda.synchronize()
    assert int(status[0].item()) == 0, hex(int(status[0].item()) & 0xffffffff)
    ref = _bs_reference(aq, as_, bq, bs)
    _check(out, ref, 1e-2)
    _check(out, a.bfloat16().float() @ b.bfloat16().float().t(), 6e-2)


def test_pow2_quantisation_bytes_match_scales(native_lib):
    from commbench_b200.ops.gemm import quantize_blockscaled_pow2, sf_exponents

    g = torch.Generator(device="cuda").manual_seed(3)
    x = (torch.randn(300, 640, device="cuda", generator=g) * 3).bfloat16()
    for rb in (1, 128):
        q, s, sf = quantize_blockscaled_pow2(x, rb)
        assert sf.shape == (2, 300)
        assert torch.equal(torch.exp2(torch.log2(s).round()), s)          # powers of two
        per_row = s.repeat_interleave(rb, dim=0)[:300]
        assert torch.equal(torch.exp2(sf_exponents(sf, 5).float() - 127.0), per_row)
        assert bool((sf_exponents(sf, 8)[:, 5:] == 127).all())             # padding = 1.0
        amax = x.float().view(300, 5, 128).abs().amax(-1)
        if rb == 1:
            assert bool((s >= amax / 448.0).all()) and bool((s < 2 * amax / 448.0 + 1e-30).all())


@pytest.mark.parametrize("pair", [True, False])
@pytest.mark.parametrize("shape", [(128, 192, 128), (128, 192, 512), (256, 384, 1024),
                                   (1000, 1304, 640), (512, 8192, 2048)])
def test_fp8_gemm_with_hardware_block_scales(native_lib, shape, pair):
    """Power-of-two 1x128 / 128x128 block scales applied by the tensor core: against the fp32
    product of the same quantised operands with the same scales."""
    from commbench_b200.ops.gemm import gemm_fp8_mx, quantize_blockscaled_pow2

    M, N, K = shape
    g = torch.Generator(device="cuda").manual_seed(9 + M + N + K)
    a = torch.randn(M, K, device="cuda", generator=g) * \
        (1.0 + torch.arange(K // 128, device="cuda").float().repeat_interleave(128))[None, :] * \
        (1.0 + (torch.arange(M, device="cuda") % 7).float())[:, None]
    b = torch.randn(N, K, device="cuda", generator=g) * 0.02 * \
        (1.0 + (torch.arange(N, device="cuda") // 128).float())[:, None]
    aq, as_, asf = quantize_blockscaled_pow2(a.bfloat16().contiguous(), 1)
    bq, bs, bsf = quantize_blockscaled_pow2(b.bfloat16().contiguous(), 128)
    status = torch.zeros(4, dtype=torch.int32, device="cuda")
    out = gemm_fp8_mx(aq, asf, bq, bsf, pair=pair, status_ptr=status.data_ptr())
    torch.cuda.synchronize()
    assert int(status[0].item()) == 0, hex(int(status[0].item()) & 0xffffffff)
    ref = _bs_reference(aq, as_, bq, bs)
    _check(out, ref, 1e-2)


@pytest.mark.gpu
@pytest.mark.parametrize("rows,k", [(1, 128), (3, 640), (4, 512), (37, 384), (130, 1152)])
@pytest.mark.parametrize("pow2", [False, True])
def test_quantize_rows_is_exact(native_lib, rows, k, pow2):
    """The warp-per-512-columns kernel at ragged row groups and K groups: scales, e4m3 bytes and
    packed words equal the formula bit for bit (zero and huge blocks among them)."""
    from commbench_b200.ops.gemm import quantize_blockscaled, quantize_blockscaled_pow2

    g = torch.Generator(device="cuda").manual_seed(rows * 1000 + k)
    x = (torch.randn(rows, k, device="cuda", generator=g)
         * torch.logspace(-6, 6, rows, device="cuda")[:, None]).bfloat16()
    x[0, :128] = 0
    x[-1, -1] = 3e38
    f = x.float().view(rows, k // 128, 128)
    amax = f.abs().amax(dim=-1)
    s = torch.where(amax > 0, amax / torch.full_like(amax, 448.0), torch.ones_like(amax))
    if pow2:
        m, e = torch.frexp(s)
        s = torch.ldexp(torch.ones_like(s), torch.where(m == 0.5, e - 1, e))
    # the kernel saturates, torch's cast may not: clamp in fp32 first
    ref = (f * (1.0 / s)[..., None]).clamp(-448, 448).to(torch.float8_e4m3fn).view(rows, k)
    if pow2:
        q, sc, sf = quantize_blockscaled_pow2(x, 1)
        kg = (k // 128 + 3) // 4
        byte = torch.full((rows, kg * 4), 127, dtype=torch.uint8, device="cuda")
        byte[:, :k // 128] = (torch.frexp(s)[1] + 126).to(torch.uint8)
        words = byte.view(rows, kg, 4).permute(1, 0, 2).contiguous().view(torch.int32).view(kg, rows)
        assert torch.equal(sf, words)
    else:
        q, sc = quantize_blockscaled(x, 1)
    assert torch.equal(sc, s)
    assert torch.equal(q.view(torch.uint8), ref.view(torch.uint8))


@pytest.mark.parametrize("fp8", [False, True])
@pytest.mark.parametrize("split", [1, 2, 4, 8])
@pytest.mark.parametrize("bn", [64, 128, 256])
@pytest.mark.parametrize("shape", [(1, 8, 1024), (7, 72, 1040), (128, 264, 1536), (129, 520, 1040),
                                   (300, 136, 2064)])
def test_small_gemm_splits(native_lib, shape, bn, split, fp8):
    """Split-K kernel at the edges of its tiles: one row, ragged row groups, columns short of a
    tile, a last K block of 16 elements, K blocks that do not divide by the splits or the ring
    stage.  Against fp32: the bf16 result is off by at most half a unit (2^-9 of the value), the
    fp32 sums by far less, so 2-norm 3e-3 and 1e-2 of the largest value.  Two runs give the same
    bits; rows of C beyond M stay untouched."""
    from commbench_b200 import _native as N

    M, Nn, K = shape
    g = torch.Generator(device="cuda").manual_seed(M + Nn + K)
    a = torch.randn(M, K, device="cuda", generator=g).mul_(0.5).bfloat16()
    b = torch.randn(Nn, K, device="cuda", generator=g).mul_(0.5).bfloat16()
    if fp8:
        a, b = a.to(torch.float8_e4m3fn), b.to(torch.float8_e4m3fn)
    lib = N.load()
    status = torch.zeros(4, dtype=torch.int32, device="cuda")
    outs = []
    for _ in range(2):
        c = torch.full((M + 3, Nn), 7.0, device="cuda", dtype=torch.bfloat16)
        rc = lib.cb_gemm_small(a.data_ptr(), b.data_ptr(), c.data_ptr(), M, Nn, K, 0.5, int(fp8), bn,
                               split, status.data_ptr(), N.raw_stream())
        assert rc == 0, N.last_error()
        outs.append(c)
    ref = _ref(a, b, 0.5)
    assert int(status.abs().sum()) == 0
    assert torch.equal(outs[0], outs[1])
    assert bool((outs[0][M:] == 7.0).all())
    err = outs[0][:M].float() - ref
    assert err.norm() <= 3e-3 * ref.norm()
    assert err.abs().max() <= 1e-2 * ref.abs().max()


def test_gemm_choice_covers_the_range(native_lib):
    """The size rule: split K where tiles are few, the pair kernel where they are many; whatever it
    picks is right (bf16 rounding, 2-norm 3e-3)."""
    from commbench_b200 import _native as N
    from commbench_b200.ops.gemm import gemm

    lib = N.load()
    assert lib.cb_gemm_choice(48, 3584, 8192, 0) >= 2000          # split
    assert lib.cb_gemm_choice(8192, 8192, 8192, 0) == 512         # persistent pairs
    g = torch.Generator(device="cuda").manual_seed(9)
    for M, Nn, K in [(1, 512, 8), (17, 4096, 4096), (129, 1032, 3080), (700, 2000, 520)]:
        a = torch.randn(M, K, device="cuda", generator=g).bfloat16()
        b = torch.randn(Nn, K, device="cuda", generator=g).bfloat16()
        ref = _ref(a, b)
        assert (gemm(a, b).float() - ref).norm() <= 3e-3 * ref.norm()
        out = gemm(a, b, max_ctas=16)                             # a CTA limit keeps the persistent kernels
        assert (out.float() - ref).norm() <= 3e-3 * ref.norm()


@pytest.mark.parametrize("bn", [512, 256])
def test_role_trace_runs_with_one_tracing_lane(native_lib, bn):
    """Only lane 0 of the first epilogue warp traces: the waits, which are warp-collective, must not
    depend on it."""
    from commbench_b200.ops.gemm import gemm_role_trace

    a = torch.randn(300, 1024, device="cuda").bfloat16()
    b = torch.randn(520, 1024, device="cuda").bfloat16()
    r = gemm_role_trace(a, b, bn)
    assert r["mma_cycles"] > 0
    assert all(0.0 <= v <= 1.0 for k, v in r.items() if k != "mma_cycles"), r


@pytest.mark.parametrize("path", ["bf16", "mx", "blockscaled"])
def test_gemm_on_a_side_stream_leaves_blocks_of_the_current_stream_alone(native_lib, path):
    """A result made inside a call that is given a stream does not take a block that the current stream
    has freed but still has a copy queued from."""
    from commbench_b200.ops.gemm import (gemm, gemm_fp8_blockscaled, gemm_fp8_mx, quantize_blockscaled,
                                         quantize_blockscaled_pow2)

    a = torch.randn(512, 1024, device="cuda").bfloat16()
    b = torch.randn(2048, 1024, device="cuda").bfloat16()
    if path == "bf16":
        run = lambda **kw: gemm(a, b, **kw)
    elif path == "mx":
        (aq, _, asf), (bq, _, bsf) = quantize_blockscaled_pow2(a, 1), quantize_blockscaled_pow2(b, 128)
        run = lambda **kw: gemm_fp8_mx(aq, asf, bq, bsf, **kw)
    else:
        (aq, as_), (bq, bs) = quantize_blockscaled(a, 1), quantize_blockscaled(b, 128)
        run = lambda **kw: gemm_fp8_blockscaled(aq, as_, bq, bs, **kw)
    ref = run()
    side = torch.cuda.Stream()
    for _ in range(3):
        block = torch.full((ref.numel() * 2,), 0x5a, dtype=torch.uint8, device="cuda")
        kept = torch.empty_like(block)
        torch.cuda.synchronize()
        torch.cuda._sleep(20_000_000)                 # about 10 ms: the copy stays queued behind it
        kept.copy_(block)
        del block
        out = run(stream=side)
        torch.cuda.synchronize()
        assert bool((kept == 0x5a).all()) and torch.equal(out, ref)


@pytest.mark.parametrize("fp8", [False, True])
@pytest.mark.parametrize("max_ctas", [1, 2, 3])
def test_gemm_with_a_limit_of_few_ctas(native_lib, max_ctas, fp8):
    """A limit below a CTA pair: a shape for which the size rule picks pairs runs on single CTAs, and an
    explicit pair tile is refused instead of leaving the result unwritten.  bf16 rounding, 2-norm
    3e-3."""
    from commbench_b200 import _native as N
    from commbench_b200.ops.gemm import GemmError, gemm

    M, Nn, K = 3000, 2568, 1040
    assert N.load().cb_gemm_choice(M, Nn, K, int(fp8)) == 512
    g = torch.Generator(device="cuda").manual_seed(17)
    a = torch.randn(M, K, device="cuda", generator=g).bfloat16()
    b = torch.randn(Nn, K, device="cuda", generator=g).bfloat16()
    if fp8:
        a, b = a.to(torch.float8_e4m3fn), b.to(torch.float8_e4m3fn)
    ref = _ref(a, b)
    for bn in (0, 256, 128, 64) + ((512,) if max_ctas > 1 else ()):
        out = torch.full((M, Nn), float("nan"), device="cuda", dtype=torch.bfloat16)
        gemm(a, b, out=out, bn=bn, max_ctas=max_ctas)
        assert (out.float() - ref).norm() <= 3e-3 * ref.norm(), bn
    if max_ctas == 1:
        with pytest.raises(GemmError, match="pair"):
            gemm(a, b, bn=512, max_ctas=1)


@pytest.mark.parametrize("m", [1, 48, 300])
def test_split_k_gemm_in_a_cuda_graph(native_lib, m):
    """Two split-K GEMMs in a row, chained with programmatic dependent launch, captured and replayed on
    new inputs: the bits of the plain calls."""
    from commbench_b200 import _native as N
    from commbench_b200.ops.gemm import gemm

    assert N.load().cb_gemm_choice(m, 1024, 2048, 0) >= 1000 and N.load().cb_gemm_choice(m, 2048, 1024, 0) >= 1000
    x = torch.randn(m, 2048, device="cuda").bfloat16()
    w1 = (torch.randn(1024, 2048, device="cuda") * 0.05).bfloat16()
    w2 = (torch.randn(2048, 1024, device="cuda") * 0.05).bfloat16()
    gemm(gemm(x, w1), w2)
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        y = gemm(gemm(x, w1), w2)
    for seed in range(3):
        x.copy_(torch.randn(m, 2048, device="cuda", generator=torch.Generator("cuda").manual_seed(seed)))
        graph.replay()
        assert torch.equal(y, gemm(gemm(x, w1), w2))


@pytest.mark.parametrize("fp8", [False, True])
@pytest.mark.parametrize("shape", [(1, 8, 64), (256, 224, 128), (257, 216, 192), (300, 232, 320),
                                   (513, 904, 512), (700, 1112, 1040)])
def test_gemm_pair_tiles_224_wide_exact_on_small_ints(native_lib, shape, fp8):
    """256 x 224 tiles: three store boxes of 64 columns and one of 32 per row group; widths that end in
    each of them, row counts around the tile height."""
    from commbench_b200.ops.gemm import gemm

    M, N, K = shape
    g = torch.Generator(device="cuda").manual_seed(M + N)
    a = torch.randint(-3, 4, (M, K), device="cuda", generator=g).float()
    b = torch.randint(-3, 4, (N, K), device="cuda", generator=g).float()
    dt = torch.float8_e4m3fn if fp8 else torch.bfloat16
    guard = torch.full((M + 2, N), 7.0, device="cuda", dtype=torch.bfloat16)
    out = guard[1:M + 1]
    gemm(a.to(dt), b.to(dt), out=out, bn=448)
    # |sums| < 9 * 1040 are exact in fp32; the result is their rounding to bf16
    assert torch.equal(out.float(), _ref(a, b).bfloat16().float())
    assert bool((guard[0] == 7).all()) and bool((guard[M + 1] == 7).all())


@pytest.mark.parametrize("n", [3584, 3568, 3544, 3400])
def test_fp8_gemm_with_hardware_block_scales_224_wide(native_lib, n):
    """Shapes at which 256 x 224 tiles take fewer waves than 256 x 192, the last column tile whole,
    ending inside its half box, inside a whole box, and nearly empty."""
    from commbench_b200.ops.gemm import gemm_fp8_mx, quantize_blockscaled_pow2

    M, K = 8100, 640
    g = torch.Generator(device="cuda").manual_seed(n)
    a = torch.randn(M, K, device="cuda", generator=g) * (1.0 + (torch.arange(M, device="cuda") % 7))[:, None]
    b = torch.randn(n, K, device="cuda", generator=g) * 0.02 * (1 + torch.arange(n, device="cuda") // 128)[:, None]
    aq, as_, asf = quantize_blockscaled_pow2(a.bfloat16().contiguous(), 1)
    bq, bs, bsf = quantize_blockscaled_pow2(b.bfloat16().contiguous(), 128)
    out = gemm_fp8_mx(aq, asf, bq, bsf)
    _check(out, _bs_reference(aq, as_, bq, bs), 1e-2)
    # the same K order on one CTA per 128 x 192 tile: the same bits
    assert torch.equal(out, gemm_fp8_mx(aq, asf, bq, bsf, pair=False))


@pytest.mark.parametrize("fp8", [False, True])
@pytest.mark.parametrize("bn", [64, 128, 256])
@pytest.mark.parametrize("m", [1, 8, 9, 40, 65, 120, 121, 128, 130])
def test_small_gemm_ring_slots_of_every_height(native_lib, m, bn, fp8):
    """Ring slots follow the rows of A, 10 of them at one row and 3 or 4 at 128: K long enough to go round
    several times, and short enough to leave slots unused."""
    from commbench_b200 import _native as N

    lib = N.load()
    for n, k in ((264, 2704), (64, 80)):
        g = torch.Generator(device="cuda").manual_seed(m + n)
        a = torch.randint(-3, 4, (m, k), device="cuda", generator=g).float()
        b = torch.randint(-3, 4, (n, k), device="cuda", generator=g).float()
        dt = torch.float8_e4m3fn if fp8 else torch.bfloat16
        aq, bq = a.to(dt), b.to(dt)
        for split in (1, 4):
            if split > (k * aq.element_size() + 127) // 128:
                continue
            out = torch.full((m, n), float("nan"), device="cuda", dtype=torch.bfloat16)
            N.check(lib.cb_gemm_small(aq.data_ptr(), bq.data_ptr(), out.data_ptr(), m, n, k, 1.0, int(fp8), bn,
                                      split, 0, N.raw_stream()), "cb_gemm_small")
            # |sums| < 9 * 2704 are exact in fp32
            assert torch.equal(out.float(), _ref(a, b).bfloat16().float()), (n, k, split)


@pytest.mark.parametrize("shape", [(8100, 3584, 1024), (8100, 3544, 1152), (8100, 3400, 1024), (1718, 4296, 640),
                                   (1718, 4272, 128)])
def test_hardware_block_scales_224_wide_where_the_choice_takes_them(native_lib, shape):
    """At the shortest K of the rule and below it; the last column tile whole, ending inside its half box, inside
    a whole box and nearly empty.  The same K order as on one CTA per 128 x 192 tile: the same bits."""
    from commbench_b200.ops.gemm import gemm_fp8_mx, quantize_blockscaled_pow2

    M, n, K = shape
    assert native_lib.cb_gemm_mx_choice(M, n, K) == 224
    g = torch.Generator(device="cuda").manual_seed(n)
    a = torch.randn(M, K, device="cuda", generator=g) * (1.0 + (torch.arange(M, device="cuda") % 7))[:, None]
    b = torch.randn(n, K, device="cuda", generator=g) * 0.02 * (1 + torch.arange(n, device="cuda") // 128)[:, None]
    aq, as_, asf = quantize_blockscaled_pow2(a.bfloat16().contiguous(), 1)
    bq, bs, bsf = quantize_blockscaled_pow2(b.bfloat16().contiguous(), 128)
    out = gemm_fp8_mx(aq, asf, bq, bsf)
    _check(out, _bs_reference(aq, as_, bq, bs), 1e-2)
    assert torch.equal(out, gemm_fp8_mx(aq, asf, bq, bsf, pair=False))
