"""tcgen05 flash-attention forward and the exact merge of partial results, against a plain
PyTorch fp32 reference."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _qkv(B, Sq, Skv, Hq, Hkv, seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    q = torch.randn(B, Sq, Hq, 128, device="cuda", generator=g).bfloat16()
    k = torch.randn(B, Skv, Hkv, 128, device="cuda", generator=g).bfloat16()
    v = torch.randn(B, Skv, Hkv, 128, device="cuda", generator=g).bfloat16()
    return q, k, v


@pytest.mark.parametrize("impl", [1, 4])
@pytest.mark.parametrize("causal", [True, False])
@pytest.mark.parametrize("shape", [(1, 128, 128, 1, 1), (1, 256, 256, 4, 1), (2, 384, 384, 4, 2),
                                   (1, 200, 200, 2, 2), (1, 1024, 1024, 8, 2),
                                   (1, 2048, 2048, 4, 1)])
def test_flash_attention_matches_reference(native_lib, shape, causal, impl):
    from commbench_b200.ops.cp import flash_attention, reference_attention

    B, Sq, Skv, Hq, Hkv = shape
    q, k, v = _qkv(B, Sq, Skv, Hq, Hkv, 11 + Sq)
    o, lse = flash_attention(q, k, v, causal=causal, impl=impl)
    torch.cuda.synchronize()
    ro, rl = reference_attention(q, k, v, causal=causal)
    assert torch.allclose(o.float(), ro, atol=2e-2, rtol=2e-2), (o.float() - ro).abs().max()
    assert torch.allclose(lse, rl, atol=2e-2, rtol=1e-3)


def test_chunked_attention_with_offsets_merges_to_full(native_lib):
    """Keys split in three chunks (one entirely in the future of some queries); the merged
    result must equal attention over the whole sequence - the ring-attention invariant."""
    from commbench_b200.ops.cp import attn_merge, flash_attention, reference_attention

    B, S, Hq, Hkv = 1, 384, 4, 2
    q, k, v = _qkv(B, S, S, Hq, Hkv, 77)
    q_off = 128                      # queries are positions 128..511 of a longer sequence
    kfull = torch.cat([k, k.flip(1)], dim=1)[:, :640].contiguous()
    vfull = torch.cat([v, v.flip(1)], dim=1)[:, :640].contiguous()
    o_acc = torch.empty(B, S, Hq, 128, dtype=torch.float32, device="cuda")
    l_acc = torch.empty(B, Hq, S, dtype=torch.float32, device="cuda")
    bounds = [(0, 256), (256, 512), (512, 640)]
    for i, (a, b) in enumerate(bounds):
        o, lse = flash_attention(q, kfull[:, a:b].contiguous(), vfull[:, a:b].contiguous(),
                                 causal=True, q_offset=q_off, kv_offset=a)
        attn_merge(o_acc, l_acc, o, lse, first=(i == 0))
    ro, rl = reference_attention(q, kfull, vfull, causal=True, q_offset=q_off, kv_offset=0)
    assert torch.allclose(o_acc, ro, atol=2e-2, rtol=2e-2)
    assert torch.allclose(l_acc, rl, atol=2e-2, rtol=1e-3)


def test_ring_and_ulysses_single_rank(native_lib):
    from commbench_b200.ops.cp import RingAttention, reference_attention, ulysses_attention
    from commbench_b200.runtime.context import CommContext

    ctx = CommContext(heap_bytes=64 << 20)
    q, k, v = _qkv(1, 512, 512, 4, 1, 5)
    ring = RingAttention(ctx, 1, 512, 4, 1)
    o, lse = ring.forward(q, k, v, causal=True)
    ro, rl = reference_attention(q, k, v, causal=True)
    assert torch.allclose(o.float(), ro, atol=2e-2, rtol=2e-2)
    assert torch.allclose(lse, rl, atol=2e-2, rtol=1e-3)
    o2 = ulysses_attention(ctx, q, k, v, causal=True)
    assert torch.allclose(o2.float(), ro, atol=2e-2, rtol=2e-2)
    ctx.check_status()
    ctx.close()


def _full(B, S, Hq, Hkv, seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    q = torch.randn(B, S, Hq, 128, device="cuda", generator=g).bfloat16()
    k = torch.randn(B, S, Hkv, 128, device="cuda", generator=g).bfloat16()
    v = torch.randn(B, S, Hkv, 128, device="cuda", generator=g).bfloat16()
    return q, k, v


@pytest.mark.parametrize("world", [2, 4])
@pytest.mark.parametrize("zigzag", [True, False])
@pytest.mark.parametrize("causal", [True, False])
def test_ring_attention_kernel_virtual_ranks(native_lib, world, zigzag, causal):
    """W virtual ranks on one GPU (their launches pull from each other's buffers, none waits
    for another): every rank's rows must equal full-sequence attention, over three calls."""
    from commbench_b200.ops.cp import RingAttention, reference_attention, zigzag_shard
    from commbench_b200.runtime.context import EmuContext

    B, Sl, Hq, Hkv = 2, 512, 4, 2
    S = Sl * world
    q, k, v = _full(B, S, Hq, Hkv, 31 + world)
    ro, rl = reference_attention(q, k, v, causal=causal)
    if zigzag:
        shard = lambda x, r: zigzag_shard(x, world, r)
    else:
        shard = lambda x, r: x[:, r * Sl:(r + 1) * Sl].contiguous()
    ctx = EmuContext(world)
    ring = RingAttention(ctx, B, Sl, Hq, Hkv, zigzag=zigzag, num_comm=2)
    qs = [shard(q, r) for r in range(world)]
    ks = [shard(k, r) for r in range(world)]
    vs = [shard(v, r) for r in range(world)]
    for it in range(3):
        outs, lses = ring.forward(qs, ks, vs, causal=causal)
        ctx.check_status()
        for r in range(world):
            assert torch.allclose(outs[r].float(), shard(ro, r), atol=2e-2, rtol=2e-2), (it, r)
            ref_l = shard(rl.permute(0, 2, 1), r).permute(0, 2, 1)
            assert torch.allclose(lses[r], ref_l, atol=2e-2, rtol=1e-3), (it, r)
    # the same object with the other mask: the list of pieces to pull changes
    ro2, _ = reference_attention(q, k, v, causal=not causal)
    for it in range(2):
        outs, _ = ring.forward(qs, ks, vs, causal=not causal)
        ctx.check_status()
        for r in range(world):
            assert torch.allclose(outs[r].float(), shard(ro2, r), atol=2e-2, rtol=2e-2), (it, r)


@pytest.mark.parametrize("world", [2, 4])
@pytest.mark.parametrize("causal", [True, False])
def test_ulysses_attention_kernel_virtual_ranks(native_lib, world, causal):
    """Sequence-sharded in and out; each virtual rank attends for its head slice over the whole
    sequence, reading Q from and writing O to the other ranks' tensors."""
    from commbench_b200.ops.cp import UlyssesAttention, reference_attention
    from commbench_b200.runtime.context import EmuContext

    B, Sl, Hq, Hkv = 1, 512, 8, 4
    S = Sl * world
    q, k, v = _full(B, S, Hq, Hkv, 57 + world)
    ro, _ = reference_attention(q, k, v, causal=causal)
    ctx = EmuContext(world)
    op = UlyssesAttention(ctx, B, Sl, Hq, Hkv, num_comm=2)
    sh = lambda x, r: x[:, r * Sl:(r + 1) * Sl].contiguous()
    for it in range(3):
        outs = op.forward([sh(q, r) for r in range(world)], [sh(k, r) for r in range(world)],
                          [sh(v, r) for r in range(world)], causal=causal)
        ctx.check_status()
        for r in range(world):
            assert torch.allclose(outs[r].float(), sh(ro, r), atol=2e-2, rtol=2e-2), (it, r)


# (B, Sq, Skv, Hq, Hkv, q_offset, kv_offset): one block and one key; a group of one, three (no
# divisor of 128) and 64; ragged keys; more items than CTAs; items cut over many CTAs; a query tile
# that sees no key; several query tiles with a causal diagonal.
SPLIT_SHAPES = [(1, 1, 1, 1, 1, 0, 0), (1, 1, 129, 4, 1, 128, 0), (3, 2, 1000, 6, 2, 998, 0),
                (2, 1, 640, 128, 2, 639, 0), (40, 1, 300, 8, 8, 299, 0), (1, 1, 16384, 8, 1, 16383, 0),
                (2, 4, 5000, 32, 8, 4996, 0), (1, 100, 260, 8, 2, 0, 70), (1, 300, 1077, 4, 1, 777, 0)]


@pytest.mark.parametrize("causal", [True, False])
@pytest.mark.parametrize("shape", SPLIT_SHAPES)
def test_split_key_attention_matches_reference(native_lib, shape, causal):
    """Split-key kernel and merge against fp32.  o: rounding of the bf16 result (2^-9 of values of
    order one) plus bf16 probabilities, 1e-2 of the largest value; lse is fp32 throughout, 1e-4."""
    import ctypes as C
    import math

    from commbench_b200 import _native as N
    from commbench_b200.ops.cp import reference_attention

    B, Sq, Skv, Hq, Hkv, qo, ko = shape
    q, k, v = _qkv(B, Sq, Skv, Hq, Hkv, 31 + Skv)
    lib = N.load()
    nbytes = 64 << 20
    ws = torch.full((nbytes,), 0xff, dtype=torch.uint8, device="cuda")     # NaN everywhere
    o, lse = torch.empty_like(q), torch.empty(B, Hq, Sq, device="cuda")
    status = torch.zeros(4, dtype=torch.int32, device="cuda")
    rc = lib.cb_attn_split(N.ptr(q), N.ptr(k), N.ptr(v), N.ptr(o), N.ptr(lse), B, Sq, Skv, Hq, Hkv,
                           qo, ko, int(causal), C.c_float(1.0 / math.sqrt(128)), N.ptr(ws),
                           C.c_longlong(nbytes), N.ptr(status), N.stream_ptr())
    assert rc == 0, N.last_error()
    ro, rl = reference_attention(q, k, v, causal=causal, q_offset=qo, kv_offset=ko)
    assert int(status.abs().sum()) == 0
    assert (o.float() - ro).abs().max() <= 1e-2 * ro.abs().max()
    seen = rl > float("-inf")
    assert torch.equal(lse > float("-inf"), seen)
    assert (lse - rl)[seen].abs().max() < 1e-4


def test_split_and_pair_kernels_agree_on_the_public_call(native_lib):
    """The size rule sends decode to the split kernel and a full prefill to the tile-pair kernel; both
    give the same on one call (each within 1e-2 of the largest value of fp32, lse within 1e-4); a
    workspace that is too small is refused."""
    import ctypes as C
    import math

    from commbench_b200 import _native as N
    from commbench_b200.ops.cp import flash_attention, reference_attention

    lib = N.load()
    assert lib.cb_attn_split_bytes(4, 1, 3000, 16, 4, 2999, 0, 1) > 0
    assert lib.cb_attn_split_bytes(1, 16384, 16384, 32, 8, 0, 0, 1) == -1
    q, k, v = _qkv(4, 1, 3000, 16, 4, 3)
    o, lse = flash_attention(q, k, v, causal=True, q_offset=2999)
    ro, rl = reference_attention(q, k, v, causal=True, q_offset=2999)
    assert (o.float() - ro).abs().max() <= 1e-2 * ro.abs().max()
    assert (lse - rl).abs().max() < 1e-4
    o4, lse4 = torch.empty_like(o), torch.empty_like(lse)
    rc = lib.cb_attn_fwd4(N.ptr(q), N.ptr(k), N.ptr(v), N.ptr(o4), N.ptr(lse4), 4, 1, 3000, 16, 4, 2999,
                          0, 1, 1.0 / math.sqrt(128), 0, N.stream_ptr())
    assert rc == 0, N.last_error()
    assert (o.float() - o4.float()).abs().max() <= 2e-2 * ro.abs().max()
    assert (lse - lse4).abs().max() < 2e-4
    rc = lib.cb_attn_split(N.ptr(q), N.ptr(k), N.ptr(v), N.ptr(o), N.ptr(lse), 4, 1, 3000, 16, 4, 2999,
                           0, 1, C.c_float(0.1), N.ptr(o), C.c_longlong(16), C.c_void_p(0),
                           N.stream_ptr())
    assert rc != 0 and "workspace" in N.last_error()


@pytest.mark.parametrize("causal,kv_offset", [(False, 0), (True, 0), (True, 400)])
def test_persistent_tile_pairs(native_lib, causal, kv_offset):
    """More tile pairs than SMs, so a CTA walks several of different lengths: ragged rows and keys, and
    with kv_offset whole pairs that see no key (zero rows, lse -inf) between ones that do.
    Bounds as for the split-key kernel."""
    import ctypes as C
    import math

    from commbench_b200 import _native as N
    from commbench_b200.ops.cp import reference_attention

    B, Sq, Skv, Hq, Hkv = 2, 700, 300, 64, 4
    q, k, v = _qkv(B, Sq, Skv, Hq, Hkv, 41)
    o, lse = torch.empty_like(q), torch.empty(B, Hq, Sq, device="cuda")
    status = torch.zeros(4, dtype=torch.int32, device="cuda")
    rc = N.load().cb_attn_fwd4(N.ptr(q), N.ptr(k), N.ptr(v), N.ptr(o), N.ptr(lse), B, Sq, Skv, Hq, Hkv,
                               0, kv_offset, int(causal), C.c_float(1.0 / math.sqrt(128)),
                               N.ptr(status), N.stream_ptr())
    assert rc == 0, N.last_error()
    ro, rl = reference_attention(q, k, v, causal=causal, kv_offset=kv_offset)
    assert int(status.abs().sum()) == 0
    assert (o.float() - ro).abs().max() <= 1e-2 * ro.abs().max()
    seen = rl > float("-inf")
    assert torch.equal(lse > float("-inf"), seen)
    assert (lse - rl)[seen].abs().max() < 1e-4


@pytest.mark.parametrize("shape", [(1, 1, 2000, 1, 1), (4, 1, 3000, 16, 4), (2, 4, 5000, 32, 8),
                                   (2, 5, 700, 6, 2)])
def test_split_key_attention_repeats_its_bits(native_lib, shape):
    """Tiles with fewer than 128 rows: what other kernels leave in shared memory where rows are missing
    must not show in the result."""
    from commbench_b200.ops.cp import flash_attention

    B, Sq, Skv, Hq, Hkv = shape
    q, k, v = _qkv(B, Sq, Skv, Hq, Hkv, 23)
    # a full tile of queries with large scores, of another size each time
    others = [_qkv(8, 128, 2048, 8, 8, 29 + i) for i in range(4)]
    ref = flash_attention(q, k, v, q_offset=Skv - Sq)
    for i in range(12):
        qn, kn, vn = others[i % 4]
        flash_attention(qn * float(1 + i), kn, vn, causal=False)
        o, lse = flash_attention(q, k, v, q_offset=Skv - Sq)
        assert torch.equal(o, ref[0]) and torch.equal(lse, ref[1]), i


@pytest.mark.parametrize("given", [True, False])
def test_call_on_a_side_stream_leaves_blocks_of_the_current_stream_alone(native_lib, given):
    """A block that the current stream has freed but still has a copy queued from is not handed to a
    call that runs on another stream, neither as its workspace nor as a result made inside."""
    from commbench_b200 import _native as N
    from commbench_b200.ops.cp import flash_attention

    B, Skv, Hq, Hkv = 4, 3000, 16, 4
    q, k, v = _qkv(B, 1, Skv, Hq, Hkv, 19)
    ref_o, ref_l = flash_attention(q, k, v, q_offset=Skv - 1)
    sizes = [N.load().cb_attn_split_bytes(B, 1, Skv, Hq, Hkv, Skv - 1, 0, 1), ref_o.numel() * 2,
             ref_l.numel() * 4]
    assert min(sizes) > 0
    out, lse = (torch.empty_like(ref_o), torch.empty_like(ref_l)) if given else (None, None)
    side = torch.cuda.Stream()
    for _ in range(3):
        blocks = [torch.full((n,), 0x5a, dtype=torch.uint8, device="cuda") for n in sizes]
        kept = [torch.empty_like(b) for b in blocks]
        torch.cuda.synchronize()
        torch.cuda._sleep(20_000_000)                 # about 10 ms: the copies stay queued behind it
        for a, b in zip(kept, blocks):
            a.copy_(b)
        del a, b, blocks
        o, l = flash_attention(q, k, v, q_offset=Skv - 1, out=out, lse=lse, stream=side)
        torch.cuda.synchronize()
        assert all(bool((x == 0x5a).all()) for x in kept)
        assert torch.equal(o, ref_o) and torch.equal(l, ref_l)


@pytest.mark.parametrize("op", ["ring", "ulysses"])
def test_context_parallel_call_runs_wholly_on_its_stream(native_lib, op):
    """Inputs outside the op's own buffers, with the current stream busy: copies and launch follow
    each other on the given stream and read what that stream was given to wait for."""
    from commbench_b200.ops.cp import RingAttention, UlyssesAttention, reference_attention
    from commbench_b200.runtime.context import CommContext

    ctx = CommContext(heap_bytes=64 << 20)
    attn = (RingAttention if op == "ring" else UlyssesAttention)(ctx, 1, 512, 4, 1)
    side = torch.cuda.Stream()
    for seed in (5, 6):
        q, k, v = _qkv(1, 512, 512, 4, 1, seed)
        ro, _ = reference_attention(q, k, v)
        side.wait_stream(torch.cuda.current_stream())
        torch.cuda._sleep(20_000_000)
        o = attn.forward(q, k, v, stream=side)
        o = o[0] if op == "ring" else o
        side.synchronize()                            # the current stream is still asleep
        with torch.cuda.stream(side):
            assert torch.allclose(o.float(), ro, atol=2e-2, rtol=2e-2)
        torch.cuda.synchronize()
    ctx.check_status()
    ctx.close()


@pytest.mark.parametrize("shape", [(4, 1, 3000, 16, 4), (60, 16, 1501, 128, 8), (2, 130, 1500, 8, 2)])
def test_split_key_workspace_is_two_tiles_per_cta(native_lib, shape):
    """The bytes asked for are enough - nothing behind them is written, the result is right (bounds as
    above) - and do not grow with the batch."""
    import math

    from commbench_b200 import _native as N
    from commbench_b200.ops.cp import reference_attention

    B, Sq, Skv, Hq, Hkv = shape
    q, k, v = _qkv(B, Sq, Skv, Hq, Hkv, 3)
    lib = N.load()
    nbytes = lib.cb_attn_split_bytes(B, Sq, Skv, Hq, Hkv, Skv - Sq, 0, 1)
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    assert 0 < nbytes <= 2 * sms * 128 * 520
    ws = torch.full((nbytes + 4096,), 0xff, dtype=torch.uint8, device="cuda")
    o, lse = torch.empty_like(q), torch.empty(B, Hq, Sq, device="cuda")
    rc = lib.cb_attn_split(q.data_ptr(), k.data_ptr(), v.data_ptr(), o.data_ptr(), lse.data_ptr(), B, Sq,
                           Skv, Hq, Hkv, Skv - Sq, 0, 1, 1.0 / math.sqrt(128), ws.data_ptr(), nbytes,
                           0, N.raw_stream())
    assert rc == 0, N.last_error()
    assert bool((ws[nbytes:] == 0xff).all())
    ro, rl = reference_attention(q, k, v, q_offset=Skv - Sq)
    assert (o.float() - ro).abs().max() <= 1e-2 * ro.abs().max()
    assert (lse - rl).abs().max() < 1e-4


@pytest.mark.parametrize("kv_offset", [0, 900])
def test_tile_pairs_beside_a_kernel_that_holds_sms(native_lib, kv_offset):
    """More tile pairs than SMs while a GEMM on another stream holds some of these: the same bits as
    without it.  With kv_offset some pairs see no key."""
    import math

    from commbench_b200 import _native as N
    from commbench_b200.ops.gemm import gemm

    B, S, Hq, Hkv = 2, 2000, 32, 8
    q, k, v = _qkv(B, S, S, Hq, Hkv, 47)
    status = torch.zeros(4, dtype=torch.int32, device="cuda")
    a = torch.randn(4096, 4096, device="cuda").bfloat16()
    side = torch.cuda.Stream()

    def run():
        o, lse = torch.empty_like(q), torch.empty(B, Hq, S, device="cuda")
        rc = N.load().cb_attn_fwd4(q.data_ptr(), k.data_ptr(), v.data_ptr(), o.data_ptr(), lse.data_ptr(),
                                   B, S, S, Hq, Hkv, 0, kv_offset, 1, 1.0 / math.sqrt(128),
                                   status.data_ptr(), N.raw_stream())
        assert rc == 0, N.last_error()
        return o, lse

    ref = run()
    c = torch.empty(4096, 4096, dtype=torch.bfloat16, device="cuda")
    for n in (1, 8, 100):
        torch.cuda.synchronize()
        gemm(a, a, out=c, bn=256, max_ctas=n, stream=side)
        torch.cuda._sleep(100_000)                    # the GEMM is there first
        for _ in range(3):
            o, lse = run()
            assert torch.equal(o, ref[0]) and torch.equal(lse, ref[1])
    torch.cuda.synchronize()
    assert int(status.abs().sum()) == 0


@pytest.mark.parametrize("s,hq,hkv,split", [(1024, 4, 1, True), (2304, 32, 8, False)])
def test_ring_on_one_real_rank_takes_either_kernel(native_lib, s, hq, hkv, split):
    """One rank of a real context: few query tiles go to the split-key kernel, more tile pairs than SMs
    to the tile-pair kernel, persistent since there is nothing to pull.  Both masks in turn on one object;
    bounds as for the two kernels."""
    from commbench_b200 import _native as N
    from commbench_b200.ops.cp import RingAttention, reference_attention
    from commbench_b200.runtime.context import CommContext

    assert (N.load().cb_attn_split_bytes(1, s, s, hq, hkv, 0, 0, 1) >= 0) == split
    ctx = CommContext(heap_bytes=64 << 20)
    ring = RingAttention(ctx, 1, s, hq, hkv)
    q, k, v = _qkv(1, s, s, hq, hkv, 61)
    for causal in (True, True, False, True):
        o, lse = ring.forward(q, k, v, causal=causal)
        o2, none = ring.forward(q, ring.k_local(), ring.v_local(), causal=causal, want_lse=False)
        ro, rl = reference_attention(q, k, v, causal=causal)
        assert (o.float() - ro).abs().max() <= 1e-2 * ro.abs().max()
        assert (lse - rl).abs().max() < 1e-4
        assert none is None and torch.equal(o, o2)
    ctx.check_status()
    ctx.close()


@pytest.mark.parametrize("shape", [(4, 1, 3000, 16, 4), (1, 1100, 1100, 32, 8)])
def test_attention_in_a_cuda_graph(native_lib, shape):
    """Split-key kernel, its merge and the workspace made inside the call, and the tile-pair kernel with
    more items than SMs, captured and replayed on new inputs: the bits of the plain call."""
    from commbench_b200.ops.cp import flash_attention

    B, Sq, Skv, Hq, Hkv = shape
    q, k, v = _qkv(B, Sq, Skv, Hq, Hkv, 71)
    flash_attention(q, k, v, q_offset=Skv - Sq)
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        o, lse = flash_attention(q, k, v, q_offset=Skv - Sq)
    for seed in range(3):
        for t, x in zip((q, k, v), _qkv(B, Sq, Skv, Hq, Hkv, seed)):
            t.copy_(x)
        graph.replay()
        ro, rl = flash_attention(q, k, v, q_offset=Skv - Sq)
        assert torch.equal(o, ro) and torch.equal(lse, rl)
