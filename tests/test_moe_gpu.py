"""MoE kernels: router, layout, and the whole expert-parallel layer with virtual ranks on one
GPU, against plain PyTorch fp32 references."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def test_router_topk_matches_torch(native_lib):
    from commbench_b200.ops.moe import router_topk

    g = torch.Generator(device="cuda").manual_seed(5)
    logits = torch.randn(777, 256, device="cuda", generator=g)
    idx, w = router_topk(logits, 8)
    p = torch.softmax(logits, dim=-1)
    tw, ti = torch.topk(p, 8, dim=-1)
    tw = tw / tw.sum(-1, keepdim=True)
    assert torch.equal(idx.long(), ti)
    assert torch.allclose(w, tw, atol=1e-5, rtol=1e-4)


@pytest.mark.parametrize("T,K,R", [(257, 1, 1), (1024, 2, 2), (4096, 8, 8), (4097, 4, 4)])
def test_dispatch_layout_matches_cpu_reference(native_lib, T, K, R):
    from commbench_b200.ops.moe import dispatch_layout

    E = 32
    g = torch.Generator(device="cuda").manual_seed(T + K)
    # k distinct experts per token; some patterns put several experts on the same rank
    idx = torch.rand(T, E, device="cuda", generator=g).argsort(dim=1)[:, :K].int()
    idx[::7, 0] = -1                      # masked selections are skipped
    per_e, per_r, in_r = dispatch_layout(idx, R, E)
    ci = idx.cpu()
    ref_e = torch.zeros(E, dtype=torch.int32)
    ref_in = torch.zeros(T, R, dtype=torch.bool)
    for k in range(K):
        col = ci[:, k]
        ok = col >= 0
        ref_e += torch.bincount(col[ok].long(), minlength=E).int()
        ref_in[ok.nonzero().squeeze(1), (col[ok] // (E // R)).long()] = True
    assert torch.equal(per_e.cpu(), ref_e)
    assert torch.equal(in_r.cpu(), ref_in)
    assert torch.equal(per_r.cpu(), ref_in.sum(0).int())


@pytest.mark.parametrize("dispatch", ["per_pair", "per_token"])
@pytest.mark.parametrize("fused_swiglu", [True, False])
@pytest.mark.parametrize("world", [1, 2, 4])
def test_moe_layer_virtual_ranks(native_lib, world, fused_swiglu, dispatch):
    from commbench_b200.ops.moe import MoELayer, reference_moe, router_topk
    from commbench_b200.runtime.context import EmuContext

    T, H, I, E, K = 96, 512, 256, 8, 2
    ctx = EmuContext(world)
    layer = MoELayer(ctx, T, H, I, E, K, capacity_factor=float(world) * 2,
                     fused_swiglu=fused_swiglu, dispatch=dispatch)
    assert layer.launches_per_call == (8 if fused_swiglu else 10)
    xs, idxs, ws = [], [], []
    for r in range(world):
        g = torch.Generator(device="cuda").manual_seed(100 + r)
        xs.append(torch.randn(T, H, device="cuda", generator=g).bfloat16())
        i, w = router_topk(torch.randn(T, E, device="cuda", generator=g), K)
        idxs.append(i)
        ws.append(w)
    w1_all = torch.cat([layer.weights(r)[0] for r in range(world)])
    w2_all = torch.cat([layer.weights(r)[1] for r in range(world)])
    for it in range(2):     # second call: counters and flags were reset by the first
        ys = layer.forward(xs, idxs, ws)
        ctx.check_status()
        for r in range(world):
            ref = reference_moe(xs[r], idxs[r], ws[r], w1_all, w2_all, I)
            err = (ys[r].float() - ref).abs().max().item()
            scale = ref.abs().max().item() + 1e-6
            assert err / scale < 3e-2, (it, r, err, scale)
        # the receive kernel re-armed its own counters (no fill launch between two calls)
        for st in layer.states:
            assert int(layer._local(layer.arrived, st).view(torch.int32).abs().sum()) == 0
            assert int(st.recv_ctas.abs().sum()) == 0
            assert int(layer._local(layer.done, st).view(torch.int32).abs().sum()) == 0
    # the two optional bias inputs of the combine reduction (shared expert / residual)
    b0 = [torch.randn(T, H, device="cuda").bfloat16() for _ in range(world)]
    b1 = [torch.randn(T, H, device="cuda").bfloat16() for _ in range(world)]
    ys = layer.forward(xs, idxs, ws, bias0=b0, bias1=b1)
    ctx.check_status()
    for r in range(world):
        ref = reference_moe(xs[r], idxs[r], ws[r], w1_all, w2_all, I) + b0[r].float() + b1[r].float()
        err = (ys[r].float() - ref).abs().max().item()
        assert err / (ref.abs().max().item() + 1e-6) < 3e-2, (r, err)


@pytest.mark.parametrize("n,E", [(100, 4), (4096 * 8, 256), (777, 33)])
def test_expert_sort_is_a_stable_sort(native_lib, n, E):
    from commbench_b200.ops.moe import expert_sort

    g = torch.Generator(device="cuda").manual_seed(n)
    idx = torch.randint(0, E, (n,), device="cuda", generator=g, dtype=torch.int32)
    idx[::11] = -1
    sp, counts = expert_sort(idx, E)
    valid = (idx >= 0).nonzero().squeeze(1)
    order = valid[torch.sort(idx[valid].long(), stable=True).indices]
    assert torch.equal(sp[:order.numel()].long(), order)
    assert bool((sp[order.numel():] == -1).all())
    assert torch.equal(counts.long(), torch.bincount(idx[valid].long(), minlength=E))


@pytest.mark.parametrize("dispatch", ["per_pair", "per_token"])
@pytest.mark.parametrize("T,H,K,world", [(1, 256, 1, 1), (33, 2304, 5, 2), (19, 7168, 8, 1),
                                         (9, 1024, 40, 2)])
def test_moe_dispatch_edges(native_lib, T, H, K, world, dispatch):
    """Dispatch kernel at its edges: one token, hidden sizes of one, several and a ragged number
    of 1024-column slices, more than 32 selections, masked and repeated experts; rows for the own
    rank go straight to the GEMM input, the others through the fp8 buffers.  3e-2 of the largest
    value, as in the layer test above."""
    from commbench_b200.ops.moe import MoELayer, reference_moe
    from commbench_b200.runtime.context import EmuContext

    I, E = 256, 8
    ctx = EmuContext(world)
    layer = MoELayer(ctx, T, H, I, E, K, capacity_factor=2.0 * world, dispatch=dispatch)
    w1_all = torch.cat([layer.weights(r)[0] for r in range(world)])
    w2_all = torch.cat([layer.weights(r)[1] for r in range(world)])
    g = torch.Generator(device="cuda").manual_seed(T + H)
    xs = [torch.randn(T, H, device="cuda", generator=g).bfloat16() for _ in range(world)]
    idxs = [torch.randint(0, E, (T, K), device="cuda", generator=g, dtype=torch.int32)
            for _ in range(world)]
    ws = [torch.rand(T, K, device="cuda", generator=g) + 0.1 for _ in range(world)]
    for idx in idxs:
        idx[::3, K - 1] = -1
    for _ in range(2):
        ys = layer.forward(xs, idxs, ws)
    ctx.check_status()
    for r in range(world):
        wr = torch.where(idxs[r] >= 0, ws[r], torch.zeros_like(ws[r]))
        ref = reference_moe(xs[r], idxs[r], wr, w1_all, w2_all, I)
        err = (ys[r].float() - ref).abs().max().item()
        assert err / (ref.abs().max().item() + 1e-6) < 3e-2, (r, err)


@pytest.mark.parametrize("dispatch", ["per_pair", "per_token"])
def test_moe_layer_on_one_real_rank(native_lib, dispatch):
    """A context of one real rank takes its own counts as the count matrix (no gather, one launch less).
    3e-2 of the largest value, as in the layer test above."""
    from commbench_b200.ops.moe import MoELayer, reference_moe, router_topk
    from commbench_b200.runtime.context import CommContext

    T, H, I, E, K = 96, 512, 256, 8, 2
    ctx = CommContext(heap_bytes=64 << 20)
    layer = MoELayer(ctx, T, H, I, E, K, dispatch=dispatch)
    assert layer.launches_per_call == 7
    w1, w2 = layer.weights()
    for seed in range(3):
        g = torch.Generator(device="cuda").manual_seed(seed)
        x = torch.randn(T, H, device="cuda", generator=g).bfloat16()
        idx, w = router_topk(torch.randn(T, E, device="cuda", generator=g), K)
        y = layer.forward(x, idx, w)
        ref = reference_moe(x, idx, w, w1, w2, I)
        assert (y.float() - ref).abs().max() <= 3e-2 * ref.abs().max()
    ctx.check_status()
    ctx.close()


@pytest.mark.parametrize("fused_swiglu", [True, False])
@pytest.mark.parametrize("narrow", [False, True])
def test_grouped_gemm_forms_at_ragged_row_counts(native_lib, narrow, fused_swiglu):
    """Experts with 0, 1, 31 ... 385 rows, tiles of 256 and of 128 columns, weights fetched before the wait for
    the kernel before and after it."""
    from commbench_b200.ops.moe import MoELayer, reference_moe
    from commbench_b200.runtime.context import CommContext

    counts = [1, 31, 32, 0, 33, 127, 128, 129, 255, 256, 257, 385]
    E, H, I, T = len(counts), 512, 512, sum(counts)
    g = torch.Generator(device="cuda").manual_seed(11)
    idx = torch.repeat_interleave(torch.arange(E), torch.tensor(counts)).int()[torch.randperm(T)]
    idx = idx.view(T, 1).cuda()
    w = torch.rand(T, 1, device="cuda", generator=g) + 0.5
    x = torch.randn(T, H, device="cuda", generator=g).bfloat16()
    ctx = CommContext(heap_bytes=64 << 20)
    layer = MoELayer(ctx, T, H, I, E, 1, seed=3, fused_swiglu=fused_swiglu)
    layer.narrow_up = layer.narrow_down = layer.weights_early = narrow
    w1, w2 = layer.weights()
    ref = reference_moe(x, idx, w, w1, w2, I)
    for _ in range(2):
        y = layer.forward(x, idx, w).float()
        torch.cuda.synchronize()
        ctx.check_status()
        # bf16 roundings of the two products, as in the layer's other tests
        assert (y - ref).abs().max().item() < 3e-2 * ref.abs().max().item()
    for layer.narrow_up in (False, True):
        for layer.weights_early in (False, True):
            layer.narrow_down = not layer.narrow_up
            assert torch.equal(layer.forward(x, idx, w).float(), y)    # same K order: the same bits
    torch.cuda.synchronize()
    ctx.close()


@pytest.mark.parametrize("narrow", [False, True])
def test_weights_in_the_default_gate_up_order(native_lib, narrow):
    """interleave_gate_up's default order is the one that the gated product reads, whatever its tile width.
    3e-2 of the largest value, as in the layer tests above."""
    from commbench_b200.ops.moe import MoELayer, interleave_gate_up, reference_moe, router_topk
    from commbench_b200.runtime.context import CommContext

    T, H, I, E, K = 40, 512, 768, 8, 2
    ctx = CommContext(heap_bytes=64 << 20)
    layer = MoELayer(ctx, T, H, I, E, K, seed=5)
    layer.narrow_up = narrow
    g = torch.Generator(device="cuda").manual_seed(6)
    w1, w2 = layer.weights()
    w1.copy_(torch.randn(w1.shape, device="cuda", generator=g) * 0.02)
    layer.states[0].w1_gated = interleave_gate_up(w1)
    x = torch.randn(T, H, device="cuda", generator=g).bfloat16()
    idx, w = router_topk(torch.randn(T, E, device="cuda", generator=g), K)
    y = layer.forward(x, idx, w)
    ref = reference_moe(x, idx, w, w1, w2, I)
    assert (y.float() - ref).abs().max() <= 3e-2 * ref.abs().max()
    ctx.check_status()
    ctx.close()
