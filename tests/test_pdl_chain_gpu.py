"""Kernels that start while the ones before them end: chains whose buffers are overwritten round after round,
called in a row and captured, give the bits that they give with a synchronisation after every call."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _dense(sync):
    """Persistent GEMMs around attention, both ways of splitting it; then a quantiser before each of the two
    block-scaled products.  Every buffer is written again in the next round."""
    from commbench_b200.ops import gemm as G
    from commbench_b200.ops.cp import flash_attention

    g = torch.Generator(device="cuda").manual_seed(1)
    s, h = 1024, 16
    d = h * 128

    def randn(*shape, scale=1.0):
        return (torch.randn(*shape, device="cuda", generator=g) * scale).bfloat16()

    x0, wq, wk, wv, wo = randn(s, d), *(randn(d, d, scale=0.02) for _ in range(4))
    bq, bs = G.quantize_blockscaled(wo, 128)
    mq, _, msf = G.quantize_blockscaled_pow2(wo, 128)
    x, q, k, v, o, y = (torch.empty_like(x0) for _ in range(6))
    lse = torch.empty(1, h, s, device="cuda")

    def round_():
        for w, t in ((wq, q), (wk, k), (wv, v)):
            G.gemm(x, w, out=t, bn=512)
            sync()
        flash_attention(*(t.view(1, s, h, 128) for t in (q, k, v)), out=o.view(1, s, h, 128), lse=lse)
        sync()
        G.gemm(o, wo, out=y, bn=448)
        sync()
        last = slice(s - 8, s)                            # few queries: the split-key kernel
        part, _ = flash_attention(q[last].view(1, 8, h, 128), k.view(1, s, h, 128), v.view(1, s, h, 128),
                                  q_offset=s - 8)
        sync()
        small = G.gemm(part.view(8, d), wo)               # the split-K kernel
        sync()
        yq, ys = G.quantize_blockscaled(y, 1)
        sync()
        G.gemm_fp8_blockscaled(yq, ys, bq, bs, out=q)
        sync()
        zq, _, zsf = G.quantize_blockscaled_pow2(q, 1)
        sync()
        G.gemm_fp8_mx(zq, zsf, mq, msf, out=x)
        sync()
        x[last].add_(small)

    def start():
        x.copy_(x0)

    return start, round_, (x, q, k, v, o, y, lse), []


def _experts(sync):
    """Two expert layers in a row whose weights are rewritten right before each call."""
    from commbench_b200.ops.moe import MoELayer, interleave_gate_up, router_topk
    from commbench_b200.runtime.context import CommContext

    T, H, I, E, K = 24, 512, 512, 8, 2
    g = torch.Generator(device="cuda").manual_seed(2)
    layers = []
    for seed in range(2):
        layer = MoELayer(CommContext(heap_bytes=32 << 20), T, H, I, E, K, seed=seed)
        assert layer.weights_early
        st = layer.states[0]
        sets = []
        for _ in range(2):
            w1 = (torch.randn(st.w1.shape, device="cuda", generator=g) * 0.03).bfloat16()
            sets.append((interleave_gate_up(w1), torch.flip(st.w2, [0]) if sets else st.w2.clone()))
        layers.append((layer, st, sets))
    idx, w = router_topk(torch.randn(T, E, device="cuda", generator=g), K)
    x0 = torch.randn(T, H, device="cuda", generator=g).bfloat16()
    x = torch.empty_like(x0)
    seen = [torch.empty_like(x0) for _ in range(4)]

    def round_():
        for n in range(4):
            layer, st, sets = layers[n % 2]
            st.w1_gated.copy_(sets[n // 2][0])
            st.w2.copy_(sets[n // 2][1])
            sync()
            y = layer.forward(x, idx, w)
            sync()
            seen[n].copy_(y)
            x.add_(y)

    def start():
        x.copy_(x0)

    return start, round_, (x, *seen), [layer.ctx for layer, _, _ in layers]


@pytest.mark.parametrize("captured", [False, True])
@pytest.mark.parametrize("chain", [_dense, _experts])
def test_chain_gives_the_bits_of_single_calls(native_lib, chain, captured):
    results = []
    for sync in (torch.cuda.synchronize, lambda: None):
        start, round_, buffers, contexts = chain(sync)
        start()
        round_()                                          # attributes of the kernels are set outside a capture
        start()
        if captured and results:
            graph = torch.cuda.CUDAGraph()
            torch.cuda.synchronize()
            with torch.cuda.graph(graph):
                round_()
            step = graph.replay
        else:
            step = round_
        start()
        for _ in range(6):
            step()
        torch.cuda.synchronize()
        results.append([t.clone() for t in buffers])
        for ctx in contexts:
            ctx.check_status()
            ctx.close()
    for a, b in zip(*results):
        assert bool(torch.isfinite(a.float()).all())
        assert torch.equal(a.view(torch.uint8), b.view(torch.uint8))
