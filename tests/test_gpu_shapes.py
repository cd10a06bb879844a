"""Edges of the tile shapes and dispatch rules: remainders, the smallest and the largest of each kernel variant's range."""
import numpy as np
import pytest

from conftest import rel_err

pytestmark = pytest.mark.gpu

F32_TOL = 1e-5


# The f32 products: 32-, 64- and 128-wide tiles around their edges, k around the slab length and split over a cluster, row
# pitches that rule out 16-byte copies (odd k or n), few rows, few columns.
@pytest.mark.parametrize("m,k,n", [(1, 1, 1), (31, 63, 33), (33, 65, 31), (64, 32, 64), (65, 96, 63), (300, 192, 576), (2048, 64, 8),
                                   (64, 2048, 64), (65, 2050, 12), (1100, 200, 1030), (130, 4097, 129)])
@pytest.mark.parametrize("mode", ["NN", "TN", "NT"])
def test_f32_product_tile_edges(gpu, m, k, n, mode):
    import torch
    import asca_b200
    from asca_b200 import ops

    g = torch.Generator(device="cuda").manual_seed(m + 7 * k + 13 * n)
    a, b = (torch.randn(*s, generator=g, device="cuda") for s in ((m, k), (k, n)))
    bias, c0 = torch.randn(n, generator=g, device="cuda"), torch.randn(m, n, generator=g, device="cuda")
    out = c0.clone()
    ops.gemm(gpu, a.t().contiguous() if mode == "TN" else a, b.t().contiguous() if mode == "NT" else b, getattr(asca_b200, mode), bias=bias,
             out=out, accumulate=True)
    gpu.sync()
    ref = a.double() @ b.double() + bias.double() + c0.double()
    assert rel_err(out.cpu().numpy(), ref.cpu().numpy()) < F32_TOL


# The grouped f32 products of the expert layer: empty experts, experts of one token, ragged tiles, widths that are no
# multiple of four.
@pytest.mark.parametrize("n,d,F,E,vocab", [(1, 64, 128, 4, 256), (33, 48, 30, 8, 3), (257, 30, 66, 5, 256), (1500, 192, 384, 8, 256)])
def test_f32_expert_products_tile_edges(orc, gpu, n, d, F, E, vocab):
    g = np.random.default_rng(n)
    ids = g.integers(0, vocab, n).astype(np.uint32)
    xn, dout = (g.standard_normal((n, d)).astype(np.float32) for _ in range(2))
    w1, w2 = (g.standard_normal(s).astype(np.float32) * 0.1 for s in ((d, E * F), (E * F, d)))
    b1, b2 = (g.standard_normal(s).astype(np.float32) * 0.1 for s in (E * F, d))
    ref_out, pre, hid = orc.moe_ffn_forward(xn, w1, b1, w2, b2, ids, F, E, want_cache=True)
    want = orc.moe_ffn_backward(xn, w1, w2, pre, hid, ids, dout, F, E)
    out, dev = gpu.moe_forward_dev(xn, w1, b1, w2, b2, ids, F)
    r = gpu.moe_bwd_dev(dev, dout)
    assert rel_err(out, ref_out) < F32_TOL
    for got, ref in zip((r.d_w1, r.d_b1, r.d_w2, r.d_b2, r.dxn), want):
        assert rel_err(got, ref) < F32_TOL


# f32 decode: every cluster width (1 .. 8 CTAs a stream), head dims, more CTAs than heads and the other way round, hidden and
# vocabulary slices that leave CTAs without work, and the two shapes that fall back to single kernels (an odd number of heads;
# states too large for shared memory).
@pytest.mark.parametrize("cfg,ns", [((256, 64, 4, 2, 4, 256), 1), ((256, 64, 4, 2, 4, 256), 70), ((256, 96, 6, 1, 8, 20), 3),
                                    ((256, 192, 6, 3, 8, 640), 19), ((48, 64, 2, 2, 3, 36), 150), ((256, 128, 1, 2, 2, 64), 2),
                                    ((256, 256, 4, 1, 2, 128), 40), ((256, 80, 5, 2, 4, 64), 3), ((256, 512, 4, 12, 2, 64), 2)])
def test_f32_decode_cluster_widths_and_fallbacks(orc, gpu, cfg, ns):
    import asca_b200

    V = cfg[0]
    ref = orc.Model(*cfg)
    ref.params[:] = orc.Rng(sum(cfg)).normal(ref.n, 0.8 * cfg[1] ** -0.5)
    dev = asca_b200.Model(gpu, *cfg)
    dev.set_params(ref.params)
    ids = orc.Rng(ns).below(V, ns)
    state = dev.new_decode_state(ns)
    toks = dev.decode_greedy(state, ids.copy(), 3)
    logits, nxt = dev.decode_step(state, toks[-1].copy())
    for s in sorted({0, ns // 2, ns - 1}):
        st, tok = ref.new_decode_state(), ids[s]
        for t in range(3):
            lg = ref.step(tok, st)
            tok = int(lg.argmax())
            assert tok == toks[t, s]
        lg = ref.step(tok, st)
        assert rel_err(logits[s:s + 1], lg) < F32_TOL and nxt[s] == lg.argmax()
        assert rel_err(state[:, s].cpu().numpy(), st) < F32_TOL
    dev.free()
