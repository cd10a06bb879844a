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


# f32 decode past one wave of streams: where a launch of its own for every stream costs more than the batched step, the call takes
# the batched step (two steps a call: from the fifth wave of 148 streams on at d 64, from the second at d 256); the same tokens, logits
# and states on both sides of the line.
@pytest.mark.parametrize("cfg,ns,steps,one", [((256, 64, 4, 2, 4, 256), 148, 2, True), ((256, 64, 4, 2, 4, 256), 592, 2, True),
                                              ((256, 64, 4, 2, 4, 256), 593, 2, False), ((256, 256, 4, 2, 4, 512), 148, 2, True),
                                              ((256, 256, 4, 2, 4, 512), 149, 2, False)])
def test_f32_decode_more_streams_than_fit_at_once(orc, gpu, cfg, ns, steps, one):
    import asca_b200

    V = cfg[0]
    ref = orc.Model(*cfg)
    ref.params[:] = orc.Rng(sum(cfg)).normal(ref.n, 0.8 * cfg[1] ** -0.5)
    dev = asca_b200.Model(gpu, *cfg)
    dev.set_params(ref.params)
    ids = orc.Rng(ns).below(V, ns)
    state = dev.new_decode_state(ns)
    before = gpu.launch_count()
    toks = dev.decode_greedy(state, ids.copy(), steps)
    assert (gpu.launch_count() - before == 1) == one
    logits, nxt = dev.decode_step(state, toks[-1].copy())
    for s in sorted({0, ns // 2, ns - 1}):
        st, tok = ref.new_decode_state(), ids[s]
        for t in range(steps):
            tok = int(ref.step(tok, st).argmax())
            assert tok == toks[t, s]
        lg = ref.step(tok, st)
        assert rel_err(logits[s:s + 1], lg) < F32_TOL and nxt[s] == lg.argmax()
        assert rel_err(state[:, s].cpu().numpy(), st) < F32_TOL
    dev.free()


# Logits that do not compare (a head of NaNs, or all of them -inf): the choice is token 0, in every form of the step, and the next step
# reads that row of the embedding and no other.
@pytest.mark.parametrize("cfg,ns,mode", [((256, 64, 4, 1, 4, 64), 3, "F32"), ((256, 80, 5, 1, 4, 64), 3, "F32"), ((256, 128, 2, 1, 4, 64), 5, "BF16"),
                                         ((256, 128, 2, 1, 4, 64), 300, "BF16"), ((256, 128, 1, 1, 4, 64), 5, "BF16")])
@pytest.mark.parametrize("bad", [float("nan"), float("-inf")])
def test_greedy_choice_without_a_largest_logit(orc, gpu, cfg, ns, mode, bad):
    import asca_b200

    m = asca_b200.Model(gpu, *cfg)
    params = np.abs(orc.Rng(5).normal(m.n, 0.1)) + 0.01   # positive throughout: -inf weights give -inf logits
    V, d = cfg[:2]
    params[V * d:2 * V * d] = bad
    m.set_params(params)
    m.set_compute(getattr(asca_b200, mode))
    ids = orc.Rng(6).below(V, ns)
    for _ in range(3):
        st = m.new_decode_state(ns)
        assert not m.decode_greedy(st, ids.copy(), 3).any()
        assert not m.decode_step(st, ids.copy())[1].any() and bool(st.isfinite().all())
    assert not m.prefill(m.new_decode_state(ns), np.tile(ids[:, None], (1, 5)))[1].any()
    m.free()


# The f32 recurrence with one, two and four value columns per lane group (few chains to many), ragged stages, decay strong enough
# to be folded in step by step, and the three-kernel backward with every width of its chain kernel.
@pytest.mark.parametrize("B,T,H,dh", [(1, 1, 1, 16), (2, 33, 2, 16), (40, 70, 20, 16), (1, 65, 1, 32), (60, 40, 20, 32), (130, 16, 20, 32),
                                      (3, 64, 2, 64), (20, 50, 8, 64), (40, 129, 8, 64), (1, 130, 1, 128), (6, 24, 8, 128), (12, 80, 8, 128)])
@pytest.mark.parametrize("decay", [2.0, -3.0])
def test_f32_delta_column_splits(orc, gpu, B, T, H, dh, decay):
    import torch
    from asca_b200 import ops

    g = np.random.default_rng(B + T + dh)
    n, d = B * T, H * dh
    q, k, v, d_o = (g.standard_normal((n, d)).astype(np.float32) for _ in range(4))
    qn, kn = (np.linalg.norm(x.reshape(n, H, dh), axis=-1).astype(np.float32) for x in (q, k))
    q, k = ((x.reshape(n, H, dh) / xn[..., None]).reshape(n, d).astype(np.float32) for x, xn in ((q, qn), (k, kn)))
    alpha = (1 / (1 + np.exp(-(decay + 0.5 * g.standard_normal((n, H)))))).astype(np.float32)
    beta = (1 / (1 + np.exp(-g.standard_normal((n, H))))).astype(np.float32)
    tq, tk, tv, ta, tb, tqn, tkn, tdo = (torch.from_numpy(x).cuda() for x in (q, k, v, alpha, beta, qn, kn, d_o))
    o, s_fin, ckpt = ops.delta_fwd(gpu, tq, tk, tv, ta, tb, B, T, H, dh, want_final=True)
    d_qkv, d_gate = ops.delta_bwd(gpu, tq, tk, tv, ta, tb, tqn, tkn, tdo, ckpt, B, T, H, dh)
    gpu.sync()
    b = B - 1   # the last sequence of the batch stands for all: sequences are independent
    rows = slice(b * T, B * T)
    o_ref, s_ref = orc.delta_scan(q[rows], k[rows], v[rows], alpha[rows], beta[rows], 1, T, H, dh)[:2]
    dq_ref, dg_ref = orc.delta_bptt(q[rows], k[rows], v[rows], alpha[rows], beta[rows], qn[rows], kn[rows], d_o[rows], 1, T, H, dh)
    assert rel_err(o[rows].cpu().numpy(), o_ref) < F32_TOL
    assert rel_err(s_fin[b].cpu().numpy(), s_ref.reshape(H, dh, dh)) < F32_TOL
    assert rel_err(d_qkv[rows].cpu().numpy(), dq_ref) < F32_TOL
    assert rel_err(d_gate[rows].cpu().numpy(), dg_ref) < F32_TOL


# The state buffers of the f32 forward may start at any float, in every split of the value columns.
@pytest.mark.parametrize("B,H,dh", [(2, 2, 32), (30, 20, 32), (80, 20, 32), (20, 8, 64), (40, 8, 64), (2, 8, 128), (6, 8, 128), (12, 8, 128)])
def test_f32_delta_forward_unaligned_states(gpu, B, H, dh):
    import ctypes as C
    import torch

    g = torch.Generator(device="cuda").manual_seed(B + dh)
    T, n, size = 70, B * 70, B * H * dh * dh
    q, k, v = (torch.randn(n, H * dh, generator=g, device="cuda") * dh ** -0.5 for _ in range(3))
    alpha, beta = (torch.sigmoid(torch.randn(n, H, generator=g, device="cuda")) for _ in range(2))
    s0 = torch.randn(size, generator=g, device="cuda")
    got = []
    for off in (0, 1):
        init, fin, ck = (torch.zeros(m + 8, device="cuda") for m in (size, size, 2 * size))
        init[off:off + size] = s0
        o = torch.empty_like(q)
        torch.cuda.synchronize()
        ptr = lambda t: t.data_ptr() + 4 * off  # noqa: E731
        i64 = C.c_int64
        gpu._call("asca_delta_fwd", gpu._ctx, *(C.c_void_p(t.data_ptr()) for t in (q, k, v, alpha, beta)), i64(B), i64(T), i64(H), i64(dh), i64(64),
                  C.c_int(0), C.c_void_p(o.data_ptr()), C.c_void_p(ptr(init)), C.c_void_p(ptr(fin)), C.c_void_p(ptr(ck)))
        gpu.sync()
        got.append((o, fin[off:off + size].clone(), ck[off:off + 2 * size].clone()))
        assert not fin[off + size:].any() and not ck[off + 2 * size:].any()
    assert all(torch.equal(a, b) for a, b in zip(*got))


# The f32 backward where its chunks do not fit the scratch of one launch (27,473 tiles at dh 16, 8,923 at dh 128): segments of one
# long chain, segments of many chains, groups of chains, both, and a device without room for any of it (the single kernel). The
# scratch stays below 1.6 GB; the reference is the single kernel on checkpoints every 32 tokens (both are held to F32_TOL of the
# oracle, so twice that between them).
@pytest.mark.parametrize("B,T,H,dh,left", [(1, 27483 * 64 - 5, 1, 16, None), (60, 32 * 64 - 1, 16, 16, None), (150, 19 * 64, 16, 16, None),
                                           (150, 33 * 64 + 7, 16, 16, None), (2, 4500 * 64 + 1, 1, 128, None), (60, 32 * 64 - 1, 16, 16, 64 << 20),
                                           (60, 32 * 64 - 1, 16, 16, 600 << 20)])
def test_f32_delta_backward_in_bounded_scratch(gpu, B, T, H, dh, left):
    import ctypes as C
    import torch
    from asca_b200 import ops

    g = torch.Generator(device="cuda").manual_seed(B + T)
    n, d = B * T, H * dh
    norm = lambda *shape: torch.randn(*shape, generator=g, device="cuda")  # noqa: E731
    q, k = norm(n, H, dh), norm(n, H, dh)
    qn, kn = q.norm(dim=-1), k.norm(dim=-1)
    q, k = ((x / xn[..., None]).reshape(n, d) for x, xn in ((q, qn), (k, kn)))
    v, d_o = norm(n, d), norm(n, d)
    alpha, beta = torch.sigmoid(4 + norm(n, H)), torch.sigmoid(norm(n, H))   # decay slow enough to cross segments
    ckpt = ops.delta_fwd(gpu, q, k, v, alpha, beta, B, T, H, dh, chunk=32)[2]
    want = ops.delta_bwd(gpu, q, k, v, alpha, beta, qn, kn, d_o, ckpt, B, T, H, dh, chunk=32)
    ckpt = ops.delta_fwd(gpu, q, k, v, alpha, beta, B, T, H, dh)[2]
    got = [torch.empty_like(x) for x in want]
    torch.cuda.empty_cache()
    gpu._call("asca_ctx_trim", gpu._ctx)
    before, hog = torch.cuda.mem_get_info()[0], C.c_void_p()
    if left:
        gpu._call("asca_malloc", gpu._ctx, C.c_size_t(before - left), C.byref(hog))
    gpu.profile(True)
    ops.delta_bwd(gpu, q, k, v, alpha, beta, qn, kn, d_o, ckpt, B, T, H, dh, d_qkv=got[0], d_gate=got[1])
    kernels = [name for name, _ in gpu.profile_read()]
    gpu.profile(False)
    used = before - torch.cuda.mem_get_info()[0]
    if left:
        gpu._call("asca_free", gpu._ctx, hog)
        gpu._call("asca_ctx_trim", gpu._ctx)
        assert kernels == ["delta_bwd_kernel"] if left == 64 << 20 else kernels.count("delta_bwd_chain_kernel") > 4
    else:
        assert used < 1600 << 20 and kernels.count("delta_bwd_chain_kernel") > 1
    for a, b in zip(got, want):
        assert float((a - b).abs().max() / b.abs().max()) < 2 * F32_TOL


# Buffers off the 16-byte grid where the aligned ones move 16 bytes at a time: same results from rows moved, AdamW, the bf16 expert layer
# (which leaves the tensor cores for it) and the bf16 recurrence's final state; its d_qkv is refused.
def test_unaligned_device_buffers(gpu):
    import ctypes as C
    import torch
    import asca_b200
    from asca_b200 import ops

    g = torch.Generator(device="cuda").manual_seed(3)
    norm = lambda *s: torch.randn(*s, generator=g, device="cuda")  # noqa: E731
    i64, vp = C.c_int64, lambda t: C.c_void_p(t.data_ptr())  # noqa: E731

    def off(t):   # the same values one element further on
        buf = torch.empty(t.numel() + 8, dtype=t.dtype, device="cuda")
        buf[1:1 + t.numel()] = t.reshape(-1)
        return buf[1:1 + t.numel()].reshape(t.shape)

    src, idx = norm(50, 64), torch.randperm(50, generator=g, device="cuda").int()
    for call in ("asca_gather_rows", "asca_scatter_rows"):
        dst = [torch.zeros(50, 64, device="cuda"), off(torch.zeros(50, 64, device="cuda"))]
        torch.cuda.synchronize()
        for s, d in zip((src, off(src)), dst):
            gpu._call(call, gpu._ctx, vp(s), vp(idx), i64(50), i64(64), vp(d))
        gpu.sync()
        assert torch.equal(*dst) and dst[0].any()

    p, m, v, gr = norm(1003), norm(1003), norm(1003).abs(), norm(1003)
    both = [[t.clone() for t in (p, gr, m, v)], [off(t) for t in (p, gr, m, v)]]
    torch.cuda.synchronize()
    for a in both:
        gpu._call("asca_adamw", gpu._ctx, *(vp(t) for t in a), i64(1003), *(C.c_float(x) for x in (1e-2, 0.9, 0.95, 1e-8, 1e-3)))
    gpu.sync()
    # (the two loops may contract other multiply-add pairs: a few units of 2^-24 on values of order one)
    assert all(rel_err(b.cpu().numpy(), a.cpu().numpy()) < 1e-6 for a, b in zip(*both)) and not torch.equal(both[0][0], p)

    n, d, F, E = 300, 128, 192, 4
    xn, w1, w2 = norm(n, d).bfloat16(), norm(d, E * F).mul(0.1).bfloat16(), norm(E * F, d).mul(0.1).bfloat16()
    b1, b2, dout = norm(E * F), norm(d), norm(n, d)
    perm, offs = ops.moe_dispatch(gpu, torch.randint(0, 99, (n,), generator=g, device="cuda", dtype=torch.int32), E)
    got = []
    for x, do in ((xn, dout), (off(xn), dout), (xn, off(dout))):
        out, pre, hid = ops.moe_fwd(gpu, x, w1, b1, w2, b2, perm, offs, F, E)
        got.append((out, *ops.moe_bwd(gpu, x, w1, w2, pre, hid, do, perm, offs, F, E)))
    gpu.sync()
    for other in got[1:]:
        for a, b in zip(got[0], other):
            assert rel_err(b.cpu().numpy(), a.cpu().numpy()) < 2e-2

    B, T, H, dh = 2, 130, 2, 64
    q, k, v, d_o = (torch.nn.functional.normalize(norm(B * T, H, dh), dim=-1).reshape(B * T, H * dh).bfloat16() for _ in range(4))
    alpha, beta, qn = torch.sigmoid(2 + norm(B * T, H)), torch.sigmoid(norm(B * T, H)), torch.ones(B * T, H, device="cuda")
    fins = [torch.zeros(B, H, dh, dh, device="cuda"), off(torch.zeros(B, H, dh, dh, device="cuda"))]
    o, ckpt = torch.empty_like(q), torch.empty(ops.delta_ckpt_floats(gpu, B, T, H, dh, 64), device="cuda")
    torch.cuda.synchronize()
    for fin in fins:
        gpu._call("asca_delta_fwd", gpu._ctx, *(vp(t) for t in (q, k, v, alpha, beta)), i64(B), i64(T), i64(H), i64(dh), i64(64),
                  C.c_int(asca_b200.BF16), vp(o), None, vp(fin), vp(ckpt))
    gpu.sync()
    assert torch.equal(*fins) and fins[0].any()
    d_gate = torch.empty(B * T, 2 * H, device="cuda")
    with pytest.raises(asca_b200.AscaError, match="d_qkv must be 16-byte aligned"):
        gpu._call("asca_delta_bwd", gpu._ctx, *(vp(t) for t in (q, k, v, alpha, beta, qn, qn, d_o, ckpt)), i64(B), i64(T), i64(H), i64(dh), i64(64),
                  C.c_int(asca_b200.BF16), vp(off(torch.empty(B * T, 3 * H * dh, device="cuda"))), vp(d_gate))


# The one-kernel dispatch up to its limits (16,384 tokens, 256 experts) and just past them.
@pytest.mark.parametrize("n,e", [(1, 1), (32, 4), (33, 256), (1025, 7), (16384, 64), (16384, 256), (16385, 64), (2000, 257)])
def test_dispatch_small_and_past_it(orc, gpu, n, e):
    ids = np.random.default_rng(n + e).integers(0, 4096, n).astype(np.uint32)
    for got, want in zip(gpu.moe_dispatch(ids, e), orc.moe_dispatch(ids, e)):
        assert np.array_equal(got, want)


# A repeated f32 training step is replayed as a graph from its third call on: same losses and gradients, bit for bit, as the
# direct launches (a gradient hook keeps those), with a second shape and an accumulating backward in between.
def test_f32_training_step_graph_equals_direct_launches(orc, gpu):
    import asca_b200

    cfg = (256, 64, 4, 2, 4, 256)
    params = orc.Rng(5).normal(331408, 0.02)
    runs = []
    for hooked in (False, True):
        m = asca_b200.Model(gpu, *cfg)
        m.set_params(params)
        if hooked:
            m.set_grad_hook(lambda off, cnt: None)
        out = []
        for step in range(6):
            m.zero_grads()
            for B, T in ((4, 96), (2, 130)):
                ids, tg = (orc.Rng(100 * step + s).below(256, B * T) for s in (1, 2))
                out.append(m.forward_backward(ids, tg, B))
            out.append(m.get()[1])
            m.adamw_step(1e-3)
        runs.append(out)
        m.free()
    for a, b in zip(*runs):
        assert np.array_equal(a, b)


# The replay survives a scratch that moves: given back by a trim (between any two steps), or grown by another call.
@pytest.mark.parametrize("before", [1, 2, 4])
@pytest.mark.parametrize("how", ["trim", "grow"])
def test_f32_training_step_graph_after_the_scratch_moved(orc, gpu, before, how):
    import asca_b200

    m = asca_b200.Model(gpu, 256, 64, 4, 2, 4, 256)
    m.set_params(orc.Rng(5).normal(m.n, 0.02))
    ids, tg = (orc.Rng(s).below(256, 384) for s in (1, 2))
    gpu._call("asca_ctx_trim", gpu._ctx)

    def step():
        n = gpu.graph_launch_count()
        m.zero_grads()
        loss = m.forward_backward(ids, tg, 4)
        return gpu.graph_launch_count() - n, loss, m.get()[1]

    first = [step() for _ in range(before)]
    assert [n for n, _, _ in first] == [0, 0, 1, 1][:before]
    if how == "trim":
        gpu._call("asca_ctx_trim", gpu._ctx)
    else:   # a far larger expert layer takes a far larger scratch
        x = np.zeros((20000, 256), np.float32)
        _, dev = gpu.moe_forward_dev(x, np.zeros((256, 1024), np.float32), np.zeros(1024, np.float32), np.zeros((1024, 256), np.float32),
                                     np.zeros(256, np.float32), np.zeros(20000, np.uint32), 512)
        gpu.moe_bwd_dev(dev, x)
        dev.free()
    after = [step() for _ in range(4)]
    assert after[0][0] == 0 and after[-1][0] == 1
    for _, loss, g in after:
        assert loss == first[0][1] and np.array_equal(g, first[0][2])
    m.free()


# A trim gives back what the replayed steps hold (a training plan of 80 MB, a decode plan), and both go on afterwards with the
# results they had; a model may go before or after the context that its plans came from.
def test_trim_gives_back_the_replayed_steps(orc, gpu):
    import torch
    import asca_b200

    ids, tg = (orc.Rng(s).below(256, 8192) for s in (1, 2))

    def work(m, st):
        st.zero_()
        m.set_compute(asca_b200.F32)
        m.zero_grads()
        out = [m.forward_backward(ids, tg, 16), m.get()[1]]
        m.set_compute(asca_b200.BF16)
        return out + [m.decode_greedy(st, ids[:64].copy(), 40)]

    def free():
        gpu._call("asca_ctx_trim", gpu._ctx)
        return torch.cuda.mem_get_info()[0]

    for rest in range(2):   # (the first round loads the kernels)
        m = asca_b200.Model(gpu, 256, 128, 2, 2, 4, 256)
        m.set_params(orc.Rng(5).normal(m.n, 0.05))
        st = m.new_decode_state(64)
        first = work(m, st)
        before = free()
        n = gpu.graph_launch_count()
        for _ in range(3):
            work(m, st)
        assert gpu.graph_launch_count() > n + 40
        if rest:
            assert before - free() < 16 << 20
        for a, b in zip(first, work(m, st)):
            assert np.array_equal(a, b)
        m.free()

    for model_first in (True, False):
        g2 = asca_b200.Gpu(0)
        m = asca_b200.Model(g2, 256, 64, 4, 1, 2, 64)
        m.set_params(orc.Rng(5).normal(m.n, 0.05))
        for _ in range(4):
            loss = m.forward_backward(ids[:64], tg[:64], 1)
        assert g2.graph_launch_count() > 0 and np.isfinite(loss)
        (m.free if model_first else g2.close)()
        (g2.close if model_first else m.free)()


# A bf16 decode step takes the buffers of its own form only: no f32 pre-activations (16 MB here) beside the packed products.
def test_bf16_decode_takes_the_buffers_of_its_form(orc, gpu):
    import torch
    import asca_b200

    m = asca_b200.Model(gpu, 256, 128, 2, 1, 4, 16384)
    m.set_params(orc.Rng(9).normal(m.n, 0.02))
    m.set_compute(asca_b200.BF16)
    st, ids = m.new_decode_state(256), orc.Rng(3).below(256, 256)
    m.decode_step(st, ids)   # loads the kernels, makes the weight copies
    gpu._call("asca_ctx_trim", gpu._ctx)
    before = torch.cuda.mem_get_info()[0]
    m.decode_step(st, ids)
    assert before - torch.cuda.mem_get_info()[0] < 16 << 20
    m.free()


# Where the projection's epilogue writes q, k and v, the f32 qkv matrix (50 MB here) is not allocated.
@pytest.mark.parametrize("what", ["train", "prefill"])
def test_fused_qkv_allocates_no_f32_matrix(orc, gpu, what):
    import torch
    import asca_b200

    m = asca_b200.Model(gpu, 256, 256, 2, 1, 4, 256)
    m.set_params(orc.Rng(9).normal(m.n, 0.05))
    m.set_compute(asca_b200.BF16)
    ids = orc.Rng(3).below(256, 16384)
    used = {}
    for fused in (False, True, False, True):   # (the first two load the kernels)
        m.set_fused_qkv(fused)
        gpu._call("asca_ctx_trim", gpu._ctx)
        before = torch.cuda.mem_get_info()[0]
        if what == "train":
            m.zero_grads()
            m.forward_backward(ids, ids, 4)
        else:
            m.prefill(m.new_decode_state(4), ids.reshape(4, -1))
        used[fused] = before - torch.cuda.mem_get_info()[0]
    assert used[False] - used[True] > 40 << 20
    m.free()


# Pageable host arrays around the sizes where the copies change form: staged, one piece more, one slot of the ring and one
# byte more, more than the whole ring.
@pytest.mark.parametrize("n", [1, 65536, 65537, 1 << 20, (1 << 20) + 1, (8 << 20) + 3, (19 << 20) + 70001])
def test_host_copies(gpu, n):
    import ctypes as C
    import torch

    src, back = np.random.default_rng(n).integers(0, 256, n).astype(np.uint8), np.zeros(n + 2, np.uint8)
    buf = torch.zeros(n + 64, dtype=torch.uint8, device="cuda")
    torch.cuda.synchronize()
    for _ in range(2):
        gpu._call("asca_memcpy_h2d", gpu._ctx, C.c_void_p(buf.data_ptr()), C.c_void_p(src.ctypes.data), C.c_size_t(n))
        gpu._call("asca_memcpy_d2h", gpu._ctx, C.c_void_p(back.ctypes.data + 1), C.c_void_p(buf.data_ptr()), C.c_size_t(n))
        assert np.array_equal(back[1:-1], src) and back[0] == back[-1] == 0
        src = src[::-1].copy()
    assert not buf[n:].any()


# A device address where a host array belongs is an error code, in both directions and at both copy forms, and the context goes
# on working; pinned arrays are taken.
def test_device_address_as_host_array_is_refused(gpu):
    import ctypes as C
    import torch
    import asca_b200

    n = 1 << 20
    dev, back = torch.arange(2 * n, dtype=torch.uint8, device="cuda"), torch.zeros(n, dtype=torch.uint8).pin_memory()
    torch.cuda.synchronize()
    at = dev.data_ptr()
    for size in (64, n):
        for call in ("asca_memcpy_h2d", "asca_memcpy_d2h"):
            with pytest.raises(asca_b200.AscaError, match="device address"):
                gpu._call(call, gpu._ctx, C.c_void_p(at), C.c_void_p(at + n), C.c_size_t(size))
        gpu._call("asca_memcpy_d2h", gpu._ctx, C.c_void_p(back.data_ptr()), C.c_void_p(at), C.c_size_t(size))
        assert torch.equal(back[:size], dev[:size].cpu())
    m = asca_b200.Model(gpu, 256, 64, 4, 1, 2, 64)
    ids = np.zeros(4, np.uint32)
    with pytest.raises(asca_b200.AscaError, match="device address"):
        gpu._call("asca_model_forward_backward_host", gpu._ctx, m._h, C.c_void_p(ids.ctypes.data), C.c_void_p(ids.ctypes.data), C.c_int64(1),
                  C.c_int64(4), C.c_void_p(at), None)
    assert np.isfinite(m.forward_backward(ids, ids, 1))
    m.free()


# A repeated bf16 decode step is replayed as a graph; profiled calls launch directly. Same tokens and logits either way, for
# two batch sizes in turn.
def test_bf16_decode_graph_equals_direct_launches(orc, gpu):
    import asca_b200

    m = asca_b200.Model(gpu, 256, 128, 2, 2, 4, 256)
    m.set_params(orc.Rng(9).normal(m.n, 0.05))
    m.set_compute(asca_b200.BF16)
    runs = []
    for direct in (False, True):
        gpu.profile(direct)
        states = {ns: m.new_decode_state(ns) for ns in (5, 16)}
        out = []
        for step in range(6):
            for ns, st in states.items():
                out += list(m.decode_step(st, orc.Rng(step + ns).below(256, ns)))
                if step % 2:
                    out.append(m.decode_greedy(st, orc.Rng(step).below(256, ns), 3 + step))
        gpu.profile(False)
        runs.append(out)
    for a, b in zip(*runs):
        assert np.array_equal(a, b)
    m.free()


# The decode graph belongs to a number of streams, not to a state buffer: requests that come with states of their own are replayed
# from the third on, eleven states in turn go on being replayed, and a call longer than the token buffer (1024 steps of 256
# streams) is replayed in parts.
def test_bf16_decode_graph_serves_any_state(orc, gpu):
    import asca_b200

    m = asca_b200.Model(gpu, 256, 128, 2, 1, 4, 256)
    m.set_params(orc.Rng(9).normal(m.n, 0.05))
    m.set_compute(asca_b200.BF16)
    states = [m.new_decode_state(5) for _ in range(11)]
    for rest in range(3):
        for i, st in enumerate(states):
            n = gpu.graph_launch_count()
            got = m.decode_step(st, orc.Rng(i + 20 * rest).below(256, 5))
            assert gpu.graph_launch_count() - n == (0 if rest == 0 and i < 2 else 1)
            if i == 7:
                first = (got[0], st.clone())
    gpu.profile(True)
    other = m.new_decode_state(5)
    for rest in range(3):
        want = m.decode_step(other, orc.Rng(7 + 20 * rest).below(256, 5))
    gpu.profile(False)
    assert np.array_equal(first[0], want[0]) and bool((first[1] == other).all())

    ids, toks = orc.Rng(1).below(256, 256), []
    for replayed in (False, False, True):
        n = gpu.graph_launch_count()
        st = m.new_decode_state(256)
        toks.append((m.decode_greedy(st, ids, 1030), st))
        assert gpu.graph_launch_count() - n == (1030 if replayed else 0)
    assert np.array_equal(toks[0][0], toks[2][0]) and bool((toks[0][1] == toks[2][1]).all())
    m.free()


# The tensor-core products around their tile shapes: pairs from half the chip on (37 tiles), one 128 x 128 tile an SM, two CTAs
# an SM; ragged last rows and columns, rows off the 32-byte grid, k below and between k-tiles, bias and accumulation.
@pytest.mark.parametrize("m,k,n", [(1536, 64, 1600), (1537, 72, 1604), (2560, 1032, 2050), (1100, 200, 1030), (130, 520, 40), (2100, 136, 2100)])
@pytest.mark.parametrize("mode", ["NN", "TN", "NT"])
def test_bf16_product_tile_edges(gpu, m, k, n, mode):
    import torch
    import asca_b200
    from asca_b200 import ops

    g = torch.Generator(device="cuda").manual_seed(m + 7 * k + 13 * n)
    a, b = (torch.randn(*s, generator=g, device="cuda").bfloat16() for s in ((m, k), (k, n)))
    bias, c0 = torch.randn(n, generator=g, device="cuda"), torch.randn(m, n, generator=g, device="cuda")
    out = c0.clone()
    ops.gemm(gpu, a.t().contiguous() if mode == "TN" else a, b.t().contiguous() if mode == "NT" else b, getattr(asca_b200, mode), bias=bias,
             out=out, accumulate=True)
    gpu.sync()
    ref = a.double() @ b.double() + bias.double() + c0.double()
    assert rel_err(out.cpu().numpy(), ref.cpu().numpy()) < F32_TOL


# The bf16 expert layer with a skewed load, experts of no token in long runs and in turn with experts of one k-tile (whose claims are
# held back by the epilogue and by the ring), and segments around the tile and cluster sizes.
@pytest.mark.parametrize("n,d,F,E,vocab", [(1025, 512, 1024, 256, 1), (4096, 256, 320, 4, 256), (6000, 256, 512, 8, 3), (640, 128, 1088, 2, 256),
                                           (700, 256, 512, 512, 256), (700, 128, 128, 1024, 200), (130, 256, 256, 1500, 4096)])
def test_bf16_expert_layer_edges(gpu, n, d, F, E, vocab):
    import torch
    from asca_b200 import ops

    g = torch.Generator(device="cuda").manual_seed(n)
    ids = torch.randint(0, vocab, (n,), generator=g, device="cuda", dtype=torch.int32)
    perm, offs = ops.moe_dispatch(gpu, ids, E)
    xn = torch.randn(n, d, generator=g, device="cuda").bfloat16()
    w1, w2 = (torch.randn(*s, generator=g, device="cuda").mul_(s[0] ** -0.5 if s[0] == d else F ** -0.5).bfloat16() for s in ((d, E * F), (E * F, d)))
    b1, b2 = torch.randn(E * F, generator=g, device="cuda"), torch.randn(d, generator=g, device="cuda")
    dout = torch.randn(n, d, generator=g, device="cuda")
    out, pre, hid = ops.moe_fwd(gpu, xn, w1, b1, w2, b2, perm, offs, F, E)
    d_w1, d_b1, d_w2, d_b2, dxn = ops.moe_bwd(gpu, xn, w1, w2, pre, hid, dout, perm, offs, F, E)
    gpu.sync()
    o = offs.cpu().tolist()
    close = lambda got, want: rel_err(got.float().cpu().numpy(), want.float().cpu().numpy()) < 2e-2
    assert close(d_b2, dout.sum(0))
    for e in range(E):
        rows, f = perm[o[e]:o[e + 1]].long(), slice(e * F, (e + 1) * F)
        if o[e] == o[e + 1]:
            assert not (d_w1[:, f].any() or d_w2[f].any() or d_b1[f].any())
            continue
        x, dy = xn[rows].float(), dout[rows]
        p = x @ w1[:, f].float() + b1[f]
        s = torch.sigmoid(p)
        h, dp = p * s, (dy @ w2[f].float().t()) * (s * (1 + p * (1 - s)))
        assert close(out[rows], h @ w2[f].float() + b2) and close(dxn[rows], dp @ w1[:, f].float().t())
        assert close(d_w1[:, f], x.t() @ dp) and close(d_w2[f], h.t() @ dy) and close(d_b1[f], dp.sum(0))


# q, k and v from the projection's epilogue (one head of 128 or two of 64 a warp, ragged last rows) against the separate pass:
# a prefill's states and logits.
@pytest.mark.parametrize("d,H,ns,T", [(256, 4, 33, 97), (256, 2, 16, 192), (768, 12, 9, 301)])
def test_prefill_with_the_fused_qkv_epilogue(orc, gpu, d, H, ns, T):
    import asca_b200

    m = asca_b200.Model(gpu, 256, d, H, 2, 4, 256)
    m.set_params(orc.Rng(d + H).normal(m.n, 0.05))
    m.set_compute(asca_b200.BF16)
    ids = orc.Rng(T).below(256, ns * T).reshape(ns, T)
    got = []
    for fused in (False, True):
        m.set_fused_qkv(fused)
        st = m.new_decode_state(ns)
        logits, _ = m.prefill(st, ids)
        got.append((np.asarray(logits), st.cpu().numpy()))
    m.free()
    for a, b in zip(*got):
        assert rel_err(b, a) < 5e-3


# bf16 delta on the tensor cores: a sequence's last, ragged chunk must not read the next sequence's rows (zero times NaN is NaN),
# and what comes out is as close to 64-bit arithmetic as bf16 operands allow.
@pytest.mark.parametrize("dh", [64, 128])
@pytest.mark.parametrize("B,T,H", [(2, 1, 1), (2, 63, 2), (3, 65, 1), (2, 129, 3)])
def test_delta_tc_sequences_do_not_mix(gpu, B, T, H, dh):
    import torch
    from asca_b200 import ops

    g = torch.Generator(device="cuda").manual_seed(7 * T + dh)
    n = B * T

    def norm(*s):
        return torch.randn(*s, generator=g, device="cuda")

    q, k = (torch.nn.functional.normalize(norm(n, H, dh), dim=-1).reshape(n, H * dh).bfloat16() for _ in range(2))
    v, d_o = norm(n, H * dh).bfloat16(), norm(n, H * dh).bfloat16()
    al, be, qn = torch.sigmoid(2 + norm(n, H)), torch.sigmoid(norm(n, H)), 1 + torch.rand(n, H, generator=g, device="cuda")

    def run(q, k, v, d_o):
        o, fin, ck = ops.delta_fwd(gpu, q, k, v, al, be, B, T, H, dh, want_final=True)
        d_qkv, d_gate = ops.delta_bwd(gpu, q, k, v, al, be, qn, qn, d_o, ck, B, T, H, dh)
        gpu.sync()
        return o, fin, d_qkv, d_gate

    want = run(q, k, v, d_o)
    bad = [x.clone() for x in (q, k, v, d_o)]
    for x in bad:
        x[T:2 * T] = float("nan")   # the second sequence
    got = run(*bad)
    keep = torch.ones(n, dtype=torch.bool, device="cuda")
    keep[T:2 * T] = False
    seqs = torch.arange(B, device="cuda") != 1
    for a, b, m in zip(got, want, (keep, seqs, keep, keep)):
        assert torch.equal(a[m], b[m]) and not torch.isnan(b).any()
    assert torch.isnan(got[0][~keep]).any()

    # the recurrence in 64 bits on the same bf16 inputs, gradients by autograd
    q64, k64, v64, do64 = (x.double().view(B, T, H, dh).transpose(1, 2).clone().requires_grad_() for x in (q, k, v, d_o))
    la = al.double().log().view(B, T, H).transpose(1, 2).clone().requires_grad_()
    b64 = be.double().view(B, T, H).transpose(1, 2).clone().requires_grad_()
    S, outs = torch.zeros(B, H, dh, dh, dtype=torch.float64, device="cuda"), []
    for t in range(T):
        S = la[:, :, t].exp()[..., None, None] * S
        u = b64[:, :, t, None] * (v64[:, :, t] - torch.einsum("bhai,bha->bhi", S, k64[:, :, t]))
        S = S + k64[:, :, t, :, None] * u[:, :, None, :]
        outs.append(torch.einsum("bhai,bha->bhi", S, q64[:, :, t]))
    o64 = torch.stack(outs, 2)
    (o64 * do64).sum().backward()

    def back(x, y):   # the L2 norm's backward
        return (x.grad - y * (y * x.grad).sum(-1, keepdim=True)) / qn.double().view(B, T, H).transpose(1, 2)[..., None]

    def flat(x):
        return x.transpose(1, 2).reshape(n, -1)

    d64 = torch.cat([flat(back(q64, q64.detach())), flat(back(k64, k64.detach())), flat(v64.grad)], 1)
    g64 = torch.cat([flat(la.grad * (1 - la.exp())), flat(b64.grad * b64 * (1 - b64))], 1)
    # a handful of bf16 roundings (2^-9 each) on the way to every value
    for got_, ref in zip(want, (flat(o64), S, d64, g64)):
        ref = ref.detach()
        assert (got_.double() - ref).norm() < 8e-3 * ref.norm()


# bf16 delta: chains over many chunks, more chains than SMs (the requests ahead into L2 switch off, heads of 64 share an SM): within a handful
# of bf16 roundings of the f32 kernels, and bit for bit what the sequences give in smaller launches.
@pytest.mark.parametrize("dh", [64, 128])
@pytest.mark.parametrize("B,T,H", [(1, 2111, 2), (20, 130, 16)])
def test_delta_tc_many_chunks_and_many_chains(gpu, B, T, H, dh):
    import torch
    from asca_b200 import ops

    g = torch.Generator(device="cuda").manual_seed(B + dh)
    n = B * T

    def norm(*s):
        return torch.randn(*s, generator=g, device="cuda")

    q, k = (torch.nn.functional.normalize(norm(n, H, dh), dim=-1).reshape(n, H * dh).bfloat16() for _ in range(2))
    v, d_o = norm(n, H * dh).bfloat16(), norm(n, H * dh).bfloat16()
    al, be, qn = torch.sigmoid(3 + norm(n, H)), torch.sigmoid(norm(n, H)), 1 + torch.rand(n, H, generator=g, device="cuda")

    def run(b0, b1, cast):
        part = [x[b0 * T:b1 * T].contiguous() for x in (q, k, v, d_o, al, be, qn)]
        q_, k_, v_, do_ = (cast(x) for x in part[:4])
        o, fin, ck = ops.delta_fwd(gpu, q_, k_, v_, *part[4:6], b1 - b0, T, H, dh, want_final=True)
        d_qkv, d_gate = ops.delta_bwd(gpu, q_, k_, v_, *part[4:6], part[6], part[6], do_, ck, b1 - b0, T, H, dh)
        gpu.sync()
        return o, fin.view(b1 - b0, -1), d_qkv, d_gate

    got = run(0, B, lambda x: x)
    for a, b in zip(got, run(0, B, lambda x: x.float())):
        assert (a.double() - b.double()).norm() < 8e-3 * b.double().norm()
    cut = B * 9 // 20   # (9 x 16 chains: fewer than SMs)
    if cut:
        for a, b, c in zip(got, run(0, cut, lambda x: x), run(cut, B, lambda x: x)):
            assert torch.equal(a, torch.cat([b, c]))


# What the bf16 delta gradients hold in f32 between their products: inputs for which everything else is exact in bf16, one chain per
# entry, so that a value rounded to bf16 on the way (2^-9) stands out. The bound: a dozen f32 roundings, exp and log among them.
def _delta_tc_gates(gpu, q, k, v, al, be, d_o, s_init=None):
    """d_gate (B, T, 2, H) of float tensors (B, T, H, dh) / (B, T, H) with unit norms."""
    import torch
    from asca_b200 import ops

    B, T, H, dh = q.shape
    q, k, v, d_o = (x.reshape(B * T, H * dh).bfloat16() for x in (q, k, v, d_o))
    al, be = (x.reshape(B * T, H).contiguous() for x in (al, be))
    one = torch.ones(B * T, H, device="cuda")
    _, _, ck = ops.delta_fwd(gpu, q, k, v, al, be, B, T, H, dh, s_init=s_init)
    _, d_gate = ops.delta_bwd(gpu, q, k, v, al, be, one, one, d_o, ck, B, T, H, dh)
    gpu.sync()
    return d_gate.view(B, T, 2, H).double()


def _bf16_values(g, *shape):
    import torch

    return (torch.rand(*shape, generator=g, device="cuda") + 1).bfloat16().float()   # eight significant bits


@pytest.mark.parametrize("dh", [64, 128])
@pytest.mark.parametrize("T", [65, 128, 300])
def test_delta_tc_state_gradient_meets_the_state_in_f32(gpu, dh, T):
    """Nothing is written (beta 0), no output of the first chunk counts: d log alpha_0 = alpha_0 <S, Q^T dO of the chunks behind>."""
    import torch

    B, H = 2, 8
    g = torch.Generator(device="cuda").manual_seed(T + dh)
    q, k, v, d_o = (_bf16_values(g, B, T, H, dh) for _ in range(4))
    d_o[:, :64] = 0.0
    al, be = torch.ones(B, T, H, device="cuda"), torch.zeros(B, T, H, device="cuda")
    al[:, 0] = 0.75
    s_init = torch.zeros(B, H, dh, dh, device="cuda")
    at = torch.randint(0, dh * dh, (B, H, 1), generator=g, device="cuda")
    s_init.view(B, H, -1).scatter_(2, at, 1.0)
    got = _delta_tc_gates(gpu, q, k, v, al, be, d_o, s_init)[:, 0, 0]
    d_s = torch.einsum("bthi,bthj->bhij", q.double(), d_o.double())
    want = 0.25 * 0.75 * d_s.reshape(B, H, -1).gather(2, at)[..., 0]
    # (f32 sums on the tensor cores: sixteen products a step, each step within 2^-23 of the sum so far)
    assert ((got - want).abs() <= 2.0 ** -18 * want.abs()).all()


@pytest.mark.parametrize("dh", [64, 128])
@pytest.mark.parametrize("t0,t1", [(0, 1), (2, 40), (17, 63)])
def test_delta_tc_gate_sums_within_a_chunk_in_f32(gpu, dh, t0, t1):
    """Token t0 writes, t1 reads (d log alpha) and overwrites (d beta): sums of (dO U^T) o (Q K^T) and (dR U^T) o (K K^T) with one entry."""
    import torch

    B, H, T = 2, 8, t1 + 1
    g = torch.Generator(device="cuda").manual_seed(dh + t1)
    al, be = torch.ones(B, T, H, device="cuda"), torch.zeros(B, T, H, device="cuda")
    al[:, t1], be[:, t0] = 0.75, 1.0
    q, k, v, d_o = (torch.zeros(B, T, H, dh, device="cuda") for _ in range(4))
    q[:, t1, :, 1], k[:, t0, :, 1] = _bf16_values(g, B, H), 1.0
    v[:, t0, :, dh - 3], d_o[:, t1, :, dh - 3] = _bf16_values(g, B, H), _bf16_values(g, B, H)
    got = _delta_tc_gates(gpu, q, k, v, al, be, d_o)
    x = (v[:, t0, :, dh - 3].double() * d_o[:, t1, :, dh - 3].double()) * 0.75
    want = 0.25 * x * q[:, t1, :, 1].double()
    assert ((got[:, t1, 0] - want).abs() <= 2.0 ** -19 * want).all()
    q[:, t1, :, 1], k[:, t1, :, 1], be[:, t1] = 1.0, 1.0, 0.5
    got = _delta_tc_gates(gpu, q, k, v, al, be, d_o)
    want = -0.25 * x
    assert ((got[:, t1, 1] - want).abs() <= 2.0 ** -19 * want.abs()).all()


@pytest.mark.parametrize("dh", [64, 128])
def test_delta_tc_value_gradient_meets_the_state_in_f32(gpu, dh):
    """One token on a state with one entry: d beta = -dR . (S^T k), dR = (q . k) dO a product of two eight-bit numbers."""
    import torch

    B, H = 2, 8
    g = torch.Generator(device="cuda").manual_seed(dh)
    q, k, v, d_o = (torch.zeros(B, 1, H, dh, device="cuda") for _ in range(4))
    q[..., 3], k[..., 3] = _bf16_values(g, B, 1, H), 1.0
    d_o[..., dh - 2] = _bf16_values(g, B, 1, H)
    s_init = torch.zeros(B, H, dh, dh, device="cuda")
    s_init[..., 3, dh - 2] = 1.0
    al, be = torch.ones(B, 1, H, device="cuda"), torch.full((B, 1, H), 0.5, device="cuda")
    got = _delta_tc_gates(gpu, q, k, v, al, be, d_o, s_init)[:, 0, 1]
    want = -0.25 * (q[..., 3] * d_o[..., dh - 2]).double()[:, 0]
    assert ((got - want).abs() <= 2.0 ** -19 * want.abs()).all()


# f32 delta backward: a row's gradients are divided by its norm through the reciprocal; zero, infinite and tiny norms behave as a division.
@pytest.mark.parametrize("dh", [32, 64, 128])
def test_delta_f32_norm_division_at_its_edges(gpu, dh):
    import torch
    from asca_b200 import ops

    B, T, H = 1, 70, 2
    g = torch.Generator(device="cuda").manual_seed(dh)
    q, k = (torch.nn.functional.normalize(torch.randn(T, H, dh, generator=g, device="cuda"), dim=-1).reshape(T, H * dh) for _ in range(2))
    v, d_o = (torch.randn(T, H * dh, generator=g, device="cuda") for _ in range(2))
    al, be = (torch.sigmoid(torch.randn(T, H, generator=g, device="cuda")) for _ in range(2))
    one = torch.ones(T, H, device="cuda")
    _, _, ck = ops.delta_fwd(gpu, q, k, v, al, be, B, T, H, dh)
    want, want_g = ops.delta_bwd(gpu, q, k, v, al, be, one, one, d_o, ck, B, T, H, dh)
    norm = 10.0 ** torch.empty(T, H, device="cuda").uniform_(-30, 30, generator=g)
    norm[3], norm[5], norm[66] = 0.0, float("inf"), 3.0
    got, got_g = ops.delta_bwd(gpu, q, k, v, al, be, norm, norm, d_o, ck, B, T, H, dh)
    gpu.sync()
    assert torch.equal(got_g, want_g)
    for part in range(2):
        a, w = (x.view(T, 3, H, dh)[:, part] for x in (got, want))
        w = w / norm[..., None]
        fin = torch.isfinite(w)
        assert torch.equal(fin, torch.isfinite(a)) and torch.equal(torch.isnan(a), torch.isnan(w))
        # one rounding of the quotient on each side; denormal results on the spacing of denormals
        assert ((a - w)[fin].abs() <= 2 ** -22 * w[fin].abs() + 2 ** -148).all()


# The same division by norms without a finite reciprocal (below 2^-128, denormal ones among them): finite quotients, infinities and the zeros of rows
# without a gradient as in 64 bits.
@pytest.mark.parametrize("dh", [32, 64, 128])
def test_delta_f32_norms_without_a_reciprocal(gpu, dh):
    import torch
    from asca_b200 import ops

    B, T, H = 1, 70, 2
    g = torch.Generator(device="cuda").manual_seed(dh + 1)
    q, k = (torch.nn.functional.normalize(torch.randn(T, H, dh, generator=g, device="cuda"), dim=-1).reshape(T, H * dh) for _ in range(2))
    v, d_o = (torch.randn(T, H * dh, generator=g, device="cuda") for _ in range(2))
    d_o *= 10.0 ** torch.empty(T, 1, device="cuda").uniform_(-8, 0, generator=g)
    d_o[2:7] = 0.0    # dq of these rows is zero
    al, be = (torch.sigmoid(torch.randn(T, H, generator=g, device="cuda")) for _ in range(2))
    one = torch.ones(T, H, device="cuda")
    _, _, ck = ops.delta_fwd(gpu, q, k, v, al, be, B, T, H, dh)
    want, _ = ops.delta_bwd(gpu, q, k, v, al, be, one, one, d_o, ck, B, T, H, dh)
    norm = (10.0 ** torch.empty(T, H, device="cuda", dtype=torch.float64).uniform_(-44, -36, generator=g)).float()
    norm[4], norm[9], norm[68], norm[69] = 2.0 ** -149, 2.0 ** -100, 2.0 ** -128, 2.0 ** -129
    got, _ = ops.delta_bwd(gpu, q, k, v, al, be, norm, norm, d_o, ck, B, T, H, dh)
    gpu.sync()
    assert (norm > 0).all()
    for part in range(2):
        a, w = (x.view(T, 3, H, dh)[:, part] for x in (got, want))
        w = (w.double() / norm.double()[..., None]).float()
        fin = torch.isfinite(w)
        assert (fin & (w != 0)).any() and not fin.all()
        assert torch.equal(fin, torch.isfinite(a)) and not torch.isnan(a).any() and torch.equal(a[~fin], w[~fin])
        assert ((a - w)[fin].abs() <= 2 ** -22 * w[fin].abs()).all()   # one rounding of the quotient on each side
    assert (got.view(T, 3, H, dh)[2:7, 0] == 0).all()


# Expert products of a few tokens: ones whose k range two or four CTAs share and ones past the rule (more tokens, shorter k), experts without tokens
# and with more than one token tile; against f64 sums over the hidden rows as they were stored.
@pytest.mark.parametrize("tokens,experts,d,F", [(1, 16, 768, 3072), (3, 16, 768, 3072), (12, 16, 768, 3072), (13, 16, 768, 3072), (70, 2, 128, 1664), (300, 6, 64, 832), (200, 40, 64, 448)])
def test_few_tokens_per_expert_with_a_shared_k_range(gpu, tokens, experts, d, F):
    import torch
    from asca_b200 import ops

    g = torch.Generator(device="cuda").manual_seed(tokens)

    def norm(*s, scale=1.0):
        return torch.randn(*s, generator=g, device="cuda") * scale

    xn, w1, w2 = norm(tokens, d).bfloat16(), norm(d, experts * F, scale=d ** -0.5).bfloat16(), norm(experts * F, d, scale=F ** -0.5).bfloat16()
    b1, b2 = norm(experts * F), norm(d)
    ids = torch.randint(0, 256, (tokens,), generator=g, device="cuda", dtype=torch.int32)
    perm, offs = ops.moe_dispatch(gpu, ids, experts)
    out, _, hid = ops.moe_fwd(gpu, xn, w1, b1, w2, b2, perm, offs, F, experts)
    out2, _, _ = ops.moe_fwd(gpu, xn, w1, b1, w2, b2, perm, offs, F, experts)
    gpu.sync()
    assert torch.equal(out, out2)
    route = torch.repeat_interleave(torch.arange(experts, device="cuda"), (offs[1:] - offs[:-1]).long())
    want = torch.empty(tokens, d, dtype=torch.float64, device="cuda")
    for e in range(experts):
        rows = (route == e).nonzero().flatten()
        if len(rows):   # from the hidden rows as they were stored (bf16)
            want[perm[rows].long()] = hid[rows].double() @ w2[e * F:(e + 1) * F].double() + b2.double()
    assert (out - want).abs().max() < 4e-6 * F ** 0.5


# The same with more tiles than clusters run at a time (148 SMs: 37 of four CTAs, 74 of two), so that some take a second tile into slots
# and an accumulator buffer that the first one's readers have to leave; odd and even numbers of k-tiles.
@pytest.mark.parametrize("counts,share,F", [([33] * 15 + [1] * 17, 4, 2048), ([1] * 17 + [33] * 15, 4, 2112), ([33] * 30 + [1] * 34, 2, 2048), ([1] * 34 + [33] * 30, 2, 2624)])
def test_shared_k_range_over_several_tiles_a_cluster(gpu, counts, share, F):
    import torch
    from asca_b200 import ops

    E, tokens, d = len(counts), sum(counts), 128
    assert tokens == 16 * E and sum((c + 31) // 32 for c in counts) > 148 // share   # (one feature tile each)
    g = torch.Generator(device="cuda").manual_seed(F + E)

    def norm(*s, scale=1.0):
        return torch.randn(*s, generator=g, device="cuda") * scale

    xn, w1, w2 = norm(tokens, d).bfloat16(), norm(d, E * F, scale=d ** -0.5).bfloat16(), norm(E * F, d, scale=F ** -0.5).bfloat16()
    b1, b2 = norm(E * F), norm(d)
    offs = torch.tensor([0] + counts, device="cuda").cumsum(0).int()
    perm = torch.randperm(tokens, generator=g, device="cuda").int()
    out, _, hid = ops.moe_fwd(gpu, xn, w1, b1, w2, b2, perm, offs, F, E)
    out2, _, _ = ops.moe_fwd(gpu, xn, w1, b1, w2, b2, perm, offs, F, E)
    gpu.sync()
    assert torch.equal(out, out2)
    for e in range(E):
        rows = slice(int(offs[e]), int(offs[e + 1]))
        want = hid[rows].double() @ w2[e * F:(e + 1) * F].double() + b2.double()
        assert (out[perm[rows].long()] - want).abs().max() < 4e-6 * F ** 0.5


# The residual adds in the epilogues of the attention's and the experts' second product, on both sides of where the row-tiled kernel
# takes either product (rows past 256; more than 64 tokens per expert), ragged rows and 64-column remainders included: logits and
# loss of three blocks against the f32 oracle, within the bf16 mode's 2e-2.
@pytest.mark.parametrize("B,T,E", [(1, 100, 2), (1, 200, 2), (2, 150, 8), (1, 257, 2), (3, 301, 3)])
def test_residual_in_the_products_epilogues(orc, gpu, B, T, E):
    import asca_b200

    cfg = (256, 192, 3, 3, E, 320)
    ref = orc.Model(*cfg)
    ref.init_reference(orc.Rng(T))
    dev = asca_b200.Model(gpu, *cfg)
    dev.set_params(ref.params)
    dev.set_compute(asca_b200.BF16)
    ids = orc.Rng(T + E).below(256, B * T)
    loss_ref, g_ref = ref.forward_backward(ids, ids, B)
    dev.zero_grads()
    loss = dev.forward_backward(ids, ids, B)
    _, g = dev.get()
    assert abs(loss - loss_ref) < 2e-2 * abs(loss_ref)
    for name in ref.names:   # (the gate biases, sums that cancel, are held at larger sizes)
        a, b = ref.tensor(name, g), ref.tensor(name, g_ref)
        assert b.size < 64 or rel_err(a, b) < 2e-2, name
    state = dev.new_decode_state(B)
    logits, _ = dev.prefill(state, ids.reshape(B, T))
    last = np.empty_like(logits)
    for s in range(B):
        st = ref.new_decode_state()
        for t in range(T):
            last[s] = ref.step(int(ids[s * T + t]), st)[0]
    assert rel_err(logits, last) < 2e-2
    dev.free()


# SiLU and its derivative in the expert products' epilogues (few rows, row tiles), from large negative arguments to large positive ones, against
# 64 bits: the bf16 rounding of the result (eight significant bits: 2^-8) and (|x| + 5) 2^-23 of the sigmoid inside it.
@pytest.mark.parametrize("tokens", [8, 256])
def test_silu_over_the_range_of_its_argument(gpu, tokens):
    import torch
    from asca_b200 import ops

    d, F, E = 128, 512, 2
    x = torch.cat([torch.linspace(-110, 110, F // 2), torch.linspace(-9, 9, F // 2 - 4), torch.tensor([0.0, -1.2784645, 3e4, -3e4])]).cuda()
    xn = torch.zeros(tokens, d, device="cuda").bfloat16()
    w1, w2 = torch.zeros(d, E * F, device="cuda").bfloat16(), torch.zeros(E * F, d, device="cuda").bfloat16()
    w2[:, 0] = 1.0
    perm, offs = ops.moe_dispatch(gpu, torch.arange(tokens, device="cuda", dtype=torch.int32), E)
    _, _, hid = ops.moe_fwd(gpu, xn, w1, x.repeat(E), w2, torch.zeros(d, device="cuda"), perm, offs, F, E)
    dout = torch.zeros(tokens, d, device="cuda")
    dout[0, 0] = 1.0
    _, d_b1, _, _, _ = ops.moe_bwd(gpu, xn, w1, w2, x.repeat(tokens, 1), hid, dout, perm, offs, F, E)
    gpu.sync()
    x64 = x.double()
    sg = torch.sigmoid(x64)
    want, rel = x64 * sg, 2.0 ** -8 + (x64.abs() + 6) * 2.0 ** -23
    assert ((hid.double() - want).abs() <= rel * want.abs() + 2e-36).all()
    want = sg * (1 + x64 * (1 - sg))
    off = 2.0 ** -8 * want.abs() + sg * (1 + 2 * x64.abs()) * (x64.abs() + 6) * 2.0 ** -23 + 2e-36
    assert ((d_b1.view(E, F).double().sum(0) - want).abs() <= off).all()


# Weight gradients of experts whose token counts end a 64-token tile anywhere (empty experts, sixteens, one past them): nothing of a
# neighbour's rows, 1e4 times as large, enters a sum. d_w2 from the hidden rows as they were stored, within the bound of f32 sums.
# The long form: runs of tiles without a ragged end, more than a CTA's 16 claims at a time, between ragged ones.
@pytest.mark.parametrize("d,F,long", [(256, 512, False), (128, 128, False), (1024, 2048, True)])   # CTA pairs; single CTAs; CTA pairs
def test_ragged_token_counts_in_weight_gradients(gpu, d, F, long):
    import torch
    from asca_b200 import ops

    counts = [0, 1, 64, 15, 16, 17, 0, 63, 65, 79, 80, 81, 127, 128, 129, 448, 449, 511, 512, 513, 900, 33, 48, 2, 320, 7]
    if long:
        counts = [65, 7] + [64] * 46 + [129, 1, 0, 190] + [128, 64] * 24 + [63]
    E, N = len(counts), sum(counts)
    g = torch.Generator(device="cuda").manual_seed(F)

    def norm(*s):
        return torch.randn(*s, generator=g, device="cuda")

    offs = torch.tensor([0] + counts, device="cuda").cumsum(0).int()
    perm = torch.randperm(N, generator=g, device="cuda").int()
    xn, w1, w2 = norm(N, d).bfloat16(), (norm(d, E * F) * d ** -0.5).bfloat16(), norm(E * F, d).bfloat16()
    _, pre, hid = ops.moe_fwd(gpu, xn, w1, norm(E * F), w2, norm(d), perm, offs, F, E)
    dout = norm(N, d)
    for e in range(0, E, 2):
        dout[perm[offs[e]:offs[e + 1]].long()] *= 1e4
    _, _, d_w2, _, _ = ops.moe_bwd(gpu, xn, w1, w2, pre, hid, dout, perm, offs, F, E)
    gpu.sync()
    for e, n in enumerate(counts):
        h, dy = hid[offs[e]:offs[e + 1]].double(), dout[perm[offs[e]:offs[e + 1]].long()].bfloat16().double()
        err = (d_w2[e * F:(e + 1) * F].double() - h.t() @ dy).abs()
        assert (err <= n * 2.0 ** -22 * (h.abs().t() @ dy.abs())).all(), (e, n)
