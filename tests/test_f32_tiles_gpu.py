"""The FP32 tile kernels (csrc/gemm_f32.cuh: channel chains, mixing; csrc/spectral_f32.cu: transforms) at the edges of
their 64-row tiles and column tiles, with 16-byte aligned and with misaligned buffers: the two must agree bit for bit
(same products, same order), and both must match the same operation in float64 torch.

Tolerance: a chain of two contractions of length <= 3C = 288 in FP32 rounds each partial sum by 2^-24 of its size, so the
relative error (max over max) is below 2 * 288 * 2^-24 = 3.5e-5 in the worst case; transforms of length K stay below
K * 2^-24 <= 1.6e-5 for K <= 260. 4e-5 covers both, and the activations' few ulp."""
import pytest
import torch
import torch.nn.functional as F

pytestmark = pytest.mark.gpu

TOL = 4e-5


def _buf(shape, off, gen=None):
    """A float32 buffer that starts `off` floats past a 512-byte boundary, random or (gen None) NaN."""
    n = 1
    for s in shape:
        n *= s
    base = torch.full((n + off,), float("nan"), device="cuda")
    t = base[off:].view(*shape)
    if gen is not None:
        t.copy_(torch.randn(*shape, generator=gen))
    return t


def _both(run):
    """run(off) -> outputs; aligned and misaligned outputs must have the same bits."""
    a, b = run(0), run(1)
    for x, y in zip(a, b):
        assert torch.equal(x, y)
    return a


def _close(got, want):
    err = ((got.double() - want).abs().max() / want.abs().max()).item()
    assert err < TOL, err


@pytest.mark.parametrize("C", [16, 32, 64, 96])
@pytest.mark.parametrize("V", [1, 63, 65, 200])
def test_chains_match_float64_and_do_not_need_alignment(C, V):
    from ffnoml_gb300 import _native as nat
    s = torch.cuda.current_stream().cuda_stream
    P = nat.lib().ffno_stats_parts(V)

    def run(off):
        g = torch.Generator().manual_seed(C * 1000 + V)
        x, xd, pre, up = (_buf((V, C), off, g) for _ in range(4))
        w = lambda k, n: _buf((k, n), off, g).mul_(k ** -0.5)
        g1, g2, m1, m2 = w(C, C), w(C, C), w(C, 2 * C), w(2 * C, C)
        dw = _buf((V,), off, g).abs_()
        coefs = _buf((3, C), off, g)
        tr = lambda t: _buf(tuple(t.t().shape), off).copy_(t.t())
        m1t, m2t, g1t, g2t = tr(m1), tr(m2), tr(g1), tr(g2)
        gate, x1, out, ab, jv, gj, gb = (_buf((V, C), off) for _ in range(7))
        parts = torch.empty(P, 8, 3, dtype=torch.float64, device="cuda")
        coef_out, gst = torch.empty(3, C, device="cuda"), torch.empty(8, 3, dtype=torch.float64, device="cuda")
        one, zero = torch.ones(C, device="cuda"), torch.zeros(C, device="cuda")
        p = lambda t: t.data_ptr()
        nat.call("ffno_gate_fwd", p(x), V, C, p(g1), p(g2), None, None, p(gate), s)
        nat.call("ffno_mlp2_fwd", 1, p(x), p(pre), p(coefs), 0.7, p(x1), V, C, p(m1), p(m2), p(dw), p(out), p(parts),
                 P, 8, s)
        nat.call("ffno_gn_finalize", p(parts), P, C, 8, p(one), p(zero), 1e-5, p(coef_out), p(gst), s)
        nat.call("ffno_mlp2_bwd", p(x), p(up), p(pre), V, C, p(m1), p(m2t), p(m1t), p(ab), s)
        nat.call("ffno_mlp2_jvp", p(x), p(xd), V, C, p(m1), p(m2), p(jv), s)
        nat.call("ffno_gate_jvp", p(x), p(xd), V, C, p(g1), p(g2), p(gj), s)
        nat.call("ffno_gate_bwd", p(x), p(up), p(xd), p(pre), V, C, p(g1), p(g2), p(g2t), p(g1t), p(g1), p(g2),
                 p(g2t), p(g1t), None, p(gb), None, s)
        torch.cuda.synchronize()
        run.inputs = [t.double() for t in (x, xd, pre, up, g1, g2, m1, m2, dw, coefs)]
        return gate, x1, out, ab, jv, gj, gb, gst

    gate, x1, out, ab, jv, gj, gb, gst = _both(run)
    x, xd, pre, up, g1, g2, m1, m2, dw, cf = run.inputs
    f_gate = lambda a: a * torch.sigmoid(F.gelu(a @ g1) @ g2)
    f_mlp = lambda a: F.gelu(a @ m1) @ m2
    _close(gate, f_gate(x))
    a1 = x + 0.7 * F.gelu((pre - cf[0]) * cf[1] + cf[2])
    _close(x1, a1)
    _close(out, f_mlp(a1))
    grp = out.double().reshape(V, 8, C // 8)
    tot = dw.sum() * (C // 8)
    mean = (dw[:, None, None] * grp).sum((0, 2)) / tot
    var = (dw[:, None, None] * (grp - mean[:, None]) ** 2).sum((0, 2)) / tot
    _close(gst[:, 0], mean)
    _close(gst[:, 1], (var + 1e-5).rsqrt())
    _close(gst[:, 2], tot.expand(8))
    _close(ab, pre + torch.autograd.functional.vjp(f_mlp, x, up)[1])
    _close(jv, torch.func.jvp(f_mlp, (x,), (xd,))[1])
    _close(gj, torch.func.jvp(f_gate, (x,), (xd,))[1])
    vjp = lambda v: torch.autograd.functional.vjp(f_gate, x, v)[1]
    _close(gb, pre + vjp(up) + vjp(xd))


@pytest.mark.parametrize("C", [16, 32, 64, 96])
@pytest.mark.parametrize("V", [1, 70, 129])
def test_fusion_chain(C, V):
    from ffnoml_gb300 import _native as nat
    s = torch.cuda.current_stream().cuda_stream
    P = nat.lib().ffno_stats_parts(V)

    def run(off):
        g = torch.Generator().manual_seed(C + V)
        x, sp, vp, xd, sd, vd, up, base = (_buf((V, C), off, g) for _ in range(8))
        w = lambda k, n: _buf((k, n), off, g).mul_(k ** -0.5)
        wg1, wg2, wf1, wf2 = w(3 * C, C), w(C, 2 * C), w(2 * C, 2 * C), w(2 * C, C)
        tr = lambda t: _buf(tuple(t.t().shape), off).copy_(t.t())
        wg1t, wg2t, wf1t, wf2t = tr(wg1), tr(wg2), tr(wf1), tr(wf2)
        bg = _buf((2 * C,), off, g)
        sc, vc = _buf((3, C), off, g), _buf((3, C), off, g)
        dw = _buf((V,), off, g).abs_()
        out, od, xb, sb, vb = (_buf((V, C), off) for _ in range(5))
        parts = torch.empty(P, 8, 3, dtype=torch.float64, device="cuda")
        p = lambda t: t.data_ptr()
        nat.call("ffno_fuse_fwd", p(x), p(sp), p(sc), p(vp), p(vc), V, C, p(wg1), p(wg2), p(bg), p(wf1), p(wf2), p(dw),
                 p(out), p(parts), P, 8, s)
        nat.call("ffno_fuse_jvp", p(x), p(xd), p(sp), p(sc), p(vp), p(vc), p(sd), p(vd), V, C, p(wg1), p(wg2), p(bg),
                 p(wf1), p(wf2), p(od), s)
        nat.call("ffno_fuse_bwd", p(x), p(sp), p(sc), p(vp), p(vc), p(up), p(base), V, C, p(wg1), p(wg2), p(bg), p(wf1),
                 p(wf2t), p(wf1t), p(wg2t), p(wg1t), p(xb), p(sb), p(vb), s)
        torch.cuda.synchronize()
        run.inputs = [t.double() for t in (x, sp, vp, xd, sd, vd, up, base, wg1, wg2, wf1, wf2, bg, sc, vc)]
        return out, od, xb, sb, vb

    out, od, xb, sb, vb = _both(run)
    x, sp, vp, xd, sd, vd, up, base, wg1, wg2, wf1, wf2, bg, sc, vc = run.inputs

    def f(a, s_, v_):
        gates = torch.sigmoid(F.gelu(torch.cat([a, s_, v_], 1) @ wg1) @ wg2 + bg)
        b = torch.cat([s_, v_], 1) * gates
        return F.gelu(b @ wf1) @ wf2 + 0.5 * (b[:, :C] + b[:, C:])

    s_, v_ = F.gelu((sp - sc[0]) * sc[1] + sc[2]), F.gelu((vp - vc[0]) * vc[1] + vc[2])
    _close(out, f(x, s_, v_))
    _close(od, torch.func.jvp(f, (x, s_, v_), (xd, sd, vd))[1])
    gx, gs, gv = torch.autograd.functional.vjp(f, (x, s_, v_), up)[1]
    _close(xb, base + gx)
    _close(sb, gs)
    _close(vb, gv)


@pytest.mark.parametrize("M,K,N,nb", [(1, 1, 16, 3), (16, 17, 64, 5), (33, 16, 96, 2), (50, 15, 32, 7), (66, 101, 64, 3),
                                      (96, 90, 16, 9), (128, 130, 64, 2), (130, 33, 96, 3), (145, 40, 64, 1),
                                      (260, 48, 20, 4), (24, 20, 7, 5)])
def test_transform_shapes(M, K, N, nb):
    """Every row split (M), ragged K, column tiles across batch elements, N not a multiple of four, accumulation, a table
    per batch element; in a two-part input row layout."""
    from ffnoml_gb300 import _native as nat
    s = torch.cuda.current_stream().cuda_stream
    half = (K + 1) // 2

    def run(off):
        g = torch.Generator().manual_seed(M * K + N)
        T = _buf((nb, M, K), off, g)
        rows = _buf((2, nb, half, N), off, g)       # k < half in part 0, the rest in part 1
        start = _buf((nb, M, N), off, g)
        once, twice, per = (_buf((nb, M, N), off) for _ in range(3))
        twice.copy_(start)
        d = nat.XformDesc(nb=nb, nb2=1, in_b1=half * N, in_b2=0, out_b1=M * N, out_b2=0, K=K, M=M, N=N, in_split=half,
                          in_hi=nb * half * N, in_lo=N, out_split=1 << 30, out_hi=0, out_lo=N)
        nat.call("ffno_xform", T.data_ptr(), rows.data_ptr(), once.data_ptr(), d, 0, s)
        nat.call("ffno_xform", T.data_ptr(), rows.data_ptr(), twice.data_ptr(), d, 1, s)
        nat.call("ffno_xform_pt", T.data_ptr(), M * K, rows.data_ptr(), per.data_ptr(), d, 0, s)
        torch.cuda.synchronize()
        run.inputs = (T.double(), torch.cat([rows[0], rows[1]], 1)[:, :K].double(), start.double())
        return once, twice, per

    once, twice, per = _both(run)
    T, x, start = run.inputs
    _close(once, T[0] @ x)
    _close(twice, start + T[0] @ x)
    _close(per, T @ x)


@pytest.mark.parametrize("C", [16, 32, 64, 96])
@pytest.mark.parametrize("rank", [0, 1, 8, 16])
def test_mixing(C, rank):
    from ffnoml_gb300 import _native as nat
    s = torch.cuda.current_stream().cuda_stream
    Fq, nb = 3, 70

    def run(off):
        g = torch.Generator().manual_seed(C + rank)
        x = _buf((2, Fq, nb, C), off, g)
        w = _buf((2 * C, 2 * C), off, g).mul_((2 * C) ** -0.5)
        gt = _buf((Fq, 2), off, g)
        u, v = (_buf((Fq, C, rank), off, g), _buf((Fq, rank, C), off, g).mul_(C ** -0.5)) if rank else (None, None)
        y = _buf((2, Fq, nb, C), off)
        ptr = lambda t: None if t is None else t.data_ptr()
        nat.call("ffno_spectral_mix", x.data_ptr(), y.data_ptr(), Fq, nb, nb * C, C, Fq * nb * C, C, w.data_ptr(),
                 gt.data_ptr(), ptr(u), ptr(v), rank, s)
        torch.cuda.synchronize()
        run.inputs = [None if t is None else t.double() for t in (x, w, gt, u, v)]
        return (y,)

    (y,) = _both(run)
    x, w, gt, u, v = run.inputs
    big = torch.cat([x[0], x[1]], -1) @ w
    a = torch.complex(big[..., :C], big[..., C:]) * torch.complex(gt[:, 0], gt[:, 1])[:, None, None]
    if rank:
        z = torch.complex(x[0], x[1])
        a = a + (z @ v.transpose(1, 2).to(z.dtype)) @ u.transpose(1, 2).to(z.dtype)
    _close(y, torch.stack([a.real, a.imag]))
