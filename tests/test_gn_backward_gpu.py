"""GroupNorm-backward statistics and application against float64: every width and activation mode of the eight-group
kernels, sizes around a warp's and a round's voxels, and other group counts (the general kernels)."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _act_grad(mode, y):
    if mode == 0:
        return torch.ones_like(y)
    return torch.special.ndtr(y) + y * torch.exp(-y * y / 2) / (2 * torch.pi) ** 0.5


@pytest.mark.parametrize("mode", [0, 1, 2])
@pytest.mark.parametrize("C,groups,V", [(C, 8, V) for C in (16, 32, 64, 96) for V in (1, 31, 4097, 40003)]
                         + [(64, 4, 4097), (96, 6, 4097), (16, 2, 31)])
def test_gn_backward(C, groups, V, mode):
    from ffnoml_gb300 import _native as nat
    g = torch.Generator().manual_seed(C + V + mode)
    rnd = lambda *s: torch.randn(*s, generator=g).cuda()  # noqa: E731
    u, pre, gamma, beta = rnd(V, C), 0.5 + 1.5 * rnd(V, C), 1 + 0.2 * rnd(C), 0.1 * rnd(C)
    dw = 0.5 + torch.rand(V, generator=g).cuda()
    wbar0, r, eps, cpg = rnd(V), 0.75, 1e-5, C // groups
    x = pre.double().reshape(V, groups, cpg)
    wd = dw.double()[:, None, None]
    T = dw.double().sum() * cpg
    mean = (x * wd).sum((0, 2)) / T
    rstd = ((((x - mean[None, :, None]) ** 2) * wd).sum((0, 2)) / T + eps).rsqrt()
    gst = torch.stack([mean, rstd, T.expand(groups)], 1).contiguous()
    xh = (x - mean[None, :, None]) * rstd[None, :, None]
    gm, bt = gamma.double().reshape(groups, cpg), beta.double().reshape(groups, cpg)
    ug = r * u.double().reshape(V, groups, cpg) * gm
    gh = ug * _act_grad(mode, xh * gm + bt)
    S1, S2 = gh.sum((0, 2)), (gh * xh).sum((0, 2))
    s = torch.cuda.current_stream().cuda_stream
    P = 152 * 3
    part = torch.full((P, groups, 2), float("nan"), dtype=torch.float64, device="cuda")
    sums = torch.empty(groups, 2, dtype=torch.float64, device="cuda")
    nat.call("ffno_gn_bwd_stats", mode, u.data_ptr(), r, pre.data_ptr(), gamma.data_ptr(), beta.data_ptr(),
             gst.data_ptr(), V, C, groups, part.data_ptr(), P, s)
    nat.call("ffno_gn_bwd_final", part.data_ptr(), P, groups, sums.data_ptr(), s)
    # A term gh has a relative rounding error of a few 2^-24, the activation derivative an absolute one of up to 1.5e-6
    # (mode 2's approximation), xhat one of a few 2^-24 (|mean| <= |x| + 4 std): 4e-6 of the sums of magnitudes.
    lim = 4e-6
    m1, m2 = ug.abs().sum((0, 2)), (ug * xh).abs().sum((0, 2)) + ug.abs().sum((0, 2))
    assert ((sums[:, 0] - S1).abs() <= lim * m1).all()
    assert ((sums[:, 1] - S2).abs() <= lim * m2).all()
    sums.copy_(torch.stack([S1, S2], 1))
    out, wbar = torch.empty_like(u), wbar0.clone()
    nat.call("ffno_gn_bwd_apply", mode, u.data_ptr(), r, pre.data_ptr(), gamma.data_ptr(), beta.data_ptr(),
             gst.data_ptr(), sums.data_ptr(), dw.data_ptr(), V, C, groups, eps, out.data_ptr(), wbar.data_ptr(), s)
    torch.cuda.synchronize()
    c1, c2, rs = S1[None, :, None] / T, S2[None, :, None] / T, rstd[None, :, None]
    ref = rs * (gh - wd * (c1 + xh * c2))
    mag = rs * (ug.abs() + wd * (c1.abs() + (1 + xh.abs()) * c2.abs()))
    assert ((out.double().reshape(V, groups, cpg) - ref).abs() <= lim * mag).all()
    vr2 = (1 - eps * rstd * rstd)[None, :, None]
    wref = wbar0.double() + (-c1 * xh - 0.5 * c2 * (xh * xh - vr2)).sum((1, 2))
    wmag = wbar0.double().abs() + (c1.abs() * (1 + xh.abs()) + c2.abs() * (1 + xh * xh)).sum((1, 2))
    assert ((wbar.double() - wref).abs() <= lim * wmag).all()
