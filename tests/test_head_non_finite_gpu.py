"""Non-finite values and unusual constants in the level-fraction head: what is infinite or not a number in the float64
oracle is so here too, with the same sign, and every other output keeps its accuracy (FP32 precision: one float32 rounding
of the output and one of the oracle's own inputs, 2^-23; split-BF16 precision: FP32 level weights, 1e-5; both of the
larger of the output and 1, the bounds of test_head_ranges_gpu.py)."""
import math

import pytest
import torch

from golden_io import model_config

pytestmark = pytest.mark.gpu

CFG = dict(width=16, n_layers=1, hidden_spectral=16, hidden_vertical=16, z_min_wavelength=0.5, atoms=["H", "CA"])
INF = float("inf")


def _model(precision):
    from ffnoml_gb300 import FFNO3D
    torch.manual_seed(0)
    m = FFNO3D(**model_config(CFG)).cuda().eval().set_precision(precision)
    m.set_normalization([4.75, 0, 0, 0, 17.5, -8.0], [0.72, 5, 5, 5, 2.0, 2.3], 20 * torch.ones(12), 3 * torch.ones(12))
    return m


def _voxels(n=40):
    g = torch.Generator().manual_seed(3)
    head = torch.randn(1, 14, n, 1, 1, generator=g)
    x = 0.5 * torch.randn(1, 6, n, 1, 1, generator=g)
    return head, x


@pytest.mark.parametrize("precision", ["fp32", "bf16"])
@pytest.mark.parametrize("bad", [float("nan"), INF, -INF])
@pytest.mark.parametrize("where", ["density", "level", "total"])
def test_head_output_of_non_finite_values(precision, bad, where):
    from oracle.ffno_oracle import OracleFFNO3D
    m = _model(precision)
    head, x = _voxels()
    {"density": x[0, 5], "level": head[0, 2], "total": head[0, 6]}[where][5] = bad
    y = m.head_output(head.cuda(), x.cuda()).double().cpu()
    state = {k: v.double().cpu() for k, v in m.state_dict().items()}
    ref = OracleFFNO3D(state, model_config(CFG), torch.float64).head(head.double(), x.double())
    assert torch.equal(torch.isnan(y), torch.isnan(ref))
    assert torch.equal(torch.isposinf(y), torch.isposinf(ref)) and torch.equal(torch.isneginf(y), torch.isneginf(ref))
    fine = torch.isfinite(ref)
    err = ((y - ref).abs() / ref.abs().clamp_min(1.0))[fine]
    assert err.max().item() <= (2.0 ** -23 if precision == "fp32" else 1e-5)


def _dual(m, x, z, t):
    import torch.autograd.forward_ad as forward_ad
    with torch.no_grad(), forward_ad.dual_level():
        return [v.clone() for v in forward_ad.unpack_dual(m(forward_ad.make_dual(x, t), z, 48e3, 48e3))]


def _head_calls(m):
    """head_output and its VJP on voxels, and the model's forward-mode derivative on a small cube."""
    head, x = _voxels()
    hc, xc = head.cuda().requires_grad_(True), x.cuda().requires_grad_(True)
    y = m.head_output(hc, xc)
    y.backward(torch.randn(y.shape, generator=torch.Generator().manual_seed(2)).cuda())
    g = torch.Generator().manual_seed(4)
    cube, tangent = torch.randn(2, 1, 6, 12, 6, 5, generator=g).cuda()
    z = torch.linspace(2.0, 0.0, 12)[None, :, None, None].expand(1, 12, 6, 5).contiguous().cuda()
    return [y.detach(), hc.grad, xc.grad] + _dual(m, cube, z, tangent)


@pytest.mark.parametrize("precision", ["fp32", "bf16"])
def test_total_bound_of_zero(precision):
    """A bound of zero holds the total at log10 rho: what a bound far below one rounding gives, bit for bit."""
    m = _model(precision)
    with torch.no_grad():
        for i in (6, 13):       # totals away from zero (0 / 0 is not a number)
            m.proj2.bias[i] = 1.0
    m.total_bound = 1e-30
    want = _head_calls(m)
    m = _model(precision)
    with torch.no_grad():
        for i in (6, 13):
            m.proj2.bias[i] = 1.0
    m.total_bound = 0.0
    for a, b in zip(_head_calls(m), want):
        assert bool(torch.isfinite(b).all())
        assert torch.equal(a, b)


@pytest.mark.parametrize("precision", ["fp32", "bf16"])
def test_total_of_zero_over_a_bound_of_zero(precision):
    """0 / 0 is not a number in the total term, nor in the levels that it is added to."""
    from oracle.ffno_oracle import OracleFFNO3D
    m = _model(precision)
    m.total_bound = 0.0
    head, x = _voxels()
    head[0, 6, 5] = 0.0
    y = m.head_output(head.cuda(), x.cuda()).cpu()
    state = {k: v.double().cpu() for k, v in m.state_dict().items()}
    ref = OracleFFNO3D(state, dict(model_config(CFG), total_bound=0.0), torch.float64).head(head.double(), x.double())
    assert bool(torch.isnan(ref[0, :6, 5]).all())
    assert torch.equal(torch.isnan(y), torch.isnan(ref))


@pytest.mark.parametrize("precision", ["fp32", "bf16"])
@pytest.mark.parametrize("bound", [1e-3, 1e5, 1e7, 1e14])
def test_total_bounds_from_small_to_none(precision, bound):
    """A large bound leaves the totals as they are: to the accuracy of the other outputs, not to that of the bound."""
    from oracle.ffno_oracle import OracleFFNO3D
    m = _model(precision)
    m.total_bound = bound
    head, x = _voxels()
    y = m.head_output(head.cuda(), x.cuda()).double().cpu()
    state = {k: v.double().cpu() for k, v in m.state_dict().items()}
    ref = OracleFFNO3D(state, dict(model_config(CFG), total_bound=torch.tensor(bound).item()), torch.float64).head(
        head.double(), x.double())
    err = (y - ref).abs() / ref.abs().clamp_min(1.0)
    assert err.max().item() <= (2.0 ** -23 if precision == "fp32" else 1e-5)


def test_output_scale_of_zero():
    """A level whose scale std_Y is zero: its outputs and its species' totals' gradients are infinite, as a division by
    zero makes them, not undefined."""
    m = _model("fp32")
    m.std_Y[2] = 0.0
    y, hb, xb, p, t = _head_calls(m)
    assert bool(torch.isinf(y[0, 2]).all()) and bool(torch.isinf(p[0, 2]).all())
    assert bool(torch.isinf(t[0, 2]).all())
    assert bool(torch.isinf(xb[0, 5]).all())                                   # the gradient in log10 rho
    assert bool(torch.isfinite(y[0, 6:]).all()) and bool(torch.isfinite(t[0, 6:]).all())


@pytest.mark.parametrize("precision", ["fp32", "bf16"])
@pytest.mark.parametrize("sign", [1.0, -1.0])      # x86's inf - inf is a NaN with the sign bit set, Arm's without
def test_level_energy_that_is_not_a_number(precision, sign):
    """A level energy that is not a number leaves every level of its species undefined, and the other species alone."""
    m = _model(precision)
    want = _head_calls(m)
    m = _model(precision)
    lg, ev, nd, di = (list(t) for t in m.lte_tables)
    ev[2] = math.copysign(float("nan"), sign)
    m.lte_tables = (lg, ev, nd, di)
    got = _head_calls(m)
    for i in (0, 3, 4):
        assert bool(torch.isnan(got[i][0, :6]).all())
        assert torch.equal(got[i][0, 6:], want[i][0, 6:])
    assert bool(torch.isnan(got[1][0, :6]).all()) and torch.equal(got[1][0, 7:], want[1][0, 7:])
