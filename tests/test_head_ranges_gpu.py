"""The level-fraction head's own FP64 exp, log and tanh (tables and Newton steps, csrc/common.cuh) over and past the
range where they are used, against the float64 oracle, and its two-float assembly of the split-BF16 path: forward and
VJP on cold and hot, thin and dense voxels, head channels from tiny to huge, and non-finite inputs.

Bounds: FP32 precision evaluates everything in FP64 and rounds once, so an output is within one float32 rounding
(2^-24) of the oracle's, taken twice for the oracle's own rounding of its inputs; the split-BF16 precision has FP32 level
weights: 1e-5 of the largest output (the bound of the head's other tests)."""
import pytest
import torch

from golden_io import model_config

pytestmark = pytest.mark.gpu

CFG = dict(width=16, n_layers=1, hidden_spectral=16, hidden_vertical=16, z_min_wavelength=0.5, atoms=["H", "CA"])


def _model(precision):
    from ffnoml_gb300 import FFNO3D
    torch.manual_seed(0)
    m = FFNO3D(**model_config(CFG)).cuda().eval().set_precision(precision)
    m.set_normalization([4.75, 0, 0, 0, 17.5, -8.0], [0.72, 5, 5, 5, 2.0, 2.3], 20 * torch.ones(12), 3 * torch.ones(12))
    return m


def _voxels(scale, n=64):
    g = torch.Generator().manual_seed(int(scale * 1e3) + 1)
    head = scale * torch.randn(1, 14, n, 1, 1, generator=g)
    x = torch.randn(1, 6, n, 1, 1, generator=g)
    lt = torch.linspace(0.3, 16.0, n)           # log10 T: both sides of the range of the tables
    x[0, 0, :, 0, 0] = (lt - 4.75) / 0.72
    x[0, 4, :, 0, 0] = (torch.linspace(-45.0, 45.0, n)[torch.randperm(n, generator=g)] - 17.5) / 2.0
    return head, x


@pytest.mark.parametrize("scale", [1e-6, 1.0, 30.0, 3e4, 1e7])
@pytest.mark.parametrize("precision", ["fp32", "bf16"])
def test_head_over_its_range(scale, precision):
    from oracle.ffno_oracle import OracleFFNO3D
    m = _model(precision)
    head, x = _voxels(scale)
    if precision == "bf16":                     # FP32 level weights overflow far outside the atmosphere
        x[:, 0] = ((x[:, 0] * 0.72 + 4.75).clamp(3.3, 7.0) - 4.75) / 0.72
        x[:, 4] = ((x[:, 4] * 2.0 + 17.5).clamp(12.0, 23.0) - 17.5) / 2.0
    y = m.head_output(head.cuda(), x.cuda()).double().cpu()
    state = {k: v.double().cpu() for k, v in m.state_dict().items()}
    ref = OracleFFNO3D(state, model_config(CFG), torch.float64).head(head.double(), x.double())
    # the two rounded inputs log10 T, log10 ne enter the oracle and the kernel as the same float32 values
    big = ref.abs().clamp_min(1.0)
    err = ((y - ref).abs() / big)
    assert torch.equal(torch.isfinite(y), torch.isfinite(ref.float()))
    fine = torch.isfinite(ref)
    print(f"{precision} {scale:g}: {err[fine].max().item():.2e}")
    assert err[fine].max().item() <= (2.0 ** -23 if precision == "fp32" else 1e-5)


@pytest.mark.parametrize("scale", [1e-6, 1.0, 30.0])
def test_head_vjp_over_its_range(scale):
    from oracle.ffno_oracle import OracleFFNO3D
    m = _model("fp32")
    head, x = _voxels(scale)
    keep = ((x[0, 0, :, 0, 0] * 0.72 + 4.75) > 2.5) & ((x[0, 4, :, 0, 0] * 2.0 + 17.5) < 30)
    head, x = head[:, :, keep], x[:, :, keep]
    cot = torch.randn(1, 12, head.shape[2], 1, 1, generator=torch.Generator().manual_seed(2))
    hc, xc = head.cuda().requires_grad_(True), x.cuda().requires_grad_(True)
    m.head_output(hc, xc).backward(cot.cuda())
    state = {k: v.double().cpu() for k, v in m.state_dict().items()}
    hr, xr = head.double().requires_grad_(True), x.double().requires_grad_(True)
    hb, xb = torch.autograd.grad(OracleFFNO3D(state, model_config(CFG), torch.float64).head(hr, xr), (hr, xr),
                                 cot.double())
    for got, want in ((hc.grad, hb), (xc.grad, xb)):
        d = (got.double().cpu() - want).abs()
        # per voxel: one float32 rounding of sums whose terms are at most the voxel's largest gradient (14 terms)
        size = want.abs().amax(1, keepdim=True).clamp_min(1e-30)
        assert (d / size).max().item() <= 14 * 2.0 ** -23


@pytest.mark.parametrize("precision", ["fp32", "bf16"])
@pytest.mark.parametrize("bad", [float("nan"), float("inf"), -float("inf")])
@pytest.mark.parametrize("where", ["total", "level", "temperature"])
def test_non_finite_voxels_stay_their_own(precision, bad, where):
    """A non-finite value leaves the other voxels' bits alone, and its own voxel is not made finite by the tables."""
    m = _model(precision)
    head, x = _voxels(1.0, 40)
    x[:, 0] = 0.1
    x[:, 4] = 0.1
    good = m.head_output(head.cuda(), x.cuda())
    h2, x2 = head.clone(), x.clone()
    {"total": h2[0, 6], "level": h2[0, 2], "temperature": x2[0, 0]}[where][5] = bad
    y = m.head_output(h2.cuda(), x2.cuda())
    rest = torch.arange(40) != 5
    assert torch.equal(y[:, :, rest], good[:, :, rest])
    if where == "total" and bad == bad:          # tanh of an infinite total is the bound
        assert bool(torch.isfinite(y[0, :6, 5]).all())
    else:
        assert not bool(torch.isfinite(y[0, :6, 5]).all())
