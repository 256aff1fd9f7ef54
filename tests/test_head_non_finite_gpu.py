"""Non-finite values in the level-fraction head: what is infinite or not a number in the float64 oracle is so here too,
with the same sign, and every other output keeps its accuracy (FP32 precision: one float32 rounding of the output and one
of the oracle's own inputs, 2^-23; split-BF16 precision: FP32 level weights, 1e-5; both of the larger of the output and 1,
the bounds of test_head_ranges_gpu.py)."""
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
