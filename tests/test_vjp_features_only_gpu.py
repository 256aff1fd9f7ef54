"""The input VJP when the heights take no gradient (z_scale.requires_grad False): the feature gradient is the one of the
full VJP bit for bit, z_scale gets none, on shared and per-column height grids, in both precisions, for two samples."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", ["fp32", "bf16"])
@pytest.mark.parametrize("columns", [False, True])
@pytest.mark.parametrize("width", [32, 96])
def test_feature_gradient_does_not_depend_on_the_heights_gradient(precision, columns, width):
    from ffnoml_gb300 import create_ffno3d
    torch.manual_seed(3)
    m = create_ffno3d(6, 6, atoms=["H"], width=width, n_layers=2, hidden_spectral=16, hidden_vertical=16,
                      z_min_wavelength=40.0 / 15).cuda().eval().set_precision(precision)
    B, D, H, W = 2, 19, 6, 7
    g = torch.Generator().manual_seed(1)
    x = torch.randn(B, 6, D, H, W, generator=g).cuda()
    z = torch.linspace(14.0, -1.0, D)[None, :, None, None].expand(B, D, H, W).clone()
    if columns:
        z = z * (1.0 + 0.01 * torch.rand(B, 1, H, W, generator=g))
    cot = torch.randn(B, 6, D, H, W, generator=g).cuda()

    def grads(heights):
        xx, zz = x.clone().requires_grad_(True), z.cuda().requires_grad_(heights)
        m(xx, zz, 48e3, 48e3).backward(cot)
        return xx.grad, zz.grad

    full, zbar = grads(True)
    alone, none = grads(False)
    assert torch.equal(full, alone)
    assert zbar is not None and bool(torch.isfinite(zbar).all()) and none is None
