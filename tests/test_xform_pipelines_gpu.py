"""Tensor-core transforms against float64 where the number of pipelines an SM (resident tables: four, three, two) or of
CTAs an SM (streamed tables: three, two) changes, with ragged rows, columns and items and with more items than slots."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("N", [64, 200])
@pytest.mark.parametrize("nb", [3, 701])
@pytest.mark.parametrize("kind,M,K", [("resident", 30, 40), ("resident", 128, 150), ("resident", 129, 100),
                                      ("resident", 160, 33), ("resident", 161, 96), ("streamed", 100, 300),
                                      ("streamed", 128, 33), ("streamed", 129, 31), ("streamed", 256, 200)])
def test_xform_pipelines(kind, M, K, nb, N):
    from ffnoml_gb300 import _native as nat
    from ffnoml_gb300.executor import TcXform
    g = torch.Generator().manual_seed(M + K + nb + N)
    T = torch.randn(M, K, generator=g, dtype=torch.float64)
    x = torch.randn(nb, K, N, generator=g).cuda()
    out = torch.full((nb, M, N), float("nan"), device="cuda")
    err = torch.zeros(1, dtype=torch.int32, device="cuda")
    d = nat.XformDesc(nb=nb, nb2=1, in_b1=K * N, in_b2=0, out_b1=M * N, out_b2=0, K=K, M=M, N=N, in_split=K, in_hi=0,
                      in_lo=N, out_split=M, out_hi=0, out_lo=N)
    (_, _, _, _, packed, res), = TcXform(T.numpy(), torch.device("cuda")).slices
    s = torch.cuda.current_stream().cuda_stream
    if kind == "resident":
        nat.call("ffno_xform_tcr", res[0].data_ptr(), res[1], res[2], x.data_ptr(), out.data_ptr(), d, 0,
                 err.data_ptr(), s)
    else:
        nat.call("ffno_xform_tc", packed.data_ptr(), x.data_ptr(), out.data_ptr(), d, 0, err.data_ptr(), s)
    torch.cuda.synchronize()
    assert int(err.item()) == 0
    Tc = T.cuda()
    ref, mag = Tc @ x.double(), Tc.abs() @ x.double().abs()
    # split BF16: the dropped lo * lo product and the two roundings of lo are 2^-18 each, and 3 K additions in FP32
    # (2^-23 each where the accumulator truncates)
    assert ((out.double() - ref).abs() <= (3 * 2.0 ** -18 + 3 * K * 2.0 ** -23) * mag).all()
