"""The f32 matrix product of the eager operators at the edges of its tiles, slabs and K ranges, against float64."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("batch,m,n,k", [(1, 1, 1, 1), (3, 5, 7, 3), (2, 64, 64, 16), (1, 65, 63, 17), (1, 128, 132, 1024), (1, 61, 60, 4864),
                                         (1, 2000, 1500, 33), (1, 1024, 2432, 68), (4, 130, 66, 300), (1, 1530, 1500, 68),
                                         (1, 1536, 1531, 17)])
@pytest.mark.parametrize("trans_b", [0, 1])
def test_matmul_f32(batch, m, n, k, trans_b):
    from mobilefinetuner_b200 import _lib as L
    L.init(0)
    g = torch.Generator(device="cuda").manual_seed(m * 7919 + n * 31 + k)
    a = torch.randn(batch, m, k, device="cuda", generator=g)
    b = torch.randn((batch, n, k) if trans_b else (batch, k, n), device="cuda", generator=g)
    c = torch.full((batch, m, n), float("nan"), device="cuda")
    L.call("mft_matmul_f32", a.data_ptr(), b.data_ptr(), c.data_ptr(), batch, m, n, k, m * k, n * k, m * n, trans_b,
           torch.cuda.current_stream().cuda_stream)
    bd = b.double().transpose(1, 2) if trans_b else b.double()
    # every f32 summation order of k products stays within k * 2^-24 * sum |a||b|
    bound = (k + 1) * 2.0 ** -24 * (a.double().abs() @ bd.abs())
    assert bool(((c.double() - a.double() @ bd).abs() <= bound).all())
