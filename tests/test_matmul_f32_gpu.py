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


@pytest.mark.parametrize("batch,m,n,k", [(1, 32, 32, 1), (1, 33, 31, 32), (1, 128, 128, 447), (1, 128, 128, 448), (1, 128, 130, 255), (1, 64, 64, 256),
                                         (148, 32, 32, 33), (149, 7, 9, 31), (149, 7, 9, 32), (296, 16, 16, 100), (297, 16, 16, 100)])
@pytest.mark.parametrize("trans_b", [0, 1])
def test_small_products_on_both_sides_of_the_rule(batch, m, n, k, trans_b):
    test_matmul_f32(batch, m, n, k, trans_b)


@pytest.mark.parametrize("off", [(1, 0, 0), (0, 1, 0), (0, 0, 1), (2, 3, 1)])       # elements that A, B, C start after a 16-byte boundary
@pytest.mark.parametrize("m,n,k", [(8, 12, 16), (512, 512, 64), (64, 64, 1024), (1536, 1532, 20)])
def test_operands_off_16_bytes(m, n, k, off):
    from mobilefinetuner_b200 import _lib as L
    L.init(0)
    g = torch.Generator(device="cuda").manual_seed(m + k)
    bufs = [torch.randn(3 + 2 * (r * c + 1), device="cuda", generator=g) for r, c in ((m, k), (k, n), (m, n))]
    # two products whose operands lie an odd number of elements apart
    views = [[buf[o + i * (r * c + 1):][:r * c].view(r, c) for i in range(2)] for buf, o, (r, c) in zip(bufs, off, ((m, k), (k, n), (m, n)))]
    (a, b, c) = views
    L.call("mft_matmul_f32", a[0].data_ptr(), b[0].data_ptr(), c[0].data_ptr(), 2, m, n, k, m * k + 1, k * n + 1, m * n + 1, 0,
           torch.cuda.current_stream().cuda_stream)
    for i in range(2):
        bound = (k + 1) * 2.0 ** -24 * (a[i].double().abs() @ b[i].double().abs())      # as above
        assert bool(((c[i].double() - a[i].double() @ b[i].double()).abs() <= bound).all())
