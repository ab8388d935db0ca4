"""RMSNorm forward kernels by row count: the same row gives the same bits whichever kernel takes the call."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rows,dim", [(3000, 264), (3001, 512), (2048, 520), (2049, 640), (2051, 776), (3003, 1024), (2050, 1152), (2048, 1536),
                                      (2688, 1544), (6001, 1800), (6000, 2048)])
@pytest.mark.parametrize("bf16_in", [False, True])
def test_single_norm(rows, dim, bf16_in):
    from mobilefinetuner_b200 import ops as O
    g = torch.Generator(device="cuda").manual_seed(rows + dim)
    x = torch.randn(rows, dim, device="cuda", generator=g)
    x = x.bfloat16() if bf16_in else x
    w = torch.randn(dim, device="cuda", generator=g) * 0.1
    y, rstd = O.rms_norm_fwd(x, w, 1e-6, 1, out_dtype=torch.float32)[:2]
    for lo in range(0, rows, 1500):                  # calls of few rows: the other kernel
        ys, rs = O.rms_norm_fwd(x[lo:lo + 1500], w, 1e-6, 1, out_dtype=torch.float32)[:2]
        assert torch.equal(y[lo:lo + 1500], ys) and torch.equal(rstd[lo:lo + 1500], rs)
    xd = x.double()
    want = xd * (xd.square().mean(-1, keepdim=True) + 1e-6).rsqrt() * (1.0 + w.double())
    # f32 sums of dim squares (relative error below dim * 2^-24, halved by the root) and four roundings
    assert bool(((y.double() - want).abs() <= (dim / 2 + 8) * 2.0 ** -24 * want.abs()).all())


@pytest.mark.parametrize("rows,dim", [(8192, 8), (8193, 256), (8195, 640), (8192, 1152), (8194, 1544), (8192, 2048)])
def test_norm_pair(rows, dim):
    from mobilefinetuner_b200 import ops as O
    g = torch.Generator(device="cuda").manual_seed(rows + dim)
    y, x = torch.randn(rows, dim, device="cuda", generator=g).bfloat16(), torch.randn(rows, dim, device="cuda", generator=g)
    wp, wn = (torch.randn(dim, device="cuda", generator=g) * 0.1 for _ in range(2))
    got = O.rms_norm_add_norm_fwd(y, wp, x, wn, 1e-6)
    for lo in range(0, rows, 4000):
        part = O.rms_norm_add_norm_fwd(y[lo:lo + 4000], wp, x[lo:lo + 4000], wn, 1e-6)
        assert all(torch.equal(a[lo:lo + 4000], b) for a, b in zip(got, part))
    # and the two separate calls, which take their kernels by their own rules
    _, rp, s = O.rms_norm_fwd(y, wp, 1e-6, 1, out_dtype=torch.bfloat16, residual=x)
    h, rn = O.rms_norm_fwd(s, wn, 1e-6, 1, out_dtype=torch.bfloat16)[:2]
    assert all(torch.equal(a, b) for a, b in zip(got, (s, rp, h, rn)))
