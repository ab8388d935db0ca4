"""bf16 GEMM with K cut over the CTAs of a cluster, at the edges of its tiles, k-blocks and K ranges, against float64."""
import pytest
import torch

pytestmark = pytest.mark.gpu
BF = torch.bfloat16


def _check(m, n, k, k2, bias):
    from mobilefinetuner_b200 import ops as O
    g = torch.Generator(device="cuda").manual_seed(m * 131 + n * 7 + k)

    def rnd(r, c, scale=1.0):
        return (torch.randn(r, c, device="cuda", generator=g) * scale).to(BF)
    a, b = rnd(m, k), rnd(n, k, 0.05)
    a2 = b2 = None
    if k2:           # panels of 64 columns: what lies past the second segment must not be read
        a2, b2 = torch.full((m, 64), float("nan"), device="cuda", dtype=BF), torch.full((n, 64), float("nan"), device="cuda", dtype=BF)
        a2[:, :k2], b2[:, :k2] = rnd(m, k2), rnd(n, k2, 0.05)
        a2, b2 = a2[:, :k2], b2[:, :k2]
    bs = torch.randn(n, device="cuda", generator=g) if bias else None
    ld = (n + 7) // 8 * 8
    out = torch.full((m + 1, ld), 7.0, device="cuda", dtype=BF)
    O.gemm_nt(a, b, a2=a2, b2=b2, bias=bs, alpha=0.5, out=out[:m, :n])
    want, mag = a.double() @ b.double().T, a.double().abs() @ b.double().abs().T
    if k2:
        want, mag = want + a2.double() @ b2.double().T, mag + a2.double().abs() @ b2.double().abs().T
    want = 0.5 * want + (bs.double() if bias else 0.0)
    # bf16 rounding of the result (2^-9 relative) and the f32 sums of k + k2 exact products, alpha, bias and the slices
    bound = 2.0 ** -8 * want.abs() + (k + k2 + 16) * 2.0 ** -24 * (mag + 1.0)
    assert bool(((out[:m, :n].double() - want).abs() <= bound).all())
    assert bool((out[m] == 7.0).all()) and bool((out[:m, n:] == 7.0).all())
    assert O.device_status() == 0


@pytest.mark.parametrize("m,n,k,k2,bias", [
    (512, 16, 13824, 0, False), (512, 48, 1152, 0, False), (129, 40, 2048, 0, False), (512, 1152, 13824, 32, False), (512, 1536, 1152, 48, False),
    (1, 64, 4096, 0, False), (1, 8, 4104, 0, True), (129, 72, 1352, 16, True), (437, 640, 2048, 8, False), (437, 8, 2048, 0, False), (512, 2304, 768, 8, True),
    (65, 128, 1000, 0, True), (1170, 896, 4864, 0, False), (300, 200, 1160, 64, True), (512, 50, 6912, 0, True), (1000, 768, 3072, 0, False)])
def test_gemm_ksplit(m, n, k, k2, bias):
    from mobilefinetuner_b200 import ops as O
    cols, ranges = O.gemm_nt_ksplit_plan(m, n, k, k2)
    assert cols in (64, 128) and 2 <= ranges <= 8, "the shape no longer reaches the K-split kernel"
    _check(m, n, k, k2, bias)


@pytest.mark.parametrize("m,n,k,k2", [(2100, 2200, 640, 16), (2305, 2000, 1152, 0), (4097, 1160, 264, 8)])
def test_pair_kernel_ragged_bf16(m, n, k, k2):
    """Ragged bf16 outputs of many tiles: the K-split kernel leaves them to 256-wide pair tiles."""
    from mobilefinetuner_b200 import ops as O
    assert O.gemm_nt_ksplit_plan(m, n, k, k2) == (0, 1) and O.gemm_nt_tile_cols(m, n, k, k2) == 256
    _check(m, n, k, k2, True)


@pytest.mark.parametrize("m,n,k,k2,bias", [(130, 40, 520, 0, False), (1, 64, 704, 0, False), (437, 8, 640, 0, False), (1985, 896, 4864, 0, False)])
def test_shapes_of_the_other_kernels(m, n, k, k2, bias):
    from mobilefinetuner_b200 import ops as O
    assert O.gemm_nt_ksplit_plan(m, n, k, k2) == (0, 1)
    _check(m, n, k, k2, bias)


# the gated-MLP calls have the bits of the plain product and the activation kernel, also where that product is K-split;
# gate|up and its gradient with row strides of their own
@pytest.mark.parametrize("swiglu", [False, True])
@pytest.mark.parametrize("m,inter,k,r", [(512, 2048, 640, 0), (512, 2048, 640, 16), (257, 448, 1160, 16), (300, 256, 2048, 0)])
def test_gated_mlp_calls_keep_the_bits(swiglu, m, inter, k, r):
    from mobilefinetuner_b200 import _lib as L
    from mobilefinetuner_b200 import ops as O
    kind = L.ACT_SWIGLU if swiglu else L.ACT_GEGLU
    g = torch.Generator(device="cuda").manual_seed(m + inter)
    st = torch.cuda.current_stream().cuda_stream

    def rnd(rows, cols, scale=1.0):
        return (torch.randn(rows, cols, device="cuda", generator=g) * scale).to(BF)
    dy, wd, gu_wide = rnd(m, k), rnd(inter, k, 0.05), rnd(m, 2 * inter + 16)
    gu = gu_wide[:, :2 * inter]
    a2, b2 = (rnd(m, 64)[:, :r], rnd(inter, 64, 0.05)[:, :r]) if r else (None, None)
    assert O.gemm_nt_ksplit_plan(m, inter, k, r)[0] > 0

    def bwd(gu, dgu):
        L.call("mft_glu_linear_bwd", kind, dy.data_ptr(), k, wd.data_ptr(), k, m, inter, k, a2.data_ptr() if r else None, 64, b2.data_ptr() if r else None,
               64, r, gu.data_ptr(), gu.stride(0), dgu.data_ptr(), dgu.stride(0), st)
    dgu_wide = torch.full((m + 1, 2 * inter + 8), 3.0, device="cuda", dtype=BF)
    bwd(gu, dgu_wide[:m, :2 * inter])
    dg, du = O.act_bwd(kind, O.gemm_nt(dy, wd, a2=a2, b2=b2), gu[:, :inter].contiguous(), gu[:, inter:].contiguous())
    assert torch.equal(dgu_wide[:m, :inter], dg) and torch.equal(dgu_wide[:m, inter:2 * inter], du)
    assert bool((dgu_wide[m] == 3.0).all()) and bool((dgu_wide[:, 2 * inter:] == 3.0).all())
    # in place over the saved gate|up: taken as before, equal to the rounding of d(act) to bf16
    both = gu.contiguous()
    bwd(both, both)
    for x, y in ((both[:, :inter], dg), (both[:, inter:], du)):
        assert (x.float() - y.float()).norm() <= 2.0 ** -8 * y.float().norm()
    # forward
    if inter % 128 == 0 and O.gemm_nt_ksplit_plan(m, 2 * inter, k, r)[0] > 0:
        x, w = dy, rnd(2 * inter, k, 0.05)
        xa, bp = (rnd(m, 64)[:, :r], rnd(2 * inter, 64, 0.05)[:, :r]) if r else (None, None)
        bias = torch.randn(2 * inter, device="cuda", generator=g)
        gu_f, act_wide = torch.empty(m, 2 * inter + 8, device="cuda", dtype=BF)[:, :2 * inter], torch.full((m, inter + 8), 3.0, device="cuda", dtype=BF)
        L.call("mft_glu_linear_fwd", kind, x.data_ptr(), k, w.data_ptr(), k, m, inter, k, xa.data_ptr() if r else None, 64, bp.data_ptr() if r else None, 64, r,
               bias.data_ptr(), gu_f.data_ptr(), gu_f.stride(0), act_wide.data_ptr(), act_wide.stride(0), st)
        want = O.gemm_nt(x, w, a2=xa, b2=bp, bias=bias)
        assert torch.equal(gu_f, want) and torch.equal(act_wide[:, :inter], O.act_fwd(kind, want[:, :inter], want[:, inter:]))
        assert bool((act_wide[:, inter:] == 3.0).all())
    assert O.device_status() == 0
