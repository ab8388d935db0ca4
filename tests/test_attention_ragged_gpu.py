"""tcgen05 attention kernels on sequences that are no multiple of their 128-row tiles, against f32 torch."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _reference(q, k, v, d_o, scale, window):
    q, k, v = (x.float().detach().requires_grad_() for x in (q, k, v))
    rep, s = q.shape[1] // k.shape[1], q.shape[2]
    kk, vv = k.repeat_interleave(rep, 1), v.repeat_interleave(rep, 1)
    i, j = torch.arange(s, device=q.device)[:, None], torch.arange(s, device=q.device)[None, :]
    mask = (j <= i) & ((i - j < window) if window > 0 else True)
    logits = (q @ kk.transpose(-1, -2) * scale).masked_fill(~mask, float("-inf"))
    o = logits.softmax(-1) @ vv
    grads = torch.autograd.grad(o, (q, k, v), d_o.float())
    return (o, logits.logsumexp(-1), *grads)


# around the 128-row tile, the 64- / 32-key and 32-query tiles, the 32-query rule of the statistics' bulk copy, and both
# sides of the lengths from which the kernels are taken
@pytest.mark.parametrize("hd,heads,kv,seq,window", [
    (256, 4, 1, 2, 0), (256, 4, 1, 31, 0), (256, 4, 1, 97, 33), (256, 2, 1, 127, 0), (256, 4, 1, 129, 0), (256, 4, 1, 161, 64),
    (256, 4, 1, 256, 0), (256, 4, 1, 257, 0), (256, 4, 1, 1001, 512), (256, 4, 2, 640 + 32, 100), (64, 14, 2, 193, 0), (64, 14, 2, 385, 0),
    (64, 4, 2, 513, 0), (64, 4, 2, 544, 0), (64, 4, 1, 1023, 70), (128, 4, 2, 129, 0), (128, 4, 2, 600, 0), (128, 2, 1, 515, 96)])
def test_ragged_sequences(hd, heads, kv, seq, window):
    from mobilefinetuner_b200 import ops as O
    g = torch.Generator(device="cuda").manual_seed(seq)

    def rnd(n):
        return torch.randn(3, seq, n, hd, device="cuda", generator=g).bfloat16().permute(0, 2, 1, 3)
    q, k, v, d_o = rnd(heads), rnd(kv), rnd(kv), rnd(heads)
    # the sample in the middle is not a number: none of it may reach its neighbours through a tile's rows past the end
    for x in (q, k, v, d_o):
        x[1] = float("nan")
    scale = hd ** -0.5
    o, lse = O.attention_fwd(q, k, v, scale, window)
    got = (o, lse, *O.attention_bwd(q, k, v, o, d_o, lse, scale, window))
    keep = [0, 2]
    ref = _reference(q[keep], k[keep], v[keep], d_o[keep], scale, window)
    for name, a, b in zip(("o", "lse", "dq", "dk", "dv"), got, ref):
        a = a[keep].float()
        assert torch.isfinite(a).all(), name
        # P, dS and the results are rounded to bf16 (2^-9 each, sums of independent roundings below): 4 * 2^-9
        assert (a - b).norm() <= 2 ** -7 * b.norm(), (name, ((a - b).norm() / b.norm()).item())
        # no row is off on its own (rows of a few keys carry the full rounding of their terms)
        row = (a - b).norm(dim=-1) if a.dim() == 4 else (a - b).abs()
        size = b.norm(dim=-1) if a.dim() == 4 else b.abs()
        assert (row <= 2 ** -5 * (size + size.mean())).all(), name


# the mma.sync kernels store 4 bytes at a time and take outputs that start on any 4 bytes; the tensor-memory kernels do not
@pytest.mark.parametrize("hd,heads,kv,seq", [(64, 14, 2, 401), (64, 4, 4, 512), (128, 4, 4, 201), (128, 4, 2, 1000), (256, 4, 1, 300), (256, 2, 2, 384)])
@pytest.mark.parametrize("shift", [2, 4])       # elements of 2 bytes that the outputs start after a 16-byte boundary
def test_outputs_off_16_bytes(hd, heads, kv, seq, shift):
    from mobilefinetuner_b200 import _lib as L
    from mobilefinetuner_b200 import ops as O
    b = 2
    g = torch.Generator(device="cuda").manual_seed(seq + shift)

    def rnd(n):
        return torch.randn(b, seq, n, hd, device="cuda", generator=g).bfloat16().permute(0, 2, 1, 3)

    def off(n):
        buf = torch.full((b * seq * n * hd + 8,), float("nan"), device="cuda").bfloat16()
        return buf[shift:shift + b * seq * n * hd].view(b, seq, n, hd).permute(0, 2, 1, 3), buf
    q, k, v, d_o = rnd(heads), rnd(kv), rnd(kv), rnd(heads)
    (o, o_buf), (dq, dq_buf), (dk, dk_buf), (dv, dv_buf) = off(heads), off(heads), off(kv), off(kv)
    lse, delta = torch.empty(b, heads, seq, device="cuda"), torch.empty(b, heads, seq, device="cuda")
    acc = torch.empty(2 * b * seq * kv * hd, device="cuda")
    scale, st = hd ** -0.5, torch.cuda.current_stream().cuda_stream
    L.init(0)

    def ps(*ts):
        return [x for t in ts for x in (t.data_ptr(), O._strides_bhsd(t))]
    L.call("mft_attn_fwd", *ps(q, k, v, o), lse.data_ptr(), b, seq, heads, kv, hd, scale, 0, st)
    L.call("mft_attn_bwd", *ps(q, k, v, o, d_o), lse.data_ptr(), dq.data_ptr(), dk.data_ptr(), dv.data_ptr(), delta.data_ptr(), acc.data_ptr(),
           b, seq, heads, kv, hd, scale, 0, st)
    ref = _reference(q, k, v, d_o, scale, 0)
    for name, x, r in zip(("o", "lse", "dq", "dk", "dv"), (o, lse, dq, dk, dv), ref):
        assert (x.float() - r).norm() <= 2 ** -7 * r.norm(), name       # as above
    for buf in (o_buf, dq_buf, dk_buf, dv_buf):
        assert bool(buf[:shift].isnan().all()) and bool(buf[buf.numel() - 8 + shift:].isnan().all())


# short calls with grouped heads: dK / dV are added over the heads of a group inside a cluster, in head order.  Group sizes up
# to eight (nine goes another way), one and several 64-key tiles, both sides of the grid limits and of the lengths
@pytest.mark.parametrize("hd,heads,kv,seq,window,batch", [
    (64, 14, 2, 2, 0, 1), (64, 14, 2, 65, 0, 2), (64, 8, 1, 192, 70, 3), (64, 6, 2, 130, 0, 8), (64, 9, 1, 63, 0, 2), (64, 4, 2, 64, 0, 80),
    (128, 8, 2, 100, 0, 1), (128, 6, 2, 128, 33, 2), (128, 8, 1, 64, 0, 16), (256, 4, 1, 40, 0, 2), (256, 4, 1, 64, 20, 30), (256, 8, 1, 33, 0, 1),
    (256, 4, 1, 64, 0, 31), (256, 6, 2, 17, 0, 3)])
def test_short_grouped_backward(hd, heads, kv, seq, window, batch):
    from mobilefinetuner_b200 import ops as O
    g = torch.Generator(device="cuda").manual_seed(seq + batch)

    def rnd(n):
        return torch.randn(batch, seq, n, hd, device="cuda", generator=g).bfloat16().permute(0, 2, 1, 3)
    q, k, v, d_o = rnd(heads), rnd(kv), rnd(kv), rnd(heads)
    scale = hd ** -0.5
    o, lse = O.attention_fwd(q, k, v, scale, window)
    got = O.attention_bwd(q, k, v, o, d_o, lse, scale, window)
    ref = _reference(q, k, v, d_o, scale, window)
    for name, a, b in zip(("dq", "dk", "dv"), got, ref[2:]):
        assert (a.float() - b).norm() <= 2 ** -7 * b.norm(), name       # as above
    tiles = (seq + 63) // 64 * heads * batch
    if heads // kv <= 8 and tiles <= (296 if hd == 64 else 120):        # by clusters (148 SMs): the same bits every time
        for _ in range(10):
            again = O.attention_bwd(q, k, v, o, d_o, lse, scale, window)
            assert all(torch.equal(a, b) for a, b in zip(got, again))
