"""The forwards that split the query rows themselves, against float64: one head a block, two, wide heads, walks split along the keys and
windows whose sums leave the accumulators; rows far smaller than their neighbours, whole tensors far from one; and the backward
that reads q after the forward, its gradient written over it.  Tolerance in the 2-norm: operands of 22 bits and at most 48 truncated
additions (half of 2^-23 each) give S 3e-6 of its size at 256 columns, half of that at 128; O is truncated 12 times a key tile at
two thirds of its final size on average, 4e-8 each."""
import pytest
import torch

from test_gpu_backward64 import gradients
from test_gpu_forward_short import forward64

pytestmark = pytest.mark.gpu


def inputs(B, T, H, G, D, scale, spread):
    gen = torch.Generator(device="cuda")
    gen.manual_seed(29)
    q, k, v, do = (torch.randn((B, T, w * D), device="cuda", generator=gen) * c for w, c in zip((H, G, G, H), (*scale, 1.0)))
    if spread:  # every row by a power of two of its own, the largest 1
        q *= 2.0 ** -torch.randint(0, spread, (B, T, 1), device="cuda", generator=gen).float()
    return q, k, v, do


def bound(D, keys):
    return (1.5e-6 if D <= 128 else 3e-6) + 12 * -(-keys // 64) * 4e-8


@pytest.mark.parametrize("B,T,H,G,D,scale,spread", [
    (1, 129, 4, 2, 32, (1, 1, 1), 30), (3, 200, 3, 3, 60, (1, 1, 1), 0), (2, 161, 6, 2, 80, (1, 1, 1), 30),   # one head a block
    (1, 1100, 2, 1, 128, (1, 1, 1), 0),                                                                      # split along the keys
    (20, 200, 8, 2, 64, (1, 1, 1), 30), (30, 130, 12, 2, 100, (1, 1, 1), 0), (13, 257, 8, 2, 128, (1, 1, 1), 30),  # two heads a block
    (2, 131, 3, 1, 160, (1, 1, 1), 30), (1, 300, 4, 2, 192, (1, 1, 1), 0), (2, 129, 2, 2, 256, (1, 1, 1), 30),     # wide heads
    (1, 200, 4, 2, 128, (1e-25, 1e25, 1), 30), (20, 200, 8, 2, 64, (1e20, 1e-20, 1e-20), 0), (1, 200, 2, 1, 256, (1e-30, 1, 1), 0),
])
def test_against_float64(zt, B, T, H, G, D, scale, spread):
    q, k, v, do = inputs(B, T, H, G, D, scale, spread)
    ws = zt.BackwardWorkspace(B, T, H, G, D)
    out, lse = zt.attention_forward(q, k, v, H, G, D, want_lse=True, keep=ws)
    torch.cuda.synchronize()
    assert zt.lib.tc_status() == 0 and zt.lib.last_path() == "tcgen05"
    ref, ref_lse = forward64(q, k, v, H, G, D, 0)
    assert float((out.double() - ref).norm()) <= bound(D, T) * float(ref.norm())
    assert float((lse.double().view_as(ref_lse) - ref_lse).abs().max()) <= 2e-5
    if scale != (1, 1, 1):
        return
    got = zt.attention_backward(q, k, v, out, lse, do, H, G, D, workspace=ws, kept=True)
    torch.cuda.synchronize()
    assert zt.lib.tc_status() == 0 and zt.lib.tc_saturated() == 0
    for name, x, r in zip(("dq", "dk", "dv"), got, gradients(q, k, v, do, H, G, D)):
        assert float((x.double() - r).norm()) <= 1e-5 * float(r.norm()), name  # (what the calls are measured to)


@pytest.mark.parametrize("t,off,H,G,D", [
    (130, 1200, 3, 3, 64), (200, 2100, 8, 2, 128), (40, 1500, 2, 1, 256), (600, 1400, 32, 8, 64),
    # as many tiles as no accumulator is flushed after, and one more: one head a block, two, wide heads; narrow ones; rows that are not a warp's
    (519, 1529, 32, 32, 128), (519, 1530, 32, 32, 100), (1223, 313, 16, 16, 36), (1001, 1100, 16, 16, 60), (1025, 999, 32, 8, 100), (603, 421, 32, 32, 192),
    (603, 422, 32, 32, 164),
])
def test_windows(zt, t, off, H, G, D):
    attn = zt.Attn(off + t, H, G, D)
    gen = torch.Generator(device="cuda")
    gen.manual_seed(3)
    for x in (attn.q, attn.k, attn.v):
        x.normal_(generator=gen)
    attn.forward_at(1, 64, off, off + t, t)
    torch.cuda.synchronize()
    assert zt.lib.tc_status() == 0
    q, k, v = attn.q[: t * H * D].view(1, t, H * D), attn.k.view(1, -1, G * D), attn.v.view(1, -1, G * D)
    ref = forward64(q, k, v, H, G, D, off)[0]
    assert float((attn.out[: t * H * D].double().view_as(ref) - ref).norm()) <= bound(D, 1024) * float(ref.norm())  # (flushed every 16 tiles)


@pytest.mark.parametrize("B,T,H,G,D", [(2, 200, 4, 2, 64), (1, 300, 8, 2, 128), (1, 1100, 2, 1, 256)])
def test_gradient_of_q_over_q(zt, B, T, H, G, D):
    q, k, v, do = inputs(B, T, H, G, D, (1, 1, 1), 0)
    ws = zt.BackwardWorkspace(B, T, H, G, D)
    out, lse = zt.attention_forward(q, k, v, H, G, D, want_lse=True, keep=ws)
    token = ws.token
    want = zt.attention_backward(q, k, v, out, lse, do, H, G, D, workspace=ws, kept=True)
    zt.attention_forward(q, k, v, H, G, D, want_lse=True, keep=ws)
    assert ws.token > token
    dk, dv, delta = torch.empty_like(k), torch.empty_like(v), torch.empty_like(lse)
    assert zt.lib.load().zt_attn_backward_batched_kept(
        *(x.data_ptr() for x in (q, k, v, out, lse, do, q, dk, dv, delta, ws.buf)), ws.nbytes, B, T, H, G, D,
        torch.cuda.current_stream().cuda_stream, ws.token) == 0, zt.lib.last_error()
    torch.cuda.synchronize()
    for a, b in zip((q, dk, dv), want):  # (sums that are made in memory come in no fixed order)
        assert float((a.double() - b.double()).norm()) <= 1e-6 * float(b.double().norm())


def rotated(x, heads, D, pos, theta):
    """x in float64 with its heads rotated as src/rope.zig does."""
    B, T, _ = x.shape
    i = torch.arange(D // 2, dtype=torch.float64, device=x.device)
    angle = (pos + torch.arange(T, dtype=torch.float64, device=x.device))[:, None] / theta ** (2 * i / D)
    c, s = angle.cos()[None, :, None], angle.sin()[None, :, None]
    lo, hi = x.double().view(B, T, heads, 2, D // 2).unbind(3)
    return torch.stack((lo * c - hi * s, hi * c + lo * s), 3).reshape(B, T, heads * D)


@pytest.mark.parametrize("B,T,H,G,D", [
    (1, 200, 4, 2, 64), (1, 140, 6, 2, 80), (12, 300, 8, 2, 64), (40, 130, 3, 1, 40),  # one head a block; two blocks an SM
    (14, 257, 8, 2, 128), (20, 130, 8, 4, 96), (1, 150, 4, 2, 256), (1, 300, 2, 1, 160),  # two heads; wide heads
])
def test_rotated_rows_and_the_planes_of_out(zt, B, T, H, G, D):
    q, k, v, _ = inputs(B, T, H, G, D, (1, 1, 1), 0)
    out, lse = zt.attention_forward_rope(q, k, v, H, G, D, pos=5, want_lse=True)
    torch.cuda.synchronize()
    assert zt.lib.tc_status() == 0
    theta = zt.ops.ROPE_THETA
    ref, ref_lse = forward64(rotated(q, H, D, 5, theta), rotated(k, G, D, 5, theta), v.double(), H, G, D, 0)
    assert float((out.double() - ref).norm()) <= (bound(D, T) + 1e-6) * float(ref.norm())  # (a rotation is an f32 product sum)
    assert float((lse.double().view_as(ref_lse) - ref_lse).abs().max()) <= 2e-5
    if H * D % 64:
        return
    wo = torch.randn(H * D, 64, device="cuda") / (H * D) ** 0.5
    block = zt.AttentionBlock(B, T, H, G, D, 64)
    y, y2 = (block.forward(q, k, v, wo, fused=f) for f in (True, False))
    assert float((y - y2).abs().max()) <= 1e-6 * float(y2.abs().max())


@pytest.mark.parametrize("B,T,H,G,D,kernel", [
    # more than a block an SM and fewer than two: by the length; from two on whatever it is
    (1, 1536, 16, 16, 64, "attn_fwd_tc16n"), (1, 1537, 16, 16, 64, "attn_fwd_tc16"), (1, 3001, 8, 2, 40, "attn_fwd_tc16"), (3, 1537, 8, 4, 64, "attn_fwd_tc16n"),
])
def test_long_sequences_in_few_blocks(zt, B, T, H, G, D, kernel):
    q, k, v, _ = inputs(B, T, H, G, D, (1, 1, 1), 0)
    zt.lib.profile(True)
    zt.lib.profile_read()
    out, lse = zt.attention_forward(q, k, v, H, G, D, want_lse=True)
    torch.cuda.synchronize()
    names = {x for x in zt.lib.profile_read() if x.startswith("attn_")}
    zt.lib.profile(False)
    assert names == {kernel} and zt.lib.tc_status() == 0
    ref, ref_lse = forward64(q, k, v, H, G, D, 0)
    assert float((out.double() - ref).norm()) <= bound(D, T) * float(ref.norm())
    assert float((lse.double().view_as(ref_lse) - ref_lse).abs().max()) <= 2e-5


@pytest.mark.parametrize("B,T,H,G,D", [
    (1, 200, 4, 2, 128), (1, 140, 6, 2, 80), (1, 1100, 2, 1, 128),  # one head a block, split along the keys
    (20, 200, 8, 2, 64), (24, 130, 12, 4, 40),                      # two blocks an SM
    (13, 257, 8, 2, 128), (2, 131, 3, 1, 160), (1, 300, 2, 2, 256),  # two heads, wide heads
])
def test_rows_that_are_not_numbers(zt, B, T, H, G, D):
    """A NaN or an infinity in one query row of one head makes that row's output NaN and changes no bit of any other: a row's scale is its own.
    A NaN in a key's row reaches the queries that see the key, in its group's heads, and none before them."""
    q, k, v, _ = inputs(B, T, H, G, D, (1, 1, 1), 0)
    out, lse = zt.attention_forward(q, k, v, H, G, D, want_lse=True)
    spoilt = q.clone()
    spoilt[0, 70, 3] = float("nan")
    spoilt[B - 1, T - 2, H * D - 1] = float("inf")
    got, got_lse = zt.attention_forward(spoilt, k, v, H, G, D, want_lse=True)
    torch.cuda.synchronize()
    assert zt.lib.tc_status() == 0
    hit = torch.zeros(B, T, H, dtype=torch.bool, device="cuda")
    hit[0, 70, 0] = hit[B - 1, T - 2, H - 1] = True
    rows, rows0 = got.view(B, T, H, D), out.view(B, T, H, D)
    assert rows[hit].isnan().all() and torch.equal(rows[~hit], rows0[~hit])
    assert torch.equal(got_lse.view(B, T, H)[~hit], lse.view(B, T, H)[~hit])
    spoilt = k.clone()
    spoilt[B - 1, 90, G * D - 2] = float("nan")
    got = zt.attention_forward(q, spoilt, v, H, G, D).view(B, T, H, D)
    torch.cuda.synchronize()
    assert zt.lib.tc_status() == 0
    hit.zero_()
    hit[B - 1, 90:, H - H // G:] = True
    assert got[hit].isnan().all() and torch.equal(got[~hit], rows0[~hit])
