"""Forwards of up to 128 keys, which run as one launch, against float64: lengths around the tile's and the MMAs' steps, padded heads,
windows, several sequences, inputs far from one.  Tolerance in the 2-norm: operands of 22 bits (1.2e-7 of a value each) and an f32
accumulator truncated at each of at most 24 additions (half of 2^-23 each) give S and O 1.2e-6 of their size; a score's error is its
probability's, and scores of N(0, 1) inputs are of size one: 3e-6 in all.  An error of 1.2e-6 in a score is one of the log-sum-exp."""
import pytest
import torch

from test_gpu_backward64 import gradients

pytestmark = pytest.mark.gpu


def forward64(q, k, v, H, G, D, off):
    B, T, _ = q.shape
    n = off + T
    qq = q.double().view(B, T, H, D).transpose(1, 2)
    kk, vv = (x.double()[:, :n].view(B, n, G, D).transpose(1, 2).repeat_interleave(H // G, 1) for x in (k, v))
    s = (qq @ kk.transpose(-1, -2) / D ** 0.5).masked_fill(torch.ones(T, n, device=q.device).triu(1 + off).bool(), float("-inf"))
    return (s.softmax(-1) @ vv).transpose(1, 2).reshape(B, T, H * D), s.logsumexp(-1).transpose(1, 2)


@pytest.mark.parametrize("B,T,H,G,D,scale", [
    (1, 33, 4, 2, 32, (1, 1, 1)), (1, 48, 2, 1, 64, (1, 1, 1)), (3, 63, 6, 2, 36, (1, 1, 1)), (1, 77, 32, 8, 128, (1, 1, 1)),
    (2, 64, 8, 8, 68, (1, 1, 1)), (1, 65, 12, 4, 80, (1, 1, 1)), (9, 96, 32, 8, 96, (1, 1, 1)), (1, 127, 4, 4, 128, (1, 1, 1)),
    (2, 128, 8, 2, 40, (1, 1, 1)), (1, 128, 16, 4, 112, (1, 1, 1)), (5, 113, 3, 1, 124, (1, 1, 1)),
    (1, 90, 4, 2, 128, (1e-15, 1e15, 1e12)), (1, 90, 4, 2, 64, (1e10, 1e-10, 1e-20)),
])
def test_against_float64(zt, B, T, H, G, D, scale):
    gen = torch.Generator(device="cuda")
    gen.manual_seed(11)
    q, k, v = (torch.randn((B, T, w * D), device="cuda", generator=gen) * c for w, c in zip((H, G, G), scale))
    n0 = zt.lib.launch_count()
    out, lse = zt.attention_forward(q, k, v, H, G, D, want_lse=True)
    assert zt.lib.launch_count() - n0 == 1
    torch.cuda.synchronize()
    assert zt.lib.tc_status() == 0
    ref, ref_lse = forward64(q, k, v, H, G, D, 0)
    assert float((out.double() - ref).norm()) <= 3e-6 * float(ref.norm())
    assert float((lse.double().view_as(ref_lse) - ref_lse).abs().max()) <= 1e-5
    assert torch.equal(out, zt.attention_forward(q, k, v, H, G, D))


@pytest.mark.parametrize("t,off,D", [(1, 40, 64), (16, 17, 128), (50, 78, 80), (20, 100, 32)])
def test_windows_of_short_prompts(zt, t, off, D):
    H, G = 8, 2
    attn = zt.Attn(200, H, G, D)
    gen = torch.Generator(device="cuda")
    gen.manual_seed(5)
    for x in (attn.q, attn.k, attn.v):
        x.normal_(generator=gen)
    attn.forward_at(1, 64, off, off + t, t)
    torch.cuda.synchronize()
    q, k, v = attn.q[: t * H * D].view(1, t, H * D), attn.k[: (off + t) * G * D].view(1, -1, G * D), attn.v[: (off + t) * G * D].view(1, -1, G * D)
    ref = forward64(q, k, v, H, G, D, off)[0]
    assert float((attn.out[: t * H * D].double().view_as(ref) - ref).norm()) <= 3e-6 * float(ref.norm())


def test_values_that_are_not_finite_stay_in_their_rows(zt):
    H, G, D, T = 2, 1, 64, 70
    q, k, v = (torch.randn(1, T, w * D, device="cuda") for w in (H, G, G))
    q[0, 40, 3] = float("nan")
    out = zt.attention_forward(q, k, v, H, G, D).view(T, H, D)
    assert torch.isnan(out[40, 0]).all() and not torch.isnan(out[:40]).any() and not torch.isnan(out[41:]).any()
    assert not torch.isnan(out[40, 1]).any()


@pytest.mark.parametrize("T", [100, 128])
@pytest.mark.parametrize("D", [32, 64, 96, 128])
def test_a_backward_finds_the_short_forwards_scores(zt, T, D):
    """Scores that rise with the key, where the softmax is saturated and dP - delta cancels: dq after the short forward against dq
    after the planes' forward (`keep`), each against float64.  Both forwards add S's terms in the backward's order, and what they
    differ in otherwise (the planes' scales, the order of P.V's terms) was seen to move dq's error by 4 % at most; with the small
    terms of S first it was 1.38 to 2.5 times the other."""
    H, G = 8, 2
    short = planes = 0.0
    for seed in range(3):
        gen = torch.Generator(device="cuda")
        gen.manual_seed(seed)
        q, k, v, do = (torch.randn((1, T, w * D), device="cuda", generator=gen) for w in (H, G, G, H))
        q += 1.0
        k += (torch.arange(T, device="cuda") * (12.0 / (64.0 * D ** 0.5 * 1.4427)))[None, :, None]
        ref = gradients(q, k, v, do, H, G, D)[0]
        ws = zt.BackwardWorkspace(1, T, H, G, D)
        n0 = zt.lib.launch_count()
        out, lse = zt.attention_forward(q, k, v, H, G, D, want_lse=True)
        assert zt.lib.launch_count() - n0 == 1
        dq = zt.attention_backward(q, k, v, out, lse, do, H, G, D, workspace=ws)[0]
        short = max(short, float((dq.double() - ref).norm() / ref.norm()))
        out, lse = zt.attention_forward(q, k, v, H, G, D, want_lse=True, keep=ws)
        dq = zt.attention_backward(q, k, v, out, lse, do, H, G, D, workspace=ws, kept=True)[0]
        planes = max(planes, float((dq.double() - ref).norm() / ref.norm()))
    assert short <= 1.15 * planes, (short, planes)
