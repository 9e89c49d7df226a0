"""The backward of heads of up to 64 columns, whose steps are 128 query rows, against float64: lengths around its tiles and
flushes, split and whole walks, padded heads, and inputs far from one.  Tolerance in the 2-norm: operands are split into two f16
pieces (22 bits, 2^-23 = 1.2e-7 of a value each; three operands and two roundings on the way to a gradient: 6e-7), and the
tensor core truncates its f32 accumulator at each of n additions, half of 2^-23 on average and always toward zero, of a sum that is
two thirds of its final size on average: n 4e-8.  n is 24 for dq; for dk and dv 24 a step, over the steps between two
flushes, which are the heads of the group times at most four tiles of 128 rows."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def gradients(q, k, v, do, H, G, D):
    B, T, _ = q.shape
    heads = lambda x, n: x.double().view(B, T, n, D).transpose(1, 2)
    qq, g = heads(q, H), heads(do, H)
    kk, vv = (heads(x, G).repeat_interleave(H // G, 1) for x in (k, v))
    s = (qq @ kk.transpose(-1, -2) / D ** 0.5).masked_fill(torch.ones(T, T, device=q.device).triu(1).bool(), float("-inf"))
    p = s.softmax(-1)
    dp = g @ vv.transpose(-1, -2)
    ds = p * (dp - (dp * p).sum(-1, keepdim=True))
    flat = lambda x, n: x.transpose(1, 2).reshape(B, T, n * D)
    group = lambda x: flat(x.reshape(B, G, H // G, T, D).sum(2), G)
    return flat(ds @ kk / D ** 0.5, H), group(ds.transpose(-1, -2) @ qq / D ** 0.5), group(p.transpose(-1, -2) @ g)


@pytest.mark.parametrize("B,T,H,G,D,scale", [
    (1, 127, 2, 1, 64, (1, 1, 1, 1)), (1, 128, 4, 2, 64, (1, 1, 1, 1)), (2, 129, 4, 4, 32, (1, 1, 1, 1)), (1, 256, 4, 2, 32, (1, 1, 1, 1)),
    (1, 257, 6, 2, 36, (1, 1, 1, 1)), (4, 1000, 16, 4, 64, (1, 1, 1, 1)),  # (split by heads)
    (1, 900, 3, 3, 60, (1, 1, 1, 1)), (1, 1300, 2, 2, 48, (1, 1, 1, 1)),   # (by ranges of query tiles, past a flush inside the walk)
    (8, 700, 32, 8, 64, (1, 1, 1, 1)), (20, 640, 8, 8, 32, (1, 1, 1, 1)),  # (whole walks, tile by tile and sequence by sequence)
    (1, 333, 4, 2, 64, (1e-15, 1e-15, 1, 1)), (1, 333, 4, 2, 64, (1, 1, 1e15, 1e15)), (1, 333, 4, 2, 40, (1, 1, 1e-12, 1e-12)),
])
def test_gradients_against_float64(zt, B, T, H, G, D, scale):
    gen = torch.Generator(device="cuda")
    gen.manual_seed(7)
    q, k, v, do = (torch.randn((B, T, w * D), device="cuda", generator=gen) * c for w, c in zip((H, G, G, H), scale))
    ws = zt.BackwardWorkspace(B, T, H, G, D)
    out, lse = zt.attention_forward(q, k, v, H, G, D, want_lse=True, keep=ws)
    got = zt.attention_backward(q, k, v, out, lse, do, H, G, D, workspace=ws, kept=True)
    torch.cuda.synchronize()
    assert zt.lib.tc_status() == 0 and zt.lib.tc_saturated() == 0
    for name, x, ref in zip(("dq", "dk", "dv"), got, gradients(q, k, v, do, H, G, D)):
        # (norms of float64 values, so that no square leaves their range)
        n = 24 if name == "dq" else 24 * (H // G) * min(4, max(1, (T + 127) // 128 - 1))
        assert float((x.double() - ref).norm()) <= (6e-7 + 4e-8 * n) * float(ref.norm()), name
    again = zt.attention_backward(q, k, v, out, lse, do, H, G, D, workspace=ws)
    assert torch.equal(got[1], again[1]) and torch.equal(got[2], again[2])  # (sums of dk and dv are made in the order of the walk)


@pytest.mark.parametrize("B,T,H,G,D", [
    (1, 33, 4, 2, 32), (2, 48, 8, 2, 64), (3, 63, 3, 3, 36), (5, 64, 16, 16, 60), (1, 64, 32, 4, 64),  # (the last one: split by heads)
    (64, 37, 32, 4, 32), (40, 64, 16, 4, 40), (1, 65, 8, 2, 64),  # (tile by tile; sequence by sequence; the first of steps of 128)
])
def test_steps_of_64_rows(zt, B, T, H, G, D):
    test_gradients_against_float64(zt, B, T, H, G, D, (1, 1, 1, 1))
