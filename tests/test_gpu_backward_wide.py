"""The backward of heads above 128 columns against float64, where a tile of a product is one unit (up to 1024 keys; dQ is stored) and
where it is several (added to a zeroed dq): lengths around the tiles and that line, odd numbers of heads, padded heads.  Tolerance in
the 2-norm, as in the 64-column backward's test: 6e-7 for the operands, 4e-8 for each addition to a truncating accumulator: at most 48
of a score's contraction and 192 of a product's piece."""
import pytest
import torch

from test_gpu_backward64 import gradients

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("B,T,H,G,D", [
    (1, 64, 2, 1, 256), (1, 128, 4, 4, 192), (3, 129, 3, 1, 160), (2, 700, 6, 2, 132), (1, 1000, 4, 1, 256), (5, 1024, 3, 3, 256),
    (1, 1025, 4, 2, 192), (2, 1300, 3, 1, 256),
])
def test_gradients_against_float64(zt, B, T, H, G, D):
    gen = torch.Generator(device="cuda")
    gen.manual_seed(13)
    q, k, v, do = (torch.randn((B, T, w * D), device="cuda", generator=gen) for w in (H, G, G, H))
    ws = zt.BackwardWorkspace(B, T, H, G, D)
    out, lse = zt.attention_forward(q, k, v, H, G, D, want_lse=True, keep=ws)
    got = zt.attention_backward(q, k, v, out, lse, do, H, G, D, workspace=ws, kept=ws.token != 0)
    torch.cuda.synchronize()
    assert zt.lib.last_path() == "tcgen05" and zt.lib.tc_status() == 0 and zt.lib.tc_saturated() == 0
    for name, x, ref in zip(("dq", "dk", "dv"), got, gradients(q, k, v, do, H, G, D)):
        assert float((x.double() - ref).norm()) <= (6e-7 + 4e-8 * 240) * float(ref.norm()), name


@pytest.mark.parametrize("B,T,H,G,D", [(23, 100, 4, 2, 160), (23, 256, 2, 1, 256), (15, 380, 3, 1, 192), (12, 1024, 4, 2, 132)])
def test_units_of_the_products_in_turn(zt, B, T, H, G, D):
    """Enough heads for a head's units of the three products to go in turn (45 of them on 148 SMs at these lengths, 89 of up to 128 rows)."""
    test_gradients_against_float64(zt, B, T, H, G, D)


@pytest.mark.parametrize("T,D,kept", [(130, 256, True), (130, 160, False), (1100, 192, True)])
def test_query_rows_of_small_gradients_keep_their_scores(zt, T, D, kept):
    """Rows whose dout, and whose q, are 2^-11 of their neighbours': dK wants q's rows scaled down with dout's, under which the low pieces of
    such a row leave f16's range; the scores are made of the planes as they are.  dq of these rows, relative to them: q's 22 bits at
    2^-11 of the maximum leave S (some 4 here) 2^-22 and the three products' additions 1e-6 of its size."""
    gen = torch.Generator(device="cuda")
    gen.manual_seed(5)
    q, k, v, do = (torch.randn((1, T, w * D), device="cuda", generator=gen) for w in (4, 2, 2, 4))
    small = torch.arange(T, device="cuda") % 3 == 1
    q[:, small] *= 2.0 ** -11
    do[:, small] *= 2.0 ** -12
    k *= 2.0 ** 13
    ws = zt.BackwardWorkspace(1, T, 4, 2, D)
    out, lse = zt.attention_forward(q, k, v, 4, 2, D, want_lse=True, keep=ws)
    dq = zt.attention_backward(q, k, v, out, lse, do, 4, 2, D, workspace=ws, kept=kept)[0]
    torch.cuda.synchronize()
    assert zt.lib.tc_status() == 0 and zt.lib.tc_saturated() == 0
    ref = gradients(q, k, v, do, 4, 2, D)[0][:, small]
    assert float((dq[:, small].double() - ref).norm()) <= 1e-5 * float(ref.norm())
