"""The backward's pre-pass in one launch, at the ends of what it takes: units (rows times heads of a group) around its blocks' and clusters'
sizes, heads narrower than their planes, rows of dout far from one another; and its neighbours that take two launches: more
rows, wider heads, an out on a 4-byte boundary, an out that the gradient of q is written over.  Tolerance: that of the 64-column
backward's tests."""
import pytest
import torch

from test_gpu_backward64 import gradients

pytestmark = pytest.mark.gpu


def step(zt, B, T, H, G, D, out_shift=0, out_is_dq=False):
    gen = torch.Generator(device="cuda")
    gen.manual_seed(B + T)
    q, k, v, do = (torch.randn((B, T, w * D), device="cuda", generator=gen) for w in (H, G, G, H))
    do *= 2.0 ** -torch.randint(0, 8, (B, T, 1), device="cuda", generator=gen).float()
    ws = zt.BackwardWorkspace(B, T, H, G, D)
    out, lse = zt.attention_forward(q, k, v, H, G, D, want_lse=True, keep=ws)
    if out_shift:
        flat = torch.empty(out.numel() + 4, device="cuda")
        flat[out_shift:out_shift + out.numel()] = out.flatten()
        out = flat[out_shift:out_shift + out.numel()].view_as(out)
    dq = out if out_is_dq else torch.full_like(q, float("nan"))
    dk, dv, delta = torch.empty_like(k), torch.empty_like(v), torch.empty_like(lse)
    zt.lib.profile(True)
    zt.lib.profile_read()
    assert zt.lib.load().zt_attn_backward_batched_kept(
        *(x.data_ptr() for x in (q, k, v, out, lse, do, dq, dk, dv, delta, ws.buf)), ws.nbytes, B, T, H, G, D,
        torch.cuda.current_stream().cuda_stream, ws.token) == 0, zt.lib.last_error()
    torch.cuda.synchronize()
    launched = zt.lib.profile_read()
    zt.lib.profile(False)
    assert zt.lib.tc_status() == 0 and zt.lib.tc_saturated() == 0
    n = 24 * (H // G) * min(4, max(1, (T + 127) // 128))
    for name, x, ref in zip(("dq", "dk", "dv"), (dq, dk, dv), gradients(q, k, v, do, H, G, D)):
        assert float((x.double() - ref).norm()) <= (6e-7 + 4e-8 * (24 if name == "dq" else n)) * float(ref.norm()), name
    return "pass_backward_kernel" in launched


@pytest.mark.parametrize("B,T,H,G,D", [
    (1, 40, 1, 1, 32), (1, 64, 4, 4, 32), (1, 65, 4, 4, 36), (2, 33, 6, 2, 60), (1, 256, 4, 2, 32), (3, 200, 3, 1, 64), (64, 100, 8, 2, 64),
    (1, 640, 2, 2, 64), (1, 639, 1, 1, 40), (5, 320, 4, 2, 64), (1, 1280, 1, 1, 32), (40, 160, 8, 2, 48), (130, 35, 2, 2, 64),
])
def test_one_launch(zt, B, T, H, G, D):
    assert step(zt, B, T, H, G, D)


def test_two_launches(zt):
    assert not step(zt, 1, 641, 2, 2, 64) and not step(zt, 1, 1281, 1, 1, 32) and not step(zt, 1, 70, 4, 2, 68)
    assert not step(zt, 130, 257, 8, 8, 64)  # (two blocks for each of 1040 (sequence, group)s: more than dout's slots)
    assert not step(zt, 2, 90, 4, 2, 64, out_shift=1) and not step(zt, 2, 90, 4, 2, 64, out_is_dq=True)
