"""The one-launch pre-pass of small forwards at the sizes where its two forms begin and end (units of a sequence's group of heads:
rows times heads): outputs against float64, and gradients from the planes it leaves.  Tolerances are those of the short forward's and
the backwards' tests.  Where pass_one_kernel ends, a form of pass_planes_kernel goes on that holds the rows in clusters of blocks, still
in one launch; where that ends, pass_stats_kernel goes before pass_planes_kernel."""
import pytest
import torch

from test_gpu_backward64 import gradients
from test_gpu_forward_short import forward64
from test_gpu_query_rows import bound

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("B,T,H,G,D,one", [
    (3, 64, 8, 2, 32, True), (1, 65, 8, 2, 32, True), (1, 256, 4, 1, 32, True), (1, 257, 4, 1, 32, False),     # 256 and 1024 units
    (2, 128, 3, 3, 64, True), (1, 129, 3, 3, 64, True), (1, 170, 6, 2, 60, True), (1, 171, 6, 2, 64, False),   # 128 and 512
    (1, 64, 2, 2, 96, True), (5, 106, 3, 1, 80, True), (1, 107, 3, 1, 80, False),                              # 64 and 320
    (1, 64, 4, 1, 128, True), (1, 65, 4, 1, 128, False), (7, 53, 3, 1, 192, True), (1, 54, 3, 1, 160, False),  # 64, 256; 32, 160
    (2, 128, 2, 2, 256, True), (1, 129, 2, 2, 200, False),                                                     # 32, 128
])
def test_planes_of_small_forwards(zt, B, T, H, G, D, one):
    gen = torch.Generator(device="cuda")
    gen.manual_seed(17)
    q, k, v, do = (torch.randn((B, T, w * D), device="cuda", generator=gen) * c for w, c in zip((H, G, G, H), (1, 1, 1e3, 1e-3)))
    ws = zt.BackwardWorkspace(B, T, H, G, D)
    zt.lib.profile(True)
    zt.lib.profile_read()
    out, lse = zt.attention_forward(q, k, v, H, G, D, want_lse=True, keep=ws)
    launched = zt.lib.profile_read()
    zt.lib.profile(False)
    assert ("pass_one_kernel" in launched) == one and ("pass_planes_kernel" in launched) != one
    got = zt.attention_backward(q, k, v, out, lse, do, H, G, D, workspace=ws, kept=ws.token != 0)
    torch.cuda.synchronize()
    assert zt.lib.tc_status() == 0 and zt.lib.tc_saturated() == 0
    ref, ref_lse = forward64(q, k, v, H, G, D, 0)
    assert float((out.double() - ref).norm()) <= 3e-6 * float(ref.norm())
    assert float((lse.double().view_as(ref_lse) - ref_lse).abs().max()) <= 1e-5
    for name, x, r in zip(("dq", "dk", "dv"), got, gradients(q, k, v, do, H, G, D)):
        assert float((x.double() - r).norm()) <= (6e-7 + 4e-8 * 240) * float(r.norm()), name


@pytest.mark.parametrize("B,T,H,G,D,one", [
    (36, 64, 16, 4, 64, True), (64, 64, 16, 4, 64, False),     # a quarter of the room in use, groups of four: five waves of blocks
    (64, 78, 16, 4, 64, True), (128, 78, 16, 4, 64, False),    # 0.305: 7.4
    (9, 33, 32, 4, 32, True), (24, 33, 32, 4, 32, False),      # 0.107, groups of eight: 0.9
    (64, 130, 16, 16, 64, True), (128, 130, 16, 16, 64, False),  # 0.254, no groups: 29
    (128, 103, 16, 4, 64, True), (64, 60, 16, 16, 128, True),  # two fifths: any number; the form of 4 float4
])
def test_planes_of_small_forwards_in_many_blocks(zt, B, T, H, G, D, one):
    test_planes_of_small_forwards(zt, B, T, H, G, D, one)


ONE, HELD, TWO = {"pass_one_kernel"}, {"pass_planes_kernel"}, {"pass_stats_kernel", "pass_planes_kernel"}


@pytest.mark.parametrize("B,T,H,G,D,launched", [
    (1, 256, 4, 1, 32, ONE), (1, 257, 4, 1, 32, HELD), (1, 170, 6, 2, 60, ONE), (1, 171, 6, 2, 64, HELD), (1, 107, 3, 1, 80, HELD),
    (1, 65, 4, 1, 128, HELD), (1, 54, 3, 1, 160, HELD), (64, 64, 16, 4, 64, HELD), (24, 33, 32, 4, 32, HELD),
    # the clusters' sizes: eight blocks of 4 float4 a thread, three of 16, eight of these, and more
    (1, 256, 1, 1, 256, HELD), (1, 257, 1, 1, 256, HELD), (1, 1024, 1, 1, 256, HELD), (1, 1025, 1, 1, 256, TWO),
    (2, 1280, 1, 1, 160, HELD), (2, 1281, 1, 1, 160, TWO), (1, 2049, 1, 1, 128, TWO),
    # and their slots, 2048 a tensor
    (128, 129, 32, 8, 64, HELD), (150, 140, 16, 16, 64, TWO),
    # single blocks of 16 float4 a thread, where those of 4 have no slots: full enough or not
    (65, 100, 16, 8, 256, HELD), (130, 45, 24, 8, 256, TWO), (128, 130, 16, 16, 64, TWO),
])
def test_the_launches_of_a_forwards_pre_pass(zt, B, T, H, G, D, launched):
    gen = torch.Generator(device="cuda")
    gen.manual_seed(B + T)
    q, k, v, do = (torch.randn((B, T, w * D), device="cuda", generator=gen) * c for w, c in zip((H, G, G, H), (1, 1, 1e3, 1e-3)))
    ws = zt.BackwardWorkspace(B, T, H, G, D)
    zt.lib.profile(True)
    zt.lib.profile_read()
    out, lse = zt.attention_forward(q, k, v, H, G, D, want_lse=True, keep=ws)
    names = {x for x in zt.lib.profile_read() if x.startswith("pass_")}
    zt.lib.profile(False)
    assert names == launched
    got = zt.attention_backward(q, k, v, out, lse, do, H, G, D, workspace=ws, kept=ws.token != 0)
    torch.cuda.synchronize()
    assert zt.lib.tc_status() == 0 and zt.lib.tc_saturated() == 0
    ref, ref_lse = forward64(q, k, v, H, G, D, 0)
    assert float((out.double() - ref).norm()) <= bound(D, T) * float(ref.norm())
    assert float((lse.double().view_as(ref_lse) - ref_lse).abs().max()) <= 2e-5
    for name, x, r in zip(("dq", "dk", "dv"), got, gradients(q, k, v, do, H, G, D)):
        assert float((x.double() - r).norm()) <= 1e-5 * float(r.norm()), name


@pytest.mark.parametrize("B,T,k,n,launched", [
    (1, 128, 128, 128, ONE), (1, 600, 64, 576, HELD), (3, 600, 64, 576, HELD), (1, 4096, 64, 4096, HELD),
    # two tensors that need different numbers of blocks: in the form of 4 float4 a thread, and in that of 16 too
    (1, 641, 64, 576, HELD), (1, 1300, 128, 1088, TWO), (12, 300, 512, 64, TWO),
])
def test_a_projections_pre_pass(zt, B, T, k, n, launched):
    gen = torch.Generator(device="cuda")
    gen.manual_seed(B + T)
    ctx, w = torch.randn((B, T, k), device="cuda", generator=gen) * 1e2, torch.randn((k, n), device="cuda", generator=gen) * 1e-2
    zt.lib.profile(True)
    zt.lib.profile_read()
    y = zt.proj_forward(ctx, w)
    torch.cuda.synchronize()
    names = {x for x in zt.lib.profile_read() if x.startswith("pass_")}
    zt.lib.profile(False)
    assert names == launched and zt.lib.tc_status() == 0
    ref = ctx.double() @ w.double()
    # two operands of 22 bits, and three truncated additions (half of 2^-23 on average) for every 16 of the contraction
    assert float((y.double() - ref).norm()) <= (2 * 2.0 ** -22 + 3 * (k // 16) * 2.0 ** -24) * float(ref.norm())


def test_clusters_in_a_captured_graph(zt):
    """A step whose pre-passes are clusters, forward and backward, and a projection's, recorded once and replayed on other inputs."""
    B, T, H, G, D = 2, 200, 6, 2, 64
    gen = torch.Generator(device="cuda")
    gen.manual_seed(3)
    q, k, v, do = (torch.randn((B, T, w * D), device="cuda", generator=gen) for w in (H, G, G, H))
    ctx, w = torch.randn((1, 600, 64), device="cuda", generator=gen), torch.randn((64, 576), device="cuda", generator=gen)
    ws, pws = zt.BackwardWorkspace(B, T, H, G, D), zt.ProjWorkspace(1, 600, 64, 576)

    def step():
        out, lse = zt.attention_forward(q, k, v, H, G, D, want_lse=True, keep=ws)
        return (out, lse, *zt.attention_backward(q, k, v, out, lse, do, H, G, D, workspace=ws, kept=True), zt.proj_forward(ctx, w, workspace=pws))

    zt.lib.profile(True)
    zt.lib.profile_read()
    step()
    names = {x for x in zt.lib.profile_read() if x.startswith("pass_")}
    zt.lib.profile(False)
    assert names == {"pass_planes_kernel", "pass_backward_kernel"}
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        captured = step()
    for _ in range(2):
        for x in (q, k, v, do, ctx, w):
            x.normal_(generator=gen)
        graph.replay()
        got = [x.clone() for x in captured]
        torch.cuda.synchronize()
        assert zt.lib.tc_status() == 0 and zt.lib.tc_saturated() == 0
        for a, b in zip(got, step()):  # (sums that are made in memory come in no fixed order)
            assert float((a.double() - b.double()).norm()) <= 1e-6 * float(b.double().norm())
