"""Calls that could do without scratch -- windows of a prompt, sequences under 128 rows, head widths between the tiles' -- take
it in the order of their stream: they may overlap on the GPU and be captured without a word to the library."""
import subprocess
import sys
import threading

import pytest
import torch

pytestmark = pytest.mark.gpu
ROOT = __file__.rsplit("/tests/", 1)[0]


def normal(seed, *shape):
    return torch.randn(shape, generator=torch.Generator(device="cuda").manual_seed(seed), device="cuda")


def window(zt, seed, ctx, t, H, Hkv, D):
    a = zt.Attn(ctx, H, Hkv, D)
    for i, x in enumerate((a.q, a.k, a.v)):
        x.copy_(normal(seed + i, x.numel()))

    def call():
        a.forward_at(1, 64, ctx - t, ctx, t)
        return a.out[: t * H * D]
    return call


def whole(zt, seed, B, T, H, Hkv, D):
    q, k, v = (normal(seed + i, B, T, w * D) for i, w in enumerate((H, Hkv, Hkv)))
    return lambda: zt.attention_forward(q, k, v, H, Hkv, D)


def reference_abi_backward(zt, seed, T, H, Hkv, D):
    a = zt.Attn(T, H, Hkv, D)
    for i, x in enumerate((a.q, a.k, a.v, a.dout)):
        x.copy_(normal(seed + i, x.numel()))

    def call():
        a.backward()
        return a.dk
    return call


def calls(zt, seed):
    return [window(zt, seed, 3000, 64, 8, 2, 128), window(zt, seed + 10, 900, 300, 4, 1, 64), whole(zt, seed + 20, 4, 100, 8, 2, 128),
            whole(zt, seed + 30, 2, 700, 8, 2, 80), whole(zt, seed + 40, 1, 500, 4, 2, 200), reference_abi_backward(zt, seed + 50, 400, 4, 2, 72)]


@pytest.mark.parametrize("threads", [False, True])
def test_calls_on_two_streams_overlap(zt, threads):
    """Each stream's calls give bit for bit what they give alone, whatever the other stream's do meanwhile."""
    sides = [calls(zt, 100), calls(zt, 500)]
    torch.cuda.synchronize()
    want = [[f().clone() for f in side] for side in sides]
    torch.cuda.synchronize()
    streams = [torch.cuda.Stream() for _ in sides]
    got = [[], []]

    def run(i):
        with torch.cuda.stream(streams[i]):
            # the other stream's order, so that unlike calls meet
            for f in (sides[i] if i == 0 else sides[i][::-1]):
                got[i].append(f().clone())

    for _ in range(5):
        if threads:
            ts = [threading.Thread(target=run, args=(i,)) for i in range(2)]
            [t.start() for t in ts]
            [t.join() for t in ts]
        else:
            run(0), run(1)
    torch.cuda.synchronize()
    assert zt.lib.tc_status() == 0
    n = len(want[0])
    for i in range(2):
        order = list(range(n)) if i == 0 else list(range(n))[::-1]
        assert len(got[i]) == 5 * n
        for j, x in enumerate(got[i]):
            assert torch.equal(x, want[i][order[j % n]]), (i, j)


def test_captured_without_reserving_and_replayed_side_by_side(zt):
    """A process of its own, whose arena nothing has grown: each call is captured into a graph without zt_attn_reserve
    (the holders' own reservation aside), and the graphs of both sides replay on two streams at once."""
    code = """
import importlib, sys, torch
sys.path.insert(0, "tests")
zt = importlib.import_module("z-transformer_b200")
import test_gpu_streams as t
q, k, v = (t.normal(i, 2, 300, w * 80) for i, w in enumerate((8, 2, 2)))
L = zt.lib.load()
assert L.zt_attn_arena_bytes() == 0
side = torch.cuda.Stream()
first = torch.cuda.CUDAGraph()
torch.cuda.synchronize()
zt.attention_forward(q[:1, :200].contiguous(), k[:1, :200].contiguous(), v[:1, :200].contiguous(), 8, 2, 80)  # (loads the kernels)
torch.cuda.synchronize()
with torch.cuda.graph(first, stream=side):
    out = zt.attention_forward(q, k, v, 8, 2, 80)
first.replay()
torch.cuda.synchronize()
assert L.zt_attn_arena_bytes() == 0 and zt.lib.last_path() == "tcgen05"
assert torch.equal(out, zt.attention_forward(q, k, v, 8, 2, 80))
sides = [t.calls(zt, 100), t.calls(zt, 500)]
want = [[f().clone() for f in side_] for side_ in sides]
torch.cuda.synchronize()
graphs, outs = [[], []], [[], []]
for i, fs in enumerate(sides):
    for f in fs:
        g = torch.cuda.CUDAGraph()
        with torch.cuda.graph(g, stream=side):
            outs[i].append(f().clone())
        graphs[i].append(g)
streams = [torch.cuda.Stream(), torch.cuda.Stream()]
for _ in range(5):
    for a, b in zip(graphs[0], graphs[1][::-1]):
        for s, g in zip(streams, (a, b)):
            with torch.cuda.stream(s):
                g.replay()
torch.cuda.synchronize()
for i in range(2):
    for x, w in zip(outs[i], want[i]):
        assert torch.equal(x, w)
assert zt.lib.tc_status() == 0
"""
    r = subprocess.run([sys.executable, "-c", code], cwd=ROOT, capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stderr[-2000:]


def test_reserved_windows_map_no_memory(zt):
    """After the holder's reservation the pool holds what its windows take: free memory stays as it is, also where the
    device was waited for in between."""
    window(zt, 7, 1300, 512, 8, 2, 64)()  # (loads the kernels)
    f = window(zt, 7, 4096, 512, 8, 2, 64)
    torch.cuda.synchronize()
    free = torch.cuda.mem_get_info()[0]
    for _ in range(3):
        f()
        torch.cuda.synchronize()
        assert torch.cuda.mem_get_info()[0] == free
