"""The per-device arena behind the entry points that take no workspace (zt_attn_forward, zt_attn_backward,
zt_attn_forward_batched): it may allocate, so it must never do so inside a stream capture, and a caller can size
it up front with zt_attn_reserve.  (This file sorts before the full-size tests so that the arena is still small
when it runs; it also works after them.)"""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def dev():
    assert torch.cuda.is_available(), "these tests need a CUDA device"
    return torch.device("cuda:0")


def test_reference_abi_refuses_to_grow_its_arena_inside_a_capture(zt, dev):
    """zt_attn_forward takes its operand planes from the per-device arena.  Growing the arena means cudaMalloc,
    which must not happen while the caller's stream is being captured: the call is refused (return 1, nothing
    launched, the capture intact) and works once zt_attn_reserve has sized the arena beforehand."""
    L = zt.lib.load()
    H, Hkv, D = 8, 2, 128
    # a sequence whose operand planes (T x (8 + 2 + 2) x 128 x 4 bytes) need more than the arena holds now
    T = max(9000, int(L.zt_attn_arena_bytes() * 1.25) // ((H + 2 * Hkv) * D * 4))
    g = torch.Generator(device=dev).manual_seed(3)
    q = torch.randn((T, H * D), generator=g, device=dev)
    k, v = (torch.randn((T, Hkv * D), generator=g, device=dev) for _ in range(2))
    out = torch.full_like(q, 7.0)
    graph = torch.cuda.CUDAGraph()
    side = torch.cuda.Stream(dev)
    L.zt_attn_set_verbose(0)
    rcs = []
    with torch.cuda.stream(side):
        with torch.cuda.graph(graph, stream=side):
            st = torch.cuda.current_stream(dev).cuda_stream
            rcs.append(L.zt_attn_forward(q.data_ptr(), k.data_ptr(), v.data_ptr(), out.data_ptr(), T, H, Hkv, D, 1, 64, 0, T, st))
    L.zt_attn_set_verbose(1)
    assert rcs == [1] and "zt_attn_reserve" in zt.lib.last_error()
    graph.replay()  # an empty graph: the refused call enqueued nothing and did not break the capture
    torch.cuda.synchronize()
    assert bool((out == 7.0).all())
    assert L.zt_attn_reserve(1, T, H, Hkv, D) == 0
    graph2 = torch.cuda.CUDAGraph()
    # eager once (sets the kernels' shared-memory attributes), then captured
    assert L.zt_attn_forward(q.data_ptr(), k.data_ptr(), v.data_ptr(), out.data_ptr(), T, H, Hkv, D, 1, 64, 0, T,
                             torch.cuda.current_stream(dev).cuda_stream) == 0
    torch.cuda.synchronize()
    want = out.clone()
    with torch.cuda.stream(side):
        with torch.cuda.graph(graph2, stream=side):
            st = torch.cuda.current_stream(dev).cuda_stream
            assert L.zt_attn_forward(q.data_ptr(), k.data_ptr(), v.data_ptr(), out.data_ptr(), T, H, Hkv, D, 1, 64, 0, T, st) == 0
    out.fill_(float("nan"))
    graph2.replay()
    torch.cuda.synchronize()
    assert torch.equal(out, want) and zt.lib.tc_status() == 0


def test_reserving_a_shape_covers_a_shorter_one_that_is_split(zt):
    """32/8 heads of 128, one sequence: 2304 rows want more scratch than 2432 (the backward's walk is split there).  A
    process of its own, whose arena nothing else has grown."""
    import subprocess
    import sys
    code = """
import importlib, torch
zt = importlib.import_module("z-transformer_b200")
L, shape = zt.lib.load(), (32, 8, 128)
assert L.zt_attn_backward_workspace_bytes(1, 2304, *shape) > L.zt_attn_backward_workspace_bytes(1, 2432, *shape)
assert L.zt_attn_reserve(1, 2432, *shape) == 0
held = L.zt_attn_arena_bytes()
assert held == L.zt_attn_reserve_bytes(1, 2432, *shape)
a = zt.Attn(2304, *shape)
for x in ("q", "k", "v", "dout"):
    getattr(a, x).normal_()
a.backward()
torch.cuda.synchronize()
assert L.zt_attn_arena_bytes() == held and zt.lib.last_path() == "tcgen05" and zt.lib.tc_status() == 0
"""
    root = __file__.rsplit("/tests/", 1)[0]
    r = subprocess.run([sys.executable, "-c", code], cwd=root, capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stderr[-2000:]


def rel(a, b):
    return float((a - b).norm() / b.norm())


@pytest.mark.parametrize("H,Hkv,D", [(4, 2, 128), (3, 1, 64), (4, 2, 192), (2, 1, 256)])
def test_a_workspace_for_the_longest_sequence_serves_the_shorter_ones(zt, dev, H, Hkv, D):
    """The backward, plain and with the forward's planes kept, in every workspace between what a longer sequence is told
    to bring and what this one would like: the split, or the heads that go through memory together, take what is there."""
    L = zt.lib.load()
    if D <= 128:
        T = next(t for t in range(256, 4000, 64) if L.zt_attn_backward_workspace_bytes(1, t, H, Hkv, D) >
                 L.zt_attn_backward_workspace_bytes(1, t + 128, H, Hkv, D))
        room = L.zt_attn_backward_workspace_bytes(1, T + 128, H, Hkv, D)
    else:  # (two planes of P and two of dS a head: room for one KV group instead of all)
        T = 300
        room = L.zt_attn_backward_workspace_bytes(1, T, H, Hkv, D) - 8 * 384 ** 2 * (H - H // Hkv)
    best = L.zt_attn_backward_workspace_bytes(1, T, H, Hkv, D)
    g = torch.Generator(device=dev).manual_seed(11)
    q, do = (torch.randn((1, T, H * D), generator=g, device=dev) for _ in range(2))
    k, v = (torch.randn((1, T, Hkv * D), generator=g, device=dev) for _ in range(2))
    results = []
    for nbytes in (best, room):
        # (guarded: what lies behind the workspace is not the call's)
        ws = torch.full((nbytes + 4096,), 85, dtype=torch.uint8, device=dev)
        out, lse, delta = torch.empty_like(q), torch.empty((1, T, H), device=dev), torch.empty((1, T, H), device=dev)
        token = zt.lib.C.c_ulonglong(0)
        st = torch.cuda.current_stream().cuda_stream
        assert L.zt_attn_forward_batched_keep(q.data_ptr(), k.data_ptr(), v.data_ptr(), out.data_ptr(), lse.data_ptr(), ws.data_ptr(),
                                              nbytes, 1, T, H, Hkv, D, st, zt.lib.C.byref(token)) == 0, zt.lib.last_error()
        assert token.value != 0
        for tok in (token.value, 0):
            dq, dk, dv = torch.empty_like(q), torch.empty_like(k), torch.empty_like(v)
            assert L.zt_attn_backward_batched_kept(*(x.data_ptr() for x in (q, k, v, out, lse, do, dq, dk, dv, delta, ws)), nbytes,
                                                   1, T, H, Hkv, D, st, tok) == 0, zt.lib.last_error()
            torch.cuda.synchronize()
            assert zt.lib.last_path() == "tcgen05" and zt.lib.tc_status() == 0
            results.append((out, lse, dq, dk, dv))
        assert bool((ws[nbytes:] == 85).all())
    for r in results[1:]:
        for name, a, b in zip(("out", "lse", "dq", "dk", "dv"), r, results[0]):
            # the same products with their sums cut elsewhere: the truncating accumulator costs either 3.7e-6 at most
            # between two flushes (kFlushKeyTiles in csrc/tc_fwd16.cuh; the backward flushes as often)
            assert rel(a, b) <= 8e-6, name


@pytest.mark.parametrize("T,D", [(300, 80), (100, 64), (140, 160), (90, 256)])
def test_shapes_that_can_do_without_a_workspace(zt, dev, oracle, T, D):
    """Widths between the tiles' and short sequences: without a workspace, or with too little, the CUDA cores take them."""
    L = zt.lib.load()
    H, Hkv = 2, 1
    q, k, v, do = (oracle.fill_normal((T, w * D), 12, i) for i, w in enumerate((H, Hkv, Hkv, H)))
    tq, tk, tv, tdo = (torch.from_numpy(x).to(dev) for x in (q, k, v, do))
    out, lse = zt.attention_forward(tq[None], tk[None], tv[None], H, Hkv, D, want_lse=True)
    want = oracle.attention_backward(q, k, v, do, H, Hkv, D)
    delta = torch.empty((1, T, H), device=dev)
    some = torch.empty(1024, dtype=torch.uint8, device=dev)
    for ws, nbytes in ((None, 0), (some.data_ptr(), 1024)):
        dq, dk, dv = torch.empty_like(tq), torch.empty_like(tk), torch.empty_like(tv)
        assert L.zt_attn_backward_batched(*(x.data_ptr() for x in (tq, tk, tv, out, lse, tdo, dq, dk, dv, delta)), ws, nbytes, 1, T, H,
                                          Hkv, D, torch.cuda.current_stream().cuda_stream) == 0, zt.lib.last_error()
        torch.cuda.synchronize()
        assert zt.lib.last_path() == "simt"
        for got, ref in zip((dq, dk, dv), want):
            ref = torch.from_numpy(ref)
            assert bool(((got.cpu() - ref).abs() <= 1e-5 + 1e-4 * ref.abs()).all())  # (the stated bar of this path)
