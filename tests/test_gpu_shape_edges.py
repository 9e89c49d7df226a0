"""Shapes at the edges of the tensor-core kernels' tiles, through the public calls, against the CPU oracle: head widths
that no tile has (padded to the next wider one), sequences shorter than a tile of query rows, and windows of a prompt
at an offset.  Tolerance: the stated bar of this path, |got - ref| <= 1e-5 + 1e-4 |ref|, element-wise."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def close(got, ref, what):
    got, ref = got.cpu().numpy().astype(np.float64), np.asarray(ref, np.float64)
    assert got.shape == ref.shape, what
    bad = ~(np.abs(got - ref) <= 1e-5 + 1e-4 * np.abs(ref))
    assert not bad.any(), (what, int(bad.sum()), float(np.nanmax(np.abs(got - ref))))


def normal(oracle, shape, stream):
    return oracle.fill_normal(shape, 93, stream)


@pytest.mark.parametrize("B,T,H,Hkv,D", [
    (2, 33, 4, 2, 36), (1, 64, 3, 1, 40), (1, 1, 4, 2, 64), (2, 65, 4, 4, 60), (1, 2, 2, 1, 128), (1, 127, 4, 2, 68),
    (2, 129, 6, 2, 80), (1, 32, 4, 1, 124), (1, 100, 4, 2, 132), (1, 63, 2, 2, 200), (1, 257, 2, 1, 252), (3, 31, 8, 2, 256),
    # few key tiles for the chip: the backward's walk is split by heads, then by ranges of query tiles
    (1, 1000, 4, 2, 64), (1, 700, 3, 3, 40), (2, 300, 8, 1, 128), (1, 1100, 2, 1, 72),
    # the 192-column tile: its narrowest and widest heads, several key tiles a block, more than one piece of a contraction
    (1, 385, 3, 3, 132), (2, 300, 4, 2, 192), (1, 1290, 2, 1, 188),
    # more than one block an SM: the blocks go tile by tile through the sequences (and with odd ones among them)
    (20, 130, 8, 4, 64), (30, 140, 3, 3, 128), (11, 260, 9, 3, 160), (40, 150, 4, 2, 96),
    # planes narrower than the tile, on either side of where they become so
    (1, 300, 4, 2, 32), (2, 200, 2, 1, 72), (1, 200, 2, 2, 96), (1, 200, 4, 2, 100),
])
def test_widths_and_short_sequences(zt, oracle, B, T, H, Hkv, D):
    q, k, v, do = (normal(oracle, (B, T, w * D), i) for i, w in enumerate((H, Hkv, Hkv, H)))
    tq, tk, tv, tdo = (torch.from_numpy(x).cuda() for x in (q, k, v, do))
    ws = zt.BackwardWorkspace(B, T, H, Hkv, D)
    o, lse = zt.attention_forward(tq, tk, tv, H, Hkv, D, want_lse=True, keep=ws)
    grads = zt.attention_backward(tq, tk, tv, o, lse, tdo, H, Hkv, D, workspace=ws, kept=ws.token != 0)
    torch.cuda.synchronize()
    assert zt.lib.last_path() == "tcgen05" and zt.lib.tc_status() == 0 and zt.lib.tc_saturated() == 0
    for b in range(B):
        ro, rl = oracle.attention_forward(q[b], k[b], v[b], H, Hkv, D, want_lse=True, threads=4)
        ref = oracle.attention_backward(q[b], k[b], v[b], do[b], H, Hkv, D, threads=4)
        for name, got, want in zip(("out", "lse", "dq", "dk", "dv"), (o, lse, *grads), (ro, rl, *ref)):
            close(got[b], want, f"{name}[{b}]")


@pytest.mark.parametrize("T,q_offset,ctx,H,Hkv,D", [
    (33, 1, 40, 4, 2, 32), (64, 63, 127, 3, 1, 64), (128, 64, 192, 4, 1, 80), (200, 313, 600, 8, 2, 128),
    (129, 511, 700, 6, 3, 96), (40, 0, 64, 2, 2, 192), (70, 250, 320, 4, 2, 256), (96, 1000, 1500, 32, 8, 128),
    # many key tiles: the row sums leave the tensor core's accumulator every sixteen of them
    (129, 2900, 3100, 2, 1, 128), (300, 2100, 2400, 4, 1, 64), (40, 1500, 1540, 2, 1, 256),
    # few rows: the keys are split over the chip (parts that some rows see nothing of, parts that sum in memory too)
    (2, 700, 702, 4, 2, 64), (16, 3000, 3016, 2, 1, 96), (150, 5000, 5200, 4, 4, 64), (100, 2500, 2600, 2, 2, 256),
    (700, 1, 701, 2, 1, 64), (250, 9000, 9250, 8, 2, 40),
    (300, 2100, 2400, 4, 1, 192), (100, 2500, 2600, 2, 2, 160),
    # not split, and the planes narrower than the tile: one of the two running sums lives in the query rows' planes
    (40, 2100, 2140, 76, 76, 72),
])
def test_windows_of_a_prompt(zt, oracle, T, q_offset, ctx, H, Hkv, D):
    """device.Attn.forward_at: rows at q_offset over the first q_offset + T keys; what lies beyond is never read."""
    q = normal(oracle, (T, H * D), 0)
    n_keys = q_offset + T
    k, v = (normal(oracle, (n_keys, Hkv * D), i) for i in (1, 2))
    holder = zt.Attn(ctx, H, Hkv, D)
    holder.k.fill_(float("nan")), holder.v.fill_(float("nan")), holder.q.zero_()
    for name, x in (("q", q), ("k", k), ("v", v)):
        holder.upload(getattr(holder, name), x)
    holder.forward_at(1, 64, q_offset, n_keys, T)
    torch.cuda.synchronize()
    assert zt.lib.last_path() == "tcgen05" and zt.lib.tc_status() == 0
    ref = oracle.attention_forward_at(q, k, v, H, Hkv, D, q_offset, n_keys)
    got = holder.out[: q.size].view(q.shape)
    close(got, ref, "window")
    # the CUDA-core kernels served these calls with rounded f32 sums: as a whole no further off than they are
    assert float(np.linalg.norm(got.cpu().numpy() - ref) / np.linalg.norm(ref)) <= 5e-6


def test_split_launches_are_reproducible(zt, oracle):
    """Parts are put together in a fixed order: out, lse, dk and dv come out bit for bit the same (dq is summed in memory)."""
    T, H, Hkv, D = 900, 4, 1, 64
    q, k, v, do = (torch.from_numpy(normal(oracle, (1, T, w * D), i)).cuda() for i, w in enumerate((H, Hkv, Hkv, H)))
    runs = []
    for _ in range(2):
        o, lse = zt.attention_forward(q, k, v, H, Hkv, D, want_lse=True)
        runs.append((o, lse, *zt.attention_backward(q, k, v, o, lse, do, H, Hkv, D)[1:]))
    for a, b in zip(*runs):
        assert torch.equal(a, b)


@pytest.mark.parametrize("T,H,Hkv,D,pos", [(70, 4, 2, 40, 3), (150, 2, 1, 136, 0), (90, 2, 2, 68, 5)])
def test_rope_at_widths_between_the_tiles(zt, oracle, T, H, Hkv, D, pos):
    """Halves that are multiples of four ride in the pre-pass; others are rotated before it."""
    q, k, v, do = (normal(oracle, (1, T, w * D), i) for i, w in enumerate((H, Hkv, Hkv, H)))
    tq, tk, tv, tdo = (torch.from_numpy(x).cuda() for x in (q, k, v, do))
    ws = zt.RopeWorkspace(1, T, H, Hkv, D)
    o, lse = zt.attention_forward_rope(tq, tk, tv, H, Hkv, D, pos=pos, workspace=ws, want_lse=True)
    dq, dk, dv = zt.attention_backward_rope(tq, tk, tv, o, lse, tdo, H, Hkv, D, pos=pos, workspace=ws, kept=ws.token != 0)
    torch.cuda.synchronize()
    assert zt.lib.last_path() == "tcgen05" and zt.lib.tc_status() == 0
    qr, kr = oracle.rope_forward(q[0], pos, D), oracle.rope_forward(k[0], pos, D)
    close(o[0], oracle.attention_forward(qr, kr, v[0], H, Hkv, D), "out")
    rdq, rdk, rdv = oracle.attention_backward(qr, kr, v[0], do[0], H, Hkv, D)
    for name, got, want in (("dq", dq, oracle.rope_backward(rdq, pos, D)), ("dk", dk, oracle.rope_backward(rdk, pos, D)), ("dv", dv, rdv)):
        close(got[0], want, name)


@pytest.mark.parametrize("B,T,k,n", [(1, 1000, 1088, 1216), (2, 1100, 1600, 1536)])
def test_projection_on_wide_tiles(zt, oracle, B, T, k, n):
    """Large enough for the 128 x 256 tiles (the second in all three products, several to a block), with tails in rows
    and columns, a half of a tile beyond the columns, and contractions cut into pieces.  The reference reduces in f32, so
    the gate is its own, relative to the tensor's largest magnitude (src/train.zig:706)."""
    ctx, dy = normal(oracle, (B, T, k), 0), normal(oracle, (B, T, n), 1)
    wo, dwo0 = normal(oracle, (k, n), 2) / np.float32(np.sqrt(k)), normal(oracle, (k, n), 3)
    tctx, two, tdy, tdwo = (torch.from_numpy(np.ascontiguousarray(x)).cuda() for x in (ctx, wo, dy, dwo0))
    ws = zt.ProjWorkspace(B, T, k, n)
    y = zt.proj_forward(tctx, two, workspace=ws)
    dctx = zt.proj_backward(tctx, two, tdy, tdwo, workspace=ws)
    torch.cuda.synchronize()
    assert zt.lib.tc_status() == 0
    ref_dwo = dwo0.copy()
    pairs = []
    for b in range(B):
        pairs += [(y[b], oracle.matmul(ctx[b], wo, threads=8)), (dctx[b], oracle.input_grad(dy[b], wo, threads=8))]
        oracle.weight_grad(ref_dwo, ctx[b], dy[b], threads=8)
    for got, ref in pairs + [(tdwo, ref_dwo)]:
        err = np.abs(got.cpu().numpy().astype(np.float64) - ref)
        assert float(np.where(np.isnan(err), np.inf, err).max()) <= 1e-4 * float(np.abs(ref).max())


@pytest.mark.parametrize("B,T,H,Hkv,D", [(2, 70, 4, 2, 32), (1, 150, 4, 2, 96), (1, 140, 3, 3, 128), (1, 200, 2, 1, 160), (1, 90, 2, 2, 256)])
def test_backward_takes_an_output_on_a_four_byte_boundary(zt, B, T, H, Hkv, D):
    """Of out only the row sums with dout are wanted, so it need not start where the tensor copies of q, k, v and dout
    do: an out at an odd offset of a larger buffer gives what the same values give in a buffer of their own (delta is the
    same sum; dq, and above 128 columns dk and dv, are added in memory in no fixed order)."""
    gen = torch.Generator(device="cuda").manual_seed(4)
    q, k, v, do = (torch.randn((B, T, w * D), generator=gen, device="cuda") for w in (H, Hkv, Hkv, H))
    ws = zt.BackwardWorkspace(B, T, H, Hkv, D)
    out, lse = zt.attention_forward(q, k, v, H, Hkv, D, want_lse=True)
    want = zt.attention_backward(q, k, v, out, lse, do, H, Hkv, D, workspace=ws)
    for odd in (1, 2, 3):
        moved = torch.empty(out.numel() + 4, device="cuda")[odd:odd + out.numel()].view(out.shape).copy_(out)
        assert moved.data_ptr() % 16 == 4 * odd
        got = zt.attention_backward(q, k, v, moved, lse, do, H, Hkv, D, workspace=ws)
        torch.cuda.synchronize()
        assert zt.lib.last_path() == "tcgen05" and zt.lib.tc_status() == 0
        for name, a, b in zip(("dq", "dk", "dv"), got, want):
            # two orders of at most ten f32 additions
            assert float((a - b).abs().max()) <= 1e-5 * float(b.abs().max()), name


def test_a_flag_whose_truth_raises(zt):
    """want_lse is asked for its truth in native code: what it raises is what the caller sees."""
    q, k, v = (torch.randn((1, 40, w * 32), device="cuda") for w in (2, 1, 1))
    both = np.array([True, False])
    with pytest.raises(ValueError):
        zt.attention_forward(q, k, v, 2, 1, 32, want_lse=both)
    nk = torch.full((1,), 40, dtype=torch.int32, device="cuda")
    with pytest.raises(ValueError):
        zt.decode_attention(q[:, 0].contiguous(), k, v, nk, 2, 1, 32, workspace=zt.DecodeWorkspace(1, 40, 2, 1, 32), want_lse=both)


@pytest.mark.parametrize("path,T,q_offset,H,Hkv,D", [
    # two heads a block, whose row sums leave the accumulator on the way: forced, the planes as wide as the tile and narrower
    (7, 129, 2900, 2, 1, 128), (7, 300, 2100, 4, 1, 72), (7, 70, 1500, 4, 2, 64), (7, 33, 5, 2, 1, 96),
    # and where enough blocks make it the default
    (0, 1200, 1100, 32, 8, 64),
])
def test_windows_two_heads_a_block(zt, oracle, path, T, q_offset, H, Hkv, D):
    n_keys = q_offset + T
    q = normal(oracle, (T, H * D), 0)
    k, v = (normal(oracle, (n_keys, Hkv * D), i) for i in (1, 2))
    holder = zt.Attn(n_keys, H, Hkv, D)
    for name, x in (("q", q), ("k", k), ("v", v)):
        holder.upload(getattr(holder, name), x)
    L = zt.lib.load()
    L.zt_attn_set_path(path)
    try:
        L.zt_attn_profile(1)
        holder.forward_at(1, 64, q_offset, n_keys, T)
        torch.cuda.synchronize()
        names = kernels_timed(zt)
    finally:
        L.zt_attn_profile(0)
        L.zt_attn_set_path(0)
    assert "attn_fwd_tc16g" in names and zt.lib.tc_status() == 0
    ref = oracle.attention_forward_at(q, k, v, H, Hkv, D, q_offset, n_keys, threads=8)
    got = holder.out[: q.size].view(q.shape)
    close(got, ref, "window")
    assert float(np.linalg.norm(got.cpu().numpy() - ref) / np.linalg.norm(ref)) <= 5e-6


def kernels_timed(zt):
    """Names of the kernels timed since zt_attn_profile(1)."""
    import ctypes
    buf = ctypes.create_string_buffer(4096)
    zt.lib.load().zt_attn_profile_read(buf, 4096)
    return {line.split()[0] for line in buf.value.decode().splitlines()}


@pytest.mark.parametrize("D", [160, 192, 256])
def test_wide_heads_tile_by_tile(zt, oracle, D):
    """More blocks than SMs and at most twice as many, odd numbers of heads and tiles: the wide forward goes tile by tile."""
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    T, H, Hkv = 260, 9, 3  # 27 blocks a sequence
    B = sms // 27 + 2
    assert sms < 27 * B <= 2 * sms
    q, k, v = (normal(oracle, (B, T, w * D), i) for i, w in enumerate((H, Hkv, Hkv)))
    o, lse = zt.attention_forward(*(torch.from_numpy(x).cuda() for x in (q, k, v)), H, Hkv, D, want_lse=True)
    torch.cuda.synchronize()
    assert zt.lib.last_path() == "tcgen05" and zt.lib.tc_status() == 0
    for b in range(B):
        ro, rl = oracle.attention_forward(q[b], k[b], v[b], H, Hkv, D, want_lse=True, threads=8)
        close(o[b], ro, f"out[{b}]"), close(lse[b], rl, f"lse[{b}]")


@pytest.mark.parametrize("B,T,H,Hkv,D", [(2, 70, 4, 2, 40), (1, 200, 2, 1, 80), (1, 150, 3, 1, 96), (1, 33, 2, 2, 100), (2, 129, 4, 2, 160),
                                         (1, 260, 2, 1, 192), (1, 90, 2, 1, 252)])
def test_earlier_backward_forms_at_widths_between_the_tiles(zt, oracle, B, T, H, Hkv, D):
    """zt_attn_set_path(8): the two-kernel backward, and the scores that load every operand per tile, on padded heads."""
    q, k, v, do = (normal(oracle, (B, T, w * D), i) for i, w in enumerate((H, Hkv, Hkv, H)))
    tq, tk, tv, tdo = (torch.from_numpy(x).cuda() for x in (q, k, v, do))
    L = zt.lib.load()
    L.zt_attn_set_path(8)
    try:
        o, lse = zt.attention_forward(tq, tk, tv, H, Hkv, D, want_lse=True)
        L.zt_attn_profile(1)
        grads = zt.attention_backward(tq, tk, tv, o, lse, tdo, H, Hkv, D)
        torch.cuda.synchronize()
        names = kernels_timed(zt)
    finally:
        L.zt_attn_profile(0)
        L.zt_attn_set_path(0)
    assert ("attn_bwd_dq_tc" if D <= 128 else "bwd_wide_scores") in names and zt.lib.tc_status() == 0
    for b in range(B):
        ref = oracle.attention_backward(q[b], k[b], v[b], do[b], H, Hkv, D, threads=4)
        for name, got, want in zip(("dq", "dk", "dv"), grads, ref):
            close(got[b], want, f"{name}[{b}]")
