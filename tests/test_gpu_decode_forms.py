"""Both forms of the decode step -- clusters in one launch, and chunks whose partial results a second kernel puts together --
at every width and group the kernel is compiled for, with the shortest and longest prefixes and with refused ones.
Tolerance: the stated bar of this path, |got - ref| <= 1e-5 + 1e-4 |ref|, element-wise."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

# more keys than eight blocks of a cluster take (768 each): two launches, whatever the device
LONG = 6300


def check(zt, oracle, n_ctx, H, Hkv, D, n_keys, launches):
    B = len(n_keys)
    k, v = (oracle.fill_normal((B, n_ctx, Hkv * D), 51, i) for i in (1, 2))
    q = oracle.fill_normal((B, H * D), 51, 0)
    ws = zt.DecodeWorkspace(B, n_ctx, H, Hkv, D)
    ws.buf.fill_(255)  # (NaN partial results, and a count that has to be written)
    nk = torch.tensor(n_keys, dtype=torch.int32, device="cuda")
    tq, tk, tv = (torch.from_numpy(x).cuda() for x in (q, k, v))
    out, lse = zt.decode_attention(tq, tk, tv, nk, H, Hkv, D, workspace=ws, want_lse=True)
    before = zt.lib.launch_count()
    again, _ = zt.decode_attention(tq, tk, tv, nk, H, Hkv, D, workspace=ws, want_lse=True)
    assert zt.lib.launch_count() - before == launches and zt.lib.last_path() == "decode-splitk"
    torch.cuda.synchronize()
    assert ws.bad_sequences() == sum(not 1 <= n <= n_ctx for n in n_keys)
    assert torch.equal(out.nan_to_num(7.0), again.nan_to_num(7.0))
    out, lse = out.cpu().numpy(), lse.cpu().numpy()
    for b, n in enumerate(n_keys):
        if not 1 <= n <= n_ctx:
            assert np.isnan(out[b]).all() and np.isnan(lse[b]).all()
            continue
        for got, ref in zip((out[b], lse[b]), oracle.attn_step_raw(q[b], k[b], v[b], n, H, Hkv, D, threads=8)):
            err = np.abs(got.astype(np.float64) - ref)
            assert (err <= 1e-5 + 1e-4 * np.abs(ref)).all(), (b, n, float(np.nanmax(err)))


@pytest.mark.parametrize("H,Hkv,D", [
    # every (lanes, chunks) of a row at one, two and four heads a pass; groups of three and six fill a pass in part, of
    # eight take two passes
    (2, 2, 32), (4, 2, 32), (4, 1, 32), (2, 2, 64), (6, 1, 64), (2, 1, 96), (8, 1, 96), (2, 2, 128), (3, 1, 128),
    (2, 2, 192), (4, 2, 160), (4, 1, 192), (1, 1, 256), (2, 1, 256), (8, 1, 256), (4, 1, 36), (4, 2, 252),
])
def test_two_launches(zt, oracle, H, Hkv, D):
    # one key; a chunk's edge and its neighbours; full; refused ones among them, first and last
    check(zt, oracle, LONG, H, Hkv, D, [0, 1, 128, 129, 127, LONG, 2049, 3000, LONG + 1, -5], 2)


@pytest.mark.parametrize("B,n_ctx,H,Hkv,D", [
    # widths of which an SM holds one block: one wave of clusters, and two
    (4, 1024, 32, 8, 256), (8, 1024, 16, 4, 192), (16, 300, 32, 8, 256), (16, 900, 16, 8, 192), (32, 200, 32, 8, 256),
    # two blocks an SM
    (8, 500, 32, 8, 128), (30, 70, 8, 8, 64), (1, 6144, 4, 1, 32), (5, 400, 16, 2, 96), (3, 500, 16, 16, 128),
])
def test_clusters(zt, oracle, B, n_ctx, H, Hkv, D):
    n_keys = [n_ctx, 1, 0, n_ctx // 2, 63, 64, 65, n_ctx - 1] * B
    check(zt, oracle, n_ctx, H, Hkv, D, n_keys[:B], 1)


def test_many_sequences_of_short_prefixes(zt, oracle):
    """More (sequence, KV head) pairs than places for clusters: two launches of few chunks each."""
    check(zt, oracle, 200, 16, 8, 64, [1 + (37 * i) % 200 for i in range(98)] + [0, 201], 2)


def test_static_scratch_in_two_launches(zt, oracle):
    """zt_attn_decode_static over the built-in scratch: the two-launch form's results and count, twice over its own leftovers."""
    import ctypes
    L = zt.lib.load()
    H, Hkv, D = 4, 2, 64
    n_keys = [LONG, 0, 129, 5000, LONG + 1, 1]
    B = len(n_keys)
    k, v = (torch.from_numpy(oracle.fill_normal((B, LONG, Hkv * D), 52, i)).cuda() for i in (1, 2))
    nk = torch.tensor(n_keys, dtype=torch.int32, device="cuda")
    for seed in (0, 3):
        q = torch.from_numpy(oracle.fill_normal((B, H * D), 52, seed)).cuda()
        want, want_lse = zt.decode_attention(q, k, v, nk, H, Hkv, D, workspace=zt.DecodeWorkspace(B, LONG, H, Hkv, D), want_lse=True)
        out, lse = torch.full_like(q, 9.0), torch.full((B, H), 9.0, device="cuda")
        before = zt.lib.launch_count()
        assert L.zt_attn_decode_static(*(x.data_ptr() for x in (q, k, v, nk, out, lse)), B, LONG, H, Hkv, D,
                                       torch.cuda.current_stream().cuda_stream) == 0, zt.lib.last_error()
        assert zt.lib.launch_count() - before == 2
        torch.cuda.synchronize()
        bad = ctypes.c_int(-1)
        assert L.zt_attn_decode_status(None, ctypes.byref(bad)) == 0 and bad.value == 2
        for a, b in ((out, want), (lse, want_lse)):
            assert torch.equal(a.isnan(), b.isnan()) and torch.equal(a.nan_to_num(7.0), b.nan_to_num(7.0))
