"""The calls whose speed this framework is judged by: what a training program and a serving program make of it.

listed() names twelve fixed cases, draw() makes more of the same ranges.  Every case goes through the public entry
points of the package and returns its whole outputs.  Kinds:

  prefill     attention_forward over whole prompts (inference: no log-sum-exp, nothing kept for a backward)
  window      device.Attn.forward_at: a chunk of a prompt at q_offset, over the keys cached so far
  train       attention_forward(keep=...) then attention_backward(kept=True) on a workspace that outlives the step
  block       AttentionBlock: rope, attention and the output projection, forward and backward
  completion  a run of decode steps from a cached prompt: KV append, then attention, one row per sequence and step
  decode      one attention step over caches that are already filled (uniform or ragged lengths)
"""
import importlib
import math

import torch

zt = importlib.import_module("z-transformer_b200")

#: (query heads, KV heads): GPT-mini, small GQA, no grouping, and the Llama-3-8B geometry of the benchmark
HEADS = ((4, 2), (8, 2), (12, 4), (16, 16), (32, 8))
#: head widths of the benchmark sweep and the harness table, each as likely as its use
WIDTHS = (32, 64, 64, 96, 128, 128, 128, 192, 256)
MAX_FLOPS = 1.0e12         # of a drawn compute case: a quarter of the largest listed step
MAX_CACHE_BYTES = 8 << 30  # of a drawn decode case: a quarter of the largest listed cache


def listed():
    return [
        # a short prompt in a server: one sequence, Llama-3-8B heads, shorter than one tile of 128 rows
        {"name": "prompt-t77-d128", "kind": "prefill", "batch": 1, "t": 77, "heads": 32, "kv_heads": 8, "dim": 128},
        # a chunk of a long prompt: 512 rows against the 4096 keys cached so far
        {"name": "window-t512-of-4096", "kind": "window", "t": 512, "q_offset": 3584, "ctx": 4096, "heads": 32,
         "kv_heads": 8, "dim": 128},
        # the reference's own training shape (GPT-mini, context 256), one sequence: launches and host work
        {"name": "train-gptmini-t256", "kind": "train", "batch": 1, "t": 256, "heads": 4, "kv_heads": 2, "dim": 32},
        # the short end of the benchmark sweep
        {"name": "train-t512-d64", "kind": "train", "batch": 8, "t": 512, "heads": 32, "kv_heads": 8, "dim": 64},
        # a head width between the sweep's and a length that no tile divides
        {"name": "train-t1000-d80", "kind": "train", "batch": 4, "t": 1000, "heads": 16, "kv_heads": 4, "dim": 80},
        # the widest heads of the sweep
        {"name": "train-t1024-d256", "kind": "train", "batch": 8, "t": 1024, "heads": 32, "kv_heads": 8, "dim": 256},
        # the headline training point of bench.py
        {"name": "train-t4096-d128", "kind": "train", "batch": 8, "t": 4096, "heads": 32, "kv_heads": 8, "dim": 128},
        # long-context training: one sequence
        {"name": "train-t32768-d128", "kind": "train", "batch": 1, "t": 32768, "heads": 32, "kv_heads": 8, "dim": 128},
        # a transformer block's attention part, forward and backward, at the Llama-3-8B widths
        {"name": "block-t2048-d128", "kind": "block", "batch": 2, "t": 2048, "heads": 32, "kv_heads": 8, "dim": 128,
         "d_model": 4096},
        # sixteen tokens for one user: latency of the append and attention calls
        {"name": "completion-b1-ctx1000", "kind": "completion", "batch": 1, "ctx": 2048, "filled": 1000, "steps": 16,
         "heads": 32, "kv_heads": 8, "dim": 128},
        # a serving batch of equal lengths (the benchmark's decode configuration)
        {"name": "decode-b64-ctx8192", "kind": "decode", "batch": 64, "ctx": 8192, "ragged": False, "heads": 32,
         "kv_heads": 8, "dim": 128},
        # a serving batch of unequal lengths (the benchmark's ragged configuration)
        {"name": "decode-b256-ragged16384", "kind": "decode", "batch": 256, "ctx": 16384, "ragged": True, "heads": 32,
         "kv_heads": 8, "dim": 128},
    ]


def _log_int(rng, low, high):
    return max(low, min(high, round(math.exp(rng.uniform(math.log(low), math.log(high))))))


def draw(rng):
    kind = rng.choice(("prefill", "prefill", "window", "train", "train", "train", "train", "block", "completion",
                       "decode", "decode"))
    heads, kv_heads = rng.choice(HEADS)
    # one width in four is another multiple of 8 (40, 72, 80, 112, 160, ...)
    dim = 8 * rng.randint(4, 32) if rng.random() < 0.25 else rng.choice(WIDTHS)
    case = {"kind": kind, "heads": heads, "kv_heads": kv_heads, "dim": dim}
    if kind in ("prefill", "train"):
        case["batch"] = _log_int(rng, 1, 16)
        case["t"] = _log_int(rng, 16 if kind == "prefill" else 64, 8192)
    elif kind == "window":
        case["ctx"] = _log_int(rng, 256, 16384)
        case["t"] = _log_int(rng, 16, max(16, case["ctx"] // 2))
        case["q_offset"] = rng.randint(0, case["ctx"] - case["t"])
    elif kind == "block":
        # the projection takes extents that are multiples of 64
        case["dim"] = rng.choice((32, 64, 96, 128, 128, 256))
        case["batch"] = _log_int(rng, 1, 8)
        case["t"] = _log_int(rng, 128, 4096)
        case["d_model"] = heads * case["dim"]
    elif kind == "completion":
        case["batch"] = _log_int(rng, 1, 16)
        case["ctx"] = _log_int(rng, 128, 8192)
        case["steps"] = 16
        case["filled"] = rng.randint(1, case["ctx"] - case["steps"] - 1)
    else:
        case["batch"] = _log_int(rng, 1, 256)
        case["ctx"] = _log_int(rng, 64, 16384)
        case["ragged"] = rng.random() < 0.5
    while work(case)["flops"] > MAX_FLOPS or _cache_bytes(case) > MAX_CACHE_BYTES:
        if case.get("batch", 1) > 1:
            case["batch"] = case["batch"] * 2 // 3
        elif kind == "window":
            case["t"] = max(16, case["t"] * 2 // 3)
        else:
            case["t"] = case["t"] * 4 // 5
    return case


def _cache_bytes(case):
    if case["kind"] not in ("completion", "decode"):
        return 0
    return 2 * 4 * case["batch"] * case["ctx"] * case["kv_heads"] * case["dim"]


class _Inputs:
    """N(0, 1) tensors on the GPU from one seed."""

    def __init__(self, seed):
        self.gen = torch.Generator(device="cuda")
        self.gen.manual_seed(seed)

    def __call__(self, *shape, scale=1.0):
        x = torch.randn(shape, dtype=torch.float32, device="cuda", generator=self.gen)
        return x if scale == 1.0 else x.mul_(scale)


def prepare(case, seed):
    normal = _Inputs(seed)
    kind, H, G, D = case["kind"], case["heads"], case["kv_heads"], case["dim"]
    wq, wk = H * D, G * D
    s = {"case": case}
    if kind in ("prefill", "train", "block"):
        B, T = case["batch"], case["t"]
        s.update(q=normal(B, T, wq), k=normal(B, T, wk), v=normal(B, T, wk))
        if kind == "train":
            s["dout"] = normal(B, T, wq)
            s["workspace"] = zt.BackwardWorkspace(B, T, H, G, D)
        elif kind == "block":
            n = case["d_model"]
            s["wo"] = normal(wq, n, scale=wq ** -0.5)
            s["dy"] = normal(B, T, n)
            s["dwo"] = torch.zeros((wq, n), dtype=torch.float32, device="cuda")
            s["block"] = zt.AttentionBlock(B, T, H, G, D, n)
    elif kind == "window":
        attn = zt.Attn(case["ctx"], H, G, D)
        for name in ("q", "k", "v"):
            getattr(attn, name).normal_(generator=normal.gen)
        attn.out.zero_()
        s["attn"] = attn
    else:
        B = case["batch"]
        layer = zt.kv_cache.Layer(case["ctx"], wk, B)
        layer.k.normal_(generator=normal.gen)
        layer.v.normal_(generator=normal.gen)
        s["layer"] = layer
        s["workspace"] = zt.DecodeWorkspace(B, case["ctx"], H, G, D)
        if kind == "completion":
            n = case["steps"]
            s.update(q=normal(n, B, wq), k=normal(n, B, wk), v=normal(n, B, wk))
            s["filled"] = torch.full((B,), case["filled"], dtype=torch.int32)
        else:
            s["q"] = normal(B, wq)
            if case["ragged"]:
                host = torch.Generator()
                host.manual_seed(seed)
                layer.set_lens(torch.randint(1, case["ctx"] + 1, (B,), generator=host, dtype=torch.int32))
            else:
                layer.set_lens(torch.full((B,), case["ctx"], dtype=torch.int32))
    return s


def run(s):
    case = s["case"]
    kind, H, G, D = case["kind"], case["heads"], case["kv_heads"], case["dim"]
    if kind == "prefill":
        return zt.attention_forward(s["q"], s["k"], s["v"], H, G, D)
    if kind == "window":
        t = case["t"]
        s["attn"].forward_at(1, 64, case["q_offset"], case["q_offset"] + t, t)
        return s["attn"].out[: t * H * D]
    if kind == "train":
        q, k, v, ws = s["q"], s["k"], s["v"], s["workspace"]
        out, lse = zt.attention_forward(q, k, v, H, G, D, want_lse=True, keep=ws)
        # off the tensor-core path the forward keeps nothing, which its workspace says with token 0
        dq, dk, dv = zt.attention_backward(q, k, v, out, lse, s["dout"], H, G, D, workspace=ws, kept=ws.token != 0)
        return out, lse, dq, dk, dv
    if kind == "block":
        y = s["block"].forward(s["q"], s["k"], s["v"], s["wo"])
        s["dwo"].zero_()
        dq, dk, dv = s["block"].backward(s["dy"], s["dwo"])
        return y, dq, dk, dv, s["dwo"]
    layer = s["layer"]
    if kind == "completion":
        layer.set_lens(s["filled"])  # back to the prompt: another completion of it begins
        outs = []
        for i in range(case["steps"]):
            layer.append(s["k"][i], s["v"][i])
            outs.append(zt.kv_cache.attn_step(s["q"][i], layer, H, G, D, workspace=s["workspace"]))
        return outs, layer.k, layer.v, layer.len
    return zt.kv_cache.attn_step(s["q"], layer, H, G, D, workspace=s["workspace"])


def work(case):
    """Inputs read once, outputs written once; the multiply-adds of the visible (query, key) pairs."""
    kind, H, G, D = case["kind"], case["heads"], case["kv_heads"], case["dim"]
    if kind == "window":
        t, end = case["t"], case["q_offset"] + case["t"]
        pairs = t * case["q_offset"] + t * (t + 1) // 2
        return {"bytes": 4 * (2 * t * H * D + 2 * end * G * D), "flops": 4 * H * D * pairs}
    if kind in ("prefill", "train", "block"):
        B, T = case["batch"], case["t"]
        rows, forward = B * T, 2 * B * H * D * T * (T + 1)
        wq, wk = H * D, G * D
        if kind == "prefill":
            return {"bytes": 4 * rows * (2 * wq + 2 * wk), "flops": forward}
        if kind == "train":  # q, k, v, dout in; out, lse, dq, dk, dv out
            return {"bytes": 4 * rows * (4 * wq + 4 * wk + H), "flops": 3.5 * forward}
        n = case["d_model"]  # q, k, v, dy, wo in; y, dq, dk, dv, dwo out
        return {"bytes": 4 * (rows * (2 * wq + 4 * wk + 2 * n) + 2 * wq * n), "flops": 3.5 * forward + 6 * rows * wq * n}
    B = case["batch"]
    if kind == "completion":
        n = case["steps"]
        keys = B * (n * case["filled"] + n * (n + 1) // 2)
        rows = n * B * (2 * H * D + 4 * G * D)
    else:
        keys = B * (case["ctx"] + 1) / 2 if case["ragged"] else B * case["ctx"]
        rows = 2 * B * H * D
    return {"bytes": 4 * (keys * 2 * G * D + rows), "flops": 4 * keys * H * D}


def tolerance(case):
    """f32 results of sums over up to 32768 keys and their gradients."""
    return {"rel": 1e-5}
