"""The workloads whose speed this library is judged by, as a program that serves a model calls it.

A case is one attention layer's share of a model step, through the public entry points of `warp34_b200.kv` (or
the C ABI where a step has no Python wrapper): new K and V rows are appended to the layer's paged cache, then the
step's queries attend to everything cached.  Kinds:

  step     append, then paged attention (with the layer's output gate where `gate` says so).  `new` tokens per
           sequence on top of contexts spread evenly over [ctx_lo, ctx_hi]: 1 is a decode step, 2 to 4 verify
           drafted tokens, more are prefill chunks (spread over [new_lo, new])
  host     the same decode step with its inputs and its result in host memory (`kv.DecodeStep`, graph replay)
  append   a prompt's K and V rows appended on their own, as slices of packed projection rows; with
           `producer` the K rows go through the layer's norm and rotary embedding in the same call
  sparse   query-sparse attention of one decode step over selected 4-token groups

Storage (`kv`): "tq4" (4-bit rotated rows, the main format), "fp8" and "q8" (8-bit boundary layers), "bf16"
(uncompressed).  Values are synthetic (`warp34_b200.synth`): normal with four x20 outlier channels per head; page
tables come from a shuffled free list.  Nothing is committed after a pass, so a pass can be repeated.
"""
import ctypes as C
import math

import numpy as np
import torch

from warp34_b200 import ffi, kv, synth

TQ4 = (ffi.KV_FORMAT_TQ4, ffi.KV_FORMAT_TQ4, ffi.KV_TRANSFORM_RADEMACHER_WHT256, ffi.KV_TRANSFORM_RADEMACHER_WHT256)
FP8 = (ffi.KV_FORMAT_FP8_E4M3, ffi.KV_FORMAT_FP8_E4M3, ffi.KV_TRANSFORM_IDENTITY, ffi.KV_TRANSFORM_IDENTITY)
Q8 = (ffi.KV_FORMAT_Q8_0, ffi.KV_FORMAT_Q8_0, ffi.KV_TRANSFORM_IDENTITY, ffi.KV_TRANSFORM_IDENTITY)
FORMATS = {"tq4": TQ4, "fp8": FP8, "q8": Q8, "bf16": tuple(kv.BF16_KV_FORMATS)}
ROW_BYTES = {"tq4": 132, "fp8": 264, "q8": 272, "bf16": 512}
D = 256
SM_SCALE = 1.0 / 16.0
ROTARY, SECTIONS, THETA, EPS = 64, (11, 11, 10), 1.0e6, 1e-6


def step(name, kv_format, q_heads, kv_heads, batch, ctx_lo, ctx_hi, new=1, new_lo=None, gate=0):
    return {"name": name, "kind": "step", "kv": kv_format, "q_heads": q_heads, "kv_heads": kv_heads, "batch": batch,
            "ctx_lo": ctx_lo, "ctx_hi": ctx_hi, "new": new, "new_lo": new if new_lo is None else new_lo, "gate": gate}


def listed():
    return [
        # one user, a short conversation, the layer's sigmoid gate fused: latency and launches
        step("decode_1_short", "tq4", 24, 4, 1, 317, 317, gate=1),
        # a small serving batch, gate and Hadamard-rotated output projection
        step("decode_16", "tq4", 24, 4, 16, 1024, 8192, gate=2),
        # the benchmark's headline batch
        step("decode_64", "tq4", 24, 4, 64, 8192, 32768),
        # speculative decoding: four drafted tokens per sequence are verified
        step("verify_128x4", "tq4", 24, 4, 128, 2048, 16384, new=4),
        # one very long document
        step("decode_256k", "tq4", 16, 4, 1, 262143, 262143),
        # the same batch decode on a boundary layer kept in 8 bits
        step("decode_64_fp8", "fp8", 24, 4, 64, 4096, 16384),
        # a scheduler's mixed step of short and ragged prompts, some after a cached prefix
        step("prefill_ragged", "tq4", 24, 4, 5, 0, 2053, new=899, new_lo=37, gate=1),
        # long prompts in 2048-token chunks, half way through
        step("prefill_8x2048", "tq4", 16, 4, 8, 8192, 8192, new=2048),
        # a prompt's chunk on a boundary layer
        step("prefill_fp8", "fp8", 24, 4, 2, 3072, 4096, new=1024),
        # the end-to-end call of a serving loop whose model runs elsewhere: host buffers in and out
        {"name": "host_decode_4", "kind": "host", "kv": "tq4", "q_heads": 24, "kv_heads": 4, "batch": 4, "ctx_lo": 8192,
         "ctx_hi": 32768},
        # a prefill batch's K and V written to the cache, K normalised and rotated on the way
        {"name": "append_32k", "kind": "append", "kv": "tq4", "q_heads": 24, "kv_heads": 4, "tokens": 32768, "producer": True},
        # query-sparse decode: each of 64 sequences attends to 256 selected groups
        {"name": "sparse_64x256", "kind": "sparse", "kv": "tq4", "q_heads": 24, "kv_heads": 4, "tokens": 64, "groups": 256,
         "ctx": 8192, "gate": 1},
    ]


def _log_int(rng, lo, hi):
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi + 1)))))))


def draw(rng):
    kv_heads = rng.choice((1, 2, 4, 4))
    q_heads = kv_heads * rng.choice((4, 6))
    what = rng.choice(("decode", "decode", "verify", "prefill", "prefill", "host", "append", "sparse"))
    if what in ("decode", "verify"):
        fmt = rng.choice(("tq4", "tq4", "tq4", "fp8", "q8", "bf16"))
        batch = _log_int(rng, 1, 128)
        ctx_hi = _log_int(rng, 64, min(262144, 1200000 // batch))
        case = step("", fmt, q_heads, kv_heads, batch, max(1, ctx_hi // rng.choice((1, 4))), ctx_hi,
                    new=1 if what == "decode" else rng.randint(2, 4), gate=0 if fmt == "bf16" else rng.randint(0, 2))
    elif what == "prefill":
        fmt = rng.choice(("tq4", "tq4", "tq4", "fp8", "q8"))
        batch = _log_int(rng, 1, 8 if fmt == "tq4" else 2)
        new = _log_int(rng, 16, 2048 if fmt == "tq4" else 1024)
        ctx_hi = rng.choice((0, _log_int(rng, 16, 8192)))
        case = step("", fmt, q_heads, kv_heads, batch, ctx_hi // rng.choice((1, 4)), ctx_hi, new=new,
                    new_lo=max(1, new // rng.choice((1, 8))), gate=rng.randint(0, 2))
    elif what == "host":
        ctx_hi = _log_int(rng, 256, 32768)
        case = {"kind": "host", "kv": "tq4", "q_heads": q_heads, "kv_heads": kv_heads, "batch": _log_int(rng, 1, 16),
                "ctx_lo": max(1, ctx_hi // 4), "ctx_hi": ctx_hi}
    elif what == "append":
        fmt = rng.choice(("tq4", "tq4", "fp8", "q8"))
        case = {"kind": "append", "kv": fmt, "q_heads": q_heads, "kv_heads": kv_heads, "tokens": _log_int(rng, 512, 32768),
                "producer": fmt == "tq4" and rng.random() < 0.5}
    else:
        groups = _log_int(rng, 16, 512)
        case = {"kind": "sparse", "kv": rng.choice(("tq4", "tq4", "fp8")), "q_heads": q_heads, "kv_heads": kv_heads,
                "tokens": _log_int(rng, 1, 128), "groups": groups, "ctx": groups * 4 * rng.randint(2, 8), "gate": rng.randint(0, 2)}
    case.pop("name", None)
    return case


def _spread(lo, hi, n):
    """n whole numbers spread evenly over [lo, hi], the largest first."""
    return [hi] if n == 1 else [hi - (hi - lo) * i // (n - 1) for i in range(n)]


def _lens(case):
    """Context and new tokens of every sequence.  Long prompts go with short prefixes."""
    n = case["batch"]
    return _spread(case["ctx_lo"], case["ctx_hi"], n), _spread(case.get("new_lo", 1), case.get("new", 1), n)[::-1]


def prepare(case, seed):
    return {"step": _prepare_step, "host": _prepare_host, "append": _prepare_append, "sparse": _prepare_sparse}[case["kind"]](case, seed)


def run(state):
    return state["run"](state)


def _prepare_step(case, seed):
    ctx, new = _lens(case)
    hq, hkv, bf16 = case["q_heads"], case["kv_heads"], case["kv"] == "bf16"
    wl = synth.PagedWorkload(ctx, new, hkv, seed=seed, formats=FORMATS[case["kv"]])
    ex = kv.Executor()
    wl.fill_context(ex, seed)
    n = sum(new)
    k, v = synth.make_kv(n, hkv, seed + 17, device="cuda")
    q = synth.make_q(n, hq, seed + 17, device="cuda")
    gate = synth.make_q(n, hq, seed + 18, device="cuda") * 2
    if bf16:
        k, v, q = (t.to(torch.bfloat16) for t in (k, v, q))
    return {"run": _run_step_bf16 if bf16 else _run_step, "wl": wl, "layer": wl.layer, "ex": ex, "batch": wl.step(sm_scale=SM_SCALE),
            "k": k, "v": v, "q": q, "gate": gate, "out": torch.zeros_like(q), "hq": hq, "mode": case["gate"]}


def _outputs(s, out):
    return {"out": out, "k": s["layer"].k, "v": s["layer"].v}


def _run_step(s):
    kv.kv_cache_write(s["ex"], s["layer"], s["batch"], s["k"], s["v"])
    if s["mode"]:
        kv.paged_attention_gated(s["ex"], s["layer"], s["batch"], s["q"], s["gate"], s["out"], s["hq"], hadamard64=s["mode"] == 2)
    else:
        kv.paged_attention(s["ex"], s["layer"], s["batch"], s["q"], s["out"], s["hq"])
    return _outputs(s, s["out"])


def _run_step_bf16(s):
    kv.kv_cache_write_bf16(s["ex"], s["layer"], s["batch"], s["k"], s["v"])
    kv.paged_attention_bf16kv(s["ex"], s["layer"], s["batch"], s["q"], s["out"], s["hq"])
    return _outputs(s, s["out"])


def _prepare_host(case, seed):
    ctx, new = _lens(case)
    hq, hkv = case["q_heads"], case["kv_heads"]
    wl = synth.PagedWorkload(ctx, new, hkv, seed=seed, formats=FORMATS[case["kv"]])
    wl.fill_context(kv.Executor(), seed)
    step_ = kv.DecodeStep(wl.layer, wl.seqs, hq)
    k, v = synth.make_kv(len(ctx), hkv, seed + 17)
    step_.k_host.copy_(k)
    step_.v_host.copy_(v)
    step_.q_host.copy_(synth.make_q(len(ctx), hq, seed + 17))
    return {"run": _run_host, "wl": wl, "layer": wl.layer, "step": step_, "new": new}


def _run_host(s):
    return _outputs(s, s["step"].run(s["new"], SM_SCALE, graph=True))


def _prepare_append(case, seed):
    n, hkv = case["tokens"], case["kv_heads"]
    lens = [n - n // 2, n // 2 - n // 8, n // 8]
    wl = synth.PagedWorkload([0, 0, 0], lens, hkv, seed=seed, formats=FORMATS[case["kv"]])
    k, v = synth.make_kv(n, hkv, seed + 17, device="cuda")
    # rows [q and gate of every q head | k | v], as a projection writes them
    off = case["q_heads"] * 2 * D
    packed = torch.zeros(n, off + 2 * hkv * D, dtype=torch.float16, device="cuda")
    packed[:, off:off + hkv * D] = k
    packed[:, off + hkv * D:] = v
    gen = torch.Generator(device="cuda")
    gen.manual_seed(seed + 5)
    norm_w = (torch.randn(D, generator=gen, device="cuda") * 0.2).to(torch.float16)
    pos = torch.cat([torch.arange(x, dtype=torch.int32) for x in lens])
    return {"run": _run_append_producer if case["producer"] else _run_append, "wl": wl, "layer": wl.layer, "ex": kv.Executor(1 << 20),
            "batch": wl.step(sm_scale=SM_SCALE), "k": packed[:, off:off + hkv * D], "v": packed[:, off + hkv * D:], "norm_w": norm_w,
            "pos": torch.stack([pos, pos, pos]).contiguous().cuda(), "tokens": n}


def _run_append(s):
    kv.kv_cache_write(s["ex"], s["layer"], s["batch"], s["k"], s["v"])
    return {"k": s["layer"].k, "v": s["layer"].v}


def _run_append_producer(s):
    k, v = s["k"], s["v"]
    rc = ffi.kernels().warp34_fused_k_rmsnorm_rope_kv_cache_write_f16(
        C.byref(s["ex"].ex), C.byref(s["layer"].layout), C.byref(s["batch"].desc), k.data_ptr(), v.data_ptr(), s["norm_w"].data_ptr(),
        s["pos"].data_ptr(), s["tokens"], ROTARY, *SECTIONS, k.stride(0), v.stride(0), THETA, EPS)
    if rc != 0:
        raise RuntimeError(f"warp34_fused_k_rmsnorm_rope_kv_cache_write_f16: {rc}")
    return {"k": s["layer"].k, "v": s["layer"].v}


def _prepare_sparse(case, seed):
    n, groups, hq, hkv = case["tokens"], case["groups"], case["q_heads"], case["kv_heads"]
    ctx = [case["ctx"] + 5 * t for t in range(n)]
    wl = synth.PagedWorkload(ctx, [0] * n, hkv, seed=seed, formats=FORMATS[case["kv"]])
    ex = kv.Executor()
    wl.fill_context(ex, seed)
    rng = np.random.default_rng(seed)
    phys, logical = np.full((n, groups), -1, np.int32), np.zeros((n, groups), np.int32)
    for t, c in enumerate(ctx):      # the token's own group and a random choice of the others
        own = (c - 1) // 4
        pick = np.concatenate([[own], rng.choice(own, groups - 1, replace=False)])
        logical[t] = pick
        phys[t] = np.asarray(wl.seqs[t].pages, np.int64)[pick // 4] * 4 + pick % 4
    q = synth.make_q(n, hq, seed + 17, device="cuda")
    lists = [torch.from_numpy(a).cuda() for a in (phys, logical, np.full(n, groups, np.int32), np.asarray(ctx, np.int32) - 1)]
    return {"run": _run_sparse, "wl": wl, "layer": wl.layer, "ex": ex, "q": q, "gate": synth.make_q(n, hq, seed + 18, device="cuda"),
            "lists": lists, "out": torch.zeros_like(q), "hq": hq, "groups": groups, "mode": case["gate"]}


def _run_sparse(s):
    lib = ffi.kernels()
    fn = lib.warp34_qsa_sparse_paged_attn_hadamard_f16 if s["mode"] == 2 else lib.warp34_qsa_sparse_paged_attn_f16
    rc = fn(C.byref(s["ex"].ex), s["q"].data_ptr(), s["gate"].data_ptr() if s["mode"] else None, C.byref(s["layer"].layout),
            *(t.data_ptr() for t in s["lists"]), None, s["out"].data_ptr(), s["q"].shape[0], s["hq"], s["groups"], SM_SCALE)
    if rc != 0:
        raise RuntimeError(f"warp34_qsa_sparse_paged_attn: {rc}")
    return s["out"]


def work(case):
    """Bytes: the cached rows that are read and the rows that are written, the new K and V rows, queries, gate and
    output once.  Operations: two products per query row, visible key and channel."""
    hq, hkv, row = case["q_heads"], case["kv_heads"], 2 * case["kv_heads"] * ROW_BYTES[case["kv"]]
    if case["kind"] == "append":
        n = case["tokens"]
        return {"bytes": n * (2 * hkv * D * 2 + row), "flops": n * 2 * hkv * D * 8 * 2}     # the 256-point rotation
    if case["kind"] == "sparse":
        keys = case["tokens"] * case["groups"] * 4
        io = case["tokens"] * hq * D * 2 * (3 if case["gate"] else 2)
        return {"bytes": keys * row + io + 8 * case["tokens"] * case["groups"], "flops": 4 * hq * D * keys}
    ctx, new = _lens(case)
    cached = sum(c + n for c, n in zip(ctx, new))
    pairs = sum(n * c + n * (n + 1) // 2 for c, n in zip(ctx, new))
    io = sum(new) * (hq * D * 2 * (3 if case.get("gate") else 2) + 2 * hkv * D * 2 + row)
    return {"bytes": cached * row + io + 4 * cached // 16, "flops": 4 * hq * D * pairs}


def tolerance(case):
    """Packed rows are the same bytes.  Attention outputs are 16-bit: two correct implementations differ by their last
    rounding and, on channels where large values cancel, by a little more."""
    if case["kind"] == "append":
        return "exact"
    return {"rel": 5e-3, "max": 3e-2} if case["kv"] == "bf16" else {"rel": 1e-3, "max": 1e-2}
