"""Batches over 8-bit layers that mix decode rows with prompt chunks: the stream kernel serves the short requests and the CTA-pair
kernel the others; against the fp32 dequant-then-attend entry point on the same pool.  Which kernel took what is read from the plan
header that the stream kernel's plan leaves at the start of the workspace (status, items, units, units per worker)."""
import numpy as np
import pytest

from util import plain_parity

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def env(native_libs):
    assert torch.cuda.is_available(), "GPU tests need a CUDA device"
    from warp34_b200 import ffi, kv, synth
    return dict(ffi=ffi, kv=kv, synth=synth)


@pytest.mark.parametrize("fmt", ["FP8_E4M3", "Q8_0"])
@pytest.mark.parametrize("ctx,new,kw,gate,stream_items", [
    ([3000] * 40 + [100], [1] * 40 + [130], {}, 0, 4 * 40),                             # decode rows beside one chunk
    ([40] + [2500] * 30 + [700], [64] + [1, 4, 2] * 10 + [200], {}, 2, 4 * 10 * (1 + 3 + 2)),
    ([3000] * 30 + [0], [1] * 30 + [257], {"drop": True, "sliding_window": 900}, 1, 4 * 29),
    ([100] * 64, [5] * 64, {}, 0, 4 * 64 * 4),                                          # many requests of 30 rows: all of them
    ([0, 300], [500, 129], {}, 0, None),                                                # chunks only
])
def test_each_request_goes_to_the_kernel_that_is_faster_for_it(env, fmt, ctx, new, kw, gate, stream_items):
    ffi, kv, synth = env["ffi"], env["kv"], env["synth"]
    f, tr = getattr(ffi, "KV_FORMAT_" + fmt), ffi.KV_TRANSFORM_IDENTITY
    hq, hkv, n = 24, 4, sum(new)
    wl = synth.PagedWorkload(ctx, new, hkv, seed=11, fill=0x7F, formats=(f, f, tr, tr))
    ex = kv.Executor(64 << 20)
    wl.fill_context(ex, 11)
    k, v = synth.make_kv(n, hkv, 12, device="cuda")
    kv.kv_cache_write(ex, wl.layer, wl.step(), k, v)
    q, g = synth.make_q(n, hq, 12, device="cuda"), synth.make_q(n, hq, 13, device="cuda")
    kw = dict(kw)
    live = np.ones(n, bool)
    if kw.pop("drop", False):       # a masked decode request, a masked token of the chunk
        kw["valid_req_mask"] = np.array([0] + [1] * (len(ctx) - 1), np.uint8)
        kw["valid_token_mask"] = np.ones(n, np.uint8)
        kw["valid_token_mask"][n - 3] = 0
        live[[0, n - 3]] = False
    b = wl.step(**kw)
    ex.scratch.fill_(0xA5)
    out, want = (torch.full((n, hq, 256), -7.0, dtype=torch.float16, device="cuda") for _ in range(2))
    if gate:
        kv.paged_attention_gated(ex, wl.layer, b, q, g, out, hq, hadamard64=gate == 2)
    else:
        kv.paged_attention(ex, wl.layer, b, q, out, hq)
    torch.cuda.synchronize()
    status, items = ex.scratch[:8].view(torch.int32).tolist()
    assert status == 0
    if stream_items is not None:
        assert items == stream_items
    kv.paged_attention(ex, wl.layer, b, q, want, hq, scalar=True)
    torch.cuda.synchronize()
    if gate:       # the two steps on their own, on the reference output
        fn = getattr(ffi.kernels(), "warp34_apply_attn_output_gate_hadamard_f16" if gate == 2 else "warp34_apply_attn_output_gate_f16")
        import ctypes as C
        assert fn(C.byref(ex.ex), want.data_ptr(), g.data_ptr(), want.data_ptr(), b.desc.valid_token_mask or None, n, hq * 256) == 0
        torch.cuda.synchronize()
    live = torch.as_tensor(live, device="cuda")
    assert (out[~live] == -7.0).all()
    a, w = out[live].float().cpu().numpy(), want[live].float().cpu().numpy()
    if gate == 2:      # an output mixes 64 gated values: the bound of their sum
        tol = (2e-3 + 1e-2 * np.abs(w)).reshape(-1, 64).sum(1, keepdims=True) / 8
        assert (np.abs(a - w).reshape(-1, 64) <= tol).all()
    else:
        ok, msg = plain_parity(a, w)
        assert ok, msg


@pytest.mark.parametrize("scratch", [256, 8 << 20])
def test_small_workspaces(env, scratch):
    """Without room for the stream kernel's partials the pair kernel serves every request."""
    ffi, kv, synth = env["ffi"], env["kv"], env["synth"]
    f, tr = ffi.KV_FORMAT_FP8_E4M3, ffi.KV_TRANSFORM_IDENTITY
    ctx, new = [900] * 20 + [50], [1] * 20 + [90]
    wl = synth.PagedWorkload(ctx, new, 4, seed=3, fill=0x7F, formats=(f, f, tr, tr))
    wl.fill_context(kv.Executor(1 << 20), 3)
    n = sum(new)
    k, v = synth.make_kv(n, 4, 4, device="cuda")
    q = synth.make_q(n, 24, 4, device="cuda")
    ex = kv.Executor(scratch)
    b = wl.step()
    kv.kv_cache_write(ex, wl.layer, b, k, v)
    out, want = torch.zeros_like(q), torch.zeros_like(q)
    kv.paged_attention(ex, wl.layer, b, q, out, 24)
    kv.paged_attention(ex, wl.layer, b, q, want, 24, scalar=True)
    torch.cuda.synchronize()
    ok, msg = plain_parity(out.float().cpu().numpy(), want.float().cpu().numpy())
    assert ok, msg
