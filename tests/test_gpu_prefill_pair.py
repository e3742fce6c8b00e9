"""The two-CTA chunk kernel (value + residual operands on tcgen05) at the edges of its tiles: 256 query rows, 64-key
blocks, 32-key halves, 16-token pages, head groups that do not divide 256, windows and masks, for every storage format,
against the fp32 dequant-then-attend entry point on the same pool."""
import numpy as np
import pytest

from util import plain_parity

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def env(native_libs):
    assert torch.cuda.is_available(), "GPU tests need a CUDA device"
    from warp34_b200 import ffi, kv, synth
    return dict(ffi=ffi, kv=kv, synth=synth, ex=kv.Executor(64 << 20))


@pytest.mark.parametrize("fmt", ["TQ4", "FP8_E4M3", "Q8_0"])
@pytest.mark.parametrize("hq,hkv,ctx,new,kw", [
    (4, 1, [0], [7], {}),                                          # one page, 28 rows
    (4, 1, [0, 1, 15], [32, 33, 63], {}),                          # rows 128 / 132 / 252, last keys 32, 34, 78
    (4, 2, [0, 48, 63], [64, 65, 129], {}),                        # rows 256, 260, 516; keys 64, 113, 192
    (12, 2, [17, 500], [43, 42], {}),                              # 42 tokens fill a tile of 6 heads
    (10, 2, [3, 130], [51, 52], {}),                               # 5 heads: rows straddle the two CTAs
    (8, 1, [300], [100], {"sliding_window": 70}),                  # keys from the middle of a block on
    (8, 2, [40, 90], [80, 20], {"mask_mode": 1, "sliding_window": 33}),
    (32, 1, [64], [9], {"drop": 4}),                               # 32 heads, a masked token and a masked request
])
def test_chunks_at_tile_edges_match_dequant_then_attend(env, fmt, hq, hkv, ctx, new, kw):
    ffi, kv, synth = env["ffi"], env["kv"], env["synth"]
    f = getattr(ffi, "KV_FORMAT_" + fmt)
    tr = ffi.KV_TRANSFORM_RADEMACHER_WHT256 if fmt == "TQ4" else ffi.KV_TRANSFORM_IDENTITY
    if fmt != "TQ4" and hq // hkv > 8:
        pytest.skip("the fp32 kernel of these formats serves up to 8 heads per kv head")
    kw = dict(kw)
    drop = kw.pop("drop", None)
    ctx, new = ctx + ctx[:1], new + new[:1]                        # the last request is masked when `drop` says so
    wl = synth.PagedWorkload(ctx, new, hkv, seed=7, fill=0x7F, formats=(f, f, tr, tr))     # 0x7f: NaN codes as e4m3
    wl.fill_context(env["ex"], 7)
    n = sum(new)
    vtm = np.ones(n, np.uint8)
    if drop is not None:
        vtm[drop] = 0
        kw.update(valid_token_mask=vtm, valid_req_mask=np.array([1] * (len(ctx) - 1) + [0], np.uint8))
    b = wl.step(**kw)
    k, v = synth.make_kv(n, hkv, 9, device="cuda")
    q = synth.make_q(n, hq, 9, device="cuda")
    append = wl.step()
    kv.kv_cache_write(env["ex"], wl.layer, append, k, v)
    out, want = (torch.full((n, hq, 256), -7.0, dtype=torch.float16, device="cuda") for _ in range(2))
    kv.paged_attention(env["ex"], wl.layer, b, q, out, hq)
    torch.cuda.synchronize()
    assert int(env["ex"].scratch[:4].view(torch.int32).item()) == 0
    kv.paged_attention(env["ex"], wl.layer, b, q, want, hq, scalar=True)
    torch.cuda.synchronize()
    ok, msg = plain_parity(out.float().cpu().numpy(), want.float().cpu().numpy())
    assert ok, msg
    if drop is not None:
        assert (out[drop] == -7.0).all() and (out[n - new[-1]:] == -7.0).all()


@pytest.mark.parametrize("fmt", ["TQ4", "FP8_E4M3", "Q8_0"])
@pytest.mark.parametrize("hq,hkv,ctx,new,gate", [
    (4, 1, [2000], [7], 0),                            # more ranges than tiles, one row in 32 in use
    (24, 4, [700, 64, 1500], [40, 33, 50], 2),         # requests whose last ranges are empty
    (6, 2, [3000], [129], 1),
])
def test_split_chunks_equal_the_unsplit_ones(env, fmt, hq, hkv, ctx, new, gate):
    """Few tiles after a long context: the keys are cut into ranges whose states are merged.  Without a workspace there is one
    range; both meet the bound, with the output epilogue applied to the merged rows."""
    ffi, kv, synth = env["ffi"], env["kv"], env["synth"]
    f = getattr(ffi, "KV_FORMAT_" + fmt)
    tr = ffi.KV_TRANSFORM_RADEMACHER_WHT256 if fmt == "TQ4" else ffi.KV_TRANSFORM_IDENTITY
    wl = synth.PagedWorkload(ctx, new, hkv, seed=3, fill=0x7F, formats=(f, f, tr, tr))
    wl.fill_context(env["ex"], 3)
    n = sum(new)
    k, v = synth.make_kv(n, hkv, 4, device="cuda")
    q, g = synth.make_q(n, hq, 4, device="cuda"), synth.make_q(n, hq, 5, device="cuda")
    vtm = np.ones(n, np.uint8)
    vtm[1] = 0
    b = wl.step(valid_token_mask=vtm)
    kv.kv_cache_write(env["ex"], wl.layer, wl.step(), k, v)
    outs = []
    for ex in (env["ex"], kv.Executor(256)):
        out = torch.full((n, hq, 256), -7.0, dtype=torch.float16, device="cuda")
        if gate:
            kv.paged_attention_gated(ex, wl.layer, b, q, g, out, hq, hadamard64=gate == 2)
        else:
            kv.paged_attention(ex, wl.layer, b, q, out, hq)
        torch.cuda.synchronize()
        assert (out[1] == -7.0).all()
        outs.append(out.float().cpu().numpy())
    ok, msg = plain_parity(outs[0], outs[1])
    assert ok, msg
    if not gate:
        want = torch.full((n, hq, 256), -7.0, dtype=torch.float16, device="cuda")
        kv.paged_attention(env["ex"], wl.layer, b, q, want, hq, scalar=True)
        torch.cuda.synchronize()
        ok, msg = plain_parity(outs[0], want.float().cpu().numpy())
        assert ok, msg
