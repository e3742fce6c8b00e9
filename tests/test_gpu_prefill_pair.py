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


@pytest.mark.parametrize("fmt", ["TQ4", "FP8_E4M3", "Q8_0"])
@pytest.mark.parametrize("k_exp,v_exp,where", [(-10, 0, "all"), (0, -9, "all"), (-13, 0, "all"), (6, 6, "all"), (-10, -9, "pages"),
                                               (-13, 0, "ends"), (0, -13, "ends"), (-13, -13, "ends")])
def test_accuracy_does_not_depend_on_the_magnitude_of_k_and_v(env, fmt, k_exp, v_exp, where):
    """K times 2^a under Q times 2^-a, or V times 2^b: the stored codes are the same and every scale is the same but for a power
    of two, so the outputs are those of magnitude 1 (times 2^b).  At magnitude 1 about 3 % of the outputs are not the float64
    result's nearest fp16 value (1 % for 8-bit rows), so at most twice that many may differ here (measured: 2.6 and 0.5 %).
    `pages`: only the tokens of every other page are scaled; `ends`: only the first and the last 64 tokens, all others are times 4 (the exponents that
    a tile takes from its ends do not fit the rows between): the comparison is then with the fp32 kernel."""
    ffi, kv, synth = env["ffi"], env["kv"], env["synth"]
    f = getattr(ffi, "KV_FORMAT_" + fmt)
    tr = ffi.KV_TRANSFORM_RADEMACHER_WHT256 if fmt == "TQ4" else ffi.KV_TRANSFORM_IDENTITY
    hq, hkv, ctx, new = 12, 2, [400, 77], [70, 130]
    total, n = sum(ctx) + sum(new), sum(new)
    tok = torch.cat([torch.arange(c + m) for c, m in zip(ctx, new)]).cuda()
    left = torch.cat([torch.arange(c + m).flip(0) for c, m in zip(ctx, new)]).cuda()
    scaled = {"all": tok >= 0, "pages": tok // 16 % 2 == 0, "ends": (tok < 64) | (left < 64 + 15)}[where]
    outs = {}
    for a, b in ((0, 0), (k_exp, v_exp)):
        wl = synth.PagedWorkload([0, 0], [c + m for c, m in zip(ctx, new)], hkv, seed=7, fill=0x7F, formats=(f, f, tr, tr))
        k, v = synth.make_kv(total, hkv, 9, device="cuda")
        q = synth.make_q(n, hq, 9, device="cuda").float()
        k, v = (k.float() * 16).round() / 16, (v.float() * 16).round() / 16      # eleven bits or fewer, so exact at every scale
        other = 4.0 if where == "ends" else 1.0
        k, v = (k * torch.where(scaled, 2.0 ** x, other if x else 1.0)[:, None] for k, x in ((k, a), (v, b)))
        q = (q * 2.0 ** -a if where == "all" else q).half()
        kv.kv_cache_write(env["ex"], wl.layer, wl.step(), k.half(), v.half())
        for s, c in zip(wl.seqs, ctx):
            s.commit(c)
        step = wl.step(q_lens=new)
        out = torch.zeros(n, hq, 256, dtype=torch.float16, device="cuda")
        kv.paged_attention(env["ex"], wl.layer, step, q, out, hq)
        torch.cuda.synchronize()
        assert int(env["ex"].scratch[:4].view(torch.int32).item()) == 0
        outs[(a, b)] = out.float()
        if where != "all":
            want = torch.zeros_like(out)
            kv.paged_attention(env["ex"], wl.layer, step, q, want, hq, scalar=True)
            torch.cuda.synchronize()
            ok, msg = plain_parity(out.float().cpu().numpy(), want.float().cpu().numpy())
            assert ok, msg
    if where != "all":
        return
    base, got = outs[(0, 0)], outs[(k_exp, v_exp)] * 2.0 ** -v_exp
    ok, msg = plain_parity(got.cpu().numpy(), base.cpu().numpy())
    assert ok, msg
    normal = base.abs() >= 2.0 ** (-13 - min(v_exp, 0))     # fp16 has all its bits on both sides
    differ = float((got != base)[normal].float().mean())
    assert differ <= (0.06 if fmt == "TQ4" else 0.025), differ


@pytest.mark.parametrize("ctx,new", [([300, 20], [70, 50]), ([3000], [20])])      # one range of keys; several, merged
def test_nan_rows_of_a_tq4_chunk_come_out_as_nan(env, ctx, new):
    """A query row with a NaN, and only that row, gives NaN, as the fp32 kernel's does; it is not passed off as zeros."""
    kv, synth = env["kv"], env["synth"]
    hq, hkv, n = 12, 2, sum(new)
    wl = synth.PagedWorkload(ctx, new, hkv, seed=7, fill=0x7F)
    wl.fill_context(env["ex"], 7)
    k, v = synth.make_kv(n, hkv, 9, device="cuda")
    q = synth.make_q(n, hq, 9, device="cuda")
    b = wl.step()
    kv.kv_cache_write(env["ex"], wl.layer, b, k, v)
    clean = torch.zeros_like(q)
    kv.paged_attention(env["ex"], wl.layer, b, q, clean, hq)
    q[5, 3, 100] = float("nan")
    out = torch.zeros_like(q)
    kv.paged_attention(env["ex"], wl.layer, b, q, out, hq)
    torch.cuda.synchronize()
    assert torch.isnan(out[5, 3]).all()
    out[5, 3] = clean[5, 3]
    assert torch.equal(out, clean)
