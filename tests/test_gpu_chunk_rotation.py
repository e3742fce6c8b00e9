"""The chunk kernel rotates its query rows and its outputs in groups of four: groups that end inside a tile, head groups that do not
divide four, masked tokens inside a group, rows off a 16-byte boundary, with and without the output gate, and bf16 activations (which
have no gated entry point), against the fp32 dequant-then-attend path of the same entry point."""
import ctypes as C

import pytest

from util import plain_parity

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("hq,hkv,new,off,mode,drop", [
    (1, 1, [25], 0, 0, ()),                     # 25 rows: the last group has one
    (3, 1, [43, 9], 0, 1, (0, 2, 50)),          # 129 rows: one row of the second CTA; masked tokens inside groups
    (6, 1, [5, 64], 0, 2, ()),                  # 30 rows, and 384: the second tile ends at its 128th row
    (10, 2, [51, 52], 4, 1, (3,)),              # 5 heads, rows 8 bytes off a 16-byte boundary
    (12, 2, [43], 4, 2, ()),
])
def test_row_groups_match_dequant_then_attend(native_libs, hq, hkv, new, off, mode, drop):
    import numpy as np
    from warp34_b200 import ffi, kv, synth
    f, tr = ffi.KV_FORMAT_TQ4, ffi.KV_TRANSFORM_RADEMACHER_WHT256
    wl = synth.PagedWorkload([70] * len(new), new, hkv, seed=3, formats=(f, f, tr, tr))
    ex = kv.Executor(64 << 20)
    wl.fill_context(ex, 3)
    n = sum(new)
    k, v = synth.make_kv(n, hkv, 4, device="cuda")
    kv.kv_cache_write(ex, wl.layer, wl.step(), k, v)
    vtm = np.ones(n, np.uint8)
    vtm[list(drop)] = 0
    b = wl.step(valid_token_mask=vtm)

    def shifted(t):
        store = torch.zeros(t.numel() + 8, dtype=t.dtype, device="cuda")
        store[off:off + t.numel()] = t.reshape(-1)
        return store[off:off + t.numel()].view(n, hq, 256)

    q, gate = shifted(synth.make_q(n, hq, 5, device="cuda")), shifted(synth.make_q(n, hq, 6, device="cuda"))
    outs = []
    for flags in (0, ffi.EXEC_FLAG_PRECISE_ATTENTION):
        ex.ex.flags = flags
        out = shifted(torch.full((n, hq, 256), -7.0, dtype=torch.float16, device="cuda"))
        if mode:
            kv.paged_attention_gated(ex, wl.layer, b, q, gate, out, hq, hadamard64=mode == 2)
        else:
            kv.paged_attention(ex, wl.layer, b, q, out, hq)
        torch.cuda.synchronize()
        outs.append(out.float().cpu().numpy())
    keep = vtm.astype(bool)
    assert (outs[0][~keep] == -7.0).all()
    got, want = outs[0][keep], outs[1][keep]
    if mode == 2:      # an output mixes 64 gated values, each within its own bound: compared before the mixing
        h = torch.ones(1, 1)
        for _ in range(6):
            h = torch.cat([torch.cat([h, h], 1), torch.cat([h, -h], 1)], 0)
        got, want = ((x.reshape(-1, 64) @ (h / 8).numpy()) for x in (got, want))
    ok, msg = plain_parity(got, want)
    assert ok, msg


@pytest.mark.parametrize("hq,hkv,new,off,drop", [(3, 1, [43, 9], 0, (0, 2, 50)), (6, 1, [5, 64], 4, ()), (10, 2, [51, 52], 1, (3,))])
def test_bf16_row_groups_match_dequant_then_attend(native_libs, hq, hkv, new, off, drop):
    """Both outputs are rounded to bf16: 2^-9 of the value each, on top of the plain bound."""
    import numpy as np
    from util import ATOL, RTOL
    from warp34_b200 import ffi, kv, synth
    wl = synth.PagedWorkload([70] * len(new), new, hkv, seed=3)
    ex = kv.Executor(64 << 20)
    wl.fill_context(ex, 3)
    n = sum(new)
    k, v = synth.make_kv(n, hkv, 4, device="cuda")
    kv.kv_cache_write(ex, wl.layer, wl.step(), k, v)
    vtm = np.ones(n, np.uint8)
    vtm[list(drop)] = 0
    b = wl.step(valid_token_mask=vtm)

    def shifted(t):
        store = torch.zeros(t.numel() + 8, dtype=torch.bfloat16, device="cuda")
        store[off:off + t.numel()] = t.reshape(-1).to(torch.bfloat16)
        return store[off:off + t.numel()].view(n, hq, 256)

    q, outs = shifted(synth.make_q(n, hq, 5, device="cuda")), []
    for flags in (0, ffi.EXEC_FLAG_PRECISE_ATTENTION):
        ex.ex.flags = flags
        out = shifted(torch.full((n, hq, 256), -7.0, device="cuda"))
        assert native_libs[0].warp34_tq4_paged_attention_bf16(C.byref(ex.ex), C.byref(wl.layer.layout), C.byref(b.desc), q.data_ptr(), out.data_ptr(), hq) == 0
        torch.cuda.synchronize()
        outs.append(out.float().cpu().numpy())
    keep = vtm.astype(bool)
    assert (outs[0][~keep] == -7.0).all()
    got, want = outs[0][keep], outs[1][keep]
    bound = ATOL + (RTOL + 2.0 ** -8) * np.abs(want)
    assert (np.abs(got - want) <= bound).all(), float((np.abs(got - want) / bound).max())


@pytest.mark.parametrize("reqs", [8, 9, 32, 33, 70])
def test_pairs_find_their_request_among_many(native_libs, reqs):
    """Requests of 0 to 90 tokens (0 to 3 tiles of 42): the request of a pair is searched one by one up to 8 requests and 32 at a time
    from 9 on."""
    import numpy as np
    from warp34_b200 import ffi, kv, synth
    f, tr = ffi.KV_FORMAT_TQ4, ffi.KV_TRANSFORM_RADEMACHER_WHT256
    new = [(7 * r * r + 5 * r) % 91 if r % 5 else 0 for r in range(reqs)]
    new[-1] = 90
    wl = synth.PagedWorkload([0] * reqs, new, 1, seed=3, formats=(f, f, tr, tr))
    ex = kv.Executor(64 << 20)
    n = sum(new)
    k, v = synth.make_kv(n, 1, 4, device="cuda")
    b = wl.step()
    kv.kv_cache_write(ex, wl.layer, b, k, v)
    q = synth.make_q(n, 6, 5, device="cuda")
    outs = []
    for flags in (0, ffi.EXEC_FLAG_PRECISE_ATTENTION):
        ex.ex.flags = flags
        out = torch.full((n, 6, 256), -7.0, dtype=torch.float16, device="cuda")
        kv.paged_attention(ex, wl.layer, b, q, out, 6)
        torch.cuda.synchronize()
        outs.append(out.float().cpu().numpy())
    ok, msg = plain_parity(*outs)
    assert ok, msg
