"""Decode items of at most four query rows share an MMA between values and residuals: one to four rows, several tokens on few heads,
contexts around the two-page step, windows, masked tokens, query-sparse lists and a request with more tokens than the batch
declares, against the fp32 dequant-then-attend path."""
import ctypes as C

import pytest

from util import plain_parity

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


def _workload(hkv, ctx, new):
    from warp34_b200 import ffi, kv, synth
    f, tr = ffi.KV_FORMAT_TQ4, ffi.KV_TRANSFORM_RADEMACHER_WHT256
    wl = synth.PagedWorkload(ctx, new, hkv, seed=11, formats=(f, f, tr, tr))
    ex = kv.Executor(32 << 20)
    wl.fill_context(ex, 11)
    n = sum(new)
    if n:
        k, v = synth.make_kv(n, hkv, 12, device="cuda")
        kv.kv_cache_write(ex, wl.layer, wl.step(), k, v)
    return wl, ex


def _both(ex, call):
    from warp34_b200 import ffi
    outs, status = [], None
    for flags in (0, ffi.EXEC_FLAG_PRECISE_ATTENTION):
        ex.ex.flags = flags
        outs.append(call())
        torch.cuda.synchronize()
        if status is None:
            status = int(ex.scratch[:4].view(torch.int32).item())
    ex.ex.flags = 0
    return outs, status


@pytest.mark.parametrize("hq,hkv,ctx,new,kw", [
    (1, 1, [0, 14, 15, 16, 31, 32, 33, 700], [1] * 8, {}),
    (2, 1, [5, 40, 3000], [2, 1, 2], {}),
    (6, 2, [17, 47, 48, 1000], [1] * 4, {}),                                   # three heads
    (16, 4, [31, 63, 64, 2500, 9000], [1] * 5, {"drop": 2}),
    (4, 4, [100, 3], [4, 3], {}),                                              # one head, four tokens: causal rows of one item
    (8, 2, [300, 90], [1, 1], {"sliding_window": 70}),
])
def test_up_to_four_rows_match_dequant_then_attend(native_libs, hq, hkv, ctx, new, kw):
    import numpy as np
    from warp34_b200 import kv, synth
    wl, ex = _workload(hkv, ctx, new)
    n, kw = sum(new), dict(kw)
    vtm = np.ones(n, np.uint8)
    drop = kw.pop("drop", None)
    if drop is not None:
        vtm[drop] = 0
    b = wl.step(valid_token_mask=vtm, **kw)
    q = synth.make_q(n, hq, 13, device="cuda")

    def call():
        out = torch.full((n, hq, 256), -7.0, dtype=torch.float16, device="cuda")
        kv.paged_attention(ex, wl.layer, b, q, out, hq)
        return out
    (got, want), status = _both(ex, call)
    assert status == 0
    ok, msg = plain_parity(got.float().cpu().numpy(), want.float().cpu().numpy())
    assert ok, msg


def test_four_row_lists_match_the_fp32_kernel(native_libs):
    import numpy as np
    from warp34_b200 import ffi, synth
    n, hq, hkv, groups = 5, 8, 2, 37
    ctx = [150 + 61 * t for t in range(n)]
    wl, ex = _workload(hkv, ctx, [0] * n)
    rng = np.random.default_rng(3)
    phys, logical = np.full((n, groups), -1, np.int32), np.zeros((n, groups), np.int32)
    for t, c in enumerate(ctx):
        pick = rng.choice((c + 3) // 4, min(groups, (c + 3) // 4), replace=False)
        logical[t, :len(pick)] = pick
        phys[t, :len(pick)] = np.asarray(wl.seqs[t].pages, np.int64)[pick // 4] * 4 + pick % 4
        phys[t, 3] = -1
    dev = [torch.from_numpy(a).cuda() for a in (phys, logical, np.full(n, groups, np.int32), np.asarray(ctx, np.int32) - 1)]
    q = synth.make_q(n, hq, 13, device="cuda")

    def call():
        out = torch.zeros(n, hq, 256, dtype=torch.float16, device="cuda")
        rc = ffi.kernels().warp34_qsa_sparse_paged_attn_f16(C.byref(ex.ex), q.data_ptr(), None, C.byref(wl.layer.layout), *(t.data_ptr() for t in dev),
                                                            None, out.data_ptr(), n, hq, groups, 1.0 / 16.0)
        assert rc == 0
        return out
    (got, want), status = _both(ex, call)
    assert status == 0
    ok, msg = plain_parity(got.float().cpu().numpy(), want.float().cpu().numpy())
    assert ok, msg


@pytest.mark.parametrize("hq,new,declared,served,status_bit", [
    (4, [2, 1], 1, [2, 1], 0),
    (4, [2, 0], 1, [2, 0], 0),
    (4, [1, 2, 0, 1], 1, [1, 2, 0, 1], 0),
    (2, [4, 0, 0, 0], 1, [4, 0, 0, 0], 0),
    (1, [5, 1, 0], 2, [5, 1, 0], 0),
    (4, [2, 0], 0, [2, 0], 0),              # an undeclared length counts as one token
    (4, [3, 0, 0], 1, [2, 0, 0], 4),        # twelve rows: an item holds eight, the rest is left alone
])
def test_more_tokens_than_declared(native_libs, hq, new, declared, served, status_bit):
    """Requests of more tokens than the batch declares, up to eight query rows per kv head: answered in full, whatever the other requests
    of the batch hold."""
    import numpy as np
    from warp34_b200 import kv, synth
    wl, ex = _workload(1, [60 + 30 * r for r in range(len(new))], new)
    n = sum(new)
    b = wl.step(max_q_len=declared)
    q = synth.make_q(n, hq, 13, device="cuda")

    def call():
        out = torch.full((n, hq, 256), -7.0, dtype=torch.float16, device="cuda")
        kv.paged_attention(ex, wl.layer, b, q, out, hq)
        return out
    (got, want), status = _both(ex, call)
    assert status == status_bit
    keep = np.concatenate([np.arange(t) < s for t, s in zip(new, served)])
    got, want = got.float().cpu().numpy(), want.float().cpu().numpy()
    ok, msg = plain_parity(got[keep], want[keep])
    assert ok, msg
    assert (got[~keep] == -7.0).all()
