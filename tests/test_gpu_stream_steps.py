"""The exact streaming path at the edges of its split: one- and two-page steps, items that end inside a step, shares that cross
items, workers without work, and neighbouring workers whose states are merged before they are written; against the fp32
dequant-then-attend entry point on the same pool."""
import pytest

from util import plain_parity

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def env(native_libs):
    assert torch.cuda.is_available(), "GPU tests need a CUDA device"
    from warp34_b200 import kv, synth
    return dict(kv=kv, synth=synth, ex=kv.Executor(64 << 20))


@pytest.mark.parametrize("hq,hkv,ctx,new", [
    (4, 1, [0], [1]),                                   # one key
    (6, 1, [15, 16, 31, 32, 47], [1] * 5),              # 1, 2, 2, 3, 3 pages
    (24, 4, [16 * n for n in range(1, 40)], [1] * 39),  # odd and even page counts, shares across items
    (24, 4, [3000, 10, 900], [4, 2, 3]),                # 24 rows: the tcgen05 stream kernel (one-warp items of such steps: below)
    (6, 1, [38000], [1]),                               # one item over every worker: two units and a remainder each
    (12, 2, [20000, 77, 31000], [1, 1, 1]),             # neighbours hold one item, a CTA with three
])
def test_decode_and_draft_batches_at_split_edges(env, hq, hkv, ctx, new):
    kv, synth = env["kv"], env["synth"]
    wl = synth.PagedWorkload(ctx, new, hkv, seed=5, fill=0x7F)
    wl.fill_context(env["ex"], 5)
    n = sum(new)
    k, v = synth.make_kv(n, hkv, 6, device="cuda")
    q = synth.make_q(n, hq, 6, device="cuda")
    b = wl.step()
    kv.kv_cache_write(env["ex"], wl.layer, b, k, v)
    out, want = torch.zeros_like(q), torch.zeros_like(q)
    env["ex"].scratch.fill_(0xA5)                       # nothing an earlier call left is read
    kv.paged_attention(env["ex"], wl.layer, b, q, out, hq)
    torch.cuda.synchronize()
    assert int(env["ex"].scratch[:4].view(torch.int32).item()) == 0
    kv.paged_attention(env["ex"], wl.layer, b, q, want, hq, scalar=True)
    torch.cuda.synchronize()
    ok, msg = plain_parity(out.float().cpu().numpy(), want.float().cpu().numpy())
    assert ok, msg


@pytest.mark.parametrize("hq,hkv,ctx,new", [
    (24, 4, [3000, 10, 900], [4, 2, 3]),                # three row groups per request, a short one between
    (24, 4, [38000], [4]),                              # three groups of one request over every worker: shares that cross groups
    (12, 1, [16 * n for n in range(1, 60)], [2] * 59),  # 24 rows, odd and even page counts
    (9, 1, [700, 333], [1, 2]),                         # 9 and 18 rows: a last group of one and of two
])
def test_several_row_groups_per_request(env, hq, hkv, ctx, new):
    """Steps of 9 to 24 rows, which the dispatch gives to the tcgen05 stream kernel, as 8-row items of the one-warp kernel: by the
    test selector, and because the workspace has no room for the other's items."""
    import ctypes as C
    from warp34_b200 import ffi
    kv, synth = env["kv"], env["synth"]
    wl = synth.PagedWorkload(ctx, new, hkv, seed=5, fill=0x7F)
    wl.fill_context(env["ex"], 5)
    n = sum(new)
    k, v = synth.make_kv(n, hkv, 6, device="cuda")
    q = synth.make_q(n, hq, 6, device="cuda")
    b = wl.step()
    kv.kv_cache_write(env["ex"], wl.layer, b, k, v)
    want, out = torch.zeros_like(q), torch.zeros_like(q)
    kv.paged_attention(env["ex"], wl.layer, b, q, want, hq, scalar=True)
    env["ex"].scratch.fill_(0xA5)
    rc = ffi.kernels().warp34_paged_attention_f16_force_kernel_for_test(C.byref(env["ex"].ex), C.byref(wl.layer.layout), C.byref(b.desc),
                                                                       q.data_ptr(), out.data_ptr(), hq, 0)
    torch.cuda.synchronize()
    status, items = env["ex"].scratch[:8].view(torch.int32).tolist()      # the plan's header
    assert rc == 0 and status == 0
    assert items == hkv * sum(-(-m * (hq // hkv) // 8) for m in new)
    ok, msg = plain_parity(out.float().cpu().numpy(), want.float().cpu().numpy())
    assert ok, msg
    small, out = kv.Executor(2 << 20), torch.zeros_like(q)
    kv.paged_attention(small, wl.layer, b, q, out, hq)
    torch.cuda.synchronize()
    assert int(small.scratch[:4].view(torch.int32).item()) == 0
    ok, msg = plain_parity(out.float().cpu().numpy(), want.float().cpu().numpy())
    assert ok, msg
