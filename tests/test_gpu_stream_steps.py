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
    (24, 4, [3000, 10, 900], [4, 2, 3]),                # several row groups per request, a short one between
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
