"""Steps of 9 to 24 query rows per request and kv head on the tensor-memory streaming kernel: row counts around its tile sizes,
blocks of 128 keys that end early, shares that cross requests, windows, masks, the row-triple output, and an unknown sequence
limit; against the fp32 dequant-then-attend entry point on the same pool."""
import numpy as np
import pytest

from util import plain_parity

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def env(native_libs):
    assert torch.cuda.is_available(), "GPU tests need a CUDA device"
    from warp34_b200 import kv, synth
    return dict(kv=kv, synth=synth, ex=kv.Executor(64 << 20))


def _setup(env, hq, hkv, ctx, new, **kw):
    wl = env["synth"].PagedWorkload(ctx, new, hkv, seed=5, fill=0x7F)
    wl.fill_context(env["ex"], 5)
    n = sum(new)
    k, v = env["synth"].make_kv(n, hkv, 6, device="cuda")
    b = wl.step(**kw)
    env["kv"].kv_cache_write(env["ex"], wl.layer, b, k, v)
    q = env["synth"].make_q(n, hq, 6, device="cuda")
    want = torch.zeros_like(q)
    env["kv"].paged_attention(env["ex"], wl.layer, b, q, want, hq, scalar=True)
    env["ex"].scratch.fill_(0xA5)                       # nothing an earlier call left is read
    return wl, b, q, want


def _check(env, out, want):
    torch.cuda.synchronize()
    assert int(env["ex"].scratch[:4].view(torch.int32).item()) == 0
    ok, msg = plain_parity(out.float().cpu().numpy(), want.float().cpu().numpy())
    assert ok, msg


@pytest.mark.parametrize("hq,hkv,ctx,new,kw", [
    (9, 1, [125], [1], {}),                                            # 9 rows of 16; one block of keys, cut short
    (8, 2, [126, 127, 128, 129], [4] * 4, {}),                         # 16 rows; a block, and one key more
    (17, 1, [255, 257], [1, 1], {}),                                   # 17 rows of 24
    (24, 4, [3000, 10, 900], [4, 2, 3], {}),                           # fewer rows than the longest request has
    (24, 4, [16 * n for n in range(1, 40)], [4] * 39, {}),             # shares across items and requests
    (6, 1, [40000], [4], {}),                                          # one item over every worker
    (24, 4, [20000, 77, 31000], [2, 2, 1], {}),
    (8, 1, [300, 1000], [3, 3], {"sliding_window": 70}),               # keys from the middle of a block on
    (8, 2, [400, 90], [2, 2], {"mask_mode": 1, "sliding_window": 33}),
])
def test_parity(env, hq, hkv, ctx, new, kw):
    wl, b, q, want = _setup(env, hq, hkv, ctx, new, **kw)
    out = torch.zeros_like(q)
    env["kv"].paged_attention(env["ex"], wl.layer, b, q, out, hq)
    _check(env, out, want)


def test_unknown_sequence_limit(env):
    wl, b, q, want = _setup(env, 8, 2, [900, 500], [2, 2])
    b.desc.max_seq_len = 0                              # the limit is optional
    out = torch.zeros_like(q)
    env["kv"].paged_attention(env["ex"], wl.layer, b, q, out, 8)
    _check(env, out, want)


@pytest.mark.parametrize("gated", [False, True])
def test_masks_and_gate(env, gated):
    new = [3, 4, 2]
    vtm = np.ones(sum(new), np.uint8)
    vtm[[0, 4]] = 0
    wl, b, q, want = _setup(env, 24, 4, [700, 1500, 300], new, valid_token_mask=vtm, valid_req_mask=np.array([1, 1, 0], np.uint8))
    out = torch.full_like(q, 7.0)
    if gated:
        gate = env["synth"].make_q(sum(new), 24, 9, device="cuda")
        env["kv"].paged_attention_gated(env["ex"], wl.layer, b, q, gate, out, 24)
        want = (want.float() * torch.sigmoid(gate.float())).to(q.dtype)
    else:
        env["kv"].paged_attention(env["ex"], wl.layer, b, q, out, 24)
    live = torch.as_tensor((vtm != 0) & (np.arange(sum(new)) < 7), device="cuda")
    assert bool((out[~live] == 7.0).all())              # masked rows stay as they were
    _check(env, out[live], want[live])


def test_row_triples(env):
    wl, b, q, want = _setup(env, 16, 4, [130, 2000, 4097], [4, 3, 4])
    triples = torch.full((q.shape[0], 16, 258), float("nan"), device="cuda")
    env["kv"].paged_attention_partial(env["ex"], wl.layer, b, q, triples, 16)
    assert bool((triples[..., 257] > 0).all()) and bool(torch.isfinite(triples).all())
    out = torch.zeros_like(q)
    env["kv"].paged_attention(env["ex"], wl.layer, b, q, out, 16)
    _check(env, out, want)


@pytest.mark.parametrize("hq,hkv,exps", [(24, 4, (-10, -10)), (16, 4, (-13, -13)), (24, 4, (-13, 3)), (24, 4, (6, -9))])
def test_accuracy_does_not_depend_on_the_magnitude_of_v(env, hq, hkv, exps):
    """V times 2^b: the stored codes are the same and every scale is the same but for a power of two, so the outputs are those of
    magnitude 1 times 2^b.  At magnitude 1 about 1 % of them are not the float64 result's nearest fp16 value: at most twice that
    many differ.  Two exponents: the second one for the tokens from 700 on, and the comparison is with the fp32 kernel."""
    kv, synth = env["kv"], env["synth"]
    ctx, new = [2000, 600, 1300], [4, 4, 3]
    n, outs, ones = sum(new), {}, (0, 0)
    for e in (ones, exps):
        wl = synth.PagedWorkload([0] * 3, [c + m for c, m in zip(ctx, new)], hkv, seed=5, fill=0x7F)
        k, v = synth.make_kv(sum(ctx) + n, hkv, 6, device="cuda")
        tok = torch.cat([torch.arange(c + m) for c, m in zip(ctx, new)]).cuda()
        v = (v.float() * 16).round() / 16 * torch.where(tok < 700, 2.0 ** e[0], 2.0 ** e[1])[:, None]
        kv.kv_cache_write(env["ex"], wl.layer, wl.step(), k, v.half())
        for s, c in zip(wl.seqs, ctx):
            s.commit(c)
        b = wl.step(q_lens=new)
        q = synth.make_q(n, hq, 6, device="cuda")
        out, want = torch.zeros_like(q), torch.zeros_like(q)
        env["ex"].scratch.fill_(0xA5)
        kv.paged_attention(env["ex"], wl.layer, b, q, out, hq)
        kv.paged_attention(env["ex"], wl.layer, b, q, want, hq, scalar=True)
        _check(env, out, want)
        outs[e] = out.float()
    if exps[0] == exps[1]:
        base, got = outs[ones], outs[exps] * 2.0 ** -exps[0]
        normal = base.abs() >= 2.0 ** (-13 - exps[0])           # fp16 has all its bits on both sides
        assert float((got != base)[normal].float().mean()) <= 0.02
