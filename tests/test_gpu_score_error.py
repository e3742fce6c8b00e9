"""What the one-warp stream kernel's operands leave of a score's error, against float64: contexts of one key, where the partial output's
m + log2 l is the score itself.

The query is held as an fp16 value and a residual in steps of 1/255 of the row's largest one; K as a centroid's fp16 value and residual.
With all rotated columns of a query row of one magnitude (a single nonzero channel) and the residual's step as the only rounding, a
score is off by at most 2^-10 / (510 sqrt(3)) = 1.1e-6 of the scores' root mean square.  Items of more than four rows leave the product of
both residuals out: it is computed here, and the error may follow it about once, not several times."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

LUT_SCALE = np.float32(0.954016)     # the centroids' common factor (tq4_attention.cu)


@pytest.mark.parametrize("hq", [24, 16])      # eight-row and four-row items
def test_scores_against_float64(native_libs, oracle_lib, hq):
    from oracle import qsa
    from warp34_b200 import kv, synth
    n, hkv, sm = 600, 4, 1.0 / 16.0
    g = torch.Generator().manual_seed(11)
    wl = synth.PagedWorkload([0] * n, [1] * n, hkv, seed=5)
    ex = kv.Executor(64 << 20)
    b = wl.step(sm_scale=sm)
    k, v = (torch.randn(n, hkv * 256, generator=g).half().cuda() for _ in range(2))
    kv.kv_cache_write(ex, wl.layer, b, k, v)
    q = torch.zeros(n, hq, 256).scatter_(2, torch.randint(0, 256, (n, hq, 1), generator=g), 8 + 8 * torch.rand(n, hq, 1, generator=g)).half()
    triples = torch.zeros(n, hq, 258, device="cuda")
    kv.paged_attention_partial(ex, wl.layer, b, q.cuda(), triples, hq)
    torch.cuda.synchronize()
    assert int(ex.scratch[:4].view(torch.int32).item()) == 0
    t = triples.cpu().numpy().astype(np.float64)
    got = t[..., 256] + np.log2(t[..., 257])

    rows = wl.layer.k.cpu().numpy().reshape(-1, hkv, 16, 132)[[s.pages[0] for s in wl.seqs], :, 0].reshape(-1, 132)
    scale = rows.reshape(-1, 2, 66)[..., :2].copy().view(np.float16).astype(np.float64)
    keys = np.stack([oracle_lib.decode_row(r) for r in rows]).astype(np.float64).reshape(n, hkv, 1, 2, 128)
    scale = scale.reshape(n, hkv, 1, 2, 1)
    rotated = np.einsum("ij,nhj->nhi", qsa._H256 * qsa.signs()[None, :], q.numpy().astype(np.float64)).reshape(n, hkv, -1, 2, 128)
    want = (rotated * keys).sum((-1, -2)) * sm * np.log2(np.e)
    err = (got.reshape(want.shape) - want).ravel()
    rel = np.sqrt((err ** 2).mean() / (want ** 2).mean())

    # the product of the residuals, in the kernel's units: Q' = q sm log2(e) / LUT_SCALE, K' = LUT_SCALE centroid
    qp = (rotated * (sm * np.log2(np.e) / LUT_SCALE)).astype(np.float32)
    below = qp.astype(np.float16)
    below = np.where(below.astype(np.float32) > qp, np.nextafter(below, np.float16(-np.inf)), below)
    centroid = LUT_SCALE * (keys / scale).astype(np.float32)
    left_out = (((qp - below.astype(np.float32)) * (centroid - centroid.astype(np.float16).astype(np.float32))).astype(np.float64) * scale).sum((-1, -2)).ravel()
    times = -(err * left_out).sum() / (left_out ** 2).sum()
    spread = np.sqrt((err ** 2).mean() / (left_out ** 2).sum())      # standard deviation of `times`
    print(f"[margin] {hq} heads: error {rel:.2e} of the scores, left-out product {np.sqrt((left_out ** 2).mean()):.1e} taken {times:.2f} +- {spread:.2f} times")
    assert rel < 2.0 ** -10 / (510 * 3 ** 0.5)
    assert spread < 0.5 and abs(times - (1.0 if hq > 16 else 0.0)) < 1.0 + 4 * spread
