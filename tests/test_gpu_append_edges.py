"""TQ4 append at the edges of its layout (rows off 16-byte boundaries, rows whose destination is 2-byte aligned, one to nine
heads, fewer rows than a warp takes, NaN, infinity, zeros, values at the fp16 limits) against the CPU oracle: the same codes,
scales within the oracle's one unit in the last place."""
import numpy as np
import pytest

from util import host_layout, tq4_rows_equal_up_to_scale_ulp

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("hkv,n,shift", [(1, 1, 0), (1, 3, 2), (3, 5, 8), (4, 33, 1), (9, 7, 4)])
def test_rows_of_any_alignment_and_value(native_libs, hkv, n, shift):
    import oracle
    from warp34_b200 import kv, synth
    wl = synth.PagedWorkload([0], [n], hkv, seed=3, fill=0x3C)
    b = wl.step()
    k, v = synth.make_kv(n, hkv, 4)
    k[0, :7] = torch.tensor([65504.0, -65504.0, 6e-8, -0.0, 0.0, 1.0, -1.0], dtype=torch.float16)
    v[n - 1] = 0
    stride = hkv * 256 + 16
    kd = torch.zeros(n, stride, dtype=torch.float16, device="cuda")
    vd = torch.zeros(n, stride, dtype=torch.float16, device="cuda")
    kd[:, shift:shift + hkv * 256], vd[:, shift:shift + hkv * 256] = k.cuda(), v.cuda()
    kv.kv_cache_write(kv.Executor(1 << 16), wl.layer, b, kd[:, shift:], vd[:, shift:])
    torch.cuda.synchronize()
    hk, hv = np.full(wl.layer.k.numel(), 0x3C, np.uint8), np.full(wl.layer.v.numel(), 0x3C, np.uint8)
    oracle.kv_cache_write(host_layout(wl.layer.layout, hk, hv), b.host_desc(), k.numpy().view(np.uint16), v.numpy().view(np.uint16),
                          hkv * 256, hkv * 256, nthreads=2)
    for got, want in ((wl.layer.k, hk), (wl.layer.v, hv)):
        codes, scales, ulp = tq4_rows_equal_up_to_scale_ulp(got.cpu().numpy(), want)
        assert codes == 0 and ulp <= 1, (codes, scales, ulp)


def test_two_byte_aligned_destinations_and_non_finite_rows(native_libs):
    """The 16-bit store path writes what the 32-bit one does; a row with NaN or infinity leaves its neighbours alone: every other
    (token, head) row, of K and of V, is what it is when those two values are finite."""
    from warp34_b200 import kv, synth
    n, hkv = 20, 2
    k, v = synth.make_kv(n, hkv, 9, device="cuda")
    clean = synth.PagedWorkload([0], [n], hkv, seed=3, fill=0x3C)
    kv.kv_cache_write(kv.Executor(1 << 16), clean.layer, clean.step(), k, v)
    torch.cuda.synchronize()
    k[3, 5], v[7, 300] = float("nan"), float("inf")
    pools = []
    for off in (0, 2):
        wl = synth.PagedWorkload([0], [n], hkv, seed=3, fill=0x3C)
        base = torch.full((wl.layer.k.numel() + 16,), 0x3C, dtype=torch.uint8, device="cuda")
        wl.layer.layout.k_base = base.data_ptr() + off
        kv.kv_cache_write(kv.Executor(1 << 16), wl.layer, wl.step(), k, v)
        torch.cuda.synchronize()
        pools.append((base[off:off + wl.layer.k.numel()].cpu(), wl.layer.v.cpu()))
    assert torch.equal(pools[0][0], pools[1][0]) and torch.equal(pools[0][1], pools[1][1])
    assert (pools[0][0] != 0x3C).any()
    pages = clean.seqs[0].pages      # the same seed: the same pages
    for got, want, token, head in ((pools[0][0], clean.layer.k.cpu(), 3, 0), (pools[0][1], clean.layer.v.cpu(), 7, 1)):
        differ = (got.view(-1, hkv, 16, 132) != want.view(-1, hkv, 16, 132)).any(-1)
        poisoned = torch.zeros_like(differ)
        poisoned[pages[token // 16], head, token % 16] = True
        assert differ[poisoned].all() and not differ[~poisoned].any(), torch.nonzero(differ & ~poisoned)[:4]


@pytest.mark.parametrize("dtype", ["f16", "bf16"])
def test_products_and_sums_are_rounded_one_by_one(native_libs, dtype):
    """Rows whose stored scale or codes change when a product and the add behind it become one rounding, which the assembler makes of the
    packed forms where it can (22 of a million scales): 48 of each activation type out of 400 million normal rows, with the bytes that scalar
    __fmul_rn / __fadd_rn arithmetic writes (golden/tq4_append_sums.npz: found by comparing both forms)."""
    import ctypes as C
    import os
    from util import GOLDEN
    from warp34_b200 import kv, synth
    data = np.load(os.path.join(os.path.dirname(GOLDEN), "tq4_append_sums.npz"))
    want = data[dtype + "_bytes"]
    n = len(want)
    x = torch.from_numpy(data[dtype + "_rows"].view(np.int16)).cuda().view(torch.float16 if dtype == "f16" else torch.bfloat16)
    wl = synth.PagedWorkload([0], [n], 1, seed=3)
    ex, b = kv.Executor(1 << 16), wl.step()
    fn = native_libs[0].warp34_kv_cache_write_strided if dtype == "f16" else native_libs[0].warp34_tq4_kv_cache_write_strided_bf16
    assert fn(C.byref(ex.ex), C.byref(wl.layer.layout), C.byref(b.desc), x.data_ptr(), x.data_ptr(), 256, 256) == 0
    torch.cuda.synchronize()
    for pool in (wl.layer.k, wl.layer.v):
        got = pool.cpu().numpy().reshape(-1, 16, 132)[np.asarray(wl.seqs[0].pages)].reshape(-1, 132)[:n]
        assert (got == want).all(), f"{(got != want).any(1).sum()} of {n} rows differ"
