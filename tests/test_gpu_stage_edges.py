"""Stage kernels at the edges of their tiles, against the definitions in
numpy: harmonic sums (128 bins per warp), the two compaction kernels (runs
and parts), statistics, baseline removal and normalisation (128-bit and
unaligned forms)."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _at(torch, a, shift):
    """`a` on the device at an address `shift` floats past a 256-byte boundary."""
    buf = torch.zeros(len(a) + 64, device="cuda")
    v = buf[shift:shift + len(a)]
    v.copy_(torch.from_numpy(a))
    return v


@pytest.mark.parametrize("nharms", [1, 2, 3, 4, 5])
@pytest.mark.parametrize("n", [1, 31, 33, 127, 128, 129, 4097, 70001])
def test_harmonic_sum_tile_edges_bit_exact(psx, cuda, n, nharms):
    """A warp takes 128 bins: sizes around it, every fold, against the
    definition in float with the reference's double scales."""
    torch = cuda
    x = np.random.default_rng(n).standard_normal(n).astype(np.float32)
    d = torch.from_numpy(x).cuda()
    outs = [torch.full((n + 1,), -5.0, device="cuda") for _ in range(nharms)]
    ptrs = (C.c_void_p * nharms)(*[o.data_ptr() for o in outs])
    assert psx.psx_harmonic_sum(C.c_void_p(d.data_ptr()), ptrs, n, nharms, None) == 0
    torch.cuda.synchronize()
    i, val = np.arange(n), x.copy()
    for h in range(1, nharms + 1):
        for m in ([3, 1] if h == 2 else range(1, 1 << h, 2)):
            val = (val + x[(i * m + (1 << (h - 1))) >> h]).astype(np.float32)
        want = (val.astype(np.float64) * (1.0 / np.sqrt(2.0 ** h))).astype(np.float32)
        got = outs[h - 1].cpu().numpy()
        assert got[n] == -5.0
        # the double factors rsqrt(2^h) of the device may differ from the
        # host's in their last bit: at most one float rounding apart
        assert np.max(np.abs(got[:n] - want) / np.spacing(np.abs(want) + 1e-30)) <= 1.0


@pytest.mark.parametrize("n,start,every", [(1, 0, 1), (300, 7, 1), (2048, 0, 3), (2049, 0, 2048),
                                           (70001, 13, 1), (1 << 21, 255, 4099),
                                           ((1 << 22) + 5, 1, 1 << 21)])
def test_find_peaks_runs_against_definition(psx, cuda, n, start, every):
    """Runs and parts of the two compaction kernels: dense and rare hits,
    a last run of one bin, hits at both ends of a run, a short buffer."""
    torch = cuda
    x = np.zeros(n, np.float32)
    x[start::every] = 5.0 + np.arange(len(x[start::every])) % 97
    x[-1] = 200.0
    x[n // 2] = np.nan
    d = torch.from_numpy(x).cuda()
    with np.errstate(invalid="ignore"):
        want = np.flatnonzero(x[start:] > 4.0) + start
    for cap in (len(want), len(want) // 2):
        idx = torch.full((len(want) + 1,), -1, dtype=torch.int32, device="cuda")
        val = torch.full((len(want) + 1,), -1.0, device="cuda")
        cnt = C.c_int()
        rc = psx.psx_find_peaks(C.c_void_p(d.data_ptr()), n, start, 4.0,
                                C.c_void_p(idx.data_ptr()), C.c_void_p(val.data_ptr()), cap,
                                C.byref(cnt), None)
        assert rc == (0 if cap == len(want) else 5) and cnt.value == len(want)
        assert np.array_equal(idx.cpu().numpy()[:cap], want[:cap])
        assert np.array_equal(val.cpu().numpy()[:cap], x[want[:cap]])
        assert np.all(idx.cpu().numpy()[cap:] == -1)
        # the same spectrum whole, from its middle, empty and again in one call
        starts = (C.c_int * 4)(start, n // 2, n, start)
        ptrs = (C.c_void_p * 4)(*[d.data_ptr()] * 4)
        hi, hv = np.full((4, cap + 1), -1, np.int32), np.zeros((4, cap + 1), np.float32)
        hi, hv = hi[:, :cap].copy(), hv[:, :cap].copy()
        cnts = (C.c_int * 4)()
        rc = psx.psx_find_peaks_host(ptrs, (C.c_int * 4)(*[n] * 4), starts, 4, 4.0,
                                     hi.ctypes.data, hv.ctypes.data, cap, cnts, None)
        half = want[want >= n // 2]
        assert rc == (0 if cap == len(want) else 5)
        assert list(cnts) == [len(want), len(half), 0, len(want)]
        if rc == 0:
            for k, w in ((0, want), (1, half), (3, want)):
                assert np.array_equal(hi[k, :len(w)], w) and np.array_equal(hv[k, :len(w)], x[w])


@pytest.mark.parametrize("shift", [0, 1])
@pytest.mark.parametrize("n", [1, 3, 5, 1003, 300001])
def test_series_statistics_and_baseline_edges(psx, cuda, n, shift):
    """Aligned (128-bit) and unaligned forms, tails of 1 to 3 samples, one
    pass and several (a mean far above its float rounding)."""
    torch = cuda
    x = (np.random.default_rng(n).standard_normal(n) * 3 + 40).astype(np.float32)
    for mean in (0.0, 3e5):
        a = (x + np.float32(mean)).astype(np.float32)
        d = _at(torch, a, shift)
        m, r, s = C.c_float(), C.c_float(), C.c_float()
        assert psx.psx_stats(C.c_void_p(d.data_ptr()), n, 0, C.byref(m), C.byref(r), C.byref(s),
                             None) == 0
        assert abs(m.value - a.astype(np.float64).mean()) <= 1e-6 * abs(m.value)
        passes = C.c_int()
        assert psx.psx_remove_baseline(C.c_void_p(d.data_ptr()), n, C.byref(passes), None) == 0
        # the definition: float mean of the double sum, subtracted in float
        w, want = a.copy(), 0
        while True:
            mu = np.float32(np.float32(w.astype(np.float64).sum()) / np.float32(n))
            w = (w - mu).astype(np.float32)
            want += 1
            if want > 101 or not abs(float(mu)) > 5e-7 * n:
                break
        assert passes.value == want
        # one float rounding of a sample per pass
        assert np.max(np.abs(d.cpu().numpy() - w)) <= want * np.spacing(np.float32(np.abs(a).max()))
        d = _at(torch, a, shift)
        assert psx.psx_normalise(C.c_void_p(d.data_ptr()), 2.5, 1.5, n, None) == 0
        got = d.cpu().numpy()
        assert np.array_equal(got, ((a - np.float32(2.5)) / np.float32(1.5)).astype(np.float32))
