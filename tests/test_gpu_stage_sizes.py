"""Stage kernels on both sides of the sizes where their shape changes, against
numpy."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

LONG = 3 << 17  # bins from which a lane of the harmonic sums takes four


@pytest.mark.parametrize("nharms", [1, 2, 3, 4, 5])
@pytest.mark.parametrize("n", [63, 64, 65, LONG - 1, LONG, LONG + 1, LONG + 127, LONG + 128,
                               LONG + 131])
def test_harmonic_sums_of_two_and_four_bins_a_lane(psx, cuda, n, nharms):
    """The definition in float with the reference's double scales (their last
    bit may differ between device and host: one float rounding)."""
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
        assert np.max(np.abs(got[:n] - want) / np.spacing(np.abs(want) + 1e-30)) <= 1.0


def test_short_harmonic_sums_keep_a_lane_s_chain_short(psx, cuda):
    """24,577 bins do not fill the device: their time is a lane's reads, 4.3 us
    with two bins a lane and 5.6 with four (five folds), against 6.9 for
    393,217 bins in either case."""
    torch = cuda
    best = {}
    for n in (24577, LONG + 1):
        x = torch.randn(n, device="cuda")
        outs = [torch.empty(n, device="cuda") for _ in range(5)]
        ptrs = (C.c_void_p * 5)(*[o.data_ptr() for o in outs])
        g = torch.cuda.CUDAGraph()
        s = torch.cuda.Stream()
        with torch.cuda.graph(g, stream=s):
            for _ in range(100):
                psx.psx_harmonic_sum(C.c_void_p(x.data_ptr()), ptrs, n, 5,
                                     C.c_void_p(s.cuda_stream))
        for _ in range(6):
            e = [torch.cuda.Event(enable_timing=True) for _ in range(2)]
            e[0].record()
            g.replay()
            e[1].record()
            torch.cuda.synchronize()
            best[n] = min(best.get(n, 1e9), e[0].elapsed_time(e[1]) * 10.0)
    assert best[24577] < 0.72 * best[LONG + 1], best


@pytest.mark.parametrize("shift", [0, 1])
@pytest.mark.parametrize("n", [3, 5, 1003, 300001, (1 << 20) + 3])
def test_rms_and_deviation(psx, cuda, n, shift):
    """Both forms of the statistics against 64 bits.  The float results: a
    few roundings of mean and rms (2^-22 relative), and for the deviation the
    roundings of rms^2 and mean^2 before their difference."""
    torch = cuda
    x = (np.random.default_rng(n).standard_normal(n) * 3 + 5).astype(np.float32)
    for first in (0, 2):
        buf = torch.zeros(n + 8, device="cuda")
        buf[shift:shift + n] = torch.from_numpy(x)
        m, r, s = C.c_float(), C.c_float(), C.c_float()
        assert psx.psx_stats(C.c_void_p(buf.data_ptr() + 4 * shift), n, first, C.byref(m),
                             C.byref(r), C.byref(s), None) == 0
        y = x[first:].astype(np.float64)
        cnt = float(n - first)
        mean, rms = y.sum() / cnt, np.sqrt((y * y).sum() / cnt)
        std = np.sqrt(max(rms * rms - mean * mean, 0.0))
        assert abs(m.value - mean) <= 2.0 ** -22 * abs(mean)
        assert abs(r.value - rms) <= 2.0 ** -22 * rms
        if std > 1e-3 * rms:
            assert abs(s.value - std) <= 2.0 ** -22 * ((rms * rms + mean * mean) / std + std)
