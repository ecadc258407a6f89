"""The per-DM prologue on the library's own transform (batched mode, fft_form
3) against the same instance on cuFFT's (fft_form 1): the dereddened series
and the statistics, over lengths with every column shape, padded and odd
series, unaligned and host input, birdies at both ends of the spectrum, means
that take several baseline passes and more than the device makes.

Tolerance: single-precision transforms of either library are within about
1e-6 of the result's RMS of the exact ones (forward and back), so the two
agree within 1e-5 of it; mean and deviation, sums over all bins, within 1e-5
relative."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _series(n, seed, mean):
    rng = np.random.default_rng(seed)
    t = np.arange(n)
    x = rng.standard_normal(n) + mean + 0.3 * np.sin(t * 0.02) + 2.0 * np.sin(t * 2e-5)
    return x.astype(np.float32)


def _tap(n, series, form, **kw):
    from peasoup_b200 import search, synth
    s = search.AccelSearch(search.SearchParams(
        fft_size=n, tsamp=64e-6, cfreq_hz=synth.CFREQ_HZ, ch_bw_hz=synth.CH_BW_HZ, acc_lo=0.0,
        acc_hi=0.0, nharmonics=2, min_snr=8.0, batch=2, fft_form=form, **kw))
    s.search(series)
    info = s.info()
    assert info["fft_form"] == form
    tim, _, _, norm = s.debug_tap(0)
    s.close()
    return tim, norm, info


# length, samples, mean, birdie edges (Hz; the last above Nyquist)
BIRDIES = np.array([0.0, 0.05, 60.0, 7812.4, 9000.0], np.float32)
CASES = [(1 << 19, 1 << 19, 0.0), (1 << 19, 400_001, 100.0), (3 << 17, 3 << 17, 50.0),
         (3 << 18, (3 << 18) - 1, 1e4), (1 << 21, 2_000_003, 128.0), (1 << 20, (1 << 20) + 77, 5.0),
         (1 << 26, (1 << 26) - 3, 3.0)]


@pytest.mark.parametrize("n,nsamps,mean", CASES)
def test_matches_cufft_prologue(cuda, n, nsamps, mean):
    torch = cuda
    x = _series(nsamps, n % 1009 + nsamps % 7, mean)
    kw = dict(birdie_freqs=BIRDIES, birdie_widths=np.full(len(BIRDIES), 0.3, np.float32))
    tim, norm, info = _tap(n, x, 3, **kw)
    want, wnorm, winfo = _tap(n, x, 1, **kw)
    assert info["baseline_passes"] == winfo["baseline_passes"]
    assert np.max(np.abs(tim - want)) <= 1e-5 * np.sqrt(np.mean(want.astype(np.float64) ** 2))
    assert np.all(np.abs(norm - wnorm) <= 1e-5 * np.abs(wnorm))
    if n > 1 << 22:
        return
    # device series, aligned and one float past it: the same bits
    buf = torch.zeros(nsamps + 1, device="cuda")
    for shift in (0, 1):
        d = buf[shift:shift + nsamps]
        d.copy_(torch.from_numpy(x))
        got, gnorm, _ = _tap(n, d, 3, **kw)
        assert np.array_equal(got, tim) and np.array_equal(gnorm, norm)


def test_more_baseline_passes_than_the_device_makes(cuda):
    """A mean of 1e12 leaves residual means far above the threshold after
    each float subtraction: the host's loop takes over."""
    n = 1 << 19
    x = (_series(n, 3, 0.0) * 1e9 + np.float32(1e12)).astype(np.float32)
    tim, norm, info = _tap(n, x, 3)
    want, wnorm, winfo = _tap(n, x, 1)
    assert np.max(np.abs(tim - want)) <= 1e-5 * np.sqrt(np.mean(want.astype(np.float64) ** 2))
    assert np.all(np.abs(norm - wnorm) <= 1e-5 * np.abs(wnorm))


def test_retarget_replaces_the_birdies(cuda):
    """A retargeted instance zaps the new list, or none."""
    import ctypes as C
    from peasoup_b200 import search, synth
    from peasoup_b200._lib import check, load
    n = 1 << 19
    x = _series(n, 9, 10.0)
    base = dict(fft_size=n, tsamp=64e-6, cfreq_hz=synth.CFREQ_HZ, ch_bw_hz=synth.CH_BW_HZ,
                nharmonics=2, min_snr=8.0, batch=2)
    lists = [np.zeros(0, np.float32), np.array([50.0, 160.0], np.float32),
             np.array([700.0], np.float32), np.zeros(0, np.float32)]
    s = search.AccelSearch(search.SearchParams(**base))
    for f in lists:
        p = search.SearchParams(birdie_freqs=f, birdie_widths=np.full(len(f), 2.0, np.float32),
                                **base)
        cfg, keep = p.to_c()
        check(load().psx_search_retarget(s._handle, C.byref(cfg)), "retarget")
        s.search(x)
        got = s.debug_tap(0)
        fresh = search.AccelSearch(p)
        fresh.search(x)
        want = fresh.debug_tap(0)
        fresh.close()
        assert np.array_equal(got[0], want[0]) and np.array_equal(got[3], want[3])
        del keep
    s.close()


@pytest.mark.parametrize("n", [1 << 17, 1 << 18])
def test_short_lengths_take_it_by_default(cuda, oracle, n):
    """2^17 and 2^18 points (256-row columns): the default form; series and
    statistics against cuFFT's prologue, the trials' gathered series bit for
    bit and their spectra against 64 bits (1e-5, as the longer lengths'), and
    an explicit fft_form 3 refused there as before."""
    from test_gpu_fft4 import _fp64_spectrum, err_vs_mag_or_rms
    from peasoup_b200 import search, synth
    from peasoup_b200._lib import PsxError
    from peasoup_b200.transforms import AccelerationPlan
    x = _series(n - 1001, 5, 70.0)
    base = dict(fft_size=n, tsamp=64e-6, cfreq_hz=synth.CFREQ_HZ, ch_bw_hz=synth.CH_BW_HZ,
                acc_lo=-300.0, acc_hi=300.0, nharmonics=2, min_snr=8.0,
                birdie_freqs=BIRDIES, birdie_widths=np.full(len(BIRDIES), 0.3, np.float32))
    with pytest.raises(PsxError):
        search.AccelSearch(search.SearchParams(fft_form=3, **base))
    want, wnorm, _ = _tap(n, x, 1, birdie_freqs=BIRDIES,
                          birdie_widths=np.full(len(BIRDIES), 0.3, np.float32))
    s = search.AccelSearch(search.SearchParams(**base))
    s.search(x)
    assert s.info()["fft_form"] == 3
    accs = AccelerationPlan(-300.0, 300.0, 1.10, 64e-6, n, 64e-6, synth.CFREQ_HZ,
                            synth.CH_BW_HZ).generate_accel_list(0.0, 0.0)
    for t in sorted({0, len(accs) // 2, len(accs) - 1}):
        tim, tr, ps, norm = s.debug_tap(t)
        idx = oracle.resampleII_index(n, float(accs[t]), 64e-6)
        assert np.array_equal(tr, tim[idx.astype(np.int64)])
        assert err_vs_mag_or_rms(ps, _fp64_spectrum(tim, idx, norm)) < 1e-5
    s.close()
    assert np.max(np.abs(tim - want)) <= 1e-5 * np.sqrt(np.mean(want.astype(np.float64) ** 2))
    assert np.all(np.abs(norm - wnorm) <= 1e-5 * np.abs(wnorm))


def test_default_harmonic_shape_per_launch_group(cuda):
    """With no harmonic shape asked for, launch groups of 2^20 points take
    the three-row kernel where its rows carry them (multiples of 3, 12 and
    more) and the single-row one otherwise: the same candidates, bit for bit,
    as the single-row shape throughout."""
    from peasoup_b200 import search, synth
    from peasoup_b200.transforms import AccelerationPlan
    n, ts = 1 << 20, 64e-6
    x = synth.make_series_np(synth.SeriesSpec(
        nsamps=n, tsamp=ts, pulsars=[synth.Pulsar(5.1e-3, 100.0, 0.05, 0.4)]), 2)
    seen = set()
    for acc in (50.0, 150.0, 300.0, 450.0, 800.0, 900.0):
        base = dict(fft_size=n, tsamp=ts, cfreq_hz=synth.CFREQ_HZ, ch_bw_hz=synth.CH_BW_HZ,
                    acc_lo=-acc, acc_hi=acc, nharmonics=4, min_snr=5.5, batch=14)
        seen.add(len(AccelerationPlan(-acc, acc, 1.10, 64e-6, n, ts, synth.CFREQ_HZ,
                                      synth.CH_BW_HZ).generate_accel_list(0.0, 0.0)))
        got = []
        for shape in (0, 4):
            s = search.AccelSearch(search.SearchParams(harm_shape=shape, **base))
            got.append(s.search(x, 1.0, 2, per_dm=False))
            s.close()
        assert len(got[0][0]) > 0
        for a, b in zip(*got):
            assert np.array_equal(a, b)
    # group sizes on both sides of the rule
    assert len({k % 3 for k in seen}) > 1, seen
