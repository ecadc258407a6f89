"""psx_search_retarget between configurations whose defaults differ from what
is spelled out: a retargeted instance searches as a fresh one does, and what
does not match the instance stays refused."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _params(n, acc, **kw):
    from peasoup_b200 import search, synth
    return search.SearchParams(fft_size=n, tsamp=64e-6, cfreq_hz=synth.CFREQ_HZ,
                               ch_bw_hz=synth.CH_BW_HZ, acc_lo=-acc, acc_hi=acc, nharmonics=4,
                               min_snr=5.5, **kw)


def _series(n, count):
    from peasoup_b200 import synth
    return np.stack([synth.make_series_np(synth.SeriesSpec(
        nsamps=n, tsamp=64e-6, pulsars=[synth.Pulsar(5.1e-3 + 1e-3 * d, 30.0, 0.05, 0.5)]), 7 + d)
        for d in range(count)])


def _retarget(s, p):
    from peasoup_b200._lib import load
    cfg, keep = p.to_c()
    rc = load().psx_search_retarget(s._handle, C.byref(cfg))
    del keep
    return rc


def _block(s, xs):
    return s.search_block(xs, np.linspace(0.0, 20.0, len(xs)).astype(np.float32), per_dm=False)


def _equal_to_fresh(s, p, xs):
    from peasoup_b200 import search
    got, info = _block(s, xs), s.info()
    fresh = search.AccelSearch(p)
    want, winfo = _block(fresh, xs), fresh.info()
    fresh.close()
    assert len(want[0]) > 0
    for a, b in zip(got, want):
        assert np.array_equal(a, b)
    for k in ("fft_form", "batch", "group_dms", "ntrials", "harm_shape", "kernel_launches"):
        assert info[k] == winfo[k], k
    return winfo


@pytest.mark.parametrize("first,then", [(4, 0), (0, 4)])
def test_harmonic_shape_asked_for_and_by_default(cuda, first, then):
    """Groups of twelve trials at 2^21 points take the three-row shape by
    default: its tensor maps are there also where the instance was made for
    the single-row one."""
    from peasoup_b200 import search
    n = 1 << 21
    xs = _series(n, 1)
    kw = dict(batch=12)
    s = search.AccelSearch(_params(n, 800.0, harm_shape=first, **kw))
    for shape in (then, first, then):
        p = _params(n, 800.0, harm_shape=shape, **kw)
        assert _retarget(s, p) == 0
        info = _equal_to_fresh(s, p, xs)
        assert info["ntrials"] >= 12
    s.close()


def test_what_does_not_match_stays_refused(cuda):
    from peasoup_b200 import _lib, search
    n = 1 << 20
    base = dict(batch=12)
    s = search.AccelSearch(_params(n, 100.0, **base))
    for bad in (_params(n, 100.0, batch=12, harm_shape=6), _params(n, 100.0, batch=11),
                _params(n, 100.0, batch=12, fft_form=1), _params(n, 100.0, batch=12, group_dms=5),
                _params(n, 100.0, batch=12, lanes=2), _params(n // 2, 100.0, batch=12),
                _params(n, 100.0, batch=12, mode="plain")):
        assert _retarget(s, bad) == _lib.PSX_ERR_INVALID
    _equal_to_fresh(s, _params(n, 100.0, **base), _series(n, 1))
    s.close()


@pytest.mark.parametrize("first,then", [(0, 4), (4, 0)])
def test_grouping_asked_for_and_by_default(cuda, first, then):
    """Four DM trials to a grouped prologue, by name or as the default's
    least, match; what the default takes at this length (16) is made anew."""
    from peasoup_b200 import search
    n = 1 << 19
    xs = _series(n, 26)
    s = search.AccelSearch(_params(n, 0.0, group_dms=first))
    for g in (then, first):
        p = _params(n, 0.0, group_dms=g)
        assert _retarget(s, p) == 0
        assert _equal_to_fresh(s, p, xs)["group_dms"] == (4 if g else 9)
    s.close()


@pytest.mark.parametrize("own_stream", [True, False])
def test_short_lengths_with_cufft_asked_for_and_by_default(cuda, own_stream):
    """2^17 points: the default and cuFFT's transform by name match, and
    launch groups count as its powers of two; birdies go along."""
    from peasoup_b200 import search
    n = 1 << 17
    xs = _series(n, 7)
    birdies = dict(birdie_freqs=np.array([50.0], np.float32),
                   birdie_widths=np.array([0.5], np.float32))
    s = search.AccelSearch(_params(n, 40.0, batch=16, **birdies))
    st = cuda.cuda.Stream()
    if not own_stream:
        s.set_stream(st.cuda_stream)
    for kw in (dict(batch=16, fft_form=1), dict(batch=24), dict(batch=24, fft_form=1, **birdies),
               dict(batch=16, **birdies), dict(batch=16)):
        p = _params(n, 40.0, **kw)
        assert _retarget(s, p) == 0
        info = _equal_to_fresh(s, p, xs)
        assert info["fft_form"] == (1 if kw.get("fft_form") else 3)
    s.close()
