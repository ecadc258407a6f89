"""What psx_search_last_info reports is what ran: kernel launches and the
harmonic kernel's shape."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _search(n, **kw):
    from peasoup_b200 import search, synth
    return search.AccelSearch(search.SearchParams(
        fft_size=n, tsamp=64e-6, cfreq_hz=synth.CFREQ_HZ, ch_bw_hz=synth.CH_BW_HZ, nharmonics=4,
        min_snr=30.0, **kw))


# A trial's four kernels and the prologue's eight beside the means: one kernel
# up to 2^21 samples (from four rows 2^23), four above.  Five DM trials of 2^22
# points go in groups of four and one, eight of 2^19 in two of four, with one
# launch of each of a trial's kernels to a group.
@pytest.mark.parametrize("n,ndm,want", [
    (1 << 17, 1, 13), (1 << 19, 1, 13), (1 << 21, 1, 13), (1 << 22, 1, 16), (1 << 22, 3, 48),
    (1 << 22, 5, 13 + 16), (1 << 19, 8, 2 * 13)])
def test_kernel_launches(cuda, n, ndm, want):
    torch = cuda
    s = _search(n)
    x = torch.randn(ndm, n, device="cuda")
    for _ in range(2):
        s.search_block([x[d] for d in range(ndm)], np.zeros(ndm, np.float32))
        info = s.info()
        assert info["ntrials"] == ndm and info["fft_launches"] == 0
        assert info["kernel_launches"] == want, info
    s.close()


@pytest.mark.parametrize("batch,shape,want", [(12, 0, 6), (4, 0, 4), (12, 4, 4), (12, 6, 6)])
def test_harmonic_shape_of_the_largest_group(cuda, batch, shape, want):
    n = 1 << 21
    s = _search(n, acc_lo=-200.0, acc_hi=200.0, batch=batch, harm_shape=shape)
    x = cuda.randn(n, device="cuda")
    for _ in range(3):  # launched, captured and replayed
        s.search(x)
        assert s.info()["ntrials"] >= batch and s.info()["harm_shape"] == want
    s.close()


@pytest.mark.parametrize("lg,folds,batch,want", [
    (20, 4, 3, 4), (20, 4, 12, 4), (20, 5, 16, 4), (20, 4, 24, 6), (20, 4, 32, 4), (21, 4, 3, 4),
    (21, 4, 6, 6), (21, 3, 14, 4), (21, 4, 20, 6), (22, 4, 3, 6), (22, 4, 8, 4), (22, 4, 10, 6),
    (22, 1, 12, 4), (22, 2, 14, 4), (23, 4, 8, 6)])
def test_default_harmonic_shape(cuda, lg, folds, batch, want):
    """Per launch group, the shape that was measured to be the faster one."""
    from peasoup_b200 import search, synth
    n = 1 << lg
    s = search.AccelSearch(search.SearchParams(
        fft_size=n, tsamp=76e-6, cfreq_hz=synth.CFREQ_HZ, ch_bw_hz=synth.CH_BW_HZ, acc_lo=-2000.0,
        acc_hi=2000.0 if lg < 22 else -1800.0, nharmonics=folds, min_snr=30.0, batch=batch,
        group_dms=1))
    s.search(cuda.randn(n, device="cuda"))
    assert s.info()["ntrials"] >= batch and s.info()["harm_shape"] == want
    s.close()


@pytest.mark.parametrize("acc", [60.0, 100.0, 150.0, 250.0, 300.0])
def test_default_harmonic_shape_equals_the_single_row_one(cuda, acc):
    """2^21 points in groups of up to 20 and 6 trials: the same candidates,
    bit for bit, whichever shape the groups take."""
    from peasoup_b200 import search, synth
    n = 1 << 21
    x = synth.make_series_np(synth.SeriesSpec(
        nsamps=n, tsamp=64e-6, pulsars=[synth.Pulsar(5.1e-3, 100.0, 0.05, 0.4)]), 2)
    for batch in (20, 6):
        got = []
        for shape in (0, 4):
            s = search.AccelSearch(search.SearchParams(
                fft_size=n, tsamp=64e-6, cfreq_hz=synth.CFREQ_HZ, ch_bw_hz=synth.CH_BW_HZ,
                acc_lo=-acc, acc_hi=acc, nharmonics=4, min_snr=5.5, batch=batch, harm_shape=shape))
            got.append(s.search(x, 1.0, 2, per_dm=False))
            s.close()
        assert len(got[0][0]) > 0
        for a, b in zip(*got):
            assert np.array_equal(a, b)


def test_host_baseline_loop_takes_over(cuda):
    """A mean of 1e12 leaves residual means above the threshold after every
    float subtraction that the device makes: on either transform the host's
    loop goes on from there."""
    from peasoup_b200 import search, synth
    n = 1 << 19
    x = (np.random.default_rng(3).standard_normal(n) * 1e9 + 1e12).astype(np.float32)
    for form in (3, 1):
        s = search.AccelSearch(search.SearchParams(
            fft_size=n, tsamp=64e-6, cfreq_hz=synth.CFREQ_HZ, ch_bw_hz=synth.CH_BW_HZ,
            nharmonics=2, min_snr=8.0, batch=2, fft_form=form))
        s.search(x)
        assert s.info()["baseline_passes"] == -1
        s.search((x - np.float32(1e12)) / np.float32(1e9))
        assert s.info()["baseline_passes"] in (1, 2, 3)
        s.close()
