"""The means of the prologue's baseline loop depend on the samples alone: not
on the DM trials that share a launch, the CTAs of a row or the address of the
series.  The series here are sums of exact zero (paired values of 2^54 to
2^64 and of 2^20), whose double sum is what the order of its additions
rounds to, of the size of the loop's threshold: another order shows in the
number of passes (sums over 8 CTAs, 16 CTAs and the whole device disagreed in
every case here, as did the sums of a series 4 bytes further on)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

# samples, magnitude of the large values (their rounding errors add up to
# about the threshold, 5e-7 samples^2), DM trials to a group
CASES = [(1 << 16, 2.0 ** 54, 12), (1 << 16, 2.0 ** 54, 5), ((1 << 22) - 3, 2.0 ** 64, 4)]


def _series(n, big, seed):
    rng = np.random.default_rng(seed)

    def pairs(count, scale):
        v = (scale * (1.0 + rng.random(count // 2))).astype(np.float32)
        return rng.permutation(np.concatenate([v, -v]))
    x = np.zeros(n, np.float32)
    m = n // 4 * 4
    x[0:m:2] = pairs(m // 2, big)
    x[1:m:2] = pairs(m // 2, 2.0 ** 20)
    return x


@pytest.mark.parametrize("nsamps,big,group", CASES)
def test_means_do_not_depend_on_the_launch(cuda, nsamps, big, group):
    from peasoup_b200 import search, synth
    torch = cuda
    n = 1 << max(17, (nsamps - 1).bit_length())
    base = dict(fft_size=n, tsamp=64e-6, cfreq_hz=synth.CFREQ_HZ, ch_bw_hz=synth.CH_BW_HZ,
                nharmonics=1, min_snr=9.0, batch=4)
    alone = search.AccelSearch(search.SearchParams(group_dms=1, **base))
    grouped = search.AccelSearch(search.SearchParams(group_dms=group, **base))
    dms = np.zeros(2 * group, np.float32)
    for seed in range(8):
        buf = torch.zeros(nsamps + 4, device="cuda")
        passes = []
        for shift in (0, 1):
            d = buf[shift:shift + nsamps]
            d.copy_(torch.from_numpy(_series(nsamps, big, seed)))
            alone.search(d)
            passes.append(alone.info()["baseline_passes"])
        # two full groups of the same series: the last DM trial's passes
        grouped.search_block([d] * (2 * group), dms)
        assert grouped.info()["group_dms"] == group
        passes.append(grouped.info()["baseline_passes"])
        assert len(set(passes)) == 1, (seed, passes)
    alone.close()
    grouped.close()
