"""Series that lie elsewhere than in the search's own device memory: the
search copies them first, with the same result."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _tap(s, ptrs, nsamps, on_device):
    from peasoup_b200 import _lib
    from peasoup_b200._lib import load
    n = len(ptrs)
    arr = (C.c_void_p * n)(*ptrs)
    dms, idx = np.zeros(n, np.float32), np.arange(n, dtype=np.int32)
    count = C.c_size_t()
    assert load().psx_search_block(s._handle, arr, nsamps, on_device, dms.ctypes.data,
                                   idx.ctypes.data, n, _lib.PSX_OUT_DM, s._out.ctypes.data,
                                   s._na.ctypes.data, s._tr.ctypes.data, None, s._cap,
                                   C.byref(count)) == 0
    return s.debug_tap(0)


@pytest.mark.parametrize("ndm", [1, 6])
@pytest.mark.parametrize("shift", [0, 1])
@pytest.mark.parametrize("where", ["mapped", "managed"])
def test_series_called_the_devices(cuda, where, shift, ndm):
    """Pinned host and managed memory given as device series, alone and in a
    group, aligned and one float further on."""
    from peasoup_b200 import search, synth
    torch = cuda
    n, nsamps = 1 << 19, 400_001
    x = (np.random.default_rng(1).standard_normal(nsamps) + 3.0).astype(np.float32)
    s = search.AccelSearch(search.SearchParams(
        fft_size=n, tsamp=64e-6, cfreq_hz=synth.CFREQ_HZ, ch_bw_hz=synth.CH_BW_HZ, nharmonics=2,
        min_snr=9.0, group_dms=4 if ndm > 1 else 1))
    d = torch.from_numpy(x).cuda()
    want = _tap(s, [d.data_ptr()] * ndm, nsamps, 1)
    if where == "mapped":
        t = torch.zeros(nsamps + 4).pin_memory()
        t[shift:shift + nsamps] = torch.from_numpy(x)
        ptr = t.data_ptr() + 4 * shift
    else:
        rt = C.CDLL("libcudart.so.12")
        base = C.c_void_p()
        assert rt.cudaMallocManaged(C.byref(base), C.c_size_t(4 * (nsamps + 4)), C.c_uint(1)) == 0
        ptr = base.value + 4 * shift
        C.memmove(ptr, x.ctypes.data, x.nbytes)
    got = _tap(s, [ptr] * ndm, nsamps, 1)
    for a, b in zip(got, want):
        assert np.array_equal(a, b)
    s.close()
    if where == "managed":
        assert rt.cudaFree(base) == 0
