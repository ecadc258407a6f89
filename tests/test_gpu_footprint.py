"""psx_search_footprint against the device memory an instance takes."""
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1 << 17, 1 << 19, 3 << 18, 1 << 21, 1 << 22, 1 << 23])
@pytest.mark.parametrize("group", [0, 1, 12])
def test_footprint_is_what_an_instance_holds(cuda, n, group):
    """At least what the instance takes less 16 MB (the device hands out whole
    pages of 2 MB), at most a quarter more."""
    from peasoup_b200 import search
    torch = cuda
    p = search.SearchParams(fft_size=n, tsamp=64e-6, batch=16, group_dms=group)
    warm = search.AccelSearch(p)  # modules and tables a process loads once
    free0 = torch.cuda.mem_get_info()[0]
    s = search.AccelSearch(p)
    held = free0 - torch.cuda.mem_get_info()[0]
    s.close()
    warm.close()
    assert held - (16 << 20) <= search.footprint(p) <= 1.25 * held, (held, search.footprint(p))
