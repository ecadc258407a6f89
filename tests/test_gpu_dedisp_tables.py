"""A dedispersion plan keeps the shift tables of every form its calls need:
short and long outputs, and sample widths, in turn."""
import ctypes as C
import time

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _plan(psx, nchans, ndm, dmax):
    h = C.c_void_p()
    assert psx.psx_dedisp_create(nchans, 64e-6, 1500.0, -200.0 / nchans, C.byref(h)) == 0
    dms = np.linspace(0.0, dmax, ndm).astype(np.float32)
    assert psx.psx_dedisp_set_dm_list(h, dms.ctypes.data, ndm) == 0
    return h, dms


def test_calls_in_turn_do_not_rebuild_tables(psx, cuda):
    """Host time of calls that take turns (a long output, a short one, 8 and
    2 bits) against that of a call after the DM list was set again, which
    builds and uploads its tables: with them kept, far below."""
    torch = cuda
    nchans, ndm = 1024, 200
    h, dms = _plan(psx, nchans, ndm, 40.0)
    md = psx.psx_dedisp_get_max_delay(h)
    short, long_ = 2048, 160 * 1024
    rows = torch.randint(0, 256, ((long_ + md) * nchans,), dtype=torch.uint8, device="cuda")
    out = torch.empty((ndm, long_), device="cuda")

    def call(nout, nbits):
        torch.cuda.synchronize()
        t = time.perf_counter()
        rc = psx.psx_dedisp_execute(h, nout + md, C.c_void_p(rows.data_ptr()), nbits,
                                    C.c_void_p(out.data_ptr()), long_, 0, None)
        t = time.perf_counter() - t
        assert rc == 0
        return t

    kinds = [(long_, 8), (short, 8), (long_, 2), (short, 2)]
    for k in kinds:
        call(*k)
    turns = [sum(call(*k) for k in kinds) for _ in range(5)]
    built = []
    for _ in range(3):
        s = 0.0
        for k in kinds:
            assert psx.psx_dedisp_set_dm_list(h, dms.ctypes.data, ndm) == 0
            s += call(*k)
        built.append(s)
    psx.psx_dedisp_destroy(h)
    assert min(turns) < 0.3 * min(built), (turns, built)


@pytest.mark.parametrize("nbits", [2, 8, 16])
def test_turns_and_changes_of_the_plan_equal_a_fresh_one(psx, cuda, nbits):
    """Long, short and long again, with another channel mask and DM list in
    between: the same floats as a plan made for the call."""
    torch = cuda
    nchans, ndm = 64, 70
    rng = np.random.default_rng(nbits)
    mask = (rng.random(nchans) > 0.2).astype(np.int32)
    h, dms = _plan(psx, nchans, ndm, 30.0)
    long_, short = 120 * 1024, 3000
    ns = long_ + 4096
    rows = torch.from_numpy(rng.integers(0, 256, ns * nchans * nbits // 8, dtype=np.uint8)).cuda()

    def run(plan, nout):
        md = psx.psx_dedisp_get_max_delay(plan)
        assert nout + md <= ns
        o = torch.full((ndm, long_), -1.0, device="cuda")
        assert psx.psx_dedisp_execute(plan, nout + md, C.c_void_p(rows.data_ptr()), nbits,
                                      C.c_void_p(o.data_ptr()), long_, 0, None) == 0
        return o.cpu().numpy()

    for km, top in ((None, 30.0), (mask, 30.0), (mask, 45.0), (None, 30.0)):
        d = np.linspace(0.0, top, ndm).astype(np.float32)
        p = km.ctypes.data if km is not None else None
        assert psx.psx_dedisp_set_dm_list(h, d.ctypes.data, ndm) == 0
        assert psx.psx_dedisp_set_killmask(h, p) == 0
        for nout in (long_, short, long_):
            fresh, _ = _plan(psx, nchans, ndm, top)
            assert psx.psx_dedisp_set_killmask(fresh, p) == 0
            assert np.array_equal(run(h, nout), run(fresh, nout))
            psx.psx_dedisp_destroy(fresh)
    psx.psx_dedisp_destroy(h)
