"""A dedispersion plan keeps the shift tables of every form its calls need:
short and long outputs, and sample widths, in turn."""
import ctypes as C
import time

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _plan(psx, nchans, ndm, dmax, band=200.0):
    h = C.c_void_p()
    assert psx.psx_dedisp_create(nchans, 64e-6, 1500.0, -band / nchans, C.byref(h)) == 0
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


@pytest.mark.parametrize("nchans,nbits,ndm,dmax", [(9, 8, 17, 3.0), (64, 16, 33, 8.0),
                                                   (64, 2, 32, 60.0), (256, 4, 64, 60.0),
                                                   (136, 1, 50, 30.0), (64, 8, 40, 12.0)])
def test_outputs_of_any_number_equal_definition(psx, cuda, oracle, nchans, nbits, ndm, dmax):
    """Numbers of outputs on both sides of where the form changes (launches of
    one to four CTAs an SM, whole and part tiles) through one plan: the
    definition in whole numbers."""
    from peasoup_b200 import sigproc
    torch = cuda
    tile = 512 if nbits == 16 else 1024
    h, dms = _plan(psx, nchans, ndm, dmax)
    md, most = psx.psx_dedisp_get_max_delay(h), 440 * tile
    delays = oracle.delay_table(nchans, 64e-6, 1500.0, -200.0 / nchans)
    v = np.random.default_rng(ndm).integers(0, 1 << nbits, (most + md, nchans), dtype=np.uint32)
    v[:, : nchans // 2] = (1 << nbits) - 1  # the largest sums
    x = torch.from_numpy(v.T.astype(np.int32)).cuda().contiguous()
    rows = torch.from_numpy(sigproc.pack_samples(v, nbits)).cuda()
    shift = np.rint(dms[:, None] * delays[None, :]).astype(np.int64)
    want = torch.zeros((ndm, most), dtype=torch.int32, device="cuda")
    for d in range(ndm):
        for c in range(nchans):
            want[d] += x[c, shift[d, c]:shift[d, c] + most]
    want = want.float()
    for tiles in (1, 36, 73, 74, 110, 148, 149, 222, 296, 297, 439):
        for tail in (0, 1, tile - 1):
            nout = tiles * tile + tail
            out = torch.full((ndm, most + 4), -1.0, device="cuda")
            assert psx.psx_dedisp_execute(h, nout + md, C.c_void_p(rows.data_ptr()), nbits,
                                          C.c_void_p(out.data_ptr()), most + 4, 1, None) == 0
            assert torch.equal(out[:, :nout], want[:, :nout]), (tiles, tail)
            assert torch.all(out[:, nout:] == -1.0)
    psx.psx_dedisp_destroy(h)


@pytest.mark.parametrize("nbits", [2, 8])
def test_half_a_device_of_ctas_is_no_step_in_time(psx, cuda, nbits):
    """32 DM trials of 64 channels: a 74th tile of outputs is no reason for a
    form whose 74 CTAs take half as long again as the direct form's 296."""
    torch = cuda
    h, _ = _plan(psx, 64, 32, 60.0, band=70.0)
    md = psx.psx_dedisp_get_max_delay(h)
    rows = torch.randint(0, 256, ((75 * 1024 + md) * 8 * nbits,), dtype=torch.uint8, device="cuda")
    out = torch.empty((32, 75 * 1024), device="cuda")
    best = {}
    for _ in range(5):
        for tiles in (73, 74):
            e = [torch.cuda.Event(enable_timing=True) for _ in range(2)]
            for k in range(24):
                if k == 4:
                    e[0].record()
                assert psx.psx_dedisp_execute(h, tiles * 1024 + md, C.c_void_p(rows.data_ptr()),
                                              nbits, C.c_void_p(out.data_ptr()), 75 * 1024, 0,
                                              None) == 0
            e[1].record()
            torch.cuda.synchronize()
            best[tiles] = min(best.get(tiles, 1e9), e[0].elapsed_time(e[1]))
    psx.psx_dedisp_destroy(h)
    assert best[74] < 1.25 * best[73], best


@pytest.mark.parametrize("nchans", [62, 64, 66, 130])
@pytest.mark.parametrize("nsamps", [1, 63, 64, 65, 192])
@pytest.mark.parametrize("shift", [0, 2])
def test_16_bit_rows_turned_whole_and_in_part(psx, cuda, nchans, nsamps, shift):
    """64 samples x 64 channels at a time with every load first, where a tile
    is whole and rows are whole words; word by word or byte by byte elsewhere:
    each channel alone comes out as it went in."""
    torch = cuda
    h, _ = _plan(psx, nchans, 1, 0.0)
    rng = np.random.default_rng(nsamps)
    v = rng.integers(0, 1 << 16, (nsamps, nchans), dtype=np.uint16)
    buf = torch.zeros(v.nbytes + 16, dtype=torch.uint8, device="cuda")
    buf[shift:shift + v.nbytes] = torch.from_numpy(v.view(np.uint8).reshape(-1)).cuda()
    out = torch.empty((1, (nsamps + 3) // 4 * 4), device="cuda")
    for c in (0, 1, 31, 61, nchans - 1):
        km = np.zeros(nchans, np.int32)
        km[c] = 1
        assert psx.psx_dedisp_set_killmask(h, km.ctypes.data) == 0
        assert psx.psx_dedisp_execute(h, nsamps, C.c_void_p(buf.data_ptr() + shift), 16,
                                      C.c_void_p(out.data_ptr()), out.shape[1], 1, None) == 0
        assert np.array_equal(out[0, :nsamps].cpu().numpy(), v[:, c].astype(np.float32))
    psx.psx_dedisp_destroy(h)


@pytest.mark.parametrize("ndm", [32, 3])
def test_plans_of_several_threads_launch_one_kernel(psx, cuda, ndm):
    """Threads, each with a plan and a stream of its own, whose windows need
    different amounts of shared memory of the same kernel: every launch
    succeeds."""
    import threading
    torch = cuda
    nchans, nout = 64, 4096
    rows = torch.randint(0, 256, ((nout + 8192) * nchans,), dtype=torch.uint8, device="cuda")
    bad = []

    def work(k):
        h = _plan(psx, nchans, ndm, (5.0, 60.0)[k % 2], band=70.0)[0]
        o = torch.empty((ndm, nout), device="cuda")
        st = torch.cuda.Stream()
        md = psx.psx_dedisp_get_max_delay(h)
        args = (h, nout + md, C.c_void_p(rows.data_ptr()), 8, C.c_void_p(o.data_ptr()), nout, 0,
                C.c_void_p(st.cuda_stream))
        for i in range(4000):
            rc = psx.psx_dedisp_execute(*args)
            if rc:
                bad.append((k, i, rc, psx.psx_last_error()))
                break
            if i % 50 == 49:
                st.synchronize()
        st.synchronize()
        psx.psx_dedisp_destroy(h)

    threads = [threading.Thread(target=work, args=(k,)) for k in range(8)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not bad, bad


@pytest.mark.parametrize("nbits", [2, 8, 16])
def test_captured_after_a_call_of_another_size(psx, cuda, nbits):
    """A call is capturable once the plan has run, whatever outputs that call
    had: short outputs (the direct form) are captured after long ones, run
    again after further calls and replayed."""
    torch = cuda
    nchans, ndm, long_, short = 64, 64, 120 * 1024, 4 * 1024
    h, _ = _plan(psx, nchans, ndm, 20.0)
    md = psx.psx_dedisp_get_max_delay(h)
    rows = torch.randint(0, 256, ((long_ + md) * nchans * nbits // 8,), dtype=torch.uint8,
                         device="cuda")
    out, cap = torch.empty((ndm, long_), device="cuda"), torch.zeros((ndm, short), device="cuda")

    def run(o, nout, stream):
        return psx.psx_dedisp_execute(h, nout + md, C.c_void_p(rows.data_ptr()), nbits,
                                      C.c_void_p(o.data_ptr()), o.shape[1], 0,
                                      C.c_void_p(stream))

    assert run(out, long_, 0) == 0
    torch.cuda.synchronize()
    g, s = torch.cuda.CUDAGraph(), torch.cuda.Stream()
    with torch.cuda.graph(g, stream=s):
        rc = run(cap, short, s.cuda_stream)
    assert rc == 0
    want = torch.empty_like(cap)
    for _ in range(2):
        cap.zero_()
        g.replay()
        torch.cuda.synchronize()
        assert run(want, short, 0) == 0 and run(out, long_, 0) == 0
        torch.cuda.synchronize()
        assert torch.equal(cap, want) and torch.equal(out[:, :short], want)
    del g
    psx.psx_dedisp_destroy(h)
