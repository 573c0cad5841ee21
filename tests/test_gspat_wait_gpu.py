"""GS-PAT's bounded waits: above 64 foci the iteration's blocks wait for each other's entries.  With one
block's entries withheld every wait runs out: the solve must fail with an error, leave the system's
drive as it was, fail a served request, and leave the context usable.  The focus counts are those of
the iteration's forms (R in registers: 65, 300; R in L2: 400)."""
import ctypes

import numpy as np
import pytest

import workloads as W
from serving_client import Engine, slice_desc

pytestmark = pytest.mark.gpu


def _problem(m):
    rng = np.random.default_rng(m)
    pos = W.tiled_array(1, 1)
    n = len(pos)
    rec = W.t4010a1_records(pos, 1.0, 0.25)
    cen = W.array_center(pos)
    foci = np.empty((m, 3), np.float32)
    foci[:, :2] = cen[:2] + rng.uniform(-100, 100, (m, 2))
    foci[:, 2] = rng.uniform(100, 300, m)
    return (rec, np.full(n, W.wavenumber(), np.float32), np.zeros(n, np.float32), foci,
            rng.uniform(0.5, 1.0, m).astype(np.float32), cen)


@pytest.mark.parametrize("m", [65, 300, 400])
def test_a_wait_that_runs_out_fails_the_solve(gpu, m):
    afc = gpu
    rec, k, a, foci, amps, _ = _problem(m)
    ref = afc.UniformSystem(300.0)
    ref.add_records(1, rec, k, a)
    afc.Optimizer.gs_pat(ref, foci, amps)
    s = afc.UniformSystem(300.0)
    s.add_records(1, rec, k, a)
    afc.DLL.AFC_ClearLastError()
    afc.DLL.AFO_GSPATWaitTest(s.handle, foci.ctypes.data_as(ctypes.c_void_p),
                              amps.ctypes.data_as(ctypes.POINTER(ctypes.c_float)), ctypes.c_ulong(m), 1)
    assert "ran out" in afc.last_error()
    np.testing.assert_array_equal(s.records(), rec)
    afc.Optimizer.gs_pat(s, foci, amps)  # the next solve of the same system
    np.testing.assert_array_equal(s.records(), ref.records())
    assert np.all(np.isfinite(s.records()))


def test_a_wait_that_runs_out_fails_the_request(gpu):
    afc = gpu
    rec, k, a, foci, amps, cen = _problem(100)
    desc, _ = slice_desc(afc, cen[:2], 150.0, half=10.0)
    e = Engine(afc, 64 << 20, 16 << 20, 1)  # one slot: every request uses the same status word
    try:
        gid = e.add_geometry(1, rec, k, a)
        good, out0, ap0 = e.submit_gspat(gid, len(k), foci, amps, desc)
        m = int(desc.count[0] * desc.count[1] * desc.count[2])
        out, ap = np.full(m, 7.0, np.float32), np.full(2 * len(k), 7.0, np.float32)
        bad = afc.DLL.AFC_ServeSubmitGspatWaitTest(e.h, gid, foci.ctypes.data, amps.ctypes.data, len(amps),
                                                   ctypes.byref(desc), out.ctypes.data, ap.ctypes.data)
        assert bad > 0
        again, out1, ap1 = e.submit_gspat(gid, len(k), foci, amps, desc)
        e.wait(good)
        with pytest.raises(RuntimeError, match="ran out"):
            e.wait(bad)
        e.wait(again)
        assert np.all(out == 7.0) and np.all(ap == 7.0)
        np.testing.assert_array_equal(out0, out1)
        np.testing.assert_array_equal(ap0, ap1)
        assert np.all(np.isfinite(ap1))
        s = e.stats()
        assert s["completed"] == 2 and s["failed"] == 1
    finally:
        e.close()
