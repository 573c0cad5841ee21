"""Serving: a field request that fits the engine's device budget without the partial sums of its cut over
work items is accepted, and gives the field of AFC_Calculate; one that does not fit stays refused.

619,000 grid points make just fewer tiles than the work items a lone request is cut into, so that its partial
sums (two per point) take twice its result.
"""
import numpy as np
import pytest

import workloads as W
from serving_client import Engine

pytestmark = pytest.mark.gpu


def test_budget_without_partial_sums(gpu):
    afc = gpu
    n = 996
    pos = W.tiled_array(2, 2)
    cen = W.array_center(pos)
    rng = np.random.default_rng(0)
    amp, ph = W.random_pattern(rng, n)
    rec = W.sphere_records(pos, amp, ph)
    k, a = np.full(n, W.wavenumber(), np.float32), np.zeros(n, np.float32)
    spec = W.GridSpec(3, [(cen[0] - 40.0, cen[0] - 40.0 + 92.7), (cen[1] - 90.0, cen[1] - 90.0 + 184.7),
                          (80.0, 84.2)], 0.5, (W.AXIS_X, W.AXIS_Y, W.AXIS_Z))
    area = afc.grid_from_spec(spec)
    desc = area.grid_desc()
    m = int(desc.count[0] * desc.count[1] * desc.count[2])
    assert m == 186 * 370 * 9
    need = (8 + 48) * n + 8 * m  # drive, packed sources, complex result
    s = afc.UniformSystem(300.0)
    s.add_records(0, rec, k, a)
    ref = np.asarray(afc.GpuCalculator().calculate(s, area, afc.ComplexPressureFieldBuffer())).reshape(-1)
    for budget in (need + (1 << 20), need + (64 << 20)):
        e = Engine(afc, budget, 64 << 20, 2)
        try:
            gid = e.add_geometry(0, rec, k, a)
            rid, out = e.submit_field(gid, amp, ph, 2, grid=desc)
            e.wait(rid)
        finally:
            e.close()
        err = np.max(np.abs(out.view(np.complex64) - ref)) / np.max(np.abs(ref))
        print(f"budget {budget}: {err:.2e}")
        assert err <= 1e-5
    e = Engine(afc, need - (1 << 20), 64 << 20, 2)
    try:
        gid = e.add_geometry(0, rec, k, a)
        with pytest.raises(RuntimeError, match="HBM budget"):
            e.submit_field(gid, amp, ph, 2, grid=desc)
    finally:
        e.close()
