"""Small point sets: the cluster split of a few point tiles, the chunked launch of any number of points
against many sources, and the source groups of the one- and two-pair bodies (counts that leave a
remainder after groups of two, near-edge points among them), against the oracle.

Tolerance: the stated bar, max |p_gpu - p_ref| <= 1e-4 max |p_ref|.
"""
import numpy as np
import pytest

import oracle as O
import workloads as W

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("calc", ["GpuCalculator", "AccurateCalculator"])
@pytest.mark.parametrize("n,m", [(1, 1), (2, 3), (33, 100), (249, 511), (249, 513), (300, 20001),
                                 (996, 1000), (1535, 97), (1536, 97), (2490, 1), (2490, 2047)])
def test_small_scatter_sets(gpu, calc, n, m):
    afc = gpu
    rng = np.random.default_rng(10 * n + m)
    pos = W.tiled_array(5, 2)[:n]
    cen = pos.mean(axis=0)
    amp, ph = W.random_pattern(rng, n)
    rec = W.t4010a1_records(pos, amp, ph)
    k = np.full(n, W.wavenumber(), np.float32)
    a = np.full(n, 1.15e-2, np.float32)
    pts = np.empty((m, 3), np.float32)
    pts[:, :2] = cen[:2] + rng.uniform(-100, 100, (m, 2))
    pts[:, 2] = rng.uniform(50, 200, m)
    # a third of the points on 30 and 60 degree cones of some source
    for i in range(0, m, 3):
        th, az = np.deg2rad((30.0, 60.0)[i % 2]), rng.uniform(0, 2 * np.pi)
        r = pts[i, 2] / np.cos(th)
        pts[i, :2] = pos[i % n, :2] + r * np.sin(th) * np.array([np.cos(az), np.sin(az)])
    s = afc.UniformSystem(300.0)
    s.add_records(1, rec, k, a)
    area = afc.ScatterArea()
    area.add_observe_points(pts)
    out = getattr(afc, calc)().calculate(s, area, afc.ComplexPressureFieldBuffer())
    ref = O.field_f32(1, rec, k, a, pts, O.FIELD_COMPLEX)
    err = float(np.max(np.abs(out - ref)) / np.max(np.abs(ref)))
    print(f"{calc} n={n} m={m}: {err:.2e}")
    assert err <= 1e-4
