"""Sphere sources on both sides of the launch choice's lines (one pair a thread below 1,024 sources and
7e7 evaluations, four pairs above; no rows tiling with one pair), with counts that leave a remainder
after groups of two and four sources, and the T4010A1 grids whose pairs the model chooses (768 to 1,023
sources), against the oracle.

Tolerance: the stated bar, max |p_gpu - p_ref| <= 1e-4 max |p_ref|.
"""
import numpy as np
import pytest

import oracle as O
import workloads as W

pytestmark = pytest.mark.gpu


def _check(afc, st, n, grid=None, m=0):
    rng = np.random.default_rng(n + m + (sum(grid) if grid else 0))
    pos = W.tiled_array(5, 2)[:n]
    cen = pos.mean(axis=0)
    amp, ph = W.random_pattern(rng, n)
    rec = (W.t4010a1_records if st == 1 else W.sphere_records)(pos, amp, ph)
    k, a = np.full(n, W.wavenumber(), np.float32), np.full(n, 1.15e-2, np.float32)
    s = afc.UniformSystem(300.0)
    s.add_records(st, rec, k, a)
    if grid:
        lo = [float(np.float32(c)) for c in (cen[0] - 40, cen[1] - 30, 60)]
        dim = 3 if grid[2] > 1 else 2
        lohi = [(lo[i], lo[i] + 0.5 * (grid[i] - 1) + (0.25 if grid[i] > 1 else 0)) for i in range(3)]
        spec = W.GridSpec(dim, lohi, 0.5, (W.AXIS_X, W.AXIS_Y, W.AXIS_Z))
        area = afc.grid_from_spec(spec)
        pts = O.grid_points(dim, *spec.lo_hi(), spec.res, spec.axes)
        assert len(pts) == grid[0] * grid[1] * grid[2]
    else:
        pts = np.empty((m, 3), np.float32)
        pts[:, :2] = cen[:2] + rng.uniform(-100, 100, (m, 2))
        pts[:, 2] = rng.uniform(50, 200, m)
        area = afc.ScatterArea()
        area.add_observe_points(pts)
    out = afc.GpuCalculator().calculate(s, area, afc.ComplexPressureFieldBuffer())
    ref = O.field_f32(st, rec, k, a, pts, O.FIELD_COMPLEX)
    err = float(np.max(np.abs(np.asarray(out).reshape(-1) - ref)) / np.max(np.abs(ref)))
    print(f"st={st} n={n} {grid or m}: {err:.2e}")
    assert err <= 1e-4


@pytest.mark.parametrize("n,m", [(1, 33000), (3, 1), (249, 45954), (249, 281124), (249, 281125),
                                 (1023, 33001), (1023, 70001), (1024, 40000), (1537, 515)])
def test_sphere_scatter(gpu, n, m):
    _check(gpu, 0, n, m=m)


@pytest.mark.parametrize("n,grid", [(249, (163, 124, 1)), (249, (55, 67, 16)), (498, (218, 123, 2)),
                                    (1023, (90, 33, 13)), (1023, (287, 250, 1)), (1026, (65, 67, 9))])
def test_sphere_grids(gpu, n, grid):
    _check(gpu, 0, n, grid=grid)


@pytest.mark.parametrize("n,grid", [(768, (64, 42, 2)), (768, (125, 144, 1)), (996, (44, 45, 9)),
                                    (996, (49, 32, 9)), (1023, (155, 110, 1)), (767, (101, 101, 1))])
def test_t4010a1_grids_of_either_pairs(gpu, n, grid):
    _check(gpu, 1, n, grid=grid)
