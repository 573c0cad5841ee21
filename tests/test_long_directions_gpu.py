"""T4010A1 directions that are not unit vectors on grids, where cos(theta) leaves [-1, 1]: the reference's
acos is then NaN and its directivity 1 (t4010a1.rs:107-120), on either side.  Sources tilted every way,
points in front, beside and behind; lengths inside and outside what the grid body's table covers, alone and
mixed with unit directions; grids of each pair count and of the cluster split, both sums, batch plans' and
the scatter sets' bodies.

Tolerance: the stated bar, max |p_gpu - p_ref| <= 1e-4 max |p_ref|.
"""
import numpy as np
import pytest

import oracle as O
import workloads as W

pytestmark = pytest.mark.gpu


def _problem(n, lengths, seed, mixed):
    rng = np.random.default_rng(seed)
    pos = rng.uniform(-60, 60, (n, 3)).astype(np.float32)
    pos[:, 2] = rng.uniform(60, 120, n)
    nv = rng.normal(size=(n, 3))
    nv /= np.linalg.norm(nv, axis=1, keepdims=True)
    scale = rng.choice(lengths, n)
    if mixed:
        scale[rng.random(n) < 0.7] = 1.0
    rec = np.zeros((n, 9), np.float32)
    rec[:, :3], rec[:, 3:6] = pos, nv * scale[:, None]
    rec[:, 6], rec[:, 7], rec[:, 8] = rng.uniform(0.3, 1, n), rng.uniform(0, 6, n), 40000
    return rec, np.full(n, W.wavenumber(), np.float32), np.full(n, 1e-3, np.float32)


@pytest.mark.parametrize("calc", ["GpuCalculator", "AccurateCalculator"])
@pytest.mark.parametrize("lengths", [[0.5, 1.0001, 1.3], [1.97, 1.99, 2.0], [2.5, 3.0], [3.5, 10.0, 1e4]])
@pytest.mark.parametrize("n,grid,mixed", [(300, (40, 64, 9), False), (1600, (1, 76, 63), True),
                                          (130, (128, 160, 1), True), (249, (70, 64, 32), True)])
def test_grids(gpu, calc, lengths, n, grid, mixed):
    afc = gpu
    rec, k, a = _problem(n, lengths, n + int(10 * lengths[0]), mixed)
    s = afc.UniformSystem(300.0)
    s.add_records(1, rec, k, a)
    lo = (-20.0, -31.0, 30.0)
    dim = 3 if grid[2] > 1 else 2
    lohi = [(lo[i], lo[i] + (grid[i] - 1) + (0.5 if grid[i] > 1 else 0)) for i in range(3)]
    spec = W.GridSpec(dim, lohi, 1.0, (W.AXIS_X, W.AXIS_Y, W.AXIS_Z))
    pts = O.grid_points(dim, *spec.lo_hi(), spec.res, spec.axes)
    assert len(pts) == grid[0] * grid[1] * grid[2]
    out = getattr(afc, calc)().calculate(s, afc.grid_from_spec(spec), afc.ComplexPressureFieldBuffer())
    ref = O.field_f32(1, rec, k, a, pts, O.FIELD_COMPLEX)
    err = float(np.max(np.abs(np.asarray(out).reshape(-1) - ref)) / np.max(np.abs(ref)))
    print(f"{calc} n={n} {grid} {lengths}: {err:.2e}")
    assert err <= 1e-4
