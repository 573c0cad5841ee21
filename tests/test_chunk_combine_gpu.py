"""The sums of a chunked launch around its two combine kernels: few points of up to a GPU's blocks of
segments (one point, a warp's 32 points and one more, two tiles, several), and more points, whose
segments are fewer than the wide kernel takes; some points lie on a source (NaN sums).
Against the oracle; tolerance: the stated bar, 1e-4 of the peak finite |p|.
"""
import numpy as np
import pytest

import oracle as O
import workloads as W

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("st", [0, 1])
@pytest.mark.parametrize("m", [1, 32, 33, 2049, 12289, 20480, 20481, 78000])
def test_chunk_combine(gpu, st, m):
    afc = gpu
    rng = np.random.default_rng(77 + m)
    n = 1600
    pos = W.tiled_array(4, 2)[:n]
    n = len(pos)
    amp = rng.uniform(0.2, 1.0, n).astype(np.float32)
    ph = rng.uniform(-np.pi, np.pi, n).astype(np.float32)
    rec = (W.t4010a1_records if st else W.sphere_records)(pos, amp, ph)
    k = np.full(n, W.wavenumber(), np.float32)
    a = np.full(n, 1.15e-2, np.float32)
    pts = np.empty((m, 3), np.float32)
    pts[:, :2] = pos.mean(axis=0)[:2] + rng.uniform(-100, 100, (m, 2))
    pts[:, 2] = rng.uniform(50, 200, m)
    on = np.unique(rng.integers(0, m, 5)) if m > 1 else np.zeros(0, int)
    pts[on] = pos[: len(on)]
    s = afc.UniformSystem(300.0)
    s.add_records(st, rec, k, a)
    area = afc.ScatterArea()
    area.add_observe_points(pts)
    out = np.asarray(afc.GpuCalculator().calculate(s, area, afc.ComplexPressureFieldBuffer()))
    with np.errstate(all="ignore"):
        ref = O.field_f32(st, rec, k, a, pts, O.FIELD_COMPLEX)
    for part in (np.real, np.imag):
        o, r = part(out), part(ref).astype(np.float32)
        np.testing.assert_array_equal(np.isnan(o), np.isnan(r))
        np.testing.assert_array_equal(np.isinf(o), np.isinf(r))
        np.testing.assert_array_equal(o[np.isinf(r)], r[np.isinf(r)])
    finite = np.isfinite(ref.real) & np.isfinite(ref.imag)
    assert finite.sum() == m - len(on)
    err = float(np.max(np.abs(out - ref)[finite]) / np.max(np.abs(ref[finite])))
    print(f"st={st} m={m}: {err:.2e}")
    assert err <= 1e-4
