"""Levenberg-Marquardt around the sizes of its step's launches (one focus, more columns than 1,024
strided threads take at once, partial blocks of 128 columns and of 32 rows, more than 32 foci): the
phases alone change, every value is finite, and problems of other sizes in between, larger and
smaller, change no bit of a result (its device and pinned blocks are kept between calls).

The values are compared with float64 in test_nls_gpu.py.  At these sizes 200 float32 steps from the
zero drive end too far from 200 float64 steps for a bound to say anything (one focus and 249 sources:
1.2 % of |p|), and the iteration does not lower the focal amplitudes' distance from their targets
(the float64 one neither), so nothing more is asked here.
"""
import numpy as np
import pytest

import workloads as W

pytestmark = pytest.mark.gpu

SIZES = [(1, (1, 1), 1), (0, (1, 1), 7), (1, (5, 2), 5), (1, (1, 1), 33)]


def _problem(st, tiles, m):
    rng = np.random.default_rng(500 + m)
    pos = W.tiled_array(*tiles)
    n = len(pos)
    cen = W.array_center(pos)
    rec = (W.t4010a1_records if st == 1 else W.sphere_records)(pos, 1.0, 0.4)
    foci = np.empty((m, 3), np.float32)
    foci[:, :2] = cen[:2] + rng.uniform(-40, 40, (m, 2))
    foci[:, 2] = rng.uniform(100, 160, m)
    return (rec, np.full(n, W.wavenumber(), np.float32), np.zeros(n, np.float32), foci,
            rng.uniform(0.2, 0.5, m).astype(np.float32))


def _solve(afc, st, rec, k, a, foci, amps):
    s = afc.UniformSystem(300.0)
    s.add_records(st, rec, k, a)
    afc.Optimizer.lm(s, foci, amps)
    return s.records().copy()


@pytest.mark.parametrize("st,tiles,m", SIZES)
def test_lm_sizes(gpu, st, tiles, m):
    problem = _problem(st, tiles, m)
    rec, k, a, foci, amps = problem
    got = _solve(gpu, st, *problem)
    i = 7 if st == 1 else 4
    np.testing.assert_array_equal(got[:, :i], rec[:, :i])  # the phases alone change
    assert np.all(np.isfinite(got))
    for other in SIZES:
        if other != (st, tiles, m):
            _solve(gpu, other[0], *_problem(*other))
    np.testing.assert_array_equal(_solve(gpu, st, *problem), got)
