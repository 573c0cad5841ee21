"""Horn around the sizes where its SDP kernel changes: rows a warp (8, 16, 32 coordinates), columns a
lane (32, 64, 96, 128), and x in L2 (129), against the oracle's float64 steps.

Tolerance: the drive within max(1e-3, 3 d) of the float64 one in units of its peak, with d the distance
that float64 Horn itself moves when G is perturbed by 1e-5 of each entry, about the accuracy of the
float32 G (its phases k r of some hundred radians): the regularised inverse magnifies that where
the foci are close for the wavelength.
"""
import numpy as np
import pytest

import oracle as O
import workloads as W

pytestmark = pytest.mark.gpu


def _horn64(g, amps):
    m = len(amps)
    mm, g_pinv = O.horn_mm_f64(g, amps)
    x = O.horn_sdp_f64(mm, O.horn_indices(m, 100 * m))
    u = np.linalg.eigh(x)[1][:, -1]
    u = u * (abs(u[0]) / u[0])  # the first entry real and positive
    q = g_pinv @ (amps * u)
    return q / np.max(np.abs(q.real) + np.abs(q.imag))


@pytest.mark.parametrize("st,m", [(1, 1), (1, 9), (0, 16), (1, 17), (1, 32), (1, 33), (1, 65), (1, 96),
                                  (1, 97), (1, 129)])
def test_horn_sizes(gpu, st, m):
    afc = gpu
    rng = np.random.default_rng(2000 + m)
    pos = W.tiled_array(2, 2)
    n = len(pos)
    cen = W.array_center(pos)
    rec = (W.t4010a1_records if st == 1 else W.sphere_records)(pos, 1.0, 0.0)
    k = np.full(n, W.wavenumber(), np.float32)
    a = np.zeros(n, np.float32)
    foci = np.empty((m, 3), np.float32)
    foci[:, :2] = cen[:2] + rng.uniform(-150, 150, (m, 2))
    foci[:, 2] = rng.uniform(100, 300, m)
    amps = rng.uniform(0.5, 1.0, m).astype(np.float32)
    s = afc.UniformSystem(300.0)
    s.add_records(st, rec, k, a)
    afc.Optimizer.horn(s, foci, amps)
    got = s.records()
    i = 6 if st == 1 else 3
    q = got[:, i].astype(np.float64) * np.exp(1j * got[:, i + 1].astype(np.float64))
    g = O.build_g_f64(st, rec, k, a, foci)
    noise = rng.normal(size=g.shape) + 1j * rng.normal(size=g.shape)
    ref, moved = (_horn64(x, amps.astype(np.float64)) for x in (g, g * (1 + 1e-5 * noise)))
    e, d = (float(np.max(np.abs(x - ref)) / np.max(np.abs(ref))) for x in (q, moved))
    print(f"Horn st={st} m={m}: {e:.2e} of the peak drive (1e-5 of G moves it {d:.2e})")
    assert e <= max(1e-3, 3 * d)
