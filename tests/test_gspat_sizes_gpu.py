"""GS-PAT around the sizes where its kernels change: one warp (8 foci), the register columns of the
single-block iteration (16, 32, 48, 64), the cluster iteration (65; 128, 256 and 384 with R in
registers, 385 with R in L2), partial 4 x 4 tiles of R and partial chunks of 64 foci, with source
counts that leave partial blocks of 32 columns.

Tolerance: GS-PAT amplifies rounding where the foci make R ill-conditioned, so the drive must lie
within max(1e-4, 3 times the float32 restatement's own distance) of float64, in units of its peak.
The foci are drawn from a 300 x 300 x 200 mm box, where they are far apart for a wavelength of 8.5 mm.
"""
import numpy as np
import pytest

import oracle as O
import workloads as W

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("st,tiles,m", [
    (1, (2, 2), 1), (1, (2, 2), 9), (0, (2, 2), 16), (1, (1, 1), 17), (1, (2, 2), 33), (1, (2, 2), 49),
    (1, (2, 2), 65), (0, (1, 1), 66), (1, (2, 2), 96), (1, (2, 2), 127), (1, (2, 2), 129),
    (1, (5, 2), 256), (1, (5, 2), 257), (0, (5, 2), 385),
])
def test_gspat_sizes(gpu, st, tiles, m):
    afc = gpu
    rng = np.random.default_rng(1000 + m)
    pos = W.tiled_array(*tiles)
    n = len(pos)
    cen = W.array_center(pos)
    amp = rng.uniform(0.5, 1.0, n).astype(np.float32) * np.where(np.arange(n) % 7 == 0, -1, 1)
    rec = (W.t4010a1_records if st == 1 else W.sphere_records)(pos, amp.astype(np.float32), 0.3)
    k = np.full(n, W.wavenumber(), np.float32)
    a = np.full(n, 1e-3, np.float32)
    foci = np.empty((m, 3), np.float32)
    foci[:, :2] = cen[:2] + rng.uniform(-150, 150, (m, 2))
    foci[:, 2] = rng.uniform(100, 300, m)
    amps = rng.uniform(0.5, 1.0, m).astype(np.float32)
    s = afc.UniformSystem(300.0)
    s.add_records(st, rec, k, a)
    afc.Optimizer.gs_pat(s, foci, amps)
    got = s.records()
    i = 6 if st == 1 else 3
    q = got[:, i].astype(np.float64) * np.exp(1j * got[:, i + 1].astype(np.float64))
    _, q64 = O.gspat_f64(st, rec, k, a, foci, amps)
    _, q32 = O.gspat_f32(st, rec, k, a, foci, amps)
    peak = np.max(np.abs(q64))
    e, e32 = np.max(np.abs(q - q64)) / peak, np.max(np.abs(q32 - q64)) / peak
    print(f"GS-PAT st={st} n={n} m={m}: {e:.2e} of the peak drive (f32 restatement {e32:.2e})")
    assert e <= max(1e-4, 3 * e32)
