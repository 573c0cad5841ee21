"""The transfer matrix's padding columns (AFC_MultiPatternBuildG rounds the sources up) are zero for
every point, so a row's patterns are finite wherever its sources' fields are: also at a point as far
along x as a stand-in for a missing source might lie.  Source counts that fill none, half and all of a
warp's columns, and that leave a thread with one source.

Tolerance: the stated bars for the near points; a far row must be finite and at most the sum of its
sources' amplitudes over their distance, which is 9.9e7 or more (D <= 1; 1 % for the 16-bit elements).
"""
import numpy as np
import pytest

import oracle as O
import workloads as W

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("prec,bar", [(1, 1e-4), (2, 1e-3)])
@pytest.mark.parametrize("st", [0, 1])
@pytest.mark.parametrize("n", [1, 32, 49, 249, 300, 498])
def test_padding_is_zero(gpu, prec, bar, st, n):
    torch = pytest.importorskip("torch")
    afc = gpu
    rng = np.random.default_rng(n)
    pos = W.tiled_array(2, 1)[:n]
    rec = (W.t4010a1_records if st == 1 else W.sphere_records)(pos, 1.0, 0.0)
    k, a = np.full(n, W.wavenumber(), np.float32), np.zeros(n, np.float32)
    m, K = 70, 4
    pts = rng.uniform(-60, 60, (m, 3)).astype(np.float32) + np.float32([60, 60, 160])
    far = np.float32([[1e8, 0, 0], [0, 1e8, 0], [-1e8, 0, 0], [1e8, 1e8, 1e8], [9.9999992e7, 0, 0]])
    rows = [0, 3, 31, 32, 69]
    pts[rows] = far
    amps = rng.uniform(0.5, 1.0, (K, n)).astype(np.float32)
    phases = rng.uniform(0, 2 * np.pi, (K, n)).astype(np.float32)
    t = [torch.from_numpy(np.ascontiguousarray(x).reshape(-1)).cuda() for x in (rec, k, a, pts, amps, phases)]
    wsb = afc.DLL.AFC_MultiPatternWorkspaceBytes(n, m, K, prec)
    ws = torch.full((wsb + 256,), 0xFF, dtype=torch.uint8, device="cuda")
    base = (ws.data_ptr() + 255) // 256 * 256
    out = torch.empty(2 * m * K, device="cuda")
    stream = torch.cuda.current_stream().cuda_stream
    rc = afc.DLL.AFC_MultiPatternBuildG(st, prec, t[0].data_ptr(), t[1].data_ptr(), t[2].data_ptr(), n,
                                        t[3].data_ptr(), m, K, base, wsb, stream)
    assert rc == 0, afc.last_error()
    rc = afc.DLL.AFC_MultiPatternApply(prec, t[4].data_ptr(), t[5].data_ptr(), n, m, K, out.data_ptr(),
                                       base, wsb, stream)
    assert rc == 0, afc.last_error()
    p = out.cpu().numpy().view(np.complex64).reshape(m, K)
    assert np.all(np.isfinite(p)), np.unique(np.argwhere(~np.isfinite(p))[:, 0])
    near = np.setdiff1d(np.arange(m), rows)
    i = 6 if st == 1 else 3
    ref = np.empty((m, K), np.complex128)
    for q in range(K):
        pat = rec.copy()
        pat[:, i], pat[:, i + 1] = amps[q], phases[q]
        ref[:, q] = O.field_f32(st, pat, k, a, pts, O.FIELD_COMPLEX)
    peak = np.max(np.abs(ref[near]))
    assert np.max(np.abs(p[near] - ref[near])) <= bar * peak
    assert np.all(np.abs(p[rows]) <= 1.01 * amps.sum(axis=1) / 9.9e7)


@pytest.mark.parametrize("st,n,m", [(1, 513, 1519), (1, 513, 1520), (0, 1025, 1600), (1, 249, 1530), (0, 2, 1519),
                                    (1, 600, 1)])
def test_row_scales_either_way(gpu, st, n, m):
    """FP16's row scales below and from 10 rows an SM (1,520 on 152), where a row's largest |G| is sought by a
    block and by a warp: the bar of the form, and rows that are finite."""
    torch = pytest.importorskip("torch")
    afc = gpu
    rng = np.random.default_rng(n + m)
    pos = W.tiled_array(5, 2)[:n]
    rec = (W.t4010a1_records if st == 1 else W.sphere_records)(pos, 1.0, 0.0)
    k, a = np.full(n, W.wavenumber(), np.float32), rng.uniform(0, 1.2e-2, n).astype(np.float32)
    pts = (pos.mean(axis=0) + rng.uniform(-90, 90, (m, 3)) + [0, 0, 120]).astype(np.float32)
    K = 3
    amps = rng.uniform(0.5, 1.0, (K, n)).astype(np.float32)
    phases = rng.uniform(0, 2 * np.pi, (K, n)).astype(np.float32)
    t = [torch.from_numpy(np.ascontiguousarray(x).reshape(-1)).cuda() for x in (rec, k, a, pts, amps, phases)]
    wsb = afc.DLL.AFC_MultiPatternWorkspaceBytes(n, m, K, 2)
    ws = torch.full((wsb + 256,), 0xFF, dtype=torch.uint8, device="cuda")
    base = (ws.data_ptr() + 255) // 256 * 256
    out = torch.empty(2 * m * K, device="cuda")
    stream = torch.cuda.current_stream().cuda_stream
    rc = afc.DLL.AFC_MultiPatternBuildG(st, 2, t[0].data_ptr(), t[1].data_ptr(), t[2].data_ptr(), n,
                                        t[3].data_ptr(), m, K, base, wsb, stream)
    assert rc == 0, afc.last_error()
    rc = afc.DLL.AFC_MultiPatternApply(2, t[4].data_ptr(), t[5].data_ptr(), n, m, K, out.data_ptr(), base, wsb,
                                       stream)
    assert rc == 0, afc.last_error()
    p = out.cpu().numpy().view(np.complex64).reshape(m, K)
    assert np.all(np.isfinite(p))
    i = 6 if st == 1 else 3
    for q in range(K):
        pat = rec.copy()
        pat[:, i], pat[:, i + 1] = amps[q], phases[q]
        ref = O.field_f32(st, pat, k, a, pts, O.FIELD_COMPLEX)
        assert np.max(np.abs(p[:, q] - ref)) <= 1e-3 * np.max(np.abs(ref))
