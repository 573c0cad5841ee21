"""AFC_MultiPatternBuildG around its blocks (512 sources, 2 to 32 points), its padding and the FP16
row scales' source boxes (64 sources; one box up to 512 sources), against the oracle's float32 field of
every pattern (float64 is no reference here: it puts pairs next to a directivity bin edge into the
other bin, and one such term among 1,025 tilted sources is 2.5e-3 of the peak).

Bars: those of the form (max |P - P_ref| / max |P_ref|): split BF16 1e-4, FP16 1e-3.  A row scale that
missed a row's largest |G| by more than a factor of two would overflow nothing, but one that came
out too small would: the FP16 rows are also checked to be finite.
"""
import numpy as np
import pytest

import oracle as O
import workloads as W

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("prec,bar", [(1, 1e-4), (2, 1e-3)])
@pytest.mark.parametrize("st,n,m,K", [
    (1, 1, 1, 1), (0, 2, 3, 5), (1, 31, 33, 3), (1, 33, 17, 130), (1, 511, 257, 9), (1, 513, 300, 9),
    (0, 577, 65, 8), (1, 1025, 1000, 8), (1, 2490, 640, 16),
])
def test_build_g_sizes(gpu, prec, bar, st, n, m, K):
    torch = pytest.importorskip("torch")
    afc = gpu
    rng = np.random.default_rng(n + m)
    pos = W.tiled_array(5, 2)[:n] if n > 600 else rng.uniform(-80, 80, (n, 3)).astype(np.float32)
    if n <= 600:
        pos[:, 2] = rng.uniform(-5, 5, n)
    cen = pos.mean(axis=0)
    rec = (W.t4010a1_records if st == 1 else W.sphere_records)(pos, 1.0, 0.0)
    if st == 1 and n % 2:
        d = rng.normal(size=(n, 3)) * 0.3 + np.array([0.0, 0.0, 1.0])
        rec[:, 3:6] = d / np.linalg.norm(d, axis=1, keepdims=True)
    k = rng.uniform(0.70, 0.75, n).astype(np.float32)
    a = rng.uniform(0.0, 1.2e-2, n).astype(np.float32)
    pts = np.empty((m, 3), np.float32)
    pts[:, :2] = cen[:2] + rng.uniform(-100, 100, (m, 2))
    pts[:, 2] = rng.uniform(20, 200, m)
    amps = rng.uniform(0.5, 1.0, (K, n)).astype(np.float32)
    phases = rng.uniform(0, 2 * np.pi, (K, n)).astype(np.float32)
    t = [torch.from_numpy(np.ascontiguousarray(x).reshape(-1)).cuda() for x in (rec, k, a, pts, amps, phases)]
    wsb = afc.DLL.AFC_MultiPatternWorkspaceBytes(n, m, K, prec)
    ws = torch.full((wsb + 256,), 0xFF, dtype=torch.uint8, device="cuda")  # NaN where nothing is written
    base = (ws.data_ptr() + 255) // 256 * 256
    out = torch.empty(2 * m * K, device="cuda")
    stream = torch.cuda.current_stream().cuda_stream
    rc = afc.DLL.AFC_MultiPatternBuildG(st, prec, t[0].data_ptr(), t[1].data_ptr(), t[2].data_ptr(), n,
                                        t[3].data_ptr(), m, K, base, wsb, stream)
    assert rc == 0, afc.last_error()
    rc = afc.DLL.AFC_MultiPatternApply(prec, t[4].data_ptr(), t[5].data_ptr(), n, m, K, out.data_ptr(),
                                       base, wsb, stream)
    assert rc == 0, afc.last_error()
    assert afc.DLL.AFC_MultiPatternStatus(prec, n, m, K, base, stream) == 0
    p = out.cpu().numpy().view(np.complex64).reshape(m, K)
    assert np.all(np.isfinite(p))
    i = 6 if st == 1 else 3
    ref = np.empty((m, K), np.complex128)
    for q in range(K):
        pat = rec.copy()
        pat[:, i], pat[:, i + 1] = amps[q], phases[q]
        ref[:, q] = O.field_f32(st, pat, k, a, pts, O.FIELD_COMPLEX)
    err = float(np.max(np.abs(p - ref)) / np.max(np.abs(ref)))
    print(f"st={st} n={n} m={m} K={K} precision {prec}: {err:.2e}")
    assert err <= bar
