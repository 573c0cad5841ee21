"""The rows body's warp boxes and directivity polynomials against the oracle: grids around the
box sizes (8 x 8 x 4 points of a volume, 16 x 16 of a slice), spacings from where almost every
(warp, source) pair takes a polynomial to where almost none does, distances down to boxes that
touch a source, and every source type and direction.

Tolerance: the stated bar, max |p_gpu - p_ref| <= 1e-4 max |p_ref| against the float32 oracle.  A
polynomial is within 2e-7 of the directivity (at most 1), so a field of n sources moves by less
than 2e-7 of the sum of the terms' moduli.
"""
import ctypes

import numpy as np
import pytest

import oracle as O
import workloads as W

pytestmark = pytest.mark.gpu


def _grid(counts, res, lo, axes=(1, 2, 3)):
    """A grid of exactly `counts` points along x, y, z (f32 counts padded by half a step)."""
    hi = [a + (c - 1) * res + 0.5 * res if c > 1 else a for a, c in zip(lo, counts)]
    dim = 3 if min(counts) > 1 else 2
    ranges = [(lo[a - 1], hi[a - 1]) for a in axes]
    return W.GridSpec(dim, ranges, res, axes)


@pytest.mark.parametrize("st,tilted", [(0, False), (1, False), (1, True)])
@pytest.mark.parametrize("counts,res,z0", [
    ((64, 64, 16), 0.25, 60.0),   # whole boxes, nearly every pair a polynomial
    ((33, 65, 17), 0.5, 50.0),    # one past the box along every axis
    ((200, 161, 1), 0.5, 150.0),  # slices: 16 x 16 boxes, ragged ends
    ((181, 182, 1), 4.0, 90.0),   # wide spacing: the table nearly everywhere
    ((31, 40, 40), 1.0, 2.0),     # boxes beside and around the sources
])
def test_boxes_and_spacings(gpu, st, tilted, counts, res, z0):
    afc = gpu
    torch = pytest.importorskip("torch")
    rng = np.random.default_rng(sum(counts) + st)
    pos = W.tiled_array(2, 2)
    n = len(pos)
    cen = W.array_center(pos)
    amp, ph = W.random_pattern(rng, n)
    rec = (W.t4010a1_records if st == 1 else W.sphere_records)(pos, amp, ph)
    if tilted:
        d = rng.normal(size=(n, 3)) * 0.3 + np.array([0.0, 0.0, 1.0])
        rec[:, 3:6] = d / np.linalg.norm(d, axis=1, keepdims=True)
    k = np.full(n, W.wavenumber(), np.float32)
    a = np.full(n, 1.15e-2, np.float32)
    spec = _grid(counts, res, [float(cen[0]) - counts[0] * res / 2,
                               float(cen[1]) - counts[1] * res / 2, z0])
    area = afc.grid_from_spec(spec)
    desc = area.grid_desc()
    assert tuple(desc.count) == tuple(counts)
    m = int(np.prod(counts))
    d_src, d_k, d_a = (torch.from_numpy(x.reshape(-1)).cuda() for x in (rec, k, a))
    out = torch.empty(2 * m, device="cuda")
    wsb = afc.DLL.AFC_FieldWorkspaceBytes(n)
    ws = torch.empty(wsb, dtype=torch.uint8, device="cuda")
    lo, hi = spec.lo_hi()
    pts = O.grid_points(spec.dim, lo, hi, spec.res, spec.axes)
    sel = rng.choice(m, min(m, 4000), replace=False)
    ref = O.field_f32(st, rec, k, a, pts[sel], O.FIELD_COMPLEX)
    for sum_mode in (0, 1):
        rc = afc.DLL.AFC_FieldGridDevice(st, 2, sum_mode, d_src.data_ptr(), d_k.data_ptr(),
                                         d_a.data_ptr(), n, ctypes.byref(desc), out.data_ptr(),
                                         ws.data_ptr(), wsb,
                                         torch.cuda.current_stream().cuda_stream)
        assert rc == 0, afc.last_error()
        torch.cuda.synchronize()
        p = out.cpu().numpy().view(np.complex64)[sel]
        err = float(np.max(np.abs(p - ref)) / np.max(np.abs(ref)))
        print(f"{counts} res {res} st {st} tilted {tilted} sum {sum_mode}: {err:.2e}")
        assert err <= 1e-4
