"""Levenberg-Marquardt's and Gauss-Newton's first step, value by value, against float64 on the G that
the device built: K = B B^H and its largest column, the step h, and at the point it leads to F, max Jtf, |x|^2,
|h|^2, the gain's denominator, Jtf, U Jtf and L.  Sizes around the launches' edges: n across K's chunk of
1,024 columns, one focus, a full and a partial second block of 32 rows, and more than 1,024 entries of L.

Tolerances: a float32 sum of n terms in 32 lanes (or 1,024 threads) is within (n / 32 + 10) 2^-24 of the sum
of its terms' magnitudes, plus four roundings a term; a sum of computed values adds their errors.  t = exp(i x)
is within 2^-23 and the term's magnitudes bound every value, so each is compared with that bound times
the magnitudes' sum.  K is exact in its products: a double's n 2^-53.  h solves (M + mu) y = U Jtf in double
with M from K and L: it is within the condition of M + mu times 2^-17, 128 roundings of the float32 sums.
"""
import ctypes

import numpy as np
import pytest

import workloads as W

pytestmark = pytest.mark.gpu

EPS = 2.0 ** -24


def step(afc, lm, st, rec, k, a, foci, amps):
    from afc import nativemethods as nm

    n, m = len(k), len(amps)
    o = dict(g=np.empty((m, n), np.complex64), k=np.empty((m, m), np.complex128), a_max=np.empty(1),
             x=np.empty(n + m, np.float32), h=np.empty(n + m, np.float32),
             jtf0=np.empty(n + m, np.float32), jtf=np.empty(n + m, np.float32),
             scalars=np.empty(5, np.float32), u_jtf=np.empty(2 * m, np.float32),
             l=np.empty((m, m), np.complex64))
    out = nm.NlsStep(**{name: v.ctypes.data for name, v in o.items()})
    args = [np.ascontiguousarray(v, np.float32) for v in (rec, k, a, foci, amps)]
    rc = afc.DLL.AFO_NlsStepTest(lm, st, *(v.ctypes.data for v in args[:3]), n, args[3].ctypes.data,
                                 args[4].ctypes.data, m, ctypes.byref(out))
    assert rc == 0, afc.last_error()
    return o


def problem(st, n, m):
    rng = np.random.default_rng(7 * n + m)
    pos = W.tiled_array(5, 2)[:n]
    cen = pos.mean(axis=0)
    rec = (W.t4010a1_records if st == 1 else W.sphere_records)(pos, 1.0, 0.4)
    foci = np.empty((m, 3), np.float32)
    foci[:, :2] = cen[:2] + rng.uniform(-60, 60, (m, 2))
    foci[:, 2] = rng.uniform(80, 160, m)
    return (rec, np.full(n, W.wavenumber(), np.float32), np.full(n, 1e-3, np.float32), foci,
            rng.uniform(0.2, 0.5, m).astype(np.float32))


def within(name, got, ref, bound):
    err = np.abs(np.asarray(got, np.complex128) - ref)
    worst = float(np.max(err / np.maximum(bound, 1e-300)))
    print(f"  {name}: {worst:.3f} of the bound")
    assert np.all(err <= bound), name


@pytest.mark.parametrize("lm", [1, 0])
@pytest.mark.parametrize("st,n,m", [(1, 1, 1), (0, 130, 1), (1, 1023, 5), (1, 1024, 32), (0, 1025, 33),
                                    (1, 2490, 65), (1, 700, 32), (0, 2490, 1)])
def test_first_step(gpu, lm, st, n, m):
    rec, k, a, foci, amps = problem(st, n, m)
    o = step(gpu, lm, st, rec, k, a, foci, amps)
    s = (n / 32 + 14) * EPS  # of a sum of n float32 terms, a term's own roundings included
    g = o["g"].astype(np.complex128)
    p = amps.astype(np.float64)
    B = np.hstack([g, -np.diag(p)])
    aB = np.abs(B)
    # K and the largest diagonal entry of JtJ
    K = B @ B.conj().T
    within("K", o["k"], K, 2 * (n + m) * 2.0 ** -53 * (aB @ aB.T))
    amax = np.max(np.sum(aB ** 2, axis=0))
    within("a_max", o["a_max"][0], amax, (m + 4) * 2.0 ** -52 * amax)

    def at(x):
        t = np.exp(1j * x)
        r = B @ t
        return t, r, np.imag(t * (r.conj() @ B))  # Im(t_b conj((B^H r)_b))

    R = aB.sum(axis=1)            # a row's magnitudes
    rb = (s + 4 * EPS) * R        # r's bound
    # Jtf_b sums m terms conj(B_ib) r_i
    jb = aB.T @ (rb + (m + 8) * EPS * R)
    _, _, j0 = at(np.zeros(n + m))
    within("Jtf at 0", o["jtf0"], j0, jb)
    x = o["x"].astype(np.float64)
    h = o["h"].astype(np.float64)
    assert np.array_equal(o["x"], o["h"])  # from x = 0
    t, r, j = at(x)
    within("Jtf", o["jtf"], j, jb)
    sc = o["scalars"].astype(np.float64)
    within("F", sc[0], np.sum(np.abs(r) ** 2), np.sum(2 * np.abs(r) * rb + rb ** 2 + (m + 14) * EPS * R ** 2))
    within("max Jtf", sc[1], np.max(j), np.max(jb))
    within("|x|^2", sc[2], np.sum(x * x), 2 * s * np.sum(x * x))
    within("|h|^2", sc[3], np.sum(h * h), 2 * s * np.sum(h * h))
    mu = 1e-3 * o["a_max"][0]
    jj = o["jtf0"].astype(np.float64)
    within("h.(mu h - Jtf)", sc[4], np.sum(h * (mu * h - jj)),
           2 * s * np.sum(np.abs(h) * (mu * np.abs(h) + np.abs(jj))))
    C = B * t
    jf = o["jtf"].astype(np.float64)
    ub = (s + 8 * EPS) * (aB @ np.abs(jf)) + 4 * EPS * (aB @ np.abs(jf))
    within("U Jtf", o["u_jtf"], np.concatenate([C.real @ jf, C.imag @ jf]), np.concatenate([ub, ub]))
    within("L", o["l"], C @ C.T, (s + 16 * EPS) * (aB @ aB.T))
    if lm:
        # h = -(Jtf0 - U^T y) / mu, (mu + U U^T) y = U Jtf0 at x = 0
        U = np.vstack([B.real, B.imag])
        M = U @ U.T
        y = np.linalg.solve(M + mu * np.eye(2 * m), U @ j0)
        ref = -(j0 - U.T @ y) / mu
        lam = np.linalg.eigvalsh(M)
        cond = (lam[-1] + mu) / max(mu, lam[0] + mu)
        e = np.linalg.norm(h - ref) / np.linalg.norm(ref)
        print(f"  h: {e:.2e} of |h|, cond {cond:.1e}")
        assert e <= cond * 2.0 ** -17


def test_many_columns(gpu):
    """One focus and more sources than a grid has rows of 128 columns (8.39 million).  Only K and a_max, the
    largest of the |G|^2 and of the focus amplitude's square, are compared: the columns' launch alone
    depends on their number."""
    n = 8_400_000
    rng = np.random.default_rng(1)
    rec = np.zeros((n, 6), np.float32)
    rec[:, :2] = rng.uniform(0, 500, (n, 2)).astype(np.float32)
    rec[:, 3], rec[:, 5] = 1.0, 40000.0
    rec[n - 3, :3] = (250, 250, 97)  # the nearest source is one of the last
    foci, amps = np.float32([[250, 250, 100]]), np.float32([0.3])
    o = step(gpu, 1, 0, rec, np.full(n, W.wavenumber(), np.float32), np.zeros(n, np.float32), foci, amps)
    g2 = np.abs(o["g"][0].astype(np.complex128)) ** 2
    assert abs(g2[n - 3] - 1 / 9) < 1e-5 and np.argmax(g2) == n - 3
    within("a_max", o["a_max"][0], g2.max(), 4 * 2.0 ** -52 * g2.max())
    k = g2.sum() + float(amps[0]) ** 2
    within("K", o["k"][0, 0], k, 2 * n * 2.0 ** -53 * k)
