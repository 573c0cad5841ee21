"""The host's eigenvector of the largest eigenvalue (Horn's last step) against numpy's eigh: full
matrices, matrices that fall into decoupled parts, and the identity (equal eigenvalues: the first).

Tolerance: both solvers are backward stable, so each vector is exact for a matrix within about
k eps ||A|| of A and turns by that over the gap to the next eigenvalue; 20 k eps ||A|| / gap is allowed.
"""
import ctypes
import os
import subprocess

import numpy as np
import pytest

CSRC = os.path.join(os.path.dirname(os.path.abspath(__file__)), "..", "acoustic-field-calculator_gb300",
                    "csrc")
WRAPPER = """
#include "dense_host.h"
extern "C" void principal(const double* a, int k, double* out) {
    std::vector<std::complex<double>> m(static_cast<size_t>(k) * k), v;
    for (size_t i = 0; i < m.size(); ++i) m[i] = {a[2 * i], a[2 * i + 1]};
    afc::dense::principal_eigenvector(m, k, v);
    for (int i = 0; i < k; ++i) out[2 * i] = v[i].real(), out[2 * i + 1] = v[i].imag();
}
"""


@pytest.fixture(scope="module")
def principal(tmp_path_factory):
    d = tmp_path_factory.mktemp("eig")
    (d / "w.cpp").write_text(WRAPPER)
    so = str(d / "w.so")
    subprocess.run(["g++", "-O3", "-std=c++17", "-ffp-contract=off", "-shared", "-fPIC", "-I", CSRC,
                    str(d / "w.cpp"), "-o", so], check=True)
    fn = ctypes.CDLL(so).principal

    def call(a):
        a = np.ascontiguousarray(a, np.complex128)
        out = np.empty(len(a), np.complex128)
        fn(a.ctypes.data_as(ctypes.c_void_p), len(a), out.ctypes.data_as(ctypes.c_void_p))
        return out
    return call


@pytest.mark.parametrize("kind", ["full", "decoupled", "tail", "identity"])
@pytest.mark.parametrize("k", [1, 2, 3, 8, 31, 64, 129])
def test_principal_eigenvector(principal, kind, k):
    rng = np.random.default_rng(k)
    u = np.exp(2j * np.pi * rng.uniform(size=k))
    a = 0.5 * np.outer(u, u.conj()) + 0.1 * (rng.normal(size=(k, k)) + 1j * rng.normal(size=(k, k)))
    i = np.arange(k)
    if kind == "decoupled":  # every third coordinate apart from the others
        a[(i % 3 == 1)[:, None] != (i % 3 == 1)[None, :]] = 0
    if kind == "tail":       # the first two coordinates alone
        a[:2], a[:, :2] = 0, 0
    if kind == "identity":
        a[:] = 0
    a = np.tril(a, -1)
    a = a + a.conj().T + np.eye(k)
    lam, vec = np.linalg.eigh(a)
    got = principal(a)
    if np.array_equal(a, np.eye(k)):  # also two coordinates apart: equal eigenvalues
        assert np.array_equal(got, np.eye(k)[0])
        return
    ref = vec[:, -1]
    first = np.flatnonzero(np.abs(ref) > 1e-12)[0]
    ref = ref * (abs(ref[first]) / ref[first])
    gap = lam[-1] - lam[-2] if k > 1 else 1.0
    err = np.max(np.abs(got - ref))
    assert err <= 20 * k * np.finfo(float).eps * np.max(np.abs(lam)) / gap
    assert got[first].imag == 0 and got[first].real > 0
