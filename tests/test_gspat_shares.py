"""The shares of rows of the GS-PAT cluster iteration: contiguous, even starts (rows are stored in pairs),
no block without a row (a block without one does not re-arm the barriers that the others' stores
count on), none above the size that the launch's threads and registers are chosen for."""
import ctypes
import os
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(os.path.abspath(__file__)), "..", "acoustic-field-calculator_gb300",
                    "csrc")
WRAPPER = """
#include "gspat_share.h"
extern "C" long long first(long long m, long long rank) { return afc::iter_first(m, rank); }
extern "C" long long share(long long m) { return afc::iter_share(m); }
extern "C" int blocks() { return afc::kIterCluster; }
"""


@pytest.fixture(scope="module")
def shares(tmp_path_factory):
    d = tmp_path_factory.mktemp("share")
    (d / "w.cpp").write_text(WRAPPER)
    so = str(d / "w.so")
    subprocess.run(["g++", "-O1", "-std=c++17", "-shared", "-fPIC", "-I", CSRC, str(d / "w.cpp"), "-o", so],
                   check=True)
    lib = ctypes.CDLL(so)
    lib.first.argtypes, lib.share.argtypes = [ctypes.c_longlong] * 2, [ctypes.c_longlong]
    lib.first.restype = lib.share.restype = ctypes.c_longlong
    return lib


def test_every_block_has_rows(shares):
    blocks = shares.blocks()
    for m in list(range(65, 400)) + [511, 513, 1000, 1023, 4095, 4096]:
        starts = [min(shares.first(m, r), m) for r in range(blocks + 1)]
        assert starts[0] == 0 and starts[blocks] == m
        sizes = [b - a for a, b in zip(starts, starts[1:])]
        assert min(sizes) >= 1, (m, sizes)
        assert max(sizes) <= shares.share(m), (m, sizes)
        assert all(s % 2 == 0 for s in starts[:blocks])


@pytest.mark.gpu
@pytest.mark.parametrize("m", [70, 84, 97, 98])
def test_gspat_uneven_shares(gpu, m):
    """Focus counts whose rows do not divide over the blocks.  Tolerance as in test_gspat_sizes.py: within
    max(1e-4, 3 times the float32 restatement's own distance) of float64, in units of the peak."""
    import numpy as np

    import oracle as O
    import workloads as W

    rng = np.random.default_rng(2000 + m)
    pos = W.tiled_array(2, 2)
    n = len(pos)
    cen = W.array_center(pos)
    rec = W.t4010a1_records(pos, rng.uniform(0.5, 1.0, n).astype(np.float32), 0.3)
    k, a = np.full(n, W.wavenumber(), np.float32), np.full(n, 1e-3, np.float32)
    foci = np.empty((m, 3), np.float32)
    foci[:, :2] = cen[:2] + rng.uniform(-150, 150, (m, 2))
    foci[:, 2] = rng.uniform(100, 300, m)
    amps = rng.uniform(0.5, 1.0, m).astype(np.float32)
    s = gpu.UniformSystem(300.0)
    s.add_records(1, rec, k, a)
    gpu.Optimizer.gs_pat(s, foci, amps)
    got = s.records()
    q = got[:, 6].astype(np.float64) * np.exp(1j * got[:, 7].astype(np.float64))
    _, q64 = O.gspat_f64(1, rec, k, a, foci, amps)
    _, q32 = O.gspat_f32(1, rec, k, a, foci, amps)
    peak = np.max(np.abs(q64))
    e, e32 = np.max(np.abs(q - q64)) / peak, np.max(np.abs(q32 - q64)) / peak
    print(f"GS-PAT m={m}: {e:.2e} of the peak drive (f32 restatement {e32:.2e})")
    assert e <= max(1e-4, 3 * e32)
