"""The blocks that LM (with Gauss-Newton and gradient descent) and Horn (with Long) keep between calls are
given back with the last system, also while another thread captures a stream, and the next calls
give the same results."""
import gc
import threading

import numpy as np
import pytest

import workloads as W

pytestmark = pytest.mark.gpu


def _system(afc, n):
    pos = W.tiled_array(5, 2)[:n]
    s = afc.UniformSystem(300.0)
    s.add_records(1, W.t4010a1_records(pos, 1.0, 0.3), np.full(n, W.wavenumber(), np.float32),
                  np.zeros(n, np.float32))
    return s, pos.mean(axis=0)


def _solve(afc, name, n, m):
    s, cen = _system(afc, n)
    rng = np.random.default_rng(m)
    foci = np.float32(cen + np.c_[rng.uniform(-60, 60, (m, 2)), rng.uniform(100, 200, m)])
    getattr(afc.Optimizer, name)(s, foci, rng.uniform(0.3, 0.6, m).astype(np.float32))
    out = s.records().copy()
    return s, out


def test_blocks_go_with_the_last_system(gpu):
    torch = pytest.importorskip("torch")
    afc = gpu
    # 2,490 x 200: 4 MB of G, 0.6 MB of m x m matrices
    gc.collect()
    keep, _ = _system(afc, 1)
    first = {}
    for name, m in (("horn", 120), ("lm", 3)):
        s, first[name] = _solve(afc, name, 2490, m)
        del s
    free0 = torch.cuda.mem_get_info()[0]
    del keep
    gc.collect()
    free1 = torch.cuda.mem_get_info()[0]
    assert free1 - free0 >= 2 << 20, (free0, free1)
    for name, m in (("horn", 120), ("lm", 3)):  # from no block
        s, again = _solve(afc, name, 2490, m)
        np.testing.assert_array_equal(again, first[name])
        del s


def test_freeing_does_not_break_a_capture(gpu):
    torch = pytest.importorskip("torch")
    afc = gpu
    gc.collect()
    s, _ = _solve(afc, "horn", 996, 20)
    x = torch.zeros(1000, device="cuda")
    torch.cuda.synchronize()
    box = [s]
    del s

    def drop():
        box.clear()

    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):  # global capture mode
        y = x + 1
        t = threading.Thread(target=drop)
        t.start()
        t.join()
        z = y * 2
    x.fill_(3)
    g.replay()
    torch.cuda.synchronize()
    assert float(z[7]) == 8.0
    s, out = _solve(afc, "horn", 996, 20)
    assert np.all(np.isfinite(out))
