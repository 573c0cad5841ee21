"""The launch model (csrc/launch_model.h): the chunked launch is weighed against the launch that would run
instead, and has to model the stated margin below it.  Slots are those of a GB300's 152 SMs."""
import ctypes
import os
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(os.path.abspath(__file__)), "..", "acoustic-field-calculator_gb300",
                    "csrc")
SLOTS = {1: 304, 2: 304, 3: 291, 4: 296, 5: 290, 6: 276, 7: 266, 8: 288}
WRAPPER = """
#include "launch_model.h"
using namespace afc::model;
static long long g_slots[9];
static long long slots(long long s) { return g_slots[s]; }
extern "C" void set_slots(const long long* v) { for (int i = 0; i < 9; ++i) g_slots[i] = v[i]; }
extern "C" long long width(long long t, long long n) { return split_width(t, n, slots); }
extern "C" double chunk(long long t, long long n, long long b) { return chunk_cost(t, n, b, 152); }
extern "C" double bar(long long t, long long n, long long s, double margin) {
    return chunk_bar(t, n, s, g_slots[s], 152, margin);
}
extern "C" int overlaps(long long blocks, long long n, long long s) {
    return split_overlaps_packing(blocks, n, s, g_slots[s]);
}
extern "C" double pass(long long t, long long n, long long s) { return pass_cost(t, n, s, g_slots[s], 152); }
"""


@pytest.fixture(scope="module")
def model(tmp_path_factory):
    d = tmp_path_factory.mktemp("model")
    (d / "w.cpp").write_text(WRAPPER)
    so = str(d / "w.so")
    subprocess.run(["g++", "-O1", "-std=c++17", "-shared", "-fPIC", "-I", CSRC, str(d / "w.cpp"), "-o", so],
                   check=True)
    lib = ctypes.CDLL(so)
    i = ctypes.c_longlong
    lib.width.argtypes, lib.width.restype = [i, i], i
    lib.chunk.argtypes, lib.chunk.restype = [i, i, i], ctypes.c_double
    lib.bar.argtypes, lib.bar.restype = [i, i, i, ctypes.c_double], ctypes.c_double
    lib.pass_ = lib["pass"]
    lib.pass_.argtypes, lib.pass_.restype = [i, i, i], ctypes.c_double
    lib.overlaps.argtypes = [i, i, i]
    lib.set_slots((i * 9)(0, *(SLOTS[s] for s in range(1, 9))))
    return lib


@pytest.mark.parametrize("margin", [0.97, 1.0])
@pytest.mark.parametrize("n", [2, 40, 249, 996, 1200, 2490, 3984])
def test_bar_is_the_launch_that_runs(model, n, margin):
    for tiles in list(range(1, 700)) + list(range(700, 9000, 37)):
        s = model.width(tiles, n)
        assert 1 <= s <= 8 and (s == 1 or n // s >= 32)
        waves = -(-tiles * s // SLOTS[s])
        cost = waves * (-(-n // s) + 11 + (2 if s > 1 else 0))
        assert model.pass_(tiles, n, s) == pytest.approx(cost)
        bar = model.bar(tiles, n, s, margin)
        # a single pass always keeps its margin, whatever narrower or wider splits would model
        assert bar == pytest.approx(cost * (0.95 if s == 1 else margin if waves > 1 else 1.0))


def test_a_single_pass_keeps_its_margin(model):
    # launches that run as a single pass, where the chunked launch models less than 5 % below it and some
    # split models between the two, which used to open the chunked launch
    seen = 0
    for n in (996, 2490, 3984):
        for tiles in range(1, 9000):
            if model.width(tiles, n) != 1:
                continue
            direct, chunk = model.pass_(tiles, n, 1), model.chunk(tiles, n, 304)
            split = min(model.pass_(tiles, n, s) for s in range(2, 9))
            if 0.95 * direct <= chunk < split < direct:
                seen += 1
                assert not chunk < model.bar(tiles, n, 1, 1.0)
    assert seen > 0  # the case exists


def test_costs_in_shared_slots(model):
    # three blocks an SM share its issue slots
    assert model.chunk(456, 1000, 456) == pytest.approx(1.5 * (1000 + 22))


def test_crowded_clusters_wait_for_the_packing(model):
    # many packing blocks and a last wave that needs nearly all slots: a plain launch
    for s in range(3, 9):
        full = SLOTS[s] // s * s
        for n in (1025, 2490, 3984):
            assert not model.overlaps(full, n, s) and not model.overlaps(SLOTS[s] + full - s, n, s)
            assert model.overlaps(full // 2 // s * s, n, s)
            assert model.overlaps(SLOTS[s] + s, n, s)  # the last wave is short
        assert model.overlaps(full, 996, s)
    assert model.overlaps(304, 3984, 2)
