"""The closed form of how long the busiest of several workers takes, against dealing the units one by one; and its cost, which every
call of the tensor-core products with a new number of tiles pays."""
import ctypes
import os
import random
import subprocess
import time

import pytest

CSRC = os.path.join(os.path.dirname(os.path.abspath(__file__)), "..", "openequivariance_b200", "csrc")


@pytest.fixture(scope="module")
def busiest(tmp_path_factory):
    d = tmp_path_factory.mktemp("dealing")
    (d / "t.cpp").write_text('#include "dealing.h"\nextern "C" double f(long long u, int n, const double* p, double e, int w)'
                             " { return busiest_load(u, n, p, e, w); }\n")
    subprocess.run(["g++", "-O2", "-std=c++17", "-shared", "-fPIC", f"-I{CSRC}", str(d / "t.cpp"), "-o", str(d / "t.so")], check=True)
    f = ctypes.CDLL(str(d / "t.so")).f
    f.restype, f.argtypes = ctypes.c_double, [ctypes.c_longlong, ctypes.c_int, ctypes.c_void_p, ctypes.c_double, ctypes.c_int]
    return lambda units, part, each, workers: f(units, len(part), (ctypes.c_double * len(part))(*part), each, workers)


def test_matches_dealing_one_by_one(busiest):
    rng = random.Random(0)
    for _ in range(600):
        workers, n = rng.choice([1, 2, 3, 7, 108, 132, 148]), rng.randint(1, 8)
        part, each = [rng.randint(1, 60) / 2 for _ in range(n)], rng.choice([2.0, 8.0])
        units = rng.choice([1, n, workers, workers - 1, workers + 1, rng.randint(1, 3 * workers * n)]) or 1
        load = [0.0] * workers
        for u in range(units):
            load[u % workers] += part[u % n] + each
        assert busiest(units, part, each, workers) == max(load), (workers, part, units)


def test_costs_no_loop_over_units(busiest):
    part = [float(i) for i in range(1, 9)]
    best = {}
    for units in (1000, 10 ** 9):
        best[units] = min(_timed(busiest, units, part) for _ in range(5))
    assert best[10 ** 9] < 10 * best[1000] + 1e-3


def _timed(busiest, units, part):
    start = time.perf_counter()
    busiest(units, part, 8.0, 148)
    return time.perf_counter() - start


@pytest.fixture(scope="module")
def best(tmp_path_factory):
    """(parts, list) for two lists of costs, tiles and workers."""
    d = tmp_path_factory.mktemp("parts")
    (d / "t.cpp").write_text('#include "dealing.h"\nextern "C" int f(int n0, const double* c0, int n1, const double* c1, long long t, double each, double extra,'
                             " int w, int* list) { Cuts a, b; a.cost.assign(c0, c0 + n0); b.cost.assign(c1, c1 + n1); cut_into_parts(a); cut_into_parts(b);"
                             " const Cuts* l[2] = {&a, &b}; return best_parts(l, t, each, extra, w, list); }\n")
    subprocess.run(["g++", "-O2", "-std=c++17", "-shared", "-fPIC", f"-I{CSRC}", str(d / "t.cpp"), "-o", str(d / "t.so")], check=True)
    f = ctypes.CDLL(str(d / "t.so")).f
    array = lambda v: (ctypes.c_double * len(v))(*v)  # noqa: E731

    def call(c0, c1, tiles, each=3000.0, extra=0.0, workers=148):
        which = ctypes.c_int()
        return f(len(c0), array(c0), len(c1), array(c1), ctypes.c_longlong(tiles), ctypes.c_double(each), ctypes.c_double(extra), workers,
                 ctypes.byref(which)), which.value
    return call


def test_a_number_of_parts_that_makes_no_cut_does_not_hide_the_next(best):
    assert best([7000.0] * 4, [7000.0] * 4, 20) == (4, 0)             # three parts of four equal pieces are two
    assert best([48000.0], [4000.0] * 12, 4) == (12, 1)               # seven to eleven of twelve are six
    assert best([7000.0] * 4, [7000.0] * 4, 148) == (1, 0)            # a tile for each worker
