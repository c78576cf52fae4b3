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
