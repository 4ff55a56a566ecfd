"""The split of a batch over clusters (warpvbd_b200/csrc/vbd_plan.h), compiled for the host:
the schedule against a plain simulation, the choice against the shapes it is made for."""
import ctypes
import os
import subprocess

import numpy as np
import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "warpvbd_b200",
                    "csrc")


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    d = tmp_path_factory.mktemp("plan")
    (d / "plan.cpp").write_text("""#include "vbd_plan.h"
static std::vector<double> v(const double* p, int n) { return std::vector<double>(p, p + n); }
extern "C" {
double schedule(const double* j, int n, int places) { return vbd::list_schedule(v(j, n), places); }
double launch_time(const double* a, const double* b, int n, int h, int C, int k, int sms) {
  return vbd::launch_time(v(a, n), v(b, n), h, C, k, sms);
}
int split_count(const double* a, const double* b, int n, int C, int k, int sms, int bound) {
  return vbd::split_count(v(a, n), v(b, n), C, k, sms, bound);
}
int pick_cluster(int preferred, const int* clusters, const double* time) {
  return vbd::pick_cluster(preferred, [&](int C) { return clusters[C]; },
                           [&](int C, int) { return time[C]; });
}
}
""")
    subprocess.run(["g++", "-O2", "-std=c++17", "-fPIC", "-shared", f"-I{CSRC}",
                    str(d / "plan.cpp"), "-o", str(d / "plan.so")], check=True)
    L = ctypes.CDLL(str(d / "plan.so"))
    p, i = ctypes.POINTER(ctypes.c_double), ctypes.c_int
    L.schedule.argtypes, L.schedule.restype = [p, i, i], ctypes.c_double
    L.launch_time.argtypes = [p, p, i, i, i, i, i]
    L.launch_time.restype = ctypes.c_double
    L.split_count.argtypes = [p, p, i, i, i, i, i]
    return L


def _p(a):
    return np.ascontiguousarray(a, float).ctypes.data_as(ctypes.POINTER(ctypes.c_double))


@pytest.mark.parametrize("n,places", [(1, 1), (5, 2), (40, 7), (7, 40), (64, 33)])
def test_schedule(lib, n, places):
    jobs = np.random.default_rng(n).uniform(1, 10, n)
    free = np.zeros(places)
    for j in jobs:
        k = free.argmin()
        free[k] += j
    assert lib.schedule(_p(jobs), n, places) == pytest.approx(free.max())


def _split(lib, one, split, C, clusters, bound, sms=148):
    one, split = np.asarray(one, float), np.asarray(split, float)
    h = lib.split_count(_p(one), _p(split), len(one), C, clusters, sms, bound)
    t = [lib.launch_time(_p(one), _p(split), len(one), k, C, clusters, sms)
         for k in range(len(one) + 1)]
    return h, t


def test_blocks_that_start_late_count_in_full(lib):
    """64 equal environments, 33 clusters of 4: 32 split ones leave the singles to a second
    wave (598 + 1396 us measured); all of them split run in two waves of 598."""
    h, t = _split(lib, [1396.0] * 64, [598.0] * 64, 4, 33, bound=32)
    assert t[32] == 598 + 1396 and t[64] == 2 * 598 and t[0] == 1396
    assert h == 64


def test_nothing_is_split_when_everything_fits_an_sm_each(lib):
    """100 equal environments, 33 clusters: splitting 33 puts the others behind them."""
    h, t = _split(lib, [470.0] * 100, [423.0] * 100, 4, 33, bound=33)
    assert t[33] == 470 + 423 and h == 0


def test_the_longest_are_split_when_all_start_together(lib):
    one = [900.0, 850.0] + [300.0] * 14
    split = [280.0, 270.0] + [200.0] * 14
    h, t = _split(lib, one, split, 8, 16, bound=2)
    assert h in (2, 14, 16) and t[h] <= min(t[2], t[0])


@pytest.mark.parametrize("seed", range(20))
def test_the_choice_is_never_worse_than_its_candidates(lib, seed):
    rng = np.random.default_rng(seed)
    n, C = int(rng.integers(2, 200)), int(rng.choice([2, 4, 8, 16]))
    one = np.sort(rng.uniform(100, 2000, n))[::-1]
    split = one / C + rng.uniform(50, 150)
    bound, clusters = int(rng.integers(0, n + 1)), int(rng.integers(1, 74))
    h, t = _split(lib, one, split, C, clusters, bound)
    assert t[h] <= min(t[0], t[n], t[bound]) * 1.002


@pytest.mark.parametrize("preferred,clusters,time,want", [
    (16, {16: 7, 8: 16, 4: 33, 2: 70}, {16: 10, 8: 10, 4: 10, 2: 10}, 16),
    (16, {16: 7, 8: 16, 4: 33, 2: 70}, {16: 25, 8: 13, 4: 15, 2: 24}, 8),
    (8, {8: 16, 4: 33, 2: 70}, {8: 10, 4: 9.5, 2: 9.2}, 8),   # within the model's error
    (16, {16: 0, 8: 16, 4: 33, 2: 70}, {16: 1, 8: 10, 4: 10, 2: 10}, 8),  # none resident
    (16, {16: 0, 8: 0, 4: 0, 2: 3}, {16: 1, 8: 1, 4: 1, 2: 9}, 2),
    (4, {4: 0, 2: 0}, {4: 1, 2: 1}, 1),
])
def test_default_cluster_size(lib, preferred, clusters, time, want):
    k, t = np.zeros(17, np.int32), np.zeros(17)
    for C in clusters:
        k[C], t[C] = clusters[C], time[C]
    lib.pick_cluster.argtypes = [ctypes.c_int, ctypes.POINTER(ctypes.c_int32),
                                 ctypes.POINTER(ctypes.c_double)]
    assert lib.pick_cluster(preferred, k.ctypes.data_as(ctypes.POINTER(ctypes.c_int32)),
                            _p(t)) == want
