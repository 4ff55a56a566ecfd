"""The setup's host threads (warpvbd_b200/csrc/vbd_parallel.h), compiled for the host: every
index once, whatever fails to start, and an exception of the work handed on."""
import os
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "warpvbd_b200",
                    "csrc")

SOURCE = r"""
#include <cstdio>
#include <cstdlib>
#include <new>
#include <stdexcept>
#include <system_error>
#include "vbd_parallel.h"

static int started = 0, limit = 0, kind = 0;
// a thread of which only `limit` can be started
struct Thread {
  std::thread t;
  template <class F>
  explicit Thread(F f) {
    if (started++ >= limit) {
      if (kind) throw std::bad_alloc();
      throw std::system_error(std::make_error_code(std::errc::resource_unavailable_try_again));
    }
    t = std::thread(f);
  }
  Thread(Thread&&) = default;
  void join() { t.join(); }
};

int main(int, char** a) {
  const int n = std::atoi(a[1]), bad = std::atoi(a[4]);
  limit = std::atoi(a[2]);
  kind = std::atoi(a[3]);
  std::vector<std::atomic<int>> seen(n > 0 ? n : 1);
  try {
    vbd::for_each_parallel<Thread>(n, [&](int k) {
      ++seen[k];
      if (k == bad) throw std::runtime_error("work");
    });
  } catch (const std::runtime_error&) {
    std::puts("thrown");
    return 0;
  }
  for (int k = 0; k < n; ++k)
    if (seen[k] != 1) return 1;
  std::puts("done");
}
"""


@pytest.fixture(scope="module")
def program(tmp_path_factory):
    d = tmp_path_factory.mktemp("parallel")
    (d / "p.cpp").write_text(SOURCE)
    subprocess.run(["g++", "-O2", "-std=c++17", "-pthread", f"-I{CSRC}", str(d / "p.cpp"), "-o",
                    str(d / "p")], check=True)
    return str(d / "p")


@pytest.mark.parametrize("n", [0, 1, 2, 100])
@pytest.mark.parametrize("limit", [0, 1, 99])
@pytest.mark.parametrize("kind", [0, 1])
def test_every_index_once_whatever_starts(program, n, limit, kind):
    r = subprocess.run([program, str(n), str(limit), str(kind), "-1"], capture_output=True)
    assert r.returncode == 0 and r.stdout == b"done\n"


@pytest.mark.parametrize("limit,kind", [(0, 1), (2, 0), (2, 1), (99, 0)])
def test_an_exception_of_the_work_is_handed_on(program, limit, kind):
    r = subprocess.run([program, "50", str(limit), str(kind), "7"], capture_output=True)
    assert r.returncode == 0 and r.stdout == b"thrown\n"
