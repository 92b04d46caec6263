"""The ring that brings results to the host, compiled from its header with parts that
arrive on a timer instead of from a device: every byte arrives whatever the sizes, an
error ends it, helpers that cannot be started are done without, and waiting costs no
processor time."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

SOURCE = r"""
#include <sys/resource.h>
#include <chrono>
#include <cstdio>
#include <cstdlib>
#include <new>
#include <system_error>
#include "dycgraph_b200/csrc/ring.h"
using namespace dycg;

static int allowed = 99, bad_alloc = 0;  // threads that can be started, what the next one throws
struct Limited {
  std::thread t;
  Limited() = default;
  template <class F>
  explicit Limited(F f) {
    if (allowed-- <= 0) {
      if (bad_alloc) throw std::bad_alloc();
      throw std::system_error(std::make_error_code(std::errc::resource_unavailable_try_again));
    }
    t = std::thread(f);
  }
  void join() { t.join(); }
};

int main(int, char **arg) {
  const uint32_t total = std::atoi(arg[1]), slots = std::atoi(arg[2]);
  const uint32_t send_fails = std::atoi(arg[3]), wait_fails = std::atoi(arg[4]);
  const int pause_ms = std::atoi(arg[5]);
  allowed = std::atoi(arg[6]);
  bad_alloc = std::atoi(arg[7]);
  std::vector<uint32_t> ring(slots, ~0u);
  std::vector<std::atomic<uint32_t>> got(total);
  for (auto &g : got) g = ~0u;
  const auto t0 = std::chrono::steady_clock::now();
  const int x = run_ring<Limited>(
      total, slots,
      [&](uint32_t i) {
        if (i == send_fails) return 7;
        ring[i % slots] = i;  // (a part stored late would find another's number)
        return 0;
      },
      [&](uint32_t i) {
        if (i == wait_fails) return 9;
        if (pause_ms) std::this_thread::sleep_for(std::chrono::milliseconds(pause_ms));
        return 0;
      },
      [&](uint32_t i) { got[i] = ring[i % slots]; });
  const double wall =
      std::chrono::duration<double>(std::chrono::steady_clock::now() - t0).count();
  uint32_t right = 0, wrong = 0;
  for (uint32_t i = 0; i < total; i++) {
    right += got[i] == i;
    wrong += got[i] != i && got[i] != ~0u;
  }
  rusage u;
  getrusage(RUSAGE_SELF, &u);
  const double cpu = u.ru_utime.tv_sec + u.ru_stime.tv_sec +
                     (u.ru_utime.tv_usec + u.ru_stime.tv_usec) * 1e-6;
  std::printf("%d %u %u %f %f\n", x, right, wrong, wall, cpu);
}
"""

NEVER = 1_000_000


@pytest.fixture(scope="module")
def ring(tmp_path_factory):
    if shutil.which("g++") is None:
        pytest.skip("no C++ compiler")
    at = tmp_path_factory.mktemp("ring")
    (at / "ring.cpp").write_text(SOURCE)
    subprocess.run(["g++", "-std=c++17", "-O2", "-Wall", "-Werror", "-pthread", "-I", ROOT,
                    str(at / "ring.cpp"), "-o", str(at / "ring")], check=True)

    def run(total, slots, send_fails=NEVER, wait_fails=NEVER, pause_ms=0, threads=99, bad_alloc=0):
        out = subprocess.run([str(at / "ring")] + [str(x) for x in (
            total, slots, send_fails, wait_fails, pause_ms, threads, bad_alloc)],
            check=True, capture_output=True, text=True, timeout=60).stdout.split()
        return [int(x) for x in out[:3]] + [float(x) for x in out[3:]]

    return run


@pytest.mark.parametrize("threads", [0, 1, 99])
@pytest.mark.parametrize("total,slots", [(0, 4), (1, 1), (1, 8), (7, 8), (8, 8), (9, 8), (50, 1),
                                         (2000, 8)])
def test_every_part_is_stored_once(ring, total, slots, threads):
    assert ring(total, slots, threads=threads)[:3] == [0, total, 0]


@pytest.mark.parametrize("threads", [0, 99])
@pytest.mark.parametrize("at", [0, 3, 7, 8, 15, 19])
def test_an_error_ends_it(ring, at, threads):
    x, right, wrong, *_ = ring(20, 8, wait_fails=at, threads=threads)
    assert (x, wrong) == (9, 0) and right <= at
    x, right, wrong, *_ = ring(20, 8, send_fails=at, threads=threads)
    assert (x, wrong) == (7, 0) and right <= at


@pytest.mark.parametrize("threads", [0, 1, 2])
@pytest.mark.parametrize("bad_alloc", [0, 1])
def test_helpers_that_cannot_be_started(ring, threads, bad_alloc):
    assert ring(100, 8, threads=threads, bad_alloc=bad_alloc)[:3] == [0, 100, 0]


def test_waiting_takes_no_processor_time(ring):
    # 12 parts, 50 ms apart: three helpers that turned would take 1.8 s of it
    x, right, wrong, wall, cpu = ring(12, 8, pause_ms=50)
    assert (x, right, wrong) == (0, 12, 0) and wall > 0.55
    assert cpu < 0.15
