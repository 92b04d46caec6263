"""The mutation kernel's launch size, compiled from its header: an explicit limit means
CTAs of eight warps, as it does for a caller who set one before the kernel's CTAs grew
to sixteen, and no launch exceeds it or what is resident."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

SOURCE = """
#include <cstdio>
#include "dycgraph_b200/csrc/mutation_grid.h"
using namespace dycg;
int main() {
  unsigned asked, sms, records, dirs;
  unsigned long long bytes, resident;
  while (std::scanf("%u %u %llu %u %u %llu", &asked, &sms, &bytes, &records, &dirs, &resident) == 6) {
    std::printf("%u %d\\n", mutation_grid(records, dirs, asked, sms, bytes, resident), MUT_BLOCK / 32);
  }
}
"""


@pytest.mark.skipif(shutil.which("g++") is None, reason="no C++ compiler")
def test_launch_sizes(tmp_path):
    src, exe = tmp_path / "grid.cpp", tmp_path / "grid"
    src.write_text(SOURCE)
    subprocess.run(["g++", "-std=c++17", "-Wall", "-Werror", "-I", ROOT, str(src), "-o", str(exe)],
                   check=True)
    asks = [(asked, 148, gb << 30, records, dirs, resident)
            for asked in (0, 1, 2, 3, 8, 37, 148, 296, 0xFFFFFFFF) for gb in (1, 4, 5, 40)
            for records in (1, 3, 16, 1000, 50_000, 0x3FFFFFFF) for dirs in (1, 2)
            for resident in (1, 100, 148)]
    out = subprocess.run([str(exe)], input="\n".join(" ".join(map(str, a)) for a in asks),
                         check=True, capture_output=True, text=True).stdout.split("\n")
    for (asked, sms, size, records, dirs, resident), line in zip(asks, out):
        grid, warps = map(int, line.split())
        most = (asked + 1) // 2 if asked else sms
        assert 1 <= grid <= min(most, resident)
        assert grid >= min(8, most, resident)
        if asked:
            assert warps * grid <= 8 * (asked + 1)
        if records == 0x3FFFFFFF:  # (any arena is densely hit)
            assert grid == min(most, resident)
        if not asked and records == 50_000 and resident == sms:
            # R-MAT 26's batches; the same in 1 GB; the density rule's own arithmetic
            fits = (5 << 30) / size * records / 256
            assert grid == (sms if size <= 4 << 30 else min(sms, max(sms // 4, int(fits))))
