"""Memory of coset-word waves (csrc/coset_bytes.h), compiled for the host,
against the sum of what a wave allocates: words of two layers for every job, a
visited buffer over the rows up to the last directed job, flags, order,
descriptors and tables."""
import math
import subprocess
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parents[1] / "multigpubfs_b200" / "csrc"

MAIN = r"""
#include "coset_bytes.h"
#include <cstdio>
int main() {
  uint32_t n, gens, closed;
  std::vector<mgbfs2::CosetJob> jobs;
  while (std::scanf("%u %u %u", &n, &gens, &closed) == 3) jobs.push_back({n, gens, nullptr, closed != 0});
  std::printf("%llu\n", static_cast<unsigned long long>(mgbfs2::coset_wave_bytes(jobs, 1024)));
}
"""


@pytest.fixture(scope="module")
def counted(tmp_path_factory):
    out = tmp_path_factory.mktemp("coset_bytes")
    (out / "main.cpp").write_text(MAIN)
    subprocess.run(["g++", "-std=c++17", "-Wall", "-Werror", "-I", str(CSRC), str(out / "main.cpp"), "-o",
                    str(out / "main")], check=True)
    return lambda jobs: int(subprocess.run([str(out / "main")], check=True, capture_output=True, text=True,
                                           input="\n".join("%d %d %d" % j for j in jobs)).stdout)


def _words(jobs):
    """Bytes of a wave's word buffers, flags, order and descriptors."""
    def rows(n):
        per_row = 630 * (8 << min(3, max(0, (n - 7) // 2)))  # states of a row
        return max(1, math.factorial(max(n, 7)) // per_row)
    width = 8 if jobs[0][0] >= 13 else 4
    total = sum(rows(n) for n, _, _ in jobs)
    directed = [k for k, (_, _, closed) in enumerate(jobs) if not closed]
    visited = sum(rows(n) for n, _, _ in jobs[:directed[-1] + 1]) if directed else 0
    return (2 * total + visited) * 640 * width + sum(rows(n) * (16 + 4 + 8 * g) for n, g, _ in jobs)


@pytest.mark.parametrize("jobs", [
    [(13, 3, 1)], [(13, 3, 0)], [(14, 32, 0)], [(2, 1, 1)], [(12, 4, 1)],
    [(13, 3, 1), (13, 3, 0)], [(13, 3, 0), (13, 3, 1)],
    [(12, 4, 1)] * 7 + [(7, 2, 0)], [(7, 2, 0)] + [(12, 4, 1)] * 7,
    [(8, 2, 0), (9, 4, 1), (10, 6, 0), (11, 8, 1), (12, 2, 1)]])
def test_every_buffer_of_a_wave_is_counted(counted, jobs):
    table = 5040 * 640 * 4
    fixed = table + 5040 + (16 + 8 * len(jobs)) * 1026 + 16000
    got = counted(jobs)
    assert _words(jobs) + fixed <= got <= _words(jobs) + fixed + 1024 * 64 + 1024 * len(jobs)
