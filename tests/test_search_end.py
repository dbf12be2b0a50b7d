"""The host's end of a persistent search (csrc/search_end.h), compiled for the
host: what a report of a search whose barrier gave up may hold, and the tables
of searches that ended."""
import subprocess
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parents[1] / "multigpubfs_b200" / "csrc"

MAIN = r"""
#include "search_end.h"
#include <cstdio>
using namespace mgbfs2;
static void show(uint32_t steps, uint32_t error, uint32_t stride, std::vector<unsigned long long> counts, uint32_t jobs) {
  const SearchEnd end = search_end(steps, error, stride, 16);
  counts.resize(static_cast<size_t>(jobs) * end.columns);
  std::printf("%u %u", end.fatal, end.columns);
  for (const auto& table : layer_tables(counts.data(), jobs, end)) {
    std::printf(" |");
    for (uint64_t s : table) std::printf(" %llu", static_cast<unsigned long long>(s));
  }
  std::printf("\n");
}
int main() {
  show(0, 0, 100, {0}, 1);             // no report, a fresh buffer
  show(0, 2, 100, {987654321}, 1);     // no report, another search's buffer
  show(3, 16, 100, {1, 4, 7, 9}, 1);   // a report of a search that failed
  show(3, 0, 100, {1, 4, 2, 0}, 1);
  show(1, 0, 100, {1, 0}, 1);
  show(4, 0, 4, {1, 4, 2, 7}, 1);      // a full table
  show(3, 0, 100, {1, 4, 2, 0, 1, 0, 0, 0}, 2);
  std::printf("lists:");
  for (int rc = 0; rc < 3000; ++rc)
    if (lists_instead(rc)) std::printf(" %d", rc);
  std::printf("\n");
}
"""


@pytest.fixture(scope="module")
def lines(tmp_path_factory):
    out = tmp_path_factory.mktemp("search_end")
    (out / "main.cpp").write_text(MAIN)
    subprocess.run(["g++", "-std=c++17", "-Wall", "-Werror", "-fsanitize=address", "-I", str(CSRC), str(out / "main.cpp"),
                    "-o", str(out / "main")], check=True)
    return subprocess.run([str(out / "main")], check=True, capture_output=True, text=True).stdout.splitlines()


def test_a_search_without_a_report_keeps_its_start_only(lines):
    assert lines[0] == "16 1 | 1" and lines[1] == "16 1 | 1"
    assert lines[2] == "16 4 | 1"


def test_tables_of_searches_that_ended(lines):
    assert lines[3:7] == ["0 4 | 1 4 2", "0 2 | 1", "0 4 | 1 4 2 7", "0 4 | 1 4 2 | 1"]


def test_list_layers_take_over_for_memory_and_residency_only(lines):
    """UNSUPPORTED, OUT_OF_MEMORY, and cudaErrorCooperativeLaunchTooLarge (720)
    and cudaErrorNotSupported (801) on the base of CUDA codes; no other error,
    an illegal address (700) least of all, starts a second search."""
    assert lines[7] == "lists: 2 3 1720 1801"
