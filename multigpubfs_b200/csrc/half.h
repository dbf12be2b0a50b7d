// Half-rank layers: exact BFS of permutations with repeated labels whose rank
// is the sum of two table entries.
//
// The multinomial rank of a state splits at its middle: the states that start
// with a smaller first half come before it whatever the second half, and within
// one first half the second is ranked among the arrangements of its own labels
// (the labels left over are fixed by the first half).  So
//     rank(first, second) = before[first] + within[second]
// with one table entry per half instead of a division chain over every symbol
// (multiset_rank, device.cuh), and the bitmap is the same.  States are coded in
// one to three bits a symbol, so starts of more than 16 positions and at most
// four labels fit one word too; those otherwise take the wide hash path.  Both
// lists hold the bound of the reachable states, 16 bytes each in all, whatever
// the orbit: 32 states of a shift of 32 positions map 9.2 GB the first time (5.2
// ms a call, the wide hash 1.1) and find them mapped afterwards (0.41, 0.98).
#pragma once
#include <cuda_runtime.h>

#include <cstdint>
#include <vector>

#include "device.cuh"
#include "engine.h"

namespace mgbfs2 {

constexpr uint32_t kHalfMaxLabels = 6, kHalfMaxGens = 32, kHalfSmall = 1000;
constexpr uint32_t kHalfIndexBits = 21;  // table entries of a half

struct HalfMemory {
  DeviceBuffer arena, list[2];
  void* report = nullptr;  // pinned, from pinned_take
  const uint64_t* deepest = nullptr;  // the last search's deepest layer, in one of the lists
  uint64_t key_mask = 0;              // its words without their tags
  uint32_t bits = 0;                  // bits a symbol
  void set_stream(cudaStream_t s) {
    arena.stream = list[0].stream = list[1].stream = s;
  }
  void free() {
    deepest = nullptr;
    arena.free();
    for (DeviceBuffer& b : list) b.free();
  }
  void release_to_cache(int device) {
    arena.release_to_cache(device);
    for (DeviceBuffer& b : list) b.release_to_cache(device);
    pinned_give(report);
    report = nullptr;
  }
  uint64_t bytes() const { return arena.bytes + list[0].bytes + list[1].bytes; }
};

// One search: n positions, codes of the start, generators (gens x n), label counts.
struct HalfJob {
  uint32_t n = 0, distinct = 0, gens = 0;
  const uint32_t* codes = nullptr;
  const uint32_t* counts = nullptr;
  const uint32_t* perms = nullptr;
  bool inverse_closed = false;
  uint64_t total = 0;     // rank domain
  uint64_t capacity = 0;  // largest possible layer
};

struct HalfResult {
  std::vector<uint64_t> layers;
  std::vector<double> seconds;
  std::vector<uint64_t> previous, deepest;  // up to kHalfSmall states each, `bits` bits a symbol
  uint32_t bits = 0, fatal = 0, launches = 0;
  bool overflow = false;
  double kernel_seconds = 0.0;
};

// job.perms: the generators' displacement terms are counted too.
bool half_supported(const HalfJob& job);
uint64_t half_bytes(const HalfJob& job, uint32_t max_layers);

// Runs the search with its visited states in `bitmap` (ceil(total / 64) words,
// cleared here).  With `front`, the deepest layer is written there as packed
// words of `front_bits` bits a symbol.
int half_wave(const HalfJob& job, uint32_t max_layers, int sm_count, cudaStream_t stream, HalfMemory* memory,
              DeviceBuffer* bitmap, DeviceBuffer* front, uint32_t front_bits, HalfResult* out);

}  // namespace mgbfs2
