// Coset-word layers: exact BFS over S_n (n <= 14, distinct labels) with the
// frontier as a bitmap whose words are cosets of label swaps.
//
// Swapping two labels commutes with every generator (a generator permutes
// positions), so the labels are split into pairs and all states that differ
// only by which label of each pair comes first share one machine word, one bit
// per choice.  A generator maps a whole word onto a whole word and only XORs
// the bit index, so one load, one byte permute and one OR carry 8 to 64 edges;
// the per-edge rank, random atomic and frontier append of the list layers
// (packed_kernels.cuh, grouped_kernels.cuh) disappear.
//
// Coordinates of a state over m = max(n, 7) symbols (symbols from n up stay in
// place, so smaller groups are embedded):
//   row   positions of the outer labels 7 .. m-1: pairs (7,8), (9,10), (11,12)
//         in turn, as unordered pairs among the positions still free, then the
//         label left over when m - 7 is odd; mixed radix.
//   node  the seven positions left free are slots 0..6; positions of the inner
//         pairs (0,1), (2,3), (4,5) as unordered pairs of slots (21 x 10 x 3 =
//         630 nodes, the last pair fastest), label 6 in the slot left over.
//   bit   inner choice r (3 bits: bit j set = the smaller label of inner pair j
//         sits in its higher slot) and outer choice q (one bit per outer pair).
//         64-bit words (m >= 13): byte r, bit q.  32-bit words: nibble r, bit q.
// A generator takes a row to one row, its nodes by one of the 5,040
// permutations of the slots (a table row of node numbers and inner flips) and
// its words by one outer flip.
//
// A layer is pulled: a word of layer d + 1 is the OR over the generators of
// its parents' words of layer d, minus what was visited.  On inverse-closed
// graphs the neighbours of layer d lie in layers d - 1, d and d + 1, so two
// buffers suffice and layer d + 1 replaces layer d - 1 in place; other graphs
// keep a third buffer of visited states.
#pragma once
#include <cuda_runtime.h>

#include <cstdint>
#include <vector>

#include "../../include/mgbfs2.h"
#include "coset_bytes.h"
#include "engine.h"

namespace mgbfs2 {

constexpr uint32_t kCosetMaxDegree = 14;
constexpr uint32_t kCosetMaxGens = 32;
constexpr uint32_t kCosetNodes = 630;    // nodes of a row
constexpr uint32_t kCosetParts = 5;

// Device memory of a wave.  Word buffers from kCosetOwnWords bytes up are
// allocations of their own: given back to the device cache they have the size
// of a Lehmer bitmap, which a later search in list layers takes without
// holding the rest of a larger block (S14 routed layers need the memory).
constexpr uint64_t kCosetOwnWords = 1ull << 29;
struct CosetMemory {
  DeviceBuffer arena, words[3];
  void* report = nullptr;  // pinned, from pinned_take
  void set_stream(cudaStream_t s) {
    arena.stream = s;
    for (DeviceBuffer& b : words) b.stream = s;
  }
  void free() {
    arena.free();
    for (DeviceBuffer& b : words) b.free();
  }
  void release_to_cache(int device) {
    arena.release_to_cache(device);
    for (DeviceBuffer& b : words) b.release_to_cache(device);
    pinned_give(report);
    report = nullptr;
  }
  uint64_t bytes() const { return arena.bytes + words[0].bytes + words[1].bytes + words[2].bytes; }
};

// Host-visible result of a wave: layer tables of every job, the wave's step
// times, and, for a wave of one job, the states of the deepest layer and of the
// layer before it where these are small.
struct CosetResult {
  std::vector<std::vector<uint64_t>> layers;
  std::vector<uint8_t> overflow;          // job ran past max_depth layers
  std::vector<double> step_seconds;       // step d expanded layer d
  std::vector<uint64_t> previous_small;   // packed words, 4 bits per code
  std::vector<uint64_t> deepest_small;    // the deepest layer, up to kCosetSmall states
  uint32_t fatal = 0;
  uint32_t steps = 0;
  uint32_t launches = 0;
  double kernel_seconds = 0.0;
};

bool coset_supported(uint32_t n, uint32_t gens);

// Runs every job to the end (or max_depth layers) in one cooperative launch
// on `stream`, in `memory` (grown as needed).  With `collect`, the wave holds
// one job and its deepest layer is written to *collect as packed words (codes
// mapped through start_word).
int coset_wave(const std::vector<CosetJob>& jobs, uint32_t max_depth, int sm_count, cudaStream_t stream,
               CosetMemory* memory, CosetResult* out, DeviceBuffer* collect = nullptr, uint64_t start_word = 0);

}  // namespace mgbfs2
