// Unipotent-ring layers: exact BFS of invertible 2x2 matrices over a prime field
// with the frontier as one bit ring per first column and determinant.
//
// Generators multiply from the left, so the p matrices that differ by a column
// operation (the second column plus t times the first) share a ring of p bits
// and a generator maps a ring onto a ring, rotated: one table entry, one load of
// the ring and one rotation carry p edges.  The list layers (packed_kernels.cuh,
// bucket_kernels.cuh) do a product, a rank and an atomic for each edge.
//
// Node: the determinant, then the first column (a, c) as a p + c - 1.  Bit t is
// the second column w + t (a, c), with w = (0, det / a), or (-det / c, 0) where a
// is 0.  A generator m leads from (v, det) to (m v, det m det); its shift is
// det times a number of v and m alone, so one table of moves serves all
// determinants.
//
// Nodes are kept by determinant because a layer holds few of them where the
// generators' determinants generate the group slowly (a diagonal generator, or
// none but 1): a pass visits the determinants that layer d leads to, 8 % of the
// work at GL(2,211).
//
// A layer is pulled as in coset.h: inverse-closed sets only, two buffers, layer
// d + 1 in the place of layer d - 1.
#pragma once
#include <cuda_runtime.h>

#include <cstdint>
#include <vector>

#include "engine.h"

namespace mgbfs2 {

constexpr uint32_t kRingMaxGens = 32;
constexpr uint32_t kRingMinPrime = 17, kRingMaxPrime = 257;  // rings of 17 to 257 bits
constexpr uint32_t kRingSmall = 1000;  // layers of fewer states are kept for samples

struct RingMemory {
  DeviceBuffer arena, words[2];
  void* report = nullptr;  // pinned, from pinned_take
  void set_stream(cudaStream_t s) {
    arena.stream = words[0].stream = words[1].stream = s;
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
  uint64_t bytes() const { return arena.bytes + words[0].bytes + words[1].bytes; }
};

struct RingResult {
  std::vector<uint64_t> layers;          // sizes from the layer after the one given
  std::vector<double> seconds;           // of each
  std::vector<uint64_t> previous_small;  // the layer before the deepest, when it was made here and is small
  std::vector<uint64_t> deepest_small;   // up to kRingSmall states of the deepest layer
  bool overflow = false;                 // more layers than the table holds
  uint32_t fatal = 0, launches = 0;
  double kernel_seconds = 0.0;
};

uint64_t ring_nodes(uint32_t p);
uint64_t ring_bytes(uint32_t p, uint32_t gens, uint32_t max_layers);

// Goes on from a frontier list (`front`, `count` packed words of `bits`-bit
// entries) and the list of the layer before it (`before`, `before_count`, may
// be empty) to the end of the search.  `coef`: gens x 4 coefficients mod p.
// The deepest layer found here is written to *collect; with no layer found
// *collect is untouched.
int ring_wave(uint32_t p, uint32_t bits, uint32_t gens, const uint32_t* coef, const void* front, uint64_t count,
              const void* before, uint64_t before_count, uint64_t key_mask, uint32_t max_layers, int sm_count,
              cudaStream_t stream, RingMemory* memory, DeviceBuffer* collect, RingResult* out);

}  // namespace mgbfs2
