// Scalar-ring layers: exact BFS of 2x2 matrices over a prime field with the
// frontier as one bit ring per matrix up to a scalar.
//
// Scalars commute with every generator, so the p - 1 nonzero multiples of a
// matrix share a ring of p - 1 bits (bit t = g^t times the node's matrix, g a
// primitive root) and a generator maps a ring onto a ring, rotated by the
// discrete logarithm of the scalar that makes the product canonical: one
// 2x2 product, one 32-byte load and one rotation carry p - 1 edges.  The list
// layers (packed_kernels.cuh, bucket_kernels.cuh) do a product, a rank and an
// atomic for each edge.
//
// Node: a nonzero matrix (a b; c d) whose first nonzero entry in the order a,
// c, b, d is 1.  Index, with a = 1: (c p + b) p + d, then the p^2 nodes with a
// = 0, c = 1, then a = c = 0, b = 1, then d = 1.  The first column decides the
// block of p^2 nodes, and generators act on columns: a block's parents come
// from one block per generator, read whole.
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
constexpr uint32_t kRingMinPrime = 17, kRingMaxPrime = 257;  // rings of 16 to 256 bits
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
uint64_t ring_bytes(uint32_t p, uint32_t max_layers);

// Goes on from a frontier list (`front`, `count` packed words of `bits`-bit
// entries) and the list of the layer before it (`before`, `before_count`, may
// be empty) to the end of the search.  `coef`: gens x 4 coefficients mod p.
// The deepest layer found here is written to *collect; with no layer found
// *collect is untouched.
int ring_wave(uint32_t p, uint32_t bits, uint32_t gens, const uint32_t* coef, const void* front, uint64_t count,
              const void* before, uint64_t before_count, uint64_t key_mask, uint32_t max_layers, int sm_count,
              cudaStream_t stream, RingMemory* memory, DeviceBuffer* collect, RingResult* out);

}  // namespace mgbfs2
