// Unipotent-ring layers (see ring.h): seeding from frontier lists, the persistent
// wave kernel and its host side.
#include "ring.h"
#include "search_end.h"

#include <algorithm>
#include <cstring>

#define MG_CHECK_RING(expr)                        \
  do {                                             \
    cudaError_t _e = (expr);                       \
    if (_e != cudaSuccess) return cuda_status(_e); \
  } while (0)

namespace mgbfs2 {
namespace {

constexpr uint32_t kRingBlock = 256;
constexpr uint32_t kRingReportLayers = 256;

struct RingCtl {
  uint32_t arrived, error;
  unsigned long long collected;
};

struct RingReport {
  uint32_t steps, error, previous_count, pad;
  unsigned long long counts[kRingReportLayers], stamps[kRingReportLayers];
  unsigned long long previous[kRingSmall], deepest[kRingSmall];
};

constexpr uint32_t kRingClasses = 256;  // determinants
constexpr uint32_t kMoveBits = 17;      // a first column: fewer than 257^2

struct RingParams {
  uint32_t p, bits, gens, magic;   // magic: floor(2^32 / p)
  uint32_t vectors, low;           // p^2 - 1 first columns; unused low bits of a ring's first word
  uint32_t nodes, max_steps;
  const uint16_t* inverse;         // p entries
  uint32_t* moves;                 // gens x vectors: the product's first column, its shift << kMoveBits
  uint32_t* buf[2];
  unsigned long long* counts;      // max_steps + 2 layer sizes; 0 = the seeded layer
  uint32_t* classes;               // 4 x kRingClasses: layer d's states by determinant in row (d + 1) & 3
  unsigned long long* stamps;
  uint32_t* small_count;
  unsigned long long* small;       // 2 x kRingSmall (node << 9 | bit), by step parity
  RingReport* report;
  unsigned long long* front;
  unsigned long long front_cap;
  RingCtl* ctl;
  uint32_t coef[4 * kRingMaxGens], det[kRingMaxGens];
};

__device__ __forceinline__ uint32_t reduce(uint32_t x, const RingParams& r) {
  uint32_t y = x - __umulhi(x, r.magic) * r.p;  // quotient short by at most one
  return y >= r.p ? y - r.p : y;
}

// Node and ring bit of an invertible matrix.
__device__ __forceinline__ uint32_t node_of(uint32_t a, uint32_t b, uint32_t c, uint32_t d, const RingParams& r,
                                            uint32_t* bit) {
  const uint32_t det = reduce(a * d + (r.p - b) * c, r);
  *bit = a ? reduce(b * r.inverse[a], r) : reduce(d * r.inverse[c], r);
  return (det - 1) * r.vectors + a * r.p + c - 1;
}

__device__ __forceinline__ unsigned long long pack_matrix(uint32_t node, uint32_t bit, const RingParams& r) {
  const uint32_t det = node / r.vectors + 1, column = node - (det - 1) * r.vectors + 1;
  const uint32_t a = column / r.p, c = column - a * r.p;
  const uint32_t w = reduce(det * r.inverse[a ? a : c], r);
  const uint32_t b = a ? reduce(bit * a, r) : r.p - w, d = a ? reduce(bit * c + w, r) : reduce(bit * c, r);
  return static_cast<unsigned long long>(a) | (static_cast<unsigned long long>(b) << r.bits) |
         (static_cast<unsigned long long>(c) << (2 * r.bits)) | (static_cast<unsigned long long>(d) << (3 * r.bits));
}

// Words between rings in memory: whole 8- or 16-byte loads.
template <int NW>
constexpr uint32_t ring_stride() {
  return NW <= 2 ? NW : (NW + 3) / 4 * 4;
}

// Marks the states of a list in a buffer; `which` 0 = the frontier, 1 = the
// layer before it.
template <int NW>
__global__ void __launch_bounds__(kRingBlock) ring_seed(RingParams r, const unsigned long long* list,
                                                        unsigned long long count, unsigned long long key_mask,
                                                        uint32_t which) {
  __shared__ uint32_t classes[kRingClasses];
  for (uint32_t i = threadIdx.x; i < kRingClasses; i += blockDim.x) classes[i] = 0;
  __syncthreads();
  uint32_t* buf = which ? r.buf[1] : r.buf[0];
  const uint32_t mask = (1u << r.bits) - 1u;
  for (unsigned long long k = blockIdx.x * static_cast<unsigned long long>(blockDim.x) + threadIdx.x; k < count;
       k += static_cast<unsigned long long>(gridDim.x) * blockDim.x) {
    const unsigned long long w = list[k] & key_mask;
    uint32_t bit;
    const uint32_t node = node_of(static_cast<uint32_t>(w) & mask, static_cast<uint32_t>(w >> r.bits) & mask,
                                  static_cast<uint32_t>(w >> (2 * r.bits)) & mask,
                                  static_cast<uint32_t>(w >> (3 * r.bits)) & mask, r, &bit);
    bit += r.low;
    atomicOr(buf + static_cast<size_t>(node) * ring_stride<NW>() + (bit >> 5), 1u << (bit & 31u));
    atomicAdd(classes + node / r.vectors, 1u);
  }
  __syncthreads();
  for (uint32_t i = threadIdx.x; i < kRingClasses; i += blockDim.x)
    if (classes[i]) atomicAdd(r.classes + (which ? 0u : kRingClasses) + i, classes[i]);
  if (blockIdx.x == 0 && threadIdx.x == 0 && !which) r.counts[0] = count;
}

// The move of each generator on each first column v: the column of m v and the
// ring shift per unit of determinant.
__global__ void __launch_bounds__(kRingBlock) ring_moves(RingParams r) {
  const uint32_t all = r.gens * r.vectors;
  for (uint32_t k = blockIdx.x * blockDim.x + threadIdx.x; k < all; k += gridDim.x * blockDim.x) {
    const uint32_t g = k / r.vectors, column = k - g * r.vectors + 1, a = column / r.p, c = column - a * r.p;
    const uint32_t m0 = r.coef[4 * g], m1 = r.coef[4 * g + 1], m2 = r.coef[4 * g + 2], m3 = r.coef[4 * g + 3];
    const uint32_t a2 = reduce(m0 * a + m1 * c, r), c2 = reduce(m2 * a + m3 * c, r);
    // The node's second column at bit 0 and determinant 1: (0, 1/a) or (-1/c, 0).
    const uint32_t w = r.inverse[a ? a : c];
    const uint32_t top = a ? m1 * w : m0 * (r.p - w), bottom = a ? m3 * w : m2 * (r.p - w);
    const uint32_t shift = a2 ? reduce(reduce(top, r) * r.inverse[a2], r) : reduce(reduce(bottom, r) * r.inverse[c2], r);
    r.moves[k] = (a2 * r.p + c2 - 1) | (shift << kMoveBits);
  }
}

template <int NW>
__device__ __forceinline__ void load_ring(const uint32_t* at, uint32_t (&w)[NW]) {
  if constexpr (NW >= 3) {
#pragma unroll
    for (int i = 0; i < NW; i += 4) {
      const uint4 x = *reinterpret_cast<const uint4*>(at + i);
      w[i] = x.x;
      if (i + 1 < NW) w[i + 1] = x.y;
      if (i + 2 < NW) w[i + 2] = x.z;
      if (i + 3 < NW) w[i + 3] = x.w;
    }
  } else if constexpr (NW == 2) {
    const uint2 x = *reinterpret_cast<const uint2*>(at);
    w[0] = x.x, w[1] = x.y;
  } else {
    w[0] = *at;
  }
}

template <int NW>
__device__ __forceinline__ void store_ring(uint32_t* at, const uint32_t (&w)[NW]) {
  if constexpr (NW >= 3) {
#pragma unroll
    for (int i = 0; i < NW; i += 4)
      *reinterpret_cast<uint4*>(at + i) = make_uint4(w[i], i + 1 < NW ? w[i + 1] : 0u, i + 2 < NW ? w[i + 2] : 0u,
                                                     i + 3 < NW ? w[i + 3] : 0u);
  } else if constexpr (NW == 2) {
    *reinterpret_cast<uint2*>(at) = make_uint2(w[0], w[1]);
  } else {
    *at = w[0];
  }
}

// The words that the smaller moves still need, `by` words down if s asks for it.
template <int NW, int by>
__device__ __forceinline__ void move_down(uint32_t (&y)[2 * NW], uint32_t s) {
  const bool down = (s >> 5) & by;
#pragma unroll
  for (int i = 0; i < NW + by; ++i) y[i] = down ? (i + by < 2 * NW ? y[i + by] : 0u) : y[i];
}

// acc |= the ring rotated right by s < p.  A ring fills its words from the top
// (bit t at low + t), so the copy that follows it starts on a word: words by
// selects, the rest by one funnel shift a word.  The caller drops the low bits.
template <int NW>
__device__ __forceinline__ void or_rotated(uint32_t (&acc)[NW], const uint32_t (&x)[NW], uint32_t s, uint32_t low) {
  uint32_t y[2 * NW];
#pragma unroll
  for (int i = 0; i < NW; ++i) {
    y[i] = x[i];
    y[NW + i] = __funnelshift_r(x[i], i + 1 < NW ? x[i + 1] : 0u, low);
  }
  if constexpr (NW > 8) move_down<NW, 8>(y, s);
  if constexpr (NW > 4) move_down<NW, 4>(y, s);
  if constexpr (NW > 2) move_down<NW, 2>(y, s);
  if constexpr (NW > 1) move_down<NW, 1>(y, s);
#pragma unroll
  for (int i = 0; i < NW; ++i) acc[i] |= __funnelshift_r(y[i], y[i + 1], s & 31u);
}

// Block 0's report of the layers up to d.
__device__ void ring_report(const RingParams& r, uint32_t d, bool exhausted) {
  const uint32_t kept = exhausted ? min(r.small_count[d], kRingSmall) : 0u;
  for (uint32_t k = threadIdx.x; k < kept; k += blockDim.x) {
    const unsigned long long at = r.small[(d & 1u) * kRingSmall + k];
    r.report->previous[k] = pack_matrix(static_cast<uint32_t>(at >> 9), static_cast<uint32_t>(at & 511u), r);
  }
  for (uint32_t k = threadIdx.x; k < kRingReportLayers && k <= d + 1; k += blockDim.x) {
    r.report->counts[k] = __ldcg(r.counts + k);
    r.report->stamps[k] = r.stamps[k];
  }
  if (threadIdx.x == 0) {
    r.report->previous_count = kept;
    r.report->steps = d + 1;
    r.report->error = r.ctl->error;
  }
}

// A layer is a pass over the rings of the determinants that it can hold, a
// warp per 32 rings: per generator one coalesced move, one ring of 32 bytes and
// its rotation, most of the instructions.  No unit is full (integer pipe 48 % of
// its rate, issue slots 43 %, DRAM 0.6 TB/s): the warps wait for the ring loads,
// whose addresses hang on the moves, and at the barrier behind uneven layers.  GL(2,211),
// 111 layers, whole call: 4.8 ms, 30 to 60 us a layer; rings of the 210 scalar
// multiples, which mix all determinants (520 us a layer): 58.8 ms; list layers:
// 271 ms.  GL(2,257): 9.4 ms.
template <int NW>
__global__ void __launch_bounds__(kRingBlock, 4) ring_wave_kernel(RingParams r) {
  __shared__ uint32_t here[kRingClasses], list[kRingClasses], live[kRingClasses], lists[kRingBlock / 32];
  constexpr uint32_t kStride = ring_stride<NW>();
  constexpr uint32_t kOwn = 1u << 8, kOld = 1u << 9;  // in list: the class holds states of layer d, of d - 1
  const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
  const uint32_t first = (blockIdx.x * kRingBlock + threadIdx.x) >> 5, warps = gridDim.x * (kRingBlock / 32);
  const uint32_t per_class = (r.vectors + 31u) / 32u;
  uint32_t epoch = 0;
  for (uint32_t d = 0;; ++d) {
    if (blockIdx.x == 0 && threadIdx.x == 0) r.stamps[d] = global_ns();
    const uint32_t* cur = d & 1u ? r.buf[1] : r.buf[0];
    uint32_t* nxt = d & 1u ? r.buf[0] : r.buf[1];
    uint32_t* counted = r.classes + ((d + 2) & 3u) * kRingClasses;
    const bool keep = d && __ldcg(r.counts + d - 1) < kRingSmall;
    // The determinants to visit: those that a generator leads to from layer d
    // and those that layer d - 1 has left states of in the buffer.
    static_assert(kRingBlock == kRingClasses, "a thread per determinant");
    here[threadIdx.x] = __ldcg(r.classes + ((d + 1) & 3u) * kRingClasses + threadIdx.x);
    const uint32_t before = __ldcg(r.classes + (d & 3u) * kRingClasses + threadIdx.x);
    if (blockIdx.x == 0) __stcg(r.classes + ((d + 3) & 3u) * kRingClasses + threadIdx.x, 0u);
    __syncthreads();
    uint32_t from = 0;
    if (threadIdx.x < r.p - 1)
      for (uint32_t g = 0; g < r.gens; ++g)
        if (here[reduce((threadIdx.x + 1) * r.det[g], r) - 1]) from |= 1u << g;
    const bool listed = from || before;
    const uint32_t votes = __ballot_sync(kFullMask, listed);
    if (lane == 0) lists[warp] = __popc(votes);
    __syncthreads();
    uint32_t at = __popc(votes & ((1u << lane) - 1u)), all = 0;
#pragma unroll
    for (uint32_t w = 0; w < kRingBlock / 32; ++w) {
      if (w < warp) at += lists[w];
      all += lists[w];
    }
    if (listed) {
      list[at] = threadIdx.x | (here[threadIdx.x] ? kOwn : 0u) | (before ? kOld : 0u);
      live[at] = from;
    }
    __syncthreads();
    const uint32_t items = all * per_class;
    unsigned long long total = 0;
    for (uint32_t item = first; item < items; item += warps) {
      const uint32_t slot = item / per_class, entry = list[slot], cls = entry & 255u;
      const uint32_t v = (item - slot * per_class) * 32u + lane;
      uint32_t found = 0;
      if (v < r.vectors) {
        uint32_t acc[NW];
#pragma unroll
        for (int i = 0; i < NW; ++i) acc[i] = 0;
        const uint32_t* moves = r.moves + v;
        uint32_t left = live[slot];
        uint32_t ahead = left ? __ldg(moves + (__ffs(static_cast<int>(left)) - 1) * r.vectors) : 0u;
        while (left) {
          // The set is inverse-closed: its products are the parents.
          const uint32_t g = __ffs(static_cast<int>(left)) - 1, move = ahead;
          left &= left - 1;
          if (left) ahead = __ldg(moves + (__ffs(static_cast<int>(left)) - 1) * r.vectors);
          const uint32_t parent = (reduce((cls + 1) * r.det[g], r) - 1) * r.vectors + (move & ((1u << kMoveBits) - 1u));
          uint32_t w[NW];
          load_ring<NW>(cur + static_cast<size_t>(parent) * kStride, w);
          or_rotated<NW>(acc, w, reduce((cls + 1) * (move >> kMoveBits), r), r.low);
        }
        acc[0] &= 0xffffffffu << r.low;
        const size_t ring = static_cast<size_t>(cls * r.vectors + v) * kStride;
        uint32_t old[NW], changed = 0;
        if (entry & kOwn) {
          load_ring<NW>(cur + ring, old);
#pragma unroll
          for (int i = 0; i < NW; ++i) acc[i] &= ~old[i];
        }
        if (entry & kOld) {
          load_ring<NW>(nxt + ring, old);
#pragma unroll
          for (int i = 0; i < NW; ++i) {
            acc[i] &= ~old[i];
            changed |= old[i];
          }
          if (keep) {
            // The small layer d - 1 is about to be overwritten.
#pragma unroll
            for (int i = 0; i < NW; ++i)
              for (uint32_t o = old[i]; o; o &= o - 1) {
                const uint32_t k = atomicAdd(r.small_count + d, 1u);
                if (k < kRingSmall)
                  r.small[(d & 1u) * kRingSmall + k] = (static_cast<unsigned long long>(cls * r.vectors + v) << 9) |
                                                       (32u * i + __ffs(static_cast<int>(o)) - 1u - r.low);
              }
          }
        }
#pragma unroll
        for (int i = 0; i < NW; ++i) {
          found += __popc(acc[i]);
          changed |= acc[i];
        }
        if (changed) store_ring<NW>(nxt + ring, acc);
      }
      found = __reduce_add_sync(kFullMask, found);
      if (found && lane == 0) atomicAdd(counted + cls, found);
      total += found;
    }
    if (total && lane == 0) atomicAdd(r.counts + d + 1, total);
    if (!arrival_barrier(&r.ctl->arrived, &r.ctl->error, &epoch)) return;
    const bool more = __ldcg(r.counts + d + 1) != 0;
    if (more && d < r.max_steps) continue;
    if (blockIdx.x == 0) {
      if (threadIdx.x == 0) r.stamps[d + 1] = global_ns();
      __syncthreads();
      ring_report(r, d, !more);
    }
    return;
  }
}

// The states of layer d (from the seeded one) as packed words.
template <int NW>
__global__ void __launch_bounds__(kRingBlock) ring_collect(RingParams r, uint32_t d) {
  const uint32_t* buf = d & 1u ? r.buf[1] : r.buf[0];
  const uint32_t* held = r.classes + ((d + 1) & 3u) * kRingClasses;
  for (uint32_t node = blockIdx.x * blockDim.x + threadIdx.x; node < r.nodes; node += gridDim.x * blockDim.x) {
    if (!__ldg(held + node / r.vectors)) continue;
    uint32_t w[NW];
    load_ring<NW>(buf + static_cast<size_t>(node) * ring_stride<NW>(), w);
    uint32_t mine = 0;
#pragma unroll
    for (int i = 0; i < NW; ++i) mine += __popc(w[i]);
    if (!mine) continue;
    unsigned long long at = atomicAdd(&r.ctl->collected, static_cast<unsigned long long>(mine));
#pragma unroll
    for (int i = 0; i < NW; ++i)
      for (uint32_t b = w[i]; b; b &= b - 1, ++at) {
        const unsigned long long s = pack_matrix(node, 32 * i + __ffs(static_cast<int>(b)) - 1 - r.low, r);
        if (at < r.front_cap) r.front[at] = s;
        if (at < kRingSmall) r.report->deepest[at] = s;
      }
  }
}

size_t al256(size_t x) { return (x + 255) / 256 * 256; }

uint32_t ring_words(uint32_t p) { return (p + 31) / 32; }

uint32_t ring_word_stride(uint32_t p) {
  const uint32_t w = ring_words(p);
  return w <= 2 ? w : (w + 3) / 4 * 4;
}

using SeedFn = void (*)(RingParams, const unsigned long long*, unsigned long long, unsigned long long, uint32_t);
using WaveFn = void (*)(RingParams);
using CollectFn = void (*)(RingParams, uint32_t);

struct RingKernels {
  SeedFn seed;
  WaveFn wave;
  CollectFn collect;
};

template <int NW>
RingKernels kernels_of() {
  return {ring_seed<NW>, ring_wave_kernel<NW>, ring_collect<NW>};
}

RingKernels kernels_for(uint32_t words) {
  switch (words) {
    case 1: return kernels_of<1>();
    case 2: return kernels_of<2>();
    case 3: return kernels_of<3>();
    case 4: return kernels_of<4>();
    case 5: return kernels_of<5>();
    case 6: return kernels_of<6>();
    case 7: return kernels_of<7>();
    case 8: return kernels_of<8>();
    default: return kernels_of<9>();
  }
}

}  // namespace

uint64_t ring_nodes(uint32_t p) {
  const uint64_t q = p;
  return (q - 1) * (q * q - 1);
}

uint64_t ring_bytes(uint32_t p, uint32_t gens, uint32_t max_layers) {
  return 2 * ring_nodes(p) * 4 * ring_word_stride(p) + 4ull * gens * (p * p - 1) + 20ull * (max_layers + 2) +
         16ull * kRingSmall + 2ull * p + 16ull * kRingClasses + 16 * 256;
}

int ring_wave(uint32_t p, uint32_t bits, uint32_t gens, const uint32_t* coef, const void* front, uint64_t count,
              const void* before, uint64_t before_count, uint64_t key_mask, uint32_t max_layers, int sm_count,
              cudaStream_t stream, RingMemory* memory, DeviceBuffer* collect, RingResult* out) {
  if (p < kRingMinPrime || p > kRingMaxPrime || gens < 1 || gens > kRingMaxGens || !count || !max_layers)
    return MGBFS2_INVALID_ARGUMENT;
  const uint32_t words = ring_words(p);
  const RingKernels k = kernels_for(words);
  RingParams r{};
  r.p = p;
  r.bits = bits;
  r.gens = gens;
  r.magic = static_cast<uint32_t>((1ull << 32) / p);
  r.vectors = p * p - 1;
  r.low = 32 * words - p;
  r.nodes = static_cast<uint32_t>(ring_nodes(p));
  r.max_steps = max_layers - 1;
  std::copy_n(coef, 4 * gens, r.coef);
  std::vector<uint16_t> tables(p, 0);
  for (uint32_t x = 1; x < p; ++x)
    for (uint32_t y = 1; y < p; ++y)
      if (x * y % p == 1) tables[x] = static_cast<uint16_t>(y);
  for (uint32_t g = 0; g < gens; ++g) {
    const uint32_t* m = r.coef + 4 * g;
    r.det[g] = (m[0] * m[3] + (p - m[1]) * m[2]) % p;
    if (!r.det[g]) return MGBFS2_INVALID_ARGUMENT;
  }
  const uint32_t stride = max_layers + 2;
  size_t off = 0;
  const auto take = [&off](size_t bytes) {
    const size_t at = off;
    off = al256(off + bytes);
    return at;
  };
  const size_t o_tables = take(tables.size() * 2);
  const size_t upload = off;
  const size_t o_counts = take(8ull * stride), o_small_count = take(4ull * stride), o_ctl = take(sizeof(RingCtl));
  const size_t o_classes = take(16ull * kRingClasses);
  const size_t cleared = off;
  const size_t o_stamps = take(8ull * stride), o_small = take(16ull * kRingSmall);
  const size_t o_moves = take(4ull * gens * r.vectors);
  int rc = memory->arena.ensure(off, true);
  const size_t word_bytes = ring_nodes(p) * 4 * ring_word_stride(p);
  for (DeviceBuffer& b : memory->words)
    if (!rc) rc = b.ensure(word_bytes, true);
  if (!rc && !memory->report) rc = pinned_take(sizeof(RingReport), &memory->report);
  if (rc) return rc;
  char* base = static_cast<char*>(memory->arena.ptr);
  RingReport* report = static_cast<RingReport*>(memory->report);
  report->steps = 0;
  r.inverse = reinterpret_cast<const uint16_t*>(base + o_tables);
  r.buf[0] = static_cast<uint32_t*>(memory->words[0].ptr);
  r.buf[1] = static_cast<uint32_t*>(memory->words[1].ptr);
  r.counts = reinterpret_cast<unsigned long long*>(base + o_counts);
  r.stamps = reinterpret_cast<unsigned long long*>(base + o_stamps);
  r.classes = reinterpret_cast<uint32_t*>(base + o_classes);
  r.moves = reinterpret_cast<uint32_t*>(base + o_moves);
  r.small_count = reinterpret_cast<uint32_t*>(base + o_small_count);
  r.small = reinterpret_cast<unsigned long long*>(base + o_small);
  r.report = report;
  r.ctl = reinterpret_cast<RingCtl*>(base + o_ctl);
  // The list given may sit in *collect, so the deepest layer is not written
  // over it: a second launch writes it once the seeds have been read.
  r.front = nullptr;
  r.front_cap = 0;
  MG_CHECK_RING(cudaMemcpyAsync(base, tables.data(), tables.size() * 2, cudaMemcpyHostToDevice, stream));
  MG_CHECK_RING(cudaMemsetAsync(base + upload, 0, cleared - upload, stream));
  for (DeviceBuffer& b : memory->words) MG_CHECK_RING(cudaMemsetAsync(b.ptr, 0, word_bytes, stream));
  const auto blocks_for = [&](uint64_t n) {
    return static_cast<uint32_t>(std::min<uint64_t>((n + kRingBlock - 1) / kRingBlock, 8ull * sm_count));
  };
  k.seed<<<blocks_for(count), kRingBlock, 0, stream>>>(r, static_cast<const unsigned long long*>(front), count, key_mask, 0);
  ring_moves<<<blocks_for(static_cast<uint64_t>(gens) * r.vectors), kRingBlock, 0, stream>>>(r);
  out->launches = 2;
  if (before_count) {
    k.seed<<<blocks_for(before_count), kRingBlock, 0, stream>>>(r, static_cast<const unsigned long long*>(before),
                                                                before_count, key_mask, 1);
    ++out->launches;
  }
  MG_CHECK_RING(cudaGetLastError());
  int per_sm = 0;
  MG_CHECK_RING(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, reinterpret_cast<const void*>(k.wave), kRingBlock, 0));
  if (per_sm < 1) return MGBFS2_UNSUPPORTED;
  const uint64_t blocks = std::min<uint64_t>((r.nodes + kRingBlock - 1) / kRingBlock,
                                             static_cast<uint64_t>(per_sm) * sm_count);
  void* args[] = {&r};
  MG_CHECK_RING(cudaLaunchCooperativeKernel(reinterpret_cast<const void*>(k.wave), dim3(static_cast<uint32_t>(blocks)),
                                            dim3(kRingBlock), args, 0, stream));
  ++out->launches;
  MG_CHECK_RING(cudaStreamSynchronize(stream));
  const SearchEnd end = search_end(report->steps, report->error, stride, ERR_WAIT_LIMIT);
  out->fatal = end.fatal;
  const uint32_t steps = report->steps, cols = end.columns;
  std::vector<unsigned long long> counts(cols), stamps(cols);
  if (cols <= kRingReportLayers) {
    std::memcpy(counts.data(), report->counts, 8ull * cols);
    std::memcpy(stamps.data(), report->stamps, 8ull * cols);
  } else {
    MG_CHECK_RING(cudaMemcpyAsync(counts.data(), r.counts, 8ull * cols, cudaMemcpyDeviceToHost, stream));
    MG_CHECK_RING(cudaMemcpyAsync(stamps.data(), r.stamps, 8ull * cols, cudaMemcpyDeviceToHost, stream));
    MG_CHECK_RING(cudaStreamSynchronize(stream));
  }
  if (out->fatal) return MGBFS2_OK;
  for (uint32_t d = 1; d < cols && counts[d]; ++d) {
    out->layers.push_back(counts[d]);
    out->seconds.push_back(static_cast<double>(stamps[d] - stamps[d - 1]) * 1e-9);
  }
  out->kernel_seconds = cols > 1 ? static_cast<double>(stamps[cols - 1] - stamps[0]) * 1e-9 : 0.0;
  out->overflow = steps > r.max_steps && counts[steps] != 0;
  if (out->overflow || out->layers.empty()) return MGBFS2_OK;
  out->previous_small.assign(report->previous, report->previous + report->previous_count);
  const uint64_t deepest = out->layers.back();
  if ((rc = collect->ensure((deepest + 2) * 8))) return rc;
  r.front = static_cast<unsigned long long*>(collect->ptr);
  r.front_cap = deepest;
  k.collect<<<static_cast<uint32_t>(blocks), kRingBlock, 0, stream>>>(r, steps - 1);
  ++out->launches;
  MG_CHECK_RING(cudaGetLastError());
  MG_CHECK_RING(cudaStreamSynchronize(stream));
  if (deepest <= kRingSmall) out->deepest_small.assign(report->deepest, report->deepest + deepest);
  return MGBFS2_OK;
}

}  // namespace mgbfs2
