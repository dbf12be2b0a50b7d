// Scalar-ring layers (see ring.h): seeding from frontier lists, the persistent
// wave kernel and its host side.
#include "ring.h"

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

struct RingParams {
  uint32_t p, bits, gens, magic;   // magic: floor(2^32 / p)
  uint32_t nodes, max_steps;
  const uint16_t* inverse;         // p entries: x^-1, then dlog x, then g^t
  uint32_t* buf[2];
  unsigned long long* counts;      // max_steps + 2 layer sizes; 0 = the seeded layer
  unsigned long long* stamps;
  uint32_t* small_count;
  unsigned long long* small;       // 2 x kRingSmall (node << 8 | bit), by step parity
  RingReport* report;
  unsigned long long* front;
  unsigned long long front_cap;
  RingCtl* ctl;
  uint32_t coef[4 * kRingMaxGens];
};

__device__ __forceinline__ uint32_t reduce(uint32_t x, const RingParams& r) {
  uint32_t y = x - __umulhi(x, r.magic) * r.p;  // quotient short by at most one
  return y >= r.p ? y - r.p : y;
}

struct Tables {
  uint16_t inverse[kRingMaxPrime], log[kRingMaxPrime], power[kRingMaxPrime];
};

__device__ __forceinline__ void load_tables(const RingParams& r, Tables& t) {
  for (uint32_t i = threadIdx.x; i < r.p; i += blockDim.x) {
    t.inverse[i] = r.inverse[i];
    t.log[i] = r.inverse[r.p + i];
    t.power[i] = r.inverse[2 * r.p + i];
  }
  __syncthreads();
}

// Node and scalar (its discrete logarithm) of a nonzero matrix.
__device__ __forceinline__ uint32_t node_of(uint32_t a, uint32_t b, uint32_t c, uint32_t d, const RingParams& r,
                                            const Tables& t, uint32_t* log) {
  const uint32_t p = r.p;
  if (a) {
    const uint32_t i = t.inverse[a];
    *log = t.log[a];
    return (reduce(c * i, r) * p + reduce(b * i, r)) * p + reduce(d * i, r);
  }
  if (c) {
    const uint32_t i = t.inverse[c];
    *log = t.log[c];
    return p * p * p + reduce(b * i, r) * p + reduce(d * i, r);
  }
  if (b) {
    *log = t.log[b];
    return p * p * p + p * p + reduce(d * t.inverse[b], r);
  }
  *log = t.log[d];
  return p * p * p + p * p + p;
}

__device__ __forceinline__ void matrix_of(uint32_t node, const RingParams& r, uint32_t* a, uint32_t* b, uint32_t* c,
                                          uint32_t* d) {
  const uint32_t p = r.p, square = p * p, cube = square * p;
  if (node < cube) {
    const uint32_t rest = node / p;
    *d = node - rest * p;
    *c = rest / p;
    *b = rest - *c * p;
    *a = 1;
    return;
  }
  node -= cube;
  *a = 0;
  if (node < square) {
    *b = node / p;
    *d = node - *b * p;
    *c = 1;
    return;
  }
  node -= square;
  *c = 0;
  *b = node < p ? 1u : 0u;
  *d = node < p ? node : 1u;
}

__device__ __forceinline__ unsigned long long pack_matrix(uint32_t node, uint32_t bit, const RingParams& r,
                                                          const Tables& t) {
  uint32_t a, b, c, d;
  matrix_of(node, r, &a, &b, &c, &d);
  const uint32_t s = t.power[bit];
  return static_cast<unsigned long long>(reduce(a * s, r)) | (static_cast<unsigned long long>(reduce(b * s, r)) << r.bits) |
         (static_cast<unsigned long long>(reduce(c * s, r)) << (2 * r.bits)) |
         (static_cast<unsigned long long>(reduce(d * s, r)) << (3 * r.bits));
}

// Marks the states of a list in a buffer.
template <int NW>
__global__ void __launch_bounds__(kRingBlock) ring_seed(RingParams r, const unsigned long long* list,
                                                        unsigned long long count, unsigned long long key_mask,
                                                        uint32_t which) {
  __shared__ Tables t;
  load_tables(r, t);
  uint32_t* buf = which ? r.buf[1] : r.buf[0];
  const uint32_t mask = (1u << r.bits) - 1u;
  for (unsigned long long k = blockIdx.x * static_cast<unsigned long long>(blockDim.x) + threadIdx.x; k < count;
       k += static_cast<unsigned long long>(gridDim.x) * blockDim.x) {
    const unsigned long long w = list[k] & key_mask;
    uint32_t log;
    const uint32_t node = node_of(static_cast<uint32_t>(w) & mask, static_cast<uint32_t>(w >> r.bits) & mask,
                                  static_cast<uint32_t>(w >> (2 * r.bits)) & mask,
                                  static_cast<uint32_t>(w >> (3 * r.bits)) & mask, r, t, &log);
    atomicOr(buf + static_cast<size_t>(node) * NW + (log >> 5), 1u << (log & 31u));
  }
  if (blockIdx.x == 0 && threadIdx.x == 0 && !which) r.counts[0] = count;
}

template <int NW>
__device__ __forceinline__ void load_ring(const uint32_t* at, uint32_t (&w)[NW]) {
  if constexpr (NW == 8) {
    const uint4 lo = *reinterpret_cast<const uint4*>(at), hi = *reinterpret_cast<const uint4*>(at + 4);
    w[0] = lo.x, w[1] = lo.y, w[2] = lo.z, w[3] = lo.w, w[4] = hi.x, w[5] = hi.y, w[6] = hi.z, w[7] = hi.w;
  } else if constexpr (NW == 4) {
    const uint4 lo = *reinterpret_cast<const uint4*>(at);
    w[0] = lo.x, w[1] = lo.y, w[2] = lo.z, w[3] = lo.w;
  } else if constexpr (NW == 2) {
    const uint2 lo = *reinterpret_cast<const uint2*>(at);
    w[0] = lo.x, w[1] = lo.y;
  } else {
    w[0] = *at;
  }
}

template <int NW>
__device__ __forceinline__ void store_ring(uint32_t* at, const uint32_t (&w)[NW]) {
  if constexpr (NW == 8) {
    *reinterpret_cast<uint4*>(at) = make_uint4(w[0], w[1], w[2], w[3]);
    *reinterpret_cast<uint4*>(at + 4) = make_uint4(w[4], w[5], w[6], w[7]);
  } else if constexpr (NW == 4) {
    *reinterpret_cast<uint4*>(at) = make_uint4(w[0], w[1], w[2], w[3]);
  } else if constexpr (NW == 2) {
    *reinterpret_cast<uint2*>(at) = make_uint2(w[0], w[1]);
  } else {
    *at = w[0];
  }
}

// acc |= the ring of `length` bits rotated right by s (bits from `length` up
// of acc are dropped by the caller).
template <int NW>
__device__ __forceinline__ void or_rotated(uint32_t (&acc)[NW], const uint32_t (&x)[NW], uint32_t s, uint32_t length) {
  const uint32_t n = s ? length - s : 0u;
  uint32_t y[NW + 1], z[NW + 1];  // y: x moved down by whole words; z: moved up, z[0] below word 0
#pragma unroll
  for (int i = 0; i < NW; ++i) y[i] = z[i + 1] = x[i];
  y[NW] = z[0] = 0;
#pragma unroll
  for (int by = NW / 2; by; by /= 2) {
    const bool down = (s >> 5) & by, up = (n >> 5) & by;
#pragma unroll
    for (int i = 0; i < NW; ++i) y[i] = down ? (i + by < NW ? y[i + by] : 0u) : y[i];
#pragma unroll
    for (int i = NW; i > 0; --i) z[i] = up ? (i - by > 0 ? z[i - by] : 0u) : z[i];
  }
#pragma unroll
  for (int i = 0; i < NW; ++i)
    acc[i] |= __funnelshift_r(y[i], y[i + 1], s & 31u) | __funnelshift_l(z[i], z[i + 1], n & 31u);
}

// The states of layer d (from the seeded one) as packed words, and block 0's report.
template <int NW>
__device__ void ring_finish(const RingParams& r, const Tables& t, uint32_t d, bool exhausted) {
  const uint32_t step = gridDim.x * blockDim.x;
  if (exhausted && d && __ldcg(r.counts + d) <= r.front_cap) {
    const uint32_t* buf = d & 1u ? r.buf[1] : r.buf[0];
    for (uint32_t node = blockIdx.x * blockDim.x + threadIdx.x; node < r.nodes; node += step) {
      uint32_t w[NW];
      load_ring<NW>(buf + static_cast<size_t>(node) * NW, w);
      uint32_t mine = 0;
#pragma unroll
      for (int i = 0; i < NW; ++i) mine += __popc(w[i]);
      if (!mine) continue;
      unsigned long long at = atomicAdd(&r.ctl->collected, static_cast<unsigned long long>(mine));
#pragma unroll
      for (int i = 0; i < NW; ++i)
        for (uint32_t b = w[i]; b; b &= b - 1, ++at) {
          const unsigned long long s = pack_matrix(node, 32 * i + __ffs(static_cast<int>(b)) - 1, r, t);
          if (at < r.front_cap) r.front[at] = s;
          if (at < kRingSmall) r.report->deepest[at] = s;
        }
    }
  }
  if (blockIdx.x) return;
  const uint32_t kept = exhausted ? min(r.small_count[d], kRingSmall) : 0u;
  for (uint32_t k = threadIdx.x; k < kept; k += blockDim.x) {
    const unsigned long long at = r.small[(d & 1u) * kRingSmall + k];
    r.report->previous[k] = pack_matrix(static_cast<uint32_t>(at >> 8), static_cast<uint32_t>(at & 255u), r, t);
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

template <int NW>
__global__ void __launch_bounds__(kRingBlock, 4) ring_wave_kernel(RingParams r) {
  __shared__ Tables t;
  load_tables(r, t);
  const uint32_t step = gridDim.x * blockDim.x, length = r.p - 1;
  uint32_t top[NW];  // bits of the ring in each word
#pragma unroll
  for (int i = 0; i < NW; ++i) {
    const int left = static_cast<int>(length) - 32 * i;
    top[i] = left >= 32 ? 0xffffffffu : (left > 0 ? (1u << left) - 1u : 0u);
  }
  uint32_t epoch = 0;
  for (uint32_t d = 0;; ++d) {
    if (blockIdx.x == 0 && threadIdx.x == 0) r.stamps[d] = global_ns();
    const uint32_t* cur = d & 1u ? r.buf[1] : r.buf[0];
    uint32_t* nxt = d & 1u ? r.buf[0] : r.buf[1];
    const bool keep = d && __ldcg(r.counts + d - 1) < kRingSmall;
    uint32_t found = 0;
    for (uint32_t node = blockIdx.x * blockDim.x + threadIdx.x; node < r.nodes; node += step) {
      uint32_t a, b, c, e;
      matrix_of(node, r, &a, &b, &c, &e);
      uint32_t acc[NW];
#pragma unroll
      for (int i = 0; i < NW; ++i) acc[i] = 0;
#pragma unroll 2
      for (uint32_t g = 0; g < r.gens; ++g) {
        // The set is inverse-closed: its products are the parents.
        const uint32_t m0 = r.coef[4 * g], m1 = r.coef[4 * g + 1], m2 = r.coef[4 * g + 2], m3 = r.coef[4 * g + 3];
        uint32_t log, w[NW];
        const uint32_t from = node_of(reduce(m0 * a + m1 * c, r), reduce(m0 * b + m1 * e, r), reduce(m2 * a + m3 * c, r),
                                      reduce(m2 * b + m3 * e, r), r, t, &log);
        load_ring<NW>(cur + static_cast<size_t>(from) * NW, w);
        or_rotated<NW>(acc, w, log, length);
      }
      uint32_t own[NW], old[NW];
      load_ring<NW>(cur + static_cast<size_t>(node) * NW, own);
      load_ring<NW>(nxt + static_cast<size_t>(node) * NW, old);
      uint32_t changed = 0;
#pragma unroll
      for (int i = 0; i < NW; ++i) {
        acc[i] &= top[i] & ~(own[i] | old[i]);
        found += __popc(acc[i]);
        changed |= acc[i] | old[i];
      }
      if (keep) {
        // The small layer d - 1 is about to be overwritten.
#pragma unroll
        for (int i = 0; i < NW; ++i)
          for (uint32_t o = old[i]; o; o &= o - 1) {
            const uint32_t at = atomicAdd(r.small_count + d, 1u);
            if (at < kRingSmall)
              r.small[(d & 1u) * kRingSmall + at] =
                  (static_cast<unsigned long long>(node) << 8) | (32u * i + __ffs(static_cast<int>(o)) - 1u);
          }
      }
      if (changed) store_ring<NW>(nxt + static_cast<size_t>(node) * NW, acc);
    }
    found = __reduce_add_sync(kFullMask, found);
    if (found && (threadIdx.x & 31u) == 0) atomicAdd(r.counts + d + 1, static_cast<unsigned long long>(found));
    if (!arrival_barrier(&r.ctl->arrived, &r.ctl->error, &epoch)) return;
    const bool more = __ldcg(r.counts + d + 1) != 0;
    if (more && d < r.max_steps) continue;
    if (blockIdx.x == 0) {
      if (threadIdx.x == 0) r.stamps[d + 1] = global_ns();
      __syncthreads();
    }
    ring_finish<NW>(r, t, d, !more);
    return;
  }
}

template <int NW>
__global__ void __launch_bounds__(kRingBlock) ring_collect(RingParams r, uint32_t last) {
  __shared__ Tables t;
  load_tables(r, t);
  ring_finish<NW>(r, t, last, true);
}

size_t al256(size_t x) { return (x + 255) / 256 * 256; }

uint32_t ring_words(uint32_t p) {
  uint32_t w = 1;
  while (32 * w < p - 1) w *= 2;
  return w;
}

using SeedFn = void (*)(RingParams, const unsigned long long*, unsigned long long, unsigned long long, uint32_t);
using WaveFn = void (*)(RingParams);
using CollectFn = void (*)(RingParams, uint32_t);

struct RingKernels {
  SeedFn seed;
  WaveFn wave;
  CollectFn collect;
};

RingKernels kernels_for(uint32_t words) {
  switch (words) {
    case 1: return {ring_seed<1>, ring_wave_kernel<1>, ring_collect<1>};
    case 2: return {ring_seed<2>, ring_wave_kernel<2>, ring_collect<2>};
    case 4: return {ring_seed<4>, ring_wave_kernel<4>, ring_collect<4>};
    default: return {ring_seed<8>, ring_wave_kernel<8>, ring_collect<8>};
  }
}

}  // namespace

uint64_t ring_nodes(uint32_t p) {
  const uint64_t q = p;
  return q * q * q + q * q + q + 1;
}

uint64_t ring_bytes(uint32_t p, uint32_t max_layers) {
  return 2 * ring_nodes(p) * 4 * ring_words(p) + 20ull * (max_layers + 2) + 16ull * kRingSmall + 6ull * p + 16 * 256;
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
  r.nodes = static_cast<uint32_t>(ring_nodes(p));
  r.max_steps = max_layers - 1;
  std::copy_n(coef, 4 * gens, r.coef);
  // Tables: inverses, logarithms and powers of the least primitive root.
  std::vector<uint16_t> tables(3 * p, 0);
  for (uint32_t g = 2;; ++g) {
    uint32_t x = 1, order = 0;
    do {
      tables[2 * p + order] = static_cast<uint16_t>(x);
      tables[p + x] = static_cast<uint16_t>(order);
      x = x * g % p;
      ++order;
    } while (x != 1);
    if (order == p - 1) break;
  }
  for (uint32_t x = 1; x < p; ++x) {
    const uint32_t log = tables[p + x];
    tables[x] = tables[2 * p + (log ? p - 1 - log : 0)];
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
  const size_t cleared = off;
  const size_t o_stamps = take(8ull * stride), o_small = take(16ull * kRingSmall);
  int rc = memory->arena.ensure(off, true);
  const size_t word_bytes = ring_nodes(p) * 4 * words;
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
  out->launches = 1;
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
  out->fatal = report->steps ? report->error : static_cast<uint32_t>(ERR_WAIT_LIMIT);  // no report: a barrier gave up
  const uint32_t steps = report->steps, cols = std::min(steps + 1, stride);
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
