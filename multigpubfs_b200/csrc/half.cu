// Half-rank layers (see half.h): tables, the persistent wave kernel and its
// host side.
#include "half.h"
#include "search_end.h"

#include <algorithm>
#include <cstring>

#define MG_CHECK_HALF(expr)                        \
  do {                                             \
    cudaError_t _e = (expr);                       \
    if (_e != cudaSuccess) return cuda_status(_e); \
  } while (0)

namespace mgbfs2 {
namespace {

constexpr uint32_t kHalfBlock = 256, kHalfReportLayers = 512;
constexpr uint32_t kHalfStage = 2048;   // winners a block stages between two reservations
constexpr uint32_t kHalfMaxTerms = 512;
constexpr uint32_t kLutSize = 1u << 12;  // four symbols of three bits

struct HalfCtl {
  uint32_t arrived, error;
};

struct HalfReport {
  uint32_t steps, error;
  unsigned long long counts[kHalfReportLayers], stamps[kHalfReportLayers];
  unsigned long long previous[kHalfSmall], deepest[kHalfSmall];
};

struct HalfParams {
  uint32_t n, bits, distinct, gens, total_terms, gen_shift, max_steps, front_bits;
  uint32_t first_symbols;      // symbols of the first half
  uint32_t counts_of[kHalfMaxLabels];
  uint32_t entries[2];         // table entries of each half
  unsigned long long total, capacity, start;
  uint32_t* before;            // per first half: states whose first half is smaller
  uint32_t* within;            // per second half: its rank among its own arrangements
  const Term* terms;
  const uint32_t* term_begin;  // gens + 1 offsets, then inverse[gens]
  uint32_t* bitmap;
  unsigned long long* list[2];
  unsigned long long* counts;
  unsigned long long* stamps;
  HalfReport* report;
  unsigned long long* front;
  unsigned long long front_cap;
  HalfCtl* ctl;
};

// Table index of up to eight symbols: the bits themselves for one or two bits
// a symbol, else the number with the symbols as digits of base `distinct`,
// four at a time through a table in shared memory.
template <int BITS>
__device__ __forceinline__ uint32_t half_index(uint32_t field, const uint16_t* lut, uint32_t quad) {
  if constexpr (BITS < 3) return field;
  else return lut[field & (kLutSize - 1)] + quad * lut[field >> 12];
}

template <int BITS>
__device__ __forceinline__ uint32_t half_rank(const HalfParams& p, unsigned long long w, const uint16_t* lut, uint32_t quad) {
  const uint32_t split = BITS * p.first_symbols;
  const uint32_t lo = static_cast<uint32_t>(w) & ((1u << split) - 1u), hi = static_cast<uint32_t>(w >> split);
  return __ldg(p.before + half_index<BITS>(lo, lut, quad)) + __ldg(p.within + half_index<BITS>(hi, lut, quad));
}

template <int BITS>
__device__ __forceinline__ void load_lut(const HalfParams& p, uint16_t* lut) {
  if constexpr (BITS == 3) {
    for (uint32_t i = threadIdx.x; i < kLutSize; i += blockDim.x) {
      uint32_t v = 0, weight = 1;
      for (uint32_t s = 0; s < 4; ++s, weight *= p.distinct) v += min((i >> (3 * s)) & 7u, p.distinct - 1) * weight;
      lut[i] = static_cast<uint16_t>(v);
    }
  }
}

// Both tables; halves that no state has keep what the recurrence gives them
// (they are never read).
template <int BITS>
__global__ void __launch_bounds__(kHalfBlock) half_tables(HalfParams p) {
  const uint32_t step = gridDim.x * blockDim.x;
  for (uint32_t t = blockIdx.x * blockDim.x + threadIdx.x; t < p.entries[0] + p.entries[1]; t += step) {
    const bool second = t >= p.entries[0];
    const uint32_t index = second ? t - p.entries[0] : t;
    const uint32_t symbols = second ? p.n - p.first_symbols : p.first_symbols;
    uint32_t left[kHalfMaxLabels], rest = index;
#pragma unroll
    for (uint32_t c = 0; c < kHalfMaxLabels; ++c) left[c] = second ? 0u : p.counts_of[c];
    unsigned long long code = 0;  // the half's symbols, four bits each past eight: two words
    unsigned long long code2 = 0;
    bool valid = true;
    for (uint32_t e = 0; e < symbols; ++e) {
      uint32_t s;
      if constexpr (BITS < 3) {
        s = rest & ((1u << BITS) - 1u);
        rest >>= BITS;
      } else {
        s = rest % p.distinct;
        rest /= p.distinct;
      }
      if (e < 16) code |= static_cast<unsigned long long>(s) << (4 * e);
      else code2 |= static_cast<unsigned long long>(s) << (4 * (e - 16));
      valid = valid && s < p.distinct;
      if (second) {
#pragma unroll
        for (uint32_t c = 0; c < kHalfMaxLabels; ++c) left[c] += s == c ? 1u : 0u;
      }
    }
    // Arrangements of what `left` holds.
    unsigned long long ways = p.total;
    uint32_t remaining = p.n;
    if (second) {
      ways = 1;
      remaining = 0;
#pragma unroll
      for (uint32_t c = 0; c < kHalfMaxLabels; ++c)
        for (uint32_t k = 1; k <= left[c]; ++k) ways = ways * ++remaining / k;
    }
    unsigned long long rank = 0;
    for (uint32_t e = 0; e < symbols && valid; ++e, --remaining) {
      const uint32_t s = static_cast<uint32_t>((e < 16 ? code >> (4 * e) : code2 >> (4 * (e - 16))) & 15u);
      uint32_t less = 0, mine = 0;
#pragma unroll
      for (uint32_t c = 0; c < kHalfMaxLabels; ++c) {
        less += c < s ? left[c] : 0u;
        mine = c == s ? left[c] : mine;
        left[c] -= c == s && left[c] ? 1u : 0u;
      }
      if (!mine) {
        valid = false;
        break;
      }
      rank += scale_floor(ways, less, remaining);
      ways = scale_floor(ways, mine, remaining);
    }
    (second ? p.within : p.before)[index] = valid ? static_cast<uint32_t>(rank) : 0u;
  }
  if (blockIdx.x == 0 && threadIdx.x == 0) {
    p.list[0][0] = p.start;
    p.counts[0] = 1;
  }
}

// A state's codes in words of front_bits a symbol (four, when it fits one word).
__device__ __forceinline__ unsigned long long widen(unsigned long long w, const HalfParams& p) {
  unsigned long long out = 0;
  for (uint32_t e = 0; e < p.n; ++e)
    out |= ((w >> (p.bits * e)) & ((1ull << p.bits) - 1ull)) << (p.front_bits * e);
  return out;
}

__device__ void half_finish(const HalfParams& p, uint32_t d) {
  const unsigned long long size = __ldcg(p.counts + d);
  const unsigned long long keep = p.gen_shift ? (1ull << p.gen_shift) - 1ull : ~0ull;
  const unsigned long long* deepest = d & 1u ? p.list[1] : p.list[0];
  if (p.front && size <= p.front_cap)
    for (unsigned long long k = blockIdx.x * static_cast<unsigned long long>(blockDim.x) + threadIdx.x; k < size;
         k += static_cast<unsigned long long>(gridDim.x) * blockDim.x)
      p.front[k] = widen(deepest[k] & keep, p);
  if (blockIdx.x) return;
  const unsigned long long before = d ? __ldcg(p.counts + d - 1) : 0ull;
  const unsigned long long* previous = d & 1u ? p.list[0] : p.list[1];
  for (uint32_t k = threadIdx.x; k < kHalfSmall; k += blockDim.x) {
    if (k < size) p.report->deepest[k] = deepest[k] & keep;
    if (k < before && before < kHalfSmall) p.report->previous[k] = previous[k] & keep;
  }
  for (uint32_t k = threadIdx.x; k < kHalfReportLayers && k <= d + 1; k += blockDim.x) {
    p.report->counts[k] = __ldcg(p.counts + k);
    p.report->stamps[k] = p.stamps[k];
  }
  if (threadIdx.x == 0) {
    p.report->steps = d + 1;
    p.report->error = p.ctl->error;
  }
}

// A whole search per launch.  A block takes tiles of 256 parents; a child costs
// its displacement terms, two table reads and one atomic on the bitmap (in L2
// for the domains taken here); winners are staged and appended with one
// reservation per flush.
template <int BITS>
__global__ void __launch_bounds__(kHalfBlock, 6) half_wave_kernel(HalfParams p) {
  __shared__ unsigned long long out[kHalfStage];
  __shared__ Term terms[kHalfMaxTerms];
  __shared__ uint32_t begin[2 * kHalfMaxGens + 1];
  __shared__ uint16_t lut[BITS == 3 ? kLutSize : 1];
  __shared__ uint32_t staged;
  __shared__ unsigned long long reserved;
  const uint32_t lane = threadIdx.x & 31u;
  load_lut<BITS>(p, lut);
  for (uint32_t i = threadIdx.x; i < p.total_terms; i += blockDim.x) terms[i] = p.terms[i];
  for (uint32_t i = threadIdx.x; i <= 2 * p.gens; i += blockDim.x) begin[i] = p.term_begin[i];
  if (threadIdx.x == 0) staged = 0;
  __syncthreads();
  const uint32_t quad = p.distinct * p.distinct * p.distinct * p.distinct;
  const unsigned long long key = p.gen_shift ? (1ull << p.gen_shift) - 1ull : ~0ull;
  uint32_t epoch = 0;
  if (blockIdx.x == 0 && threadIdx.x == 0) {
    const uint32_t r = half_rank<BITS>(p, p.start, lut, quad);
    atomicOr(p.bitmap + (r >> 5), 1u << (r & 31u));
  }
  if (!arrival_barrier(&p.ctl->arrived, &p.ctl->error, &epoch)) return;
  for (uint32_t d = 0;; ++d) {
    if (blockIdx.x == 0 && threadIdx.x == 0) p.stamps[d] = global_ns();
    const unsigned long long count = __ldcg(p.counts + d);
    const unsigned long long* cur = d & 1u ? p.list[1] : p.list[0];
    unsigned long long* nxt = d & 1u ? p.list[0] : p.list[1];
    const auto flush = [&]() {
      __syncthreads();
      const uint32_t n = staged;
      if (threadIdx.x == 0 && n) reserved = atomicAdd(p.counts + d + 1, static_cast<unsigned long long>(n));
      __syncthreads();
      bool lost = false;
      for (uint32_t k = threadIdx.x; k < n; k += blockDim.x) {
        if (reserved + k < p.capacity) nxt[reserved + k] = out[k];
        else lost = true;
      }
      if (lost) raise_error(&p.ctl->error, ERR_FRONTIER_OVERFLOW);
      __syncthreads();
      if (threadIdx.x == 0) staged = 0;
      __syncthreads();
    };
    for (unsigned long long base = static_cast<unsigned long long>(blockIdx.x) * kHalfBlock; base < count;
         base += static_cast<unsigned long long>(gridDim.x) * kHalfBlock) {
      const bool valid = base + threadIdx.x < count;
      const unsigned long long w = valid ? cur[base + threadIdx.x] : 0ull;
      const uint32_t tag = p.gen_shift ? static_cast<uint32_t>(w >> p.gen_shift) : 0u;
      const uint32_t skip = tag ? begin[p.gens + tag] : 0xffffffffu;  // inverse[tag - 1]
      const unsigned long long state = w & key;
      for (uint32_t g = 0; g < p.gens; ++g) {
        bool won = false;
        unsigned long long c = 0;
        if (valid && g != skip) {
          c = apply_terms(state, terms, begin[g], begin[g + 1]);
          const uint32_t r = half_rank<BITS>(p, c, lut, quad), bit = 1u << (r & 31u);
          won = !(atomicOr(p.bitmap + (r >> 5), bit) & bit);
        }
        const uint32_t m = __ballot_sync(kFullMask, won);
        if (m) {
          uint32_t at = 0;
          const int leader = __ffs(static_cast<int>(m)) - 1;
          if (static_cast<int>(lane) == leader) at = atomicAdd(&staged, static_cast<uint32_t>(__popc(m)));
          at = __shfl_sync(kFullMask, at, leader) + __popc(m & ((1u << lane) - 1u));
          if (won) out[at] = c | (p.gen_shift ? static_cast<unsigned long long>(g + 1) << p.gen_shift : 0ull);
        }
        // Room for the next generator's winners of every thread.
        if ((g + 1) % (kHalfStage / kHalfBlock) == 0 && g + 1 < p.gens) flush();
      }
      flush();
    }
    if (!arrival_barrier(&p.ctl->arrived, &p.ctl->error, &epoch)) return;
    const bool more = __ldcg(p.counts + d + 1) != 0;
    if (more && d < p.max_steps && !__ldcg(&p.ctl->error)) continue;
    if (blockIdx.x == 0) {
      if (threadIdx.x == 0) p.stamps[d + 1] = global_ns();
      __syncthreads();
    }
    half_finish(p, d);
    return;
  }
}

__global__ void __launch_bounds__(kHalfBlock) half_collect(HalfParams p, uint32_t last) { half_finish(p, last); }

size_t al256(size_t x) { return (x + 255) / 256 * 256; }

uint32_t half_code_bits(uint32_t distinct) { return distinct <= 2 ? 1 : (distinct <= 4 ? 2 : 3); }

uint64_t half_entries(uint32_t symbols, uint32_t bits, uint32_t distinct) {
  uint64_t e = 1;
  for (uint32_t i = 0; i < symbols; ++i) e *= bits < 3 ? 1u << bits : distinct;
  return e;
}

}  // namespace

// The generators' displacement terms: one for every distinct shift of each.
static uint32_t half_terms(const HalfJob& job) {
  uint32_t terms = 0;
  for (uint32_t g = 0; g < job.gens; ++g) {
    const uint32_t* s = job.perms + static_cast<size_t>(g) * job.n;
    uint64_t shifts[2] = {0, 0};  // bit n + s[i] - i
    for (uint32_t i = 0; i < job.n; ++i) {
      const uint32_t at = job.n + s[i] - i;
      shifts[at / 64] |= 1ull << (at % 64);
    }
    terms += static_cast<uint32_t>(__builtin_popcountll(shifts[0]) + __builtin_popcountll(shifts[1]));
  }
  return terms;
}

bool half_supported(const HalfJob& job) {
  const uint32_t n = job.n, distinct = job.distinct;
  if (n < 2 || n > 36 || distinct < 1 || distinct > kHalfMaxLabels || !job.gens || job.gens > kHalfMaxGens) return false;
  if (job.total < 1 || job.total >= UINT32_MAX) return false;
  const uint32_t bits = half_code_bits(distinct), half = (n + 1) / 2;
  // Three-bit halves are indexed as two table lookups of four symbols.  More
  // terms than a block keeps in shared memory (32 random generators of 24
  // positions: 570) go to the wide hash; 16 positions cannot have more.
  return n * bits <= 64 && half * bits <= 31 && (bits < 3 || half <= 8) &&
         half_entries(half, bits, distinct) <= (1ull << kHalfIndexBits) && half_terms(job) <= kHalfMaxTerms;
}

uint64_t half_bytes(const HalfJob& job, uint32_t max_layers) {
  const uint32_t bits = half_code_bits(job.distinct), half = (job.n + 1) / 2;
  return 8 * half_entries(half, bits, job.distinct) + 16 * (job.capacity + 2) + 16ull * (max_layers + 2) +
         24ull * kHalfMaxTerms + 16 * 256;
}

int half_wave(const HalfJob& job, uint32_t max_layers, int sm_count, cudaStream_t stream, HalfMemory* memory,
              DeviceBuffer* bitmap, DeviceBuffer* front, uint32_t front_bits, HalfResult* out) {
  if (!half_supported(job) || !max_layers) return MGBFS2_INVALID_ARGUMENT;
  HalfParams p{};
  p.n = job.n;
  p.distinct = job.distinct;
  p.bits = out->bits = half_code_bits(job.distinct);
  p.gens = job.gens;
  p.total = job.total;
  p.capacity = job.capacity;
  p.max_steps = max_layers - 1;
  p.front_bits = front_bits;
  p.first_symbols = (job.n + 1) / 2;
  for (uint32_t c = 0; c < job.distinct; ++c) p.counts_of[c] = job.counts[c];
  p.entries[0] = static_cast<uint32_t>(half_entries(p.first_symbols, p.bits, job.distinct));
  p.entries[1] = static_cast<uint32_t>(half_entries(job.n - p.first_symbols, p.bits, job.distinct));
  for (uint32_t i = 0; i < job.n; ++i) p.start |= static_cast<unsigned long long>(job.codes[i]) << (p.bits * i);
  // Displacement terms and, in the bits above the codes, the generator that
  // produced a state: its inverse leads back and is not tested.
  std::vector<Term> terms;
  std::vector<uint32_t> begin(1, 0);
  const unsigned long long symbol = (1ull << p.bits) - 1ull;
  for (uint32_t g = 0; g < job.gens; ++g) {
    const uint32_t* s = job.perms + static_cast<size_t>(g) * job.n;
    for (int disp = -static_cast<int>(job.n) + 1; disp < static_cast<int>(job.n); ++disp) {
      unsigned long long mask = 0;
      for (uint32_t i = 0; i < job.n; ++i)
        if (static_cast<int>(s[i]) - static_cast<int>(i) == disp) mask |= symbol << (p.bits * i);
      if (!mask) continue;
      const int shift = disp * static_cast<int>(p.bits);
      terms.push_back(Term{mask, shift > 0 ? static_cast<uint32_t>(shift) : 0u, shift < 0 ? static_cast<uint32_t>(-shift) : 0u});
    }
    begin.push_back(static_cast<uint32_t>(terms.size()));
  }
  p.total_terms = static_cast<uint32_t>(terms.size());
  const uint32_t tag_bits = 32 - static_cast<uint32_t>(__builtin_clz(job.gens));
  if (job.inverse_closed && job.n * p.bits + tag_bits <= 64) p.gen_shift = job.n * p.bits;
  for (uint32_t g = 0; g < job.gens; ++g) {
    const uint32_t* a = job.perms + static_cast<size_t>(g) * job.n;
    uint32_t inverse = 0xffffffffu;
    for (uint32_t h = 0; h < job.gens && inverse == 0xffffffffu; ++h) {
      const uint32_t* b = job.perms + static_cast<size_t>(h) * job.n;
      bool is = true;
      for (uint32_t i = 0; i < job.n && is; ++i) is = b[a[i]] == i;
      if (is) inverse = h;
    }
    begin.push_back(inverse);
  }
  const uint32_t stride = max_layers + 2;
  size_t off = 0;
  const auto take = [&off](size_t bytes) {
    const size_t at = off;
    off = al256(off + bytes);
    return at;
  };
  const size_t o_terms = take(terms.size() * sizeof(Term)), o_begin = take(begin.size() * 4);
  const size_t upload = off;
  const size_t o_counts = take(8ull * stride), o_ctl = take(sizeof(HalfCtl));
  const size_t cleared = off;
  const size_t o_stamps = take(8ull * stride), o_before = take(4ull * p.entries[0]), o_within = take(4ull * p.entries[1]);
  memory->deepest = nullptr;
  int rc = memory->arena.ensure(off, true);
  for (DeviceBuffer& b : memory->list)
    if (!rc) rc = b.ensure((job.capacity + 2) * 8, true);
  const size_t bitmap_bytes = (job.total + 63) / 64 * 8;
  if (!rc) rc = bitmap->ensure(bitmap_bytes);
  if (!rc && front) rc = front->ensure((kHalfSmall + 2) * 8);
  if (!rc && !memory->report) rc = pinned_take(sizeof(HalfReport), &memory->report);
  if (rc) return rc;
  HalfReport* report = static_cast<HalfReport*>(memory->report);
  report->steps = 0;
  char* base = static_cast<char*>(memory->arena.ptr);
  p.terms = reinterpret_cast<const Term*>(base + o_terms);
  p.term_begin = reinterpret_cast<const uint32_t*>(base + o_begin);
  p.counts = reinterpret_cast<unsigned long long*>(base + o_counts);
  p.ctl = reinterpret_cast<HalfCtl*>(base + o_ctl);
  p.stamps = reinterpret_cast<unsigned long long*>(base + o_stamps);
  p.before = reinterpret_cast<uint32_t*>(base + o_before);
  p.within = reinterpret_cast<uint32_t*>(base + o_within);
  p.bitmap = static_cast<uint32_t*>(bitmap->ptr);
  p.list[0] = static_cast<unsigned long long*>(memory->list[0].ptr);
  p.list[1] = static_cast<unsigned long long*>(memory->list[1].ptr);
  p.report = report;
  if (front) {
    p.front = static_cast<unsigned long long*>(front->ptr);
    p.front_cap = front->bytes / 8;
  }
  std::vector<char> host(upload);
  std::memcpy(host.data() + o_terms, terms.data(), terms.size() * sizeof(Term));
  std::memcpy(host.data() + o_begin, begin.data(), begin.size() * 4);
  MG_CHECK_HALF(cudaMemcpyAsync(base, host.data(), upload, cudaMemcpyHostToDevice, stream));
  MG_CHECK_HALF(cudaMemsetAsync(base + upload, 0, cleared - upload, stream));
  MG_CHECK_HALF(cudaMemsetAsync(bitmap->ptr, 0, bitmap_bytes, stream));
  const void* wave = p.bits == 1   ? reinterpret_cast<const void*>(half_wave_kernel<1>)
                     : p.bits == 2 ? reinterpret_cast<const void*>(half_wave_kernel<2>)
                                   : reinterpret_cast<const void*>(half_wave_kernel<3>);
  const uint32_t table_blocks = std::min<uint32_t>((p.entries[0] + p.entries[1] + kHalfBlock - 1) / kHalfBlock, 8u * static_cast<uint32_t>(sm_count));
  if (p.bits == 1) half_tables<1><<<table_blocks, kHalfBlock, 0, stream>>>(p);
  else if (p.bits == 2) half_tables<2><<<table_blocks, kHalfBlock, 0, stream>>>(p);
  else half_tables<3><<<table_blocks, kHalfBlock, 0, stream>>>(p);
  MG_CHECK_HALF(cudaGetLastError());
  const int want = size_carveout(wave, 0, 6, kHalfBlock);
  int per_sm = 0;
  MG_CHECK_HALF(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, wave, kHalfBlock, 0));
  per_sm = std::min(per_sm, want);
  if (per_sm < 1) return MGBFS2_UNSUPPORTED;
  const uint64_t tiles = (job.capacity + kHalfBlock - 1) / kHalfBlock;
  const uint32_t blocks = static_cast<uint32_t>(std::min<uint64_t>(std::max<uint64_t>(tiles, 1), static_cast<uint64_t>(per_sm) * sm_count));
  void* args[] = {&p};
  MG_CHECK_HALF(cudaLaunchCooperativeKernel(wave, dim3(blocks), dim3(kHalfBlock), args, 0, stream));
  MG_CHECK_HALF(cudaStreamSynchronize(stream));
  out->launches = 2;
  const SearchEnd end = search_end(report->steps, report->error, stride, ERR_WAIT_LIMIT);
  out->fatal = end.fatal;
  const uint32_t cols = end.columns;
  std::vector<unsigned long long> counts(cols), stamps(cols);
  if (cols <= kHalfReportLayers) {
    std::memcpy(counts.data(), report->counts, 8ull * cols);
    std::memcpy(stamps.data(), report->stamps, 8ull * cols);
  } else {
    MG_CHECK_HALF(cudaMemcpyAsync(counts.data(), p.counts, 8ull * cols, cudaMemcpyDeviceToHost, stream));
    MG_CHECK_HALF(cudaMemcpyAsync(stamps.data(), p.stamps, 8ull * cols, cudaMemcpyDeviceToHost, stream));
    MG_CHECK_HALF(cudaStreamSynchronize(stream));
  }
  if (out->fatal) {
    out->layers.assign(1, 1);
    return MGBFS2_OK;
  }
  for (uint32_t d = 0; d < cols && counts[d]; ++d) {
    out->layers.push_back(counts[d]);
    if (d) out->seconds.push_back(static_cast<double>(stamps[d] - stamps[d - 1]) * 1e-9);
  }
  out->kernel_seconds = cols > 1 ? static_cast<double>(stamps[cols - 1] - stamps[0]) * 1e-9 : 0.0;
  out->overflow = out->layers.size() > max_layers;
  if (out->overflow) return MGBFS2_OK;
  const uint64_t deepest = out->layers.back(), last = out->layers.size() - 1;
  memory->deepest = reinterpret_cast<const uint64_t*>(p.list[last & 1]);
  memory->key_mask = p.gen_shift ? (1ull << p.gen_shift) - 1ull : ~0ull;
  memory->bits = p.bits;
  out->deepest.assign(report->deepest, report->deepest + std::min<uint64_t>(deepest, kHalfSmall));
  if (last && out->layers[last - 1] < kHalfSmall)
    out->previous.assign(report->previous, report->previous + out->layers[last - 1]);
  if (!front || deepest <= p.front_cap) return MGBFS2_OK;
  if ((rc = front->ensure((deepest + 2) * 8))) return rc;
  p.front = static_cast<unsigned long long*>(front->ptr);
  p.front_cap = deepest;
  half_collect<<<blocks, kHalfBlock, 0, stream>>>(p, static_cast<uint32_t>(last));
  ++out->launches;
  MG_CHECK_HALF(cudaGetLastError());
  MG_CHECK_HALF(cudaStreamSynchronize(stream));
  return MGBFS2_OK;
}

}  // namespace mgbfs2
