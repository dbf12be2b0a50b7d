// Coset-word layers (see coset.h for the coordinates): tables, the persistent
// wave kernel, the read-out of the deepest layer, and their host side.
#include "coset.h"
#include "search_end.h"

#include <algorithm>
#include <cstring>
#include <numeric>
#include <type_traits>

#define MG_CHECK_COSET(expr)                       \
  do {                                             \
    cudaError_t _e = (expr);                       \
    if (_e != cudaSuccess) return cuda_status(_e); \
  } while (0)

namespace mgbfs2 {
namespace {

constexpr uint32_t kSlots = 7, kSlotPerms = 5040;
constexpr uint32_t kCosetBlock = 256, kCosetWarps = kCosetBlock / 32;
constexpr uint32_t kMaxUnits = 8;  // units (128 nodes) of a work item
constexpr uint32_t kWideUnits = 4, kWideRows = 36;  // 64-bit words: units of an item, rows of a chunk
constexpr size_t kSmallMaxShared = 160 << 10;  // parent words of a block of the small kernel

constexpr uint32_t kNoWalk = 0xffffffffu;

struct CosetInst {
  uint32_t m, gens, rows, inverse_closed;
  uint32_t same_layer;  // some generator is an even permutation: a layer may have edges inside it
  uint32_t perm_off;    // first byte of gens x 16 position images
  uint32_t walk;        // 64-bit words: the generator whose orbits order the rows, kNoWalk without one
  unsigned long long row_off, desc_off;  // first row in the buffers and flags; first descriptor
};

struct CosetCtl {
  uint32_t arrived, error, steps, pad;
  unsigned long long collected;  // states of the deepest layer written out
};

// What the host reads of a wave of one job: pinned memory that the kernel
// writes at its end, so that the launch and one synchronisation are the whole
// read-back.  Layers past kReportLayers are copied from the tables.
constexpr uint32_t kReportLayers = 256;
struct CosetReport {
  uint32_t steps, error, previous_count, pad;
  unsigned long long collected;
  unsigned long long counts[kReportLayers], stamps[kReportLayers];
  unsigned long long previous[kCosetSmall], deepest[kCosetSmall];
};

struct CosetParams {
  const CosetInst* inst;
  const uint32_t* item_prefix;  // count + 1: exclusive prefix of the jobs' work items
  const uint8_t* perms;
  uint32_t count, units;        // jobs; units per item (a power of two)
  uint32_t chunk;               // 64-bit words: items of a block's chunk
  uint32_t stride, max_steps;   // layer-table columns; last step that may run
  unsigned long long* counts;   // count x stride layer sizes
  uint32_t* active;             // stride: layer d of any job is not empty
  uint32_t* next_item;          // stride: work items of step d taken so far, past the first of every warp
  unsigned long long* stamps;   // stride: globaltimer at the start of step d
  uint8_t* used;                // slot permutations that some row needs
  uint32_t* order;              // 64-bit words: every job's rows in the order they are visited
  uint32_t* order_sums;         // rows of each setup block's orbits
  uint32_t* table;              // slot permutation x node -> image and flips (table_entry)
  unsigned long long* desc;     // row x generator -> parent row | slot permutation << 32 | outer flips << 48
  unsigned long long* flags[2]; // per row: byte p = part p of the buffer's row is not zero
  void* buf[2];
  void* visited;                // jobs that are not inverse-closed
  uint32_t* small_count;        // stride: states kept by step d (wave of one job)
  unsigned long long* small;    // 2 x kCosetSmall state indices, by step parity
  CosetReport* report;          // wave of one job: written at the end, else null
  unsigned long long* front;    // with report: states of the deepest layer, as far as front_cap
  unsigned long long front_cap, start;  // start: the start's codes, 4 bits each
  uint32_t n;                   // with report: symbols of the job
  unsigned long long descs;     // total descriptors
  CosetCtl* ctl;
};

__host__ __device__ __forceinline__ void pair_of(uint32_t c, uint32_t* i, uint32_t* j) {
  uint32_t b = 1;
  while (b * (b + 1) / 2 <= c) ++b;
  *j = b;
  *i = c - b * (b - 1) / 2;
}

__host__ __device__ __forceinline__ uint32_t bits_below(uint32_t mask, uint32_t p) {
  const uint32_t x = mask & ((1u << p) - 1u);
#ifdef __CUDA_ARCH__
  return __popc(x);
#else
  return static_cast<uint32_t>(__builtin_popcount(x));
#endif
}

// The i-th position not in `used`.
__host__ __device__ __forceinline__ uint32_t nth_free(uint32_t used, uint32_t i) {
  uint32_t p = 0;
  for (;; ++p)
    if (!((used >> p) & 1u) && i-- == 0) return p;
}

// Positions of the outer labels 7 .. m-1 of a row, each pair's lower position
// first, and the mask of all of them.
__host__ __device__ __forceinline__ uint32_t row_positions(uint32_t m, uint32_t row, uint8_t* pos) {
  const uint32_t outer = m - kSlots, pairs = outer / 2;
  uint32_t digit[4];
  if (outer & 1) {
    digit[pairs] = row % 8;
    row /= 8;
  }
  for (uint32_t t = pairs; t-- > 0;) {
    const uint32_t c = m - 2 * t, radix = c * (c - 1) / 2;
    digit[t] = row % radix;
    row /= radix;
  }
  uint32_t used = 0;
  for (uint32_t t = 0; t < pairs; ++t) {
    uint32_t i, j;
    pair_of(digit[t], &i, &j);
    const uint32_t a = nth_free(used, i), b = nth_free(used, j);
    pos[2 * t] = static_cast<uint8_t>(a);
    pos[2 * t + 1] = static_cast<uint8_t>(b);
    used |= (1u << a) | (1u << b);
  }
  if (outer & 1) {
    const uint32_t a = nth_free(used, digit[pairs]);
    pos[outer - 1] = static_cast<uint8_t>(a);
    used |= 1u << a;
  }
  return used;
}

// The row whose outer labels sit at `pos` (pairs in either order); *flips
// gets bit t for every pair whose first label sits at the higher position.
__host__ __device__ __forceinline__ uint32_t row_rank(uint32_t m, const uint8_t* pos, uint32_t* flips,
                                                      uint32_t* mask) {
  const uint32_t outer = m - kSlots, pairs = outer / 2;
  uint32_t used = 0, row = 0, f = 0;
  for (uint32_t t = 0; t < pairs; ++t) {
    uint32_t a = pos[2 * t], b = pos[2 * t + 1];
    if (a > b) {
      f |= 1u << t;
      const uint32_t s = a;
      a = b;
      b = s;
    }
    const uint32_t i = a - bits_below(used, a), j = b - bits_below(used, b), c = m - 2 * t;
    row = row * (c * (c - 1) / 2) + j * (j - 1) / 2 + i;
    used |= (1u << a) | (1u << b);
  }
  if (outer & 1) {
    const uint32_t a = pos[outer - 1];
    row = row * 8 + a - bits_below(used, a);
    used |= 1u << a;
  }
  *flips = f;
  *mask = used;
  return row;
}

// Slots of a node's inner labels, four bits a label, each pair's lower slot
// first.
constexpr uint32_t packed_slots(uint32_t x) {
  const uint32_t digit[3] = {x / 30, x / 3 % 10, x % 3};
  uint32_t free_slots[kSlots] = {0, 1, 2, 3, 4, 5, 6}, left = kSlots, out = 0;
  for (uint32_t t = 0; t < 3; ++t) {
    uint32_t j = 1;
    while (j * (j + 1) / 2 <= digit[t]) ++j;
    const uint32_t i = digit[t] - j * (j - 1) / 2;
    out |= (free_slots[i] | (free_slots[j] << 4)) << (8 * t);
    uint32_t kept = 0;
    for (uint32_t k = 0; k < left; ++k)
      if (k != i && k != j) free_slots[kept++] = free_slots[k];
    left = kept;
  }
  return out | (free_slots[0] << 24);
}
struct NodeSlots {
  uint32_t at[kCosetNodes];
};
constexpr NodeSlots all_node_slots() {
  NodeSlots s{};
  for (uint32_t x = 0; x < kCosetNodes; ++x) s.at[x] = packed_slots(x);
  return s;
}
__device__ const NodeSlots kNodeSlots = all_node_slots();

// Decoding: the words (4 bits per position, the start's codes) of a row's
// states share the outer labels in canonical order; an outer or inner flip
// XORs one pair's two positions.
struct RowDecode {
  unsigned long long base, flip[3];
  uint32_t slots;  // position of each slot, four bits a slot
};

__device__ __forceinline__ unsigned long long code_of(unsigned long long start, uint32_t label) {
  return (start >> (4 * label)) & 15ull;
}

__device__ RowDecode decode_row(uint32_t m, uint32_t row, unsigned long long start) {
  uint8_t pos[7];
  const uint32_t used = row_positions(m, row, pos), outer = m - kSlots;
  RowDecode r{};
  for (uint32_t l = 0; l < outer; ++l) r.base |= code_of(start, kSlots + l) << (4 * pos[l]);
#pragma unroll
  for (uint32_t t = 0; t < 3; ++t)
    if (t < outer / 2) {
      const unsigned long long x = code_of(start, kSlots + 2 * t) ^ code_of(start, kSlots + 2 * t + 1);
      r.flip[t] = (x << (4 * pos[2 * t])) | (x << (4 * pos[2 * t + 1]));
    }
  uint32_t s = 0;
  for (uint32_t at = 0; at < m; ++at)
    if (!((used >> at) & 1u)) r.slots |= at << (4 * s++);
  return r;
}

// The state of bit `bit` of a node's word.
template <bool WIDE>
__device__ __forceinline__ unsigned long long decode_state(const RowDecode& r, uint32_t node, uint32_t bit,
                                                           unsigned long long start, unsigned long long keep) {
  const uint32_t slots = kNodeSlots.at[node];
  const uint32_t inner = WIDE ? bit >> 3 : bit >> 2, outer = WIDE ? bit & 7u : bit & 3u;
  unsigned long long w = r.base;
#pragma unroll
  for (uint32_t t = 0; t < 3; ++t) {
    const uint32_t a = (r.slots >> (4 * ((slots >> (8 * t)) & 15u))) & 15u;
    const uint32_t b = (r.slots >> (4 * ((slots >> (8 * t + 4)) & 15u))) & 15u;
    const bool flip = (inner >> t) & 1u;
    w |= code_of(start, 2 * t) << (4 * (flip ? b : a));
    w |= code_of(start, 2 * t + 1) << (4 * (flip ? a : b));
    if ((outer >> t) & 1u) w ^= r.flip[t];
  }
  w |= code_of(start, 6) << (4 * ((r.slots >> (4 * ((slots >> 24) & 15u))) & 15u));
  return w & keep;
}

// tau, four bits a slot, from its Lehmer code.
__device__ __forceinline__ uint32_t slot_permutation(uint32_t code) {
  uint32_t digits = 0, tau = 0, seen = 0;
#pragma unroll
  for (uint32_t a = kSlots; a-- > 0;) {
    digits |= (code % (kSlots - a)) << (4 * a);
    code /= kSlots - a;
  }
  for (uint32_t a = 0; a < kSlots; ++a) {
    const uint32_t to = nth_free(seen, (digits >> (4 * a)) & 15u);
    tau |= to << (4 * a);
    seen |= 1u << to;
  }
  return tau;
}

// Image of a node under a slot permutation, and the inner flips.
__device__ __forceinline__ uint32_t node_image(uint32_t tau, uint32_t x, uint32_t* flips) {
  const uint32_t slots = kNodeSlots.at[x];
  uint32_t used = 0, to = 0, f = 0;
#pragma unroll
  for (uint32_t t = 0; t < 3; ++t) {
    const uint32_t a = (tau >> (4 * ((slots >> (8 * t)) & 15u))) & 15u;
    const uint32_t b = (tau >> (4 * ((slots >> (8 * t + 4)) & 15u))) & 15u;
    const uint32_t lo = min(a, b), hi = max(a, b), c = 7 - 2 * t;
    const uint32_t i = lo - bits_below(used, lo), j = hi - bits_below(used, hi);
    f |= (a > b ? 1u : 0u) << t;
    to = to * (c * (c - 1) / 2) + j * (j - 1) / 2 + i;
    used |= (1u << a) | (1u << b);
  }
  *flips = f;
  return to;
}

// Parent row of a row under a generator (position images `perm`), the slot
// permutation's Lehmer code and the outer flips.
__device__ __forceinline__ uint32_t row_image(uint32_t m, uint32_t row, const uint8_t* perm, uint32_t* code,
                                              uint32_t* flips) {
  uint8_t pos[7], image[7];
  const uint32_t used = row_positions(m, row, pos);
  for (uint32_t l = 0; l < m - kSlots; ++l) image[l] = perm[pos[l]];
  uint32_t mask;
  const uint32_t parent = row_rank(m, image, flips, &mask);
  // Slot a of the row goes to slot tau[a] of the parent row.
  uint32_t c = 0, seen = 0, at = 0;
  for (uint32_t a = 0; a < kSlots; ++a, ++at) {
    while ((used >> at) & 1u) ++at;
    const uint32_t image_at = perm[at], tau = image_at - bits_below(mask, image_at);
    c = c * (kSlots - a) + tau - bits_below(seen, tau);
    seen |= 1u << tau;
  }
  *code = c;
  return parent;
}

// Descriptors of every (row, generator), the slot permutations they need, and
// the start states.  The parent of a state under g has the label of position p
// at position g[p].
template <typename W>
__global__ void __launch_bounds__(kCosetBlock) coset_setup(CosetParams p) {
  const unsigned long long step = static_cast<unsigned long long>(gridDim.x) * blockDim.x;
  const unsigned long long thread = blockIdx.x * static_cast<unsigned long long>(blockDim.x) + threadIdx.x;
  for (unsigned long long t = thread; t < p.descs; t += step) {
    uint32_t lo = 0, hi = p.count;
    while (hi - lo > 1) {
      const uint32_t mid = (lo + hi) / 2;
      if (p.inst[mid].desc_off <= t) lo = mid;
      else hi = mid;
    }
    const CosetInst in = p.inst[lo];
    const uint32_t local = static_cast<uint32_t>(t - in.desc_off), row = local / in.gens, g = local % in.gens;
    uint32_t code, flips;
    const uint32_t parent = row_image(in.m, row, p.perms + in.perm_off + 16 * g, &code, &flips);
    p.used[code] = 1;
    if (flips) p.used[0] = 1;  // read for rows that flip outer labels only
    p.desc[t] = parent | (static_cast<unsigned long long>(code) << 32) | (static_cast<unsigned long long>(flips) << 48);
  }
  for (unsigned long long i = thread; i < p.count; i += step) {
    const CosetInst in = p.inst[i];
    // The identity: label l at position l, hence node 0 and no flips.
    uint8_t pos[7];
    for (uint32_t l = 0; l < kSlots; ++l) pos[l] = static_cast<uint8_t>(kSlots + l);
    uint32_t f, mask;
    const unsigned long long row = in.row_off + row_rank(in.m, pos, &f, &mask), w = row * kCosetStride;
    static_cast<W*>(p.buf[0])[w] = 1;
    if (!in.inverse_closed) static_cast<W*>(p.visited)[w] = 1;
    p.flags[0][row] = 1;
    p.counts[i * p.stride] = 1;
  }
  if (thread == 0) p.active[0] = 1;
}

// The order in which a layer with 64-bit words visits its rows: orbit after
// orbit of the job's generator of the greatest order, by their least row, so
// that the rows it leads to and from are the neighbours in a chunk and are read
// from L2 once.  S13 LRX (the shift's 13 rows an orbit): DRAM traffic 131 -> 86
// GB, L2 sectors 7.3 -> 5.3 G, 28.3 -> 24.7 ms a call.  Without a generator
// of order 3 or more the rank's order stays: orbits of two rows gain nothing
// (adjacent transpositions: 25.9 ms either way).  Thread t of block b stands for row 1024 b +
// t; the least row of an orbit places all of it, behind the orbits of smaller rows.
constexpr uint32_t kOrderBlock = 1024;

// Length of the orbit if the row is its least, else 0.
__device__ __forceinline__ uint32_t orbit_of_least(const CosetParams& p, const CosetInst& in, uint32_t row) {
  if (in.walk == kNoWalk) return 1;
  uint32_t length = 0, at = row;
  do {
    at = static_cast<uint32_t>(p.desc[in.desc_off + static_cast<unsigned long long>(at) * in.gens + in.walk]);
    ++length;
    if (at < row) return 0;
  } while (at != row);
  return length;
}

__device__ __forceinline__ bool job_of_row(const CosetParams& p, unsigned long long all, CosetInst* in, uint32_t* row) {
  const unsigned long long r = blockIdx.x * static_cast<unsigned long long>(kOrderBlock) + threadIdx.x;
  if (r >= all) return false;
  uint32_t lo = 0, hi = p.count;
  while (hi - lo > 1) {
    const uint32_t mid = (lo + hi) / 2;
    if (p.inst[mid].row_off <= r) lo = mid;
    else hi = mid;
  }
  *in = p.inst[lo];
  *row = static_cast<uint32_t>(r - in->row_off);
  return true;
}

__global__ void __launch_bounds__(kOrderBlock) coset_orbits(CosetParams p, unsigned long long all) {
  __shared__ uint32_t sum;
  if (threadIdx.x == 0) sum = 0;
  __syncthreads();
  CosetInst in;
  uint32_t row;
  uint32_t mine = job_of_row(p, all, &in, &row) ? orbit_of_least(p, in, row) : 0u;
  mine = __reduce_add_sync(kFullMask, mine);
  if ((threadIdx.x & 31u) == 0 && mine) atomicAdd(&sum, mine);
  __syncthreads();
  if (threadIdx.x == 0) p.order_sums[blockIdx.x] = sum;
}

__global__ void __launch_bounds__(kOrderBlock) coset_order(CosetParams p, unsigned long long all) {
  __shared__ uint32_t before, sums[kOrderBlock / 32];
  const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
  if (threadIdx.x == 0) before = 0;
  __syncthreads();
  uint32_t earlier = 0;
  for (uint32_t b = threadIdx.x; b < blockIdx.x; b += kOrderBlock) earlier += p.order_sums[b];
  earlier = __reduce_add_sync(kFullMask, earlier);
  if (lane == 0 && earlier) atomicAdd(&before, earlier);
  CosetInst in;
  uint32_t row = 0;
  const uint32_t mine = job_of_row(p, all, &in, &row) ? orbit_of_least(p, in, row) : 0u;
  uint32_t upto = mine;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const uint32_t up = __shfl_up_sync(kFullMask, upto, o);
    if (lane >= static_cast<uint32_t>(o)) upto += up;
  }
  if (lane == 31) sums[warp] = upto;
  __syncthreads();
  uint32_t at = before + upto - mine;
  for (uint32_t w = 0; w < warp; ++w) at += sums[w];
  for (uint32_t k = 0, x = row; k < mine; ++k) {
    p.order[at + k] = x;
    if (k + 1 < mine)
      x = static_cast<uint32_t>(p.desc[in.desc_off + static_cast<unsigned long long>(x) * in.gens + in.walk]);
  }
}

// A table entry in the form the pull uses without unpacking: the byte permute
// selector of the inner flips in the low half (of the low word; the high
// word's is it ^ 0x4444), the node's image in the high half.  32-bit words keep
// the lowest flip as a nibble shift of 4 in bits 16..20 and XOR bytes by the
// other two; 64-bit words XOR bytes by all three.
template <typename W>
__device__ __forceinline__ uint32_t table_entry(uint32_t node, uint32_t flips) {
  if constexpr (sizeof(W) == 8) return (node << 21) | (0x3210u ^ (flips * 0x1111u));
  else return (node << 21) | ((flips & 1u) << 18) | (0x3210u ^ ((flips >> 1) * 0x1111u));
}

// The table rows of the slot permutations that some row needs: the image of
// every node and its inner flips.  One warp takes a permutation.
template <typename W>
__device__ void coset_table(const CosetParams& p, uint32_t per_block) {
  const uint32_t lane = threadIdx.x & 31u;
  const uint32_t warps = gridDim.x * per_block, warp = blockIdx.x * per_block + (threadIdx.x >> 5);
  for (uint32_t base = 0; base * warps + warp < kSlotPerms; base += 32) {
    const uint32_t mine = (base + lane) * warps + warp;
    uint32_t found = __ballot_sync(kFullMask, mine < kSlotPerms && __ldcg(p.used + mine));
    for (; found; found &= found - 1) {
      const uint32_t perm = (base + __ffs(static_cast<int>(found)) - 1) * warps + warp;
      const uint32_t tau = slot_permutation(perm);
      for (uint32_t x = lane; x < kCosetStride; x += 32) {
        uint32_t out = table_entry<W>(x, 0);  // words past the nodes stay zero and map to themselves
        if (x < kCosetNodes) {
          uint32_t flips;
          const uint32_t to = node_image(tau, x, &flips);
          out = table_entry<W>(to, flips);
        }
        p.table[perm * kCosetStride + x] = out;
      }
    }
  }
}

// Word with its bit index XORed: inner flips of a table entry (per lane),
// outer flips q (uniform).
__device__ __forceinline__ uint32_t flip_inner(uint32_t w, uint32_t entry) {
  w = __byte_perm(w, 0u, entry);
  const uint32_t by = entry >> 16;  // shifts use the low five bits: 0 or 4
  return (__funnelshift_l(0u, w, by) & 0xf0f0f0f0u) | (__funnelshift_r(w, 0u, by) & 0x0f0f0f0fu);
}
__device__ __forceinline__ unsigned long long flip_inner(unsigned long long w, uint32_t entry) {
  const uint32_t lo = static_cast<uint32_t>(w), hi = static_cast<uint32_t>(w >> 32);
  return (static_cast<unsigned long long>(__byte_perm(lo, hi, entry ^ 0x4444u)) << 32) | __byte_perm(lo, hi, entry);
}
__device__ __forceinline__ uint32_t swap_bits(uint32_t w, uint32_t mask, int by) {
  return ((w & mask) << by) | ((w >> by) & mask);
}
__device__ __forceinline__ uint32_t flip_outer(uint32_t w, uint32_t q) {
  if (q & 1u) w = swap_bits(w, 0x55555555u, 1);
  if (q & 2u) w = swap_bits(w, 0x33333333u, 2);
  return w;
}
__device__ __forceinline__ unsigned long long flip_outer(unsigned long long w, uint32_t q) {
  uint32_t lo = static_cast<uint32_t>(w), hi = static_cast<uint32_t>(w >> 32);
  if (q & 1u) lo = swap_bits(lo, 0x55555555u, 1), hi = swap_bits(hi, 0x55555555u, 1);
  if (q & 2u) lo = swap_bits(lo, 0x33333333u, 2), hi = swap_bits(hi, 0x33333333u, 2);
  if (q & 4u) lo = swap_bits(lo, 0x0f0f0f0fu, 4), hi = swap_bits(hi, 0x0f0f0f0fu, 4);
  return (static_cast<unsigned long long>(hi) << 32) | lo;
}
// Four words by one branch a flip (the flips are the same in all lanes).
template <typename W>
__device__ __forceinline__ void flip_words(W (&w)[4], uint32_t q) {
#pragma unroll
  for (uint32_t bit = 1; bit <= (sizeof(W) == 8 ? 4u : 2u); bit *= 2)
    if (q & bit) {
#pragma unroll
      for (int k = 0; k < 4; ++k) w[k] = flip_outer(w[k], bit);
    }
}
__device__ __forceinline__ uint32_t popcount(uint32_t w) { return __popc(w); }
__device__ __forceinline__ uint32_t popcount(unsigned long long w) { return __popcll(w); }

template <typename W>
__device__ __forceinline__ uint32_t lowest_bit(W b) {
  return (sizeof(W) == 8 ? __ffsll(static_cast<long long>(b)) : __ffs(static_cast<int>(b))) - 1;
}

// The end of a wave of one job whose step d found nothing: the states of layer
// d as packed words, in any order, and block 0 writes the report.
template <typename W>
__device__ void coset_finish(const CosetParams& p, const CosetInst& in, uint32_t d, bool exhausted) {
  const uint32_t lane = threadIdx.x & 31u, per_block = blockDim.x / 32;
  const uint32_t warps = gridDim.x * per_block, warp = blockIdx.x * per_block + (threadIdx.x >> 5);
  constexpr bool kWide = sizeof(W) == 8;
  CosetReport* r = p.report;
  const unsigned long long keep = (1ull << (4 * p.n)) - 1ull;  // embedded: positions from n up are not written
  // A layer that `front` does not hold is left to coset_collect.
  if (exhausted && __ldcg(p.counts + d) <= p.front_cap) {
    const W* buf = static_cast<const W*>(p.buf[d & 1u]);
    const unsigned long long* flags = p.flags[d & 1u];
    for (uint32_t row0 = warp * 32u; row0 < in.rows; row0 += warps * 32u) {
      const uint32_t row_l = row0 + lane;
      for (uint32_t m = __ballot_sync(kFullMask, row_l < in.rows && flags[row_l]); m; m &= m - 1) {
        const uint32_t row = row0 + __ffs(static_cast<int>(m)) - 1;
        const W* words = buf + static_cast<unsigned long long>(row) * kCosetStride;
        uint32_t mine = 0;
        for (uint32_t x = lane; x < kCosetStride; x += 32u) mine += popcount(words[x]);
        uint32_t upto = mine;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
          const uint32_t up = __shfl_up_sync(kFullMask, upto, o);
          if (lane >= static_cast<uint32_t>(o)) upto += up;
        }
        unsigned long long at = 0;
        if (lane == 31) at = atomicAdd(&p.ctl->collected, static_cast<unsigned long long>(upto));
        at = __shfl_sync(kFullMask, at, 31) + upto - mine;
        const RowDecode dec = decode_row(in.m, row, p.start);
        for (uint32_t x = lane; x < kCosetStride && mine; x += 32u)
          for (W b = words[x]; b; b &= b - 1, ++at) {
            const unsigned long long s = decode_state<kWide>(dec, x, lowest_bit(b), p.start, keep);
            if (at < p.front_cap) p.front[at] = s;
            if (at < kCosetSmall) r->deepest[at] = s;
          }
      }
    }
  }
  if (blockIdx.x) return;
  const uint32_t kept = exhausted ? min(p.small_count[d], kCosetSmall) : 0u;
  for (uint32_t k = threadIdx.x; k < kept; k += blockDim.x) {
    const unsigned long long at = p.small[(d & 1u) * kCosetSmall + k], w = at / 64;
    const RowDecode dec = decode_row(in.m, static_cast<uint32_t>(w / kCosetStride), p.start);
    r->previous[k] = decode_state<kWide>(dec, static_cast<uint32_t>(w % kCosetStride), static_cast<uint32_t>(at % 64),
                                         p.start, keep);
  }
  for (uint32_t k = threadIdx.x; k < kReportLayers && k <= d + 1; k += blockDim.x) {
    r->counts[k] = __ldcg(p.counts + k);
    r->stamps[k] = p.stamps[k];
  }
  if (threadIdx.x == 0) {
    r->previous_count = kept;
    r->steps = d + 1;
    r->error = p.ctl->error;
  }
}

// Threads of a block: with 64-bit words a whole multiprocessor's.
template <typename W>
constexpr uint32_t coset_threads() {
  return sizeof(W) == 8 ? 1024 : kCosetBlock;
}

// A whole search per launch: step d pulls layer d + 1 of every job, one grid
// barrier ends it.  A work item is up to `units` units of one job; its warp
// first looks, one lane per (unit, generator), which parent rows hold anything,
// and skips units with none (early and last layers touch few rows).
template <typename W>
__global__ void __launch_bounds__(coset_threads<W>(), 1024 / coset_threads<W>()) coset_wave_kernel(CosetParams p) {
  constexpr uint32_t kWarps = coset_threads<W>() / 32;
  __shared__ uint32_t tickets[2];
  const uint32_t lane = threadIdx.x & 31u;
  const uint32_t warps = gridDim.x * kWarps, warp = blockIdx.x * kWarps + (threadIdx.x >> 5);
  const uint32_t items = p.item_prefix[p.count];
  const uint32_t unit_mask = p.units - 1u;
  uint32_t epoch = 0;
  if (threadIdx.x == 0) tickets[0] = 0;
  coset_table<W>(p, kWarps);
  if (!arrival_barrier(&p.ctl->arrived, &p.ctl->error, &epoch)) return;
  CosetInst in = p.inst[0];
  for (uint32_t d = 0;; ++d) {
    if (blockIdx.x == 0 && threadIdx.x == 0) p.stamps[d] = global_ns();
    const W* cur = static_cast<const W*>(p.buf[d & 1u]);
    W* nxt = static_cast<W*>(p.buf[(d & 1u) ^ 1u]);
    const unsigned long long* cur_flags = p.flags[d & 1u];
    unsigned long long* nxt_flags = p.flags[(d & 1u) ^ 1u];
    const bool keep = p.report && d && __ldcg(p.counts + d - 1) < kCosetSmall;
    // The job of the current item; a wave of one job has nothing to look up.
    uint32_t i = 0, i_end = p.count == 1 ? items : 0u;
    bool live = p.count == 1;
    uint32_t found = 0;  // this lane's new states of job i
    auto flush = [&]() {
      const uint32_t sum = __reduce_add_sync(kFullMask, found);
      if (sum && lane == 0) {
        atomicAdd(p.counts + static_cast<unsigned long long>(i) * p.stride + d + 1, static_cast<unsigned long long>(sum));
        p.active[d + 1] = 1;
      }
      found = 0;
    };
    // Items are taken from a counter, the next one asked for before the current
    // one is worked on: parents differ too much in what they hold for a fixed
    // split (S12, six random generators: 30 % of the warps' time went into
    // waiting at the barrier), and warps that stay close together find each
    // other's rows in L2.  A layer with fewer states than items skips nearly all
    // of them, which the counter would only slow: those go round the warps.
    // 64-bit words: a block is all of a multiprocessor and its warps share a
    // chunk of neighbouring rows, whose parents largely coincide: what one warp
    // has read the others find in L1 (64 % of the sectors on S13 LRX).
    constexpr bool kChunks = sizeof(W) == 8;
    const bool counter = !kChunks && (p.count > 1 || __ldcg(p.counts + d) >= items);
    if (kChunks && threadIdx.x == 0) tickets[(d + 1) & 1u] = 0;
    const auto take = [&]() {
      uint32_t t = 0;
      if (lane == 0) t = atomicAdd(&tickets[d & 1u], 1u);
      t = __shfl_sync(kFullMask, t, 0);
      const uint32_t c = t / p.chunk;
      return (blockIdx.x + c * gridDim.x) * p.chunk + t - c * p.chunk;
    };
    uint32_t item = kChunks ? take() : warp;
    for (uint32_t coming; item < items; item = coming) {
      coming = item + warps;
      if (kChunks) {
        coming = take();
      } else if (counter) {
        if (lane == 0) coming = warps + atomicAdd(p.next_item + d, 1u);
        coming = __shfl_sync(kFullMask, coming, 0);
      }
      if (item >= i_end) {
        if (live) flush();
        uint32_t lo = 0, hi = p.count;
        while (hi - lo > 1) {
          const uint32_t mid = (lo + hi) / 2;
          if (__ldg(p.item_prefix + mid) <= item) lo = mid;
          else hi = mid;
        }
        i = lo;
        i_end = p.item_prefix[i + 1];
        in = p.inst[i];
        live = __ldcg(p.counts + static_cast<unsigned long long>(i) * p.stride + d) != 0;
      }
      if (!live) continue;
      const uint32_t unit0 = (item - p.item_prefix[i]) * p.units, all_units = in.rows * kCosetParts;
      // Parents that hold anything, of this lane's unit.
      const uint32_t my_unit = unit0 + (lane & unit_mask);
      uint32_t parents = 0, own_cur = 0, own_nxt = 0, place = 0;  // place: row << 3 | part
      if (my_unit < all_units) {
        uint32_t row = my_unit / kCosetParts;
        const uint32_t part = my_unit - row * kCosetParts, shift = 8 * part;
        if (kChunks && in.walk != kNoWalk) row = __ldg(p.order + in.row_off + row);
        place = (row << 3) | part;
        const unsigned long long* desc = p.desc + in.desc_off + static_cast<unsigned long long>(row) * in.gens;
        for (uint32_t g = lane / p.units; g < in.gens; g += 32u / p.units)
          if (cur_flags[in.row_off + static_cast<uint32_t>(__ldg(desc + g))]) parents |= 1u << g;
        own_cur = static_cast<uint32_t>(cur_flags[in.row_off + row] >> shift) & 255u;
        own_nxt = static_cast<uint32_t>(nxt_flags[in.row_off + row] >> shift) & 255u;
      }
      for (uint32_t o = p.units; o < 32u; o <<= 1) parents |= __shfl_xor_sync(kFullMask, parents, o);
      for (uint32_t u = 0; u < p.units; ++u) {
        const uint32_t mask = __shfl_sync(kFullMask, parents, u);
        const uint32_t in_cur = __shfl_sync(kFullMask, own_cur, u), in_nxt = __shfl_sync(kFullMask, own_nxt, u);
        if (!mask && !in_nxt) continue;  // nothing comes in and nothing is to be cleared
        const uint32_t here = __shfl_sync(kFullMask, place, u), row = here >> 3, part = here & 7u;
        const uint32_t x0 = part * 128u + lane;
        // Lane g holds generator g's descriptor.
        uint32_t from_row = 0, how = 0;  // parent row; slot permutation | outer flips << 16
        if (lane < in.gens) {
          const unsigned long long e =
              __ldg(p.desc + in.desc_off + static_cast<unsigned long long>(row) * in.gens + lane);
          from_row = static_cast<uint32_t>(e);
          how = static_cast<uint32_t>(e >> 32);
        }
        // Generators that keep the free positions' order and every outer pair's
        // read the parent row as it lies, the others through their table row, two
        // at a time: eight loads in flight and one three-way OR for both.  The
        // integer pipe, at half the issue rate, bounds a full layer, and a flip
        // that is only predicated off still takes its slots: with one loop for
        // all generators 25 instructions a word and generator and the pipe at
        // 84 % on S13, adjacent transpositions (52.0 ms, 24.4 ms in these loops).
        // With 64-bit words those without outer flips go by themselves (31.9 ms
        // otherwise) and an odd one out is done twice (26.3 ms with its own tail,
        // which spills); with 32-bit words the reverse (eight S12 instances: 11.0
        // ms; 12.4 ms the other way).
        const uint32_t plain = __ballot_sync(kFullMask, how == 0) & mask;
        W acc[4] = {0, 0, 0, 0};
        if constexpr (sizeof(W) == 8) {
          const uint32_t flipped = __ballot_sync(kFullMask, (how >> 16) != 0) & mask;
          for (uint32_t left = plain; left;) {
            const int g = __ffs(static_cast<int>(left)) - 1;
            left &= left - 1u;
            const W* from_g = cur + (in.row_off + __shfl_sync(kFullMask, from_row, g)) * kCosetStride + x0;
            const int h = left ? __ffs(static_cast<int>(left)) - 1 : g;
            left &= left - 1u;
            const W* from_h = cur + (in.row_off + __shfl_sync(kFullMask, from_row, h)) * kCosetStride + x0;
            W w_g[4], w_h[4];
#pragma unroll
            for (int k = 0; k < 4; ++k) w_g[k] = from_g[32 * k], w_h[k] = from_h[32 * k];
#pragma unroll
            for (int k = 0; k < 4; ++k) acc[k] |= w_g[k] | w_h[k];
          }
          for (uint32_t left = mask & ~plain & ~flipped; left;) {
            const int g = __ffs(static_cast<int>(left)) - 1;
            left &= left - 1u;
            const uint32_t how_g = __shfl_sync(kFullMask, how, g);
            const W* from_g = cur + (in.row_off + __shfl_sync(kFullMask, from_row, g)) * kCosetStride;
            const uint32_t* table_g = p.table + (how_g & 0xffffu) * kCosetStride + x0;
            uint32_t to_g[4];
            W w_g[4];
            const int h = left ? __ffs(static_cast<int>(left)) - 1 : g;
            left &= left - 1u;
            const uint32_t how_h = __shfl_sync(kFullMask, how, h);
            const W* from_h = cur + (in.row_off + __shfl_sync(kFullMask, from_row, h)) * kCosetStride;
            const uint32_t* table_h = p.table + (how_h & 0xffffu) * kCosetStride + x0;
            uint32_t to_h[4];
            W w_h[4];
#pragma unroll
            for (int k = 0; k < 4; ++k) to_g[k] = table_g[32 * k], to_h[k] = table_h[32 * k];
#pragma unroll
            for (int k = 0; k < 4; ++k) w_g[k] = from_g[to_g[k] >> 21], w_h[k] = from_h[to_h[k] >> 21];
#pragma unroll
            for (int k = 0; k < 4; ++k) w_g[k] = flip_inner(w_g[k], to_g[k]), w_h[k] = flip_inner(w_h[k], to_h[k]);
#pragma unroll
            for (int k = 0; k < 4; ++k) acc[k] |= w_g[k] | w_h[k];
          }
          // (The identity's table row for those that only flip.)
          for (uint32_t left = flipped; left;) {
            const int g = __ffs(static_cast<int>(left)) - 1;
            left &= left - 1u;
            const uint32_t how_g = __shfl_sync(kFullMask, how, g);
            const W* from_g = cur + (in.row_off + __shfl_sync(kFullMask, from_row, g)) * kCosetStride;
            const uint32_t* table_g = p.table + (how_g & 0xffffu) * kCosetStride + x0;
            uint32_t to_g[4];
            W w_g[4];
            const int h = left ? __ffs(static_cast<int>(left)) - 1 : g;
            left &= left - 1u;
            const uint32_t how_h = __shfl_sync(kFullMask, how, h);
            const W* from_h = cur + (in.row_off + __shfl_sync(kFullMask, from_row, h)) * kCosetStride;
            const uint32_t* table_h = p.table + (how_h & 0xffffu) * kCosetStride + x0;
            uint32_t to_h[4];
            W w_h[4];
#pragma unroll
            for (int k = 0; k < 4; ++k) to_g[k] = table_g[32 * k], to_h[k] = table_h[32 * k];
#pragma unroll
            for (int k = 0; k < 4; ++k) w_g[k] = from_g[to_g[k] >> 21], w_h[k] = from_h[to_h[k] >> 21];
#pragma unroll
            for (int k = 0; k < 4; ++k) w_g[k] = flip_inner(w_g[k], to_g[k]), w_h[k] = flip_inner(w_h[k], to_h[k]);
            flip_words(w_g, how_g >> 16);
            flip_words(w_h, how_h >> 16);
#pragma unroll
            for (int k = 0; k < 4; ++k) acc[k] |= w_g[k] | w_h[k];
          }
        } else {
          for (uint32_t left = plain; left;) {
            const int g = __ffs(static_cast<int>(left)) - 1;
            left &= left - 1u;
            const W* from_g = cur + (in.row_off + __shfl_sync(kFullMask, from_row, g)) * kCosetStride + x0;
            if (!left) {
#pragma unroll
              for (int k = 0; k < 4; ++k) acc[k] |= from_g[32 * k];
              break;
            }
            const int h = __ffs(static_cast<int>(left)) - 1;
            left &= left - 1u;
            const W* from_h = cur + (in.row_off + __shfl_sync(kFullMask, from_row, h)) * kCosetStride + x0;
            W w_g[4], w_h[4];
#pragma unroll
            for (int k = 0; k < 4; ++k) w_g[k] = from_g[32 * k], w_h[k] = from_h[32 * k];
#pragma unroll
            for (int k = 0; k < 4; ++k) acc[k] |= w_g[k] | w_h[k];
          }
          for (uint32_t left = mask & ~plain; left;) {
            const int g = __ffs(static_cast<int>(left)) - 1;
            left &= left - 1u;
            const uint32_t how_g = __shfl_sync(kFullMask, how, g);
            const W* from_g = cur + (in.row_off + __shfl_sync(kFullMask, from_row, g)) * kCosetStride;
            const uint32_t* table_g = p.table + (how_g & 0xffffu) * kCosetStride + x0;
            uint32_t to_g[4];
            W w_g[4];
            if (!left) {
#pragma unroll
              for (int k = 0; k < 4; ++k) to_g[k] = table_g[32 * k];
#pragma unroll
              for (int k = 0; k < 4; ++k) w_g[k] = from_g[to_g[k] >> 21];
#pragma unroll
              for (int k = 0; k < 4; ++k) w_g[k] = flip_inner(w_g[k], to_g[k]);
              flip_words(w_g, how_g >> 16);
#pragma unroll
              for (int k = 0; k < 4; ++k) acc[k] |= w_g[k];
              break;
            }
            const int h = __ffs(static_cast<int>(left)) - 1;
            left &= left - 1u;
            const uint32_t how_h = __shfl_sync(kFullMask, how, h);
            const W* from_h = cur + (in.row_off + __shfl_sync(kFullMask, from_row, h)) * kCosetStride;
            const uint32_t* table_h = p.table + (how_h & 0xffffu) * kCosetStride + x0;
            uint32_t to_h[4];
            W w_h[4];
#pragma unroll
            for (int k = 0; k < 4; ++k) to_g[k] = table_g[32 * k], to_h[k] = table_h[32 * k];
#pragma unroll
            for (int k = 0; k < 4; ++k) w_g[k] = from_g[to_g[k] >> 21], w_h[k] = from_h[to_h[k] >> 21];
#pragma unroll
            for (int k = 0; k < 4; ++k) w_g[k] = flip_inner(w_g[k], to_g[k]), w_h[k] = flip_inner(w_h[k], to_h[k]);
            flip_words(w_g, how_g >> 16);
            flip_words(w_h, how_h >> 16);
#pragma unroll
            for (int k = 0; k < 4; ++k) acc[k] |= w_g[k] | w_h[k];
          }
        }
        const unsigned long long own = (in.row_off + row) * kCosetStride + x0;
        W old[4] = {0, 0, 0, 0};
        if (in_nxt && (in.inverse_closed || keep)) {
#pragma unroll
          for (int k = 0; k < 4; ++k) old[k] = nxt[own + 32 * k];
        }
        if (in.inverse_closed) {
#pragma unroll
          for (int k = 0; k < 4; ++k) acc[k] &= ~old[k];
          if (in_cur && in.same_layer) {
#pragma unroll
            for (int k = 0; k < 4; ++k) acc[k] &= ~cur[own + 32 * k];
          }
        } else if (mask) {
          W* visited = static_cast<W*>(p.visited) + own;
#pragma unroll
          for (int k = 0; k < 4; ++k) {
            const W v = visited[32 * k];
            acc[k] &= ~v;
            if (acc[k]) visited[32 * k] = v | acc[k];
          }
        }
        if (keep && in_nxt) {
          // The small layer d - 1 is about to be overwritten.
#pragma unroll
          for (int k = 0; k < 4; ++k)
            for (W b = old[k]; b; b &= b - 1) {
              const uint32_t at = atomicAdd(p.small_count + d, 1u);
              if (at < kCosetSmall) p.small[(d & 1u) * kCosetSmall + at] = (own + 32 * k) * 64ull + lowest_bit(b);
            }
        }
        const bool any = __any_sync(kFullMask, (acc[0] | acc[1] | acc[2] | acc[3]) != 0);
        if (any || in_nxt) {
#pragma unroll
          for (int k = 0; k < 4; ++k) {
            nxt[own + 32 * k] = acc[k];
            found += popcount(acc[k]);
          }
          if (lane == 0 && any != (in_nxt != 0))
            reinterpret_cast<uint8_t*>(nxt_flags + in.row_off + row)[part] = any ? 1 : 0;
        }
      }
    }
    if (live) flush();
    if (!arrival_barrier(&p.ctl->arrived, &p.ctl->error, &epoch)) return;
    const bool more = __ldcg(p.active + d + 1) != 0;
    if (more && d < p.max_steps) continue;
    if (blockIdx.x == 0 && threadIdx.x == 0) {
      p.stamps[d + 1] = global_ns();
      p.ctl->steps = d + 1;
    }
    if (blockIdx.x == 0) __syncthreads();
    if (p.report) coset_finish<W>(p, in, d, !more);
    return;
  }
}

// The deepest layer again, into a buffer that holds it.
template <typename W>
__global__ void __launch_bounds__(kCosetBlock) coset_collect(CosetParams p, uint32_t last) {
  coset_finish<W>(p, p.inst[0], last, true);
}

// Small searches: every unit (128 nodes) has a warp of its own for the whole
// search, which keeps its words of layers d and d - 1 (and of the visited set)
// in registers and the address and flips of every parent word in shared memory.
// A layer is then one gather from L2 per generator, one store and one barrier;
// the general kernel's chain of dependent L2 reads (items, descriptors, flags,
// table, words) took 5.5 us a layer on S8 and 9 us on S10 with nothing to
// read.  No tables are made: the descriptors are computed where they are used.
struct SmallParams {
  uint32_t n, m, gens, units, inverse_closed, max_steps;
  uint8_t perms[kCosetMaxGens * 16];
  uint32_t* buf[2];
  unsigned long long* counts;
  unsigned long long* stamps;
  // Barrier and layer size in one: arrivals in the low half, states found so
  // far in the high half (a search of up to 10! states).
  unsigned long long* arrived;
  CosetCtl* ctl;
  uint32_t* small_count;
  unsigned long long* small;  // kCosetSmall entries (node word * 64 + bit) of the last small layer overwritten, by parity
  CosetReport* report;
  unsigned long long* front;
  unsigned long long front_cap, start;
};

// Parent word of a node: index in the buffer, outer flips in bits 24..25, the
// inner nibble shift (0 or 4) in bits 26..28, the byte flips in bits 30..31.
constexpr uint32_t kSmallIndexMask = (1u << 24) - 1u;

__device__ __forceinline__ uint32_t flip_small(uint32_t w, uint32_t e) {
  w = __byte_perm(w, 0u, 0x3210u ^ ((e >> 30) * 0x1111u));
  const uint32_t by = (e >> 26) & 7u;
  w = ((w << by) & 0xf0f0f0f0u) | ((w >> by) & 0x0f0f0f0fu);
  return flip_outer(w, (e >> 24) & 3u);
}

__device__ __forceinline__ void small_states(const SmallParams& p, uint32_t unit, uint32_t lane, const uint32_t (&w)[4]) {
  const unsigned long long keep = (1ull << (4 * p.n)) - 1ull;
  const uint32_t row = unit / kCosetParts, x0 = (unit - row * kCosetParts) * 128u + lane;
  if (!(w[0] | w[1] | w[2] | w[3])) return;
  const RowDecode dec = decode_row(p.m, row, p.start);
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    if (!w[k]) continue;
    unsigned long long at = atomicAdd(&p.ctl->collected, static_cast<unsigned long long>(__popc(w[k])));
    for (uint32_t b = w[k]; b; b &= b - 1, ++at) {
      const unsigned long long s = decode_state<false>(dec, x0 + 32 * k, lowest_bit(b), p.start, keep);
      if (at < p.front_cap) p.front[at] = s;
      if (at < kCosetSmall) p.report->deepest[at] = s;
    }
  }
}

__global__ void __launch_bounds__(kCosetBlock, 4) coset_small_kernel(SmallParams p) {
  extern __shared__ uint32_t parents[];  // warp x generator x 128 nodes
  __shared__ uint32_t sums[kCosetWarps];
  __shared__ unsigned long long seen;
  const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
  const uint32_t unit = blockIdx.x * kCosetWarps + warp;
  const bool mine = unit < p.units;
  const uint32_t row = unit / kCosetParts, x0 = (unit - row * kCosetParts) * 128u + lane;
  const size_t own = static_cast<size_t>(row) * kCosetStride + x0;
  uint32_t* from = parents + warp * p.gens * 128u + lane;
  uint32_t a[4] = {0, 0, 0, 0}, b[4] = {0, 0, 0, 0}, v[4] = {0, 0, 0, 0};  // layers d and d - 1, visited
  if (mine) {
    uint32_t parent = 0, tau = 0, q = 0;
    if (lane < p.gens) {
      uint32_t code;
      parent = row_image(p.m, row, p.perms + 16 * lane, &code, &q);
      tau = slot_permutation(code);
    }
    for (uint32_t g = 0; g < p.gens; ++g) {
      const uint32_t row_g = __shfl_sync(kFullMask, parent, g), tau_g = __shfl_sync(kFullMask, tau, g);
      const uint32_t q_g = __shfl_sync(kFullMask, q, g);
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        const uint32_t x = x0 + 32 * k;
        uint32_t flips = 0;
        const uint32_t to = x < kCosetNodes ? node_image(tau_g, x, &flips) : x;
        from[g * 128u + 32 * k] =
            (row_g * kCosetStride + to) | (q_g << 24) | ((flips & 1u) << 28) | ((flips >> 1) << 30);
      }
    }
    // The identity: outer label l at position l, node 0, no flips.
    uint8_t pos[7];
    for (uint32_t l = 0; l < kSlots; ++l) pos[l] = static_cast<uint8_t>(kSlots + l);
    uint32_t f, mask;
    if (row == row_rank(p.m, pos, &f, &mask) && x0 == 0) a[0] = v[0] = 1;
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      p.buf[0][own + 32 * k] = a[k];
      p.buf[1][own + 32 * k] = 0;
    }
  }
  uint32_t epoch = 0;
  // Ends the block's part of a layer that found `found` states in this thread;
  // returns the states found so far by all, or ~0 when the wait gave up.
  const auto arrive = [&](uint32_t found) {
    const uint32_t sum = __reduce_add_sync(kFullMask, found);
    if (lane == 0) sums[warp] = sum;
    __syncthreads();
    ++epoch;
    if (threadIdx.x == 0) {
      unsigned long long add = 0, now;
      for (uint32_t w = 0; w < kCosetWarps; ++w) add += sums[w];
      add = (add << 32) | 1ull;
      const uint32_t all = epoch * gridDim.x;
      __threadfence();
      asm volatile("atom.add.release.gpu.global.u64 %0, [%1], %2;" : "=l"(now) : "l"(p.arrived), "l"(add) : "memory");
      now += add;
      const unsigned long long started = global_ns();
      for (uint32_t polls = 0; static_cast<int32_t>(static_cast<uint32_t>(now) - all) < 0; ++polls) {
        if (polls >= kBarrierPolls || ((polls & 1023u) == 1023u && global_ns() - started > kBarrierWaitNs)) {
          raise_error(&p.ctl->error, ERR_WAIT_LIMIT);
          now = ~0ull;
          break;
        }
        asm volatile("ld.acquire.gpu.global.u64 %0, [%1];" : "=l"(now) : "l"(p.arrived) : "memory");
      }
      seen = now;
    }
    __syncthreads();
    const unsigned long long all_found = seen;
    return all_found == ~0ull ? all_found : all_found >> 32;
  };
  unsigned long long total = 0;
  if (arrive(0) == ~0ull) return;
  unsigned long long size = 1, before = ~0ull;  // layers d and d - 1
  for (uint32_t d = 0;; ++d) {
    if (blockIdx.x == 0 && threadIdx.x == 0) {
      p.stamps[d] = global_ns();
      p.counts[d] = size;
    }
    uint32_t found = 0;
    if (mine) {
      const uint32_t* cur = p.buf[d & 1u];
      uint32_t acc[4] = {0, 0, 0, 0};
      // Read past L1, which may hold words of two layers ago.
#pragma unroll 2
      for (uint32_t g = 0; g < p.gens; ++g) {
        uint32_t e[4], w[4];
#pragma unroll
        for (int k = 0; k < 4; ++k) e[k] = from[g * 128u + 32 * k];
#pragma unroll
        for (int k = 0; k < 4; ++k) w[k] = __ldcg(cur + (e[k] & kSmallIndexMask));
#pragma unroll
        for (int k = 0; k < 4; ++k) acc[k] |= flip_small(w[k], e[k]);
      }
      uint32_t* nxt = p.buf[(d & 1u) ^ 1u] + own;
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        acc[k] &= p.inverse_closed ? ~(a[k] | b[k]) : ~v[k];
        v[k] |= acc[k];
        found += __popc(acc[k]);
        if (acc[k] != b[k]) nxt[32 * k] = acc[k];
        if (before < kCosetSmall)
          for (uint32_t o = b[k]; o; o &= o - 1) {
            const uint32_t at = atomicAdd(p.small_count + d, 1u);
            if (at < kCosetSmall) p.small[(d & 1u) * kCosetSmall + at] = (own + 32 * k) * 64ull + lowest_bit(o);
          }
        b[k] = a[k];
        a[k] = acc[k];
      }
    }
    const unsigned long long now = arrive(found);
    if (now == ~0ull) return;
    before = size;
    size = now - total;
    total = now;
    if (size && d < p.max_steps) continue;
    // b holds layer d, the deepest when nothing was found.
    if (!size && mine && before <= p.front_cap) small_states(p, unit, lane, b);
    if (blockIdx.x) return;
    const uint32_t kept = size ? 0u : min(__ldcg(p.small_count + d), kCosetSmall);
    const unsigned long long keep = (1ull << (4 * p.n)) - 1ull;
    for (uint32_t k = threadIdx.x; k < kept; k += blockDim.x) {
      const unsigned long long at = __ldcg(p.small + (d & 1u) * kCosetSmall + k), w = at / 64;
      const RowDecode dec = decode_row(p.m, static_cast<uint32_t>(w / kCosetStride), p.start);
      p.report->previous[k] = decode_state<false>(dec, static_cast<uint32_t>(w % kCosetStride),
                                                  static_cast<uint32_t>(at % 64), p.start, keep);
    }
    if (threadIdx.x == 0) {
      p.counts[d + 1] = size;
      p.stamps[d + 1] = global_ns();
      p.ctl->steps = d + 1;
      p.report->previous_count = kept;
      p.report->steps = d + 1;
      p.report->error = p.ctl->error;
    }
    __syncthreads();
    for (uint32_t k = threadIdx.x; k < kReportLayers && k <= d + 1; k += blockDim.x) {
      p.report->counts[k] = p.counts[k];
      p.report->stamps[k] = p.stamps[k];
    }
    return;
  }
}

// The deepest layer of a small search again, into a buffer that holds it.
__global__ void __launch_bounds__(kCosetBlock) coset_small_collect(SmallParams p, uint32_t last) {
  const uint32_t lane = threadIdx.x & 31u, unit = blockIdx.x * kCosetWarps + (threadIdx.x >> 5);
  if (unit >= p.units) return;
  const uint32_t row = unit / kCosetParts, x0 = (unit - row * kCosetParts) * 128u + lane;
  const uint32_t* words = p.buf[last & 1u] + static_cast<size_t>(row) * kCosetStride + x0;
  const uint32_t w[4] = {words[0], words[32], words[64], words[96]};
  small_states(p, unit, lane, w);
}

size_t al256(size_t x) { return (x + 255) / 256 * 256; }

static_assert(kSlots == kCosetInner && kSlotPerms == kCosetInnerPerms && sizeof(CosetInst) <= kCosetInstBytes,
              "the sizes coset_bytes.h counts with");

}  // namespace

bool coset_supported(uint32_t n, uint32_t gens) {
  return n >= 2 && n <= kCosetMaxDegree && gens >= 1 && gens <= kCosetMaxGens;
}

// Layer tables (count x end.columns sizes) and step times.
static void read_layers(const std::vector<unsigned long long>& counts, const std::vector<unsigned long long>& stamps,
                        uint32_t count, const SearchEnd& end, uint32_t max_depth, CosetResult* out) {
  const uint32_t cols = end.fatal ? 1 : end.columns;
  out->layers = layer_tables(counts.data(), count, end);
  out->overflow.assign(count, 0);
  for (uint32_t i = 0; i < count; ++i) out->overflow[i] = out->layers[i].size() > max_depth;
  out->step_seconds.clear();
  for (uint32_t d = 0; d + 1 < cols; ++d) out->step_seconds.push_back(static_cast<double>(stamps[d + 1] - stamps[d]) * 1e-9);
  out->kernel_seconds = cols > 1 ? static_cast<double>(stamps[cols - 1] - stamps[0]) * 1e-9 : 0.0;
}

// One job through the small kernel: one clear, one launch, one synchronisation.
static int coset_small(const CosetJob& job, uint32_t max_depth, uint32_t units, size_t smem, cudaStream_t stream,
                       CosetMemory* memory, CosetResult* out, DeviceBuffer* collect, uint64_t start_word) {
  SmallParams p{};
  p.n = job.n;
  p.m = coset_symbols(job.n);
  p.gens = job.gens;
  p.units = units;
  p.inverse_closed = job.inverse_closed;
  p.max_steps = max_depth - 1;
  p.start = start_word;
  for (uint32_t g = 0; g < job.gens; ++g)
    for (uint32_t k = 0; k < 16; ++k)
      p.perms[16 * g + k] = static_cast<uint8_t>(k < job.n ? job.perms[static_cast<size_t>(g) * job.n + k] : k);
  const uint32_t stride = max_depth + 2;
  size_t off = 0;
  const auto take = [&off](size_t bytes) {
    const size_t at = off;
    off = al256(off + bytes);
    return at;
  };
  const size_t o_ctl = take(sizeof(CosetCtl)), o_arrived = take(8), o_small_count = take(4ull * stride);
  const size_t cleared = off;
  const size_t o_counts = take(8ull * stride), o_stamps = take(8ull * stride), o_small = take(16ull * kCosetSmall);
  const size_t words = static_cast<size_t>(units) * 128 * sizeof(uint32_t);
  const size_t o_buf0 = take(words), o_buf1 = take(words);
  int rc = memory->arena.ensure(off, true);
  if (!rc) rc = collect->ensure((kCosetSmall + 2) * 8);
  if (!rc && !memory->report) rc = pinned_take(sizeof(CosetReport), &memory->report);
  if (rc) return rc;
  char* base = static_cast<char*>(memory->arena.ptr);
  p.ctl = reinterpret_cast<CosetCtl*>(base + o_ctl);
  p.arrived = reinterpret_cast<unsigned long long*>(base + o_arrived);
  p.small_count = reinterpret_cast<uint32_t*>(base + o_small_count);
  p.counts = reinterpret_cast<unsigned long long*>(base + o_counts);
  p.stamps = reinterpret_cast<unsigned long long*>(base + o_stamps);
  p.small = reinterpret_cast<unsigned long long*>(base + o_small);
  p.buf[0] = reinterpret_cast<uint32_t*>(base + o_buf0);
  p.buf[1] = reinterpret_cast<uint32_t*>(base + o_buf1);
  p.report = static_cast<CosetReport*>(memory->report);
  p.report->steps = 0;
  p.front = static_cast<unsigned long long*>(collect->ptr);
  p.front_cap = collect->bytes / 8;
  const uint32_t blocks = (units + kCosetWarps - 1) / kCosetWarps;
  void* args[] = {&p};
  MG_CHECK_COSET(cudaMemsetAsync(base, 0, cleared, stream));
  MG_CHECK_COSET(cudaLaunchCooperativeKernel(reinterpret_cast<const void*>(coset_small_kernel), dim3(blocks),
                                             dim3(kCosetBlock), args, smem, stream));
  MG_CHECK_COSET(cudaStreamSynchronize(stream));
  out->launches = 1;
  out->steps = p.report->steps;
  const SearchEnd end = search_end(out->steps, p.report->error, stride, ERR_WAIT_LIMIT);
  out->fatal = end.fatal;
  const uint32_t cols = end.columns;
  std::vector<unsigned long long> counts(cols, 0), stamps(cols, 0);
  if (cols <= kReportLayers) {
    std::memcpy(counts.data(), p.report->counts, 8ull * cols);
    std::memcpy(stamps.data(), p.report->stamps, 8ull * cols);
  } else {
    MG_CHECK_COSET(cudaMemcpyAsync(counts.data(), p.counts, 8ull * cols, cudaMemcpyDeviceToHost, stream));
    MG_CHECK_COSET(cudaMemcpyAsync(stamps.data(), p.stamps, 8ull * cols, cudaMemcpyDeviceToHost, stream));
    MG_CHECK_COSET(cudaStreamSynchronize(stream));
  }
  read_layers(counts, stamps, 1, end, max_depth, out);
  if (out->fatal || out->overflow[0]) return MGBFS2_OK;
  out->previous_small.assign(p.report->previous, p.report->previous + p.report->previous_count);
  const uint64_t deepest = out->layers[0].back();
  if (deepest <= kCosetSmall) out->deepest_small.assign(p.report->deepest, p.report->deepest + deepest);
  if (deepest <= p.front_cap) return MGBFS2_OK;
  if ((rc = collect->ensure((deepest + 2) * 8))) return rc;
  p.front = static_cast<unsigned long long*>(collect->ptr);
  p.front_cap = deepest;
  MG_CHECK_COSET(cudaMemsetAsync(&p.ctl->collected, 0, sizeof(unsigned long long), stream));
  coset_small_collect<<<blocks, kCosetBlock, 0, stream>>>(p, out->steps - 1);
  ++out->launches;
  MG_CHECK_COSET(cudaGetLastError());
  MG_CHECK_COSET(cudaStreamSynchronize(stream));
  return MGBFS2_OK;
}

int coset_wave(const std::vector<CosetJob>& jobs, uint32_t max_depth, int sm_count, cudaStream_t stream,
               CosetMemory* memory, CosetResult* out, DeviceBuffer* collect, uint64_t start_word) {
  const uint32_t count = static_cast<uint32_t>(jobs.size());
  if (!count || !max_depth || (collect && count != 1)) return MGBFS2_INVALID_ARGUMENT;
  const bool wide = coset_wide(jobs[0].n);
  const size_t word = wide ? 8 : 4;
  const void* kernel = wide ? reinterpret_cast<const void*>(coset_wave_kernel<unsigned long long>)
                            : reinterpret_cast<const void*>(coset_wave_kernel<uint32_t>);
  const uint32_t threads = wide ? coset_threads<unsigned long long>() : coset_threads<uint32_t>();
  int per_sm = 0;
  MG_CHECK_COSET(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, static_cast<int>(threads), 0));
  if (per_sm < 1) return MGBFS2_UNSUPPORTED;
  // Units per item: eight, fewer while that leaves warps without an item.
  uint64_t units = 0;
  for (const CosetJob& j : jobs) {
    if (!coset_supported(j.n, j.gens) || coset_wide(j.n) != wide || !j.perms) return MGBFS2_INVALID_ARGUMENT;
    units += static_cast<uint64_t>(coset_rows(j.n)) * kCosetParts;
  }
  const uint64_t warps = static_cast<uint64_t>(per_sm) * sm_count * (threads / 32);
  uint32_t per_item = kMaxUnits;
  while (per_item > 1 && units / per_item < 6 * warps) per_item /= 2;
  if (wide) per_item = kWideUnits;
  if (collect && !wide) {
    // The small kernel where every unit gets a resident warp and 10! bounds the
    // states (its layer sizes share a word with the barrier).
    const size_t smem = static_cast<size_t>(kCosetWarps) * jobs[0].gens * 128 * sizeof(uint32_t);
    int resident = 0;
    if (jobs[0].n <= 10 && smem <= kSmallMaxShared &&
        cudaFuncSetAttribute(coset_small_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(kSmallMaxShared)) == cudaSuccess &&
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&resident, coset_small_kernel, kCosetBlock, smem) == cudaSuccess &&
        units <= static_cast<uint64_t>(resident) * sm_count * kCosetWarps)
      return coset_small(jobs[0], max_depth, static_cast<uint32_t>(units), smem, stream, memory, out, collect, start_word);
    cudaGetLastError();
  }
  std::vector<CosetInst> inst(count);
  std::vector<uint32_t> prefix(count + 1, 0);
  std::vector<uint8_t> perms;
  unsigned long long rows = 0, descs = 0;
  bool walks = false;
  for (uint32_t i = 0; i < count; ++i) {
    const CosetJob& j = jobs[i];
    CosetInst& c = inst[i];
    c.m = coset_symbols(j.n);
    c.gens = j.gens;
    c.rows = coset_rows(j.n);
    c.inverse_closed = j.inverse_closed;
    c.same_layer = 0;
    c.perm_off = static_cast<uint32_t>(perms.size());
    c.row_off = rows;
    c.desc_off = descs;
    for (uint32_t g = 0; g < j.gens; ++g) {
      const uint32_t* s = j.perms + static_cast<size_t>(g) * j.n;
      for (uint32_t k = 0; k < 16; ++k) perms.push_back(static_cast<uint8_t>(k < j.n ? s[k] : k));
      uint32_t swaps = 0, seen = 0;
      for (uint32_t k = 0; k < j.n; ++k)
        for (uint32_t at = k; !((seen >> at) & 1u); at = s[at]) {
          seen |= 1u << at;
          if (s[at] != k) ++swaps;
        }
      if (!(swaps & 1u)) c.same_layer = 1;
    }
    c.walk = kNoWalk;
    uint32_t greatest = 2;
    for (uint32_t g = 0; g < j.gens; ++g) {
      const uint32_t* s = j.perms + static_cast<size_t>(g) * j.n;
      uint32_t order = 1;
      for (uint32_t k = 0; k < j.n; ++k) {
        uint32_t length = 1;
        for (uint32_t at = s[k]; at != k; at = s[at]) ++length;
        order = std::lcm(order, length);
      }
      if (wide && order > greatest) greatest = order, c.walk = g;
    }
    walks |= c.walk != kNoWalk;
    rows += c.rows;
    descs += static_cast<unsigned long long>(c.rows) * c.gens;
    prefix[i + 1] = prefix[i] + (c.rows * kCosetParts + per_item - 1) / per_item;
  }
  // Arena: uploaded block | cleared block (tables of the loop, flags, buffers) | tables.
  const uint32_t stride = max_depth + 2;
  size_t off = 0;
  const auto take = [&off](size_t bytes) {
    const size_t at = off;
    off = al256(off + bytes);
    return at;
  };
  const size_t o_inst = take(count * sizeof(CosetInst)), o_prefix = take((count + 1) * 4), o_perms = take(perms.size());
  const size_t upload = off;
  const size_t o_counts = take(8ull * count * stride), o_active = take(4ull * stride), o_next = take(4ull * stride), o_small_count = take(4ull * stride);
  const size_t o_ctl = take(sizeof(CosetCtl)), o_used = take(kSlotPerms);
  const size_t o_flags0 = take(8 * rows), o_flags1 = take(8 * rows);
  const size_t word_bytes[3] = {rows * kCosetStride * word, rows * kCosetStride * word,
                                coset_visited_rows(jobs) * kCosetStride * word};
  const bool own = word_bytes[0] >= kCosetOwnWords;
  size_t o_words[3];
  for (int k = 0; k < 3; ++k) o_words[k] = take(own ? 0 : word_bytes[k]);
  const size_t cleared = off;
  const size_t o_stamps = take(8ull * stride), o_small = take(16ull * kCosetSmall), o_table = take(coset_table_bytes());
  const size_t o_desc = take(8 * descs);
  const uint64_t order_blocks = (rows + kOrderBlock - 1) / kOrderBlock;
  const size_t o_order = take(wide ? 4 * rows : 0), o_order_sums = take(wide ? 4 * order_blocks : 0);
  int rc = memory->arena.ensure(off, true);
  for (int k = 0; k < 3 && !rc && own; ++k)
    if (word_bytes[k]) rc = memory->words[k].ensure(word_bytes[k], true);
  // Room for a small deepest layer; a larger one is written by a second pass.
  if (!rc && collect) rc = collect->ensure((kCosetSmall + 2) * 8);
  if (!rc && collect && !memory->report) rc = pinned_take(sizeof(CosetReport), &memory->report);
  if (rc) return rc;
  char* base = static_cast<char*>(memory->arena.ptr);
  void* words[3];
  for (int k = 0; k < 3; ++k) words[k] = own ? memory->words[k].ptr : base + o_words[k];
  std::vector<char> host(upload);
  std::memcpy(host.data() + o_inst, inst.data(), count * sizeof(CosetInst));
  std::memcpy(host.data() + o_prefix, prefix.data(), (count + 1) * 4);
  std::memcpy(host.data() + o_perms, perms.data(), perms.size());
  CosetParams p{};
  p.inst = reinterpret_cast<const CosetInst*>(base + o_inst);
  p.item_prefix = reinterpret_cast<const uint32_t*>(base + o_prefix);
  p.perms = reinterpret_cast<const uint8_t*>(base + o_perms);
  p.count = count;
  p.units = per_item;
  p.chunk = kWideRows * kCosetParts / kWideUnits;
  p.stride = stride;
  p.max_steps = max_depth - 1;
  p.counts = reinterpret_cast<unsigned long long*>(base + o_counts);
  p.active = reinterpret_cast<uint32_t*>(base + o_active);
  p.next_item = reinterpret_cast<uint32_t*>(base + o_next);
  p.stamps = reinterpret_cast<unsigned long long*>(base + o_stamps);
  p.used = reinterpret_cast<uint8_t*>(base + o_used);
  p.table = reinterpret_cast<uint32_t*>(base + o_table);
  p.desc = reinterpret_cast<unsigned long long*>(base + o_desc);
  p.order = reinterpret_cast<uint32_t*>(base + o_order);
  p.order_sums = reinterpret_cast<uint32_t*>(base + o_order_sums);
  p.flags[0] = reinterpret_cast<unsigned long long*>(base + o_flags0);
  p.flags[1] = reinterpret_cast<unsigned long long*>(base + o_flags1);
  p.buf[0] = words[0];
  p.buf[1] = words[1];
  p.visited = words[2];
  p.small_count = reinterpret_cast<uint32_t*>(base + o_small_count);
  p.small = reinterpret_cast<unsigned long long*>(base + o_small);
  if (collect) {
    p.report = static_cast<CosetReport*>(memory->report);
    p.report->steps = 0;
    p.front = static_cast<unsigned long long*>(collect->ptr);
    p.front_cap = collect->bytes / 8;
    p.start = start_word;
    p.n = jobs[0].n;
  }
  p.descs = descs;
  p.ctl = reinterpret_cast<CosetCtl*>(base + o_ctl);
  cudaError_t e = cudaMemcpyAsync(base, host.data(), upload, cudaMemcpyHostToDevice, stream);
  if (e == cudaSuccess) e = cudaMemsetAsync(base + upload, 0, cleared - upload, stream);
  for (int k = 0; k < 3 && own && e == cudaSuccess; ++k)
    if (word_bytes[k]) e = cudaMemsetAsync(words[k], 0, word_bytes[k], stream);
  const uint32_t per_block = wide ? p.chunk : kCosetWarps;
  const uint64_t blocks = std::min<uint64_t>((prefix[count] + per_block - 1) / per_block,
                                             static_cast<uint64_t>(per_sm) * sm_count);
  if (e == cudaSuccess) {
    const uint32_t setup = static_cast<uint32_t>(
        std::min<unsigned long long>((descs + kCosetBlock - 1) / kCosetBlock, 8ull * static_cast<uint32_t>(sm_count)));
    if (wide) coset_setup<unsigned long long><<<setup, kCosetBlock, 0, stream>>>(p);
    else coset_setup<uint32_t><<<setup, kCosetBlock, 0, stream>>>(p);
    if (walks) {
      coset_orbits<<<static_cast<uint32_t>(order_blocks), kOrderBlock, 0, stream>>>(p, rows);
      coset_order<<<static_cast<uint32_t>(order_blocks), kOrderBlock, 0, stream>>>(p, rows);
    }
    e = cudaGetLastError();
  }
  if (e == cudaSuccess) {
    void* args[] = {&p};
    e = cudaLaunchCooperativeKernel(kernel, dim3(static_cast<uint32_t>(blocks)), dim3(threads), args, 0, stream);
  }
  CosetCtl ctl{};
  if (e == cudaSuccess && !collect) e = cudaMemcpyAsync(&ctl, p.ctl, sizeof(ctl), cudaMemcpyDeviceToHost, stream);
  if (e == cudaSuccess) e = cudaStreamSynchronize(stream);
  if (e != cudaSuccess) return cuda_status(e);
  if (p.report) {
    ctl.steps = p.report->steps;
    ctl.error = p.report->error;
  }
  const SearchEnd end = search_end(ctl.steps, ctl.error, stride, ERR_WAIT_LIMIT);
  out->launches = walks ? 4 : 2;
  out->steps = ctl.steps;
  out->fatal = end.fatal;
  // Columns 0 .. steps of the layer table, and the step times.
  const uint32_t cols = end.columns;
  std::vector<unsigned long long> stamps(cols), counts(static_cast<size_t>(count) * cols);
  if (p.report && cols <= kReportLayers) {
    std::memcpy(counts.data(), p.report->counts, 8ull * cols);
    std::memcpy(stamps.data(), p.report->stamps, 8ull * cols);
  } else {
    MG_CHECK_COSET(cudaMemcpy2DAsync(counts.data(), 8ull * cols, p.counts, 8ull * stride, 8ull * cols, count,
                                     cudaMemcpyDeviceToHost, stream));
    MG_CHECK_COSET(cudaMemcpyAsync(stamps.data(), p.stamps, 8ull * cols, cudaMemcpyDeviceToHost, stream));
    MG_CHECK_COSET(cudaStreamSynchronize(stream));
  }
  read_layers(counts, stamps, count, end, max_depth, out);
  if (!collect || out->fatal || out->overflow[0]) return MGBFS2_OK;
  const CosetReport& r = *p.report;
  out->previous_small.assign(r.previous, r.previous + r.previous_count);
  const uint64_t deepest = out->layers[0].back();
  if (deepest <= kCosetSmall) out->deepest_small.assign(r.deepest, r.deepest + deepest);
  if (deepest <= p.front_cap) return MGBFS2_OK;
  if ((rc = collect->ensure((deepest + 2) * 8))) return rc;
  p.front = static_cast<unsigned long long*>(collect->ptr);
  p.front_cap = deepest;
  const uint32_t last = ctl.steps - 1;
  MG_CHECK_COSET(cudaMemsetAsync(&p.ctl->collected, 0, sizeof(unsigned long long), stream));
  if (wide) coset_collect<unsigned long long><<<static_cast<uint32_t>(blocks), kCosetBlock, 0, stream>>>(p, last);
  else coset_collect<uint32_t><<<static_cast<uint32_t>(blocks), kCosetBlock, 0, stream>>>(p, last);
  ++out->launches;
  MG_CHECK_COSET(cudaGetLastError());
  MG_CHECK_COSET(cudaStreamSynchronize(stream));
  return MGBFS2_OK;
}

}  // namespace mgbfs2
