// Sizes of coset-word searches (see coset.h).  Host code without CUDA.
#pragma once
#include <algorithm>
#include <cstdint>
#include <vector>

namespace mgbfs2 {

constexpr uint32_t kCosetStride = 640;    // words of a row in memory: 5 parts of 128
constexpr uint32_t kCosetSmall = 1000;    // layers of fewer states are kept for samples
constexpr uint32_t kCosetInner = 7, kCosetInnerPerms = 5040;
constexpr uint32_t kCosetInstBytes = 64;  // at most, of a job's description on the device

// One search of a wave.
struct CosetJob {
  uint32_t n = 0, gens = 0;
  const uint32_t* perms = nullptr;  // gens x n, child[i] = state[g[i]]
  bool inverse_closed = false;
};

// 64-bit words: jobs of one wave must agree.
inline bool coset_wide(uint32_t n) { return n >= 13; }

// Symbols of the embedded search, and its rows.
inline uint32_t coset_symbols(uint32_t n) { return std::max(n, kCosetInner); }
inline uint32_t coset_rows(uint32_t n) {
  const uint32_t m = coset_symbols(n), outer = m - kCosetInner;
  uint32_t rows = outer & 1 ? 8 : 1;
  for (uint32_t t = 0; t < outer / 2; ++t) rows *= (m - 2 * t) * (m - 2 * t - 1) / 2;
  return rows;
}

inline uint64_t coset_row_bytes(uint32_t n) { return kCosetStride * (coset_wide(n) ? 8ull : 4ull); }

// Rows of the visited buffer of a wave: those up to its last directed job's
// (closed jobs before it hold their place).
inline uint64_t coset_visited_rows(const std::vector<CosetJob>& jobs) {
  uint64_t rows = 0, visited = 0;
  for (const CosetJob& j : jobs) {
    rows += coset_rows(j.n);
    if (!j.inverse_closed) visited = rows;
  }
  return visited;
}

inline size_t coset_table_bytes() { return static_cast<size_t>(kCosetInnerPerms) * kCosetStride * sizeof(uint32_t); }

// Device bytes of a wave: per row two layers' words, two flag words, the order
// and a descriptor a generator; the visited rows; tables.
inline uint64_t coset_wave_bytes(const std::vector<CosetJob>& jobs, uint32_t max_depth) {
  uint64_t bytes = coset_table_bytes() + kCosetInnerPerms + 16ull * kCosetSmall + 20ull * (max_depth + 2) + 32 * 256;
  for (const CosetJob& j : jobs)
    bytes += coset_rows(j.n) * (2 * coset_row_bytes(j.n) + 20 + 8ull * j.gens) + kCosetInstBytes + 4 + 16ull * j.gens +
             8ull * (max_depth + 2);
  return jobs.empty() ? bytes : bytes + coset_visited_rows(jobs) * coset_row_bytes(jobs[0].n);
}

}  // namespace mgbfs2
