// What the host takes from the end of a persistent search.  The kernels write
// a report in pinned memory as they end; a search whose barrier gave up writes
// none, and the report then holds what the buffer's last user left (the
// buffers are recycled).  Host code without CUDA.
#pragma once
#include <algorithm>
#include <cstdint>
#include <vector>

#include "../../include/mgbfs2.h"

namespace mgbfs2 {

// Whether list layers run a search that a form without them returned `rc` for:
// its buffers did not fit (the plan looked at the memory, but takes none of
// theirs), or its grid cannot be resident as a whole.
constexpr int kCooperativeTooLarge = MGBFS2_CUDA_BASE + 720, kNotSupported = MGBFS2_CUDA_BASE + 801;
constexpr bool lists_instead(int rc) {
  return rc == MGBFS2_OUT_OF_MEMORY || rc == MGBFS2_UNSUPPORTED || rc == kCooperativeTooLarge || rc == kNotSupported;
}

struct SearchEnd {
  uint32_t fatal;    // device ERR_* bits
  uint32_t columns;  // columns of the layer table that the search wrote
};

// `steps` and `error` of the report, `steps` cleared before the launch;
// `no_report` is the error of a search that wrote none.
inline SearchEnd search_end(uint32_t steps, uint32_t error, uint32_t stride, uint32_t no_report) {
  return {steps ? error : no_report, std::min(steps + 1, stride)};
}

// Layer tables of `count` searches from rows of `columns` sizes, 0 past the
// deepest layer.  Of a search that failed only the start is known, whatever
// the rows hold.
inline std::vector<std::vector<uint64_t>> layer_tables(const unsigned long long* counts, uint32_t count,
                                                       const SearchEnd& end) {
  std::vector<std::vector<uint64_t>> tables(count);
  for (uint32_t i = 0; i < count; ++i) {
    const unsigned long long* row = counts + static_cast<size_t>(i) * end.columns;
    for (uint32_t d = 0; d < end.columns && row[d] && !end.fatal; ++d) tables[i].push_back(row[d]);
    if (tables[i].empty()) tables[i].push_back(1);
  }
  return tables;
}

}  // namespace mgbfs2
