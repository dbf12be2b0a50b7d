// Whole searches without frontier lists: the handle's side of coset-word
// layers (coset.h), unipotent-ring layers (ring.h) and half-rank layers (half.h).
#include <algorithm>
#include <chrono>

#include "coset.h"
#include "engine.h"
#include "half.h"
#include "ring.h"
#include "search_end.h"

namespace mgbfs2 {

static_assert(kCooperativeTooLarge == MGBFS2_CUDA_BASE + cudaErrorCooperativeLaunchTooLarge &&
                  kNotSupported == MGBFS2_CUDA_BASE + cudaErrorNotSupported,
              "the codes that cuda_status makes of a cooperative launch's errors");

#define MG_CHECK(expr)                         \
  do {                                         \
    cudaError_t _e = (expr);                   \
    if (_e != cudaSuccess) return cuda_status(_e); \
  } while (0)

namespace {
using Clock = std::chrono::steady_clock;

// List layers until a layer has this share of the ring nodes (below, a
// layer's pass over every determinant's nodes, 0.3 ms at p = 257, costs more
// than its edges; small orbits, p = 127: 129 layers in 1.6 ms), unless there are so few nodes
// that the pass costs no more than a launch (p = 67: 10 us a layer).
constexpr uint64_t kRingShare = 64, kRingFewNodes = 1ull << 20;

// The handle of a packed search that knows its start alone: one that is about
// to begin, or one that failed.
int start_only(Graph* g) {
  g->layer_sizes.assign(1, 1);
  g->layer_seconds.clear();
  g->front_grouped = false;
  for (int i = 0; i < 2; ++i) {
    g->small_layer[i].clear();
    g->small_depth[i] = UINT32_MAX;
  }
  g->keep_small(0, std::vector<uint64_t>(1, g->start_word));
  g->last_count = 1;
  if (int rc = g->front.ensure(16)) return rc;
  MG_CHECK(cudaMemcpyAsync(g->front.ptr, &g->start_word, 8, cudaMemcpyHostToDevice, g->stream));
  return MGBFS2_OK;
}
}  // namespace

// A whole search in coset-word layers, from the identity: the layer sizes do
// not depend on the start, and its states are those of the identity's search
// with the codes mapped through the start.
int Graph::coset_run(mgbfs2_status* status) {
  mgbfs2_status st{};
  const auto started = Clock::now();
  MG_CHECK(cudaEventRecord(ev_run[0], stream));
  CosetResult r;
  if (!coset) {
    coset = new CosetMemory();
    coset->set_stream(stream);
  }
  {
    TraceRange range("layers.coset");
    const int rc = coset_wave({CosetJob{elements, gens, perms.data(), inverse_closed}}, kWholeDepth, sm_count, stream,
                              coset, &r, &front, start_word);
    if (rc) return rc;
  }
  if (r.overflow[0]) {  // deeper than its layer table: the list layers have no such limit
    return run_lists(nullptr, nullptr, nullptr, status);
  }
  no_bitmap = true;
  front_grouped = false;
  layer_sizes = r.layers[0];
  const uint32_t deepest = static_cast<uint32_t>(layer_sizes.size() - 1);
  layer_seconds.assign(r.step_seconds.begin(), r.step_seconds.begin() + std::min<size_t>(deepest, r.step_seconds.size()));
  for (int i = 0; i < 2; ++i) {
    small_layer[i].clear();
    small_depth[i] = UINT32_MAX;
  }
  if (r.fatal) {
    if (int rc = start_only(this)) return rc;
  } else {
    if (deepest && layer_sizes[deepest - 1] < kCosetSmall) keep_small(deepest - 1, std::move(r.previous_small));
    if (layer_sizes[deepest] < kCosetSmall) keep_small(deepest, std::move(r.deepest_small));
    last_count = layer_sizes[deepest];
  }
  launches = r.launches;
  st.complete = r.fatal == 0;
  st.reason = r.fatal ? MGBFS2_REASON_RESOURCE : MGBFS2_REASON_FRONTIER_EXHAUSTED;
  st.fatal = r.fatal;
  st.layers = deepest + 1;
  for (uint32_t d = 0; d <= deepest; ++d) {
    const uint64_t c = layer_sizes[d];
    st.states += c;
    st.successors += c * gens;
    st.visited_tests += c * gens - (parent_skip && d > 0 ? c : 0);
  }
  if (cudaEventRecord(ev_run[1], stream) == cudaSuccess && cudaEventSynchronize(ev_run[1]) == cudaSuccess) {
    float ms = 0.f;
    if (cudaEventElapsedTime(&ms, ev_run[0], ev_run[1]) == cudaSuccess) st.device_seconds = ms * 1e-3;
  }
  st.kernel_seconds = r.kernel_seconds;
  st.bfs_seconds = std::chrono::duration<double>(Clock::now() - started).count();
  st.kernel_launches = launches;
  st.peak_device_bytes = std::max<uint64_t>(plan.device_bytes, coset->bytes() + front.bytes);
  if (status) *status = st;
  return MGBFS2_OK;
}

// A search of 2x2 matrices over a prime field: list layers while they are
// small, then unipotent-ring layers to the end.
int Graph::ring_run(mgbfs2_status* status) {
  mgbfs2_status st{};
  const auto started = Clock::now();
  const uint32_t m = moduli[0];
  if (ring_nodes(m) > kRingFewNodes) {
    list_stop = ring_nodes(m) / kRingShare;
    const int rc = run_lists(nullptr, nullptr, nullptr, &st);
    list_stop = 0;
    if (rc || st.reason != MGBFS2_REASON_LAYER_LIMIT) {
      if (status) *status = st;
      return rc;
    }
  } else {
    launches = 0;
    st.states = st.layers = 1;
    if (int rc = start_only(this)) return rc;
  }
  if (!ring) {
    ring = new RingMemory();
    ring->set_stream(stream);
  }
  std::vector<uint32_t> coef;
  for (int64_t v : matrices) {
    v %= static_cast<int64_t>(m);
    coef.push_back(static_cast<uint32_t>(v < 0 ? v + m : v));
  }
  const uint32_t from = static_cast<uint32_t>(layer_sizes.size() - 1);
  MG_CHECK(cudaEventRecord(ev_run[0], stream));
  RingResult r;
  {
    TraceRange range("layers.ring");
    const int rc = ring_wave(m, bits, gens, coef.data(), front.ptr, layer_sizes[from], next.ptr,
                             from ? layer_sizes[from - 1] : 0, key_mask, kWholeDepth, sm_count, stream, ring, &front, &r);
    if (rc) return rc;
  }
  if (r.overflow) return run_lists(nullptr, nullptr, nullptr, status);
  no_bitmap = true;
  layer_sizes.insert(layer_sizes.end(), r.layers.begin(), r.layers.end());
  layer_seconds.insert(layer_seconds.end(), r.seconds.begin(), r.seconds.end());
  const uint32_t deepest = static_cast<uint32_t>(layer_sizes.size() - 1);
  if (deepest > from) {
    if (layer_sizes[deepest - 1] < kRingSmall) keep_small(deepest - 1, std::move(r.previous_small));
    if (layer_sizes[deepest] < kRingSmall) keep_small(deepest, std::move(r.deepest_small));
    last_count = layer_sizes[deepest];
  }
  launches += r.launches;
  st.complete = r.fatal == 0;
  st.reason = r.fatal ? MGBFS2_REASON_RESOURCE : MGBFS2_REASON_FRONTIER_EXHAUSTED;
  st.fatal = r.fatal;
  st.layers = deepest + 1;
  for (uint32_t d = from; d <= deepest; ++d) {
    const uint64_t c = layer_sizes[d];
    if (d > from) st.states += c;
    st.successors += c * gens;
    st.visited_tests += c * gens - (parent_skip && d > 0 ? c : 0);
  }
  if (cudaEventRecord(ev_run[1], stream) == cudaSuccess && cudaEventSynchronize(ev_run[1]) == cudaSuccess) {
    float ms = 0.f;
    if (cudaEventElapsedTime(&ms, ev_run[0], ev_run[1]) == cudaSuccess) st.device_seconds += ms * 1e-3;
  }
  st.kernel_seconds += r.kernel_seconds;
  st.bfs_seconds = std::chrono::duration<double>(Clock::now() - started).count();
  st.kernel_launches = launches;
  st.peak_device_bytes = std::max<uint64_t>(st.peak_device_bytes, bitmap.bytes + front.bytes + next.bytes + ring->bytes());
  if (status) *status = st;
  return MGBFS2_OK;
}

// A search over repeated labels in half-rank layers, packed or wide.
int Graph::half_run(mgbfs2_status* status) {
  mgbfs2_status st{};
  const auto started = Clock::now();
  if (!half) {
    half = new HalfMemory();
    half->set_stream(stream);
  }
  const uint64_t reach = state_bound ? std::min(state_bound, rank_total) : rank_total;
  const HalfJob job{elements, distinct, gens, codes.data(), code_counts.data(), perms.data(), inverse_closed, rank_total, reach};
  MG_CHECK(cudaEventRecord(ev_run[0], stream));
  HalfResult r;
  {
    TraceRange range("layers.half");
    const int rc = half_wave(job, kWholeDepth, sm_count, stream, half, &bitmap, packed ? &front : nullptr, bits, &r);
    if (rc) return rc;
  }
  if (r.overflow) return packed ? run_lists(nullptr, nullptr, nullptr, status) : wide_run(nullptr, nullptr, nullptr, status);
  no_bitmap = false;  // the bitmap over the rank domain is the one list layers make
  front_grouped = false;
  layer_sizes = r.layers;
  layer_seconds = r.seconds;
  const uint32_t deepest = static_cast<uint32_t>(layer_sizes.size() - 1);
  for (int i = 0; i < 2; ++i) {
    small_layer[i].clear();
    small_depth[i] = UINT32_MAX;
    half_rows[i].clear();
  }
  const auto symbol = [&](uint64_t w, uint32_t i) { return (w >> (r.bits * i)) & ((1ull << r.bits) - 1ull); };
  if (packed && r.fatal) {
    if (int rc = start_only(this)) return rc;
  } else if (packed) {
    const auto words = [&](const std::vector<uint64_t>& states) {
      std::vector<uint64_t> out;
      for (uint64_t w : states) {
        uint64_t v = 0;
        for (uint32_t i = 0; i < elements; ++i) v |= symbol(w, i) << (bits * i);
        out.push_back(v);
      }
      return out;
    };
    if (deepest && layer_sizes[deepest - 1] < kHalfSmall) keep_small(deepest - 1, words(r.previous));
    if (layer_sizes[deepest] < kHalfSmall) keep_small(deepest, words(r.deepest));
    last_count = layer_sizes[deepest];
  } else {
    half_done = true;
    last_count = layer_sizes[deepest];
    const auto rows = [&](const std::vector<uint64_t>& states, std::vector<std::vector<int64_t>>* out) {
      for (uint64_t w : states) {
        std::vector<int64_t> row(elements);
        for (uint32_t i = 0; i < elements; ++i) row[i] = labels[symbol(w, i)];
        out->push_back(std::move(row));
      }
    };
    rows(r.deepest, &half_rows[0]);
    rows(r.previous, &half_rows[1]);
    if (r.fatal) half_rows[0].assign(1, start);
  }
  launches = r.launches;
  st.complete = r.fatal == 0;
  st.reason = r.fatal ? MGBFS2_REASON_RESOURCE : MGBFS2_REASON_FRONTIER_EXHAUSTED;
  st.fatal = r.fatal;
  st.layers = deepest + 1;
  for (uint32_t d = 0; d <= deepest; ++d) {
    const uint64_t c = layer_sizes[d];
    st.states += c;
    st.successors += c * gens;
    if (packed) st.visited_tests += c * gens - (parent_skip && d > 0 ? c : 0);
  }
  if (cudaEventRecord(ev_run[1], stream) == cudaSuccess && cudaEventSynchronize(ev_run[1]) == cudaSuccess) {
    float ms = 0.f;
    if (cudaEventElapsedTime(&ms, ev_run[0], ev_run[1]) == cudaSuccess) st.device_seconds = ms * 1e-3;
  }
  st.kernel_seconds = r.kernel_seconds;
  st.bfs_seconds = std::chrono::duration<double>(Clock::now() - started).count();
  st.kernel_launches = launches;
  st.peak_device_bytes = std::max<uint64_t>(plan.device_bytes, bitmap.bytes + front.bytes + half->bytes());
  if (status) *status = st;
  return MGBFS2_OK;
}

}  // namespace mgbfs2

extern "C" int mgbfs2_search_form(const mgbfs2_graph* graph, uint32_t* form) {
  if (!graph || !form) return MGBFS2_INVALID_ARGUMENT;
  const mgbfs2::Graph& g = *graph->impl;
  if (!g.planned) return MGBFS2_STATE;
  *form = g.half_ok ? MGBFS2_FORM_HALF : g.coset_ok ? MGBFS2_FORM_COSET : g.ring_ok ? MGBFS2_FORM_RING : MGBFS2_FORM_LISTS;
  return MGBFS2_OK;
}
