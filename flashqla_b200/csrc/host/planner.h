// Segment planner of the context-parallel split (host only, no CUDA): see split_sequences.
#pragma once
#include <cstdint>
#include <optional>
#include <vector>

namespace fqla_host {

constexpr int CHUNK = 64;
constexpr int MIN_SEGMENT_CHUNKS = 8;
// K = V = 128, where most segments start a few chunks early and need no state from a pass of its own:
// shorter segments pay.  LEAD_SPLIT_CHUNKS: what a split costs in any case, the three launches that find
// out whether a state has to be handed over (9 us forward, 11 backward).  Batches whose longest sequence has
// less than LEAD_MIN_CHUNKS stay whole: there the launches cost a training step, which waits for the host,
// more than the shorter chains give.
constexpr int LEAD_MIN_SEGMENT_CHUNKS = 4, LEAD_SPLIT_CHUNKS = 4, LEAD_MIN_CHUNKS = 2 * MIN_SEGMENT_CHUNKS;
// costs, in chunk steps of the recurrence kernel
constexpr int SEGMENT_OVERHEAD_CHUNKS = 2;  // handing a start state to a segment
constexpr int CTA_START_CHUNKS = 2;         // starting a CTA (tensor-memory allocation, first loads)

struct Split {
  std::vector<int64_t> seg_bounds;  // cumulative lengths of the segments
  std::vector<int64_t> seg_begin;   // [n_raw + 1]: first segment of every raw sequence
};

// Length of the schedule the hardware produces for CTAs of the given costs (each present `copies`
// times, one per head) handed out longest first to `machines` SMs, one CTA per SM: every CTA goes
// to the SM that frees up first.  Returns a value above `give_up` as soon as the length is known
// to exceed it.
int64_t makespan(std::vector<int64_t> costs, int64_t copies, int64_t machines, int64_t give_up);

// `bounds`: raw cumulative sequence lengths.  Evaluates that schedule for the unsplit batch and
// for every maximum segment length ceil(longest / p) (longer sequences are cut into equal,
// chunk-aligned parts) and keeps the coarsest split within 3 % of the cheapest; nothing when no
// split gains 3 % after `split_cost`.
std::optional<Split> split_sequences(const std::vector<int64_t>& bounds, int64_t heads, int64_t n_sm,
                                     int64_t min_chunks = MIN_SEGMENT_CHUNKS, int64_t slices = 1,
                                     int64_t split_cost = 0);

}  // namespace fqla_host
