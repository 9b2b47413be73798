// Grouped linears: many independent complete linears of ONE geometry (inputs, outputs)
// in one launch of wide_linear.cu, each with its own weights (any rate), its own gathered input
// rows and scattered output rows.  Building block of the routed-expert, SwiGLU and grouped-GEMV plans.
#pragma once
#include "backend.h"
#include "wide_linear.h"

namespace st {

constexpr int kGroupRows = 128;  // most rows of one problem: its weights are decoded once for all of them
constexpr int kDirectRows = 8;   // most rows of one problem of grouped_direct.cu
constexpr int kDirectStages = 16, kDirectSplits = 16;
constexpr double kWideStart = 10.0;  // us of a wide launch pair beyond its units, see direct_pays
constexpr size_t kDirectSmemLimit = 110 * 1024;  // two CTAs per SM

// One problem of a table in device memory.  Input row r is x + x_row[r]*x_stride, output row r is
// y + y_row[r]*y_stride (x_rows / y_rows point at the arrays of the record itself, see bind_rows).
struct GroupedProblem : WideProblem {
    int live;  // in the table's FIRST record: how many of its records a launch runs
    int x_row[kGroupRows];
    int y_row[kGroupRows];
};
// Points a host copy's row arrays at those of the device record it will be copied to.
inline void bind_rows(GroupedProblem& host, const GroupedProblem* device) {
    host.x_rows = device->x_row;
    host.y_rows = device->y_row;
}

struct GroupedPlan {
    int splits;            // typical number of CTAs that share one column block
    int scratch_splits;    // planes of partial sums per CTA
    int stages;            // weight ring slots
    int ctas_per_problem;  // CTAs of a launch of one problem
    bool direct;           // grouped_direct.cu: problems of up to kDirectRows rows; else wide_linear.cu
    int stage_stride;      // direct: bytes between ring slots
    size_t smem_bytes;     // direct
    WidePlan wide;
    size_t counter_bytes_per_problem;  // 0: nothing is counted per problem
    size_t partial_bytes_per_problem;  // core input tiles of one problem; direct: counters (zero at first) and planes
    size_t shared_bytes;               // flags and planes of a launch
    unsigned char* shared;             // the caller's memory for them
    SwigluRows swiglu;                 // not direct: input rows that the launch makes itself
};
// `rows` = most rows of one problem, `problems` = most problems of a launch; for up to kDirectRows rows
// the plan may be a direct one (direct_pays).
GroupedPlan plan_grouped(int inputs, int outputs, int max_bits, int rows, int sm_count, int problems);
// Which kernel a launch of `problems` weight sets, or `groups` groups of at most eight rows, is for.
// In us on a B200: an SM decodes a unit (128 columns x 128 of K) in 0.60 in grouped_direct.cu and in
// 0.53 in wide_linear.cu, which starts later (its input stages are a launch, its fold waits).
inline bool direct_pays(long long groups, long long problems, int inputs, int outputs, int launches, int sm_count) {
    const double units = (double)(inputs / 128) * (outputs / 128) / sm_count;
    return 0.60 * (double)groups * units + 4.0 * launches < 0.53 * (double)problems * units + kWideStart * launches;
}
// Makes `plan` a direct one for `groups` expected groups.  K partitions: of the counts up to `most`, the
// one with the least estimated time in units on one SM (two CTAs share an SM; a CTA costs about one
// unit beyond its own) plus the half-empty tail of the last CTAs.  At most 32 blocks of K per CTA: 64 KB
// of core input.
inline int direct_splits(int hblocks, int nblocks, long long groups, int sm_count, int most) {
    int splits = (hblocks + 31) / 32;
    double best = -1.0;
    for (int s = splits; s <= hblocks && s <= most; s *= 2) {
        const double ctas = (double)groups * nblocks * s, each = (double)((hblocks + s - 1) / s) + 1.0;
        const double cost = ctas * each / sm_count + 0.5 * each;
        if (best < 0.0 || cost < best) { best = cost; splits = s; }
    }
    return splits;
}
inline void plan_direct(GroupedPlan& plan, int inputs, int outputs, int max_bits, long long groups, int sm_count, int headroom) {
    const int hblocks = inputs / 128, nblocks = outputs / 128;
    // a plan that has its scratch (a window was set since) only takes another partition of it
    plan.splits = direct_splits(hblocks, nblocks, groups, sm_count, plan.direct ? plan.scratch_splits : kDirectSplits);
    const int per = (hblocks + plan.splits - 1) / plan.splits;
    plan.stage_stride = unit_bytes(max_bits);
    plan.stages = (32 * 1024) / plan.stage_stride;
    if (plan.stages > per) plan.stages = per;
    if (plan.stages > kDirectStages) plan.stages = kDirectStages;
    plan.ctas_per_problem = nblocks * plan.splits;
    plan.smem_bytes = 256 + (size_t)plan.stages * plan.stage_stride + (size_t)per * 256 * kDirectRows;
    if (plan.direct) return;
    plan.direct = true;
    int room = plan.splits * headroom < kDirectSplits ? plan.splits * headroom : kDirectSplits;
    if (room > hblocks) room = hblocks;
    plan.scratch_splits = room < plan.splits ? plan.splits : room;
    plan.partial_bytes_per_problem = align_up(align_up((size_t)nblocks * sizeof(unsigned int)) +
                                              (size_t)nblocks * plan.scratch_splits * kDirectRows * 128 * sizeof(float));
    plan.shared_bytes = 0;
}
// How many groups of at most eight rows a launch is expected to have, where the caller knows better
// than eight-row groups of `rows` in every problem (routes spread over a bank).
inline void expect_row_groups(GroupedPlan& plan, int inputs, int outputs, int max_bits, long long groups, int sm_count) {
    if (plan.direct) plan_direct(plan, inputs, outputs, max_bits, groups, sm_count, 1);
    else plan.wide.parts = accumulator_parts(inputs / 128, outputs / 128, groups, sm_count);
}
// `problems` lives in device memory; problems[0].live of its `problem_count` records are run.
cudaError_t launch_grouped(const GroupedProblem* problems, int problem_count, int inputs, int outputs,
                           int codebook, const GroupedPlan& plan, unsigned int* status, bool programmatic,
                           cudaStream_t stream);
cudaError_t launch_grouped_direct(const GroupedProblem* problems, int problem_count, int inputs, int outputs, int codebook,
                                  const GroupedPlan& plan, unsigned int* status, bool programmatic, cudaStream_t stream);

// hidden[r][c] = SwiGLU(gate[r][c], up[r][c]); gate/up contiguous [rows][width], hidden rows
// `out_stride` apart (src/tp_moe_activation.hpp:52-59).
cudaError_t launch_swiglu(const float* gate, const float* up, float* hidden, int rows, int width,
                          long long out_stride, bool programmatic, cudaStream_t stream);

// Device-side routing for a persistent expert bank: validates each token's route row and
// groups the valid routes by expert into problems of up to `window.group_rows` rows each, the first records of
// the tables, and sets their `live` counts.  The tables hold max_problems(...) (gate/up: twice that).
inline int max_problems(int routes, int bank, int group_rows) {
    const long long most = (long long)bank + routes / group_rows;  // one remainder per expert, full ones beyond
    return (int)(most < routes ? most : routes);
}
struct MoeBankEntry { DeviceWeights gate, up, down; };
// The bank is a window of the router's id space: id g is bank entry g - first_expert when that
// lies in [0, bank_count), belongs to another rank when g < experts_total (its slot runs nothing
// here and does not invalidate the row), and is invalid otherwise.  first_expert = 0 and
// experts_total = bank_count is the single-rank case.
struct MoeWindow { int first_expert, experts_total, group_rows; };
cudaError_t launch_moe_route(const unsigned int* route_ids, const float* route_scores, int tokens, int top_k,
                             const MoeBankEntry* bank, int bank_count, MoeWindow window, GroupedProblem* gate_up,
                             GroupedProblem* down, int* row_valid, bool programmatic, cudaStream_t stream);

// Routed-expert combine: y[t] = alpha * sum_{s ascending, from +0} RN32(score[t,s]*each[t,s]) + beta*y[t];
// a zero score skips its slot; a row flagged invalid becomes NaN (src/tp_moe.hip:112-164).
// With `route_ids` and a window, slots whose expert lives on another rank are skipped: the
// result is this rank's contribution (the reference's per-rank semantics, include/strix_trellis.h:215-216).
cudaError_t launch_moe_combine(const float* each, const float* scores, const int* row_valid, int tokens,
                               int top_k, int outputs, float* y, long long y_stride, float alpha, float beta,
                               bool programmatic, cudaStream_t stream, const unsigned int* route_ids = nullptr,
                               int first_expert = 0, int bank_count = 0);

}  // namespace st
