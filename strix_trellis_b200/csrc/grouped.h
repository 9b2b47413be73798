// Grouped linears: many independent complete linears of ONE geometry (inputs, outputs)
// in one launch of wide_linear.cu, each with its own weights (any rate), its own gathered input
// rows and scattered output rows.  Building block of the routed-expert, SwiGLU and grouped-GEMV plans.
#pragma once
#include "backend.h"
#include "wide_linear.h"

namespace st {

constexpr int kGroupRows = 128;  // most rows of one problem: its weights are decoded once for all of them

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
    WidePlan wide;
    size_t counter_bytes_per_problem;  // 0: nothing is counted per problem
    size_t partial_bytes_per_problem;  // core input tiles of one problem
    size_t shared_bytes;               // flags and planes of a launch
    unsigned char* shared;             // the caller's memory for them
};
// `rows` = most rows of one problem, `problems` = most problems of a launch.
GroupedPlan plan_grouped(int inputs, int outputs, int max_bits, int rows, int sm_count, int problems);
// `problems` lives in device memory; problems[0].live of its `problem_count` records are run.
cudaError_t launch_grouped(const GroupedProblem* problems, int problem_count, int inputs, int outputs,
                           int codebook, const GroupedPlan& plan, unsigned int* status, bool programmatic,
                           cudaStream_t stream);

// hidden[r][c] = SwiGLU(gate[r][c], up[r][c]); gate/up contiguous [rows][width], hidden rows
// `out_stride` apart (src/tp_moe_activation.hpp:52-59).
cudaError_t launch_swiglu(const float* gate, const float* up, float* hidden, int rows, int width,
                          long long out_stride, bool programmatic, cudaStream_t stream);

// Device-side routing for a persistent expert bank: validates each token's route row and
// groups the valid routes by expert into problems of up to kGroupRows rows each, the first records of
// the tables, and sets their `live` counts.  The tables hold max_problems(...) (gate/up: twice that).
inline int max_problems(int routes, int bank) {
    const long long most = (long long)bank + routes / kGroupRows;  // one remainder per expert, full ones beyond
    return (int)(most < routes ? most : routes);
}
struct MoeBankEntry { DeviceWeights gate, up, down; };
// The bank is a window of the router's id space: id g is bank entry g - first_expert when that
// lies in [0, bank_count), belongs to another rank when g < experts_total (its slot runs nothing
// here and does not invalidate the row), and is invalid otherwise.  first_expert = 0 and
// experts_total = bank_count is the single-rank case.
struct MoeWindow { int first_expert, experts_total; };
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
