// Linears of more than a few rows with the weights decoded on the fly (wide_linear.cu): one layer
// with up to some hundred rows, or many layers of one geometry (routed experts) in one launch.
#pragma once
#include "backend.h"

namespace st {

constexpr int kWideRows = 256;  // most rows of one problem: the MMA's N

// One problem: a complete linear over `rows` rows.  Row r of the input is x row x_rows[r] (r itself
// when null), row r of the output is y row y_rows[r].
struct WideProblem {
    DeviceWeights w;
    const void* x;
    void* y;
    const int* x_rows;
    const int* y_rows;
    long long x_stride, y_stride;
    unsigned char* tiles;  // core input, [I/128] tiles of wide_tile_bytes(rows)
    int rows;
    int x_dtype, y_dtype;
    float alpha, beta;
};

ST_RATE_FN int wide_n(int rows) { return rows <= 16 ? 16 : (rows + 15) & ~15; }  // MMA N
ST_RATE_FN size_t wide_tile_bytes(int rows) { return (size_t)wide_n(rows) * 256; }

struct WidePlan {
    int grid;
    int n_max;              // widest problem's N
    int w_slots, w_stride;  // weight ring: slots of one unit, bytes apart
    int b_slots, b_stride;  // activation ring
    size_t smem_bytes;
    size_t flag_bytes;      // [grid] counters, zeroed by launch_wide_inputs
    size_t plane_bytes;     // [grid][n_max][128] partial sums
};
// `heaviest`: the rate code with the largest tiles among the problems.
WidePlan plan_wide(int inputs, int heaviest, int rows_max, long long units, int sm_count);

// A set of problems of one geometry.  `table` (device memory) holds them, `table_stride` bytes apart;
// without a table the set is ONE layer whose `one.rows` rows are cut into problems of group_rows rows.
// `live` (device memory, may be null) overrides `count` at run time.
struct WideSet {
    const WideProblem* table;
    size_t table_stride;
    const int* live;
    WideProblem one;
    int count, group_rows;
    int inputs, outputs, codebook;
};
// Input stages of every row of every problem into its tiles; also zeroes the flags.
cudaError_t launch_wide_inputs(const WideSet& set, const WidePlan& plan, unsigned int* flags, bool programmatic,
                               cudaStream_t stream);
// The linears.  Must follow launch_wide_inputs (or another producer of tiles that zeroes the flags)
// in the stream.
cudaError_t launch_wide(const WideSet& set, const WidePlan& plan, unsigned int* flags, float* planes,
                        unsigned int* status, bool programmatic, cudaStream_t stream);

}  // namespace st
