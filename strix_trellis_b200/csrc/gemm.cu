// Routes of a GEMM (more than 8 rows) and their workspace.
//   up to kWideMaxRows   weights decoded on the fly into tensor memory (wide_linear.cu), once for each
//                        row group
//   more rows            weights decoded once into the workspace, dense GEMM (gemm_dense.cu)
#include "wide_linear.h"

#include <cmath>

namespace st {

int gemm_dense_rows_padded(int rows);
size_t gemm_dense_scratch(const DeviceWeights& w);
cudaError_t launch_gemm_dense(const LinearCall& call, unsigned char* workspace, int sm_count, bool programmatic,
                              cudaStream_t stream);

namespace {
// Measured at the crossing (4096 -> 12288, K5): 512 rows take 87 us on the fly (two decodes) and 82 us
// dense; 256 rows take one decode.
constexpr int kWideMaxRows = kWideRows;
// How a call's rows are cut into groups that each decode the weights, and how many CTAs run them: one
// group and every SM, unless so few column blocks are left that many CTAs share one and the CTA that
// finishes it adds all their planes (178 rows on 3072 -> 2048, nine CTAs a block: 51 us in one group,
// 22 us in three).  In us: a decoded unit 0.53 on its SM; a plane's chunk of 16 rows 1.0 and its
// output stages 1.5, five warp groups side by side.  With s CTAs a block that is
// 0.53 * hblocks / s + rounds * (s + 1.5), least at s = sqrt(0.53 * hblocks / rounds).
struct Cut { int groups, rows, ctas; };
Cut cut_call(const DeviceWeights& w, int rows, int sm_count) {
    const int hblocks = w.inputs / 128, nblocks = w.outputs / 128;
    Cut best{};
    double least = 0.0;
    for (int count = (rows + kWideRows - 1) / kWideRows; count <= 1 || rows / count >= 32; ++count) {
        const int each = ((rows + count - 1) / count + 15) & ~15, groups = (rows + each - 1) / each;
        const double blocks = (double)groups * nblocks, rounds = (each / 16 + 4) / 5;
        double sharers = std::sqrt(0.53 * hblocks / rounds);
        if (sharers < 1.0) sharers = 1.0;
        if (sharers > sm_count / blocks) sharers = sm_count / blocks;
        const double cost = 0.53 * hblocks / sharers + rounds * (sharers + 1.5);
        if (!best.groups || cost < least) {
            const int ctas = (int)std::ceil(blocks * sharers);
            best = Cut{groups, each < rows ? each : rows, ctas < sm_count ? ctas : sm_count};
            least = cost;
        }
    }
    return best;
}
WidePlan wide_plan(const DeviceWeights& w, const Cut& cut) {
    return plan_wide(w.inputs, w.bits, cut.rows, (long long)cut.groups * (w.inputs / 128) * (w.outputs / 128), cut.ctas);
}
}  // namespace

GemmPlan plan_gemm(const DeviceWeights& w, int rows, int sm_count) {
    GemmPlan plan{};
    plan.sm_count = sm_count;
    plan.dense = rows > kWideMaxRows && sm_count >= 2;
    if (plan.dense) {
        plan.act_bytes = align_up((size_t)gemm_dense_rows_padded(rows) * w.inputs * 2);
        plan.workspace_bytes = plan.act_bytes + gemm_dense_scratch(w);
        return plan;
    }
    const Cut cut = cut_call(w, rows, sm_count);
    const WidePlan wide = wide_plan(w, cut);
    plan.act_bytes = align_up((size_t)cut.groups * (w.inputs / 128) * wide_tile_bytes(cut.rows));
    plan.workspace_bytes = wide.flag_bytes + wide.plane_bytes + plan.act_bytes;
    return plan;
}

cudaError_t launch_gemm(const LinearCall& call, const GemmPlan& plan, void* workspace, bool programmatic_launch,
                        cudaStream_t stream) {
    if (!workspace) return cudaErrorInvalidValue;
    unsigned char* base = static_cast<unsigned char*>(workspace);
    if (plan.dense) return launch_gemm_dense(call, base, plan.sm_count, programmatic_launch, stream);
    const Cut cut = cut_call(call.w, call.rows, plan.sm_count);
    const WidePlan wide = wide_plan(call.w, cut);
    WideSet set{};
    set.count = cut.groups;
    set.group_rows = cut.rows;
    set.inputs = call.w.inputs;
    set.outputs = call.w.outputs;
    set.codebook = call.w.codebook;
    set.one = WideProblem{call.w, call.x, call.y, nullptr, nullptr, call.x_stride, call.y_stride,
                          base + wide.flag_bytes + wide.plane_bytes, call.rows, call.x_dtype, call.y_dtype, call.alpha, call.beta};
    unsigned int* flags = reinterpret_cast<unsigned int*>(base);
    const cudaError_t e = launch_wide_inputs(set, wide, flags, programmatic_launch, stream);
    if (e != cudaSuccess) return e;
    return launch_wide(set, wide, flags, reinterpret_cast<float*>(base + wide.flag_bytes), call.status, programmatic_launch, stream);
}

}  // namespace st
