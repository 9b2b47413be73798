// Routes of a GEMM (more than 8 rows) and their workspace.
//   up to kWideMaxRows   weights decoded on the fly into tensor memory (wide_linear.cu); beyond
//                        kWideRows rows every further 256 decode the weights again
//   more rows            weights decoded once into the workspace, dense GEMM (gemm_dense.cu)
#include "wide_linear.h"

namespace st {

int gemm_dense_rows_padded(int rows);
size_t gemm_dense_scratch(const DeviceWeights& w);
cudaError_t launch_gemm_dense(const LinearCall& call, unsigned char* workspace, int sm_count, bool programmatic,
                              cudaStream_t stream);

namespace {
// Measured at the crossing (4096 -> 12288, K5): 512 rows take 87 us on the fly (two decodes) and 82 us
// dense; 256 rows take one decode.
constexpr int kWideMaxRows = kWideRows;
// Weight units of all row groups of a call.
long long wide_units(const DeviceWeights& w, int rows) {
    return (long long)((rows + kWideRows - 1) / kWideRows) * (w.inputs / 128) * (w.outputs / 128);
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
    const WidePlan wide = plan_wide(w.inputs, w.bits, rows, wide_units(w, rows), sm_count);
    const size_t groups = (rows + kWideRows - 1) / kWideRows;
    plan.act_bytes = align_up(groups * (w.inputs / 128) * wide_tile_bytes(rows > kWideRows ? kWideRows : rows));
    plan.workspace_bytes = wide.flag_bytes + wide.plane_bytes + plan.act_bytes;
    return plan;
}

cudaError_t launch_gemm(const LinearCall& call, const GemmPlan& plan, void* workspace, bool programmatic_launch,
                        cudaStream_t stream) {
    if (!workspace) return cudaErrorInvalidValue;
    unsigned char* base = static_cast<unsigned char*>(workspace);
    if (plan.dense) return launch_gemm_dense(call, base, plan.sm_count, programmatic_launch, stream);
    const WidePlan wide = plan_wide(call.w.inputs, call.w.bits, call.rows, wide_units(call.w, call.rows), plan.sm_count);
    WideSet set{};
    set.count = (call.rows + kWideRows - 1) / kWideRows;
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
