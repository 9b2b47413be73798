// Routes of a GEMM (more than 8 rows) and their workspace.
//   weights decoded on the fly into tensor memory, once for each row group (wide_linear.cu)
//   weights decoded once into the workspace, dense GEMM (gemm_dense.cu)
// Beyond kWideMaxRows always the second; below, whichever the estimates here say is faster.
#include "strix_trellis_b200.h"
#include "wide_linear.h"

#include <cmath>

namespace st {

int gemm_dense_rows_padded(int rows);
bool gemm_dense_narrow(int m_tiles, int nblocks, int pairs);
size_t gemm_dense_scratch(const DeviceWeights& w);
cudaError_t launch_gemm_dense(const LinearCall& call, unsigned char* workspace, int sm_count, bool programmatic,
                              cudaStream_t stream);

namespace {
// As far as the estimates are fitted and measured; beyond, four and more decodes of a unit hardly pay.
constexpr int kWideMaxRows = 1024;

// How a call's rows are cut into groups that each decode the weights, and how many CTAs run them: one
// group and every SM, unless so few column blocks are left that many CTAs share one and the CTA that
// finishes it adds all their planes (178 rows on 3072 -> 2048, nine CTAs a block: 51 us in one group,
// 22 us in three).  Estimates in us, fitted to 150 shapes of 9 to 512 rows (rms error 10 %) and checked to 1024: a unit 0.6
// + 0.0023 a row (its activation tile comes from the L2 for every unit); a segment that is not a
// CTA's last 1.4 a chunk of 16 rows, 1.6 where its accumulators have no second buffer; in the last one
// a plane's chunk 0.9, five warp groups side by side.  With s CTAs a block that is (unit * hblocks +
// segment) / s + 0.9 * rounds * s; s is taken somewhat below the least of that, which is flat.
struct Cut { int groups, rows, ctas; double us; };
Cut cut_call(const DeviceWeights& w, int rows, int sm_count) {
    const int hblocks = w.inputs / 128, nblocks = w.outputs / 128;
    Cut best{};
    for (int count = (rows + kWideRows - 1) / kWideRows; !best.groups || rows / count >= 32; ++count) {
        const int each = ((rows + count - 1) / count + 15) & ~15, groups = (rows + each - 1) / each;
        const double blocks = (double)groups * nblocks, rounds = (each / 16 + 4) / 5;
        const double unit = 0.6 + 0.0023 * each, segment = (each > 64 ? 1.6 : 1.4) * (each / 16);
        const double block = unit * hblocks + segment;
        double sharers = std::sqrt(block / (1.4 * rounds));
        if (sharers < 1.0) sharers = 1.0;
        if (sharers > sm_count / blocks) sharers = sm_count / blocks;
        const double us = 7.8 + block / sharers + 0.9 * rounds * sharers;
        if (!best.groups || us < best.us) {
            const int ctas = (int)std::ceil(blocks * sharers);
            best = Cut{groups, each < rows ? each : rows, ctas < sm_count ? ctas : sm_count, us};
        }
    }
    return best;
}
// The dense route in us, fitted likewise: decoding and storing a unit 0.59 on its SM; then a K step of 64
// for every wave of tiles, 256 x 256 or (gemm_dense_narrow) 256 x 128, faster where a wave leaves
// pairs of SMs idle because their loads share the L2.
double dense_us(const DeviceWeights& w, int rows, int sm_count) {
    const int hblocks = w.inputs / 128, nblocks = w.outputs / 128, m_tiles = gemm_dense_rows_padded(rows) / 256, pairs = sm_count / 2;
    const bool narrow = gemm_dense_narrow(m_tiles, nblocks, pairs);
    const int tiles = m_tiles * (narrow ? nblocks : (nblocks + 1) / 2), full = tiles / pairs, rest = tiles % pairs;
    const double step = 0.485 * full + (rest ? 0.28 + 0.205 * rest / pairs : 0.0);
    return 14.5 + 0.59 * hblocks * nblocks / sm_count + (narrow ? 0.72 : 1.0) * step * 2 * hblocks;
}
WidePlan wide_plan(const DeviceWeights& w, const Cut& cut) {
    return plan_wide(w.bits, cut.rows, (long long)cut.groups * (w.inputs / 128) * (w.outputs / 128), cut.ctas);
}
}  // namespace

GemmPlan plan_gemm(const DeviceWeights& w, int rows, int sm_count) {
    GemmPlan plan{};
    plan.sm_count = sm_count;
    const Cut cut = cut_call(w, rows, sm_count);
    plan.dense = sm_count >= 2 && (rows > kWideMaxRows || dense_us(w, rows, sm_count) < cut.us);
    if (plan.dense) {
        plan.act_bytes = align_up((size_t)gemm_dense_rows_padded(rows) * w.inputs * 2);
        plan.workspace_bytes = plan.act_bytes + gemm_dense_scratch(w);
        return plan;
    }
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

// Pure host arithmetic: no context, no device.
extern "C" strix_status strix_b200_gemm_route(uint64_t inputs, uint64_t outputs, uint32_t bits_x2, uint32_t rows, uint32_t sm_count,
                                              uint64_t out[4]) {
    if (!out) return STRIX_ERROR_INVALID_ARGUMENT;
    out[0] = out[1] = out[2] = out[3] = 0;
    const int code = st::rate_code(bits_x2);
    if (!inputs || !outputs || inputs % 128 || outputs % 128 || inputs > (1u << 30) || outputs > (1u << 30) ||
        (inputs / 128) * (outputs / 128) > 0x7FFFFFFF || !code ||
        rows <= 8 || rows > 0x7FFFFFFF || !sm_count || sm_count > 4096)
        return STRIX_ERROR_INVALID_ARGUMENT;
    st::DeviceWeights w{};
    w.inputs = (int)inputs;
    w.outputs = (int)outputs;
    w.bits = code;
    const st::GemmPlan plan = st::plan_gemm(w, (int)rows, (int)sm_count);
    out[0] = plan.dense;
    out[1] = plan.workspace_bytes;
    if (!plan.dense) {
        const st::Cut cut = st::cut_call(w, (int)rows, (int)sm_count);
        out[2] = (uint64_t)cut.groups;
        out[3] = (uint64_t)cut.ctas;
    }
    return STRIX_SUCCESS;
}
