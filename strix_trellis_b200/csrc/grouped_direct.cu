// Grouped linears of a few rows with little work for each SM (see grouped.h; the rule is direct_pays):
// one CTA = (problem of up to eight rows, 128-column block, K partition).  A producer warp streams the
// partition's contiguous weight bytes through a shared-memory ring (1-D bulk copies), eight decode
// warps each own a 16-column tile and feed mma.sync.m16n8k16; partial planes go to the problem's
// scratch and the last CTA of a column block to arrive folds them in ascending K order and applies the
// output stages.  Bound by the decode's issue slots as wide_linear.cu is, and about a tenth slower
// per unit (an mma.sync costs the issue port more than a tensor-memory store), but its input stages
// need no launch of their own and its start no tensor memory: 4 tokens over 48 experts, 3200 x 640,
// 32.6 us a block against 52.6.  Same arithmetic per row as the single-layer GEMV.
// (src/tp_moe.hip:60-164, src/tp_fused_device.hpp:19-126, src/dense_r1_group*.hip)
#include "grouped.h"
#include "hadamard.cuh"
#include "launch.h"
#include "sync_primitives.cuh"
#include "trellis_decode.cuh"

namespace st {

namespace {
constexpr int kWarps = 8;
constexpr int kMaxStages = kDirectStages;
constexpr int kThreadsG = (kWarps + 1) * 32;

struct DirectArgs {
    const GroupedProblem* problems;
    int ctas_per_problem;
    int splits;
    int stages;
    int hblocks;
    int stage_stride;  // bytes between ring slots (sized for the largest rate in the group)
    size_t counter_bytes;  // of a problem: its counters, zero between launches, then its partial planes
    unsigned int* status;
};

// Decode loop of one CTA for rate K.  Returns false when a bounded wait gave up.
template <int K, int CB>
__device__ __forceinline__ bool consume(const unsigned char* ring, int stage_stride, int stages, int nblk, uint32_t full0,
                                        uint32_t empty0, const uint2* act_lane, int rows, int warp, int lane,
                                        unsigned int* status, float (&acc)[2][4]) {
    const LaneGeom<K> geom(lane);
    int st = 0;
    uint32_t use = 0;  // ring slot and use parity of unit i, stepped without divisions
    for (int i = 0; i < nblk; ++i, st = (st + 1 == stages ? 0 : st + 1), use ^= (st == 0)) {
        if (!mbar_wait(full0 + 8 * st, use, status, kTimeoutRingFull)) return false;
        const uint32_t* tiles = reinterpret_cast<const uint32_t*>(ring + (size_t)st * stage_stride) + warp * quad_words(K);
        const uint2* bsrc = act_lane + (size_t)i * rows * 32;
#pragma unroll
        for (int half = 0; half < 2; ++half) {
            uint32_t f[4][4];
            decode_quad_frag<K, CB>(tiles + half * 8 * quad_words(K), geom, f);
#pragma unroll
            for (int t = 0; t < 4; ++t) {
                const uint2 b = bsrc[(half * 4 + t) * 4];
                mma_16816(acc[t & 1], f[t], b.x, b.y);
            }
        }
        __syncwarp();
        if (lane == 0) mbar_arrive(empty0 + 8 * st);
    }
    return true;
}
}  // namespace

// At most 64 registers: a CTA of the launch after next then fits beside two of these and one of the
// small kernel between (3 tokens x 6 routes, 2048 x 768: the down projection 16.2 us with 72).
template <int CB>
__global__ void __maxnreg__(64) grouped_direct_kernel(const DirectArgs args) {
    extern __shared__ __align__(128) unsigned char smem[];
    const int pidx = blockIdx.x / args.ctas_per_problem, rem = blockIdx.x % args.ctas_per_problem;
    const GroupedProblem& pr = args.problems[pidx];
    // problem tables may have been written by the prior grid (device routing)
    pdl_wait_prior_grid();
    const int live = args.problems->live, rows = pr.rows;
    if (pidx >= live) return;
    unsigned int* counters = reinterpret_cast<unsigned int*>(pr.tiles);
    float* partials = reinterpret_cast<float*>(pr.tiles + args.counter_bytes);
    const DeviceWeights w = pr.w;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int nb = rem / args.splits, split = rem % args.splits;
    const int hblocks = args.hblocks;
    const int hb_begin = (int)((long long)hblocks * split / args.splits);
    const int hb_end = (int)((long long)hblocks * (split + 1) / args.splits);
    const int nblk = hb_end - hb_begin;
    const int stages = args.stages;
    const int stage_bytes = unit_bytes(w.bits);

    uint64_t* bars = reinterpret_cast<uint64_t*>(smem);
    unsigned char* ring = smem + 256;
    uint2* act = reinterpret_cast<uint2*>(ring + (size_t)stages * args.stage_stride);
    __shared__ int s_last, s_abort;
    const uint32_t full0 = smem_u32(bars), empty0 = smem_u32(bars + kMaxStages);
    if (threadIdx.x == 0) {
        for (int i = 0; i < stages; ++i) {
            mbar_init(full0 + 8 * i, 1);
            mbar_init(empty0 + 8 * i, kWarps);
        }
        mbar_fence_init();
        s_abort = 0;
    }
    __syncthreads();
    pdl_launch_dependents();

    if (warp == kWarps) {
        if (lane == 0) {
            const unsigned char* stream = reinterpret_cast<const unsigned char*>(w.packed) +
                ((size_t)nb * hblocks + hb_begin) * stage_bytes;
            int issued = 0;
            for (int i = 0; i < nblk; ++i) {
                const int st = i % stages;
                if (i >= stages && !mbar_wait(empty0 + 8 * st, (uint32_t)((i / stages) - 1) & 1, args.status, kTimeoutRingEmpty)) {
                    s_abort = 1;
                    break;
                }
                mbar_expect_tx(full0 + 8 * st, stage_bytes);
                bulk_load(smem_u32(ring + (size_t)st * args.stage_stride), stream + (size_t)i * stage_bytes, stage_bytes,
                          full0 + 8 * st);
                issued = i + 1;
            }
            for (int i = (issued > stages ? issued - stages : 0); i < issued; ++i)
                mbar_wait(full0 + 8 * (i % stages), (uint32_t)(i / stages) & 1, args.status, kTimeoutDrain);
        }
    } else {
        // input stages of the gathered rows for this K partition, in B-fragment order
        __half* act_h = reinterpret_cast<__half*>(act);
        for (int item = warp; item < rows * nblk; item += kWarps) {
            const int r = item / nblk, blk = item % nblk;
            const float* xr = static_cast<const float*>(pr.x) + (long long)pr.x_row[r] * pr.x_stride + (size_t)(hb_begin + blk) * 128;
            const uint16_t* su = w.suh + (size_t)(hb_begin + blk) * 128;
            float v[4];
#pragma unroll
            for (int j = 0; j < 4; ++j) v[j] = __half2float(scale_input(xr[lane + 32 * j], su[lane + 32 * j]));
            hadamard128_warp(v, lane);
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const int e = lane + 32 * j, kt = e >> 4, kk = e & 15;
                const int q = (kk & 7) >> 1, hi = kk >> 3, lo = kk & 1;
                act_h[((((size_t)blk * rows + r) * 8 + kt) * 4 + q) * 4 + hi * 2 + lo] = __float2half_rn(v[j]);
            }
        }
        named_barrier(1, kWarps * 32);

        float acc[2][4] = {{0.f, 0.f, 0.f, 0.f}, {0.f, 0.f, 0.f, 0.f}};
        const int brow = (lane >> 2) < rows ? (lane >> 2) : rows - 1;
        const uint2* act_lane = act + brow * 32 + (lane & 3);
        bool ok;
        switch (w.bits) {
        case 1: ok = consume<1, CB>(ring, args.stage_stride, stages, nblk, full0, empty0, act_lane, rows, warp, lane, args.status, acc); break;
        case 2: ok = consume<2, CB>(ring, args.stage_stride, stages, nblk, full0, empty0, act_lane, rows, warp, lane, args.status, acc); break;
        case 3: ok = consume<3, CB>(ring, args.stage_stride, stages, nblk, full0, empty0, act_lane, rows, warp, lane, args.status, acc); break;
        case 4: ok = consume<4, CB>(ring, args.stage_stride, stages, nblk, full0, empty0, act_lane, rows, warp, lane, args.status, acc); break;
        case 5: ok = consume<5, CB>(ring, args.stage_stride, stages, nblk, full0, empty0, act_lane, rows, warp, lane, args.status, acc); break;
        case 6: ok = consume<6, CB>(ring, args.stage_stride, stages, nblk, full0, empty0, act_lane, rows, warp, lane, args.status, acc); break;
        case 7: ok = consume<7, CB>(ring, args.stage_stride, stages, nblk, full0, empty0, act_lane, rows, warp, lane, args.status, acc); break;
        case 8: ok = consume<8, CB>(ring, args.stage_stride, stages, nblk, full0, empty0, act_lane, rows, warp, lane, args.status, acc); break;
        default:  // half-integer rates exist for mul1 only
            if constexpr (CB == CB_MUL1) {
                if (w.bits == 9) ok = consume<9, CB>(ring, args.stage_stride, stages, nblk, full0, empty0, act_lane, rows, warp, lane, args.status, acc);
                else if (w.bits == 10) ok = consume<10, CB>(ring, args.stage_stride, stages, nblk, full0, empty0, act_lane, rows, warp, lane, args.status, acc);
                else ok = consume<11, CB>(ring, args.stage_stride, stages, nblk, full0, empty0, act_lane, rows, warp, lane, args.status, acc);
            } else {
                ok = false;
            }
            break;
        }
        if (!ok) s_abort = 1;
        const int col = warp * 16 + (lane >> 2), r0 = 2 * (lane & 3);
        float* p = partials + (((size_t)nb * args.splits + split) * rows) * 128;
        const float v00 = acc[0][0] + acc[1][0], v01 = acc[0][1] + acc[1][1];
        const float v10 = acc[0][2] + acc[1][2], v11 = acc[0][3] + acc[1][3];
        if (r0 < rows) { p[r0 * 128 + col] = v00; p[r0 * 128 + col + 8] = v10; }
        if (r0 + 1 < rows) { p[(r0 + 1) * 128 + col] = v01; p[(r0 + 1) * 128 + col + 8] = v11; }
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        // one release/acquire atomic: the CTA's planes (ordered before it by the barrier) are
        // visible before the count, and the last arriver sees the planes of the others
        unsigned int seen;
        asm volatile("atom.add.acq_rel.gpu.global.u32 %0, [%1], 1;" : "=r"(seen) : "l"(counters + nb) : "memory");
        const int last = (seen == (unsigned int)args.splits - 1);
        if (last) counters[nb] = 0;  // visible at grid end, before any later launch
        s_last = last && !s_abort;
    }
    __syncthreads();
    if (!s_last || warp >= rows) return;
    {
        const int r = warp;
        float v[4] = {0.f, 0.f, 0.f, 0.f};
        for (int s = 0; s < args.splits; ++s) {
            const float* p = partials + (((size_t)nb * args.splits + s) * rows + r) * 128;
#pragma unroll
            for (int j = 0; j < 4; ++j) v[j] = __fadd_rn(v[j], __ldcg(p + lane + 32 * j));
        }
        hadamard128_warp(v, lane);
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const int cidx = nb * 128 + lane + 32 * j;
            float* out = static_cast<float*>(pr.y) + (long long)pr.y_row[r] * pr.y_stride + cidx;
            *out = finish_output(v[j], w.svh[cidx], w.bias, cidx, 1.0f, 0.0f, out);
        }
    }
}


// Opt-in dynamic shared memory is a per-device function attribute: set when a context is created
// on a device (configure_device), never on the launch path.
cudaError_t configure_direct_kernels() {
    cudaError_t e = cudaFuncSetAttribute(grouped_direct_kernel<CB_3INST>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kDirectSmemLimit);
    if (e == cudaSuccess)
        e = cudaFuncSetAttribute(grouped_direct_kernel<CB_MCG>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kDirectSmemLimit);
    if (e == cudaSuccess)
        e = cudaFuncSetAttribute(grouped_direct_kernel<CB_MUL1>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kDirectSmemLimit);
    return e;
}

cudaError_t launch_grouped_direct(const GroupedProblem* problems, int problem_count, int inputs, int outputs, int codebook,
                                  const GroupedPlan& plan, unsigned int* status, bool programmatic, cudaStream_t stream) {
    const DirectArgs args{problems, plan.ctas_per_problem, plan.splits, plan.stages, inputs / 128, plan.stage_stride,
                          align_up((size_t)(outputs / 128) * sizeof(unsigned int)), status};
    const long long grid = (long long)problem_count * plan.ctas_per_problem;
    if (grid > 0x7FFFFFFF || plan.smem_bytes > kDirectSmemLimit) return cudaErrorInvalidValue;
    return for_codebook(codebook, [&](auto cb) {
        return launch_pdl(grouped_direct_kernel<decltype(cb)::value>, (int)grid, kThreadsG, plan.smem_bytes, programmatic, stream, args);
    });
}

}  // namespace st
