// Fused decode GEMV of ONE activation row, the single-user decode case, where the head and the tail
// of the launch weigh as much as the loop: input stages, trellis decode, tensor-core dot, split-K
// fold and output stages in one launch.  It stands in for the reference's fused R1 variants
// (src/gemv_fused.hip:17-129, src/gemv_fused_both.hip:10-93).
//
// Work split ("stream-K"): the weights are one byte stream of units, a unit being the 64 tiles of
// (one 128-column block) x (one H128 block of K), ordered column block major -- exactly the prepared
// layout.  The grid is one persistent CTA per SM and CTA c owns a contiguous unit range
// (gemv_partition.h), streamed through a shared-memory ring by 1-D bulk copies.  Sixteen decode
// warps: warp (t, g) owns column tile t of the units of parity g.  A decoded tile is the A operand of
// mma.sync.m16n8k16 (m = output column), the activation row is its B operand.
//
// Against gemv_tmem.cu, which serves more rows: mma.sync costs the decoders about 12 % of their
// rate, but nothing of the chain tensor memory -> commit -> epilogue warp -> transposition stands
// between the last tile and the fold (16 layers of K4 in a chain of launches: 152 against 161 us).
// Layers of many units per CTA are the other way round (plan_gemv).
#include "gemv_kernels.h"
#include "hadamard.cuh"
#include "launch.h"
#include "sync_primitives.cuh"
#include "trellis_decode.cuh"

namespace st {

namespace {
constexpr int kGroups = 2;                       // k-tile parities per column tile
constexpr int kConsumers = 8 * kGroups;          // decode warps
constexpr int kThreads = (kConsumers + 2) * 32;  // + producer warp + epilogue warp
constexpr int kDumpThreads = (kConsumers + 1) * 32;  // decode warps + epilogue warp
constexpr uint32_t kEmptyWord = 0xFFFFFFFFu;      // a partial-plane word nobody has written yet
constexpr int kActBytes = 64 * 1024;             // core input a CTA can stage
constexpr size_t kGemvSmemLimit = 200 * 1024;    // dynamic shared memory a launch may ask for

struct GemvArgs {
    LinearCall call;
    Split split;               // unit range of every CTA (units / grid, units % grid)
    int stages;
    float* partials;           // [grid][2 k-groups][128], every word empty on entry and on exit
};

}  // namespace

// ---- one activation row -----------------------------------------------------------------
namespace {
constexpr int kRowHeader = 2048 + 8192 + 128 + 512;  // fold buffers, gathered planes, flag, barriers
static_assert(kRowHeader % 128 == 0, "the ring starts on a 128-byte boundary");

__device__ __forceinline__ uint4 ld_relaxed_gpu_v4(const uint4* p) {
    uint4 v;
    asm volatile("ld.relaxed.gpu.global.v4.u32 {%0,%1,%2,%3}, [%4];"
                 : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "l"(p) : "memory");
    return v;
}
__device__ __forceinline__ void st_relaxed_gpu_v4(uint4* p, uint4 v) {
    asm volatile("st.relaxed.gpu.global.v4.u32 [%0], {%1,%2,%3,%4};" ::"l"(p), "r"(v.x), "r"(v.y), "r"(v.z), "r"(v.w)
                 : "memory");
}
__device__ __forceinline__ bool any_empty(const uint4& a, const uint4& b) {
    return a.x == kEmptyWord || a.y == kEmptyWord || a.z == kEmptyWord || a.w == kEmptyWord ||
           b.x == kEmptyWord || b.y == kEmptyWord || b.z == kEmptyWord || b.w == kEmptyWord;
}

// One warp waits for one contributor's plane: lane l owns columns 4l..4l+3 of both k-group
// halves.  The first load is looked at as soon as it is back: measured on the benchmark shapes,
// most planes are already there when the finishing CTA gets here, and anything that delays the
// first look (pacing the loads, staggering them) costs more than it gains.  Returns the two
// halves (every word a value) and marks the plane empty again; false when the bounded wait
// runs out.
__device__ __forceinline__ bool await_plane(uint4* g0, uint4* g1, int lane, uint4& a, uint4& b) {
    bool have = false;
    for (uint32_t tries = 0; tries < (1u << 20) && !have; ++tries) {
        a = ld_relaxed_gpu_v4(g0 + lane);
        b = ld_relaxed_gpu_v4(g1 + lane);
        have = __all_sync(0xFFFFFFFFu, !any_empty(a, b));
    }
    if (have) {
        const uint4 empty = make_uint4(kEmptyWord, kEmptyWord, kEmptyWord, kEmptyWord);
        st_relaxed_gpu_v4(g0 + lane, empty);  // empty again for the next launch
        st_relaxed_gpu_v4(g1 + lane, empty);
    }
    return have;
}
}  // namespace

// One row, core input resident in shared memory.  Roles: 16 decode warps, one producer warp
// (bulk copies of the weight stream), one epilogue warp (finishes column blocks that lie
// wholly inside this CTA's range while the decode warps go on).
//
// Head: the producer streams weights from the moment the CTA starts (weights are immutable, so
// this does not wait for the previous kernel of the stream); the input scales of a warp's
// H128 block are fetched before the wait on the previous kernel too, so that only the load of
// the activation row and the input stages follow it, then one barrier, then the first mma.
// (Decoding a warp's first tiles into registers while that load is in flight was measured:
// 0.25 us per launch slower, the extra live registers cost more than the overlap gains.)
//
// Tail: a CTA whose range BEGINS inside a column block is a contributor to it: its decode
// warps store their accumulators straight into the CTA's plane in global scratch
// ([cta][k-group][128] floats), no shared-memory hop and no other warp involved.  The CTA whose
// range ENDS inside a block (it holds the block's first K range) finishes it: decode warp p
// waits for plane p (await_plane), the planes meet in shared memory, and warp 0 adds them in
// ascending K order from +0, its own contribution first, then H128, svh, bias, alpha, beta.
template <int K, int CB>
__global__ void __launch_bounds__(kThreads, 1) gemv_row_kernel(const GemvArgs args) {
    extern __shared__ __align__(128) unsigned char smem[];
    const LinearCall& c = args.call;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int hblocks = c.w.inputs / 128;
    const int cta = (int)blockIdx.x;
    const Range mine = cta_range(args.split, cta);
    const int my_units = mine.end - mine.begin;
    const int stages = args.stages;
    constexpr int kStage = unit_bytes(K);

    // shared memory: [2 x fold 1 KB][16 gathered planes 8 KB][flag][barriers 512 B][ring][core input]
    float* fold_base = reinterpret_cast<float*>(smem);            // [2 buffers][2 k-groups][128]
    float* gathered = reinterpret_cast<float*>(smem + 2048);      // [16][128]
    int* gave_up = reinterpret_cast<int*>(smem + 2048 + 8192);
    uint64_t* bars = reinterpret_cast<uint64_t*>(smem + 2048 + 8192 + 128);
    unsigned char* ring = smem + kRowHeader;
    uint2* act = reinterpret_cast<uint2*>(ring + (size_t)stages * kStage);

    const uint32_t full0 = smem_u32(bars), empty0 = smem_u32(bars + stages);
    // By the producer's lanes, one per ring slot.  Measured for a sweep of 96 launches and for the same sweep as
    // two chains on two streams: 864 / 758 us so; by a decode warp 892 / 781; with the CTA's first two units
    // asked for here, before the barrier, 885 / 790.
    if (warp == kConsumers && lane < stages) {
        mbar_init(full0 + 8 * lane, 1);
        mbar_init(empty0 + 8 * lane, 8);
        mbar_fence_init();
    }
    if (threadIdx.x == 0) *gave_up = 0;
    __syncthreads();
    pdl_launch_dependents();

    if (warp == kConsumers) {
        // ---- producer: weights are immutable, so this needs no wait on the launch before ----
        if (lane == 0) {
            int issued = 0;
            int st = 0;  // ring slot of the next unit and the parity of its previous use, stepped without divisions
            uint32_t prev_use = 1;
            for (; issued < my_units; ++issued) {
                if (issued >= stages && !mbar_wait(empty0 + 8 * st, prev_use, c.status, kTimeoutRingEmpty)) break;
                mbar_expect_tx(full0 + 8 * st, kStage);
                bulk_load(smem_u32(ring) + st * kStage,
                          reinterpret_cast<const unsigned char*>(c.w.packed) + (size_t)(mine.begin + issued) * kStage, kStage, full0 + 8 * st);
                if (++st == stages) { st = 0; prev_use ^= 1; }
            }
            // Never leave the CTA with a copy still landing in its shared memory.
            for (int i = (issued > stages ? issued - stages : 0); i < issued; ++i)
                mbar_wait(full0 + 8 * (i % stages), (i / stages) & 1, c.status, kTimeoutDrain);
        }
        return;
    }

    // Walk of the CTA's unit range, cut at column-block ends; shared by decode and epilogue
    // warps (each calls it once per segment, in order).
    int walk_nb = mine.begin / hblocks, walk_hb0 = mine.begin - walk_nb * hblocks;
    auto segment = [&](int done, int& nb, int& hb0, int& len) {
        nb = walk_nb;
        hb0 = walk_hb0;
        len = my_units - done;
        if (len > hblocks - hb0) len = hblocks - hb0;
        walk_hb0 += len;
        if (walk_hb0 == hblocks) { walk_hb0 = 0; ++walk_nb; }
    };
    // A segment [hb0, hb0+len) of block nb ends the block or the range.  It is `whole` when the
    // block lies inside this CTA's range.
    auto is_whole = [&](int nb) { return mine.begin <= nb * hblocks && mine.end >= (nb + 1) * hblocks; };

    if (warp == kConsumers + 1) {
        // ---- epilogue warp: output stages of the blocks that need nobody else ---------------
        // Output scales and bias of every column block this CTA touches are weights, cold in DRAM,
        // and are needed at the very end of a block: ask the L2 for them now.
        for (int nb = mine.begin / hblocks, last = (mine.end - 1) / hblocks; nb <= last && my_units > 0; ++nb) {
            if (lane < 2) prefetch_line_l2(c.w.svh + (size_t)nb * 128 + lane * 64);
            else if (lane < 6 && c.w.bias) prefetch_line_l2(c.w.bias + (size_t)nb * 128 + (lane - 2) * 32);
        }
        pdl_wait_prior_grid();  // y may belong to the prior grid
        int done = 0, flush = 0;
        while (done < my_units) {
            int nb, hb0, len;
            segment(done, nb, hb0, len);
            done += len;
            if (!is_whole(nb)) continue;
            const int buf = flush & 1;
            float sv[4], bs[4];
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const int cidx = nb * 128 + lane + 32 * j;
                sv[j] = half_bits_to_float(c.w.svh[cidx]);
                bs[j] = c.w.bias ? c.w.bias[cidx] : 0.0f;
            }
            named_barrier(2 + buf, kDumpThreads);  // all decode warps have dumped into `buf`
            const float* f0 = fold_base + buf * 256;
            float v[4];
#pragma unroll
            for (int j = 0; j < 4; ++j) v[j] = __fadd_rn(0.f, __fadd_rn(f0[lane + 32 * j], f0[128 + lane + 32 * j]));
            hadamard128_warp(v, lane);
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                float value = __fmul_rn(v[j], sv[j]);
                if (c.w.bias) value = __fadd_rn(value, bs[j]);
                scale_and_store(c.y, c.y_dtype, (long long)nb * 128 + lane + 32 * j, value, c.alpha, c.beta);
            }
            asm volatile("bar.arrive %0, %1;" ::"r"(4 + buf), "r"(kDumpThreads) : "memory");
            ++flush;
        }
        return;
    }

    // ---- decode warps -------------------------------------------------------------------
    const int ctile = warp & 7, kgroup = warp >> 3;
    const LaneGeom<K> geom(lane);
    const int need = my_units < hblocks ? my_units : hblocks;  // H128 blocks of the row this CTA touches
    const int hb_first = walk_hb0;
    int my_hb = hb_first + warp;                               // the block this warp stages (warp < need)
    if (my_hb >= hblocks) my_hb -= hblocks;
    uint16_t su[4] = {0, 0, 0, 0};
    if (warp < need) {  // input scales are weights: fetched before the wait on the prior grid
#pragma unroll
        for (int j = 0; j < 4; ++j) su[j] = c.w.suh[(size_t)my_hb * 128 + lane + 32 * j];
    }
    // The activation row may still be in flight from the prior grid, or cold in DRAM when it came
    // from the host: ask the L2 for this CTA's part of it now, read it after the wait.
    {
        const int x_bytes = c.x_dtype == DT_F32 ? 4 : 2;
        if (lane * 128 < 128 * x_bytes)
            for (int item = warp; item < need; item += kConsumers) {
                int hb = hb_first + item;
                if (hb >= hblocks) hb -= hblocks;
                prefetch_line_l2(reinterpret_cast<const unsigned char*>(c.x) + (size_t)hb * 128 * x_bytes + lane * 128);
            }
    }
    pdl_wait_prior_grid();  // x, y and the scratch may belong to the prior grid
    float xv[4] = {0.f, 0.f, 0.f, 0.f};
    if (warp < need) {
#pragma unroll
        for (int j = 0; j < 4; ++j) xv[j] = load_element(c.x, c.x_dtype, (long long)my_hb * 128 + lane + 32 * j);
    }

    bool ok = true;
    int slot = kgroup % stages;  // ring slot and use parity of the unit this warp decodes next
    uint32_t use = (uint32_t)(kgroup / stages) & 1;

    // input stages of this warp's block, written in B-fragment order:
    // act[(hb*8 + kt)*4 + q] = {half2(k0,k0+1), half2(k0+8,k0+9)}, k0 = 2q
    __half* act_h = reinterpret_cast<__half*>(act);
    for (int item = warp; item < need; item += kConsumers) {
        int hb = hb_first + item;
        if (hb >= hblocks) hb -= hblocks;
        float v[4];
        if (item == warp) {
#pragma unroll
            for (int j = 0; j < 4; ++j) v[j] = __half2float(scale_input(xv[j], su[j]));
        } else {  // more blocks than warps: the rest comes straight from memory
#pragma unroll
            for (int j = 0; j < 4; ++j)
                v[j] = __half2float(scale_input(load_element(c.x, c.x_dtype, (long long)hb * 128 + lane + 32 * j),
                                                c.w.suh[(size_t)hb * 128 + lane + 32 * j]));
        }
        hadamard128_warp(v, lane);
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const int e = lane + 32 * j, kt = e >> 4, kk = e & 15;
            const int q = (kk & 7) >> 1, hi = kk >> 3, lo = kk & 1;
            act_h[(((size_t)hb * 8 + kt) * 4 + q) * 4 + hi * 2 + lo] = __float2half_rn(v[j]);
        }
    }
    named_barrier(1, kConsumers * 32);

    // Only activation row 0 exists: lanes of every row feed it as the B operand; accumulator
    // columns of rows >= 1 are never read.
    const uint2* act_lane = act + (lane & 3);
    const int col = ctile * 16 + (lane >> 2);
    float acc[2][4] = {{0.f, 0.f, 0.f, 0.f}, {0.f, 0.f, 0.f, 0.f}};
    int done = 0, flush = 0;
    int next = kgroup;  // the unit (relative to the range) this warp decodes next
    while (done < my_units) {
        int nb, hb0, len;
        segment(done, nb, hb0, len);
        for (; next < done + len && ok; next += 2) {
            const int b = next - done, st = slot;
            ok = mbar_wait(full0 + 8 * st, use, c.status, kTimeoutRingFull);
            if (!ok) break;
            slot += 2;
            while (slot >= stages) { slot -= stages; use ^= 1; }
            const uint32_t* tiles = reinterpret_cast<const uint32_t*>(ring + (size_t)st * kStage) + ctile * quad_words(K);
            const uint2* bsrc = act_lane + (size_t)(hb0 + b) * 32;
#pragma unroll
            for (int half = 0; half < 2; ++half) {  // four independent tiles in flight
                uint32_t f[4][4];
                decode_quad_frag<K, CB>(tiles + half * 8 * quad_words(K), geom, f);
#pragma unroll
                for (int t = 0; t < 4; ++t) {
                    const uint2 bf = bsrc[(half * 4 + t) * 4];
                    mma_16816(acc[t & 1], f[t], bf.x, bf.y);
                }
            }
            __syncwarp();
            if (lane == 0) mbar_arrive(empty0 + 8 * st);
        }
        done += len;

        // ---- this CTA's contribution to column block nb is complete -------------------------
        // row 0 of the accumulators: lanes with lane % 4 == 0 hold columns col (c0) and col+8 (c2)
        const float v_lo = acc[0][0] + acc[1][0], v_hi = acc[0][2] + acc[1][2];
#pragma unroll
        for (int j = 0; j < 4; ++j) acc[0][j] = acc[1][j] = 0.f;
        const int blk_lo = nb * hblocks, blk_hi = blk_lo + hblocks;
        const bool whole = mine.begin <= blk_lo && mine.end >= blk_hi;
        if (!whole && mine.begin > blk_lo) {
            // contributor: publish straight from the registers, k-group planes apart
            if ((lane & 3) == 0) {
                uint32_t* plane = reinterpret_cast<uint32_t*>(args.partials) + ((size_t)cta * 2 + kgroup) * 128;
                st_relaxed_gpu(plane + col, __float_as_uint(v_lo));
                st_relaxed_gpu(plane + col + 8, __float_as_uint(v_hi));
            }
            continue;
        }
        const int buf = flush & 1;
        if (flush >= 2) named_barrier(4 + buf, kDumpThreads);  // the epilogue warp is done with `buf`
        if ((lane & 3) == 0) {
            float* g = fold_base + buf * 256 + kgroup * 128;
            g[col] = v_lo;
            g[col + 8] = v_hi;
        }
        ++flush;
        if (whole) {
            asm volatile("bar.arrive %0, %1;" ::"r"(2 + buf), "r"(kDumpThreads) : "memory");
            continue;
        }

        // ---- this CTA holds the block's first K range: it finishes the block ----------------
        // (the block goes on in later CTAs, so this is the end of the range)
        int first, last;
        contributors(args.split, blk_lo, blk_hi, first, last);
        const int planes = last - cta;
        float sv[4], bs[4], v[4];
        if (warp == 0) {
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const int cidx = nb * 128 + lane + 32 * j;
                sv[j] = half_bits_to_float(c.w.svh[cidx]);
                bs[j] = c.w.bias ? c.w.bias[cidx] : 0.0f;
            }
        }
        for (int base = 0; base < planes; base += kConsumers) {
            const int p = base + warp;
            if (p < planes) {
                uint4* g0 = reinterpret_cast<uint4*>(args.partials + ((size_t)(cta + 1 + p) * 2) * 128);
                uint4 a, bq;
                if (await_plane(g0, g0 + 32, lane, a, bq)) {
                    float4 sum;  // the contributor's own order: k-group 0 + k-group 1
                    sum.x = __fadd_rn(__uint_as_float(a.x), __uint_as_float(bq.x));
                    sum.y = __fadd_rn(__uint_as_float(a.y), __uint_as_float(bq.y));
                    sum.z = __fadd_rn(__uint_as_float(a.z), __uint_as_float(bq.z));
                    sum.w = __fadd_rn(__uint_as_float(a.w), __uint_as_float(bq.w));
                    reinterpret_cast<float4*>(gathered + warp * 128)[lane] = sum;
                } else if (lane == 0) {
                    atomicOr(c.status, kTimeoutFold);
                    *gave_up = 1;
                }
            }
            named_barrier(1, kConsumers * 32);  // planes of this round (and, first time, the dumps) are in shared memory
            if (warp == 0) {
                if (base == 0) {
                    const float* f0 = fold_base + buf * 256;
#pragma unroll
                    for (int j = 0; j < 4; ++j) v[j] = __fadd_rn(0.f, __fadd_rn(f0[lane + 32 * j], f0[128 + lane + 32 * j]));
                }
                const int n = planes - base < kConsumers ? planes - base : kConsumers;
                for (int q = 0; q < n; ++q) {
#pragma unroll
                    for (int j = 0; j < 4; ++j) v[j] = __fadd_rn(v[j], gathered[q * 128 + lane + 32 * j]);
                }
            }
            if (base + kConsumers < planes) named_barrier(1, kConsumers * 32);  // before `gathered` is reused
        }
        if (warp == 0 && ok && *gave_up == 0) {  // a wait that ran out leaves the block unwritten
            hadamard128_warp(v, lane);
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                float value = __fmul_rn(v[j], sv[j]);
                if (c.w.bias) value = __fadd_rn(value, bs[j]);
                scale_and_store(c.y, c.y_dtype, (long long)nb * 128 + lane + 32 * j, value, c.alpha, c.beta);
            }
        }
    }
}

// ---- host side -------------------------------------------------------------------------
bool plan_gemv_row(const DeviceWeights& w, GemvPlan& plan) {
    const int hblocks = w.inputs / 128, stride = unit_bytes(w.bits);
    const long long units = (long long)hblocks * (w.outputs / 128);
    const int per_cta = (int)((units + plan.grid - 1) / plan.grid);
    if (hblocks * 256 > kActBytes) return false;
    int stages = ((int)kGemvSmemLimit - kRowHeader - hblocks * 256) / stride;
    const int want = (128 * 1024) / stride;  // enough bytes in flight per SM to cover HBM latency
    if (stages > want) stages = want;
    if (stages > per_cta) stages = per_cta;
    if (stages > 28) stages = 28;
    if (stages < 1) stages = 1;
    plan.stages = stages;
    plan.act_blocks = hblocks;
    plan.smem_bytes = kRowHeader + (size_t)stages * stride + (size_t)hblocks * 256;
    plan.partial_bytes = align_up((size_t)plan.grid * 2 * 128 * sizeof(float));
    return true;
}

cudaError_t launch_gemv_row(const LinearCall& call, const GemvPlan& plan, Split split, float* planes, bool pdl, cudaStream_t stream) {
    const GemvArgs args{call, split, plan.stages, planes};
    return for_codebook(call.w.codebook, [&](auto cb) {
        return for_rate<decltype(cb)::value>(call.w.bits, [&](auto k) {
            return launch_pdl(gemv_row_kernel<decltype(k)::value, decltype(cb)::value>, plan.grid, kThreads, plan.smem_bytes, pdl, stream, args);
        });
    });
}

// Opt-in dynamic shared memory is a per-device function attribute: set for every instantiation
// when a context is created on a device (configure_device), never on the launch path.
template <int CB>
static cudaError_t configure_row() {
    cudaError_t e = cudaSuccess;
    for (int bits = 1; bits <= (CB == CB_MUL1 ? kRateCodes : 8) && e == cudaSuccess; ++bits)
        e = for_rate<CB>(bits, [&](auto k) {
            return cudaFuncSetAttribute(gemv_row_kernel<decltype(k)::value, CB>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                        (int)kGemvSmemLimit);
        });
    return e;
}
cudaError_t configure_gemv_row_kernels() {
    cudaError_t e = configure_row<CB_3INST>();
    if (e == cudaSuccess) e = configure_row<CB_MCG>();
    if (e == cudaSuccess) e = configure_row<CB_MUL1>();
    return e;
}

}  // namespace st
