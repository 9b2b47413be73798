// Linears of 9 to some hundred rows, one or many per launch: trellis tiles are decoded into TENSOR
// MEMORY and multiplied from there (tcgen05.mma with A in tensor memory), output stages fused.
// It stands in for the reference's tiled core at small row counts and for its per-expert
// projection kernels (src/wmma_tiled.hip:87-269, src/tp_moe.hip:60-164).
//
// Bound by the decode's issue slots: a weight is decoded once for up to 256 rows.  A decoded tile
// is, register for register, a piece of the MMA's A operand (128 weight columns = the 128 lanes of
// tensor memory), so it leaves a warp by ONE tcgen05.st per four tiles: no shared-memory stores, no
// swizzle arithmetic, no proxy fence, and none of the eight issue clocks that an mma.sync costs.
// The activation rows are the MMA's N (a multiple of 16): 16 or 256 rows cost the decoders the same.
//
// Work split (stream-K): the weights are units of (one 128-column block) x (one H128 block of K),
// ordered problem, column block, K; the grid is one persistent CTA per SM and CTA c owns a
// contiguous range of units (gemv_partition.h), whatever the shapes are.
// Roles: 16 decode warps (warp w feeds tensor-memory lane quarter w % 4, i.e. column tiles
// 2(w % 4) and +1, of every fourth unit), 4 epilogue warps, one producer thread each for
// the weight ring and the activation ring, one MMA issuer.
// Fold: a CTA whose range BEGINS inside a column block dumps its raw sums to its plane in global
// scratch (that is its first segment, done early) and counts the chunks in its flag; the CTA whose
// range holds the block's first K part finishes the block at the end of its own range and adds the
// planes in ascending K order.  Waits only point to higher CTA indices and every CTA is resident.
// The decode warps, idle at the end of the range, share the last segment's epilogue.
// Every wait is bounded and reports into the device status word.
#include "gemv_partition.h"
#include "hadamard.cuh"
#include "launch.h"
#include "sync_primitives.cuh"
#include "tmem_decode.cuh"
#include "wide_linear.h"

namespace st {

namespace {
constexpr int kUnitGroups = 4, kDecodeW = 4 * kUnitGroups, kEpiW = 4;
constexpr int kWarpMma = kDecodeW + kEpiW, kWarpWeights = kWarpMma + kIssuers, kWarpRows = kWarpWeights + 1;
constexpr int kThreadsW = (kWarpRows + 1) * 32;
constexpr int kChunkRows = 16;                       // rows of one epilogue chunk
constexpr int kStageFloats = kChunkRows * 128;       // 8 KB of transposition space per warp group
constexpr int kHeaderW = 1024 + 2 * kStageFloats * 4;  // barriers, the epilogue group's two staging areas
constexpr size_t kSmemLimitW = 224 * 1024;
constexpr int kMaxWSlots = 24, kMaxBSlots = 8;
constexpr int kRingMin = kDecodeW / 4 * kStageFloats * 4;       // the decode groups' staging of the last segment

struct WideArgs {
    const WideProblem* table;
    size_t table_stride;
    const int* live;
    WideProblem one;
    int count, group_rows, hblocks, nblocks;
    int n_max, w_slots, w_stride, b_slots, b_stride;
    // tensor memory: a_stages x 64 columns of A, then d_bufs buffers of `parts` times d_accs accumulators of n_max
    int a_stages, d_bufs, d_accs, parts, parts_log2;
    unsigned int* flags;
    float* planes;
    unsigned int* status;
};

// Problem p of the set: from the table, or row group p of the one layer.
__device__ __forceinline__ const WideProblem& problem(const WideArgs& a, int p) {
    return a.table ? *reinterpret_cast<const WideProblem*>(reinterpret_cast<const unsigned char*>(a.table) + p * a.table_stride) : a.one;
}
__device__ __forceinline__ int problem_rows(const WideArgs& a, int p) {
    if (a.table) return problem(a, p).rows;
    const int left = a.one.rows - p * a.group_rows;
    return left < a.group_rows ? left : a.group_rows;
}
__device__ __forceinline__ const unsigned char* problem_tiles(const WideArgs& a, int p) {
    return a.table ? problem(a, p).tiles : a.one.tiles + (size_t)p * a.hblocks * wide_tile_bytes(a.group_rows);
}

// First block of K part s: the blocks [part_begin(s), part_begin(s + 1)) have accumulators of their own.
__device__ __forceinline__ int part_begin(const WideArgs& a, int s) { return (a.hblocks * s) >> a.parts_log2; }
__device__ __forceinline__ int part_of(const WideArgs& a, int hb) {
    int part = 0;
    while (part_begin(a, part + 1) <= hb) ++part;
    return part;
}

// Position in a CTA's unit range; every role walks it segment by segment (a segment ends with a
// column block or with the range).
struct Walk {
    int unit, end, p, nb, hb;
    __device__ __forceinline__ Walk(const WideArgs& a, Range r) : unit(r.begin), end(r.end) {
        const int block = r.begin / a.hblocks;
        hb = r.begin - block * a.hblocks;
        p = block / a.nblocks;
        nb = block - p * a.nblocks;
    }
    __device__ __forceinline__ int length(const WideArgs& a) const {
        const int left = end - unit, block = a.hblocks - hb;
        return left < block ? left : block;
    }
    __device__ __forceinline__ void next(const WideArgs& a, int len) {
        unit += len;
        hb = 0;  // the next segment, if any, starts a block
        if (++nb == a.nblocks) { nb = 0; ++p; }
    }
};
}  // namespace

__device__ __forceinline__ unsigned int ld_acquire_gpu(const unsigned int* p) {
    unsigned int v;
    asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
    return v;
}
__device__ __forceinline__ void red_release_gpu(unsigned int* p, unsigned int v) {
    asm volatile("red.release.gpu.global.add.u32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}

// One segment's share of the epilogue by one warp group (four warps, one per tensor-memory lane
// quarter): chunks first_chunk, first_chunk + step, ... of 16 rows.  A thread reads its column of a
// chunk, adds the other CTAs' planes (finisher) or stores the sums to this CTA's plane
// (contributor); for outputs the chunk is transposed through `stage` and each warp finishes four
// rows, eight lanes per row.
template <bool PARTS>  // K in more than one part
struct Epilogue {
    const WideArgs& a;
    int cta, origin, quarter, lane, bar;  // origin: first unit of the range
    float* areas;      // staging: two areas in turn (one barrier per chunk instead of two), or one
    int area_floats;   // from one to the other; 0: one

    // false: a wait ran out (the whole group returns together)
    __device__ __forceinline__ bool segment(const Split& split, const Walk& w, int len, uint32_t dcol, int first_chunk, int step,
                                            uint32_t d_empty) const {
        const int rows = problem_rows(a, w.p), chunks = (rows + kChunkRows - 1) / kChunkRows;
        const int lo = (w.p * a.nblocks + w.nb) * a.hblocks, hi = lo + a.hblocks;
        const bool contributor = w.hb != 0;
        int last = cta;
        if (!contributor && w.hb + len < a.hblocks) last = owner(split, hi - 1);
        const WideProblem& pr = problem(a, w.p);
        // The flag of CTA c counts the chunks of its plane that are there.
        bool late = false;
        for (int c = cta + 1; c <= last && !late; ++c) {
            late = true;
            for (uint32_t tries = 0; tries < (1u << 20); ++tries)
                if (ld_acquire_gpu(a.flags + c) >= (unsigned int)chunks) { late = false; break; }
        }
        if (group_any(bar, late)) {
            if (late && lane == 0) atomicOr(a.status, kTimeoutFold);
            return false;
        }
        const int col = quarter * 32 + lane;
        const uint32_t taddr = ((uint32_t)(quarter * 32) << 16) + dcol;
        float* stage = areas;
        const int first_part = PARTS ? part_of(a, w.hb) : 0, last_part = PARTS ? part_of(a, w.hb + len - 1) : 0;  // of this segment
        int dumped = 0;
        for (int ch = first_chunk; ch < chunks; ch += step) {
            uint32_t r[16];
            // Parts in ascending K order; the running sum of a column waits in its place in `stage`.
#pragma unroll 1
            for (int part = first_part; part <= last_part; ++part) {
                // The units of this part in this segment: from two on both issuers have had some.
                const int lo = PARTS && part_begin(a, part) > w.hb ? part_begin(a, part) : w.hb;
                const int hi = PARTS && part_begin(a, part + 1) < w.hb + len ? part_begin(a, part + 1) : w.hb + len;
                const bool both = a.d_accs > 1 && hi - lo > 1;
                const int set = a.d_accs > 1 && !both ? (w.unit - origin + lo - w.hb) & 1 : 0;
                const uint32_t at = taddr + (part * a.d_accs + set * (a.d_accs >> 1)) * a.n_max + ch * kChunkRows;
                auto add = [&](uint32_t from) {
                    uint32_t q[16];
                    tmem_ld_32x16(from, q);
                    tmem_ld_wait();
#pragma unroll
                    for (int j = 0; j < 16; ++j) {
                        asm volatile("" : "+r"(q[j]), "+r"(r[j]));  // not before the wait
                        r[j] = __float_as_uint(__fadd_rn(__uint_as_float(r[j]), __uint_as_float(q[j])));
                    }
                };
                __syncwarp();
                tmem_ld_32x16(at, r);
                if (!PARTS && a.d_accs == 4) {  // one layer of up to sixteen rows
                    add(at + a.n_max);
                    if (both) {
                        uint32_t q[16], t[16];
                        tmem_ld_32x16(at + 2 * a.n_max, q);
                        tmem_ld_32x16(at + 3 * a.n_max, t);
                        tmem_ld_wait();
#pragma unroll
                        for (int j = 0; j < 16; ++j) {
                            asm volatile("" : "+r"(q[j]), "+r"(t[j]));
                            r[j] = __float_as_uint(__fadd_rn(__uint_as_float(r[j]), __fadd_rn(__uint_as_float(q[j]), __uint_as_float(t[j]))));
                        }
                    }
                } else if (both) {
                    add(at + a.n_max);
                } else {
                    tmem_ld_wait();
#pragma unroll
                    for (int j = 0; j < 16; ++j) asm volatile("" : "+r"(r[j]));
                }
                if (PARTS && part != first_part)
#pragma unroll
                    for (int j = 0; j < 16; ++j) r[j] = __float_as_uint(__fadd_rn(stage[j * 128 + col], __uint_as_float(r[j])));
                if (PARTS && part != last_part)
#pragma unroll
                    for (int j = 0; j < 16; ++j) stage[j * 128 + col] = __uint_as_float(r[j]);
            }
            if (d_empty && ch + step >= chunks) {  // the accumulators are in registers: the next segment's MMAs may start
                tc_fence_before_sync();
                __syncwarp();
                if (lane == 0) mbar_arrive(d_empty);
            }
            if (contributor) {
                float* plane = a.planes + ((size_t)cta * a.n_max + ch * kChunkRows) * 128 + col;
#pragma unroll
                for (int j = 0; j < 16; ++j) __stcg(plane + j * 128, __uint_as_float(r[j]));
                ++dumped;
                continue;
            }
            float v[16];
#pragma unroll
            for (int j = 0; j < 16; ++j) v[j] = __fadd_rn(0.f, __uint_as_float(r[j]));
            for (int c = cta + 1; c <= last; ++c) {
                const float* plane = a.planes + ((size_t)c * a.n_max + ch * kChunkRows) * 128 + col;
                float other[16];
#pragma unroll
                for (int j = 0; j < 16; ++j) other[j] = __ldcg(plane + j * 128);
#pragma unroll
                for (int j = 0; j < 16; ++j) v[j] = __fadd_rn(v[j], other[j]);
            }
#pragma unroll
            for (int j = 0; j < 16; ++j) stage[j * 128 + col] = v[j];
            named_barrier(bar, 128);
            finish_rows(pr, w, ch, rows, stage);
            if (!area_floats) named_barrier(bar, 128);  // (two areas: the next chunk's barrier does)
            stage = stage == areas ? areas + area_floats : areas;
        }
        if (contributor && dumped) {
            named_barrier(bar, 128);  // the group's stores are ordered before the count below
            if (quarter == 0 && lane == 0) red_release_gpu(a.flags + cta, (unsigned int)dumped);
        }
        return true;
    }

    __device__ __forceinline__ void finish_rows(const WideProblem& pr, const Walk& w, int ch, int rows, const float* stage) const {
        const int l8 = lane & 7;
        const int in_chunk = quarter * 4 + (lane >> 3);
        float v[4][4];
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const float4 t = *reinterpret_cast<const float4*>(stage + in_chunk * 128 + 32 * i + 4 * l8);
            v[i][0] = t.x; v[i][1] = t.y; v[i][2] = t.z; v[i][3] = t.w;
        }
        hadamard128_oct(v, lane);
        const int r = ch * kChunkRows + in_chunk;
        if (r >= rows) return;
        uint2 sv[4];
        float4 bi[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) {  // all loads before the first store
            const int c0 = w.nb * 128 + 32 * i + 4 * l8;
            sv[i] = __ldg(reinterpret_cast<const uint2*>(pr.w.svh + c0));
            bi[i] = pr.w.bias ? __ldg(reinterpret_cast<const float4*>(pr.w.bias + c0)) : make_float4(0.f, 0.f, 0.f, 0.f);
        }
        const int out_row = a.table ? (pr.y_rows ? pr.y_rows[r] : r) : w.p * a.group_rows + r;
        const bool aligned = quads_aligned(pr.y, pr.y_dtype, pr.y_stride);
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const int c0 = w.nb * 128 + 32 * i + 4 * l8;
            const uint32_t sw[2] = {sv[i].x, sv[i].y};
            const float bias[4] = {bi[i].x, bi[i].y, bi[i].z, bi[i].w};
            float o[4];
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                o[j] = __fmul_rn(v[i][j], half_bits_to_float((uint16_t)(sw[j >> 1] >> (16 * (j & 1)))));
                if (pr.w.bias) o[j] = __fadd_rn(o[j], bias[j]);
            }
            scale_and_store_quad(pr.y, pr.y_dtype, (long long)out_row * pr.y_stride + c0, aligned, o, pr.alpha, pr.beta);
        }
    }
};

// At most 72 registers: a CTA of the next call's input stages (128 threads) then fits beside this
// kernel's, is resident and has its operands in the L2 when this kernel ends.  (ptxas spills for it in
// the epilogue's chunk: 124 bytes stored and 188 loaded with K parts, 4 bytes without for mul1.)
template <int CB, bool PARTS>
__global__ void __maxnreg__(72) wide_linear_kernel(const WideArgs args) {
    extern __shared__ __align__(1024) unsigned char smem_raw[];
    unsigned char* smem = smem_raw + (-smem_u32(smem_raw) & 1023u);  // (still a shared-memory pointer to the compiler)
    const int warp = uniform_warp(), lane = threadIdx.x & 31, cta = (int)blockIdx.x;
    // Weights are immutable and a table is there before the launch before lets this one start (its own
    // wait comes first, see wide_inputs_kernel; acquiring the count acquires the table), so only the
    // activation producer waits.
    const int count = args.live ? (int)ld_acquire_gpu(reinterpret_cast<const unsigned int*>(args.live)) : args.count;
    const int units = count * args.nblocks * args.hblocks;
    const int grid = units < (int)gridDim.x ? units : (int)gridDim.x;
    if (cta >= grid) {
        // Without a live problem nobody else waits for the launch before, and a launch may only end after
        // it has: the one after this counts on that when it overwrites what the one before reads.
        if (!grid) pdl_wait_prior_grid();
        return;
    }
    const Split split = make_split(units, grid);
    const Range mine = cta_range(split, cta);
    const int my_units = mine.end - mine.begin;
    const int d_bufs = args.d_bufs, a_stages = args.a_stages;

    uint64_t* bars = reinterpret_cast<uint64_t*>(smem);
    float* epi_stage = reinterpret_cast<float*>(smem + 1024);
    unsigned char* b_ring = smem + kHeaderW;                                    // 1024-byte aligned images
    unsigned char* w_ring = b_ring + (size_t)args.b_slots * args.b_stride;
    __shared__ uint32_t s_tmem_base;
    const uint32_t w_full = smem_u32(bars), w_empty = w_full + 8 * kMaxWSlots, b_full = w_empty + 8 * kMaxWSlots,
                   b_empty = b_full + 8 * kMaxBSlots, a_full = b_empty + 8 * kMaxBSlots, a_empty = a_full + 8 * kMaxAStages,
                   d_full = a_empty + 8 * kMaxAStages, d_empty = d_full + 16, all_done = d_empty + 16;
    const int issuers = args.d_accs > 1 ? kIssuers : 1;
    if (threadIdx.x == 0) {
        for (int i = 0; i < args.w_slots; ++i) { mbar_init(w_full + 8 * i, 1); mbar_init(w_empty + 8 * i, 4); }
        for (int i = 0; i < args.b_slots; ++i) { mbar_init(b_full + 8 * i, 1); mbar_init(b_empty + 8 * i, 1); }
        for (int i = 0; i < a_stages; ++i) { mbar_init(a_full + 8 * i, 4); mbar_init(a_empty + 8 * i, 1); }
        for (int i = 0; i < 2; ++i) { mbar_init(d_full + 8 * i, issuers); mbar_init(d_empty + 8 * i, kEpiW); }
        mbar_init(all_done, issuers);
        mbar_fence_init();
    }
    if (warp == kWarpMma) tmem_alloc(smem_u32(&s_tmem_base), 512);
    tc_fence_before_sync();
    __syncthreads();
    tc_fence_after_sync();
    const uint32_t tmem = s_tmem_base;
    pdl_launch_dependents();

    auto d_column = [&](int seg) { return a_stages * 64 + (d_bufs == 2 ? (seg & 1) * args.parts * args.d_accs * args.n_max : 0); };
    auto d_parity = [&](int seg) { return (uint32_t)(d_bufs == 2 ? seg >> 1 : seg) & 1; };  // of the seg-th use
    auto d_index = [&](int seg) { return d_bufs == 2 ? seg & 1 : 0; };

    if (warp == kWarpWeights) {
        if (lane == 0) {
            int slot = 0, issued = 0;
            uint32_t prev_use = 1;
            bool ok = true;
            for (Walk w(args, mine); w.unit < w.end && ok;) {
                const int len = w.length(args);
                const DeviceWeights& dw = problem(args, w.p).w;
                const uint32_t bytes = unit_bytes(dw.bits);
                const unsigned char* src = reinterpret_cast<const unsigned char*>(dw.packed) +
                                           ((size_t)w.nb * args.hblocks + w.hb) * bytes;
                for (int i = 0; i < len; ++i, src += bytes) {
                    if (issued >= args.w_slots && !mbar_wait_long(w_empty + 8 * slot, prev_use, args.status, kTimeoutRingEmpty)) {
                        ok = false;
                        break;
                    }
                    mbar_expect_tx(w_full + 8 * slot, bytes);
                    bulk_load(smem_u32(w_ring + (size_t)slot * args.w_stride), src, bytes, w_full + 8 * slot);
                    ++issued;
                    if (++slot == args.w_slots) { slot = 0; prev_use ^= 1; }
                }
                w.next(args, len);
            }
            for (int i = (issued > args.w_slots ? issued - args.w_slots : 0); i < issued; ++i)  // nothing still landing at exit
                mbar_wait(w_full + 8 * (i % args.w_slots), (uint32_t)(i / args.w_slots) & 1, args.status, kTimeoutDrain);
        }
    } else if (warp == kWarpRows) {
        if (lane == 0) {
            pdl_wait_prior_grid();  // the tiles are the work of the launch before
            int slot = 0, issued = 0;
            uint32_t prev_use = 1;
            bool ok = true;
            for (Walk w(args, mine); w.unit < w.end && ok;) {
                const int len = w.length(args);
                const uint32_t bytes = (uint32_t)wide_tile_bytes(problem_rows(args, w.p));
                const unsigned char* src = problem_tiles(args, w.p) + (size_t)w.hb * bytes;
                for (int i = 0; i < len; ++i, src += bytes) {
                    if (issued >= args.b_slots && !mbar_wait_long(b_empty + 8 * slot, prev_use, args.status, kTimeoutTensorPipe)) {
                        ok = false;
                        break;
                    }
                    mbar_expect_tx(b_full + 8 * slot, bytes);
                    bulk_load(smem_u32(b_ring + (size_t)slot * args.b_stride), src, bytes, b_full + 8 * slot);
                    ++issued;
                    if (++slot == args.b_slots) { slot = 0; prev_use ^= 1; }
                }
                w.next(args, len);
            }
            for (int i = (issued > args.b_slots ? issued - args.b_slots : 0); i < issued; ++i)
                mbar_wait(b_full + 8 * (i % args.b_slots), (uint32_t)(i / args.b_slots) & 1, args.status, kTimeoutDrain);
        }
    } else if (warp >= kWarpMma) {
        // ---- MMA issuers, a unit each in turn: the whole warp walks, an elected lane issues ---------
        const int me = warp - kWarpMma;
        if (me < issuers) {
            // K step k of a unit goes to accumulator `me` of two, or (four) 2 me + k % 2.
            const uint32_t mine_acc = me * (args.d_accs >> 1) * args.n_max, odd = args.d_accs == 4 ? args.n_max : 0;
            int next = me, slot = me, stage = me, seg = 0;  // of this warp's next unit
            uint32_t use = 0, a_use = 0;
            bool ok = true;
            for (Walk w(args, mine); w.unit < w.end && ok; ++seg) {
                const int len = w.length(args), n = wide_n(problem_rows(args, w.p)), start = w.unit - mine.begin;
                const uint32_t idesc = umma_idesc_f16_f32(128, n), dcol = tmem + d_column(seg) + mine_acc;
                // (Waited for without a unit in the segment too: the other issuer's commit of the buffer's segment
                // before must have come before this one's.)
                if (seg >= d_bufs && !mbar_wait_long(d_empty + 8 * d_index(seg), d_parity(seg) ^ 1, args.status, kTimeoutTensorPipe)) break;
                int part = PARTS ? part_of(args, w.hb) : 0, fresh = 1;
                for (; next < start + len; next += issuers) {
                    while (PARTS && part_begin(args, part + 1) <= w.hb + next - start) { ++part; fresh = 1; }
                    const uint32_t acc = dcol + part * args.d_accs * args.n_max;
                    if (!mbar_wait_long(b_full + 8 * slot, use, args.status, kTimeoutTensorPipe) ||
                        !mbar_wait_long(a_full + 8 * stage, a_use, args.status, kTimeoutTensorPipe)) {
                        ok = false;
                        break;
                    }
                    tc_fence_after_sync();
                    const uint32_t rows0 = smem_u32(b_ring) + slot * args.b_stride, acol = tmem + stage * 64;
                    const uint64_t b0 = umma_desc_k_major_sw128(rows0), b1 = umma_desc_k_major_sw128(rows0 + n * 128);
                    if (elect_one()) {
#pragma unroll
                        for (int k = 0; k < 8; ++k)
                            umma_f16_ts(acc + (k & 1) * odd, acol + 8 * k, (k < 4 ? b0 : b1) + 2 * (k & 3), idesc, !fresh || k > 1 || (k == 1 && !odd));
                        umma_commit(a_empty + 8 * stage);
                        umma_commit(b_empty + 8 * slot);
                    }
                    __syncwarp();
                    fresh = 0;
                    if ((slot += issuers) >= args.b_slots) { slot -= args.b_slots; use ^= 1; }
                    if ((stage += issuers) >= a_stages) { stage -= a_stages; a_use ^= 1; }
                }
                if (elect_one()) umma_commit(d_full + 8 * d_index(seg));
                w.next(args, len);
            }
            if (elect_one()) umma_commit(all_done);
        }
    } else if (warp >= kDecodeW) {
        // ---- epilogue group: every segment, all of it except the last, which the decoders share ----
        // Output scales and bias are cold in DRAM and needed at the very end: ask the L2 for them now.
        for (int b = mine.begin / args.hblocks + (warp & 3), e = (mine.end - 1) / args.hblocks; b <= e; b += kEpiW) {
            const int p = b / args.nblocks, nb = b - p * args.nblocks;
            const DeviceWeights& dw = problem(args, p).w;
            if (lane < 2) prefetch_line_l2(dw.svh + (size_t)nb * 128 + lane * 64);
            else if (lane < 6 && dw.bias) prefetch_line_l2(dw.bias + (size_t)nb * 128 + (lane - 2) * 32);
        }
        const Epilogue<PARTS> epi{args, cta, mine.begin, warp & 3, lane, 1, epi_stage, kStageFloats};
        int seg = 0;
        for (Walk w(args, mine); w.unit < w.end; ++seg) {
            const int len = w.length(args);
            const bool final = w.unit + len == w.end;
            const bool ok = mbar_wait_long(d_full + 8 * d_index(seg), d_parity(seg), args.status, kTimeoutTensorPipe);
            if (group_any(1, !ok)) break;
            tc_fence_after_sync();
            if (!epi.segment(split, w, len, tmem + d_column(seg), 0, final ? 1 + kDecodeW / 4 : 1, d_empty + 8 * d_index(seg))) break;
            w.next(args, len);
        }
    } else {
        // ---- decode warps ---------------------------------------------------------------------------
        const int turn = warp >> 2, ctile = 2 * (warp & 3);
        const uint32_t taddr = tmem + ((uint32_t)(ctile * 16) << 16);
        DecodeState s{turn, turn, 1, false, turn % args.w_slots, (uint32_t)(turn / args.w_slots) & 1};
        bool ok = true;
        int seg = 0, until = 0;
        Walk w(args, mine);
        while (true) {
            const int len = w.length(args);
            until += len;
            const int bits = problem(args, w.p).w.bits;
            ok = decode_segment_rate<CB, kUnitGroups>(bits, s, until, w_ring, args.w_slots, args.w_stride, w_full, w_empty, a_full, a_empty,
                                         taddr, a_stages, ctile, lane, args.status);
            if (!ok || until >= my_units) break;
            w.next(args, len);
            ++seg;
        }
        // The range is decoded: a quarter of these warps each is a group that takes its share of the
        // last segment's epilogue, with staging space in the idle weight ring.
        const int group = warp >> 2;
        // (Not d_full: these warps may be several segments ahead of the accumulators, where its parity
        // would already look like the last segment's.)
        if (ok) ok = mbar_wait_long(all_done, 0, args.status, kTimeoutTensorPipe);
        if (!group_any(2 + group, !ok)) {
            tc_fence_after_sync();
            const Epilogue<PARTS> epi{args, cta, mine.begin, warp & 3, lane, 2 + group, reinterpret_cast<float*>(w_ring) + group * kStageFloats, 0};
            epi.segment(split, w, w.length(args), tmem + d_column(seg), 1 + group, 1 + kDecodeW / 4, 0);
            tc_fence_before_sync();
        }
    }

    tc_fence_before_sync();
    __syncthreads();
    if (warp == kWarpMma) {
        __syncwarp();
        tc_fence_after_sync();
        tmem_dealloc(tmem, 512);
    }
}

// ---- input stages: four rows of one 128-block per warp, eight lanes per row --------------------
constexpr int kInputWarps = 4;
__global__ void __launch_bounds__(32 * kInputWarps) wide_inputs_kernel(const WideArgs args, int grid_ctas) {
    if (!args.table) pdl_launch_dependents();
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, l8 = lane & 7;
    const int first = blockIdx.x * kInputWarps + warp;
    uint2 su[4];
    if (!args.table) {
        // One layer: the scales are weights, and the activations may be asked for early (the L2 is
        // the point of coherence); both are there when the launch before ends.
        const int p = blockIdx.y, rows = problem_rows(args, p), quad = first / args.hblocks, blk = first - quad * args.hblocks;
        const int row = quad * 4 + (lane >> 3);
#pragma unroll
        for (int i = 0; i < 4; ++i)
            su[i] = __ldg(reinterpret_cast<const uint2*>(args.one.w.suh + blk * 128 + 32 * i + 4 * l8));
        const int row_bytes = args.one.x_dtype == DT_F32 ? 512 : 256;  // of this block
        if (row < rows && l8 * 128 < row_bytes)
            prefetch_line_l2(static_cast<const unsigned char*>(args.one.x) +
                             ((size_t)(p * args.group_rows + row) * args.one.x_stride + blk * 128) * (row_bytes / 128) + l8 * 128);
    }
    pdl_wait_prior_grid();  // x may come from the launch before; the tiles may still be read by it
    if (args.table) pdl_launch_dependents();  // not earlier: that launch reads the table at once
    if (blockIdx.x == 0 && blockIdx.y == 0)
        for (int i = threadIdx.x; i < grid_ctas; i += blockDim.x) args.flags[i] = 0;
    const int count = args.live ? *args.live : args.count;
    for (int p = blockIdx.y; p < count; p += gridDim.y) {
        const WideProblem& pr = problem(args, p);
        const int rows = problem_rows(args, p), quads = (rows + 3) / 4;
        const size_t tile_bytes = wide_tile_bytes(rows);
        unsigned char* tiles = const_cast<unsigned char*>(problem_tiles(args, p));
        const bool aligned = quads_aligned(pr.x, pr.x_dtype, pr.x_stride);
        for (int item = first; item < quads * args.hblocks; item += gridDim.x * kInputWarps) {
            const int quad = item / args.hblocks, blk = item - quad * args.hblocks;
            const int row = quad * 4 + (lane >> 3);
            const int x_row = row >= rows ? 0 : !args.table ? p * args.group_rows + row : pr.x_rows ? pr.x_rows[row] : row;
            float v[4][4];
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                v[i][0] = v[i][1] = v[i][2] = v[i][3] = 0.f;
                if (row < rows)
                    load_quad(pr.x, pr.x_dtype, (long long)x_row * pr.x_stride + blk * 128 + 32 * i + 4 * l8, aligned, v[i]);
            }
            if (args.table || item != first) {
#pragma unroll
                for (int i = 0; i < 4; ++i)
                    su[i] = __ldg(reinterpret_cast<const uint2*>(pr.w.suh + blk * 128 + 32 * i + 4 * l8));
            }
#pragma unroll
            for (int i = 0; i < 4; ++i) scale_quad(v[i], su[i]);
            hadamard128_oct(v, lane);
            unsigned char* tile = tiles + blk * tile_bytes + 8 * (l8 & 1);
#pragma unroll
            for (int i = 0; i < 4; ++i)
                *reinterpret_cast<uint2*>(tile + (i >> 1) * (tile_bytes / 2) + sw128_chunk(row, (i & 1) * 4 + (l8 >> 1))) =
                    make_uint2(as_u32(__floats2half2_rn(v[i][0], v[i][1])), as_u32(__floats2half2_rn(v[i][2], v[i][3])));
        }
    }
}

// ---- host side -----------------------------------------------------------------------------------
WidePlan plan_wide(int heaviest, int rows_max, long long units, int sm_count) {
    WidePlan plan{};
    plan.grid = (int)(units < sm_count ? units : sm_count);
    plan.n_max = wide_n(rows_max < kWideRows ? rows_max : kWideRows);
    plan.parts = 1;
    plan.w_stride = unit_bytes(heaviest);
    plan.w_slots = (64 * 1024) / plan.w_stride;
    if (plan.w_slots > kMaxWSlots) plan.w_slots = kMaxWSlots;
    while ((size_t)plan.w_slots * plan.w_stride < kRingMin) ++plan.w_slots;  // 1 and 1.5 bits per weight
    const size_t ring = (size_t)plan.w_slots * plan.w_stride;
    plan.b_stride = plan.n_max * 256;
    plan.b_slots = (int)((kSmemLimitW - 1024 - kHeaderW - ring) / plan.b_stride);
    if (plan.b_slots > kMaxBSlots) plan.b_slots = kMaxBSlots;
    plan.smem_bytes = 1024 + kHeaderW + ring + (size_t)plan.b_slots * plan.b_stride;
    plan.flag_bytes = align_up((size_t)sm_count * sizeof(unsigned int));
    plan.plane_bytes = align_up((size_t)plan.grid * plan.n_max * 128 * sizeof(float));
    return plan;
}

static WideArgs wide_args(const WideSet& set, const WidePlan& plan, unsigned int* flags, float* planes, unsigned int* status) {
    WideArgs a{};
    a.table = set.table;
    a.table_stride = set.table_stride;
    a.live = set.live;
    a.one = set.one;
    a.count = set.count;
    a.group_rows = set.group_rows;
    a.hblocks = set.inputs / 128;
    a.nblocks = set.outputs / 128;
    a.n_max = plan.n_max;
    a.w_slots = plan.w_slots;
    a.w_stride = plan.w_stride;
    a.b_slots = plan.b_slots;
    a.b_stride = plan.b_stride;
    // Even and odd K steps have accumulators of their own where there is room, half the truncating
    // accumulations in a row; calls of up to sixteen rows have four, as those of up to eight have (distance from the
    // sum in 64 bits, 16 rows of 5120 -> 5120: 8.4e-7 of its norm with two, 4.5e-7 with four, at
    // 15.75 us instead of 15.55).  Beyond 128 rows there is room for one (129 rows of 4096 -> 12288: 2.6e-6
    // where two give 1.4e-6 for 128), as in the dense GEMM (4.9e-6).  A second buffer lets the MMAs of
    // the next segment start under this one's epilogue.  Four A stages (one for each decode group) are
    // enough, half of the columns are the accumulators'.
    a.d_accs = plan.n_max <= 16 && !set.table ? 4 : plan.n_max <= 128 ? 2 : 1;
    a.parts = plan.parts;
    while (a.parts > 1 && a.parts * a.d_accs * plan.n_max > 256) a.parts /= 2;
    while ((1 << a.parts_log2) < a.parts) ++a.parts_log2;
    a.d_bufs = 2 * a.parts * a.d_accs * plan.n_max <= 256 ? 2 : 1;
    a.a_stages = (512 - a.d_bufs * a.parts * a.d_accs * plan.n_max) / 64;
    if (a.a_stages > kMaxAStages) a.a_stages = kMaxAStages;
    a.flags = flags;
    a.planes = planes;
    a.status = status;
    return a;
}

cudaError_t launch_wide_inputs(const WideSet& set, const WidePlan& plan, unsigned int* flags, bool programmatic,
                               cudaStream_t stream) {
    const WideArgs a = wide_args(set, plan, flags, nullptr, nullptr);
    // one item per warp as far as an SM's free registers beside wide_linear_kernel go
    const int per_problem = ((plan.n_max + 3) / 4 * (set.inputs / 128) + kInputWarps - 1) / kInputWarps;
    const int y = set.count < 1024 ? set.count : 1024;
    int x = streaming_grid((long long)per_problem * y, 8) / y;
    x = x < 1 ? 1 : x > per_problem ? per_problem : x;
    return launch_pdl(wide_inputs_kernel, dim3(x, y), 32 * kInputWarps, 0, programmatic, stream, a, plan.grid);
}

cudaError_t launch_wide(const WideSet& set, const WidePlan& plan, unsigned int* flags, float* planes, unsigned int* status,
                        bool programmatic, cudaStream_t stream) {
    const WideArgs a = wide_args(set, plan, flags, planes, status);
    const long long units = (long long)set.count * a.nblocks * a.hblocks;
    if (units < 1 || units > 0x7FFFFFFF || plan.b_slots < 1 || plan.w_slots < 2 || plan.smem_bytes > kSmemLimitW ||
        (size_t)plan.w_slots * plan.w_stride < kRingMin)
        return cudaErrorInvalidValue;
    return for_codebook(set.codebook, [&](auto cb) {
        return a.parts > 1 ? launch_pdl(wide_linear_kernel<decltype(cb)::value, true>, plan.grid, kThreadsW, plan.smem_bytes, programmatic, stream, a)
                           : launch_pdl(wide_linear_kernel<decltype(cb)::value, false>, plan.grid, kThreadsW, plan.smem_bytes, programmatic, stream, a);
    });
}

// Opt-in dynamic shared memory is a per-device function attribute: set when a context is created
// on a device (configure_device), never on the launch path.
template <int CB>
static cudaError_t configure_wide_cb() {
    const cudaError_t e = cudaFuncSetAttribute(wide_linear_kernel<CB, false>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSmemLimitW);
    if (e != cudaSuccess) return e;
    return cudaFuncSetAttribute(wide_linear_kernel<CB, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSmemLimitW);
}
cudaError_t configure_wide_kernels() {
    cudaError_t e = configure_wide_cb<CB_3INST>();
    if (e == cudaSuccess) e = configure_wide_cb<CB_MCG>();
    if (e == cudaSuccess) e = configure_wide_cb<CB_MUL1>();
    // The same shared-memory carve-out as the kernel that follows: an SM that has to change its split
    // between L1 and shared memory drains first, and nothing of the two launches overlaps.
    if (e == cudaSuccess) e = cudaFuncSetAttribute(wide_inputs_kernel, cudaFuncAttributePreferredSharedMemoryCarveout, cudaSharedmemCarveoutMaxShared);
    return e;
}

}  // namespace st
