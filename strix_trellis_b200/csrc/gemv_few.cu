// Fused linear of 2..8 activation rows on a layer of few units per CTA, where the launch's head and
// tail weigh more than its loop: input stages, trellis decode, tensor-core dot, split-K fold and
// output stages in one launch, the work split of gemv_row.cu.  Sixteen decode warps: warp (t, g) owns
// column tile t of the units of parity g; a decoded tile is the A operand of mma.sync.m16n8k16 (m =
// output column), the activation rows are the B operand (n = row).  An epilogue warp turns dumped
// accumulators into planes or outputs.  (src/gemv_lds.hip:93-167)
//
// Against gemv_tmem.cu, which serves the layers of more units: no tensor memory to allocate and no chain
// tensor memory -> commit -> transposition before the fold; both sides measured stand at kFewUnits.
//
// With at most kFewUnits units a CTA has a ring slot for each of them and a slot for the core input of
// each H128 block they touch: nothing is recycled and nothing waits for a slot.
//
// Fold: a column block shared by several CTAs is finished by the CTA that holds its FIRST K range, the
// end of its own.  The others publish planes word by word, a word being either "empty" (all ones, a
// NaN no sum produces) or a value; the finishing CTA polls them (bounded), adds them in ascending K
// order from +0, its own first (src/gemv_fused.hip:81-127), and marks them empty again.  Waits only
// point to higher CTA indices and all CTAs are resident (grid <= SM count).
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

constexpr int kFewHeader = 16384 + 512;          // two fold buffers, barriers
constexpr int kFewSmem = kFewHeader + kFewUnits * (unit_bytes(8) + 256 * 8);  // the most that a launch asks for

struct GemvArgs {
    LinearCall call;
    Split split;               // unit range of every CTA (units / grid, units % grid)
    float* partials;           // [grid][rows][128], every word empty on entry and on exit
};

}  // namespace

// One output row of one column block, by one warp: this CTA's own contribution (`own`, the
// two k-group planes of the shared-memory fold buffer) first, then the planes of CTAs
// first+1 .. last in ascending K order, each polled word by word until it is no longer empty
// (bounded) and marked empty again; then output H128, svh, bias, alpha, beta.
__device__ __forceinline__ void fold_row(const GemvArgs& args, const float* own, int r, int rows, int nb, int first,
                                         int last, int lane, const float (&sv)[4], const float (&bs)[4]) {
    const LinearCall& c = args.call;
    float v[4];
#pragma unroll
    for (int j = 0; j < 4; ++j)
        v[j] = __fadd_rn(0.f, __fadd_rn(own[r * 128 + lane + 32 * j], own[1024 + r * 128 + lane + 32 * j]));
    for (int p0 = first + 1; p0 <= last; p0 += 8) {  // eight planes in flight
        uint32_t t[8][4];
        bool have = false;
        for (uint32_t tries = 0; tries < (1u << 18) && !have; ++tries) {
            bool all = true;
#pragma unroll
            for (int q = 0; q < 8; ++q) {
                const uint32_t* src =
                    reinterpret_cast<const uint32_t*>(args.partials) + ((size_t)(p0 + q) * rows + r) * 128 + lane;
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    t[q][j] = p0 + q <= last ? ld_relaxed_gpu(src + 32 * j) : 0u;
                    all = all && t[q][j] != kEmptyWord;
                }
            }
            have = __all_sync(0xFFFFFFFFu, all);
        }
        if (!have) {  // bounded: report and leave this row unwritten
            if (lane == 0) atomicOr(c.status, kTimeoutFold);
            return;
        }
#pragma unroll
        for (int q = 0; q < 8; ++q) {
            if (p0 + q <= last) {
                uint32_t* src = reinterpret_cast<uint32_t*>(args.partials) + ((size_t)(p0 + q) * rows + r) * 128 + lane;
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    v[j] = __fadd_rn(v[j], __uint_as_float(t[q][j]));
                    st_relaxed_gpu(src + 32 * j, kEmptyWord);  // empty again for the next launch
                }
            }
        }
    }
    hadamard128_warp(v, lane);
#pragma unroll
    for (int j = 0; j < 4; ++j) {
        float value = __fmul_rn(v[j], sv[j]);
        if (c.w.bias) value = __fadd_rn(value, bs[j]);
        scale_and_store(c.y, c.y_dtype, (long long)r * c.y_stride + nb * 128 + lane + 32 * j, value, c.alpha, c.beta);
    }
}

template <int K, int CB>
__global__ void __launch_bounds__(kThreads, 1) gemv_few_kernel(const GemvArgs args) {
    extern __shared__ __align__(128) unsigned char smem[];
    const LinearCall& c = args.call;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int rows = c.rows;
    const int hblocks = c.w.inputs / 128;
    const int cta = (int)blockIdx.x;
    const Range mine = cta_range(args.split, cta);
    const int my_units = mine.end - mine.begin;
    constexpr int kStage = unit_bytes(K);

    // shared memory: [2 x fold 8 KB][barriers 512 B][ring][core input]
    float* fold_base = reinterpret_cast<float*>(smem);
    uint64_t* bars = reinterpret_cast<uint64_t*>(smem + 16384);
    unsigned char* ring = smem + 16384 + 512;
    uint2* act = reinterpret_cast<uint2*>(ring + (size_t)my_units * kStage);

    const uint32_t full0 = smem_u32(bars);
    if ((int)threadIdx.x < my_units) {  // one thread per ring slot
        mbar_init(full0 + 8 * threadIdx.x, 1);
        mbar_fence_init();
    }
    __syncthreads();
    pdl_launch_dependents();

    if (warp == kConsumers) {
        // ---- producer: weights are immutable, so this needs no wait on the prior grid ----
        if (lane == 0) {
            const unsigned char* stream =
                reinterpret_cast<const unsigned char*>(c.w.packed) + (size_t)mine.begin * kStage;
            for (int i = 0; i < my_units; ++i) {
                mbar_expect_tx(full0 + 8 * i, kStage);
                bulk_load(smem_u32(ring + (size_t)i * kStage), stream + (size_t)i * kStage, kStage, full0 + 8 * i);
            }
            // Never leave the CTA with a copy still landing in its shared memory.
            for (int i = 0; i < my_units; ++i) mbar_wait(full0 + 8 * i, 0, c.status, kTimeoutDrain);
        }
        return;
    }

    // Segment walk shared by decode and epilogue warps: the CTA's unit range is cut at
    // column-block ends, where a contribution is flushed.
    // Each warp calls it once per segment, in order; the position is carried, not divided out.
    int walk_nb = mine.begin / hblocks, walk_hb0 = mine.begin - walk_nb * hblocks;
    auto segment = [&](int done, int& nb, int& hb0, int& len) {
        nb = walk_nb;
        hb0 = walk_hb0;
        len = my_units - done;
        if (len > hblocks - hb0) len = hblocks - hb0;
        walk_hb0 += len;
        if (walk_hb0 == hblocks) { walk_hb0 = 0; ++walk_nb; }
    };

    if (warp == kConsumers + 1) {
        // ---- epilogue warp: turns dumped accumulators into partial planes or outputs ------
        // Everything a flush needs that does not depend on the accumulators (contributor
        // range, output scales, bias) is resolved BEFORE the wait for the dump, while the
        // decode warps are still busy; after the dump the critical path is one plane write for
        // a contributor and, for the folding CTA, the wait for the others' plane words.
        pdl_wait_prior_grid();  // y and scratch may belong to the prior grid
        int done = 0, flush = 0;
        while (done < my_units) {
            int nb, hb0, len;
            segment(done, nb, hb0, len);
            done += len;
            const int buf = flush & 1;
            const int blk_lo = nb * hblocks, blk_hi = blk_lo + hblocks;
            const bool whole = mine.begin <= blk_lo && mine.end >= blk_hi;
            int first = cta, last = cta;
            if (!whole) contributors(args.split, blk_lo, blk_hi, first, last);
            float sv[4], bs[4];
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const int cidx = nb * 128 + lane + 32 * j;
                sv[j] = half_bits_to_float(c.w.svh[cidx]);
                bs[j] = c.w.bias ? c.w.bias[cidx] : 0.0f;
            }
            // A CTA publishes at most one plane per launch: for the block its range begins inside.
            uint32_t* plane = reinterpret_cast<uint32_t*>(args.partials) + (size_t)cta * rows * 128;

            named_barrier(2 + buf, kDumpThreads);  // all decode warps have dumped into `buf`
            const float* f0 = fold_base + buf * 2048;
            if (!whole && cta != first) {
                // contributor: publish the plane word by word (k-groups in ascending order); a
                // real sum never has the empty pattern (an all-ones NaN), so no flag and no fence
                for (int e = lane; e < rows * 128; e += 32)
                    st_relaxed_gpu(plane + e, __float_as_uint(__fadd_rn(f0[e], f0[1024 + e])));
            } else {
                // The block is finished here: it lies inside this CTA's range, or this CTA holds
                // its FIRST K range -- the end of its own unit range, so every other contributor
                // finishes at about the same time or earlier.  With several rows and planes to
                // wait for, the decode warps (idle by then) fold one row each instead.
                if (whole) {
                    for (int r = 0; r < rows; ++r) fold_row(args, f0, r, rows, nb, first, last, lane, sv, bs);
                }
            }
            // hand the buffer back (decode warps wait on this before its next reuse)
            asm volatile("bar.arrive %0, %1;" ::"r"(4 + buf), "r"(kDumpThreads) : "memory");
            ++flush;
        }
        return;
    }

    // ---- decode warps -------------------------------------------------------------------
    // Every H128 block this CTA's range touches is staged exactly once, before the loop starts: the block of
    // unit u in slot u % hblocks.
    // The input scales of a warp's first block are weights (immutable): they are fetched
    // before the wait on the prior grid, so only the activation load follows it.
    const int need = my_units < hblocks ? my_units : hblocks;
    const int hb_first = walk_hb0;
    uint16_t su_first[4] = {0, 0, 0, 0};
    if (warp < rows * need) {
        int hb = hb_first + warp % need;
        if (hb >= hblocks) hb -= hblocks;
#pragma unroll
        for (int j = 0; j < 4; ++j) su_first[j] = c.w.suh[(size_t)hb * 128 + lane + 32 * j];
    }
    pdl_wait_prior_grid();  // x may belong to the prior grid
    const int ctile = warp & 7, kgroup = warp >> 3;
    const LaneGeom<K> geom(lane);
    // Row fed by this lane as the B operand.  Rows >= `rows` only reach accumulator
    // columns that are never read, so those lanes may load any valid row.
    const int brow = (lane >> 2) < rows ? (lane >> 2) : rows - 1;
    const uint2* act_lane = act + brow * 32 + (lane & 3);
    __half* act_h = reinterpret_cast<__half*>(act);
    const int col = ctile * 16 + (lane >> 2), r0 = 2 * (lane & 3);

    // (row, H128 block) items through the input stages, written in B-fragment order:
    // act[((slot*rows + r)*8 + kt)*4 + q] = {half2(k0,k0+1), half2(k0+8,k0+9)}, k0 = 2q.
    // A warp keeps its (at most two) items in flight so that their global loads overlap.
    {
        constexpr int kItems = kFewUnits * 8 / kConsumers;
        float xv[kItems][4];
        uint16_t sc[kItems][4];
        int rr[kItems], ss[kItems];
#pragma unroll
        for (int u = 0; u < kItems; ++u) {
            const int item = warp + u * kConsumers;
            if (item < rows * need) {
                rr[u] = item / need;
                ss[u] = item % need;
                int hb = hb_first + ss[u];
                if (hb >= hblocks) hb -= hblocks;
                const long long xr = (long long)rr[u] * c.x_stride + (long long)hb * 128;
                const uint16_t* su = c.w.suh + (size_t)hb * 128;
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    xv[u][j] = load_element(c.x, c.x_dtype, xr + lane + 32 * j);
                    sc[u][j] = u == 0 ? su_first[j] : su[lane + 32 * j];
                }
            }
        }
#pragma unroll
        for (int u = 0; u < kItems; ++u) {
            if (warp + u * kConsumers < rows * need) {
                float v[4];
#pragma unroll
                for (int j = 0; j < 4; ++j) v[j] = __half2float(scale_input(xv[u][j], sc[u][j]));
                hadamard128_warp(v, lane);
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    const int e = lane + 32 * j, kt = e >> 4, kk = e & 15;
                    const int q = (kk & 7) >> 1, hi = kk >> 3, lo = kk & 1;
                    act_h[((((size_t)ss[u] * rows + rr[u]) * 8 + kt) * 4 + q) * 4 + hi * 2 + lo] = __float2half_rn(v[j]);
                }
            }
        }
        named_barrier(1, kConsumers * 32);
    }

    float acc[2][4] = {{0.f, 0.f, 0.f, 0.f}, {0.f, 0.f, 0.f, 0.f}};
    bool ok = true;
    int done = 0, flush = 0, final_nb = 0;
    int next = kgroup;  // the unit (relative to the range) this warp decodes next, and the slot of its block
    int slot = kgroup;
    while (slot >= need) slot -= need;
    while (done < my_units) {
        int nb, hb0, len;
        segment(done, nb, hb0, len);

        // this warp group takes the units of its parity
        for (; next < done + len && ok; next += 2) {
            ok = mbar_wait(full0 + 8 * next, 0, c.status, kTimeoutRingFull);
            if (!ok) break;
            __syncwarp();
            const uint32_t* tiles =
                reinterpret_cast<const uint32_t*>(ring + (size_t)next * kStage) + ctile * quad_words(K);
            const uint2* bsrc = act_lane + (size_t)slot * rows * 32;
            slot += 2;
            while (slot >= need) slot -= need;
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
        }
        done += len;

        // ---- drop this CTA's contribution to column block nb and move on --------------------
        // c0,c1: column ctile*16 + lane/4, rows 2(lane%4), +1; c2,c3: column + 8
        const int buf = flush & 1;
        if (flush >= 2) named_barrier(4 + buf, kDumpThreads);  // epilogue is done with `buf`
        {
            float* g = fold_base + buf * 2048 + kgroup * 1024;
            const float v00 = acc[0][0] + acc[1][0], v01 = acc[0][1] + acc[1][1];
            const float v10 = acc[0][2] + acc[1][2], v11 = acc[0][3] + acc[1][3];
            if (r0 < rows) { g[r0 * 128 + col] = v00; g[r0 * 128 + col + 8] = v10; }
            if (r0 + 1 < rows) { g[(r0 + 1) * 128 + col] = v01; g[(r0 + 1) * 128 + col + 8] = v11; }
#pragma unroll
            for (int j = 0; j < 4; ++j) acc[0][j] = acc[1][j] = 0.f;
        }
        asm volatile("bar.arrive %0, %1;" ::"r"(2 + buf), "r"(kDumpThreads) : "memory");
        ++flush;
        final_nb = nb;
    }

    // ---- several rows: the decode warps finish the CTA's last, shared column block ----------
    // If this CTA folds that block (it holds the block's first K range, other CTAs hold the
    // rest), warp r folds row r -- eight rows wait for their planes side by side instead of one
    // after the other in the epilogue warp.  Every decode warp reaches the barrier, whatever
    // its own waits returned, so it cannot be left short of arrivals.
    if (my_units > 0) {
        const int blk_lo = final_nb * hblocks, blk_hi = blk_lo + hblocks;
        if (!(mine.begin <= blk_lo && mine.end >= blk_hi)) {
            int first, last;
            contributors(args.split, blk_lo, blk_hi, first, last);
            if (cta == first) {
                named_barrier(1, kConsumers * 32);  // every decode warp has dumped its accumulators
                if (ok && warp < rows) {
                    float sv[4], bs[4];
#pragma unroll
                    for (int j = 0; j < 4; ++j) {
                        const int cidx = final_nb * 128 + lane + 32 * j;
                        sv[j] = half_bits_to_float(c.w.svh[cidx]);
                        bs[j] = c.w.bias ? c.w.bias[cidx] : 0.0f;
                    }
                    fold_row(args, fold_base + ((flush - 1) & 1) * 2048, warp, rows, final_nb, first, last, lane, sv, bs);
                }
            }
        }
    }
}

// ---- host side -------------------------------------------------------------------------
void plan_gemv_few(const DeviceWeights& w, int rows, int units_per_cta, GemvPlan& plan) {
    plan.stages = units_per_cta;
    plan.act_blocks = units_per_cta < w.inputs / 128 ? units_per_cta : w.inputs / 128;
    plan.smem_bytes = kFewHeader + (size_t)plan.stages * unit_bytes(w.bits) + (size_t)plan.act_blocks * 256 * rows;
}

cudaError_t launch_gemv_few(const LinearCall& call, const GemvPlan& plan, Split split, float* planes, bool pdl, cudaStream_t stream) {
    if (split.q + (split.r != 0) > kFewUnits) return cudaErrorInvalidValue;
    const GemvArgs args{call, split, planes};
    return for_codebook(call.w.codebook, [&](auto cb) {
        return for_rate<decltype(cb)::value>(call.w.bits, [&](auto k) {
            return launch_pdl(gemv_few_kernel<decltype(k)::value, decltype(cb)::value>, plan.grid, kThreads, plan.smem_bytes, pdl, stream, args);
        });
    });
}

// Opt-in dynamic shared memory is a per-device function attribute: set for every instantiation
// when a context is created on a device (configure_device), never on the launch path.
template <int CB>
static cudaError_t configure_few() {
    cudaError_t e = cudaSuccess;
    for (int bits = 1; bits <= (CB == CB_MUL1 ? kRateCodes : 8) && e == cudaSuccess; ++bits)
        e = for_rate<CB>(bits, [&](auto k) {
            return cudaFuncSetAttribute(gemv_few_kernel<decltype(k)::value, CB>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                        kFewSmem);
        });
    return e;
}
cudaError_t configure_gemv_few_kernels() {
    cudaError_t e = configure_few<CB_3INST>();
    if (e == cudaSuccess) e = configure_few<CB_MCG>();
    if (e == cudaSuccess) e = configure_few<CB_MUL1>();
    return e;
}

}  // namespace st
