// Fused linear of 1..8 activation rows in ONE launch: input stages, trellis decode, tensor-core
// dot, split-K fold, output H128, svh, bias and alpha/beta.  It stands in for the reference's
// input_transform + gemv_lds_kernel + output_transform sequence (src/backend.hip:102-151,
// src/gemv_lds.hip:93-167, src/transforms.hpp:8-52).
//
// Bound by the decode's issue slots (tmem_decode.cuh), then by the fixed time around the loop.
// The work split is that of wide_linear.cu: units of (128-column block) x (H128 block of K) in
// column-block-major order, one persistent CTA per SM with a contiguous range of them, weights
// streamed through a ring by 1-D bulk copies, tiles decoded into tensor memory, one MMA with N = 16
// per 16 inputs.  Here the activation operand is made by the CTA itself, in shared memory: eight
// helper warps run the input stages of the blocks its range touches while the decode warps are
// already at work (weights are immutable, so they do not wait for the previous kernel; only the
// MMAs wait for the activations, and the decode is up to six units ahead of them).
//
// Fold: a column block that several CTAs share is finished by the CTA that holds its FIRST K range
// (the end of its own range).  The others publish their sums word by word in global planes, where
// a word is either "empty" (all ones, a NaN no sum produces) or a value: no flag, no fence, no
// atomic.  A thread of the finishing CTA polls the very words it needs (bounded), adds them in
// ascending K order from +0, its own first (the reference's order, src/gemv_fused.hip:81-127), and
// marks them empty again for the next launch.  Waits only point to higher CTA indices and all CTAs
// are resident (grid <= SM count).  (Folding in a small second launch instead, so that no CTA waits
// for another, measured 2.6 us per layer slower: the extra launch boundary costs more.)
//
// Measured in a chain of launches against the kernel before, which fed mma.sync and staged its rows
// four 2-byte stores at a time: 16 layers, four rows, K2..K6 226 -> 179 us (four of them small ones in
// gemv_few.cu); 16384 -> 4096, eight rows, K5 29.6 -> 22.0 us; 4096 -> 129280, one row, K5 133 -> 118 us.  With two MMA
// issuers, tiles in quads and the decoder balanced between the pipes 171, 21.1 and 113 us.
#include <type_traits>

#include "gemv_kernels.h"
#include "hadamard.cuh"
#include "launch.h"
#include "tmem_decode.cuh"

namespace st {

namespace {
constexpr int kUnitGroups = 4, kDecodeT = 4 * kUnitGroups, kHelpersT = 8;
constexpr int kWarpMmaT = kDecodeT + kHelpersT, kWarpWeightsT = kWarpMmaT + kIssuers;
constexpr int kThreadsT = (kWarpWeightsT + 1) * 32;
constexpr int kRowsT = 16;                       // the MMA's N: the smallest it has; rows beyond the call's are never read
constexpr int kMaxRowsT = 8;
// A column is summed in four chains (parity of the unit, parity of the K step), each with an accumulator
// of its own, twice for the segments in turn: 128 of the 512 columns, the other 384 are six A stages.  The
// tensor cores truncate as they accumulate, so the error of a chain grows with the 1.5th power of its
// steps.  Distance from the sum in 64 bits, one chain and four, of the result's norm: 4096 -> 129280, one
// row 4.8e-6 and 1.2e-6; 16384 -> 4096, eight rows 4.0e-6 and 1.0e-6; 5120 -> 5120, four rows 1.6e-6 and
// 4.5e-7.  Four take 119.2 us instead of 118.0 for the first of these and 22.0 instead of 21.65 for the second.
constexpr int kChains = 4, kAStagesT = 6;
static_assert(kAStagesT * 64 + 2 * kChains * kRowsT <= 512 && kAStagesT >= kUnitGroups && kAStagesT <= kMaxAStages, "tensor memory");
// Activation operand of one H128 block: eight rows of both K = 64 halves.  The MMA's rows 8 to 15 are whatever
// lies behind (the other half, the next slot, the weight ring): columns of the sums that nobody reads.  With room
// for sixteen rows a layer of 4096 inputs left the weight ring 80 KB, too little for the trip to DRAM.
constexpr int kSlotBytesT = kMaxRowsT * 256;
constexpr int kStageFloats = kMaxRowsT * 128;    // transposition space of one helper group
constexpr int kMaxWSlotsT = 32, kMaxBSlotsT = 80;
constexpr int kHeaderT = 2048 + 2 * kStageFloats * 4;
constexpr size_t kSmemLimitT = 224 * 1024;
constexpr uint32_t kEmptyWord = 0xFFFFFFFFu;      // a plane word nobody has written yet
constexpr int kMinBRing = 4 * kHelpersT;          // units of one staging step of one row
static_assert((2 * kMaxWSlotsT + 2 * kMaxBSlotsT + 2 * kAStagesT + 4) * 8 <= 2048, "barriers fit the header");

struct TmemArgs {
    LinearCall call;
    Split split;
    int w_slots, b_slots;
    uint32_t row_magic;  // 2^32 / rows rounded up: high word of e * row_magic is e / rows for e < 2^28
    float* planes;       // [grid][rows][128], every word empty on entry and on exit
};
}  // namespace

template <int CB>
__global__ void __launch_bounds__(kThreadsT, 1) gemv_tmem_kernel(const TmemArgs args) {
    extern __shared__ __align__(1024) unsigned char smem_raw[];
    unsigned char* smem = smem_raw + (-smem_u32(smem_raw) & 1023u);  // (still a shared-memory pointer to the compiler)
    const LinearCall& c = args.call;
    const int warp = uniform_warp(), lane = threadIdx.x & 31, cta = (int)blockIdx.x;
    const int hblocks = c.w.inputs / 128, rows = c.rows;
    const Range mine = cta_range(args.split, cta);
    const int my_units = mine.end - mine.begin;
    const int w_stride = unit_bytes(c.w.bits);

    uint64_t* bars = reinterpret_cast<uint64_t*>(smem);
    unsigned char* b_ring = smem + kHeaderT;  // 1024-byte aligned operand images
    unsigned char* w_ring = b_ring + (size_t)args.b_slots * kSlotBytesT;
    __shared__ uint32_t s_tmem_base;
    const uint32_t w_full = smem_u32(bars), w_empty = w_full + 8 * kMaxWSlotsT, b_full = w_empty + 8 * kMaxWSlotsT,
                   b_empty = b_full + 8 * kMaxBSlotsT, a_full = b_empty + 8 * kMaxBSlotsT, a_empty = a_full + 8 * kAStagesT,
                   d_full = a_empty + 8 * kAStagesT, d_empty = d_full + 16;

    // The activation operand is staged per H128 block.  `resident`: every block the range touches has
    // a slot of its own and is staged once; else the slots are a ring in unit order.
    const int need = my_units < hblocks ? my_units : hblocks;
    const bool resident = need <= args.b_slots;
    const int first_nb = mine.begin / hblocks, first_hb = mine.begin - first_nb * hblocks;
    // Helper warps work on (block, row) elements, block-major, four per warp and step, eight lanes each.
    const int h = warp - kDecodeT, group = h >> 2, quarter = warp & 3, l8 = lane & 7, e8 = lane >> 3;
    auto unit_of = [&](int e) { return rows == 1 ? e : (int)__umulhi((uint32_t)e, args.row_magic); };  // e / rows
    auto block_of = [&](int unit) {
        int hb = first_hb + unit;
        return resident ? (hb >= hblocks ? hb - hblocks : hb) : hb % hblocks;
    };
    const int total = (resident ? need : my_units) * rows;
    uint2 su[4];  // input scales of this lane's next sixteen inputs
    auto load_scales = [&](int e) {
        const int hb = e < total ? block_of(unit_of(e)) : first_hb;
#pragma unroll
        for (int i = 0; i < 4; ++i)
            su[i] = __ldg(reinterpret_cast<const uint2*>(c.w.suh + (size_t)hb * 128 + 32 * i + 4 * l8));
    };

    // Everything that hides a DRAM round trip starts before the CTA's first barrier.  Of the weights
    // only kFirstUnits: all CTAs start together, and a whole ring requested at once would put
    // microseconds of other units before a CTA's first.
    constexpr int kFirstUnits = 2;
    const int first = args.w_slots < kFirstUnits ? args.w_slots : kFirstUnits;
    auto load_unit = [&](int unit, int slot) {
        mbar_expect_tx(w_full + 8 * slot, w_stride);
        bulk_load(smem_u32(w_ring) + slot * w_stride,
                  reinterpret_cast<const unsigned char*>(c.w.packed) + (size_t)(mine.begin + unit) * w_stride, w_stride, w_full + 8 * slot);
    };
    if (warp == kWarpWeightsT) {
        if (lane < args.w_slots) { mbar_init(w_full + 8 * lane, 1); mbar_init(w_empty + 8 * lane, 4); }
        mbar_fence_init();
        __syncwarp();
        if (lane == 0)
            for (int i = 0; i < first && i < my_units; ++i) load_unit(i, i);
    } else if (warp == kWarpMmaT) {
        tmem_alloc(smem_u32(&s_tmem_base), 512);
    } else if (warp >= kDecodeT && warp < kWarpMmaT) {
        // Scales of the first elements; the activations may be asked for early too (the L2 is the point
        // of coherence, so a line the previous kernel still writes is read correctly afterwards).
        load_scales(4 * h + e8);
        const int x_bytes = c.x_dtype == DT_F32 ? 4 : 2;
        for (int e = 4 * h + e8; e < need * rows; e += 4 * kHelpersT) {
            const int unit = unit_of(e), row = e - unit * rows;
            int hb = first_hb + unit;
            if (hb >= hblocks) hb -= hblocks;
            if (l8 < x_bytes)
                prefetch_line_l2(reinterpret_cast<const unsigned char*>(c.x) + ((size_t)row * c.x_stride + (size_t)hb * 128) * x_bytes + l8 * 128);
        }
    } else {  // one decode thread per barrier (and the second issuer, which has none)
        const int t = threadIdx.x;
        if (t < args.b_slots) { mbar_init(b_full + 8 * t, rows); mbar_init(b_empty + 8 * t, 1); }
        if (t < kAStagesT) { mbar_init(a_full + 8 * t, 4); mbar_init(a_empty + 8 * t, 1); }
        if (t < 2) { mbar_init(d_full + 8 * t, kIssuers); mbar_init(d_empty + 8 * t, 4); }
        mbar_fence_init();
    }
    tc_fence_before_sync();
    __syncthreads();
    tc_fence_after_sync();
    const uint32_t tmem = s_tmem_base, d_col = kAStagesT * 64;
    pdl_launch_dependents();

    if (warp == kWarpWeightsT) {
        // ---- weight producer: immutable, no wait on the launch before; the first units are on their way ----
        if (lane == 0) {
            int issued = my_units < first ? my_units : first;
            int slot = issued == args.w_slots ? 0 : issued;
            uint32_t prev_use = issued == args.w_slots ? 0 : 1;
            for (; issued < my_units; ++issued) {
                if (issued >= args.w_slots && !mbar_wait_long(w_empty + 8 * slot, prev_use, c.status, kTimeoutRingEmpty)) break;
                load_unit(issued, slot);
                if (++slot == args.w_slots) { slot = 0; prev_use ^= 1; }
            }
            for (int i = (issued > args.w_slots ? issued - args.w_slots : 0); i < issued; ++i)  // nothing still landing at exit
                mbar_wait(w_full + 8 * (i % args.w_slots), (uint32_t)(i / args.w_slots) & 1, c.status, kTimeoutDrain);
        }
    } else if (warp >= kWarpMmaT) {
        // ---- MMA issuers, a unit each in turn: the whole warp walks, an elected lane issues ---------
        constexpr uint32_t idesc = umma_idesc_f16_f32(128, kRowsT);
        const uint64_t b_desc = umma_desc_k_major_sw128(smem_u32(b_ring));
        const int me = warp - kWarpMmaT, b_wrap = resident ? hblocks : args.b_slots;
        int next = me, slot = me % b_wrap, stage = me, seg = 0;  // of this warp's next unit
        uint32_t use = 0, a_use = 0;
        bool ok = true;
        for (int done = 0, hb = first_hb; done < my_units && ok; ++seg, hb = 0) {
            const int left = my_units - done, len = left < hblocks - hb ? left : hblocks - hb;
            const uint32_t acc = tmem + d_col + ((seg & 1) * kChains + me * (kChains / kIssuers)) * kRowsT;
            // (Waited for without a unit in the segment too: the other issuer's commit of the segment two back
            // must have come before this one's.)
            if (seg >= 2 && !mbar_wait_long(d_empty + 8 * (seg & 1), (uint32_t)((seg >> 1) - 1) & 1, c.status, kTimeoutTensorPipe)) break;
            for (bool fresh = true; next < done + len; next += kIssuers, fresh = false) {
                if (!mbar_wait_long(b_full + 8 * slot, use, c.status, kTimeoutTensorPipe) ||
                    !mbar_wait_long(a_full + 8 * stage, a_use, c.status, kTimeoutTensorPipe)) {
                    ok = false;
                    break;
                }
                tc_fence_after_sync();
                const uint64_t b0 = b_desc + (uint32_t)(slot * (kSlotBytesT / 16));  // 16-byte units
                const uint32_t acol = tmem + stage * 64;
                if (elect_one()) {
#pragma unroll
                    for (int k = 0; k < 8; ++k)
                        umma_f16_ts(acc + (k & 1) * kRowsT, acol + 8 * k, b0 + (k < 4 ? 0 : kSlotBytesT / 32) + 2 * (k & 3), idesc, !fresh || k > 1);
                    umma_commit(a_empty + 8 * stage);
                    if (!resident) umma_commit(b_empty + 8 * slot);
                }
                __syncwarp();
                for (slot += kIssuers; slot >= b_wrap; slot -= b_wrap)
                    if (!resident) use ^= 1;  // a resident slot is filled once
                if ((stage += kIssuers) >= kAStagesT) { stage -= kAStagesT; a_use ^= 1; }
            }
            if (elect_one()) umma_commit(d_full + 8 * (seg & 1));
            done += len;
        }
    } else if (warp < kDecodeT) {
        // ---- decode warps ---------------------------------------------------------------------------
        const int turn = warp >> 2, ctile = 2 * (warp & 3);
        DecodeState s{turn, turn, 1, false, turn % args.w_slots, (uint32_t)(turn / args.w_slots) & 1};
        decode_segment_rate<CB, kUnitGroups, false>(c.w.bits, s, my_units, w_ring, args.w_slots, w_stride, w_full, w_empty, a_full, a_empty,
                                             tmem + ((uint32_t)(ctile * 16) << 16), kAStagesT, ctile, lane, c.status);
    } else {
        // ---- helper warps: input stages, then the epilogue of every other segment ---------------------
        const bool x_aligned = quads_aligned(c.x, c.x_dtype, c.x_stride);
        // Elements [begin, end) through the input stages.
        auto stage_elements = [&](int begin, int end) {
            for (int base = begin; base < end; base += 4 * kHelpersT) {
                if (resident && base + 4 * h >= end) break;
                const int e = base + 4 * h + e8;
                const bool live = e < end;
                const int unit = live ? unit_of(e) : 0, row = live ? e - unit * rows : 0, hb = block_of(unit);
                float v[4][4];
#pragma unroll
                for (int i = 0; i < 4; ++i)
                    load_quad(c.x, c.x_dtype, (long long)row * c.x_stride + (long long)hb * 128 + 32 * i + 4 * l8, x_aligned, v[i]);
                if (base) load_scales(e);
#pragma unroll
                for (int i = 0; i < 4; ++i) scale_quad(v[i], su[i]);
                hadamard128_oct(v, lane);
                const int slot = resident ? unit : unit % args.b_slots;
                // Ring slots: the helpers keep step, and a step has no more units than the ring has slots, so
                // the slot's previous use was staged in an earlier step and its parity is unambiguous.
                if (!resident) named_barrier(3, kHelpersT * 32);
                if (live && !resident && unit >= args.b_slots)
                    mbar_wait(b_empty + 8 * slot, (uint32_t)(unit / args.b_slots - 1) & 1, c.status, kTimeoutTensorPipe);
                unsigned char* tile = b_ring + (size_t)slot * kSlotBytesT + 8 * (l8 & 1);
                if (live) {
#pragma unroll
                    for (int i = 0; i < 4; ++i)
                        *reinterpret_cast<uint2*>(tile + (i >> 1) * (kSlotBytesT / 2) + sw128_chunk(row, (i & 1) * 4 + (l8 >> 1))) =
                            make_uint2(as_u32(__floats2half2_rn(v[i][0], v[i][1])), as_u32(__floats2half2_rn(v[i][2], v[i][3])));
                }
                fence_async_smem();  // the MMA reads through the async proxy
                __syncwarp();
                if (live && l8 == 0) mbar_arrive(b_full + 8 * slot);
            }
        };
        pdl_wait_prior_grid();  // x, y and the planes may belong to the launch before
        if (resident) stage_elements(0, total);
        // Output scales and bias of the range's column blocks are cold in DRAM and needed at the very
        // end: ask the L2 for them now.
        for (int nb = first_nb + h, last = (mine.end - 1) / hblocks; nb <= last; nb += kHelpersT) {
            if (lane < 2) prefetch_line_l2(c.w.svh + (size_t)nb * 128 + lane * 64);
            else if (lane < 6 && c.w.bias) prefetch_line_l2(c.w.bias + (size_t)nb * 128 + (lane - 2) * 32);
        }

        float* stage = reinterpret_cast<float*>(smem + 2048) + group * kStageFloats;
        auto epilogue = [&](int seg, int nb, int hb0, int len, int start) {
            const int c0 = nb * 128 + 4 * l8;
            const bool contributor = hb0 != 0;
            int last = cta;
            if (!contributor && len < hblocks) last = owner(args.split, (nb + 1) * hblocks - 1);
            bool good = mbar_wait_long(d_full + 8 * (seg & 1), (uint32_t)(seg >> 1) & 1, c.status, kTimeoutTensorPipe);
            __syncwarp();
            tc_fence_after_sync();
            const uint32_t at = tmem + ((uint32_t)(quarter * 32) << 16) + d_col + (seg & 1) * kChains * kRowsT;
            float v[kMaxRowsT];
            uint32_t r[2][kMaxRowsT];
#pragma unroll
            for (int j = 0; j < kMaxRowsT; ++j) v[j] = 0.f;
#pragma unroll
            for (int pair = 0; pair < kIssuers; ++pair) {  // the chains of one issuer, then of the other: both if there are two units
                if (len < 2 && pair != (start & 1)) continue;
                tmem_ld_32x8(at + pair * 2 * kRowsT, r[0]);
                tmem_ld_32x8(at + pair * 2 * kRowsT + kRowsT, r[1]);
                tmem_ld_wait();
#pragma unroll
                for (int j = 0; j < kMaxRowsT; ++j) {
                    asm volatile("" : "+r"(r[0][j]), "+r"(r[1][j]));  // not before the wait
                    v[j] = __fadd_rn(v[j], __fadd_rn(__uint_as_float(r[0][j]), __uint_as_float(r[1][j])));
                }
            }
            tc_fence_before_sync();
            __syncwarp();
            if (lane == 0) mbar_arrive(d_empty + 8 * (seg & 1));
            const int col = quarter * 32 + lane;
            uint32_t* words = reinterpret_cast<uint32_t*>(args.planes) + col;
            if (contributor) {
                if (good) {
#pragma unroll
                    for (int j = 0; j < kMaxRowsT; ++j)
                        if (j < rows) st_relaxed_gpu(words + ((size_t)cta * rows + j) * 128, __float_as_uint(v[j]));
                }
                return;
            }
            // 16 words in flight, whatever the row count: R rows of 16 / R planes
            auto fold = [&](auto width) {
                constexpr int R = decltype(width)::value, P = 16 / R;
                for (int p0 = cta + 1; p0 <= last && good; p0 += P) {
                    uint32_t t[P][R];
                    bool have = false;
                    for (uint32_t tries = 0; tries < (1u << 20) && !have; ++tries) {
                        have = true;
#pragma unroll
                        for (int p = 0; p < P; ++p)
#pragma unroll
                            for (int j = 0; j < R; ++j) {
                                t[p][j] = p0 + p <= last && j < rows ? ld_relaxed_gpu(words + ((size_t)(p0 + p) * rows + j) * 128) : 0u;
                                have = have && t[p][j] != kEmptyWord;
                            }
                    }
                    good = have;
#pragma unroll
                    for (int p = 0; p < P; ++p)
                        if (have && p0 + p <= last) {
#pragma unroll
                            for (int j = 0; j < R; ++j)
                                if (j < rows) {
                                    v[j] = __fadd_rn(v[j], __uint_as_float(t[p][j]));
                                    st_relaxed_gpu(words + ((size_t)(p0 + p) * rows + j) * 128, kEmptyWord);
                                }
                        }
                }
            };
            if (rows == 1) fold(std::integral_constant<int, 1>{});
            else if (rows == 2) fold(std::integral_constant<int, 2>{});
            else if (rows <= 4) fold(std::integral_constant<int, 4>{});
            else fold(std::integral_constant<int, 8>{});
#pragma unroll
            for (int j = 0; j < kMaxRowsT; ++j)
                if (j < rows) stage[j * 128 + col] = v[j];
            if (group_any(1 + group, !good)) {  // a wait that ran out leaves the block unwritten
                if (!good && lane == 0) atomicOr(c.status, kTimeoutFold);
                return;
            }
            if (quarter * 4 < rows) {  // four rows per warp, eight lanes per row
                const int row = quarter * 4 + e8;
                float u[4][4];
                uint2 sv[4];
                float4 bi[4];
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    sv[i] = __ldg(reinterpret_cast<const uint2*>(c.w.svh + c0 + 32 * i));
                    bi[i] = c.w.bias ? __ldg(reinterpret_cast<const float4*>(c.w.bias + c0 + 32 * i)) : make_float4(0.f, 0.f, 0.f, 0.f);
                    const float4 t = *reinterpret_cast<const float4*>(stage + row * 128 + 32 * i + 4 * l8);
                    u[i][0] = t.x; u[i][1] = t.y; u[i][2] = t.z; u[i][3] = t.w;
                }
                hadamard128_oct(u, lane);
                if (row < rows) {
                    const bool y_aligned = quads_aligned(c.y, c.y_dtype, c.y_stride);
#pragma unroll
                    for (int i = 0; i < 4; ++i) {
                        const uint32_t sw[2] = {sv[i].x, sv[i].y};
                        const float bias[4] = {bi[i].x, bi[i].y, bi[i].z, bi[i].w};
                        float o[4];
#pragma unroll
                        for (int j = 0; j < 4; ++j) {
                            o[j] = __fmul_rn(u[i][j], half_bits_to_float((uint16_t)(sw[j >> 1] >> (16 * (j & 1)))));
                            if (c.w.bias) o[j] = __fadd_rn(o[j], bias[j]);
                        }
                        scale_and_store_quad(c.y, c.y_dtype, (long long)row * c.y_stride + c0 + 32 * i, y_aligned, o, c.alpha, c.beta);
                    }
                }
            }
            named_barrier(1 + group, 128);  // before the group's next block overwrites `stage`
        };

        // Segments of the range, in order.  With a ring of activation slots a segment is staged before
        // the previous one's epilogue, never two ahead: the MMAs of a segment need the accumulator that
        // the epilogue two segments back frees.
        int seg = 0, nb = first_nb, hb = first_hb, done = 0, prev_hb = 0, prev_len = 0;
        for (; done < my_units; ++seg, ++nb, hb = 0) {
            const int left = my_units - done, len = left < hblocks - hb ? left : hblocks - hb;
            if (!resident) {
                stage_elements(done * rows, (done + len) * rows);
                if (seg && ((seg - 1) & 1) == group) epilogue(seg - 1, nb - 1, prev_hb, prev_len, done - prev_len);
                prev_hb = hb;
                prev_len = len;
            } else if ((seg & 1) == group) {
                epilogue(seg, nb, hb, len, done);
            }
            done += len;
        }
        if (!resident && ((seg - 1) & 1) == group) epilogue(seg - 1, nb - 1, prev_hb, prev_len, done - prev_len);
    }

    tc_fence_before_sync();
    __syncthreads();
    if (warp == kWarpMmaT) {
        __syncwarp();
        tc_fence_after_sync();
        tmem_dealloc(tmem, 512);
    }
}

// Marks `count` 16-byte words of a scratch area empty.  A kernel rather than a memset, so that it and
// the launch after it can both start programmatically.
__global__ void __launch_bounds__(256) empty_planes_kernel(uint4* planes, int count) {
    pdl_launch_dependents();
    pdl_wait_prior_grid();
    const int i = blockIdx.x * 256 + threadIdx.x;
    if (i < count) planes[i] = make_uint4(kEmptyWord, kEmptyWord, kEmptyWord, kEmptyWord);
}

// ---- host side -------------------------------------------------------------------------
GemvPlan plan_gemv(const DeviceWeights& w, int rows, int sm_count) {
    GemvPlan plan{};
    const int hblocks = w.inputs / 128, nblocks = w.outputs / 128, stride = unit_bytes(w.bits);
    const long long units = (long long)hblocks * nblocks;
    const int grid = (int)(units < sm_count ? units : sm_count);
    const int per_cta = (int)((units + grid - 1) / grid);
    // Activation slots for every block a range touches, as far as they leave the weight ring enough
    // bytes in flight to cover the HBM latency; the ring takes what is left.
    constexpr int kRing = 64 * 1024;
    int slots = per_cta < hblocks ? per_cta : hblocks;
    constexpr int most = (int)((kSmemLimitT - 1024 - kHeaderT - kRing) / kSlotBytesT);
    static_assert(most >= kMinBRing, "an activation ring holds a staging step");
    if (slots > most) slots = most;
    if (slots > kMaxBSlotsT) slots = kMaxBSlotsT;
    int ring = (int)((kSmemLimitT - 1024 - kHeaderT - (size_t)slots * kSlotBytesT) / stride);
    const int want = (128 * 1024) / stride;
    if (ring > want) ring = want;
    if (ring > per_cta) ring = per_cta;
    if (ring > kMaxWSlotsT) ring = kMaxWSlotsT;
    plan.grid = grid;
    plan.splits = (grid + nblocks - 1) / nblocks;  // typical K partitions of a column block
    plan.stages = ring;
    plan.act_blocks = slots;
    plan.smem_bytes = 1024 + kHeaderT + (size_t)slots * kSlotBytesT + (size_t)ring * stride;
    plan.counter_bytes = 0;  // the fold needs no counters
    plan.partial_bytes = align_up((size_t)grid * rows * 128 * sizeof(float));
    plan.row_kernel = rows == 1 && per_cta < kTmemUnits && plan_gemv_row(w, plan);
    plan.few_kernel = rows > 1 && per_cta <= kFewUnits;
    if (plan.few_kernel) plan_gemv_few(w, rows, per_cta, plan);
    return plan;
}

cudaError_t reset_gemv_scratch(void* workspace, const GemvPlan& plan, cudaStream_t stream) {
    const size_t words = (plan.counter_bytes + plan.partial_bytes) / 16;  // both are multiples of 256
    if (!words) return cudaSuccess;
    return launch_pdl(empty_planes_kernel, (int)((words + 255) / 256), 256, 0, true, stream, static_cast<uint4*>(workspace), (int)words);
}

cudaError_t launch_gemv(const LinearCall& call, const GemvPlan& plan, void* workspace, bool programmatic_launch,
                        cudaStream_t stream) {
    if (call.rows < 1 || call.rows > kMaxRowsT || !workspace) return cudaErrorInvalidValue;
    const long long units = (long long)(call.w.inputs / 128) * (call.w.outputs / 128);
    if (units > 0x7FFFFFFF || plan.grid < 1 || plan.grid > units || plan.stages < 1 || plan.act_blocks < 1) return cudaErrorInvalidValue;
    TmemArgs args{};
    args.call = call;
    args.split = make_split((int)units, plan.grid);
    args.w_slots = plan.stages;
    args.b_slots = plan.act_blocks;
    args.row_magic = call.rows == 1 ? 0 : (uint32_t)((0x100000000ull + call.rows - 1) / call.rows);
    args.planes = reinterpret_cast<float*>(static_cast<unsigned char*>(workspace) + plan.counter_bytes);
    if (plan.row_kernel) return launch_gemv_row(call, plan, args.split, args.planes, programmatic_launch, stream);
    if (plan.few_kernel) return launch_gemv_few(call, plan, args.split, args.planes, programmatic_launch, stream);
    return for_codebook(call.w.codebook, [&](auto cb) {
        return launch_pdl(gemv_tmem_kernel<decltype(cb)::value>, plan.grid, kThreadsT, plan.smem_bytes, programmatic_launch, stream, args);
    });
}

// Opt-in dynamic shared memory is a per-device function attribute: set when a context is created
// on a device (configure_device), never on the launch path.
cudaError_t configure_gemv_kernels() {
    cudaError_t e = cudaFuncSetAttribute(gemv_tmem_kernel<CB_3INST>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSmemLimitT);
    if (e == cudaSuccess)
        e = cudaFuncSetAttribute(gemv_tmem_kernel<CB_MCG>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSmemLimitT);
    if (e == cudaSuccess)
        e = cudaFuncSetAttribute(gemv_tmem_kernel<CB_MUL1>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSmemLimitT);
    return e;
}

}  // namespace st
