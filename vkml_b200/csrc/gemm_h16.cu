// GEMM on the tensor cores with half-precision operand terms: tcgen05.mma kind::f16, fp32 accumulators.
//
// Two uses of one kernel.
//
// F16 storage (one pass).  Half operands are the MMA's own format: products are exact, the accumulator
// is fp32, the result is narrowed once on the way out -- what the reference computes by widening, in
// the layout the caller already has.
//
// F32 storage (three passes).  Each operand x is scaled by a power of two s and split into
// hi = half(s x) and lo = half(2^11 (s x - hi)): 11 + 11 significant bits, the same 22 that the TF32
// split keeps, at twice the MMA rate and half the operand bytes.  hi.hi goes into one TMEM
// accumulator, the cross terms lo.hi + hi.lo, which carry the factor 2^11, into a second one; the
// epilogue adds them and takes the scales out again.  (8192^3: 4.22 -> 2.43 ms for the kernel, and a
// relative error of 9.7e-6 instead of 5.7e-5: half as many truncating additions per accumulator.)
//
// Half has five exponent bits, so s has to suit the matrix.  A first pass looks for the largest magnitude
// in a sample -- 128-element pieces spread over the whole matrix, all of it where it is small -- and s puts
// that into [2^13, 2^14): room for elements four times larger, and all 22 bits for elements down to
// 2^-26 of it.  The split checks every element against both ends.  The few that lie below the lower end, STRAYS (N(0,1) data has
// one in 3e7), are left out of the planes and noted, and their share of the product is added in fp32 behind this kernel (add_strays,
// gemm_tc.cu; 3 to 8 us where there are any): wherever they stand, each term keeps 22 bits, as with TF32 terms.  A matrix that overflows,
// that holds an infinity or a NaN, or that has more strays than kStrayFloor plus one in 2^21, is WIDE, and a product
// with a wide operand is computed by the TF32 planes queued behind this kernel instead (gemm_tc_stand_by;
// its launches return at once otherwise).  No host synchronisation decides this.  The gradient of a classifier that has
// learned something is wide -- probabilities of 1e-9 beside a label's 1 -- and shows it in the sample already: such a
// matrix gets no half planes, nor does an operand that only its product would read, so that what is left over the TF32 product
// is the range pass and two idle launches.  (8192x2048 . 2048x1000 on the gradient of logits of deviation 3: 229 us with TF32
// terms alone, 431 with half planes split first and thrown away and a standby split of one small block per SM, 234 now;
// x.W^T, g.W and x^T.g in one span 550, 765 and 532.  An outlier that the sample misses, 4096^3: 637, 800, 680.)
#include "gemm.h"
#include "tcgen05.cuh"

#include <algorithm>

#include <cuda_fp16.h>

namespace b200 {
namespace {

constexpr int kRowsM = 128;   // accumulator lanes of one CTA
constexpr int kBlockK = 64;   // halves per K-block: one 128-byte swizzle row
constexpr int kStepK = 16;    // K of one kind::f16 instruction
constexpr int kThreads = 192;
constexpr int kPatchPitch = 36;
constexpr int kGroupRows = 2048;  // M rows walked together before moving along N (L2 reuse of the B tiles)

// ---------------------------------------------------------------------------
// range of a matrix, and the split
// ---------------------------------------------------------------------------

struct MatrixArgs {
    const float* src;
    __half* hi;
    __half* lo;
    RangeSlot* range;
    int64_t b1, n_batches;            // inner batch extent, batches
    int64_t s_b0, s_b1, s_r, s_c;     // element strides
    int64_t rows, cols, pitch;        // pitch: halves per plane row (a multiple of 8)
    int vec;                          // rows start on 16 bytes and columns are dense
    // The other operand, where its being wide makes this one's planes useless: no other product of the span reads them.
    const RangeSlot* partner;
    uint32_t partner_limit;
    int64_t* strays;                  // positions of the elements left out, the first `limit` of them
    uint32_t limit;
};

struct MatrixPair {
    MatrixArgs m[2];
};

__device__ __forceinline__ const float* row_of(const MatrixArgs& a, int64_t rb, int64_t& r) {
    const int64_t b = a.n_batches == 1 ? 0 : rb / a.rows;
    r = rb - b * a.rows;
    const int64_t bo = a.s_b0 == 0 && a.b1 == 1 ? 0 : b / a.b1;
    return a.src + bo * a.s_b0 + (b - bo * a.b1) * a.s_b1 + r * a.s_r;
}

// Eight consecutive columns of one row, zeros past the end.
__device__ __forceinline__ void load8(const MatrixArgs& a, const float* row, int64_t c, float (&v)[8]) {
    if (a.vec && c + 8 <= a.cols) {
        const float4 x = __ldg(reinterpret_cast<const float4*>(row + c));
        const float4 y = __ldg(reinterpret_cast<const float4*>(row + c + 4));
        v[0] = x.x; v[1] = x.y; v[2] = x.z; v[3] = x.w;
        v[4] = y.x; v[5] = y.y; v[6] = y.z; v[7] = y.w;
        return;
    }
#pragma unroll
    for (int j = 0; j < 8; ++j) {
        v[j] = c + j < a.cols ? __ldg(row + (c + j) * a.s_c) : 0.0F;
    }
}

// The largest magnitude in a sample of each matrix, as the bits of its absolute value (infinities and
// NaNs included: they compare above every finite value), and how much of the sample is too small beside it.  Looking at all of both
// operands took 98 us at 8192^3 and 53 us at 512 x 65536 x 512; one piece in `stride`, a group to a thread, takes a few.
constexpr int kPiece = 16;  // consecutive groups of eight columns that are looked at together
constexpr int64_t kSampleGroups = int64_t(1) << 16;

__device__ __forceinline__ int64_t row_number(int64_t i, int64_t per_row, int64_t total) {
    return total < (int64_t(1) << 31) ? int64_t(uint32_t(i) / uint32_t(per_row)) : i / per_row;
}

__global__ void __launch_bounds__(256) range_kernel(MatrixPair pair) {
    pdl_prologue();
    const MatrixArgs& a = pair.m[blockIdx.y];
    const int64_t per_row = (a.cols + 7) / 8;
    const int64_t total = per_row * a.rows * a.n_batches;
    const uint32_t stride = static_cast<uint32_t>(max(int64_t(1), total / kSampleGroups));  // of the pieces, one in so many
    const uint32_t groups = static_cast<uint32_t>((total + stride - 1) / stride);           // (at most 2 * kSampleGroups)
    const bool small = total < (int64_t(1) << 31);
    const uint32_t j = blockIdx.x * blockDim.x + threadIdx.x;
    float v[8] = {};
    if (j < groups) {
        // (64-bit divisions for every group were most of this kernel's time on small matrices)
        const uint32_t piece = j / kPiece;
        // (a piece's place inside its stretch varies, so that no column pattern of the matrix is in step with it)
        const uint32_t shift = stride == 1 ? 0u : (piece * 7919u) % stride;
        const int64_t i = min(total - 1, (int64_t(piece) * stride + shift) * kPiece + j % kPiece);
        const int64_t rb = small ? int64_t(uint32_t(i) / uint32_t(per_row)) : i / per_row;
        int64_t r;
        load8(a, row_of(a, rb, r), (i - rb * per_row) * 8, v);
    }
    uint32_t top = 0;
#pragma unroll
    for (int q = 0; q < 8; ++q) top = max(top, __float_as_uint(v[q]) & 0x7FFFFFFFu);
    top = __reduce_max_sync(0xffffffffu, top);
    __shared__ uint32_t tops[8];
    if ((threadIdx.x & 31) == 0) tops[threadIdx.x >> 5] = top;
    __syncthreads();
#pragma unroll
    for (int w = 0; w < 8; ++w) top = max(top, tops[w]);
    if (threadIdx.x == 0 && top != 0) atomicMax(&a.range->max_bits, top);
    // what is too small beside the largest of this block's share of the sample is too small beside the matrix' largest
    const float low = __uint_as_float(top) * 0x1p-27F;
    uint32_t early = 0;
#pragma unroll
    for (int q = 0; q < 8; ++q) early += fabsf(v[q]) < low && v[q] != 0.0F;
    early = __reduce_add_sync(0xffffffffu, early);
    if ((threadIdx.x & 31) == 0 && early != 0) atomicAdd(&a.range->early, early);
}

__global__ void __launch_bounds__(kRangeSlots) clear_ranges_kernel(uint4* slots) {
    pdl_prologue();
    static_assert(sizeof(RangeSlot) == 2 * sizeof(uint4), "one slot to a thread");
    slots[threadIdx.x] = slots[kRangeSlots + threadIdx.x] = make_uint4(0, 0, 0, 0);
}

// Writes each matrix's two half planes, [batch][row][pitch], in the orientation the matrix has in memory: 4 bytes read, 4 written per element.
__global__ void __launch_bounds__(256) split_half_kernel(MatrixPair pair) {
    pdl_prologue();
    const MatrixArgs& a = pair.m[blockIdx.y];
    const int64_t per_row = a.pitch / 8;
    const int64_t total = per_row * a.rows * a.n_batches;
    const int64_t step = int64_t(gridDim.x) * blockDim.x;
    int64_t i = int64_t(blockIdx.x) * blockDim.x + threadIdx.x, rb = 0, c = 0;
    float v[8];
    auto fetch = [&] {
        int64_t r;
        rb = row_number(i, per_row, total);
        c = (i - rb * per_row) * 8;
        load8(a, row_of(a, rb, r), c, v);
    };
    if (i < total) fetch();  // (before the range is known: the two latencies overlap)
    __shared__ uint32_t largest;
    bool unread = false;
    if (threadIdx.x == 0) {
        const uint4 s = __ldcg(reinterpret_cast<const uint4*>(a.range));
        largest = s.x;
        unread = s.x >= 0x7F800000u || s.w > kStrayFloor;
    } else if (threadIdx.x == 1 && a.partner != nullptr) {
        unread = range_wide(a.partner, a.partner_limit);  // (its strays may still be counted beside this: what is seen only grows)
    }
    if (__syncthreads_or(unread)) return;
    const int up = range_shift(largest);
    const float s1 = exp2_int(up / 2), s2 = exp2_int(up - up / 2);
    bool over = false;
    while (i < total) {
        __half2 hi[4], lo[4];
        uint32_t few = 0;
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            float x = v[2 * j] * s1 * s2, y = v[2 * j + 1] * s1 * s2;  // exact: powers of two
            const bool stray_x = fabsf(x) < kStrayBelow && v[2 * j] != 0.0F, stray_y = fabsf(y) < kStrayBelow && v[2 * j + 1] != 0.0F;
            few |= (stray_x ? 1u : 0u) << (2 * j) | (stray_y ? 2u : 0u) << (2 * j);
            x = stray_x ? 0.0F : x;
            y = stray_y ? 0.0F : y;
            over = over || !(fmaxf(fabsf(x), fabsf(y)) < 65504.0F) || x != x || y != y;
            hi[j] = __floats2half2_rn(x, y);
            const float2 h = __half22float2(hi[j]);
            lo[j] = __floats2half2_rn((x - h.x) * 2048.0F, (y - h.y) * 2048.0F);
        }
        *reinterpret_cast<uint4*>(a.hi + rb * a.pitch + c) = *reinterpret_cast<const uint4*>(hi);
        *reinterpret_cast<uint4*>(a.lo + rb * a.pitch + c) = *reinterpret_cast<const uint4*>(lo);
        if (few != 0) {
            uint32_t at = atomicAdd(&a.range->strays, static_cast<uint32_t>(__popc(few)));
            for (; few != 0 && at < a.limit; few &= few - 1) a.strays[at++] = rb * a.cols + c + (__ffs(few) - 1);
        }
        i += step;
        if (i < total) fetch();
    }
    if (over) a.range->spoiled = 1;
}

// ---------------------------------------------------------------------------
// Main kernel
// ---------------------------------------------------------------------------

struct H16Args {
    void* out;             // C (f32 or half), or the f32 partial planes when splits > 1
    int out_half;
    // half output: the bias that a following add spreads over the rows, its result, and a relu's (each may be null)
    const __half* bias;
    __half* biased;
    __half* rectified;
    int64_t m, n, batches;
    int a_b1, b_b1;        // inner batch extents of the operand maps; 0: one matrix for every batch
    int64_t k_blocks, kb_per_split;
    int splits;
    int64_t split_stride;  // elements between partial planes
    int64_t tiles_m, tiles_n;
    int group_m;           // M-tiles walked together
    const RangeSlot* range_a;  // three passes: the operands' ranges
    const RangeSlot* range_b;
    uint32_t limit_a, limit_b;
    uint32_t* status;
};

// CG CTAs share one tile of CG*128 rows x BN columns: with CG = 2 each CTA of a cluster holds its 128
// rows of A and half of B, and one instruction issued by the even CTA drives both tensor cores
// (cta_group::2), so B's tile is fetched and stored once for 256 rows.
template <int CG, int BN, int PASSES>
struct H16Tile {
    static constexpr int kPlanes = PASSES == 3 ? 2 : 1;
    static constexpr int kABytes = kRowsM * kBlockK * 2;
    static constexpr int kBBytes = (BN / CG) * kBlockK * 2;
    static constexpr int kStageBytes = kPlanes * (kABytes + kBBytes);
    static constexpr int kFit = 200 * 1024 / kStageBytes;
    static constexpr int kStages = kFit < 8 ? kFit : 8;
    static constexpr int kAccCols = (PASSES == 3 ? 2 : 1) * BN;  // main terms, then cross terms
    static constexpr int kAccs = 2 * kAccCols <= 512 ? 2 : 1;
    static constexpr int kTmemCols = kAccs * kAccCols;
    static constexpr int kBars = kStages * kStageBytes;
    static constexpr int kTotal = kBars + 256 + 1024;
};

template <int CG>
__device__ __forceinline__ void tma_tile(uint32_t dst, const CUtensorMap* map, uint32_t bar, int c0, int c1, int c2, int c3) {
    if constexpr (CG == 2) {
        asm volatile(
            "cp.async.bulk.tensor.4d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5, %6}], [%2];"
            ::"r"(dst), "l"(reinterpret_cast<uint64_t>(map)), "r"(bar), "r"(c0), "r"(c1), "r"(c2), "r"(c3)
            : "memory");
    } else {
        tma_load_4d(dst, map, bar, c0, c1, c2, c3);
    }
}

// Bounded by the tensor cores for the large products.  Layout of the roles as in gemm_tc_kernel: warp 0 TMA,
// warp 1 tensor memory and MMA, warps 2-5 epilogue, tiles from a fixed walk.
template <int CG, int BN, int PASSES, bool A_MN, bool B_MN>
__global__ void __launch_bounds__(kThreads, 1)
gemm_h16_kernel(const __grid_constant__ CUtensorMap map_a_hi, const __grid_constant__ CUtensorMap map_a_lo,
                const __grid_constant__ CUtensorMap map_b_hi, const __grid_constant__ CUtensorMap map_b_lo, H16Args g) {
    using T = H16Tile<CG, BN, PASSES>;
    constexpr int STAGES = T::kStages;
    constexpr uint32_t kIdesc = h16_idesc(CG * kRowsM, BN, A_MN, B_MN);
    constexpr int kTileM = CG * kRowsM;
    static_assert(8 * (2 * STAGES + 2 * T::kAccs) <= 256, "barrier block");

    extern __shared__ uint8_t smem_raw[];
    const uint32_t base = (smem_u32(smem_raw) + 1023u) & ~1023u;
    const uint32_t bars = base + T::kBars;
    auto full_bar = [&](int s) { return bars + 8u * s; };              // the even CTA's: both CTAs' tiles landed
    auto empty_bar = [&](int s) { return bars + 8u * (STAGES + s); };
    auto acc_full = [&](int a) { return bars + 8u * (2 * STAGES + a); };
    auto acc_empty = [&](int a) { return bars + 8u * (2 * STAGES + T::kAccs + a); };  // the even CTA's
    __shared__ uint32_t tmem_base_slot;
    __shared__ int abort_flag;
    __shared__ __align__(16) float epi_patch[4][32][kPatchPitch];

    const int warp = threadIdx.x >> 5;
    const int lane = threadIdx.x & 31;
    const uint32_t rank = CG == 2 ? cluster_rank() : 0;

    if (threadIdx.x == 0) {
        abort_flag = 0;
        for (int s = 0; s < STAGES; ++s) {
            mbar_init(full_bar(s), 1);
            mbar_init(empty_bar(s), 1);
        }
        for (int a = 0; a < T::kAccs; ++a) {
            mbar_init(acc_full(a), 1);
            mbar_init(acc_empty(a), 4 * CG);
        }
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    }
    if (warp == 1) {
        tmem_get<CG>(smem_u32(&tmem_base_slot), T::kTmemCols);
        tc_fence_before();
    }
    __syncthreads();
    if (CG == 2) cluster_sync();  // the other CTA's barriers are initialised
    tc_fence_after();
    const uint32_t tmem_base = tmem_base_slot;
    volatile int* abort_p = &abort_flag;
    pdl_prologue();

    int64_t n_units = g.tiles_m * g.tiles_n * g.batches * g.splits;
    __shared__ int range_shifts[2];
    if (PASSES == 3) {
        if (threadIdx.x < 2) range_shifts[threadIdx.x] = range_shift(__ldcg(&(threadIdx.x == 0 ? g.range_a : g.range_b)->max_bits));
        // (the TF32 planes behind this kernel serve a wide operand's product)
        if (block_wide(RangeGuard{g.range_a, g.range_b, g.limit_a, g.limit_b})) n_units = 0;
    }
    const int64_t unit0 = blockIdx.x / CG, unit_step = gridDim.x / CG;
    auto decode = [&](int64_t u, int& split, int64_t& batch, int64_t& tm, int64_t& tn) {
        split = static_cast<int>(u % g.splits);
        int64_t t = u / g.splits;
        const int64_t per_batch = g.tiles_m * g.tiles_n;
        batch = t / per_batch;
        t -= batch * per_batch;
        const int64_t group_size = int64_t(g.group_m) * g.tiles_n;
        const int64_t group = t / group_size;
        const int64_t first_m = group * g.group_m;
        const int64_t rows_in_group = min(int64_t(g.group_m), g.tiles_m - first_m);
        const int64_t in_group = t - group * group_size;
        tm = first_m + in_group % rows_in_group;
        tn = in_group / rows_in_group;
    };

    if (warp == 0) {
        // ---------------- TMA producer (one per CTA, signalling the even CTA's barrier) ----------------
        if (lane == 0) {
            uint32_t it = 0;
            bool ok = true;
            for (int64_t u = unit0; u < n_units && ok; u += unit_step) {
                int split;
                int64_t batch, tm, tn;
                decode(u, split, batch, tm, tn);
                const int m0 = static_cast<int>(tm * kTileM + rank * kRowsM);
                const int n0 = static_cast<int>(tn * BN + rank * (BN / CG));
                const int a3 = g.a_b1 == 0 ? 0 : static_cast<int>(batch / g.a_b1), a2 = g.a_b1 == 0 ? 0 : static_cast<int>(batch - int64_t(a3) * g.a_b1);
                const int b3 = g.b_b1 == 0 ? 0 : static_cast<int>(batch / g.b_b1), b2 = g.b_b1 == 0 ? 0 : static_cast<int>(batch - int64_t(b3) * g.b_b1);
                const int64_t kb0 = int64_t(split) * g.kb_per_split;
                const int64_t kb1 = min(kb0 + g.kb_per_split, g.k_blocks);
                for (int64_t kb = kb0; kb < kb1; ++kb, ++it) {
                    const int s = it % STAGES;
                    if (!mbar_wait(empty_bar(s), ((it / STAGES) & 1) ^ 1, abort_p, g.status)) {
                        ok = false;
                        break;
                    }
                    const uint32_t stage = base + s * T::kStageBytes;
                    const int kc = static_cast<int>(kb * kBlockK);
                    const uint32_t bar = CG == 2 ? lead_addr(full_bar(s)) : full_bar(s);
                    if (rank == 0) mbar_arrive_expect_tx(full_bar(s), CG * T::kStageBytes);
                    auto load = [&](uint32_t dst, const CUtensorMap* map, bool mn, int rows, int r0, int c2, int c3) {
                        if (mn) {
                            for (int atom = 0; atom < rows / 64; ++atom) {
                                tma_tile<CG>(dst + atom * kAtomBytes, map, bar, r0 + 64 * atom, kc, c2, c3);
                            }
                        } else {
                            tma_tile<CG>(dst, map, bar, kc, r0, c2, c3);
                        }
                    };
                    load(stage, &map_a_hi, A_MN, kRowsM, m0, a2, a3);
                    load(stage + T::kPlanes * T::kABytes, &map_b_hi, B_MN, BN / CG, n0, b2, b3);
                    if (PASSES == 3) {
                        load(stage + T::kABytes, &map_a_lo, A_MN, kRowsM, m0, a2, a3);
                        load(stage + 2 * T::kABytes + T::kBBytes, &map_b_lo, B_MN, BN / CG, n0, b2, b3);
                    }
                }
            }
            drain_commits<STAGES>(empty_bar, it, abort_p, g.status);  // (from the even CTA's commits)
        }
    } else if (warp == 1) {
        // ---------------- MMA issuer (the even CTA's) ----------------
        if (lane == 0 && rank == 0) {
            uint32_t it = 0, tile_it = 0;
            bool ok = true;
            for (int64_t u = unit0; u < n_units && ok; u += unit_step, ++tile_it) {
                const int split = static_cast<int>(u % g.splits);
                const int acc = tile_it % T::kAccs;
                if (!mbar_wait(acc_empty(acc), ((tile_it / T::kAccs) & 1) ^ 1, abort_p, g.status)) break;
                tc_fence_after();
                const uint32_t d_main = tmem_base + acc * T::kAccCols;
                const uint32_t d_cross = d_main + BN;
                const int64_t kb0 = int64_t(split) * g.kb_per_split;
                const int64_t kb1 = min(kb0 + g.kb_per_split, g.k_blocks);
                for (int64_t kb = kb0; kb < kb1; ++kb, ++it) {
                    const int s = it % STAGES;
                    if (!mbar_wait(full_bar(s), (it / STAGES) & 1, abort_p, g.status)) {
                        ok = false;
                        break;
                    }
                    tc_fence_after();
                    const uint32_t stage = base + s * T::kStageBytes;
                    const uint64_t a_hi = h16_desc<A_MN>(stage);
                    const uint64_t a_lo = h16_desc<A_MN>(stage + T::kABytes);
                    const uint64_t b_hi = h16_desc<B_MN>(stage + T::kPlanes * T::kABytes);
                    const uint64_t b_lo = h16_desc<B_MN>(stage + T::kPlanes * T::kABytes + T::kBBytes);
#pragma unroll
                    for (int kk = 0; kk < kBlockK / kStepK; ++kk) {
                        const uint64_t adv_a = static_cast<uint64_t>((A_MN ? kk * kStepK * 128 : kk * kStepK * 2) >> 4);
                        const uint64_t adv_b = static_cast<uint64_t>((B_MN ? kk * kStepK * 128 : kk * kStepK * 2) >> 4);
                        const uint32_t more = (kb == kb0 && kk == 0) ? 0u : 1u;
                        if (PASSES == 3) {
                            umma_f16<CG>(d_cross, a_lo + adv_a, b_hi + adv_b, kIdesc, more);
                            umma_f16<CG>(d_cross, a_hi + adv_a, b_lo + adv_b, kIdesc, 1u);
                        }
                        umma_f16<CG>(d_main, a_hi + adv_a, b_hi + adv_b, kIdesc, more);
                    }
                    commit_all<CG>(empty_bar(s));
                }
                if (ok) commit_all<CG>(acc_full(acc));
            }
        }
    } else {
        // ---------------- epilogue (warps 2..5) ----------------
        const int quarter = warp & 3;
        float f1 = 1.0F, f2 = 1.0F, f3 = 1.0F;  // 2^-(shift_a + shift_b) in factors that stay in range
        if (PASSES == 3 && n_units > 0) {
            const int e = -(range_shifts[0] + range_shifts[1]);
            const int e1 = max(-126, min(126, e));
            const int e2 = max(-126, min(126, e - e1));
            f1 = exp2_int(e1);
            f2 = exp2_int(e2);
            f3 = exp2_int(e - e1 - e2);
        }
        const bool vec = g.n % 4 == 0 && g.split_stride % 4 == 0 && (reinterpret_cast<uintptr_t>(g.out) & 15) == 0;
        uint32_t tile_it = 0;
        for (int64_t u = unit0; u < n_units; u += unit_step, ++tile_it) {
            int split;
            int64_t batch, tm, tn;
            decode(u, split, batch, tm, tn);
            const int acc = tile_it % T::kAccs;
            if (!mbar_wait(acc_full(acc), (tile_it / T::kAccs) & 1, abort_p, g.status)) break;
            tc_fence_after();
            const int64_t row_base = tm * kTileM + rank * kRowsM + quarter * 32;
            const int64_t col0 = tn * BN;
            const int64_t at = int64_t(split) * g.split_stride + (batch * g.m + row_base) * g.n + col0;
            const uint32_t t_acc = tmem_base + (static_cast<uint32_t>(quarter * 32) << 16) + acc * T::kAccCols;
            int done_cols = 0;
            if (PASSES == 1 && g.out_half && vec && g.n % 8 == 0 && row_base < g.m) {
                // 64 columns at a time, narrowed before they go through the patch: whole 128-byte rows of halves per store
                __half* patch = reinterpret_cast<__half*>(&epi_patch[quarter][0][0]);
                constexpr int kPitch = 72;
#pragma unroll 1
                for (; done_cols + 64 <= BN && col0 + done_cols + 64 <= g.n; done_cols += 64) {
                    uint32_t r[32];
#pragma unroll
                    for (int half = 0; half < 2; ++half) {
                        tmem_ld32(t_acc + done_cols + 32 * half, r);
#pragma unroll
                        for (int j = 0; j < 4; ++j) {
                            __half2 h[4];
#pragma unroll
                            for (int q = 0; q < 4; ++q) {
                                h[q] = __floats2half2_rn(__uint_as_float(r[8 * j + 2 * q]), __uint_as_float(r[8 * j + 2 * q + 1]));
                            }
                            *reinterpret_cast<uint4*>(patch + lane * kPitch + 32 * half + 8 * j) = *reinterpret_cast<const uint4*>(h);
                        }
                    }
                    __syncwarp();
                    const int sub = lane >> 3, seg = lane & 7;
                    uint4 bias4 = make_uint4(0, 0, 0, 0);
                    if (g.bias != nullptr) bias4 = __ldg(reinterpret_cast<const uint4*>(g.bias + col0 + done_cols + seg * 8));
                    const __half2* b = reinterpret_cast<const __half2*>(&bias4);
#pragma unroll
                    for (int i = 0; i < 8; ++i) {
                        const int rl = i * 4 + sub;
                        if (row_base + rl < g.m) {
                            uint4 bits = *reinterpret_cast<const uint4*>(patch + rl * kPitch + seg * 8);
                            const int64_t o = at + int64_t(rl) * g.n + done_cols + seg * 8;
                            *reinterpret_cast<uint4*>(static_cast<__half*>(g.out) + o) = bits;
                            if (g.bias != nullptr) {
                                // every node narrows its own result (HalfIO, elementwise.cu): the sum is that of the stored halves
                                __half2* h = reinterpret_cast<__half2*>(&bits);
#pragma unroll
                                for (int q = 0; q < 4; ++q) {
                                    const float2 y = __half22float2(h[q]), w = __half22float2(b[q]);
                                    h[q] = __floats2half2_rn(__fadd_rn(y.x, w.x), __fadd_rn(y.y, w.y));
                                }
                                *reinterpret_cast<uint4*>(g.biased + o) = bits;
                                if (g.rectified != nullptr) {
#pragma unroll
                                    for (int q = 0; q < 4; ++q) {
                                        const float2 y = __half22float2(h[q]);
                                        h[q] = __floats2half2_rn(y.x <= 0.0F ? 0.0F : y.x, y.y <= 0.0F ? 0.0F : y.y);
                                    }
                                    *reinterpret_cast<uint4*>(g.rectified + o) = bits;
                                }
                            }
                        }
                    }
                    __syncwarp();
                }
            }
#pragma unroll 1
            for (int c = done_cols / 32; c < BN / 32; ++c) {
                if (col0 + c * 32 >= g.n || row_base >= g.m) break;  // uniform across the warp
                uint32_t r[32];
                tmem_ld32(t_acc + c * 32, r);
                if (PASSES == 3) {
                    uint32_t x[32];
                    tmem_ld32(t_acc + BN + c * 32, x);
#pragma unroll
                    for (int j = 0; j < 32; ++j) {
                        r[j] = __float_as_uint(fmaf(__uint_as_float(x[j]), 0x1p-11F, __uint_as_float(r[j])) * f1 * f2 * f3);
                    }
                }
                const int64_t left = g.n - (col0 + c * 32);
                if (vec && left >= 32) {
                    // through a padded patch, so that a warp stores whole row segments
                    float* patch = &epi_patch[quarter][0][0];
#pragma unroll
                    for (int j = 0; j < 8; ++j) {
                        *reinterpret_cast<uint4*>(patch + lane * kPatchPitch + 4 * j) =
                            make_uint4(r[4 * j], r[4 * j + 1], r[4 * j + 2], r[4 * j + 3]);
                    }
                    __syncwarp();
                    const int sub = lane >> 3, seg = lane & 7;
#pragma unroll
                    for (int i = 0; i < 8; ++i) {
                        const int rl = i * 4 + sub;
                        if (row_base + rl < g.m) {
                            const float4 v = *reinterpret_cast<const float4*>(patch + rl * kPatchPitch + seg * 4);
                            const int64_t o = at + int64_t(rl) * g.n + c * 32 + seg * 4;
                            if (g.out_half) {
                                __half2 h[2] = {__floats2half2_rn(v.x, v.y), __floats2half2_rn(v.z, v.w)};
                                *reinterpret_cast<uint2*>(static_cast<__half*>(g.out) + o) = *reinterpret_cast<const uint2*>(h);
                            } else {
                                *reinterpret_cast<float4*>(static_cast<float*>(g.out) + o) = v;
                            }
                        }
                    }
                    __syncwarp();
                } else {
                    // a ragged right edge, or rows that do not begin on 16 bytes: a row's 32 columns per store
                    float* patch = &epi_patch[quarter][0][0];
#pragma unroll
                    for (int j = 0; j < 8; ++j) {
                        *reinterpret_cast<uint4*>(patch + lane * kPatchPitch + 4 * j) =
                            make_uint4(r[4 * j], r[4 * j + 1], r[4 * j + 2], r[4 * j + 3]);
                    }
                    __syncwarp();
                    if (lane < left) {
                        const int rows = static_cast<int>(min(int64_t(32), g.m - row_base));
                        for (int rl = 0; rl < rows; ++rl) {
                            const float v = patch[rl * kPatchPitch + lane];
                            const int64_t o = at + int64_t(rl) * g.n + c * 32 + lane;
                            if (g.out_half) static_cast<__half*>(g.out)[o] = __float2half_rn(v);
                            else static_cast<float*>(g.out)[o] = v;
                        }
                    }
                    __syncwarp();
                }
            }
            tc_fence_before();
            __syncwarp();
            if (lane == 0) {
                if (CG == 2) mbar_arrive_cluster(lead_addr(acc_empty(acc)));
                else mbar_arrive(acc_empty(acc));
            }
        }
    }

    __syncwarp();
    __syncthreads();
    if (abort_flag != 0) {
        for (int i = 0; i < 200; ++i) __nanosleep(1000);  // copies in flight land before the CTA retires
        __syncthreads();
    }
    tc_fence_before();
    if (CG == 2) cluster_sync();  // nothing of the pair is addressed after this
    if (warp == 1) {
        tc_fence_after();
        tmem_put<CG>(tmem_base, T::kTmemCols);
    }
}

// Sums the K-slices' partial planes in split order: `splits` of this product, or `wide_splits` from the TF32 planes that stood
// by for a wide operand (one slice: the product went straight to `out`).
template <typename Out>
__global__ void __launch_bounds__(256) fold_kernel(Out* __restrict__ out, const float* __restrict__ part, int64_t n, int splits,
                                                   RangeGuard guard, int wide_splits) {
    pdl_prologue();
    if (guard.a != nullptr && block_wide(guard)) splits = wide_splits;
    if (splits <= 1) return;
    const int64_t step = int64_t(gridDim.x) * blockDim.x;
    if (n % 4 == 0) {
        for (int64_t i = int64_t(blockIdx.x) * blockDim.x + threadIdx.x; i < n / 4; i += step) {
            float4 s = __ldcg(reinterpret_cast<const float4*>(part) + i);
            for (int k = 1; k < splits; ++k) {
                const float4 v = __ldcg(reinterpret_cast<const float4*>(part + int64_t(k) * n) + i);
                s.x += v.x; s.y += v.y; s.z += v.z; s.w += v.w;
            }
            if constexpr (sizeof(Out) == 2) {
                __half2 h[2] = {__floats2half2_rn(s.x, s.y), __floats2half2_rn(s.z, s.w)};
                if (reinterpret_cast<uintptr_t>(out) % 8 == 0) {
                    reinterpret_cast<uint2*>(out)[i] = *reinterpret_cast<const uint2*>(h);
                } else {
                    for (int j = 0; j < 4; ++j) out[4 * i + j] = reinterpret_cast<const __half*>(h)[j];
                }
            } else if (reinterpret_cast<uintptr_t>(out) % 16 == 0) {
                reinterpret_cast<float4*>(out)[i] = s;
            } else {
                out[4 * i] = s.x; out[4 * i + 1] = s.y; out[4 * i + 2] = s.z; out[4 * i + 3] = s.w;
            }
        }
        return;
    }
    for (int64_t i = int64_t(blockIdx.x) * blockDim.x + threadIdx.x; i < n; i += step) {
        float s = __ldcg(part + i);
        for (int k = 1; k < splits; ++k) s += __ldcg(part + int64_t(k) * n + i);
        out[i] = static_cast<Out>(s);
    }
}

// ---------------------------------------------------------------------------
// Host side
// ---------------------------------------------------------------------------

// A half matrix as a 4-D tensor: (unit-stride axis, the other axis, inner batch, outer batch), boxes of 64 x box_rows.
CUtensorMap half_map(const __half* base, int64_t cols, int64_t rows, int64_t pitch, int64_t b1, int64_t s_b1, int64_t b0,
                     int64_t s_b0, int box_rows) {
    CUtensorMap m;
    const int64_t plane = std::max<int64_t>(rows * pitch, 8);
    if (b1 <= 1) { b1 = 1; s_b1 = plane; }
    if (b0 <= 1) { b0 = 1; s_b0 = std::max(plane, s_b1 * b1); }
    const cuuint64_t dims[4] = {cuuint64_t(cols), cuuint64_t(rows), cuuint64_t(b1), cuuint64_t(b0)};
    const cuuint64_t strides[3] = {cuuint64_t(pitch) * 2, cuuint64_t(s_b1) * 2, cuuint64_t(s_b0) * 2};
    const cuuint32_t box[4] = {kBlockK, cuuint32_t(box_rows), 1, 1};
    const cuuint32_t elem[4] = {1, 1, 1, 1};
    const CUresult rc = encode_tiled()(&m, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 4, const_cast<__half*>(base), dims, strides, box,
                                       elem, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
                                       CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (rc != CUDA_SUCCESS) {
        fail(B200_INTERNAL_ERROR, "cuTensorMapEncodeTiled (half operand) failed with code " + std::to_string(rc));
    }
    return m;
}

// One operand as the matrix it is in memory: rows x cols with `cols` the unit-stride axis where there is one.
// An operand whose M (or N) axis is that axis is consumed MN-major: nothing is transposed.
struct HalfOperand {
    bool mn = false, bcast = false;
    int64_t rows = 0, cols = 0, nb = 1, b1 = 1, s_b0 = 0, s_b1 = 0, s_r = 0, s_c = 0, pitch = 0;
    const void* src = nullptr;
    const __half* hi = nullptr;  // (one pass: the operand itself)
    const __half* lo = nullptr;
    int64_t map_b1 = 1, map_s_b1 = 0, map_b0 = 1, map_s_b0 = 0;
    RangeSlot* range = nullptr;
    PlaneKey key{};
    bool cached = false, fresh = false;
    Standby standby{};

    int64_t numel() const { return nb * rows * cols; }
    size_t plane_bytes() const { return static_cast<size_t>(align_up(nb * rows * pitch * 2, 1024)); }
    uint32_t limit() const { return std::min(kMaxStrays, kStrayFloor + static_cast<uint32_t>(std::min<int64_t>(numel() >> 21, kMaxStrays))); }
    size_t stray_bytes() const { return static_cast<size_t>(align_up(int64_t(limit()) * 8, 1024)); }
    CUtensorMap map(const __half* plane, int tile) const {
        return half_map(plane, cols, rows, pitch, map_b1, map_s_b1, map_b0, map_s_b0, mn ? kBlockK : tile);
    }
};

HalfOperand half_operand(const void* src, const int64_t (&s)[4], int mn_axis, int k_axis, int64_t mn_extent, int64_t k_extent,
                         const GemmProblem& p) {
    HalfOperand o;
    o.src = src;
    o.bcast = (s[0] == 0 || p.b0 == 1) && (s[1] == 0 || p.b1 == 1);
    o.nb = o.bcast ? 1 : p.b0 * p.b1;
    o.b1 = o.bcast ? 1 : p.b1;
    o.s_b0 = o.bcast ? 0 : s[0];
    o.s_b1 = o.bcast ? 0 : s[1];
    o.mn = s[mn_axis] == 1 && s[k_axis] != 1;
    o.rows = o.mn ? k_extent : mn_extent;
    o.cols = o.mn ? mn_extent : k_extent;
    o.s_r = o.mn ? s[k_axis] : s[mn_axis];
    o.s_c = o.mn ? s[mn_axis] : s[k_axis];
    return o;
}

HalfOperand operand_a(const GemmProblem& p) { return half_operand(p.a, p.a_s, 2, 3, p.m, p.k, p); }
HalfOperand operand_b(const GemmProblem& p) { return half_operand(p.b, p.b_s, 3, 2, p.n, p.k, p); }

// The dense layout of planes: [batch][row][pitch].
void lay_out_planes(HalfOperand& o) {
    o.pitch = align_up(o.cols, 8);
    o.map_b1 = o.nb;
    o.map_s_b1 = o.rows * o.pitch;
    o.map_b0 = 1;
    o.map_s_b0 = 0;
    o.key.src = o.src;
    const int64_t kv[9] = {o.rows, o.cols, o.s_r, o.s_c, o.b1, o.s_b0, o.s_b1, o.nb, 1};
    for (int i = 0; i < 9; ++i) o.key.v[i] = kv[i];
}

template <int CG, int BN, int PASSES, bool A_MN, bool B_MN>
void launch_tile(b200_ctx* ctx, const HalfOperand& a, const HalfOperand& b, const H16Args& g, int64_t units) {
    using T = H16Tile<CG, BN, PASSES>;
    auto kernel = gemm_h16_kernel<CG, BN, PASSES, A_MN, B_MN>;
    B200_CUDA_CHECK(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, T::kTotal));
    const CUtensorMap ah = a.map(a.hi, kRowsM), bh = b.map(b.hi, BN / CG);
    const CUtensorMap al = PASSES == 3 ? a.map(a.lo, kRowsM) : ah, bl = PASSES == 3 ? b.map(b.lo, BN / CG) : bh;
    int sms = ctx->prop.multiProcessorCount;
    if (ctx->in_grad_sync_span && ctx->comm_pending) sms = std::max(sms - ctx->comm_sms, sms / 2);
    const int grid = static_cast<int>(std::min<int64_t>(units, sms / CG)) * CG;
    // Not scheduled ahead of the kernel in front of it.  With an early start -- a CTA pair that holds tensor memory and waits while up to four
    // kernels before it still run -- a long sequence of mixed odd shapes stopped for good about once in 50000 products; five million
    // in a row have not since.  It costs 2 us at 2048x1024x1024 (33.4 -> 35.2), nothing from 2048x1000x8192 on.
    launch_kernel_clustered(ctx, kernel, grid, kThreads, T::kTotal, CG, false, ah, al, bh, bl, g);
    ctx->count_launch();
}

template <int CG, int BN, int PASSES>
void launch_major(b200_ctx* ctx, const HalfOperand& a, const HalfOperand& b, const H16Args& g, int64_t units) {
    static_assert(BN / CG >= 64, "an MN-major atom is 64 wide");
    if (a.mn && b.mn) launch_tile<CG, BN, PASSES, true, true>(ctx, a, b, g, units);
    else if (b.mn) launch_tile<CG, BN, PASSES, false, true>(ctx, a, b, g, units);
    else if (a.mn) launch_tile<CG, BN, PASSES, true, false>(ctx, a, b, g, units);
    else launch_tile<CG, BN, PASSES, false, false>(ctx, a, b, g, units);
}

struct TileChoice {
    int cg, bn;
    int64_t tiles_m, tiles_n, splits, kb_per_split, units;
    double cost;
};

// The tile whose whole waves cost least.  `width` x 128 rows of cg CTAs; a narrower or single-CTA tile moves more
// operand bytes per product (relative cost per unit of work beside the widest), so it is taken only
// where the widest one would leave SMs idle: few tiles, or a nearly empty last wave.
TileChoice choose_tile(const GemmProblem& p, int passes, int sms) {
    struct Form { int cg, bn; double cost, alone, drain; };
    // cost of one K-block of a tile in units of a 256 x 128 tile's, the same where one wave serves the product (a CTA by itself starts and
    // ends sooner than a pair, but fetches B for half as many rows), and K-blocks that its fill and drain come to.  Three
    // passes over 256 columns leave room for one pair of accumulators, so that tile's epilogue is not hidden; its operand
    // traffic per product is two thirds, which at the power cap is worth 14 % (8192^3: 3.15 -> 2.69 ms sustained).  A 64-wide tile
    // costs nearly what a 128-wide one does, the instructions being the limit.  Each form forced for 30 products of 2^32 to 2^40 operations: with
    // these figures the choice is 1 % slower than the best on average and 7 % at most.  us for 256x256, 256x128, 128x128 and 128x64:
    //   8192^3 2471 2990 3004 4732;  2048x8192x8192 703 796 760 1330;  3000^3 148 169 235 317;  6000x2000x576 77 92 92 107;
    //   1536^3 47.2 41.6 39.7 51.5;  300x8192x1000 54 54 49 57;  512x8192x512 47 43 42 48;  1200x4000x520 49 48 47 60;  20000x2000x64 139 123 125 121.
    // (256x64 was slower than one of these on every product: 6000x2000x576 108, 1200x4000x520 62.)
    static const Form three[] = {{2, 256, 1.65, 1.65, 6}, {2, 128, 1.0, 1.0, 2}, {1, 128, 1.08, 1.02, 1}, {1, 64, 0.9, 0.9, 2}};
    static const Form one[] = {{2, 256, 1.75, 1.75, 2}, {1, 128, 1.08, 1.08, 2}, {1, 64, 0.6, 0.6, 2}};
    const Form* forms = passes == 3 ? three : one;
    const int64_t batches = p.b0 * p.b1, k_blocks = ceil_div(p.k, kBlockK);
    TileChoice best{};
    double least = 0;
    for (int i = 0; i < (passes == 3 ? 4 : 3); ++i) {
        const Form& f = forms[i];
        TileChoice c{f.cg, f.bn, ceil_div(p.m, int64_t(f.cg) * kRowsM), ceil_div(p.n, int64_t(f.bn)), 1, k_blocks, 0};
        const int64_t tiles = c.tiles_m * c.tiles_n * batches, slots = sms / f.cg;
        if (tiles < slots && k_blocks >= 8) {
            // as many K-slices as keep every unit in one wave, none shorter than four K-blocks
            c.splits = std::max<int64_t>(1, std::min({slots / tiles, k_blocks / 4, int64_t(64)}));
            c.kb_per_split = ceil_div(k_blocks, c.splits);
            c.splits = ceil_div(k_blocks, c.kb_per_split);
        }
        c.units = tiles * c.splits;
        const double waves = double(ceil_div(c.units, slots));
        // (slices write and fold partial planes)
        const double cost = waves * (waves > 1 ? f.cost : f.alone) * (double(c.kb_per_split) + f.drain) + (c.splits > 1 ? 4.0 : 0.0);
        if (i == 0 || cost < least) {
            least = cost;
            best = c;
            best.cost = cost;
        }
    }
    return best;
}

void run_h16(b200_ctx* ctx, const GemmProblem& p, int passes, const TileChoice& t, const HalfOperand& a, const HalfOperand& b,
             float* partial, bool out_half, const char* label, const HalfEpilogue* epi = nullptr) {
    H16Args g{};
    if (epi != nullptr) {
        g.bias = static_cast<const __half*>(epi->bias);
        g.biased = static_cast<__half*>(epi->biased);
        g.rectified = static_cast<__half*>(epi->rectified);
    }
    const int64_t batches = p.b0 * p.b1, out_elems = batches * p.m * p.n;
    g.out = t.splits > 1 ? static_cast<void*>(partial) : static_cast<void*>(p.out);
    g.out_half = t.splits > 1 ? 0 : (out_half ? 1 : 0);
    g.m = p.m;
    g.n = p.n;
    g.batches = batches;
    g.a_b1 = a.bcast ? 0 : static_cast<int>(a.map_b1);
    g.b_b1 = b.bcast ? 0 : static_cast<int>(b.map_b1);
    g.k_blocks = ceil_div(p.k, kBlockK);
    g.kb_per_split = t.kb_per_split;
    g.splits = static_cast<int>(t.splits);
    g.split_stride = out_elems;
    g.tiles_m = t.tiles_m;
    g.tiles_n = t.tiles_n;
    g.group_m = ctx->gemm_group_m > 0 ? ctx->gemm_group_m : kGroupRows / (t.cg * kRowsM);
    g.range_a = a.range;
    g.range_b = b.range;
    g.limit_a = a.limit();
    g.limit_b = b.limit();
    g.status = ctx->d_status;
    {
        ProfScope scope(ctx, label);
#define B200_H16_CASE(CG, BN, P)                                  \
    if (t.cg == CG && t.bn == BN && passes == P) launch_major<CG, BN, P>(ctx, a, b, g, t.units);
        B200_H16_CASE(2, 256, 3)
        B200_H16_CASE(2, 128, 3)
        B200_H16_CASE(1, 128, 3)
        B200_H16_CASE(1, 64, 3)
        B200_H16_CASE(2, 256, 1)
        B200_H16_CASE(1, 128, 1)
        B200_H16_CASE(1, 64, 1)
#undef B200_H16_CASE
    }
    check_last_launch("matmul (tcgen05, half terms)");
}

template <typename Out>
void run_fold(b200_ctx* ctx, const GemmProblem& p, const float* partial, int splits, const RangeGuard& guard = {}, int wide_splits = 1) {
    if (splits <= 1 && wide_splits <= 1) return;
    ProfScope scope(ctx, "matmul.fold");
    const int64_t out_elems = p.b0 * p.b1 * p.m * p.n;
    launch_kernel(ctx, fold_kernel<Out>, grid_for(ceil_div(out_elems, 4), 256), 256, 0, reinterpret_cast<Out*>(p.out), partial, out_elems,
                  splits, guard, wide_splits);
    ctx->count_launch();
    check_last_launch("matmul (fold)");
}

bool fits_tma(const GemmProblem& p) {
    const int64_t lim = int64_t(1) << 31;
    return p.m < lim && p.n < lim && p.k < lim && p.b0 * p.b1 < lim;
}

MatrixArgs matrix_args(const HalfOperand& o) {
    MatrixArgs a{};
    a.src = static_cast<const float*>(o.src);
    a.hi = const_cast<__half*>(o.hi);
    a.lo = const_cast<__half*>(o.lo);
    a.range = o.range;
    a.b1 = o.b1;
    a.n_batches = o.nb;
    a.s_b0 = o.s_b0;
    a.s_b1 = o.s_b1;
    a.s_r = o.s_r;
    a.s_c = o.s_c;
    a.rows = o.rows;
    a.cols = o.cols;
    a.pitch = o.pitch;
    a.vec = o.s_c == 1 && o.s_r % 4 == 0 && o.s_b0 % 4 == 0 && o.s_b1 % 4 == 0 && reinterpret_cast<uintptr_t>(o.src) % 16 == 0;
    return a;
}

}  // namespace

// Products above 2^31 operations.  The range pass (a read of a sample) and the launches that stand by behind the product cost
// about 8 us together, which the halved MMA time returns from 2^32 on: 2048x1024x1024 36.2 us with TF32 terms and 34.2 with half
// terms, 512x8192x512 49.6 and 44.3, 1301x1333x1277 43.2 and 41.2, 1536^3 45 and 41.  Between 2^31 and 2^32 TF32 terms are quicker as a rule --
// 1000x1433x777 34.6 and 36.6, 1024x1536x1024 33.5 and 34.2, 1536x700x1536 28.7 and 31.0, 511x4097x513 34.5 and 42.5 -- but five times further
// from the exact product (5e-6 against 9e-7 on those), and what has half terms' error keeps it.  Below, they would be quicker by a
// third: 768x1024x768 21.3 and 30.4, 1024^3 26.8 and 29.
// What the streamed-operand kernel or the direct operands serve stays there.
bool gemm_h16_serves(const b200_ctx* ctx, const GemmProblem& p) {
    return gemm_h16_would_serve(ctx, p) && !(ctx->lone_matmul && gemm_tc_reads_directly(ctx, p));
}

bool gemm_h16_would_serve(const b200_ctx* ctx, const GemmProblem& p) {
    if (ctx->gemm_precision != B200_GEMM_3XTF32 || !ctx->gemm_half_terms || ctx->gemm_operands >= 0 || ctx->gemm_stream > 0 ||
        ctx->gemm_schedule == 1 || ctx->gemm_bn_override != 0 || !fits_tma(p)) {
        return false;
    }
    const double flops = 2.0 * double(p.m) * double(p.n) * double(p.k) * double(p.b0 * p.b1);
    // (One accumulator over more than 12288 products leaves a TF32 result about 1e-4 from the exact one -- 4096 x 16384 x 4096: 1.15e-4, from
    // half terms 1.9e-5 -- so the two would differ by more than the 1e-4 that results have kept to from version to version.)
    return flops > 2147483648.0 && !gemm_tc_streams(ctx, p) && ctx->compared.count(p.out) == 0 && gemm_tc_chain(ctx, p) <= 12288;
}

bool gemm_h16_shares(const b200_ctx* ctx, const GemmProblem& p) {
    for (HalfOperand o : {operand_a(p), operand_b(p)}) {
        lay_out_planes(o);
        const auto it = ctx->plane_uses.find(o.key);
        if (it != ctx->plane_uses.end() && it->second >= 2) return true;
    }
    return false;
}

// The planes' bytes at the rate their pass runs at, the tiles (a K-block of the 256 x 128 tile takes 0.66 us) and the launches around them.
double gemm_h16_time(const b200_ctx* ctx, const GemmProblem& p) {
    const HalfOperand a = operand_a(p), b = operand_b(p);
    return 8.0 * double(a.numel() + b.numel()) / 5.8e6 + 0.66 * choose_tile(p, 3, ctx->prop.multiProcessorCount).cost + 7.0;
}

std::string gemm_h16_tile(const b200_ctx* ctx, const GemmProblem& p) {
    const TileChoice t = choose_tile(p, 3, ctx->prop.multiProcessorCount);
    return std::to_string(t.cg * kRowsM) + "x" + std::to_string(t.bn);
}

void gemm_h16_note_uses(b200_ctx* ctx, const GemmProblem& p) {
    HalfOperand a = operand_a(p), b = operand_b(p);
    lay_out_planes(a);
    lay_out_planes(b);
    ++ctx->plane_uses[a.key];
    ++ctx->plane_uses[b.key];
}

RangeSlot* gemm_h16_slots(b200_ctx* ctx, int n) {
    if (ctx->range_next + n > kRangeSlots) return nullptr;
    if (ctx->range_next == 0) {
        // (a kernel, not a memset: it overlaps its neighbours' launches, which a memset between them would not let do so either)
        launch_kernel(ctx, clear_ranges_kernel, 1u, kRangeSlots, 0, static_cast<uint4*>(ctx->d_ranges));
        ctx->count_launch();
    }
    ctx->range_next += n;
    return static_cast<RangeSlot*>(ctx->d_ranges) + (ctx->range_next - n);
}

void gemm_h16_fold(b200_ctx* ctx, const GemmProblem& p, const float* partial, int splits, const RangeGuard& guard, int wide_splits) {
    run_fold<float>(ctx, p, partial, splits, guard, wide_splits);
}

void gemm_h16(b200_ctx* ctx, const GemmProblem& p) {
    HalfOperand a = operand_a(p), b = operand_b(p);
    const TileChoice t = choose_tile(p, 3, ctx->prop.multiProcessorCount);
    if (ctx->range_next + 2 > kRangeSlots) {
        gemm_tc(ctx, p, true);
        return;
    }
    if (ctx->range_next == 0) {
        // (a kernel, not a memset: it overlaps its neighbours' launches, which a memset between them would not let do so either)
        launch_kernel(ctx, clear_ranges_kernel, 1u, kRangeSlots, 0, static_cast<uint4*>(ctx->d_ranges));
        ctx->count_launch();
    }
    const size_t cache_limit = std::min<size_t>(size_t(16) << 30, ctx->prop.totalGlobalMem / 8);
    auto place = [&](HalfOperand& o, size_t tf32_bytes) {
        lay_out_planes(o);
        if (auto it = ctx->plane_cache.find(o.key); it != ctx->plane_cache.end()) {
            o.hi = reinterpret_cast<const __half*>(it->second.hi);
            o.lo = reinterpret_cast<const __half*>(it->second.lo);
            o.range = static_cast<RangeSlot*>(it->second.range);
            o.standby = {it->second.tf32, &o.range->tf32, it->second.strays};
            o.cached = true;
            ++ctx->plane_hits;
            return;
        }
        o.fresh = true;
        o.range = static_cast<RangeSlot*>(ctx->d_ranges) + ctx->range_next++;
        const auto uses = ctx->plane_uses.find(o.key);
        const size_t bytes = 2 * o.plane_bytes() + tf32_bytes + o.stray_bytes();
        if (uses != ctx->plane_uses.end() && uses->second >= 2 && ctx->plane_cache_bytes + bytes <= cache_limit) {
            char* block = static_cast<char*>(ctx->scratch.allocate(bytes));
            o.hi = reinterpret_cast<const __half*>(block);
            o.lo = reinterpret_cast<const __half*>(block + o.plane_bytes());
            int64_t* strays = reinterpret_cast<int64_t*>(block + 2 * o.plane_bytes() + tf32_bytes);
            o.standby = {reinterpret_cast<float*>(block + 2 * o.plane_bytes()), &o.range->tf32, strays};
            const char* begin = static_cast<const char*>(o.src);
            auto mag = [](int64_t v) { return v < 0 ? -v : v; };
            const int64_t span = (o.nb / o.b1 - 1) * mag(o.s_b0) + (o.b1 - 1) * mag(o.s_b1) + (o.rows - 1) * mag(o.s_r) +
                                 (o.cols - 1) * mag(o.s_c) + 1;
            ctx->plane_cache[o.key] = PlaneEntry{reinterpret_cast<float*>(block), reinterpret_cast<float*>(block + o.plane_bytes()),
                                                 bytes, uses->second, begin, begin + span * 4, o.range, o.standby.planes, strays};
            ctx->plane_cache_bytes += bytes;
            o.cached = true;
        }
    };
    const size_t a_tf32 = gemm_tc_plane_bytes(p, true), b_tf32 = gemm_tc_plane_bytes(p, false);
    place(a, a_tf32);
    place(b, b_tf32);  // (B may be the very matrix A just put there)

    const int64_t out_elems = p.b0 * p.b1 * p.m * p.n;
    const int wide_splits = gemm_tc_slices(ctx, p);
    const int64_t slices = std::max<int64_t>(t.splits, wide_splits);
    const size_t partial_bytes = slices > 1 ? static_cast<size_t>(align_up(out_elems * slices * 4, 1024)) : 0;
    size_t bytes = partial_bytes + 1024;
    if (!a.cached) bytes += 2 * a.plane_bytes() + a_tf32 + a.stray_bytes();
    if (!b.cached) bytes += 2 * b.plane_bytes() + b_tf32 + b.stray_bytes();
    char* ws = static_cast<char*>(ctx->ensure_workspace(bytes));
    ws = reinterpret_cast<char*>(align_up(reinterpret_cast<int64_t>(ws), 1024));
    for (HalfOperand* o : {&a, &b}) {
        if (o->cached) continue;
        o->hi = reinterpret_cast<const __half*>(ws);
        o->lo = reinterpret_cast<const __half*>(ws + o->plane_bytes());
        o->standby.planes = reinterpret_cast<float*>(ws + 2 * o->plane_bytes());
        ws += 2 * o->plane_bytes() + (o == &a ? a_tf32 : b_tf32);
        o->standby.strays = reinterpret_cast<int64_t*>(ws);
        ws += o->stray_bytes();
    }
    float* partial = reinterpret_cast<float*>(ws);

    MatrixPair pair{};
    int fresh = 0;
    int64_t largest = 0;
    for (HalfOperand* o : {&a, &b}) {
        if (!o->fresh) continue;
        pair.m[fresh] = matrix_args(*o);
        pair.m[fresh].strays = const_cast<int64_t*>(o->standby.strays);
        pair.m[fresh].limit = o->limit();
        if (!o->cached) {
            const HalfOperand& other = o == &a ? b : a;
            pair.m[fresh].partner = other.range;
            pair.m[fresh].partner_limit = other.limit();
        }
        ++fresh;
        largest = std::max(largest, o->nb * o->rows * (o->pitch / 8));
    }
    if (fresh > 0) {
        const dim3 grid(grid_for(largest, 256), static_cast<unsigned>(fresh));
        {
            ProfScope scope(ctx, "matmul.range");
            launch_kernel(ctx, range_kernel, dim3(static_cast<unsigned>(ceil_div(std::min(largest, 2 * kSampleGroups), 256)), grid.y), 256, 0, pair);
        }
        {
            ProfScope scope(ctx, "matmul.split");
            launch_kernel(ctx, split_half_kernel, grid, 256, 0, pair);
        }
        ctx->count_launch(2);
        check_last_launch("matmul (operand range and split)");
    }
    run_h16(ctx, p, 3, t, a, b, partial, false, "matmul.tcgen05_3xf16");
    const RangeGuard guard{a.range, b.range, a.limit(), b.limit()};
    gemm_tc_stand_by(ctx, p, guard, a.standby, b.standby, t.splits > 1 ? partial : p.out, partial);
    run_fold<float>(ctx, p, partial, static_cast<int>(t.splits), guard, wide_splits);
    for (HalfOperand* o : {&a, &b}) {
        if (!o->cached) continue;
        const auto it = ctx->plane_cache.find(o->key);
        if (it != ctx->plane_cache.end() && --it->second.uses_left <= 0) {
            ctx->scratch.release(it->second.hi);  // the stream is in order: only later work reuses it
            ctx->plane_cache_bytes -= it->second.bytes;
            ctx->plane_cache.erase(it);
        }
    }
}

// Half storage: products of at least 2^25 operations with a row for most of a tile's lanes (smaller ones are
// launch-bound, and served through widened copies by the CUDA cores).
bool gemm_f16_storage(b200_ctx* ctx, const GemmProblem& p, const HalfEpilogue* epi) {
    if (ctx->prop.major != 10 || encode_tiled() == nullptr || ctx->gemm_precision == B200_GEMM_FP32 || !fits_tma(p) ||
        p.m < 32 || p.n < 16 || p.k < 16) {
        return false;
    }
    if (2.0 * double(p.m) * double(p.n) * double(p.k) * double(p.b0 * p.b1) < double(1 << 25)) return false;
    HalfOperand a = operand_a(p), b = operand_b(p);
    const TileChoice t = choose_tile(p, 1, ctx->prop.multiProcessorCount);
    auto direct = [](HalfOperand& o) {
        const bool ok = o.s_c == 1 && o.s_r % 8 == 0 && o.s_r >= o.cols && reinterpret_cast<uintptr_t>(o.src) % 16 == 0 &&
                        o.s_b0 % 8 == 0 && o.s_b1 % 8 == 0 && (o.nb == 1 || ((o.b1 == 1 || o.s_b1 > 0) && (o.nb == o.b1 || o.s_b0 > 0)));
        if (ok) {
            o.pitch = o.s_r;
            o.hi = static_cast<const __half*>(o.src);
            o.map_b1 = o.b1;
            o.map_s_b1 = o.s_b1;
            o.map_b0 = o.nb / o.b1;
            o.map_s_b0 = o.s_b0;
        }
        return ok;
    };
    const bool readable = direct(a) && direct(b);
    if (!readable) return gemm_f16_any(ctx, p, epi);
    if (epi != nullptr) {
        // the epilogue adds where it stores 64 whole columns: no K-slices, no ragged edge
        for (const void* q : {static_cast<const void*>(p.out), epi->bias, static_cast<const void*>(epi->biased), static_cast<const void*>(epi->rectified)}) {
            if (reinterpret_cast<uintptr_t>(q) % 16 != 0) return false;
        }
        if (t.splits > 1 || p.n % 64 != 0 || p.b0 * p.b1 != 1) return false;
    }
    size_t bytes = 2048;
    if (t.splits > 1) bytes += static_cast<size_t>(p.b0 * p.b1 * p.m * p.n * t.splits * 4);
    char* ws = static_cast<char*>(ctx->ensure_workspace(bytes));
    ws = reinterpret_cast<char*>(align_up(reinterpret_cast<int64_t>(ws), 1024));
    run_h16(ctx, p, 1, t, a, b, reinterpret_cast<float*>(ws), true, epi != nullptr ? "matmul.tcgen05_f16_bias" : "matmul.tcgen05_f16", epi);
    run_fold<__half>(ctx, p, reinterpret_cast<const float*>(ws), static_cast<int>(t.splits));
    return true;
}

}  // namespace b200
