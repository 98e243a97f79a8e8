// Products of half storage whose rows TMA cannot read as they lie: pitches that are no multiple of 8 halves, addresses off 16 bytes.
//
// They used to run on widened copies: two conversions, the F32 product with its own passes over the operands, a narrowing, and a bias and a relu of
// their own -- 6 to 11 launches, 116 us for a 969x1327x3468 layer whose operations take 5.5.  Here warps of the product's kernel
// bring the halves into shared memory themselves: a warp reads 64 neighbours along the unit-stride axis, a word to a lane,
// and stores them in the 128-byte swizzle that TMA would give the tile.  The arithmetic is gemm_h16.cu's one pass: exact products, fp32 accumulators, one narrowing; a Linear layer's bias and relu are added
// behind it, each narrowing its own result.
//
// 128 x 128 by one CTA, or 256 x 256 by a pair, whichever takes less time in whole waves (2808x7147x621 138 us by single CTAs, 91 by pairs).  Roles as in gemm_inline.cu: warps 0-3 epilogue,
// 4 MMA (in the odd CTA of a pair it passes on that a stage has been filled), 8-23 fill the stages.
#include "gemm.h"

#include <algorithm>

#include <cuda_fp16.h>

#include "gemm_inline.cuh"

namespace b200 {
namespace {

constexpr int kRowsP = 128;   // accumulator lanes
constexpr int kRowsQ = 128;   // of Q, in one CTA
constexpr int kBlockK = 64;   // halves: one 128-byte swizzle row
constexpr int kStageK = 2 * kBlockK;  // of a stage: a handover every other block (2808x7148x621 87 -> 78 us)
constexpr int kStepK = 16;
constexpr int kRows = 16;     // a filling warp's rows of a stage
constexpr int kFirstFiller = 8;
constexpr int kFillers = (kRowsP + kRowsQ) / kRows;
constexpr int kThreads = (kFirstFiller + kFillers) * 32;
constexpr int kTileBytes = kRowsP * kBlockK * 2;
constexpr int kBlockBytes = 2 * kTileBytes;
constexpr int kStageBytes = 2 * kBlockBytes;
constexpr int kStages = 3;
constexpr int kPitch = 36;    // floats: 32 columns of the epilogue's patch
constexpr int kBars = kStages * kStageBytes;
constexpr int kTotal = kBars + 256 + 1024;

struct HalfSide {
    const __half* base;
    int64_t s_b0, s_b1, s_mn, s_k;  // element strides
    int64_t mn;
    int64_t n_batches;
    int words;                      // rows begin on 4 bytes and are whole words
};

struct F16Args {
    HalfSide p, q;  // A with its rows, B with its columns
    int64_t k, b1;
    void* out;      // C (halves), or the f32 partial planes when splits > 1
    int splits;
    const __half* bias;
    __half* biased;
    __half* rectified;
    int64_t m, n;
    UnitPlan units;
    int64_t split_stride;
    uint32_t* status;
};

__device__ __forceinline__ uint32_t load_word(const void* p) {
    uint32_t v;
    asm volatile("ld.global.nc.b32 %0, [%1];" : "=r"(v) : "l"(p));
    return v;
}

// What one lane of a filling warp reads: a pair of halves along the unit-stride axis, sixteen rows across it.  K-major: 64 K of a row, rows eight
// apart.  MN-major: 64 elements of a K-row (an atom), K-rows four apart.  Either way a warp's rows all begin on 4 bytes or all beside them; where they begin
// beside them a lane's word is the second half of its neighbour's pair and the first of its own, and one more word ends the row.  (Pairs put together
// by shuffles instead of two stores of a half: 2808x7147x621 116 -> 111 us.)  A word is only read if it holds an element of the row, so it lies in
// the row's allocation.  Past the matrix' end the last word or row is read again: what a line too many gives lies outside C, and K's end is cleared behind the
// stores.
template <bool MN, bool WORDS>
struct PairFeed {
    static constexpr int kStep = MN ? 4 : 8;
    struct Block {
        uint32_t v[kRows], end;  // lane i of `end`: the word behind row i
        bool beside;
        int left;                // of K, from the block on
    };
    const HalfSide& s;
    int lane, row, atom;
    uint32_t even, odd;  // where the pairs go: their swizzle alternates
    uint32_t before_even, before_odd, end_at;  // where the second half of the neighbour's pair goes, and of the row's last
    const char* at;      // this lane's word of the first row
    int rows_apart, to_end, last_row;  // bytes between its rows, from its word to the one behind the row; the last of the rows that exists
    bool beside;

    __device__ __forceinline__ PairFeed(const HalfSide& side, int t) : s(side) {
        const int w = t >> 5;
        lane = t & 31;
        row = MN ? w >> 1 : w;
        atom = MN ? w & 1 : 0;
        auto place_of = [&](int r, int l) { return static_cast<uint32_t>(atom * kAtomBytes + r * 128 + (((l >> 2) ^ (r & 7)) << 4) + (l & 3) * 4); };
        even = place_of(row, lane);
        odd = place_of(row + kStep, lane);
        before_even = place_of(row, lane - 1) + 2;
        before_odd = place_of(row + kStep, lane - 1) + 2;
        end_at = place_of(row + kStep * (lane & (kRows - 1)), 31) + 2;
        rows_apart = static_cast<int>(kStep * (MN ? s.s_k : s.s_mn) * 2);
    }
    __device__ __forceinline__ void place(int64_t b1, uint32_t batch, uint32_t tile, uint32_t kb, int K) {
        // (the odd CTA's rows may all lie behind the last line)
        const int line0 = min(static_cast<int>(tile * kRowsP), static_cast<int>(s.mn - 1) & ~1);
        const int k0 = min(static_cast<int>(kb * kBlockK), (K - 1) & ~(kBlockK - 1));  // (a stage's second block may lie behind K)
        const int lines = static_cast<int>(s.mn) - line0 - 1, ks = K - k0 - 1;  // behind the tile's first
        const int left = MN ? lines : ks, down = MN ? ks : lines, top = min(row, down);
        int64_t offset = 0;
        if (s.n_batches != 1) {
            const uint32_t bo = batch / static_cast<uint32_t>(b1);
            offset = int64_t(bo) * s.s_b0 + int64_t(batch - bo * static_cast<uint32_t>(b1)) * s.s_b1;
        }
        const uintptr_t start = reinterpret_cast<uintptr_t>(s.base + offset + int64_t(line0 + (MN ? 0 : top)) * s.s_mn + int64_t(k0 + (MN ? top : 0)) * s.s_k);
        beside = !WORDS && (start & 2) != 0;
        const int last = (left + (beside ? 1 : 0)) >> 1, mine = min(32 * atom + lane, last);  // words of the row
        at = reinterpret_cast<const char*>(start & ~uintptr_t(3)) + 4 * mine;
        to_end = (min(32 * atom + 32, last) - mine) * 4;
        last_row = min(kRows - 1, (down - top) / kStep);
    }
    __device__ __forceinline__ void next() { at += kBlockK * s.s_k * 2; }  // (not onto a K-block that reaches past K)
    __device__ __forceinline__ void load(Block& b) const {
        b.beside = beside;
#pragma unroll
        for (int i = 0; i < kRows; ++i) b.v[i] = load_word(at + int64_t(min(i, last_row)) * rows_apart);
        if (!WORDS && beside) b.end = load_word(at + int64_t(min(lane & (kRows - 1), last_row)) * rows_apart + to_end);
    }
    __device__ __forceinline__ uint32_t word(int i) const { return (i & 1 ? odd : even) + (i >> 1) * (2 * kStep * 128); }
    __device__ __forceinline__ void store(uint8_t* to, const Block& b) const {
        if (!WORDS && b.beside) {  // (the same for the whole warp)
            // a word holds elements 2 lane - 1 and 2 lane of the row, and the one behind it element 63
#pragma unroll
            for (int i = 0; i < kRows; ++i) {
                *reinterpret_cast<uint16_t*>(to + word(i)) = static_cast<uint16_t>(b.v[i] >> 16);
                if (lane > 0) *reinterpret_cast<uint16_t*>(to + (i & 1 ? before_odd : before_even) + (i >> 1) * (2 * kStep * 128)) = static_cast<uint16_t>(b.v[i]);
            }
            if (lane < kRows) *reinterpret_cast<uint16_t*>(to + end_at) = static_cast<uint16_t>(b.end);
        } else {
#pragma unroll
            for (int i = 0; i < kRows; ++i) *reinterpret_cast<uint32_t*>(to + word(i)) = b.v[i];
        }
    }
};

template <int CG, bool P_MN, bool Q_MN>
__global__ void __launch_bounds__(kThreads, 1) gemm_f16_any_kernel(const __grid_constant__ F16Args g) {
    constexpr int STAGES = kStages;
    constexpr int BN = CG * kRowsQ;
    constexpr int kAccs = 2;
    constexpr uint32_t kTmemCols = kAccs * BN;
    constexpr uint32_t kIdesc = h16_idesc(CG * kRowsP, BN, P_MN, Q_MN);
    static_assert(8 * (3 * STAGES + 2 * kAccs) <= 256, "barrier block");

    extern __shared__ uint8_t smem_raw[];
    const uint32_t base = (smem_u32(smem_raw) + 1023u) & ~1023u;
    uint8_t* base_ptr = smem_raw + (base - smem_u32(smem_raw));
    const uint32_t bars = base + kBars;
    auto full_bar = [&](int s) { return bars + 8u * s; };
    auto empty_bar = [&](int s) { return bars + 8u * (STAGES + s); };
    auto acc_full = [&](int a) { return bars + 8u * (2 * STAGES + a); };
    auto acc_empty = [&](int a) { return bars + 8u * (2 * STAGES + kAccs + a); };             // the even CTA's
    auto peer_bar = [&](int s) { return bars + 8u * (2 * STAGES + 2 * kAccs + s); };  // the even CTA's: a stage is filled in the odd one
    __shared__ uint32_t tmem_base_slot;
    __shared__ int abort_flag;
    __shared__ __align__(16) float epi_patch[4][32][kPitch];

    const int warp = threadIdx.x >> 5;
    const int lane = threadIdx.x & 31;
    const uint32_t rank = CG == 2 ? cluster_rank() : 0;
    const uint32_t unit0 = blockIdx.x / CG, unit_step = gridDim.x / CG;

    if (threadIdx.x == 0) {
        abort_flag = 0;
        for (int s = 0; s < STAGES; ++s) {
            mbar_init(full_bar(s), kFillers);
            mbar_init(peer_bar(s), 1);
            mbar_init(empty_bar(s), 1);
        }
        for (int a = 0; a < kAccs; ++a) {
            mbar_init(acc_full(a), 1);
            mbar_init(acc_empty(a), 4 * CG);
        }
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 4) {
        tmem_get<CG>(smem_u32(&tmem_base_slot), kTmemCols);
        tc_fence_before();
    }
    __syncthreads();
    if (CG == 2) cluster_sync();  // the other CTA's barriers are initialised
    tc_fence_after();
    const uint32_t tmem_base = tmem_base_slot;
    volatile int* abort_p = &abort_flag;
    pdl_prologue();

    // Registers: a launch of 768 threads has 80 each, and 512 x 88 + 256 x 64 are as many.
    if (warp >= kFirstFiller) {
        // ---------------- fillers ----------------
        set_registers<true, 88>();
        auto fill = [&](auto feed, const int index, const uint32_t tile_at, auto mn_tag) {
            constexpr bool MN = decltype(mn_tag)::value;
            using Block = typename decltype(feed)::Block;
            const int K = static_cast<int>(g.k);
            // where the loads are, a stage ahead of the stores
            uint32_t next_u = unit0, next_block = 0, next_end = 0;
            auto place = [&](const Unit& x, uint32_t block) { feed.place(g.b1, x.batch, (index == 0 ? x.tp : x.tq) * CG + rank, block, K); };
            auto enter = [&] {
                const Unit x = unit_of(g.units, next_u);
                next_block = 2 * x.kb0;
                next_end = 2 * x.kb1;
                place(x, next_block);
            };
            auto request = [&](Block& b) {
                if (next_u >= g.units.n_units) return;
                b.left = K - static_cast<int>(next_block) * kBlockK;
                feed.load(b);
                if (++next_block < next_end) {
                    if (static_cast<int>(next_block + 1) * kBlockK <= K) feed.next();
                    else place(unit_of(g.units, next_u), next_block);
                } else if ((next_u += unit_step) < g.units.n_units) {
                    enter();
                }
            };
            auto store = [&](uint8_t* to, const Block& b) {
                if (b.left <= 0) return;  // (nor is it multiplied)
                feed.store(to, b);
                if (b.left < kBlockK) {
                    // K past the matrix' end (a pair's second half may be another lane's store)
                    __syncwarp();
#pragma unroll 1
                    for (int e = 0; e < 2 * kRows; ++e) {
                        if ((MN ? feed.row + feed.kStep * (e >> 1) : 2 * lane + (e & 1)) < b.left) continue;
                        *reinterpret_cast<uint16_t*>(to + feed.word(e >> 1) + 2 * (e & 1)) = 0;
                    }
                }
            };
            Block b0, b1;
            enter();
            request(b0);
            request(b1);
            uint32_t it = 0;
            bool ok = true;
            for (uint32_t u = unit0; ok && u < g.units.n_units; u += unit_step) {
                const Unit now = unit_of(g.units, u);
                for (uint32_t kb = now.kb0; kb < now.kb1; ++kb, ++it) {
                    const int s = it % STAGES;
                    ok = mbar_wait(empty_bar(s), ((it / STAGES) & 1) ^ 1, abort_p, g.status);
                    if (!ok) break;
                    uint8_t* to = base_ptr + s * kStageBytes + tile_at;
                    store(to, b0);
                    request(b0);
                    store(to + kBlockBytes, b1);
                    request(b1);
                    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
                    __syncwarp();
                    if (lane == 0) mbar_arrive(full_bar(s));
                }
            }
            if (threadIdx.x == kFirstFiller * 32) drain_commits<STAGES>(empty_bar, it, abort_p, g.status);
        };
        const int t = threadIdx.x - kFirstFiller * 32;
        using PMn = std::integral_constant<bool, P_MN>;
        using QMn = std::integral_constant<bool, Q_MN>;
        if (t < kThreads / 3) {
            if (g.p.words) fill(PairFeed<P_MN, true>(g.p, t), 0, 0, PMn());
            else fill(PairFeed<P_MN, false>(g.p, t), 0, 0, PMn());
        } else {
            if (g.q.words) fill(PairFeed<Q_MN, true>(g.q, t - kThreads / 3), 1, kTileBytes, QMn());
            else fill(PairFeed<Q_MN, false>(g.q, t - kThreads / 3), 1, kTileBytes, QMn());
        }
    } else if (warp >= 4) {
        // ---------------- MMA issuer (the even CTA's) ----------------
        set_registers<false, 64>();
        if (warp == 4 && lane == 0) {
            uint32_t it = 0, tile_it = 0;
            bool ok = true;
            for (uint32_t u = unit0; u < g.units.n_units && ok; u += unit_step, ++tile_it) {
                const Unit r = unit_of(g.units, u);
                const int acc = tile_it % kAccs;
                if (rank == 0) {
                    if (!mbar_wait(acc_empty(acc), ((tile_it / kAccs) & 1) ^ 1, abort_p, g.status)) break;
                    tc_fence_after();
                }
                const uint32_t d = tmem_base + acc * BN;
                for (uint32_t kb = r.kb0; kb < r.kb1; ++kb, ++it) {
                    const int s = it % STAGES;
                    ok = mbar_wait(full_bar(s), (it / STAGES) & 1, abort_p, g.status);
                    if (CG == 2 && rank == 1) {
                        // (an arrival across the pair waits for its thread's loads, so it is not for the fillers)
                        if (!ok) break;
                        mbar_arrive_cluster(lead_addr(peer_bar(s)));
                        continue;
                    }
                    if (CG == 2) ok = ok && mbar_wait_cluster(peer_bar(s), (it / STAGES) & 1, abort_p, g.status);
                    if (!ok) break;
                    tc_fence_after();
#pragma unroll
                    for (int j = 0; j < kStageK / kBlockK; ++j) {
                        if (j > 0 && int64_t(kb) * kStageK + j * kBlockK >= g.k) break;
                        const uint32_t at = base + s * kStageBytes + j * kBlockBytes;
                        const uint64_t a = h16_desc<P_MN>(at), b = h16_desc<Q_MN>(at + kTileBytes);
#pragma unroll
                        for (int kk = 0; kk < kBlockK / kStepK; ++kk) {
                            const uint64_t adv_a = static_cast<uint64_t>((P_MN ? kk * kStepK * 128 : kk * kStepK * 2) >> 4);
                            const uint64_t adv_b = static_cast<uint64_t>((Q_MN ? kk * kStepK * 128 : kk * kStepK * 2) >> 4);
                            umma_f16<CG>(d, a + adv_a, b + adv_b, kIdesc, (kb == r.kb0 && j == 0 && kk == 0) ? 0u : 1u);
                        }
                    }
                    commit_all<CG>(empty_bar(s));
                }
                if (ok && rank == 0) commit_all<CG>(acc_full(acc));
            }
        }
    } else {
        // ---------------- epilogue ----------------
        set_registers<false, 64>();
        uint32_t tile_it = 0;
        for (uint32_t u = unit0; u < g.units.n_units; u += unit_step, ++tile_it) {
            const Unit r = unit_of(g.units, u);
            const int acc = tile_it % kAccs;
            if (!mbar_wait_parked(acc_full(acc), (tile_it / kAccs) & 1, abort_p, g.status)) break;
            tc_fence_after();
            const uint32_t t_acc = tmem_base + (static_cast<uint32_t>(warp * 32) << 16) + acc * BN;
            const int64_t p0 = (int64_t(r.tp) * CG + rank) * kRowsP + warp * 32, q0 = int64_t(r.tq) * BN;
            const int64_t p_left = g.m - p0;
            const int64_t at = int64_t(r.split) * g.split_stride + (int64_t(r.batch) * g.m + p0) * g.n + q0;
            float* patch = &epi_patch[warp][0][0];
            const int rows = static_cast<int>(min(int64_t(32), p_left));
#pragma unroll 1
            for (int c = 0; c < BN; c += 32) {
                const int64_t q_left = g.n - (q0 + c);
                if (q_left <= 0 || p_left <= 0) break;  // uniform across the warp
                uint32_t v[32];
                tmem_ld32(t_acc + c, v);
#pragma unroll
                for (int j = 0; j < 8; ++j) {
                    *reinterpret_cast<uint4*>(patch + lane * kPitch + 4 * j) = make_uint4(v[4 * j], v[4 * j + 1], v[4 * j + 2], v[4 * j + 3]);
                }
                __syncwarp();
                if (lane < q_left) {
                    const int64_t o = at + c + lane;
                    if (g.splits > 1) {
                        float* to = static_cast<float*>(g.out) + o;
#pragma unroll 4
                        for (int rl = 0; rl < rows; ++rl) to[int64_t(rl) * g.n] = patch[rl * kPitch + lane];
                    } else {
                        const float bias = g.bias != nullptr ? __half2float(g.bias[q0 + c + lane]) : 0.0F;
#pragma unroll 4
                        for (int rl = 0; rl < rows; ++rl) {
                            // every node narrows its own result: the sum is that of the stored halves
                            const int64_t i = o + int64_t(rl) * g.n;
                            const __half y = __float2half_rn(patch[rl * kPitch + lane]);
                            static_cast<__half*>(g.out)[i] = y;
                            if (g.bias != nullptr) {
                                const __half z = __float2half_rn(__fadd_rn(__half2float(y), bias));
                                g.biased[i] = z;
                                if (g.rectified != nullptr) g.rectified[i] = __half2float(z) <= 0.0F ? __ushort_as_half(0) : z;
                            }
                        }
                    }
                }
                __syncwarp();
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
        for (int i = 0; i < 200; ++i) __nanosleep(1000);  // MMAs in flight end before their memory is given up
        __syncthreads();
    }
    tc_fence_before();
    if (CG == 2) cluster_sync();  // nothing of the pair is addressed after this
    if (warp == 4) {
        tc_fence_after();
        tmem_put<CG>(tmem_base, kTmemCols);
    }
}

// The K-slices' partial planes in split order, and the layer's bias and relu behind them, whose results may lie over `out`.
__global__ void __launch_bounds__(256) fold_f16_kernel(const __grid_constant__ F16Args g, __half* out, const float* __restrict__ part, FastDiv by_n) {
    pdl_prologue();
    const int64_t total = g.split_stride, step = int64_t(gridDim.x) * blockDim.x;
    for (int64_t i = int64_t(blockIdx.x) * blockDim.x + threadIdx.x; i < total; i += step) {
        float s = __ldcg(part + i);
#pragma unroll 4
        for (int k = 1; k < g.splits; ++k) s += __ldcg(part + int64_t(k) * total + i);
        const __half y = __float2half_rn(s);
        out[i] = y;
        if (g.bias != nullptr) {
            const uint32_t col = static_cast<uint32_t>(i) - by_n.div(static_cast<uint32_t>(i)) * by_n.d;
            const __half z = __float2half_rn(__fadd_rn(__half2float(y), __half2float(g.bias[col])));
            g.biased[i] = z;
            if (g.rectified != nullptr) g.rectified[i] = __half2float(z) <= 0.0F ? __ushort_as_half(0) : z;
        }
    }
}

HalfSide side_of(const void* base, const int64_t (&s)[4], int mn_axis, int k_axis, int64_t mn, const GemmProblem& p, bool& is_mn) {
    HalfSide o{};
    const bool one = (s[0] == 0 || p.b0 == 1) && (s[1] == 0 || p.b1 == 1);
    o.base = static_cast<const __half*>(base);
    o.s_b0 = one ? 0 : s[0];
    o.s_b1 = one ? 0 : s[1];
    o.s_mn = s[mn_axis];
    o.s_k = s[k_axis];
    o.mn = mn;
    o.n_batches = one ? 1 : p.b0 * p.b1;
    is_mn = s[mn_axis] == 1 && s[k_axis] != 1;
    const int64_t across = is_mn ? o.s_k : o.s_mn;
    o.words = (is_mn ? mn : p.k) % 2 == 0 && across % 2 == 0 && o.s_b0 % 2 == 0 && o.s_b1 % 2 == 0 && reinterpret_cast<uintptr_t>(base) % 4 == 0;
    return o;
}

}  // namespace

// Any half product with a unit-stride axis in either operand; false: not a case for it.  `p`'s pointers are to halves.
bool gemm_f16_any(b200_ctx* ctx, const GemmProblem& p, const HalfEpilogue* epi) {
    bool mn[2];
    F16Args g{};
    g.p = side_of(p.a, p.a_s, 2, 3, p.m, p, mn[0]);
    g.q = side_of(p.b, p.b_s, 3, 2, p.n, p, mn[1]);
    for (int i = 0; i < 2; ++i) {
        const HalfSide& s = i == 0 ? g.p : g.q;
        if ((mn[i] ? s.s_mn : s.s_k) != 1 || std::abs(mn[i] ? s.s_k : s.s_mn) >= (int64_t(1) << 26) || reinterpret_cast<uintptr_t>(s.base) % 2 != 0) return false;
    }
    const int64_t batches = p.b0 * p.b1, lim = int64_t(1) << 30, k_blocks = ceil_div(p.k, int64_t(kStageK)), out_elems = batches * p.m * p.n;
    if (p.m >= lim || p.n >= lim || p.k >= lim || batches >= lim || out_elems >= (int64_t(1) << 31) || (epi != nullptr && batches != 1)) return false;
    const int sms = ctx->prop.multiProcessorCount;
    // One CTA or a pair, and K-slices: the least time of whole waves.  (us: a stage takes 1.8 in either, for twice the work per CTA in a pair; a pair
    // is not scheduled ahead of the kernel in front of it; slices are written, read and folded.)
    int cg = 0;
    int64_t tiles_p = 0, tiles_q = 0, tiles = 0, splits = 0, kb_per_split = 0;
    double least = 0;
    for (int c = 1; c <= 2; ++c) {
        const int64_t tp = ceil_div(p.m, int64_t(c * kRowsP)), tq = ceil_div(p.n, int64_t(c * kRowsQ)), slots = sms / c;
        int64_t n = 1;
        if (tp * tq * batches < slots && k_blocks >= 4) n = std::max<int64_t>(1, std::min({slots / (tp * tq * batches), k_blocks / 2, int64_t(64)}));
        const int64_t each = ceil_div(k_blocks, n);
        n = ceil_div(k_blocks, each);
        const double us = double(ceil_div(tp * tq * batches * n, slots)) * (1.8 * double(each) + 2.0) + (c == 2 ? 2.0 : 0.0) +
                          (n > 1 ? 3.0 + 1.4e-6 * double(n) * double(out_elems) : 0.0);
        if (cg != 0 && us >= least) continue;
        least = us;
        cg = c;
        tiles_p = tp;
        tiles_q = tq;
        tiles = tp * tq * batches;
        splits = n;
        kb_per_split = each;
    }
    if (tiles * splits >= lim) return false;
    float* partial = nullptr;
    if (splits > 1) {
        char* ws = static_cast<char*>(ctx->ensure_workspace(static_cast<size_t>(out_elems * splits * 4 + 2048)));
        partial = reinterpret_cast<float*>(align_up(reinterpret_cast<int64_t>(ws), 1024));
    }
    g.k = p.k;
    g.b1 = p.b1;
    g.out = splits > 1 ? static_cast<void*>(partial) : static_cast<void*>(p.out);
    g.splits = static_cast<int>(splits);
    if (epi != nullptr) {
        g.bias = static_cast<const __half*>(epi->bias);
        g.biased = static_cast<__half*>(epi->biased);
        g.rectified = static_cast<__half*>(epi->rectified);
    }
    g.m = p.m;
    g.n = p.n;
    g.units = unit_plan(tiles_p, tiles_q, batches, splits, k_blocks, kb_per_split, 16 / cg);
    g.split_stride = out_elems;
    g.status = ctx->d_status;
    int free_sms = sms;
    if (ctx->in_grad_sync_span && ctx->comm_pending) free_sms = std::max(sms - ctx->comm_sms, sms / 2);  // (the others are the all-reduce's)
    const int grid = static_cast<int>(std::min<int64_t>(tiles * splits, free_sms / cg)) * cg;
    auto launch = [&](auto kernel) {
        B200_CUDA_CHECK(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kTotal));
        if (cg == 2) launch_kernel_clustered(ctx, kernel, grid, kThreads, kTotal, cg, false, g);
        else launch_kernel(ctx, kernel, grid, kThreads, kTotal, g);
    };
    auto majors = [&](auto pair) {
        constexpr int CG = decltype(pair)::value;
        if (mn[0] && mn[1]) launch(gemm_f16_any_kernel<CG, true, true>);
        else if (mn[0]) launch(gemm_f16_any_kernel<CG, true, false>);
        else if (mn[1]) launch(gemm_f16_any_kernel<CG, false, true>);
        else launch(gemm_f16_any_kernel<CG, false, false>);
    };
    {
        ProfScope scope(ctx, epi != nullptr ? "matmul.tcgen05_f16_bias" : "matmul.tcgen05_f16");
        if (cg == 2) majors(std::integral_constant<int, 2>());
        else majors(std::integral_constant<int, 1>());
    }
    ctx->count_launch();
    check_last_launch("matmul (tcgen05, half storage of any pitch)");
    if (splits > 1) {
        ProfScope scope(ctx, "matmul.fold");
        launch_kernel(ctx, fold_f16_kernel, grid_for(out_elems, 256), 256, 0, g, reinterpret_cast<__half*>(p.out), static_cast<const float*>(partial),
                      FastDiv(static_cast<uint32_t>(p.n)));
        ctx->count_launch();
        check_last_launch("matmul (fold)");
    }
    return true;
}

}  // namespace b200
