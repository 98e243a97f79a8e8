// fp32 GEMM on the Blackwell tensor cores: tcgen05.mma (kind::tf32) with TMEM
// accumulators, operands staged by TMA, 3xTF32 split emulation.
//
// Arithmetic.  Each fp32 operand x is split into hi = tf32(x) (round to
// nearest) and lo = tf32(x - hi); the product a*b is accumulated in fp32 as
//     a_lo*b_hi + a_hi*b_lo + a_hi*b_hi          (small terms first)
// by three tensor-core MMAs into ONE TMEM accumulator.  The dropped a_lo*b_lo
// term is ~2^-22 relative, so the result carries fp32-grade error.  With
// B200_GEMM_TF32 only a_hi*b_hi is issued (plain TF32, explicit opt-in).
//
// Data layout.  A pre-pass (split_kernel) reads the operands through their own
// strides -- transposed views, broadcast batches, slices: whatever the graph
// hands over -- and writes K-major planes into the context's scratch buffer:
//     A_hi, A_lo : [batches_a * M][Kp]     B_hi, B_lo : [batches_b * N][Kp]
// with Kp = K rounded up to 32 and zero-filled, so every TMA tile is a legal,
// 128-byte-aligned box regardless of the caller's pitches.  A broadcast batch
// (both batch strides 0) is stored once.  An operand whose M (or N) axis is the
// contiguous one -- a transposed view as A, a row-major [K,N] matrix as B -- is
// NOT transposed: its planes keep the [Kp][M or N] layout and the MMA reads them
// through MN-major descriptors, so the split is a dense 128-bit pass.
//
// Main kernel: persistent, one CTA per SM, 6 warps:
//     warp 0   TMA producer: per K-block of 32 floats, 4 boxes
//              (A_hi, A_lo: 128 rows; B_hi, B_lo: BN rows) into a ring of
//              128B-swizzled shared-memory stages, completion on an mbarrier;
//     warp 1   allocates TMEM, one elected lane issues the tcgen05.mma
//              instructions (M=128, N=BN, K=8 each) and commits stage release /
//              accumulator-ready onto mbarriers;
//     warps 2-5  epilogue: tcgen05.ld the 128 x BN fp32 accumulator (each warp
//              its own 32-lane quarter), store to C with bounds checks.
// Two accumulators live in TMEM so the epilogue of tile i overlaps the MMAs of
// tile i+1.  Tiles are walked in groups of 16 M-tiles so the CTAs running at one
// time share operand panels in L2.  A long K with few tiles is split across CTAs
// into fp32 partial planes that a second kernel folds in split order
// (deterministic, no atomics).
//
// Every wait on an mbarrier is bounded: when the limit runs out the kernel
// records kStatusWaitTimedOut in the context's status word, all roles leave
// their loops, TMEM is freed and the kernel returns; the host reports
// B200_TIMEOUT at the next synchronize.
#include "gemm.h"
#include "tcgen05.cuh"

namespace b200 {
namespace {

constexpr int BM = 128;
constexpr int BK = 32;          // floats per K-block = one 128-byte swizzle row
constexpr int UMMA_K = 8;       // tf32
constexpr int kThreads = 192;
constexpr int kProducerThreads = 256;  // direct-operand variant: two groups of four warps
constexpr int kThreadsDirect = kThreads + kProducerThreads;
constexpr int kGroupM = 16;
constexpr int kEpiPitch = 36;   // words per row of the epilogue's staging patch (16-byte aligned rows)
constexpr int kSchedRing = 4;  // published-but-unconsumed tile numbers per CTA

// One block that waits, through the very mbar_wait the GEMM kernels use, on a barrier nobody will
// ever arrive on: the wait runs out after `limit_ns`, records kStatusWaitTimedOut and the kernel
// returns by itself.  Nothing is in flight, nothing faults; it exists so that the path from a
// bounded device wait to B200_TIMEOUT on the host can be exercised.
__global__ void wait_probe_kernel(uint32_t* status, uint64_t limit_ns) {
    __shared__ uint64_t barrier;
    __shared__ int abort_flag;
    if (threadIdx.x == 0) {
        abort_flag = 0;
        mbar_init(smem_u32(&barrier), 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        (void)mbar_wait(smem_u32(&barrier), 0, &abort_flag, status, limit_ns);
    }
}

// ---------------------------------------------------------------------------
// Operand split pre-pass
// ---------------------------------------------------------------------------

__device__ __forceinline__ void split_tf32(float x, float& hi, float& lo) {
    uint32_t h;
    asm("cvt.rna.tf32.f32 %0, %1;" : "=r"(h) : "f"(x));
    float fh = __uint_as_float(h);
    if (isinf(fh) && !isinf(x)) {
        fh = __uint_as_float(__float_as_uint(x) & 0xFFFFE000u);  // rounding overflowed: truncate instead
    }
    float fl = 0.0F;
    if (isfinite(x)) {
        uint32_t l;
        const float rest = x - fh;  // exact
        asm("cvt.rna.tf32.f32 %0, %1;" : "=r"(l) : "f"(rest));
        fl = __uint_as_float(l);
    }
    hi = fh;
    lo = fl;
}

// The same split on the integer pipe.  Conversion instructions issue at a quarter of the rate of
// integer adds, and a K-block of a 128x256 tile needs 24576 of them; adding half a TF32 ulp to
// the magnitude and clearing the 13 low bits is the same round-to-nearest, ties-away rounding
// (a mantissa carry runs into the exponent as it should).  Infinity, NaN and a rounding that
// overflows take the reference routine.
__device__ __forceinline__ void split_tf32_fast(float x, float& hi, float& lo) {
    const uint32_t b = __float_as_uint(x);
    const uint32_t h = (b + 0x1000u) & 0xFFFFE000u;
    if ((h << 1) >= 0xFF000000u) {  // x is infinite or NaN, or hi overflowed
        split_tf32(x, hi, lo);
        return;
    }
    const float fh = __uint_as_float(h);
    const uint32_t r = __float_as_uint(x - fh);  // exact
    hi = fh;
    lo = __uint_as_float((r + 0x1000u) & 0xFFFFE000u);
}

struct SplitArgs {
    const float* src;
    float* hi;
    float* lo;           // null: single-pass TF32
    int64_t b1;          // inner batch extent (outer is implied by the grid)
    int64_t rows, k, kp;
    int64_t s_b0, s_b1, s_r, s_k;  // element strides of src
    int64_t n_batches;
    int64_t out_rows;    // plane rows per batch (>= rows; the extra rows are written as zero)
    int unit, vec;       // dense along K; and every row on 16 bytes
};

// Source rows dense along K: one thread per four K-elements, 128-bit stores and, where every row lies on 16
// bytes, 128-bit loads; no shared memory.
__device__ __forceinline__ void split_rows(const SplitArgs& a) {
    const int64_t kp4 = a.kp / 4;
    const int64_t total = kp4 * a.out_rows * a.n_batches;
    const int64_t step = int64_t(gridDim.x) * blockDim.x;
    for (int64_t i = int64_t(blockIdx.x) * blockDim.x + threadIdx.x; i < total; i += step) {
        const int64_t k4 = i % kp4;
        const int64_t rb = i / kp4;
        const int64_t r = rb % a.out_rows;
        const int64_t b = rb / a.out_rows;
        const int64_t k = k4 * 4;
        float4 v = make_float4(0.0F, 0.0F, 0.0F, 0.0F);
        if (r < a.rows) {
            const float* src = a.src + (b / a.b1) * a.s_b0 + (b % a.b1) * a.s_b1 + r * a.s_r;
            if (a.vec && k + 3 < a.k) {
                v = *reinterpret_cast<const float4*>(src + k);
            } else {
                if (k < a.k) v.x = src[k];
                if (k + 1 < a.k) v.y = src[k + 1];
                if (k + 2 < a.k) v.z = src[k + 2];
                if (k + 3 < a.k) v.w = src[k + 3];
            }
        }
        float4 h, l;
        split_tf32(v.x, h.x, l.x);
        split_tf32(v.y, h.y, l.y);
        split_tf32(v.z, h.z, l.z);
        split_tf32(v.w, h.w, l.w);
        const int64_t o = rb * a.kp + k;
        *reinterpret_cast<float4*>(a.hi + o) = h;
        if (a.lo != nullptr) {
            *reinterpret_cast<float4*>(a.lo + o) = l;
        }
    }
}

// The same with 32-bit indexes, for fewer than kSmallQuads quads: divisions of 64 bits are most of a small matrix' time (64x4096x4096 35.4 us a
// product with them, 34.9 without).  In kernels of its own: with both widths in one, 1000x1433x777, whose standby launch has nothing to
// split, took 36.5 us for 36.2; and large planes are the 64-bit loop's (a CNN's at batch 231 82.4 us with it, 88.5 with this one).
constexpr int64_t kSmallQuads = int64_t(1) << 22;

__device__ __forceinline__ void split_rows_small(const SplitArgs& a) {
    const uint32_t total = static_cast<uint32_t>(a.kp / 4 * a.out_rows * a.n_batches);
    const uint32_t kp4 = static_cast<uint32_t>(a.kp / 4), out_rows = static_cast<uint32_t>(a.out_rows), b1 = static_cast<uint32_t>(a.b1);
    const uint32_t step = static_cast<uint32_t>(gridDim.x) * blockDim.x;
    for (uint32_t i = static_cast<uint32_t>(blockIdx.x) * blockDim.x + threadIdx.x; i < total; i += step) {
        const uint32_t rb = i / kp4, b = rb / out_rows;
        const int64_t k = int64_t(i - rb * kp4) * 4, r = rb - b * out_rows;
        float4 v = make_float4(0.0F, 0.0F, 0.0F, 0.0F);
        if (r < a.rows) {
            const uint32_t bo = b / b1;
            const float* src = a.src + int64_t(bo) * a.s_b0 + int64_t(b - bo * b1) * a.s_b1 + r * a.s_r;
            if (a.vec && k + 3 < a.k) {
                v = *reinterpret_cast<const float4*>(src + k);
            } else {
                if (k < a.k) v.x = src[k];
                if (k + 1 < a.k) v.y = src[k + 1];
                if (k + 2 < a.k) v.z = src[k + 2];
                if (k + 3 < a.k) v.w = src[k + 3];
            }
        }
        float4 h, l;
        split_tf32(v.x, h.x, l.x);
        split_tf32(v.y, h.y, l.y);
        split_tf32(v.z, h.z, l.z);
        split_tf32(v.w, h.w, l.w);
        const int64_t o = int64_t(rb) * a.kp + k;
        *reinterpret_cast<float4*>(a.hi + o) = h;
        if (a.lo != nullptr) {
            *reinterpret_cast<float4*>(a.lo + o) = l;
        }
    }
}

// General layouts, 64x64 (rows x k) tiles through shared memory: global reads follow
// whichever of the two axes has unit stride (so a row-major [K,N] operand is read along N
// and written K-major, i.e. transposed), writes are always dense along k.  16 elements per
// thread in flight in each phase.
constexpr int kSplitTile = 64;

template <int THREADS>
__device__ __forceinline__ void split_tiles(const SplitArgs& a, float (&tile)[kSplitTile][kSplitTile + 1]) {  // tile: [row][k]
    constexpr int kLines = THREADS / kSplitTile;  // of the tile per step
    const int fast = threadIdx.x & 63, slow = threadIdx.x >> 6;
    const int64_t tiles_k = a.kp / kSplitTile + (a.kp % kSplitTile != 0);
    const int64_t tiles_r = (a.rows + kSplitTile - 1) / kSplitTile;
    const int64_t n_tiles = tiles_k * tiles_r * a.n_batches;
    const bool k_fast = a.s_k == 1 || a.s_r != 1;
    for (int64_t t = blockIdx.x; t < n_tiles; t += gridDim.x) {
        const int64_t tk = t % tiles_k;
        const int64_t tr = (t / tiles_k) % tiles_r;
        const int64_t b = t / (tiles_k * tiles_r);
        const float* src = a.src + (b / a.b1) * a.s_b0 + (b % a.b1) * a.s_b1;
        const int64_t r0 = tr * kSplitTile, k0 = tk * kSplitTile;
        const bool full = r0 + kSplitTile <= a.rows && k0 + kSplitTile <= a.k;
        if (k_fast) {
            const float* p = src + (r0 + slow) * a.s_r + (k0 + fast) * a.s_k;
            const int64_t step = kLines * a.s_r;
#pragma unroll
            for (int j = 0; j < kSplitTile / kLines; ++j) {
                const bool ok = full || (r0 + slow + kLines * j < a.rows && k0 + fast < a.k);
                tile[slow + kLines * j][fast] = ok ? p[j * step] : 0.0F;
            }
        } else {
            const float* p = src + (r0 + fast) * a.s_r + (k0 + slow) * a.s_k;
            const int64_t step = kLines * a.s_k;
#pragma unroll
            for (int j = 0; j < kSplitTile / kLines; ++j) {
                const bool ok = full || (r0 + fast < a.rows && k0 + slow + kLines * j < a.k);
                tile[fast][slow + kLines * j] = ok ? p[j * step] : 0.0F;
            }
        }
        __syncthreads();
        if (k0 + fast < a.kp) {
            float* hi = a.hi + (b * a.rows + r0 + slow) * a.kp + k0 + fast;
            float* lo = a.lo != nullptr ? a.lo + (b * a.rows + r0 + slow) * a.kp + k0 + fast : nullptr;
            const int64_t ostep = kLines * a.kp;
#pragma unroll
            for (int j = 0; j < kSplitTile / kLines; ++j) {
                if (full || r0 + slow + kLines * j < a.rows) {
                    float h, l;
                    split_tf32(tile[slow + kLines * j][fast], h, l);
                    hi[j * ostep] = h;
                    if (lo != nullptr) {
                        lo[j * ostep] = l;
                    }
                }
            }
        }
        __syncthreads();
    }
}

__global__ void __launch_bounds__(256) split_rows_kernel(SplitArgs a) {
    pdl_prologue();
    split_rows(a);
}

__global__ void __launch_bounds__(256) split_rows_small_kernel(SplitArgs a) {
    pdl_prologue();
    split_rows_small(a);
}

__global__ void __launch_bounds__(256) split_kernel(SplitArgs a) {
    pdl_prologue();
    __shared__ float tile[kSplitTile][kSplitTile + 1];
    split_tiles<256>(a, tile);
}

struct SplitTwo {
    SplitArgs s[2];
};

// Both operands of a product side by side.
__global__ void __launch_bounds__(256) split_two_kernel(const __grid_constant__ SplitTwo p) {
    pdl_prologue();
    __shared__ float tile[kSplitTile][kSplitTile + 1];
    const SplitArgs& a = p.s[blockIdx.y];
    if (a.unit) split_rows_small(a);
    else split_tiles<256>(a, tile);
}

// Behind a half-term product, in one launch: its operands' strays, or the planes of both for a wide one.  There is mostly little or nothing
// to do, and then few large blocks cost least; for planes they keep as many loads in flight as many small ones.
constexpr int kPairThreads = 1024;

struct SplitPair {
    SplitArgs s[2];
    const uint32_t* done[2];
    RangeGuard guard;
    // the narrow case: strays of both operands
    GemmProblem p;
    const int64_t* strays[2];
    int mn[2];      // the matrix in memory has K rows
    int bcast[2];   // one matrix for every batch
    float* target;
};

// The elements that the half planes leave out (gemm_h16.cu), a few dozen in a large matrix: a row of the product gets the share of its strays
// in A, a column that of its strays in B, in fp32.  Every element of the product is added to by one thread, in the
// order of K: a row with strays takes along what its columns have, and columns leave such rows out.  A block's unit of work is 1024
// elements of one line, so the handful of strays that two N(0,1) matrices of 8192^2 have is one round of the grid.
struct Stray {
    int batch, line, k;  // line: the row of A, the column of B
};

struct StrayLists {
    Stray at[2][kMaxStrays];
    int64_t raw[2][kMaxStrays];
};
static_assert(kPairThreads == 2 * kMaxStrays, "a thread to a stray");

__device__ __forceinline__ int64_t quotient(int64_t a, int64_t b) {
    return ((a | b) >> 32) != 0 ? a / b : int64_t(uint32_t(a) / uint32_t(b));
}

__device__ void add_strays(const SplitPair& w, StrayLists& lists, const uint32_t (&counts)[2]) {
    const GemmProblem& p = w.p;
    const int64_t batches = p.b0 * p.b1;
    const uint32_t tid = threadIdx.x;
    {
        // both lists into the order of the matrix in memory, in which K ascends along a line: half of the block each
        const int o = tid < kMaxStrays ? 0 : 1;
        const uint32_t i = tid - o * kMaxStrays, n = counts[o];
        const int64_t at = i < n ? w.strays[o][i] : 0;
        if (i < n) lists.raw[o][i] = at;
        const int64_t rows = w.s[o].rows, cols = w.s[o].k, rb = quotient(at, cols), c = at - rb * cols;
        const int64_t b = w.s[o].n_batches == 1 ? 0 : quotient(rb, rows), r = rb - b * rows;
        __syncthreads();
        if (i < n) {
            uint32_t rank = 0;
#pragma unroll 1
            for (uint32_t j = 0; j < n; ++j) rank += lists.raw[o][j] < at;
            lists.at[o][rank] = Stray{static_cast<int>(b), static_cast<int>(w.mn[o] ? c : r), static_cast<int>(w.mn[o] ? r : c)};
        }
        __syncthreads();
    }
    const int64_t extent[2] = {p.n, p.m};  // along a line of the product with strays in A, in B
    int64_t tasks[2], chunks[2];
    for (int o = 0; o < 2; ++o) {
        chunks[o] = (extent[o] + kPairThreads - 1) / kPairThreads;
        tasks[o] = chunks[o] * counts[o] * (w.bcast[o] ? batches : 1);
    }
#pragma unroll 1
    for (int64_t t = blockIdx.y * gridDim.x + blockIdx.x; t < tasks[0] + tasks[1]; t += gridDim.x * gridDim.y) {
        const int o = t < tasks[0] ? 0 : 1;
        const int64_t in = o == 0 ? t : t - tasks[0], u = quotient(in, chunks[o]), pos = (in - u * chunks[o]) * kPairThreads + tid;
        const int64_t repeat = quotient(u, counts[o]);
        const uint32_t e = static_cast<uint32_t>(u - repeat * counts[o]);
        const Stray s = lists.at[o][e];
        // the first stray of a line serves the line
        if (__syncthreads_or(tid < e && lists.at[o][tid].line == s.line && lists.at[o][tid].batch == s.batch)) continue;
        if (pos >= extent[o]) continue;
        const int64_t b = w.bcast[o] ? repeat : s.batch, bo = batches == 1 ? 0 : quotient(b, p.b1), bi = b - bo * p.b1;
        const int64_t m = o == 0 ? s.line : pos, n = o == 0 ? pos : s.line;
        const float* a_row = p.a + bo * p.a_s[0] + bi * p.a_s[1] + m * p.a_s[2];
        const float* b_col = p.b + bo * p.b_s[0] + bi * p.b_s[1] + n * p.b_s[3];
        const int a_batch = w.bcast[0] ? 0 : static_cast<int>(b), b_batch = w.bcast[1] ? 0 : static_cast<int>(b);
        auto in_a = [&](int k) {  // whether A has a stray in row m, at k (k < 0: anywhere)
#pragma unroll 1
            for (uint32_t i = 0; i < counts[0]; ++i) {
                const Stray& q = lists.at[0][i];
                if (q.line == m && q.batch == a_batch && (k < 0 || q.k == k)) return true;
            }
            return false;
        };
        if (o == 1 && in_a(-1)) continue;
        float* to = w.target + (b * p.m + m) * p.n + n;
        float sum = *to;
        auto term = [&](int k) { sum = fmaf(__ldg(a_row + k * p.a_s[3]), __ldg(b_col + k * p.b_s[2]), sum); };
        if (o == 0) {
#pragma unroll 1
            for (uint32_t i = e; i < counts[0]; ++i) {
                if (lists.at[0][i].line == m && lists.at[0][i].batch == a_batch) term(lists.at[0][i].k);
            }
        }
#pragma unroll 1
        for (uint32_t i = 0; i < counts[1]; ++i) {
            const Stray& q = lists.at[1][i];
            if (q.line == n && q.batch == b_batch && (o == 1 || !in_a(q.k))) term(q.k);
        }
        *to = sum;
    }
}

__global__ void __launch_bounds__(kPairThreads, 2) split_pair_kernel(const __grid_constant__ SplitPair p) {
    pdl_prologue();
    __shared__ union {
        StrayLists lists;
        float tile[kSplitTile][kSplitTile + 1];
    } sm;
    __shared__ uint32_t counted[2];
    if (threadIdx.x < 2) counted[threadIdx.x] = __ldcg(&(threadIdx.x == 0 ? p.guard.a : p.guard.b)->strays);
    if (!block_wide(p.guard)) {
        const uint32_t counts[2] = {counted[0], counted[1]};
        if (counts[0] + counts[1] != 0) add_strays(p, sm.lists, counts);
        return;
    }
    if (p.done[blockIdx.y] != nullptr && __ldcg(p.done[blockIdx.y]) != 0) return;
    const SplitArgs& a = p.s[blockIdx.y];
    if (a.unit) split_rows(a);
    else split_tiles<kPairThreads>(a, sm.tile);
}

int64_t split_blocks(const SplitArgs& s) {
    if (s.unit) return grid_for(ceil_div((s.kp / 4) * s.out_rows * s.n_batches, 2), 256);
    return grid_for(ceil_div(s.kp, kSplitTile) * ceil_div(s.rows, kSplitTile) * s.n_batches, 1, 8);
}

void launch_split(b200_ctx* ctx, const SplitArgs& s, const char* label) {
    ProfScope scope(ctx, label);
    if (s.unit && s.kp / 4 * s.out_rows * s.n_batches < kSmallQuads) launch_kernel(ctx, split_rows_small_kernel, static_cast<unsigned>(split_blocks(s)), 256, 0, s);
    else if (s.unit) launch_kernel(ctx, split_rows_kernel, static_cast<unsigned>(split_blocks(s)), 256, 0, s);
    else launch_kernel(ctx, split_kernel, static_cast<unsigned>(split_blocks(s)), 256, 0, s);
    ctx->count_launch();
}

// ---------------------------------------------------------------------------
// Main kernel
// ---------------------------------------------------------------------------

struct TcArgs {
    float* out;            // C, or the partial planes when splits > 1
    int64_t m, n;
    int64_t batches;       // B0*B1
    int64_t a_batch_rows;  // rows between consecutive batches in the A planes (0: broadcast)
    int64_t b_batch_rows;
    int64_t k_blocks;      // Kp / 32
    int64_t kb_per_split;
    int splits;
    int64_t split_stride;  // elements between partial planes
    int64_t tiles_m, tiles_n;
    int group_m;           // M-tiles walked together before moving along N (L2 reuse of the B tiles)
    uint32_t* status;
    // Dynamic tile order: null = every CTA walks units blockIdx.x, +gridDim.x, ... ; otherwise a
    // zeroed counter from which CTAs draw their units after the first, so a CTA that starts late
    // or shares its SM with another kernel (an all-reduce) simply takes fewer tiles.
    unsigned int* sched;
    RangeGuard guard;
    uint32_t* done[2];  // (guarded: set once the planes before this launch are known to be written)
};

// Direct-operand variant: TMA brings the fp32 operand tiles themselves into the `hi` slots of a
// stage (through tensor maps over the caller's matrices: same swizzles, zero fill past the
// edges), eight converter warps split them in place into hi and lo, and only then is the stage
// handed to the MMA warp.  No plane ever exists in HBM: the kernel reads 4 bytes per operand
// element instead of 8, and the split pre-pass (4 read + 8 written) disappears.  It costs
// shared-memory bandwidth (one more read and write of every tile), so it is for products the
// plane scheme would leave waiting on HBM, not for the large compute-bound ones.
struct DirectArgs {
    int64_t b1;          // inner batch extent
    int a_bcast, b_bcast;
};

template <int BN, int STAGES>
struct Smem {
    static constexpr int kABytes = BM * BK * 4;  // one A plane tile
    static constexpr int kBBytes = BN * BK * 4;
    static constexpr int kStageBytes = 2 * kABytes + 2 * kBBytes;
    static constexpr int kBarrierBytes = 256;
    static constexpr int kTotal = STAGES * kStageBytes + kBarrierBytes + 1024;  // + alignment slack
};

template <int BN, int STAGES, bool THREE_PASS, bool A_MN, bool B_MN, bool DIRECT>
__global__ void __launch_bounds__(DIRECT ? kThreadsDirect : kThreads, 1)
gemm_tc_kernel(const __grid_constant__ CUtensorMap map_a_hi, const __grid_constant__ CUtensorMap map_a_lo,
               const __grid_constant__ CUtensorMap map_b_hi, const __grid_constant__ CUtensorMap map_b_lo,
               TcArgs g, DirectArgs da) {
    using S = Smem<BN, STAGES>;
    constexpr uint32_t kTmemCols = 2 * BN < 32 ? 32 : 2 * BN;
    constexpr uint32_t kIdesc = make_idesc(BM, BN, A_MN, B_MN);
    constexpr uint32_t kStageTx = THREE_PASS ? S::kStageBytes : (S::kABytes + S::kBBytes);

    extern __shared__ uint8_t smem_raw[];
    const uint32_t base = (smem_u32(smem_raw) + 1023u) & ~1023u;
    const uint32_t bars = base + STAGES * S::kStageBytes;
    // barrier slots (8 bytes each): full[STAGES], empty[STAGES], acc_full[2], acc_empty[2]
    auto full_bar = [&](int s) { return bars + 8u * s; };
    auto empty_bar = [&](int s) { return bars + 8u * (STAGES + s); };
    auto acc_full = [&](int a) { return bars + 8u * (2 * STAGES + a); };
    auto acc_empty = [&](int a) { return bars + 8u * (2 * STAGES + 2 + a); };
    // dynamic tile order: the producer publishes each next unit through a small ring
    auto sched_full = [&](int r) { return bars + 8u * (2 * STAGES + 4 + r); };
    auto sched_empty = [&](int r) { return bars + 8u * (2 * STAGES + 4 + kSchedRing + r); };
    auto raw_bar = [&](int s) { return bars + 8u * (2 * STAGES + 4 + 2 * kSchedRing + s); };  // direct: fp32 tile landed
    __shared__ int sched_ring[kSchedRing];
    __shared__ uint32_t tmem_base_slot;
    __shared__ int abort_flag;
    __shared__ __align__(16) float epi_patch[4][32][kEpiPitch];  // one transposing patch per epilogue warp

    const int warp = threadIdx.x >> 5;
    const int lane = threadIdx.x & 31;

    if (threadIdx.x == 0) {
        abort_flag = 0;
        for (int s = 0; s < STAGES; ++s) {
            // TMA: one arrival with the byte count; direct: every thread of a producer group
            mbar_init(full_bar(s), DIRECT ? kProducerThreads : 1);
            mbar_init(empty_bar(s), 1);
            mbar_init(raw_bar(s), 1);
        }
        for (int a = 0; a < 2; ++a) {
            mbar_init(acc_full(a), 1);
            mbar_init(acc_empty(a), 4);
        }
        for (int r = 0; r < kSchedRing; ++r) {
            mbar_init(sched_full(r), 1);
            mbar_init(sched_empty(r), 5);  // the MMA thread and the four epilogue warps
        }
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    }
    if (warp == 1) {
        tmem_alloc(smem_u32(&tmem_base_slot), kTmemCols);
        tc_fence_before();
    }
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem_base = tmem_base_slot;
    volatile int* abort_p = &abort_flag;
    // barriers and tensor memory are set up: only now wait for the previous kernel (the operand
    // split, usually), so this kernel's set-up runs under that kernel's tail
    pdl_prologue();

    const int64_t tiles_per_batch = g.tiles_m * g.tiles_n;
    const bool idle = g.guard.a != nullptr && !block_wide(g.guard);
    const int64_t n_units = idle ? 0 : tiles_per_batch * g.batches * g.splits;
    if (n_units > 0 && blockIdx.x == 0 && threadIdx.x < 2 && g.done[threadIdx.x] != nullptr) *g.done[threadIdx.x] = 1;

    // unit -> (split, batch, m tile, n tile); M-tiles walked in groups of kGroupM
    auto decode = [&](int64_t u, int& split, int64_t& batch, int64_t& tm, int64_t& tn) {
        split = static_cast<int>(u % g.splits);
        int64_t t = u / g.splits;
        batch = t / tiles_per_batch;
        t -= batch * tiles_per_batch;
        const int64_t group_size = int64_t(g.group_m) * g.tiles_n;
        const int64_t group = t / group_size;
        const int64_t first_m = group * g.group_m;
        const int64_t rows_in_group = min(int64_t(g.group_m), g.tiles_m - first_m);
        const int64_t in_group = t - group * group_size;
        tm = first_m + in_group % rows_in_group;
        tn = in_group / rows_in_group;
    };

    const bool dynamic = g.sched != nullptr;
    // unit after the t-th one of this CTA, for the MMA thread and the epilogue warps (-1: none)
    auto next_unit = [&](int64_t u, uint32_t t, bool single_thread) -> int64_t {
        if (!dynamic) {
            u += gridDim.x;
            return u < n_units ? u : -1;
        }
        const int r = t % kSchedRing;
        if (!mbar_wait(sched_full(r), (t / kSchedRing) & 1, abort_p, g.status)) {
            return -1;
        }
        const int v = *reinterpret_cast<volatile int*>(&sched_ring[r]);
        if (!single_thread) {
            __syncwarp();
        }
        if (single_thread || lane == 0) {
            mbar_arrive(sched_empty(r));
        }
        return v;
    };

    if (DIRECT && warp >= 6) {
        // ---------------- converters: split the fp32 tiles of each stage in place ----------------
        const int tc = static_cast<int>(threadIdx.x) - kThreads;  // 0 .. kProducerThreads-1
        uint32_t it = 0;
        bool ok = true;
        for (int64_t u = blockIdx.x; u < n_units && ok; u += gridDim.x) {
            int split;
            int64_t batch, tm, tn;
            decode(u, split, batch, tm, tn);
            const int64_t kb0 = int64_t(split) * g.kb_per_split;
            const int64_t kb1 = min(kb0 + g.kb_per_split, g.k_blocks);
            for (int64_t kb = kb0; kb < kb1; ++kb, ++it) {
                const int s = it % STAGES;
                const uint32_t ph = (it / STAGES) & 1;
                if (!mbar_wait(raw_bar(s), ph, abort_p, g.status)) {
                    ok = false;
                    break;
                }
                // The split is elementwise, so the tile's swizzle is irrelevant here: every float
                // of a hi slot becomes hi in place and lo at the same offset of the lo slot.  All
                // of a thread's vectors are loaded before any is stored, so the shared-memory
                // latency is paid once per stage.
                uint8_t* stage_ptr = smem_raw + (base - smem_u32(smem_raw)) + s * S::kStageBytes;
                constexpr int NA = S::kABytes / 16 / kProducerThreads;
                constexpr int NB = S::kBBytes / 16 / kProducerThreads;
                static_assert(NA >= 1 && NB >= 1, "tile smaller than the converter group");
                float4 v[NA + NB];
                float4* a_hi = reinterpret_cast<float4*>(stage_ptr) + tc;
                float4* a_lo = reinterpret_cast<float4*>(stage_ptr + S::kABytes) + tc;
                float4* b_hi = reinterpret_cast<float4*>(stage_ptr + 2 * S::kABytes) + tc;
                float4* b_lo = reinterpret_cast<float4*>(stage_ptr + 2 * S::kABytes + S::kBBytes) + tc;
#pragma unroll
                for (int j = 0; j < NA; ++j) v[j] = a_hi[j * kProducerThreads];
#pragma unroll
                for (int j = 0; j < NB; ++j) v[NA + j] = b_hi[j * kProducerThreads];
#pragma unroll
                for (int j = 0; j < NA + NB; ++j) {
                    float4 h, l;
                    split_tf32_fast(v[j].x, h.x, l.x);
                    split_tf32_fast(v[j].y, h.y, l.y);
                    split_tf32_fast(v[j].z, h.z, l.z);
                    split_tf32_fast(v[j].w, h.w, l.w);
                    float4* hi = j < NA ? a_hi + j * kProducerThreads : b_hi + (j - NA) * kProducerThreads;
                    float4* lo = j < NA ? a_lo + j * kProducerThreads : b_lo + (j - NA) * kProducerThreads;
                    *hi = h;
                    if (THREE_PASS) {
                        *lo = l;
                    }
                }
                // generic-proxy stores must be visible to the tensor core's async-proxy reads
                asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
                mbar_arrive(full_bar(s));
            }
        }
    } else if (warp == 0) {
        // ---------------- TMA producer ----------------
        if (lane == 0) {
            uint32_t it = 0;
            uint32_t t = 0;
            bool ok = true;
            for (int64_t u = blockIdx.x; u >= 0 && u < n_units && ok; ++t) {
                // draw the next unit now; its value is needed only after this tile's loads
                int64_t nxt = u + gridDim.x;
                if (dynamic) {
                    nxt = int64_t(gridDim.x) + atomicAdd(g.sched, 1u);
                }
                int split;
                int64_t batch, tm, tn;
                decode(u, split, batch, tm, tn);
                // K-major plane: coordinates (k, plane row); MN-major plane: (m or n, plane K-row)
                const int a_base = static_cast<int>(batch * g.a_batch_rows);
                const int b_base = static_cast<int>(batch * g.b_batch_rows);
                const int m0 = static_cast<int>(tm * BM), n0 = static_cast<int>(tn * BN);
                const int64_t kb0 = int64_t(split) * g.kb_per_split;
                const int64_t kb1 = min(kb0 + g.kb_per_split, g.k_blocks);
                for (int64_t kb = kb0; kb < kb1; ++kb, ++it) {
                    const int s = it % STAGES;
                    const uint32_t ph = (it / STAGES) & 1;
                    if (!mbar_wait(empty_bar(s), ph ^ 1, abort_p, g.status)) {
                        ok = false;
                        break;
                    }
                    const uint32_t stage = base + s * S::kStageBytes;
                    const int kc = static_cast<int>(kb * BK);
                    if (DIRECT) {
                        // fp32 tiles of the caller's matrices into the hi slots; coordinates are
                        // (unit-stride axis, other axis, inner batch, outer batch)
                        const uint32_t rbar = raw_bar(s);
                        mbar_arrive_expect_tx(rbar, S::kABytes + S::kBBytes);
                        const int64_t bo = batch / da.b1, bi = batch - bo * da.b1;
                        const int a1 = da.a_bcast ? 0 : static_cast<int>(bi), a0 = da.a_bcast ? 0 : static_cast<int>(bo);
                        const int b1c = da.b_bcast ? 0 : static_cast<int>(bi), b0c = da.b_bcast ? 0 : static_cast<int>(bo);
                        if (A_MN) {
#pragma unroll
                            for (int atom = 0; atom < BM / 32; ++atom) {
                                tma_load_4d(stage + atom * kMnAtomBytes, &map_a_hi, rbar, m0 + 32 * atom, kc, a1, a0);
                            }
                        } else {
                            tma_load_4d(stage, &map_a_hi, rbar, kc, m0, a1, a0);
                        }
                        const uint32_t bdst = stage + 2 * S::kABytes;
                        if (B_MN) {
#pragma unroll
                            for (int atom = 0; atom < BN / 32; ++atom) {
                                tma_load_4d(bdst + atom * kMnAtomBytes, &map_b_hi, rbar, n0 + 32 * atom, kc, b1c, b0c);
                            }
                        } else {
                            tma_load_4d(bdst, &map_b_hi, rbar, kc, n0, b1c, b0c);
                        }
                        continue;
                    }
                    const uint32_t bar = full_bar(s);
                    mbar_arrive_expect_tx(bar, kStageTx);
                    auto load_a = [&](uint32_t dst, const CUtensorMap* map) {
                        if (A_MN) {
#pragma unroll
                            for (int atom = 0; atom < BM / 32; ++atom) {
                                tma_load_2d(dst + atom * kMnAtomBytes, map, bar, m0 + 32 * atom, a_base + kc);
                            }
                        } else {
                            tma_load_2d(dst, map, bar, kc, a_base + m0);
                        }
                    };
                    auto load_b = [&](uint32_t dst, const CUtensorMap* map) {
                        if (B_MN) {
#pragma unroll
                            for (int atom = 0; atom < BN / 32; ++atom) {
                                tma_load_2d(dst + atom * kMnAtomBytes, map, bar, n0 + 32 * atom, b_base + kc);
                            }
                        } else {
                            tma_load_2d(dst, map, bar, kc, b_base + n0);
                        }
                    };
                    load_a(stage, &map_a_hi);
                    load_b(stage + 2 * S::kABytes, &map_b_hi);
                    if (THREE_PASS) {
                        load_a(stage + S::kABytes, &map_a_lo);
                        load_b(stage + 2 * S::kABytes + S::kBBytes, &map_b_lo);
                    }
                }
                if (dynamic && ok) {
                    const int r = t % kSchedRing;
                    if (!mbar_wait(sched_empty(r), ((t / kSchedRing) & 1) ^ 1, abort_p, g.status)) {
                        break;
                    }
                    *reinterpret_cast<volatile int*>(&sched_ring[r]) = nxt < n_units ? static_cast<int>(nxt) : -1;
                    mbar_arrive(sched_full(r));
                }
                u = nxt;
            }
            drain_commits<STAGES>(empty_bar, it, abort_p, g.status);
        }
    } else if (warp == 1) {
        // ---------------- MMA issuer ----------------
        if (lane == 0) {
            uint32_t it = 0;
            uint32_t tile_it = 0;
            bool ok = true;
            for (int64_t u = blockIdx.x; u >= 0 && u < n_units && ok; u = next_unit(u, tile_it, true), ++tile_it) {
                int split;
                int64_t batch, tm, tn;
                decode(u, split, batch, tm, tn);
                const int acc = tile_it & 1;
                const uint32_t aph = (tile_it >> 1) & 1;
                if (!mbar_wait(acc_empty(acc), aph ^ 1, abort_p, g.status)) {
                    break;
                }
                tc_fence_after();
                const uint32_t d_tmem = tmem_base + acc * BN;
                const int64_t kb0 = int64_t(split) * g.kb_per_split;
                const int64_t kb1 = min(kb0 + g.kb_per_split, g.k_blocks);
                for (int64_t kb = kb0; kb < kb1; ++kb, ++it) {
                    const int s = it % STAGES;
                    const uint32_t ph = (it / STAGES) & 1;
                    if (!mbar_wait(full_bar(s), ph, abort_p, g.status)) {
                        ok = false;
                        break;
                    }
                    tc_fence_after();
                    const uint32_t stage = base + s * S::kStageBytes;
                    const uint64_t a_hi = operand_desc<A_MN>(stage);
                    const uint64_t a_lo = operand_desc<A_MN>(stage + S::kABytes);
                    const uint64_t b_hi = operand_desc<B_MN>(stage + 2 * S::kABytes);
                    const uint64_t b_lo = operand_desc<B_MN>(stage + 2 * S::kABytes + S::kBBytes);
#pragma unroll
                    for (int kk = 0; kk < BK / UMMA_K; ++kk) {
                        // one K step: +32 bytes inside the swizzle row (K-major), +8 K-rows (MN-major)
                        const uint64_t adv_a = static_cast<uint64_t>((A_MN ? kk * 1024 : kk * UMMA_K * 4) >> 4);
                        const uint64_t adv_b = static_cast<uint64_t>((B_MN ? kk * 1024 : kk * UMMA_K * 4) >> 4);
                        const uint32_t first = (kb == kb0 && kk == 0) ? 0u : 1u;
                        if (THREE_PASS) {
                            umma_tf32(d_tmem, a_lo + adv_a, b_hi + adv_b, kIdesc, first);
                            umma_tf32(d_tmem, a_hi + adv_a, b_lo + adv_b, kIdesc, 1u);
                            umma_tf32(d_tmem, a_hi + adv_a, b_hi + adv_b, kIdesc, 1u);
                        } else {
                            umma_tf32(d_tmem, a_hi + adv_a, b_hi + adv_b, kIdesc, first);
                        }
                    }
                    umma_commit(empty_bar(s));  // the stage is free once these MMAs have read it
                }
                if (ok) {
                    umma_commit(acc_full(acc));
                }
            }
        }
    } else {
        // ---------------- epilogue (warps 2..5) ----------------
        const int quarter = warp & 3;  // TMEM lanes 32*quarter .. +31 belong to this warp
        uint32_t tile_it = 0;
        bool ok = true;
        for (int64_t u = blockIdx.x; u >= 0 && u < n_units && ok; u = next_unit(u, tile_it, false), ++tile_it) {
            int split;
            int64_t batch, tm, tn;
            decode(u, split, batch, tm, tn);
            const int acc = tile_it & 1;
            const uint32_t aph = (tile_it >> 1) & 1;
            if (!mbar_wait(acc_full(acc), aph, abort_p, g.status)) {
                break;
            }
            tc_fence_after();
            const int64_t col0 = tn * BN;
            const bool vec_ok = (g.n % 4 == 0) && ((reinterpret_cast<uintptr_t>(g.out) & 15) == 0) &&
                                ((g.split_stride % 4) == 0);
            const bool warp_rows_live = tm * BM + quarter * 32 < g.m;  // else nothing of this warp's is stored
#pragma unroll 2
            for (int c = 0; c < BN / 32; ++c) {
                if (col0 + c * 32 >= g.n || !warp_rows_live) {
                    break;  // uniform across the warp
                }
                uint32_t r[32];
                tmem_ld32(tmem_base + (static_cast<uint32_t>(quarter * 32) << 16) + acc * BN + c * 32, r);
                const int64_t left = g.n - (col0 + c * 32);
                if (vec_ok && left >= 32) {
                    // Each lane holds 32 columns of ITS row, so storing from here makes every warp
                    // instruction touch 32 different rows (32 wavefronts for 512 bytes).  The chunk
                    // goes through a 32 x 36-word patch of shared memory instead and leaves as four
                    // 128-byte row segments per instruction; both the row-wise writes and the
                    // quarter-warp-per-row reads of the patch are conflict-free.
                    float* patch = &epi_patch[quarter][0][0];
#pragma unroll
                    for (int j = 0; j < 8; ++j) {
                        float4 v;
                        v.x = __uint_as_float(r[4 * j]);
                        v.y = __uint_as_float(r[4 * j + 1]);
                        v.z = __uint_as_float(r[4 * j + 2]);
                        v.w = __uint_as_float(r[4 * j + 3]);
                        *reinterpret_cast<float4*>(patch + lane * kEpiPitch + 4 * j) = v;
                    }
                    __syncwarp();
                    const int sub = lane >> 3, seg = lane & 7;
                    const int64_t row_base = tm * BM + quarter * 32;
                    float* tile_dst = g.out + int64_t(split) * g.split_stride + (batch * g.m + row_base) * g.n + col0 +
                                      c * 32 + seg * 4;
#pragma unroll
                    for (int i = 0; i < 8; ++i) {
                        const int rl = i * 4 + sub;
                        if (row_base + rl < g.m) {
                            const float4 v = *reinterpret_cast<const float4*>(patch + rl * kEpiPitch + seg * 4);
                            *reinterpret_cast<float4*>(tile_dst + int64_t(rl) * g.n) = v;
                        }
                    }
                    __syncwarp();
                    continue;
                }
                // a ragged right edge, or rows that do not begin on 16 bytes: a row's 32 columns per store
                float* patch = &epi_patch[quarter][0][0];
#pragma unroll
                for (int j = 0; j < 8; ++j) {
                    *reinterpret_cast<uint4*>(patch + lane * kEpiPitch + 4 * j) = make_uint4(r[4 * j], r[4 * j + 1], r[4 * j + 2], r[4 * j + 3]);
                }
                __syncwarp();
                const int64_t row_base = tm * BM + quarter * 32;
                if (lane < left) {
                    const int rows = static_cast<int>(min(int64_t(32), g.m - row_base));
                    float* q = g.out + int64_t(split) * g.split_stride + (batch * g.m + row_base) * g.n + col0 + c * 32 + lane;
                    for (int rl = 0; rl < rows; ++rl) {
                        *q = patch[rl * kEpiPitch + lane];
                        q += g.n;
                    }
                }
                __syncwarp();
            }
            tc_fence_before();
            __syncwarp();
            if (lane == 0) {
                mbar_arrive(acc_empty(acc));
            }
        }
    }

    __syncthreads();
    if (abort_flag != 0) {
        // give copies that may still be in flight time to land before the CTA retires
        for (int i = 0; i < 200; ++i) {
            __nanosleep(1000);
        }
        __syncthreads();
    }
    if (warp == 1) {
        tc_fence_after();
        tmem_dealloc(tmem_base, kTmemCols);
    }
}

// ---------------------------------------------------------------------------
// Streamed-operand kernel: products bound by HBM, not by the tensor pipe
// ---------------------------------------------------------------------------
//
// C[b][m][n] = sum_k W[b][m][k] * S[b][k][n] with a SMALL W (few rows: a skinny left operand,
// convolution weights broadcast over the batch) and a LARGE S whose n axis is contiguous
// (a row-major [K][N] matrix, the column tensor of a convolution).  The plane scheme reads S,
// writes its two TF32 planes and reads them again -- five times S's bytes -- which is what
// bounds such a product.  Here S crosses HBM exactly once, as fp32:
//
//   * the product is computed transposed, D[n][m] = sum_k S[k][n] W[m][k], so that S is the
//     tensor core's A operand, and A may come from TENSOR MEMORY instead of shared memory;
//   * two producer warps: one brings [32 k][128 n] fp32 tiles of S (tensor map over the caller's
//     own matrix, zero fill past the edges) into a ring of 6 to 8 slots, the other the matching
//     K-blocks of W's planes into a ring of 4.  The rings are separate because their lifetimes
//     are: S's slot is free again as soon as the converters have read it, W's stays until the
//     MMAs that read it have finished.  (Measured: the deeper ring for S changes no time -- the
//     loop is bound by the rate at which tcgen05.mma instructions issue, about 98 cycles each
//     with A in tensor memory, twelve per K-block -- so its depth is headroom, not a tuning knob.)
//   * sixteen converter warps read their lane's column of the S tile (lane = n, conflict-free),
//     split every value into hi/lo in registers and put both into tensor memory with
//     tcgen05.st -- 64 columns per stage: the streamed operand never touches shared memory
//     again and no converted copy of it exists anywhere;
//   * warp 1 issues tcgen05.mma with A = [tmem] (128 lanes x 8 columns per K-step) and B = W's
//     plane tile in shared memory, three passes into one fp32 accumulator as above;
//   * warps 2-5 read the accumulator (lane = n, columns = m): for every m one warp instruction
//     stores 32 consecutive n, 128 bytes, straight from registers.
//
// S may also lie with its K axis contiguous (the transposed view of an [N][K] matrix: a Linear
// layer's weight in the forward product, the column tensor in a convolution's weight gradient).
// Then the tile is [128 n][32 k], fetched with the 128-byte swizzle so that a lane reading its own
// row (lane = n) meets no bank conflict, and everything after the converter is unchanged.
//
// W may have more rows than one accumulator holds: its 128-row chunks are separate units that run
// side by side on neighbouring SMs, so S's tile is fetched from HBM once and from L2 after that.
//
// When N is shorter than 128 and W is broadcast over the batch, one tile spans several batches
// (lanes = batch x n).  K is split across CTAs when the tiles alone cannot fill the machine, into
// partial planes that a second launch folds in split order.  (Folded in the same launch by the warp that arrived last
// at its quarter of a tile, 64 x 4096 x 4096 took 10 us longer: one warp per quarter adds up what the whole
// machine reads in 3 us.)
constexpr int kStreamStages = 4;          // W's ring in shared memory and S's ring in tensor memory
constexpr int kStreamConverters = 16;     // converter warps: four per tensor-memory lane quarter, 8 K columns each
constexpr int kStreamThreads = (7 + kStreamConverters) * 32;  // + two TMA warps, MMA and four epilogue warps
constexpr int kStreamTileBytes = BK * 128 * 4;  // one fp32 tile of S: 32 K-rows x 128 lanes
constexpr uint32_t kStreamTmemCols = 512;

struct StreamArgs {
    float* out;            // C, or the partial planes when splits > 1
    int64_t m, n;          // per batch
    int64_t batches;
    int64_t w_batch_rows;  // rows between consecutive batches in W's planes (0: broadcast)
    int64_t k_blocks, kb_per_split;
    int splits;
    int64_t split_stride;  // elements between partial planes
    int64_t tiles_m, tiles_n;
    int nt;                // n extent of one batch inside a tile (128, or N when N < 128)
    int bpt;               // batches per tile (nt * bpt == 128 when bpt > 1)
    int64_t batch_groups;  // ceil(batches / bpt)
    uint32_t* status;
};


__device__ __forceinline__ void umma_tf32_ts(uint32_t tmem_d, uint32_t tmem_a, uint64_t bdesc, uint32_t idesc,
                                             uint32_t accumulate) {
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::tf32 [%0], [%1], %2, %3, p;\n\t}"
        ::"r"(tmem_d), "r"(tmem_a), "l"(bdesc), "r"(idesc), "r"(accumulate)
        : "memory");
}

__device__ __forceinline__ void tmem_st8(uint32_t taddr, const uint32_t (&r)[8]) {
    __syncwarp();
    asm volatile(
        "tcgen05.st.sync.aligned.32x32b.x8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};"
        ::"r"(taddr), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7])
        : "memory");
}

__device__ __forceinline__ void tma_load_3d(uint32_t dst, const CUtensorMap* map, uint32_t bar, int c0, int c1,
                                            int c2) {
    asm volatile(
        "cp.async.bulk.tensor.3d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5}], [%2];"
        ::"r"(dst), "l"(reinterpret_cast<uint64_t>(map)), "r"(bar), "r"(c0), "r"(c1), "r"(c2)
        : "memory");
}

template <int BNW>
struct StreamSmem {
    static constexpr int kWBytes = BNW * BK * 4;  // one plane tile of W
    static constexpr int kWStage = 2 * kWBytes;   // hi and lo
    static constexpr int kSlots = BNW <= 64 ? 8 : 6;  // fp32 tiles of S in flight (besides the 4 in tensor memory)
    static constexpr int kWBase = kSlots * kStreamTileBytes;
    static constexpr int kBars = kWBase + kStreamStages * kWStage;
    static constexpr int kTotal = kBars + 256 + 1024;
};

template <int BNW, bool THREE_PASS, bool W_MN, bool S_KM>
__global__ void __launch_bounds__(kStreamThreads, 1)
gemm_stream_kernel(const __grid_constant__ CUtensorMap map_s, const __grid_constant__ CUtensorMap map_w_hi,
                   const __grid_constant__ CUtensorMap map_w_lo, StreamArgs g) {
    using S = StreamSmem<BNW>;
    constexpr int STAGES = kStreamStages;
    constexpr uint32_t kIdesc = make_idesc(BM, BNW, false, W_MN);
    constexpr int SLOTS = S::kSlots;
    constexpr uint32_t kWTx = (THREE_PASS ? 2 : 1) * S::kWBytes;
    constexpr uint32_t kStageCol0 = 2 * BNW;  // tensor-memory columns: two accumulators, then the S stages
    static_assert(8 * (2 * SLOTS + 3 * STAGES + 4) <= 256, "barrier block");

    extern __shared__ uint8_t smem_raw[];
    const uint32_t base = (smem_u32(smem_raw) + 1023u) & ~1023u;
    uint8_t* base_ptr = smem_raw + (base - smem_u32(smem_raw));
    const uint32_t bars = base + S::kBars;
    auto full_bar = [&](int s) { return bars + 8u * s; };                    // W's planes landed
    auto empty_bar = [&](int s) { return bars + 8u * (STAGES + s); };        // the stage's MMAs are done
    auto conv_bar = [&](int s) { return bars + 8u * (2 * STAGES + s); };     // S is in tensor memory
    auto acc_full = [&](int a) { return bars + 8u * (3 * STAGES + a); };
    auto acc_empty = [&](int a) { return bars + 8u * (3 * STAGES + 2 + a); };
    auto s_full = [&](int j) { return bars + 8u * (3 * STAGES + 4 + j); };            // an fp32 tile of S landed
    auto s_empty = [&](int j) { return bars + 8u * (3 * STAGES + 4 + SLOTS + j); };   // the converters have read it
    __shared__ uint32_t tmem_base_slot;
    __shared__ int abort_flag;

    const int warp = threadIdx.x >> 5;
    const int lane = threadIdx.x & 31;

    if (threadIdx.x == 0) {
        abort_flag = 0;
        for (int s = 0; s < STAGES; ++s) {
            mbar_init(full_bar(s), 1);
            mbar_init(empty_bar(s), 1);
            mbar_init(conv_bar(s), kStreamConverters);  // one arrival per converter warp
        }
        for (int j = 0; j < SLOTS; ++j) {
            mbar_init(s_full(j), 1);
            mbar_init(s_empty(j), kStreamConverters);
        }
        for (int a = 0; a < 2; ++a) {
            mbar_init(acc_full(a), 1);
            mbar_init(acc_empty(a), 4);
        }
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    }
    if (warp == 1) {
        tmem_alloc(smem_u32(&tmem_base_slot), kStreamTmemCols);
        tc_fence_before();
    }
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem_base = tmem_base_slot;
    volatile int* abort_p = &abort_flag;
    pdl_prologue();

    const int64_t n_units = g.tiles_m * g.splits * g.tiles_n * g.batch_groups;
    // unit -> (m tile, K split, n tile, batch group): the m tiles of one S tile run side by side
    auto decode = [&](int64_t u, int64_t& tm, int& split, int64_t& tn, int64_t& bg) {
        tm = u % g.tiles_m;
        int64_t t = u / g.tiles_m;
        split = static_cast<int>(t % g.splits);
        t /= g.splits;
        tn = t % g.tiles_n;
        bg = t / g.tiles_n;
    };

    if (warp == kStreamThreads / 32 - 1) {
        // ---------------- TMA producer of S ----------------
        if (lane == 0) {
            uint32_t it = 0;
            bool ok = true;
            for (int64_t u = blockIdx.x; u < n_units && ok; u += gridDim.x) {
                int64_t tm, tn, bg;
                int split;
                decode(u, tm, split, tn, bg);
                const int batch0 = static_cast<int>(bg * g.bpt);
                const int n0 = static_cast<int>(tn * g.nt);
                const int64_t kb0 = int64_t(split) * g.kb_per_split;
                const int64_t kb1 = min(kb0 + g.kb_per_split, g.k_blocks);
                for (int64_t kb = kb0; kb < kb1; ++kb, ++it) {
                    const int j = it % SLOTS;
                    const uint32_t ph = (it / SLOTS) & 1;
                    if (!mbar_wait(s_empty(j), ph ^ 1, abort_p, g.status)) {
                        ok = false;
                        break;
                    }
                    const uint32_t slot = base + j * kStreamTileBytes;
                    const uint32_t bar = s_full(j);
                    const int kc = static_cast<int>(kb * BK);
                    mbar_arrive_expect_tx(bar, kStreamTileBytes);
                    if (S_KM) {
                        tma_load_3d(slot, &map_s, bar, kc, n0, batch0);  // [128 n][32 k], k contiguous
                    } else {
                        tma_load_3d(slot, &map_s, bar, n0, kc, batch0);  // [32 k][128 n], n contiguous
                    }
                }
            }
        }
    } else if (warp == 0) {
        // ---------------- TMA producer of W's planes ----------------
        if (lane == 0) {
            uint32_t it = 0;
            bool ok = true;
            for (int64_t u = blockIdx.x; u < n_units && ok; u += gridDim.x) {
                int64_t tm, tn, bg;
                int split;
                decode(u, tm, split, tn, bg);
                const int batch0 = static_cast<int>(bg * g.bpt);
                const int m0 = static_cast<int>(tm * BNW);
                const int w_base = static_cast<int>(batch0 * g.w_batch_rows);
                const int64_t kb0 = int64_t(split) * g.kb_per_split;
                const int64_t kb1 = min(kb0 + g.kb_per_split, g.k_blocks);
                for (int64_t kb = kb0; kb < kb1; ++kb, ++it) {
                    const int s = it % STAGES;
                    const uint32_t ph = (it / STAGES) & 1;
                    if (!mbar_wait(empty_bar(s), ph ^ 1, abort_p, g.status)) {
                        ok = false;
                        break;
                    }
                    const uint32_t stage = base + S::kWBase + s * S::kWStage;
                    const uint32_t bar = full_bar(s);
                    const int kc = static_cast<int>(kb * BK);
                    mbar_arrive_expect_tx(bar, kWTx);
                    auto load_w = [&](uint32_t dst, const CUtensorMap* map) {
                        if (W_MN) {
#pragma unroll
                            for (int atom = 0; atom < BNW / 32; ++atom) {
                                tma_load_2d(dst + atom * kMnAtomBytes, map, bar, m0 + 32 * atom, w_base + kc);
                            }
                        } else {
                            tma_load_2d(dst, map, bar, kc, w_base + m0);
                        }
                    };
                    load_w(stage, &map_w_hi);
                    if (THREE_PASS) {
                        load_w(stage + S::kWBytes, &map_w_lo);
                    }
                }
            }
            drain_commits<STAGES>(empty_bar, it, abort_p, g.status);
        }
    } else if (warp == 1) {
        // ---------------- MMA issuer ----------------
        if (lane == 0) {
            uint32_t it = 0;
            uint32_t tile_it = 0;
            bool ok = true;
            for (int64_t u = blockIdx.x; u < n_units && ok; u += gridDim.x, ++tile_it) {
                int64_t tm, tn, bg;
                int split;
                decode(u, tm, split, tn, bg);
                const int acc = tile_it & 1;
                const uint32_t aph = (tile_it >> 1) & 1;
                if (!mbar_wait(acc_empty(acc), aph ^ 1, abort_p, g.status)) {
                    break;
                }
                tc_fence_after();
                const uint32_t d_tmem = tmem_base + acc * BNW;
                const int64_t kb0 = int64_t(split) * g.kb_per_split;
                const int64_t kb1 = min(kb0 + g.kb_per_split, g.k_blocks);
                for (int64_t kb = kb0; kb < kb1; ++kb, ++it) {
                    const int s = it % STAGES;
                    const uint32_t ph = (it / STAGES) & 1;
                    if (!mbar_wait(full_bar(s), ph, abort_p, g.status) ||
                        !mbar_wait(conv_bar(s), ph, abort_p, g.status)) {
                        ok = false;
                        break;
                    }
                    tc_fence_after();
                    const uint32_t stage = base + S::kWBase + s * S::kWStage;
                    const uint64_t w_hi = operand_desc<W_MN>(stage);
                    const uint64_t w_lo = operand_desc<W_MN>(stage + S::kWBytes);
                    const uint32_t s_hi = tmem_base + kStageCol0 + s * 64;
                    const uint32_t s_lo = s_hi + 32;
#pragma unroll
                    for (int kk = 0; kk < BK / UMMA_K; ++kk) {
                        const uint64_t adv_w = static_cast<uint64_t>((W_MN ? kk * 1024 : kk * UMMA_K * 4) >> 4);
                        const uint32_t first = (kb == kb0 && kk == 0) ? 0u : 1u;
                        if (THREE_PASS) {
                            umma_tf32_ts(d_tmem, s_lo + kk * UMMA_K, w_hi + adv_w, kIdesc, first);
                            umma_tf32_ts(d_tmem, s_hi + kk * UMMA_K, w_lo + adv_w, kIdesc, 1u);
                            umma_tf32_ts(d_tmem, s_hi + kk * UMMA_K, w_hi + adv_w, kIdesc, 1u);
                        } else {
                            umma_tf32_ts(d_tmem, s_hi + kk * UMMA_K, w_hi + adv_w, kIdesc, first);
                        }
                    }
                    umma_commit(empty_bar(s));  // W's stage and S's tensor-memory stage are both free then
                }
                if (ok) {
                    umma_commit(acc_full(acc));
                }
            }
        }
    } else if (warp < 6) {
        // ---------------- epilogue (warps 2..5) ----------------
        const int quarter = warp & 3;
        const int l = quarter * 32 + lane;  // tensor-memory lane = position along (batch, n) of the tile
        const int bl = l / g.nt;
        const int nn = l - bl * g.nt;
        uint32_t tile_it = 0;
        for (int64_t u = blockIdx.x; u < n_units; u += gridDim.x, ++tile_it) {
            int64_t tm, tn, bg;
            int split;
            decode(u, tm, split, tn, bg);
            const int acc = tile_it & 1;
            const uint32_t aph = (tile_it >> 1) & 1;
            if (!mbar_wait(acc_full(acc), aph, abort_p, g.status)) {
                break;
            }
            tc_fence_after();
            const int64_t batch = bg * g.bpt + bl;
            const int64_t n = tn * g.nt + nn;
            const bool lane_ok = batch < g.batches && n < g.n;
            const int64_t m0 = tm * BNW;
            const int64_t col = (batch * g.m) * g.n + n;  // + m * N
            float* dst = g.out + int64_t(split) * g.split_stride + col;
#pragma unroll 1
            for (int c = 0; c < BNW / 32; ++c) {
                if (m0 + c * 32 >= g.m) {
                    break;  // uniform
                }
                uint32_t r[32];
                tmem_ld32(tmem_base + (static_cast<uint32_t>(quarter * 32) << 16) + acc * BNW + c * 32, r);
                if (lane_ok) {
                    // one row of C per store: 32 lanes, 128 contiguous bytes.  The row pointer is
                    // stepped, not recomputed -- a 64-bit multiply per store would cost this
                    // single warp more than the store does.
                    const int64_t left = g.m - (m0 + c * 32);
                    float* p = dst + (m0 + c * 32) * g.n;
                    if (left >= 32) {
#pragma unroll
                        for (int j = 0; j < 32; ++j) {
                            *p = __uint_as_float(r[j]);
                            p += g.n;
                        }
                    } else {
#pragma unroll
                        for (int j = 0; j < 32; ++j) {
                            if (j < left) {
                                *p = __uint_as_float(r[j]);
                                p += g.n;
                            }
                        }
                    }
                }
            }
            tc_fence_before();
            __syncwarp();
            if (lane == 0) {
                mbar_arrive(acc_empty(acc));
            }
        }
    } else if (warp < 6 + kStreamConverters) {
        // ---------------- converters (warps 6..21): S tile -> hi / lo in tensor memory ----------------
        // Sixteen warps, four per tensor-memory lane quarter, each taking 8 of the stage's 32 K
        // columns: the split is ~7 instructions per element on 4096 elements per K-block, and it is
        // this loop, not HBM, that a thin set of warps would make the limit.
        const int quarter = warp & 3;
        const int part = (warp - 6) >> 2;  // which 8 of the stage's 32 K columns
        const int l = quarter * 32 + lane;
        const int bl = l / g.nt;
        const int nn = l - bl * g.nt;
        const uint32_t first_off = S_KM ? static_cast<uint32_t>(l * 128)
                                        : static_cast<uint32_t>(((bl * BK + part * 8) * g.nt + nn) * 4);
        const uint32_t k_step = static_cast<uint32_t>(g.nt * 4);
        // K-major tile: the row of lane l is 128 bytes, its 16-byte chunks permuted by the 128-byte
        // swizzle (chunk ^ (row & 7)); this warp's eight K values are chunks 2*part and 2*part + 1
        const uint32_t chunk0 = static_cast<uint32_t>(((2 * part) ^ (l & 7)) * 16);
        const uint32_t chunk1 = static_cast<uint32_t>(((2 * part + 1) ^ (l & 7)) * 16);
        const uint32_t lane_field = static_cast<uint32_t>(quarter * 32) << 16;
        uint32_t it = 0;
        bool ok = true;
        for (int64_t u = blockIdx.x; u < n_units && ok; u += gridDim.x) {
            int64_t tm, tn, bg;
            int split;
            decode(u, tm, split, tn, bg);
            const int64_t kb0 = int64_t(split) * g.kb_per_split;
            const int64_t kb1 = min(kb0 + g.kb_per_split, g.k_blocks);
            for (int64_t kb = kb0; kb < kb1; ++kb, ++it) {
                const int s = it % STAGES;
                const uint32_t ph = (it / STAGES) & 1;
                const int j = it % SLOTS;
                const uint32_t sph = (it / SLOTS) & 1;
                // the tile has landed, and the MMAs that read this tensor-memory stage last are done
                if (!mbar_wait_parked(s_full(j), sph, abort_p, g.status) ||
                    !mbar_wait(empty_bar(s), ph ^ 1, abort_p, g.status)) {
                    ok = false;
                    break;
                }
                tc_fence_after();
                const uint8_t* tile = base_ptr + j * kStreamTileBytes + first_off;
                float v[8];
                uint32_t top = 0;
                if (S_KM) {
                    const float4 q0 = *reinterpret_cast<const float4*>(tile + chunk0);
                    const float4 q1 = *reinterpret_cast<const float4*>(tile + chunk1);
                    v[0] = q0.x; v[1] = q0.y; v[2] = q0.z; v[3] = q0.w;
                    v[4] = q1.x; v[5] = q1.y; v[6] = q1.z; v[7] = q1.w;
                } else {
#pragma unroll
                    for (int j = 0; j < 8; ++j) {
                        v[j] = *reinterpret_cast<const float*>(tile + j * k_step);
                    }
                }
#pragma unroll
                for (int j = 0; j < 8; ++j) {
                    top = max(top, __float_as_uint(v[j]) << 1);
                }
                uint32_t hi[8], lo[8];
                if (top < 0xFEFFE000u) {
                    // every value is finite and rounds inside the TF32 range: add half a TF32 ulp,
                    // clear 13 bits (round to nearest, ties away), lo = tf32(x - hi)
#pragma unroll
                    for (int j = 0; j < 8; ++j) {
                        hi[j] = (__float_as_uint(v[j]) + 0x1000u) & 0xFFFFE000u;
                        const float rest = v[j] - __uint_as_float(hi[j]);
                        asm("cvt.rna.tf32.f32 %0, %1;" : "=r"(lo[j]) : "f"(rest));
                    }
                } else {
#pragma unroll
                    for (int j = 0; j < 8; ++j) {
                        split_tf32_select(v[j], hi[j], lo[j]);  // infinities, NaNs, values that round past the range
                    }
                }
                const uint32_t t_hi = tmem_base + lane_field + kStageCol0 + s * 64 + part * 8;
                tmem_st8(t_hi, hi);
                if (THREE_PASS) {
                    tmem_st8(t_hi + 32, lo);
                }
                asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
                tc_fence_before();
                __syncwarp();
                if (lane == 0) {
                    mbar_arrive(conv_bar(s));
                    mbar_arrive(s_empty(j));  // the values are in registers and tensor memory: the slot may be refilled
                }
            }
        }
    }

    __syncthreads();
    if (abort_flag != 0) {
        for (int i = 0; i < 200; ++i) {
            __nanosleep(1000);
        }
        __syncthreads();
    }
    if (warp == 1) {
        tc_fence_after();
        tmem_dealloc(tmem_base, kStreamTmemCols);
    }
}

__global__ void __launch_bounds__(256)
fold_partials_kernel(float* __restrict__ out, const float* __restrict__ partial, int64_t n, int splits, int quads) {
    pdl_prologue();
    const int64_t stride = int64_t(gridDim.x) * blockDim.x;
    if (quads) {
        for (int64_t i = int64_t(blockIdx.x) * blockDim.x + threadIdx.x; i < n / 4; i += stride) {
            float4 acc = __ldcg(reinterpret_cast<const float4*>(partial) + i);
#pragma unroll 4
            for (int s = 1; s < splits; ++s) {
                const float4 v = __ldcg(reinterpret_cast<const float4*>(partial + int64_t(s) * n) + i);
                acc.x += v.x;
                acc.y += v.y;
                acc.z += v.z;
                acc.w += v.w;
            }
            reinterpret_cast<float4*>(out)[i] = acc;
        }
        return;
    }
    for (int64_t i = int64_t(blockIdx.x) * blockDim.x + threadIdx.x; i < n; i += stride) {
        float acc = partial[i];
#pragma unroll 4
        for (int s = 1; s < splits; ++s) {
            acc += partial[int64_t(s) * n + i];
        }
        out[i] = acc;
    }
}

// The same with what the nodes behind the product make of it: bound by its latency at the sizes that are folded, so an element to a thread,
// whose epilogue needs no alignment, and the nodes' results cost no pass over the sum (6.4 us in a step, with the group's launch behind it 12.9 before).
// (Those results may lie over `out`.)
__global__ void __launch_bounds__(256) fold_epilogue_kernel(float* out, const float* __restrict__ partial, uint32_t n, int splits,
                                                            FastDiv by_cols, const __grid_constant__ ProductEpilogue e) {
    pdl_prologue();
    const uint32_t stride = gridDim.x * blockDim.x;
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += stride) {
        float acc = __ldcg(partial + i);
#pragma unroll 4
        for (int s = 1; s < splits; ++s) acc += __ldcg(partial + int64_t(s) * n + i);
        out[i] = acc;
        write_epilogue(e, i, i - by_cols.div(i) * by_cols.d, acc);
    }
}

// Adds the K-slices' partial planes in split order (one slice: nothing to do).
void fold_partials(b200_ctx* ctx, float* out, const float* partial, int64_t n, int splits, const ProductEpilogue* e = nullptr, int64_t cols = 0) {
    if (splits <= 1) return;
    if (e != nullptr) {
        ProfScope scope(ctx, "matmul.fold");
        launch_kernel(ctx, fold_epilogue_kernel, grid_for(n, 256), 256, 0, out, partial, static_cast<uint32_t>(n), splits,
                      FastDiv(static_cast<uint32_t>(cols)), *e);
        ctx->count_launch();
        check_last_launch("matmul (fold and epilogue)");
        return;
    }
    ProfScope scope(ctx, "matmul.fold");
    // four elements to a thread where that still fills the machine: a small result with many slices is bound by the loads in
    // flight (384 x 128 x 2 with 24 slices: the product 43.5 us with quads, 42 without)
    const bool quads = n % 4 == 0 && n / 4 >= int64_t(sm_count()) * 256 && reinterpret_cast<uintptr_t>(out) % 16 == 0 &&
                       reinterpret_cast<uintptr_t>(partial) % 16 == 0;
    launch_kernel(ctx, fold_partials_kernel, grid_for(quads ? n / 4 : n, 256), 256, 0, out, partial, n, splits, quads ? 1 : 0);
    ctx->count_launch();
    check_last_launch("matmul (fold)");
}

// ---------------------------------------------------------------------------
// Host side
// ---------------------------------------------------------------------------

// Plane [rows][pitch] of f32 (pitch in floats, a multiple of 4), boxes of 32 floats x box_rows,
// 128-byte swizzle.  K-major planes: pitch = Kp, rows = matrix rows, box_rows = tile rows.
// MN-major planes: pitch = padded M or N, rows = batches * Kp, box_rows = 32 K-rows.
CUtensorMap make_map(float* plane, int64_t rows, int64_t pitch, int box_rows, bool mn_major) {
    CUtensorMap m;
    const cuuint64_t dims[2] = {static_cast<cuuint64_t>(pitch), static_cast<cuuint64_t>(rows)};
    const cuuint64_t strides[1] = {static_cast<cuuint64_t>(pitch) * sizeof(float)};
    const cuuint32_t box[2] = {BK, static_cast<cuuint32_t>(box_rows)};
    const cuuint32_t elem[2] = {1, 1};
    const CUresult rc = encode_tiled()(&m, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 2, plane, dims, strides, box, elem,
                                       CU_TENSOR_MAP_INTERLEAVE_NONE,
                                       mn_major ? CU_TENSOR_MAP_SWIZZLE_128B_ATOM_32B : CU_TENSOR_MAP_SWIZZLE_128B,
                                       CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (rc != CUDA_SUCCESS) {
        fail(B200_INTERNAL_ERROR, "cuTensorMapEncodeTiled failed with code " + std::to_string(rc));
    }
    return m;
}

// The caller's own matrix as a 4-D tensor: (unit-stride axis, the other matrix axis, inner
// batch, outer batch), f32, boxes of 32 floats x box_rows, zero fill outside.  A broadcast
// batch axis is given extent 1 and always addressed at coordinate 0.
CUtensorMap make_raw_map(const float* base, int64_t cols, int64_t rows, int64_t pitch, int64_t b1, int64_t s_b1,
                         int64_t b0, int64_t s_b0, int box_rows, bool mn_major) {
    CUtensorMap m;
    const int64_t plane = std::max<int64_t>(rows * pitch, 4);
    if (b1 <= 1 || s_b1 == 0) {
        b1 = 1;
        s_b1 = plane;
    }
    if (b0 <= 1 || s_b0 == 0) {
        b0 = 1;
        s_b0 = std::max(plane, s_b1 * b1);
    }
    const cuuint64_t dims[4] = {static_cast<cuuint64_t>(cols), static_cast<cuuint64_t>(rows),
                                static_cast<cuuint64_t>(b1), static_cast<cuuint64_t>(b0)};
    const cuuint64_t strides[3] = {static_cast<cuuint64_t>(pitch) * sizeof(float),
                                   static_cast<cuuint64_t>(s_b1) * sizeof(float),
                                   static_cast<cuuint64_t>(s_b0) * sizeof(float)};
    const cuuint32_t box[4] = {BK, static_cast<cuuint32_t>(box_rows), 1, 1};
    const cuuint32_t elem[4] = {1, 1, 1, 1};
    const CUresult rc = encode_tiled()(&m, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 4, const_cast<float*>(base), dims, strides,
                                       box, elem, CU_TENSOR_MAP_INTERLEAVE_NONE,
                                       mn_major ? CU_TENSOR_MAP_SWIZZLE_128B_ATOM_32B : CU_TENSOR_MAP_SWIZZLE_128B,
                                       CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (rc != CUDA_SUCCESS) {
        fail(B200_INTERNAL_ERROR, "cuTensorMapEncodeTiled (operand map) failed with code " + std::to_string(rc));
    }
    return m;
}

template <int BN, int STAGES, bool THREE, bool A_MN, bool B_MN>
void launch_one(b200_ctx* ctx, const CUtensorMap& ah, const CUtensorMap& al, const CUtensorMap& bh,
                const CUtensorMap& bl, const TcArgs& g, int grid, const DirectArgs* direct) {
    using S = Smem<BN, STAGES>;
    if (direct != nullptr) {
        auto kernel = gemm_tc_kernel<BN, STAGES, THREE, A_MN, B_MN, true>;
        B200_CUDA_CHECK(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, S::kTotal));
        launch_kernel(ctx, kernel, grid, kThreadsDirect, S::kTotal, ah, al, bh, bl, g, *direct);
        return;
    }
    auto kernel = gemm_tc_kernel<BN, STAGES, THREE, A_MN, B_MN, false>;
    B200_CUDA_CHECK(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, S::kTotal));
    launch_kernel(ctx, kernel, grid, kThreads, S::kTotal, ah, al, bh, bl, g, DirectArgs{});
}

template <int BN, int STAGES>
void launch_main(b200_ctx* ctx, bool three_pass, bool a_mn, bool b_mn, const CUtensorMap& ah,
                 const CUtensorMap& al, const CUtensorMap& bh, const CUtensorMap& bl, const TcArgs& g, int grid,
                 const DirectArgs* direct = nullptr) {
#define B200_TC_CASE(T, A, B)                                                     \
    if (three_pass == T && a_mn == A && b_mn == B) {                              \
        launch_one<BN, STAGES, T, A, B>(ctx, ah, al, bh, bl, g, grid, direct);    \
        return;                                                                   \
    }
    B200_TC_CASE(true, false, false)
    B200_TC_CASE(true, false, true)
    B200_TC_CASE(true, true, false)
    B200_TC_CASE(true, true, true)
    B200_TC_CASE(false, false, false)
    B200_TC_CASE(false, false, true)
    B200_TC_CASE(false, true, false)
    B200_TC_CASE(false, true, true)
#undef B200_TC_CASE
}


// One matmul operand, described by the matrix it is in memory.
struct Operand {
    PlaneKey key{};
    bool mn = false;     // consumed MN-major (the M or N axis is the contiguous one)
    bool dense = false;  // unit stride along one axis, everything else 16-byte aligned
    bool cached = false;
    int64_t nb = 1, rows = 0, cols = 0, rows_pad = 0, cols_pad = 0;
    size_t plane_bytes = 0;
    const char* src_begin = nullptr;
    const char* src_end = nullptr;
    float* hi = nullptr;
    float* lo = nullptr;
    SplitArgs split{};
};

// `s_mn` / `s_k` are the element strides along the operand's M (or N) axis and along K.
// An operand whose M (or N) axis is contiguous keeps its [K][MN] layout and is consumed
// MN-major; everything else becomes a K-major plane [MN][Kp].  Planes of sources with a unit-stride
// axis are padded to 32 rows and 32 columns of zeros, so the same plane serves a later use
// of the same memory in the other orientation.
Operand plan_operand(const float* ptr, int64_t s_b0, int64_t s_b1, int64_t s_mn, int64_t s_k, int64_t mn_extent,
                     int64_t k_extent, bool bcast, const GemmProblem& p) {
    Operand o;
    const int64_t sb0 = bcast ? 0 : s_b0, sb1 = bcast ? 0 : s_b1;
    const bool aligned = reinterpret_cast<uintptr_t>(ptr) % 16 == 0 && sb0 % 4 == 0 && sb1 % 4 == 0;
    o.mn = s_mn == 1 && s_k != 1;
    o.nb = bcast ? 1 : p.b0 * p.b1;
    int64_t s_r, s_c;
    if (o.mn) {
        o.rows = k_extent;
        o.cols = mn_extent;
        s_r = s_k;
        s_c = 1;
    } else {
        o.rows = mn_extent;
        o.cols = k_extent;
        s_r = s_mn;
        s_c = s_k;
    }
    const bool unit = s_c == 1;
    o.dense = unit && s_r % 4 == 0 && aligned;  // as TMA and 128-bit loads want it
    o.rows_pad = unit ? align_up(o.rows, 32) : o.rows;
    o.split.unit = unit ? 1 : 0;
    o.split.vec = o.dense ? 1 : 0;
    o.cols_pad = align_up(o.cols, 32);
    o.plane_bytes = static_cast<size_t>(align_up(o.nb * o.rows_pad * o.cols_pad * 4, 1024));
    const int64_t b1 = bcast ? 1 : p.b1;
    o.key.src = ptr;
    const int64_t kv[8] = {o.rows, o.cols, s_r, s_c, b1, sb0, sb1, o.nb};
    for (int i = 0; i < 8; ++i) o.key.v[i] = kv[i];
    auto mag = [](int64_t v) { return v < 0 ? -v : v; };
    const int64_t b0 = bcast ? 1 : p.b0;
    const int64_t span = (b0 - 1) * mag(sb0) + (b1 - 1) * mag(sb1) + (o.rows - 1) * mag(s_r) + (o.cols - 1) * mag(s_c) + 1;
    o.src_begin = reinterpret_cast<const char*>(ptr);
    o.src_end = o.src_begin + span * 4;
    o.split.src = ptr;
    o.split.b1 = b1;
    o.split.s_b0 = sb0;
    o.split.s_b1 = sb1;
    o.split.n_batches = o.nb;
    o.split.rows = o.rows;
    o.split.out_rows = o.rows_pad;
    o.split.k = o.cols;
    o.split.kp = o.cols_pad;
    o.split.s_r = s_r;
    o.split.s_k = s_c;
    return o;
}

// Whether one tensor map each describes the operands as they lie.  It knows a whole broadcast over the batches (one matrix), not one of the
// two batch axes alone -- which it would read as that axis' first matrix and zeros -- and no axis that stands still or runs backwards.
bool maps_describe(const GemmProblem& p, const Operand& oa, const Operand& ob) {
    auto fits = [&](const Operand& o, const int64_t (&st)[4]) {
        const bool whole = o.nb == 1;
        return o.dense && o.split.s_r >= o.cols && (whole || ((p.b0 == 1 || st[0] > 0) && (p.b1 == 1 || st[1] > 0)));
    };
    return fits(oa, p.a_s) && fits(ob, p.b_s);
}

// Whether reading the operands directly beats splitting them into planes first.  Measured: the
// in-kernel split is bound by shared-memory traffic (the converter's loads and stores contend
// with the tensor core's operand reads) at about 147 TFLOP/s of algorithmic work -- 7.5 ms against
// 4.5 ms at 8192^3, 0.32 against 0.31 ms at 512 x 65536 x 512 -- while the plane scheme moves each
// operand five times (read, two planes written, two planes read).  It pays where
// that traffic is what the product costs: the CNN's first weight gradient, g[256][64x1024] . cols^T[256][1024x27], 74 us
// against 105; the CNN's head, 19 against 24 us (planes that another product of the span uses too cost each half) --
// and below 2^28 operations, which take under 2 us either way while a plane pass is one more launch per operand.
bool direct_pays(const b200_ctx* ctx, const GemmProblem& p, int64_t batches, const Operand& oa, const Operand& ob) {
    auto share = [&](const Operand& o) {
        const auto it = ctx->plane_uses.find(o.key);
        return it != ctx->plane_uses.end() && it->second >= 2 ? 0.5 : 1.0;
    };
    const double flops = 2.0 * double(p.m) * double(p.n) * double(p.k) * double(batches);
    if (flops < double(1 << 28)) return true;
    return flops / 147e12 < 4.0 * (double(oa.plane_bytes) * share(oa) + double(ob.plane_bytes) * share(ob)) / 6.5e12;
}

// The plane kernel's tile width and K-slices.
struct TcPlan {
    int bn;
    int64_t tiles_m, tiles_n, k_blocks, splits, kb_per_split;
};

// Whether the product is better off with operands split inside its kernel (gemm_inline.cu): where it is the only one of its span, and one wave
// serves it.  Where fp32 tiles by TMA would be taken otherwise, always: the converters hold the operands in registers, not in a stage that the tensor
// cores read (2816x1536x128 21.2 us -> 17.8, 704x1664x64 11.7 -> 10.4, 568x6746x228 32.2 -> 25.5).  Instead of planes, while K is not too long: a
// K-block takes 1 to 1.34 us for 0.57 from planes, but there are no passes over the operands in front (512^3 16.8 -> 11.5, 1024^3 26.8 -> 23.3; rows that do
// not lie on 16 bytes 637x947x201 19.0 -> 13.6, 37x8191x1999 79.5 -> 44.1, 681x1026x1021 29.1 -> 25.7; with three waves 1166x129x4131 26.2 -> 31.4;
// 1540x41875x910 935 -> 1535; both operands a float at a time, 2348x421x123 in 'nt', 20.5 -> 26.7, which planes keep).  Over 289 products of one wave
// six take more than 3 % longer than by the other form, and none more than 8 %.  A training step's products stay as they were: a CTA here takes an SM's registers whole, so neither this
// kernel nor the one behind it is scheduled ahead, which costs such a step more than the passes (MLP 248-2451x3-56 545 us -> 562, two products of the
// CNN 12 us).  A compared product of 2^28 operations, up to which fp32 tiles would serve it, keeps its planes.
bool inline_pays(const b200_ctx* ctx, const GemmProblem& p, const Operand& oa, const Operand& ob, const TcPlan& plan, bool direct) {
    if (ctx->gemm_inline == 0 || ctx->gemm_operands >= 0 || ctx->gemm_stream > 0 || ctx->gemm_bn_override != 0 || ctx->gemm_schedule == 1 ||
        (ctx->gemm_schedule < 0 && ctx->in_grad_sync_span) || !gemm_inline_fits(p, true)) {
        return false;
    }
    if (ctx->gemm_inline >= 8) return true;
    if (!ctx->lone_matmul) return false;
    const int64_t batches = p.b0 * p.b1, bn = p.n > 64 ? 128 : 64;
    if (ceil_div(p.m, int64_t(BM)) * ceil_div(p.n, bn) * batches * plan.splits > sm_count()) return false;
    if (direct) return true;
    // us: K-blocks, what is around them, and the passes over the operands (12 bytes per element)
    // (units of up to ten K-blocks stay here whatever their rows: it costs them 3 us at most, 3 x 257x301x219 in 'nt' 16.0 -> 18.7)
    const double inline_us = (plan.kb_per_split > 10 ? gemm_inline_tf32_block(p) : 1.0) * double(plan.kb_per_split) + 7.0;
    const double planes_us = 0.6 * double(plan.kb_per_split) + 12.0 * double(oa.plane_bytes + ob.plane_bytes) / 4 / 5.8e6 + 11.0;
    const double flops = 2.0 * double(p.m) * double(p.n) * double(p.k) * double(batches);
    return inline_us <= planes_us && (flops > double(1 << 28) || ctx->compared.count(p.out) == 0 || !maps_describe(p, oa, ob));
}

size_t plane_cache_limit(const b200_ctx* ctx) {
    return std::min<size_t>(size_t(16) << 30, ctx->prop.totalGlobalMem / 8);
}

void release_use(b200_ctx* ctx, const Operand& o) {
    if (!o.cached) return;
    auto it = ctx->plane_cache.find(o.key);
    if (it == ctx->plane_cache.end()) return;
    if (--it->second.uses_left <= 0) {
        ctx->scratch.release(it->second.hi);
        ctx->plane_cache_bytes -= it->second.bytes;
        ctx->plane_cache.erase(it);
    }
}

// ---- streamed-operand kernel: eligibility and launch ----

struct StreamPlan {
    bool ok = false;
    bool s_km = false;         // S's K axis is the contiguous one
    int nt = 128, bpt = 1, bnw = 64;
    int64_t pitch = 0;         // elements between consecutive rows of S (K rows, or N rows when s_km)
    int64_t batch_stride = 0;  // elements between consecutive batches of S
};

// The product qualifies when its right operand can be read by TMA as it lies in memory (n or k
// contiguous, 16-byte pitches, batches one constant stride apart) and the product is bound by
// memory rather than by the tensor pipe: a left operand of at most 256 rows (the streamed operand
// is then worth 128 flops per byte at most, and one pass over it beats reading it once, writing
// two planes and reading those), or a short K (at most 256: the result outweighs the operands --
// the column gradient of a convolution -- and re-reading S's few tiles from L2 for every 128 rows
// of W costs less than the plane passes).
StreamPlan plan_stream(const b200_ctx* ctx, const GemmProblem& p) {
    StreamPlan sp;
    if (ctx->gemm_stream == 0 || (ctx->gemm_stream < 0 && ctx->gemm_operands >= 0)) {
        return sp;  // switched off, or another operand scheme was asked for by name
    }
    const int64_t batches = p.b0 * p.b1;
    // (VKML_B200_GEMM_STREAM=1 lifts the size rule: every product whose layout allows it, for A/B runs)
    if ((ctx->gemm_stream < 1 && p.m > 256 && (p.k > 256 || p.m > 4096)) || p.n < 32 || batches < 1) return sp;
    if (p.b_s[3] == 1 && p.b_s[2] % 4 == 0 && p.b_s[2] >= p.n) {
        sp.s_km = false;
        sp.pitch = p.b_s[2];
    } else if (p.b_s[2] == 1 && p.b_s[3] % 4 == 0 && p.b_s[3] >= p.k && p.n >= 128) {
        sp.s_km = true;
        sp.pitch = p.b_s[3];
    } else {
        return sp;
    }
    if (reinterpret_cast<uintptr_t>(p.b) % 16 != 0) return sp;
    int64_t sb = std::max<int64_t>((sp.s_km ? p.n : p.k) * sp.pitch, 4);
    if (batches > 1) {
        if (p.b0 == 1) sb = p.b_s[1];
        else if (p.b1 == 1) sb = p.b_s[0];
        else if (p.b_s[0] == p.b1 * p.b_s[1]) sb = p.b_s[1];
        else return sp;
        if (sb <= 0 || sb % 4 != 0) return sp;
    }
    const bool a_bcast = (p.a_s[0] == 0 || p.b0 == 1) && (p.a_s[1] == 0 || p.b1 == 1);
    if (p.n >= 128) {
        sp.nt = 128;
        sp.bpt = 1;
    } else if ((p.n == 32 || p.n == 64) && a_bcast && batches % (128 / p.n) == 0) {
        sp.nt = static_cast<int>(p.n);  // a tile spans several batches: lanes = batch x n
        sp.bpt = static_cast<int>(128 / p.n);
    } else {
        return sp;
    }
    if (batches >= (int64_t(1) << 31) || p.n >= (int64_t(1) << 31) || sb * 4 >= (int64_t(1) << 40)) return sp;
    sp.bnw = p.m <= 64 ? 64 : 128;
    sp.batch_stride = sb;
    sp.ok = true;
    return sp;
}

CUtensorMap make_stream_map(const float* base, int64_t n, int64_t k, int64_t pitch, int64_t batches,
                            int64_t batch_stride, int nt, int bpt, bool s_km) {
    CUtensorMap m;
    // n contiguous: tiles of [32 k][nt n] as they lie; k contiguous: tiles of [128 n][32 k], whose
    // 128-byte rows take the 128-byte swizzle
    const cuuint64_t dims[3] = {static_cast<cuuint64_t>(s_km ? k : n), static_cast<cuuint64_t>(s_km ? n : k),
                                static_cast<cuuint64_t>(batches)};
    const cuuint64_t strides[2] = {static_cast<cuuint64_t>(pitch) * sizeof(float),
                                   static_cast<cuuint64_t>(batch_stride) * sizeof(float)};
    const cuuint32_t box[3] = {s_km ? cuuint32_t(BK) : static_cast<cuuint32_t>(nt), s_km ? cuuint32_t(128) : cuuint32_t(BK),
                               static_cast<cuuint32_t>(bpt)};
    const cuuint32_t elem[3] = {1, 1, 1};
    const CUresult rc = encode_tiled()(&m, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 3, const_cast<float*>(base), dims, strides,
                                       box, elem, CU_TENSOR_MAP_INTERLEAVE_NONE,
                                       s_km ? CU_TENSOR_MAP_SWIZZLE_128B : CU_TENSOR_MAP_SWIZZLE_NONE,
                                       CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (rc != CUDA_SUCCESS) {
        fail(B200_INTERNAL_ERROR, "cuTensorMapEncodeTiled (streamed operand) failed with code " + std::to_string(rc));
    }
    return m;
}

template <int BNW>
void launch_stream(b200_ctx* ctx, bool three_pass, bool w_mn, bool s_km, const CUtensorMap& ms, const CUtensorMap& wh,
                   const CUtensorMap& wl, const StreamArgs& g, int grid) {
    using S = StreamSmem<BNW>;
#define B200_STREAM_CASE(T, W)                                                                             \
    if (three_pass == T && w_mn == W && s_km) {                                                            \
        auto kernel = gemm_stream_kernel<BNW, T, W, true>;                                                 \
        B200_CUDA_CHECK(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, S::kTotal)); \
        launch_kernel(ctx, kernel, grid, kStreamThreads, S::kTotal, ms, wh, wl, g);                        \
        return;                                                                                            \
    }                                                                                                      \
    if (three_pass == T && w_mn == W) {                                                                    \
        auto kernel = gemm_stream_kernel<BNW, T, W, false>;                                                \
        B200_CUDA_CHECK(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, S::kTotal)); \
        launch_kernel(ctx, kernel, grid, kStreamThreads, S::kTotal, ms, wh, wl, g);                        \
        return;                                                                                            \
    }
    B200_STREAM_CASE(true, false)
    B200_STREAM_CASE(true, true)
    B200_STREAM_CASE(false, false)
    B200_STREAM_CASE(false, true)
#undef B200_STREAM_CASE
}

int64_t stream_slices(const b200_ctx* ctx, const GemmProblem& p, const StreamPlan& sp) {
    const int64_t tiles = ceil_div(p.m, sp.bnw) * (sp.bpt > 1 ? 1 : ceil_div(p.n, 128)) * ceil_div(p.b0 * p.b1, sp.bpt), sms = ctx->prop.multiProcessorCount;
    const int64_t k_blocks = align_up(p.k, BK) / BK;
    int64_t splits = 1;
    if (tiles < sms && k_blocks >= 16) splits = std::max<int64_t>(1, std::min<int64_t>(std::min(sms / tiles, k_blocks / 8), 64));
    return ceil_div(k_blocks, ceil_div(k_blocks, splits));
}

void gemm_stream(b200_ctx* ctx, const GemmProblem& p, bool three_pass, const StreamPlan& sp, const ProductEpilogue* epilogue) {
    const int64_t batches = p.b0 * p.b1;
    const bool a_bcast = (p.a_s[0] == 0 || p.b0 == 1) && (p.a_s[1] == 0 || p.b1 == 1);
    Operand ow = plan_operand(p.a, p.a_s[0], p.a_s[1], p.a_s[2], p.a_s[3], p.m, p.k, a_bcast, p);
    const int64_t k_blocks = align_up(p.k, BK) / BK;
    const int64_t tiles_m = ceil_div(p.m, sp.bnw);
    const int64_t tiles_n = sp.bpt > 1 ? 1 : ceil_div(p.n, 128);
    const int64_t batch_groups = ceil_div(batches, sp.bpt);
    const int64_t tiles = tiles_m * tiles_n * batch_groups;
    const int sms = ctx->prop.multiProcessorCount;
    const int64_t kb_per_split = ceil_div(k_blocks, stream_slices(ctx, p, sp)), splits = ceil_div(k_blocks, kb_per_split);
    const int64_t out_elems = batches * p.m * p.n;
    const size_t partial_bytes = splits > 1 ? static_cast<size_t>(align_up(out_elems * splits * 4, 1024)) : 0;

    // W's planes: from this span's cache, into it, or into the workspace
    const size_t planes = three_pass ? 2 : 1;
    bool hit = false;
    if (auto it = ctx->plane_cache.find(ow.key); it != ctx->plane_cache.end()) {
        ow.hi = it->second.hi;
        ow.lo = it->second.lo;
        ow.cached = hit = true;
        ++ctx->plane_hits;
    } else {
        auto uses = ctx->plane_uses.find(ow.key);
        const size_t bytes = planes * ow.plane_bytes;
        if (uses != ctx->plane_uses.end() && uses->second >= 2 &&
            ctx->plane_cache_bytes + bytes <= plane_cache_limit(ctx)) {
            char* block = static_cast<char*>(ctx->scratch.allocate(bytes));
            ow.hi = reinterpret_cast<float*>(block);
            ow.lo = three_pass ? reinterpret_cast<float*>(block + ow.plane_bytes) : nullptr;
            ctx->plane_cache[ow.key] = PlaneEntry{ow.hi, ow.lo, bytes, uses->second, ow.src_begin, ow.src_end};
            ctx->plane_cache_bytes += bytes;
            ow.cached = true;
        }
    }
    char* ws = static_cast<char*>(ctx->ensure_workspace(partial_bytes + 2048 + (ow.cached ? 0 : planes * ow.plane_bytes)));
    ws = reinterpret_cast<char*>(align_up(reinterpret_cast<int64_t>(ws), 1024));
    if (!ow.cached) {
        ow.hi = reinterpret_cast<float*>(ws);
        ow.lo = three_pass ? reinterpret_cast<float*>(ws + ow.plane_bytes) : nullptr;
        ws += planes * ow.plane_bytes;
    }
    float* partial = splits > 1 ? reinterpret_cast<float*>(ws) : nullptr;
    if (!hit) {
        ow.split.hi = ow.hi;
        ow.split.lo = ow.lo;
        launch_split(ctx, ow.split, "matmul.split_a");
        check_last_launch("matmul (operand split)");
    }

    const CUtensorMap ms = make_stream_map(p.b, p.n, p.k, sp.pitch, batches, sp.batch_stride, sp.nt, sp.bpt, sp.s_km);
    auto map_w = [&](float* plane) {
        return ow.mn ? make_map(plane, ow.nb * ow.rows_pad, ow.cols_pad, BK, true)
                     : make_map(plane, ow.nb * ow.rows_pad, ow.cols_pad, sp.bnw, false);
    };
    const CUtensorMap wh = map_w(ow.hi);
    const CUtensorMap wl = three_pass ? map_w(ow.lo) : wh;

    StreamArgs g{};
    g.out = splits > 1 ? partial : p.out;
    g.m = p.m;
    g.n = p.n;
    g.batches = batches;
    g.w_batch_rows = a_bcast ? 0 : ow.rows_pad;
    g.k_blocks = k_blocks;
    g.kb_per_split = kb_per_split;
    g.splits = static_cast<int>(splits);
    g.split_stride = out_elems;
    g.tiles_m = tiles_m;
    g.tiles_n = tiles_n;
    g.nt = sp.nt;
    g.bpt = sp.bpt;
    g.batch_groups = batch_groups;
    g.status = ctx->d_status;
    const int grid = static_cast<int>(std::min<int64_t>(tiles * splits, sms));
    {
        ProfScope scope(ctx, three_pass ? "matmul.tcgen05_3xtf32_stream" : "matmul.tcgen05_tf32_stream");
        if (sp.bnw == 64) {
            launch_stream<64>(ctx, three_pass, ow.mn, sp.s_km, ms, wh, wl, g, grid);
        } else {
            launch_stream<128>(ctx, three_pass, ow.mn, sp.s_km, ms, wh, wl, g, grid);
        }
    }
    ctx->count_launch();
    check_last_launch("matmul (tcgen05, streamed operand)");
    fold_partials(ctx, p.out, partial, out_elems, static_cast<int>(splits), epilogue, p.n);
    release_use(ctx, ow);
}

TcPlan plan_planes(const b200_ctx* ctx, const GemmProblem& p) {
    const int64_t batches = p.b0 * p.b1;
    // Tile width: 128x256 tiles are the most efficient per tile (measured 5.5 % better than two
    // 128x128 tiles), but the persistent grid runs whole waves of 148 tiles, so the narrower
    // tile wins whenever it wastes less of the last wave (M=2048, N=8192: 4 waves of 256-wide
    // tiles against 7 half-cost waves of 128-wide ones).
    int bn = 64;
    if (p.n > 64) bn = 128;
    if (p.n > 128 && p.m * p.n * batches >= int64_t(128) * 256 * sm_count()) {
        const int64_t tm = ceil_div(p.m, BM);
        const double cost256 = double(ceil_div(tm * ceil_div(p.n, 256) * batches, sm_count()));
        const double cost128 = double(ceil_div(tm * ceil_div(p.n, 128) * batches, sm_count())) * 0.5275;
        bn = cost128 < cost256 ? 128 : 256;
    }
    if (ctx->gemm_bn_override == 64 || ctx->gemm_bn_override == 128 || ctx->gemm_bn_override == 256) {
        bn = ctx->gemm_bn_override;
    }
    const int64_t tiles_m = ceil_div(p.m, BM);
    const int64_t tiles_n = ceil_div(p.n, bn);
    const int64_t tiles = tiles_m * tiles_n * batches;
    const int64_t k_blocks = ceil_div(p.k, BK);

    // split K when the tiles alone cannot fill the machine
    int64_t splits = 1;
    if (tiles < sm_count() && k_blocks >= 16) {
        // as many K-slices as keep every unit in ONE wave of the persistent grid: rounding up
        // instead (32 tiles x 5 slices = 160 units on 148 SMs) runs a second, nearly empty wave.  Slices of eight K-blocks
        // and more; of three where the tiles fill less than an eighth of the machine (a classifier's few columns: 300 x 900 x 100
        // took 21 us with three CTAs to a tile), unless the span compares the result, whose bits then stay
        const int64_t least = tiles * 8 <= sm_count() && ctx->compared.count(p.out) == 0 ? 3 : 8;
        splits = std::min<int64_t>(sm_count() / tiles, k_blocks / least);
        splits = std::max<int64_t>(1, std::min<int64_t>(splits, 64));
    }
    int64_t kb_per_split = ceil_div(k_blocks, splits);
    splits = ceil_div(k_blocks, kb_per_split);

    return TcPlan{bn, tiles_m, tiles_n, k_blocks, splits, kb_per_split};
}

}  // namespace

bool gemm_tc_eligible(const b200_ctx* ctx, const GemmProblem& p) {
    if (ctx->prop.major != 10 || encode_tiled() == nullptr) {
        return false;
    }
    const int64_t batches = p.b0 * p.b1;
    if (p.m < 32 || p.n < 16 || p.k < 16 || batches < 1) {  // K is zero-padded to the 32-wide K-block
        return false;
    }
    if (gemm_small_pays(p, plan_stream(ctx, p).ok)) {
        return false;  // one launch on the CUDA cores is cheaper
    }
    // TMA coordinates are 32-bit
    const int64_t kp = align_up(p.k, BK);
    if (kp >= (int64_t(1) << 31) || batches * p.m >= (int64_t(1) << 31) || batches * p.n >= (int64_t(1) << 31)) {
        return false;
    }
    return true;
}

int64_t gemm_tc_chain(const b200_ctx* ctx, const GemmProblem& p) { return plan_planes(ctx, p).kb_per_split * BK; }

bool gemm_tc_streams(const b200_ctx* ctx, const GemmProblem& p) { return plan_stream(ctx, p).ok; }

// Whether gemm_tc would read this product's operands directly (no planes), taken by itself: the
// same conditions as in gemm_tc below, with no other matmul of a span sharing the planes.
bool gemm_tc_reads_directly(const b200_ctx* ctx, const GemmProblem& p) {
    if (plan_stream(ctx, p).ok || ctx->gemm_operands == 0) return false;
    const int64_t batches = p.b0 * p.b1;
    const bool a_bcast = (p.a_s[0] == 0 || p.b0 == 1) && (p.a_s[1] == 0 || p.b1 == 1);
    const bool b_bcast = (p.b_s[0] == 0 || p.b0 == 1) && (p.b_s[1] == 0 || p.b1 == 1);
    const Operand oa = plan_operand(p.a, p.a_s[0], p.a_s[1], p.a_s[2], p.a_s[3], p.m, p.k, a_bcast, p);
    const Operand ob = plan_operand(p.b, p.b_s[0], p.b_s[1], p.b_s[3], p.b_s[2], p.n, p.k, b_bcast, p);
    const bool want_dynamic = ctx->gemm_schedule == 1;
    return maps_describe(p, oa, ob) && !want_dynamic && (ctx->gemm_operands == 1 || direct_pays(ctx, p, batches, oa, ob));
}

bool gemm_tc_splits_inside(const b200_ctx* ctx, const GemmProblem& p) {
    if (plan_stream(ctx, p).ok || ctx->gemm_precision != B200_GEMM_3XTF32) return false;
    const bool a_bcast = (p.a_s[0] == 0 || p.b0 == 1) && (p.a_s[1] == 0 || p.b1 == 1);
    const bool b_bcast = (p.b_s[0] == 0 || p.b0 == 1) && (p.b_s[1] == 0 || p.b1 == 1);
    const Operand oa = plan_operand(p.a, p.a_s[0], p.a_s[1], p.a_s[2], p.a_s[3], p.m, p.k, a_bcast, p);
    const Operand ob = plan_operand(p.b, p.b_s[0], p.b_s[1], p.b_s[3], p.b_s[2], p.n, p.k, b_bcast, p);
    return inline_pays(ctx, p, oa, ob, plan_planes(ctx, p), gemm_tc_reads_directly(ctx, p));
}

void gemm_tc_wait_probe(b200_ctx* ctx, uint64_t limit_ns) {
    wait_probe_kernel<<<1, 32, 0, ctx->stream>>>(ctx->d_status, limit_ns);
    ctx->count_launch();
    check_last_launch("wait probe");
}

bool gemm_tc_folds(const b200_ctx* ctx, const GemmProblem& p) {
    const StreamPlan sp = plan_stream(ctx, p);
    return (sp.ok ? stream_slices(ctx, p, sp) : plan_planes(ctx, p).splits) > 1;
}

void gemm_tc(b200_ctx* ctx, const GemmProblem& p, bool three_pass, const ProductEpilogue* epilogue) {
    if (const StreamPlan sp = plan_stream(ctx, p); sp.ok) {
        gemm_stream(ctx, p, three_pass, sp, epilogue);
        return;
    }
    const int64_t batches = p.b0 * p.b1;
    const bool a_bcast = (p.a_s[0] == 0 || p.b0 == 1) && (p.a_s[1] == 0 || p.b1 == 1);
    const bool b_bcast = (p.b_s[0] == 0 || p.b0 == 1) && (p.b_s[1] == 0 || p.b1 == 1);

    const TcPlan plan = plan_planes(ctx, p);
    const int bn = plan.bn;
    const int64_t tiles_m = plan.tiles_m, tiles_n = plan.tiles_n, tiles = tiles_m * tiles_n * batches;
    const int64_t k_blocks = plan.k_blocks, splits = plan.splits, kb_per_split = plan.kb_per_split;
    const int64_t out_elems = batches * p.m * p.n;
    const size_t partial_bytes = splits > 1 ? static_cast<size_t>(align_up(out_elems * splits * 4, 1024)) : 0;
    Operand oa = plan_operand(p.a, p.a_s[0], p.a_s[1], p.a_s[2], p.a_s[3], p.m, p.k, a_bcast, p);
    Operand ob = plan_operand(p.b, p.b_s[0], p.b_s[1], p.b_s[3], p.b_s[2], p.n, p.k, b_bcast, p);
    const bool a_mn = oa.mn, b_mn = ob.mn;

    const bool want_dynamic = ctx->gemm_schedule == 1 || (ctx->gemm_schedule < 0 && ctx->in_grad_sync_span);
    const bool direct = ctx->gemm_operands != 0 && maps_describe(p, oa, ob) && !want_dynamic &&
                        (ctx->gemm_operands == 1 || direct_pays(ctx, p, batches, oa, ob));
    if (three_pass && inline_pays(ctx, p, oa, ob, plan, direct)) {
        float* partial = nullptr;
        if (splits > 1) {
            char* ws = static_cast<char*>(ctx->ensure_workspace(partial_bytes + 2048));
            partial = reinterpret_cast<float*>(align_up(reinterpret_cast<int64_t>(ws), 1024));
        }
        gemm_inline_tf32(ctx, p, partial, splits, kb_per_split, direct ? "matmul.tcgen05_3xtf32_direct" : "matmul.tcgen05_3xtf32");
        fold_partials(ctx, p.out, partial, out_elems, static_cast<int>(splits), epilogue, p.n);
        return;
    }

    // ---- direct operands: no planes at all ----
    if (direct) {
        float* partial = nullptr;
        if (splits > 1) {
            char* ws = static_cast<char*>(ctx->ensure_workspace(partial_bytes + 2048));
            partial = reinterpret_cast<float*>(align_up(reinterpret_cast<int64_t>(ws), 1024));
        }
        DirectArgs da{};
        da.b1 = p.b1;
        da.a_bcast = a_bcast ? 1 : 0;
        da.b_bcast = b_bcast ? 1 : 0;
        // A: K-major = rows M with pitch a_s[2]; MN-major = rows K with pitch a_s[3]
        const CUtensorMap raw_a =
            a_mn ? make_raw_map(p.a, p.m, p.k, p.a_s[3], a_bcast ? 1 : p.b1, p.a_s[1], a_bcast ? 1 : p.b0, p.a_s[0], BK, true)
                 : make_raw_map(p.a, p.k, p.m, p.a_s[2], a_bcast ? 1 : p.b1, p.a_s[1], a_bcast ? 1 : p.b0, p.a_s[0], BM, false);
        const CUtensorMap raw_b =
            b_mn ? make_raw_map(p.b, p.n, p.k, p.b_s[2], b_bcast ? 1 : p.b1, p.b_s[1], b_bcast ? 1 : p.b0, p.b_s[0], BK, true)
                 : make_raw_map(p.b, p.k, p.n, p.b_s[3], b_bcast ? 1 : p.b1, p.b_s[1], b_bcast ? 1 : p.b0, p.b_s[0], bn, false);
        TcArgs g{};
        g.out = splits > 1 ? partial : p.out;
        g.m = p.m;
        g.n = p.n;
        g.batches = batches;
        g.k_blocks = k_blocks;
        g.kb_per_split = kb_per_split;
        g.splits = static_cast<int>(splits);
        g.split_stride = out_elems;
        g.tiles_m = tiles_m;
        g.tiles_n = tiles_n;
        g.group_m = ctx->gemm_group_m > 0 ? ctx->gemm_group_m : kGroupM;
        g.status = ctx->d_status;
        const int grid = static_cast<int>(std::min<int64_t>(tiles * splits, ctx->prop.multiProcessorCount));
        {
            ProfScope scope(ctx, three_pass ? "matmul.tcgen05_3xtf32_direct" : "matmul.tcgen05_tf32_direct");
            if (bn == 256) {
                launch_main<256, 2>(ctx, three_pass, a_mn, b_mn, raw_a, raw_a, raw_b, raw_b, g, grid, &da);
            } else if (bn == 128) {
                launch_main<128, 3>(ctx, three_pass, a_mn, b_mn, raw_a, raw_a, raw_b, raw_b, g, grid, &da);
            } else {
                launch_main<64, 4>(ctx, three_pass, a_mn, b_mn, raw_a, raw_a, raw_b, raw_b, g, grid, &da);
            }
        }
        ctx->count_launch();
        check_last_launch("matmul (tcgen05, direct operands)");
        fold_partials(ctx, p.out, partial, out_elems, static_cast<int>(splits), epilogue, p.n);
        return;
    }

    // ---- operand planes: from this span's cache, into it, or into the workspace ----
    const size_t planes = three_pass ? 2 : 1;
    auto from_cache = [&](Operand& o) {
        auto it = ctx->plane_cache.find(o.key);
        if (it == ctx->plane_cache.end()) return false;
        o.hi = it->second.hi;
        o.lo = it->second.lo;
        o.cached = true;
        ++ctx->plane_hits;
        return true;
    };
    auto into_cache = [&](Operand& o) {
        auto uses = ctx->plane_uses.find(o.key);
        const size_t bytes = planes * o.plane_bytes;
        if (uses == ctx->plane_uses.end() || uses->second < 2 ||
            ctx->plane_cache_bytes + bytes > plane_cache_limit(ctx)) {
            return false;
        }
        char* block = static_cast<char*>(ctx->scratch.allocate(bytes));
        o.hi = reinterpret_cast<float*>(block);
        o.lo = three_pass ? reinterpret_cast<float*>(block + o.plane_bytes) : nullptr;
        ctx->plane_cache[o.key] = PlaneEntry{o.hi, o.lo, bytes, uses->second, o.src_begin, o.src_end};
        ctx->plane_cache_bytes += bytes;
        o.cached = true;
        return true;
    };
    const bool a_hit = from_cache(oa);
    if (!a_hit) into_cache(oa);
    // (B may be the very plane A just put there: x times its own transpose)
    const bool b_hit = from_cache(ob);
    if (!b_hit) into_cache(ob);
    size_t ws_bytes = partial_bytes + 2048;
    if (!oa.cached) ws_bytes += planes * oa.plane_bytes;
    if (!ob.cached) ws_bytes += planes * ob.plane_bytes;
    char* ws = static_cast<char*>(ctx->ensure_workspace(ws_bytes));
    ws = reinterpret_cast<char*>(align_up(reinterpret_cast<int64_t>(ws), 1024));
    auto from_workspace = [&](Operand& o) {
        if (o.cached) return;
        o.hi = reinterpret_cast<float*>(ws);
        o.lo = three_pass ? reinterpret_cast<float*>(ws + o.plane_bytes) : nullptr;
        ws += planes * o.plane_bytes;
    };
    from_workspace(oa);
    from_workspace(ob);
    float* partial = splits > 1 ? reinterpret_cast<float*>(ws) : nullptr;

    oa.split.hi = oa.hi;
    oa.split.lo = oa.lo;
    ob.split.hi = ob.hi;
    ob.split.lo = ob.lo;
    auto elements = [](const SplitArgs& s) { return s.kp * s.out_rows * s.n_batches; };
    if (!a_hit && !b_hit && ctx->gemm_operands < 0 && !ctx->lone_matmul && elements(oa.split) + elements(ob.split) < 4 * kSmallQuads) {
        // (over more elements the launch saved is no longer seen: an MLP 4096-8192x3-1000 at batch 2048 561 us of splits apart, 565 together; 7 M,
        // 361x2484 and 2484x2484, 30 apart and 25 together)
        // (among a step's launches one less: 315 rows through an MLP 160-83-32 77 us a step, 64 now; 93 through 284-1130x3-201 233 and 222)
        ProfScope scope(ctx, "matmul.split");
        SplitTwo two{{oa.split, ob.split}};
        launch_kernel(ctx, split_two_kernel, dim3(static_cast<unsigned>(std::max(split_blocks(oa.split), split_blocks(ob.split))), 2), 256, 0, two);
        ctx->count_launch();
    } else {
        if (!a_hit) launch_split(ctx, oa.split, "matmul.split_a");
        if (!b_hit) launch_split(ctx, ob.split, "matmul.split_b");
    }
    if (!a_hit || !b_hit) {
        check_last_launch("matmul (operand split)");
    }

    // ---- main kernel ----
    // K-major plane: [batch][MN rows (padded)][Kp]; MN-major plane: [batch][Kp rows][MN padded]
    auto map_of = [&](float* plane, const Operand& o, int tile) {
        return o.mn ? make_map(plane, o.nb * o.rows_pad, o.cols_pad, BK, true)
                    : make_map(plane, o.nb * o.rows_pad, o.cols_pad, tile, false);
    };
    const CUtensorMap ah = map_of(oa.hi, oa, BM);
    const CUtensorMap al = three_pass ? map_of(oa.lo, oa, BM) : ah;
    const CUtensorMap bh = map_of(ob.hi, ob, bn);
    const CUtensorMap bl = three_pass ? map_of(ob.lo, ob, bn) : bh;

    TcArgs g{};
    g.out = splits > 1 ? partial : p.out;
    g.m = p.m;
    g.n = p.n;
    g.batches = batches;
    g.a_batch_rows = a_bcast ? 0 : oa.rows_pad;  // plane rows between consecutive batches
    g.b_batch_rows = b_bcast ? 0 : ob.rows_pad;
    g.k_blocks = k_blocks;
    g.kb_per_split = kb_per_split;
    g.splits = static_cast<int>(splits);
    g.split_stride = out_elems;
    g.tiles_m = tiles_m;
    g.tiles_n = tiles_n;
    g.group_m = ctx->gemm_group_m > 0 ? ctx->gemm_group_m : kGroupM;
    g.status = ctx->d_status;
    int sms = ctx->prop.multiProcessorCount;
    if (ctx->in_grad_sync_span && ctx->comm_pending) {
        sms = std::max(sms - ctx->comm_sms, sms / 2);  // leave room for the all-reduce kernels
    }
    const int grid = static_cast<int>(std::min<int64_t>(tiles * splits, sms));
    const bool dynamic = (ctx->gemm_schedule == 1 || (ctx->gemm_schedule < 0 && ctx->in_grad_sync_span)) &&
                         tiles * splits > grid && tiles * splits < (int64_t(1) << 30);
    if (dynamic) {
        g.sched = ctx->d_counters + 4096;  // past the reductions' arrival counters
        B200_CUDA_CHECK(cudaMemsetAsync(g.sched, 0, sizeof(unsigned int), ctx->stream));
    }
    {
        ProfScope scope(ctx, three_pass ? "matmul.tcgen05_3xtf32" : "matmul.tcgen05_tf32");
        if (bn == 256) {
            launch_main<256, 2>(ctx, three_pass, a_mn, b_mn, ah, al, bh, bl, g, grid);
        } else if (bn == 128) {
            launch_main<128, 3>(ctx, three_pass, a_mn, b_mn, ah, al, bh, bl, g, grid);
        } else {
            launch_main<64, 4>(ctx, three_pass, a_mn, b_mn, ah, al, bh, bl, g, grid);
        }
    }
    ctx->count_launch();
    check_last_launch("matmul (tcgen05)");

    fold_partials(ctx, p.out, partial, out_elems, static_cast<int>(splits), epilogue, p.n);
    // the stream is in order: a plane released here is only reused by later work
    release_use(ctx, oa);
    release_use(ctx, ob);
}

int gemm_tc_slices(const b200_ctx* ctx, const GemmProblem& p) { return static_cast<int>(plan_planes(ctx, p).splits); }

size_t gemm_tc_plane_limit(const b200_ctx* ctx) { return plane_cache_limit(ctx); }

size_t gemm_tc_plane_bytes(const GemmProblem& p, bool left) {
    const int64_t* s = left ? p.a_s : p.b_s;
    const bool bcast = (s[0] == 0 || p.b0 == 1) && (s[1] == 0 || p.b1 == 1);
    return 2 * plan_operand(left ? p.a : p.b, s[0], s[1], left ? s[2] : s[3], left ? s[3] : s[2], left ? p.m : p.n, p.k, bcast, p).plane_bytes;
}

void gemm_tc_stand_by(b200_ctx* ctx, const GemmProblem& p, const RangeGuard& guard, const Standby& a, const Standby& b, float* target,
                      float* partial) {
    const bool a_bcast = (p.a_s[0] == 0 || p.b0 == 1) && (p.a_s[1] == 0 || p.b1 == 1);
    const bool b_bcast = (p.b_s[0] == 0 || p.b0 == 1) && (p.b_s[1] == 0 || p.b1 == 1);
    const TcPlan plan = plan_planes(ctx, p);
    Operand oa = plan_operand(p.a, p.a_s[0], p.a_s[1], p.a_s[2], p.a_s[3], p.m, p.k, a_bcast, p);
    Operand ob = plan_operand(p.b, p.b_s[0], p.b_s[1], p.b_s[3], p.b_s[2], p.n, p.k, b_bcast, p);
    SplitPair pair{};
    pair.guard = guard;
    pair.p = p;
    pair.target = target;
    pair.bcast[0] = a_bcast ? 1 : 0;
    pair.bcast[1] = b_bcast ? 1 : 0;
    Operand* const operands[2] = {&oa, &ob};
    const Standby* const at[2] = {&a, &b};
    for (int i = 0; i < 2; ++i) {
        Operand& o = *operands[i];
        o.split.hi = o.hi = at[i]->planes;
        o.split.lo = o.lo = at[i]->planes + o.plane_bytes / sizeof(float);
        pair.s[i] = o.split;
        pair.done[i] = at[i]->done;
        pair.strays[i] = at[i]->strays;
        pair.mn[i] = o.mn ? 1 : 0;
    }
    {
        ProfScope scope(ctx, "matmul.if_wide");
        launch_kernel(ctx, split_pair_kernel, dim3(2 * ctx->prop.multiProcessorCount, 2), kPairThreads, 0, pair);
    }
    ctx->count_launch();
    auto map_of = [&](float* plane, const Operand& o, int tile) {
        return o.mn ? make_map(plane, o.nb * o.rows_pad, o.cols_pad, BK, true)
                    : make_map(plane, o.nb * o.rows_pad, o.cols_pad, tile, false);
    };
    TcArgs g{};
    g.batches = p.b0 * p.b1;
    g.splits = static_cast<int>(plan.splits);
    g.split_stride = g.batches * p.m * p.n;
    g.out = plan.splits > 1 ? partial : p.out;
    g.m = p.m;
    g.n = p.n;
    g.a_batch_rows = a_bcast ? 0 : oa.rows_pad;
    g.b_batch_rows = b_bcast ? 0 : ob.rows_pad;
    g.k_blocks = plan.k_blocks;
    g.kb_per_split = plan.kb_per_split;
    g.tiles_m = plan.tiles_m;
    g.tiles_n = plan.tiles_n;
    g.group_m = ctx->gemm_group_m > 0 ? ctx->gemm_group_m : kGroupM;
    g.status = ctx->d_status;
    g.guard = guard;
    g.done[0] = a.done;
    g.done[1] = b.done;
    int sms = ctx->prop.multiProcessorCount;
    if (ctx->in_grad_sync_span && ctx->comm_pending) sms = std::max(sms - ctx->comm_sms, sms / 2);
    const int grid = static_cast<int>(std::min<int64_t>(plan.tiles_m * plan.tiles_n * g.batches * plan.splits, sms));
    const CUtensorMap ah = map_of(oa.hi, oa, BM), al = map_of(oa.lo, oa, BM), bh = map_of(ob.hi, ob, plan.bn), bl = map_of(ob.lo, ob, plan.bn);
    {
        ProfScope scope(ctx, "matmul.if_wide");
        if (plan.bn == 256) launch_main<256, 2>(ctx, true, oa.mn, ob.mn, ah, al, bh, bl, g, grid);
        else if (plan.bn == 128) launch_main<128, 3>(ctx, true, oa.mn, ob.mn, ah, al, bh, bl, g, grid);
        else launch_main<64, 4>(ctx, true, oa.mn, ob.mn, ah, al, bh, bl, g, grid);
    }
    ctx->count_launch();
    check_last_launch("matmul (TF32 planes of a wide operand)");
}

void gemm_tc_note_uses(b200_ctx* ctx, const GemmProblem& p) {
    const int64_t batches = p.b0 * p.b1;
    (void)batches;
    const bool a_bcast = (p.a_s[0] == 0 || p.b0 == 1) && (p.a_s[1] == 0 || p.b1 == 1);
    const bool b_bcast = (p.b_s[0] == 0 || p.b0 == 1) && (p.b_s[1] == 0 || p.b1 == 1);
    ++ctx->plane_uses[plan_operand(p.a, p.a_s[0], p.a_s[1], p.a_s[2], p.a_s[3], p.m, p.k, a_bcast, p).key];
    if (plan_stream(ctx, p).ok) {
        return;  // the right operand is streamed as it is: it gets no planes
    }
    ++ctx->plane_uses[plan_operand(p.b, p.b_s[0], p.b_s[1], p.b_s[3], p.b_s[2], p.n, p.k, b_bcast, p).key];
}

void gemm_tc_invalidate(b200_ctx* ctx, const void* begin, const void* end) {
    if (ctx->plane_cache.empty()) return;
    const char* lo = static_cast<const char*>(begin);
    const char* hi = static_cast<const char*>(end);
    for (auto it = ctx->plane_cache.begin(); it != ctx->plane_cache.end();) {
        if (lo < it->second.src_end && it->second.src_begin < hi) {
            ctx->scratch.release(it->second.hi);
            ctx->plane_cache_bytes -= it->second.bytes;
            it = ctx->plane_cache.erase(it);
        } else {
            ++it;
        }
    }
}

void gemm_tc_end_span(b200_ctx* ctx) {
    for (auto& kv : ctx->plane_cache) {
        ctx->scratch.release(kv.second.hi);
    }
    ctx->plane_cache.clear();
    ctx->plane_uses.clear();
    ctx->plane_cache_bytes = 0;
    ctx->range_next = 0;
    ctx->lone_matmul = true;  // (what is asked about between two spans is a product by itself: b200_matmul_kernel)
    ctx->compared.clear();
}

}  // namespace b200
