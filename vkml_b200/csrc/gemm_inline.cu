// F32 products from two half terms per operand, split on the way into shared memory.
//
// gemm_h16.cu writes the half planes of both operands to memory before its kernel runs.  For a product that is no
// large square those passes cost as much as the product: 512 x 65536 x 512 spent 95 of 207 us on them as a pass of a program, and a
// product of a few 2^30 operations is a chain of seven launches.  Here warps of the product's own kernel read the
// caller's floats, whatever their strides, split them in registers and store the halves where the MMA reads them.
// The terms, the two accumulators, the range rules and what stands by for a wide operand are gemm_h16.cu's.
//
// Two tiles: 256 x 256 by a pair of CTAs (cta_group::2: each converts its 128 rows of either operand, 64 KB of floats per K-block for 1536 cycles
// of the tensor cores) and 128 x 64 by one, for thin results.  (128 x 128 by one CTA moves the same 64 KB through the port that L1 and shared memory
// have in common for half the work: 2650 cycles per K-block of 64, 2304 of them that port's.)
//
// Roles of a CTA's warps:
//     0-3   epilogue: tensor memory -> C, one 32-lane quarter each
//     4-7   one lane issues the MMAs (in the odd CTA of a pair it passes on that a stage is converted); for the pair's tile, whose one pair of
//           accumulators leaves nothing to issue while it is read, they are the other half of the epilogue as well
//     8-    converters: 32 floats per thread and K-block in two groups, asked for again as soon as they are converted, scaled, split, stored in the
//           128-byte swizzle that TMA would give the tile
//
// The scale comes from a sample that every CTA reads for itself -- the same elements in each, so all agree -- while
// its first K-block is on the way.  An element outside the range that the sample promised is treated as
// gemm_h16.cu's split treats it: a stray is left out and noted, by one of the CTAs that read it; an overflow,
// an infinity or a NaN, which leave a result that is not finite, make the operand wide.
//
// What bounds it: a ring of three stages of 64 K.  With the MMAs, the loads or both left out a K-block of the pair's tile takes 2375, 2560 and 1900
// cycles for 3250: converting, handing over and multiplying add up around the ring.  512x65536x512, events around the whole node: 180 us with
// planes, 120 here; as one pass of a program that has other operands each time 207 and 140.
#include "gemm.h"

#include <algorithm>
#include <type_traits>

#include <cuda_fp16.h>

#include "gemm_inline.cuh"

namespace b200 {
namespace {

constexpr int kRowsP = 128;  // accumulator lanes
constexpr int kBlockK = 64;  // halves per K-block: one 128-byte swizzle row
constexpr int kBlockTf32 = 32;  // floats of one
constexpr int kStepK = 16;
constexpr int kQuads = 8;    // float4 per converter thread and K-block
constexpr int kGroup = 4;    // ... that are asked for and converted together
constexpr int kPatchPitch = 20;  // floats: sixteen columns, rows on different banks
constexpr int kFirstConverter = 8;  // (registers are handed over by groups of four warps)
constexpr int kSamplePieces = 4;       // of 128 consecutive elements, per converter warp
constexpr int kPieces = 32;             // of one operand
constexpr uint32_t kEarlyStrays = 4;   // in a sample of 4096: more, and the matrix is taken to be wide without trying

// A thread's rows lie this many apart at most.  Their distance in bytes is held in 32 bits, which bounds the pitches that are served
// (gemm_inline_fits): 64 bits would cost a multiplication more per load, in warps that wait for nothing but their loads.
constexpr int max_row_step(bool tf32) { return tf32 ? 32 : 16; }

// One operand as the matrix with `mn` lines along K.
struct InlineSide {
    const float* base;
    int64_t s_b0, s_b1, s_mn, s_k;  // element strides
    int64_t mn;
    int64_t n_batches, b1;          // matrices it has (1: one for every batch), inner batch extent
    int quads;                      // the unit-stride axis is whole quads, each on 16 bytes
    RangeSlot* range;
    int64_t* strays;                // positions in the order of the matrix in memory
    uint32_t limit;
    int sample_step;                // bytes between neighbours along the unit-stride axis
    int64_t sample_at[kPieces];     // pieces of up to 128 of them, spread over the matrix
    uint8_t sample_len[kPieces];
};

struct InlineArgs {
    InlineSide p, q;  // the MMA's 128-row and BN-row operands
    int64_t k;
    int64_t b1;       // inner batch extent
    float* out;       // C, or the partial planes when splits > 1
    int64_t m, n;     // of C
    int swap;         // q holds C's rows
    UnitPlan units;
    int64_t split_stride;
    uint32_t* status;
};

// CG CTAs share a tile of CG * 128 x BN: each holds its 128 rows of P and BN / CG of Q.
template <int CG, int BN>
struct InlineTile {
    static constexpr int kRowsQ = BN / CG;
    static constexpr int kConverters = (kRowsP + kRowsQ) / 16;  // warps
    static constexpr int kThreads = (kFirstConverter + kConverters) * 32;
    static constexpr int kPBytes = kRowsP * kBlockK * 2;
    static constexpr int kQBytes = kRowsQ * kBlockK * 2;
    static constexpr int kStageBytes = 2 * (kPBytes + kQBytes);
    static constexpr int kStages = 192 * 1024 / kStageBytes < 4 ? 192 * 1024 / kStageBytes : 4;
    static constexpr int kAccCols = 2 * BN;  // main terms, then cross terms
    static constexpr int kAccs = 2 * kAccCols <= 512 ? 2 : 1;
    static constexpr int kTmemCols = kAccs * kAccCols;
    // One pair of accumulators: nothing is issued while it is read, so the MMA's group of warps reads half of it.
    static constexpr int kReaders = kAccs == 1 ? 2 : 1;  // groups of four warps
    static constexpr int kReaderCols = BN / kReaders;
    static constexpr int kConverterRegs = kConverters == 16 ? 88 : 112;
    static constexpr int kBars = kStages * kStageBytes;
    static constexpr int kTotal = kBars + 256 + 1024;
};

// Loads are single statements without a branch around each: where two paths meet, the loaded registers would be copied, and the copy waits for
// the load (6800 cycles per K-block).
__device__ __forceinline__ float4 load_quad(const void* p) {
    float4 v;
    asm volatile("ld.global.nc.L1::no_allocate.L2::128B.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "l"(p));
    return v;
}
__device__ __forceinline__ float load_one(const void* p) {
    float v;
    asm volatile("ld.global.nc.f32 %0, [%1];" : "=f"(v) : "l"(p));
    return v;
}
__device__ __forceinline__ float load_if(const void* p, bool there) {
    float v;
    asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %2, 0;\n\tmov.b32 %0, 0;\n\t@p ld.global.nc.f32 %0, [%1];\n\t}"
                 : "=&f"(v) : "l"(p), "r"(there ? 1 : 0));
    return v;
}

__device__ __forceinline__ int64_t batch_offset(const InlineSide& s, int64_t b1, uint32_t batch) {
    if (s.n_batches == 1) return 0;
    const uint32_t bo = batch / static_cast<uint32_t>(b1);
    return int64_t(bo) * s.s_b0 + int64_t(batch - bo * static_cast<uint32_t>(b1)) * s.s_b1;
}

// What one converter thread reads of its operand's tile and where it puts it: eight quads (TF32 terms: four) along the unit-stride axis.
// K-major: 16 (8) quads to a row of 64 (32) K.  MN-major: ROWS / 4 quads to a K-row, K-rows 8 apart.
// Past the matrix' last line or its last K the last one is read again: what a line too many gives lies outside C, and what a K too many gives is
// cleared behind the conversion.  So no load needs a predicate.
// QUAD: the unit-stride axis is whole quads, each on 16 bytes.
template <bool MN, int ROWS, bool QUAD, bool TF32 = false>
struct Feed {
    static constexpr bool kMn = MN;
    static constexpr int kBlock = TF32 ? kBlockTf32 : kBlockK;
    static constexpr int kQuads = kBlock / 8;
    static constexpr int kLanes = MN ? ROWS / 4 : kBlock / 4;
    static constexpr int kRowStep = 2 * ROWS / kLanes;
    static_assert(kRowStep <= max_row_step(TF32), "pitches are bounded by it");
    const InlineSide& s;
    int along, row;   // this thread's first element: offset along the unit axis, row of the tile
    uint32_t offset;  // of its first quad in a tile
    const char* at;   // its first quad of the K-block being requested
    int rows_apart, step[3];  // bytes between its rows; to a quad's other elements
    int last_row;     // the last of its eight rows that exists
    int k;            // K of its first element

    __device__ __forceinline__ Feed(const InlineSide& side, int t) : s(side) {
        const int c = t % kLanes;
        along = 4 * c;
        row = t / kLanes;
        if (TF32) {
            offset = MN ? (c >> 3) * kMnAtomBytes + row * 128 + ((((c & 7) >> 1) ^ (row & 3)) << 5) + (c & 1) * 16 : row * 128 + ((c ^ (row & 7)) << 4);
        } else {
            offset = MN ? (c >> 4) * kAtomBytes + row * 128 + ((((c & 15) >> 1) ^ (row & 7)) << 4) + (c & 1) * 8
                        : row * 128 + ((((c >> 1) ^ (row & 7))) << 4) + (c & 1) * 8;
        }
        rows_apart = static_cast<int>(kRowStep * (MN ? s.s_k : s.s_mn) * 4);
    }
    __device__ __forceinline__ void place(int64_t b1, uint32_t batch, uint32_t tile, uint32_t kb, int K) {
        // (the odd CTA's rows may all lie behind the last line)
        const int line0 = min(static_cast<int>(tile * ROWS), static_cast<int>(s.mn - 1) & ~3), k0 = static_cast<int>(kb * kBlock);
        const int lines = static_cast<int>(s.mn) - line0 - 1, ks = K - k0 - 1;  // behind the tile's first
        const int left = MN ? lines : ks, down = MN ? ks : lines;               // along the unit axis, across it
        const int first = QUAD ? min(along, left & ~3) : min(along, left), top = min(row, down);
        const float* base = s.base + batch_offset(s, b1, batch);
        at = reinterpret_cast<const char*>(base + int64_t(line0 + (MN ? first : top)) * s.s_mn + int64_t(k0 + (MN ? top : first)) * s.s_k);
        k = k0 + (MN ? row : along);
        last_row = min(kQuads - 1, (down - top) / kRowStep);
#pragma unroll
        for (int j = 0; j < 3; ++j) step[j] = static_cast<int>(min(j + 1, left - first) * (MN ? s.s_mn : s.s_k) * 4);
    }
    __device__ __forceinline__ void next() {  // (not onto a K-block that reaches past K)
        at += kBlock * s.s_k * 4;
        k += kBlock;
    }
    __device__ __forceinline__ float4 load(int i) const {
        const char* p = at + int64_t(min(i, last_row)) * rows_apart;
        if constexpr (QUAD) return load_quad(p);
        return make_float4(load_one(p), load_one(p + step[0]), load_one(p + step[1]), load_one(p + step[2]));
    }
    // (TF32 terms: of the sixteen elements, four to a quad)
    __device__ __forceinline__ uint32_t word(int e) const { return offset + (e >> 2) * (kRowStep * 128) + (e & 3) * 4; }
    __device__ __forceinline__ int k_of(int e) const { return MN ? row + kRowStep * (e >> 2) : along + (e & 3); }
    __device__ __forceinline__ void put(uint8_t* to, int i, const uint32_t (&v)[4]) const {
        *reinterpret_cast<uint4*>(to + word(4 * i)) = make_uint4(v[0], v[1], v[2], v[3]);
    }
};

// The same for TF32 terms where rows do not lie on 16 bytes: a warp reads 32 neighbours along the unit axis at a time -- a row of the stage
// (K-major), an atom's K-row (MN-major) -- and stores them one word to a lane.  (As four loads of a quad each, sixteen bytes from lane to lane,
// every load touched as many lines as a quad's: 1166x129x4131 33.6 us, 172x1615x2684 39.8.)
template <bool MN, int ROWS>
struct LaneFeed {
    static constexpr bool kMn = MN;
    static constexpr int kQuads = 4;  // sixteen elements, four at a time
    static constexpr int kWarps = ROWS / 16, kAtoms = ROWS / 32;
    static constexpr int kStep = MN ? 2 : kWarps;  // rows between its elements
    static_assert(kStep <= max_row_step(true), "pitches are bounded by it");
    const InlineSide& s;
    int lane, row, atom;   // of its first element
    uint32_t even, odd;    // where its elements go: their swizzle alternates
    const char* at;
    int rows_apart, last_row;

    __device__ __forceinline__ LaneFeed(const InlineSide& side, int t) : s(side) {
        const int w = t >> 5;
        lane = t & 31;
        row = MN ? w / kAtoms : w;
        atom = MN ? w % kAtoms : 0;
        auto place_of = [&](int r) {
            return static_cast<uint32_t>(MN ? atom * kMnAtomBytes + r * 128 + (((lane >> 3) ^ (r & 3)) << 5) + (lane & 7) * 4
                                            : r * 128 + (((lane >> 2) ^ (r & 7)) << 4) + (lane & 3) * 4);
        };
        even = place_of(row);
        odd = place_of(row + kStep);
        rows_apart = static_cast<int>(kStep * (MN ? s.s_k : s.s_mn) * 4);
    }
    __device__ __forceinline__ void place(int64_t b1, uint32_t batch, uint32_t tile, uint32_t kb, int K) {
        const int line0 = static_cast<int>(tile * ROWS), k0 = static_cast<int>(kb * kBlockTf32);
        const int lines = static_cast<int>(s.mn) - line0 - 1, ks = K - k0 - 1;  // behind the tile's first
        const int first = min(MN ? 32 * atom + lane : lane, MN ? lines : ks), top = min(row, MN ? ks : lines);
        const float* base = s.base + batch_offset(s, b1, batch);
        at = reinterpret_cast<const char*>(base + int64_t(line0 + (MN ? first : top)) * s.s_mn + int64_t(k0 + (MN ? top : first)) * s.s_k);
        last_row = min(15, ((MN ? ks : lines) - top) / kStep);
    }
    __device__ __forceinline__ void next() { at += kBlockTf32 * s.s_k * 4; }
    __device__ __forceinline__ float one(int e) const { return load_one(at + int64_t(min(e, last_row)) * rows_apart); }
    __device__ __forceinline__ float4 load(int i) const { return make_float4(one(4 * i), one(4 * i + 1), one(4 * i + 2), one(4 * i + 3)); }
    __device__ __forceinline__ uint32_t word(int e) const { return (e & 1 ? odd : even) + (e >> 1) * (2 * kStep * 128); }
    __device__ __forceinline__ int k_of(int e) const { return MN ? row + kStep * e : lane; }
    __device__ __forceinline__ void put(uint8_t* to, int i, const uint32_t (&v)[4]) const {
#pragma unroll
        for (int j = 0; j < 4; ++j) *reinterpret_cast<uint32_t*>(to + word(4 * i + j)) = v[j];
    }
};

// Two floats as one 64-bit operand of the paired instructions.
__device__ __forceinline__ uint64_t pair_of(float x, float y) {
    uint64_t r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(x), "f"(y));
    return r;
}
__device__ __forceinline__ float2 floats_of(uint64_t p) {
    float2 r;
    asm("mov.b64 {%0, %1}, %2;" : "=f"(r.x), "=f"(r.y) : "l"(p));
    return r;
}
__device__ __forceinline__ uint64_t mul_pair(uint64_t a, uint64_t b) {
    uint64_t r;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ uint64_t fma_pair(uint64_t a, uint64_t b, uint64_t c) {
    uint64_t r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
    return r;
}

// The scale of one operand: a power of two in one or two factors, and the smallest magnitude that keeps 22 bits under it.
struct Scale {
    float s1, s2;
    uint32_t low;  // 2 * bits - 1 of that magnitude (0: none)
    __device__ __forceinline__ explicit Scale(uint32_t max_bits) {
        const int up = range_shift(min(max_bits, 0x7F800000u));
        const bool one = up >= -126 && up <= 126;
        s1 = exp2_int(one ? up : up / 2);
        s2 = one ? 1.0F : exp2_int(up - up / 2);
        const int e = -13 - up;  // (kStrayBelow before it is scaled)
        const uint32_t bits = e > 127 ? 0x7F800000u : (e >= -126 ? static_cast<uint32_t>(e + 127) << 23 : (e >= -149 ? 1u << (e + 149) : 0u));
        low = bits == 0 ? 0u : 2 * bits - 1;
    }
};

__device__ __forceinline__ uint32_t least_of(const float4& v) {
    return min(min(2 * __float_as_uint(v.x) - 1, 2 * __float_as_uint(v.y) - 1), min(2 * __float_as_uint(v.z) - 1, 2 * __float_as_uint(v.w) - 1));
}

// x = hi + lo / 2^11, a pair of floats at a time.
__device__ __forceinline__ void half_terms(uint64_t x, uint32_t& hi, uint32_t& lo) {
    const float2 v = floats_of(x);
    const __half2 h = __floats2half2_rn(v.x, v.y);
    const float2 hf = __half22float2(h);
    const float2 r = floats_of(mul_pair(fma_pair(pair_of(hf.x, hf.y), pair_of(-1.0F, -1.0F), x), pair_of(2048.0F, 2048.0F)));  // exact
    const __half2 l = __floats2half2_rn(r.x, r.y);
    hi = *reinterpret_cast<const uint32_t*>(&h);
    lo = *reinterpret_cast<const uint32_t*>(&l);
}

// This warp's share of the sample, and the largest magnitude in it.
__device__ __forceinline__ uint32_t take_sample(const InlineSide& s, int first, int apart, float (&v)[4 * kSamplePieces]) {
    const int lane = threadIdx.x & 31;
#pragma unroll
    for (int i = 0; i < kSamplePieces; ++i) {
        const char* p = reinterpret_cast<const char*>(s.base + s.sample_at[first + i * apart]) + int64_t(lane) * s.sample_step;
#pragma unroll
        for (int j = 0; j < 4; ++j) v[4 * i + j] = load_if(p + int64_t(32 * j) * s.sample_step, lane + 32 * j < s.sample_len[first + i * apart]);
    }
    uint32_t top = 0;
#pragma unroll
    for (int i = 0; i < 4 * kSamplePieces; ++i) top = max(top, __float_as_uint(v[i]) & 0x7FFFFFFFu);
    return __reduce_max_sync(0xffffffffu, top);
}

template <int CG, int BN, bool P_MN, bool Q_MN>
__global__ void __launch_bounds__(InlineTile<CG, BN>::kThreads, 1) gemm_inline_kernel(const __grid_constant__ InlineArgs g) {
    using T = InlineTile<CG, BN>;
    constexpr int STAGES = T::kStages;
    constexpr uint32_t kIdesc = h16_idesc(CG * kRowsP, BN, P_MN, Q_MN);
    static_assert(8 * (3 * STAGES + 6) <= 256, "barrier block");

    extern __shared__ uint8_t smem_raw[];
    const uint32_t base = (smem_u32(smem_raw) + 1023u) & ~1023u;
    uint8_t* base_ptr = smem_raw + (base - smem_u32(smem_raw));
    const uint32_t bars = base + T::kBars;
    auto full_bar = [&](int s) { return bars + 8u * s; };               // a stage is converted
    auto empty_bar = [&](int s) { return bars + 8u * (STAGES + s); };   // its MMAs are done
    auto acc_full = [&](int a) { return bars + 8u * (2 * STAGES + a); };
    auto acc_empty = [&](int a) { return bars + 8u * (2 * STAGES + 2 + a); };  // the even CTA's
    const uint32_t sample_bar = bars + 8u * (2 * STAGES + 4), verdict_bar = sample_bar + 8u;  // the sample's maxima; what it says
    auto peer_bar = [&](int s) { return bars + 8u * (2 * STAGES + 6 + s); };  // the even CTA's: a stage is converted in the odd one
    __shared__ uint32_t tmem_base_slot;
    __shared__ int abort_flag;
    __shared__ uint32_t sample_max[2], sample_small[2];
    __shared__ __align__(16) float epi_patch[4 * T::kReaders][32][kPatchPitch];

    const int warp = threadIdx.x >> 5;
    const int lane = threadIdx.x & 31;
    const uint32_t rank = CG == 2 ? cluster_rank() : 0;
    const uint32_t unit0 = blockIdx.x / CG, unit_step = gridDim.x / CG;

    if (threadIdx.x == 0) {
        abort_flag = 0;
        sample_max[0] = sample_max[1] = sample_small[0] = sample_small[1] = 0;
        for (int s = 0; s < STAGES; ++s) {
            mbar_init(full_bar(s), T::kConverters);
            mbar_init(peer_bar(s), 1);
            mbar_init(empty_bar(s), 1);
        }
        for (int a = 0; a < 2; ++a) {
            mbar_init(acc_full(a), 1);
            mbar_init(acc_empty(a), 4 * T::kReaders * CG);
        }
        mbar_init(sample_bar, T::kConverters);
        mbar_init(verdict_bar, T::kConverters);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 4) {
        tmem_get<CG>(smem_u32(&tmem_base_slot), T::kTmemCols);
        tc_fence_before();
    }
    __syncthreads();
    if (CG == 2) cluster_sync();  // the other CTA's barriers are initialised
    tc_fence_after();
    const uint32_t tmem_base = tmem_base_slot;
    volatile int* abort_p = &abort_flag;
    pdl_prologue();

    auto decode = [&](uint32_t u) { return unit_of(g.units, u); };
    // whether the sample has shown that an operand is wide: nothing is computed then
    auto verdict = [&]() {
        return mbar_wait(verdict_bar, 0, abort_p, g.status) && ((volatile uint32_t*)sample_small)[0] <= kEarlyStrays &&
               ((volatile uint32_t*)sample_small)[1] <= kEarlyStrays;
    };

    // Registers: a launch of 768 threads has 80 each, and 512 x 88 + 256 x 64 are as many; one of 640 has 96, and 384 x 112 + 256 x 64 are fewer.
    if (warp >= kFirstConverter) {
        // ---------------- converters ----------------
        set_registers<true, T::kConverterRegs>();
        auto convert = [&](auto feed, const InlineSide& side, const int index, const uint32_t tile_at, const uint32_t plane_bytes, const int part,
                           const int parts, auto mn_tag) {
            constexpr bool MN = decltype(mn_tag)::value;
            const int K = static_cast<int>(g.k);
            uint32_t u = unit0;
            Unit at = decode(u);
            auto tile_of = [&](const Unit& x) { return (index == 0 ? x.tp : x.tq) * CG + rank; };
            auto place = [&](const Unit& x, uint32_t kb) { feed.place(g.b1, x.batch, tile_of(x), kb, K); };
            float4 v[kQuads];
            place(at, at.kb0);
#pragma unroll
            for (int i = 0; i < kQuads; ++i) v[i] = feed.load(i);
            bool ok = true;
            {
                float seen[4 * kSamplePieces];
                const uint32_t top = take_sample(side, part * (kPieces / parts), kPieces / (parts * kSamplePieces), seen);
                if (lane == 0) {
                    atomicMax(&sample_max[index], top);
                    mbar_arrive(sample_bar);
                }
                __syncwarp();
                ok = mbar_wait(sample_bar, 0, abort_p, g.status);
                const uint32_t low = Scale(((volatile uint32_t*)sample_max)[index]).low;
                uint32_t small = 0;
#pragma unroll
                for (int i = 0; i < 4 * kSamplePieces; ++i) small += 2 * __float_as_uint(seen[i]) - 1 < low;
                small = __reduce_add_sync(0xffffffffu, small);
                if (lane == 0) {
                    if (small != 0) atomicAdd(&sample_small[index], small);
                    mbar_arrive(verdict_bar);
                }
                __syncwarp();
                ok = ok && verdict();
                if (!ok && blockIdx.x == 0 && lane == 0) side.range->spoiled = 1;
            }
            const Scale scale(((volatile uint32_t*)sample_max)[index]);
            const uint64_t s1 = pair_of(scale.s1, scale.s1);
            const bool two = scale.s2 != 1.0F;
            uint32_t it = 0;
            for (; ok && u < g.units.n_units; u += unit_step) {
                const Unit now = at;
                for (uint32_t kb = now.kb0; kb < now.kb1; ++kb, ++it) {
                    const int s = it % STAGES;
                    const bool partial = static_cast<int>(kb + 1) * kBlockK > K;
                    bool more = true;
                    if (kb + 1 < now.kb1) {
                        if (static_cast<int>(kb + 2) * kBlockK <= K) feed.next();
                        else place(now, kb + 1);
                    } else if (u + unit_step < g.units.n_units) {
                        at = decode(u + unit_step);
                        place(at, at.kb0);
                    } else {
                        more = false;
                    }
                    if (!mbar_wait_parked(empty_bar(s), ((it / STAGES) & 1) ^ 1, abort_p, g.status)) {
                        ok = false;
                        break;
                    }
                    uint8_t* to = base_ptr + s * T::kStageBytes + tile_at + feed.offset;
                    uint32_t least = 0xFFFFFFFFu;  // 2 * bits - 1 of the smallest magnitude that is not zero
                    // two groups of four quads: a group is asked for anew as soon as it is converted, so that its loads are the only ones
                    // that its next conversion waits for (a warp has six scoreboards, shared by all eight quads if they take turns one by one)
#pragma unroll
                    for (int from = 0; from < kQuads; from += kGroup) {
                        if (two) {
#pragma unroll
                            for (int i = from; i < from + kGroup; ++i) {
                                least = min(least, least_of(v[i]));
                                v[i] = make_float4(v[i].x * scale.s2, v[i].y * scale.s2, v[i].z * scale.s2, v[i].w * scale.s2);
                            }
                        }
#pragma unroll
                        for (int i = from; i < from + kGroup; ++i) {
                            if (!two) least = min(least, least_of(v[i]));
                            uint2 hi, lo;
                            half_terms(mul_pair(pair_of(v[i].x, v[i].y), s1), hi.x, lo.x);
                            half_terms(mul_pair(pair_of(v[i].z, v[i].w), s1), hi.y, lo.y);
                            uint8_t* p = to + i * feed.kRowStep * 128;
                            *reinterpret_cast<uint2*>(p) = hi;
                            *reinterpret_cast<uint2*>(p + plane_bytes) = lo;
                        }
                        if (more) {
#pragma unroll
                            for (int i = from; i < from + kGroup; ++i) v[i] = feed.load(i);
                        }
                    }
                    if (partial || least < scale.low) {
                        // K past the matrix' end is cleared; so is what is too small for two halves beside the sample's largest, and it is noted once
                        auto again = feed;
                        again.place(g.b1, now.batch, tile_of(now), kb, K);
                        const bool note = (index == 0 ? now.tq : now.tp) == 0 && (side.n_batches != 1 || now.batch == 0);
                        const int64_t b = side.n_batches == 1 ? 0 : now.batch;
#pragma unroll 1
                        for (int i = 0; i < kQuads; ++i) {
                            const float4 q = again.load(i);
#pragma unroll
                            for (int j = 0; j < 4; ++j) {
                                const float e = j == 0 ? q.x : (j == 1 ? q.y : (j == 2 ? q.z : q.w));
                                const int64_t k = again.k + (MN ? 8 * i : j), line = int64_t(tile_of(now)) * (index == 0 ? kRowsP : T::kRowsQ) +
                                                                                      (MN ? feed.along + j : feed.row + i * feed.kRowStep);
                                const bool beyond = k >= K, stray = 2 * __float_as_uint(e) - 1 < scale.low;
                                if (!beyond && !stray) continue;
                                uint16_t* h = reinterpret_cast<uint16_t*>(to + i * feed.kRowStep * 128) + j;
                                *h = 0;
                                h[plane_bytes / 2] = 0;
                                if (beyond || !note || line >= side.mn) continue;
                                const uint32_t slot = atomicAdd(&side.range->strays, 1u);
                                if (slot < side.limit) side.strays[slot] = MN ? (b * g.k + k) * side.mn + line : (b * side.mn + line) * g.k + k;
                            }
                        }
                    }
                    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
                    __syncwarp();
                    if (lane == 0) mbar_arrive(full_bar(s));
                }
            }
            if (threadIdx.x == kFirstConverter * 32) drain_commits<STAGES>(empty_bar, it, abort_p, g.status);
        };
        constexpr int kPWarps = kRowsP / 16;
        const int t = threadIdx.x - kFirstConverter * 32;
        auto p_side = [&](auto quad) {
            convert(Feed<P_MN, kRowsP, decltype(quad)::value>(g.p, t), g.p, 0, 0, T::kPBytes, warp - kFirstConverter, kPWarps,
                    std::integral_constant<bool, P_MN>());
        };
        auto q_side = [&](auto quad) {
            convert(Feed<Q_MN, T::kRowsQ, decltype(quad)::value>(g.q, t - kPWarps * 32), g.q, 1, 2 * T::kPBytes, T::kQBytes, warp - kFirstConverter - kPWarps, T::kRowsQ / 16,
                    std::integral_constant<bool, Q_MN>());
        };
        if (warp < kFirstConverter + kPWarps) {
            if (g.p.quads) p_side(std::true_type());
            else p_side(std::false_type());
        } else {
            if (g.q.quads) q_side(std::true_type());
            else q_side(std::false_type());
        }
    } else {
        // ---------------- MMA issue (one lane of the even CTA's warp 4) and epilogue ----------------
        set_registers<false, 64>();
        const bool any = verdict();
        float f1 = 1.0F, f2 = 1.0F, f3 = 1.0F;  // 2^-(shifts) in factors that stay in range
        if (any) {
            const int e = -(range_shift(((volatile uint32_t*)sample_max)[0]) + range_shift(((volatile uint32_t*)sample_max)[1]));
            const int e1 = max(-126, min(126, e));
            const int e2 = max(-126, min(126, e - e1));
            f1 = exp2_int(e1);
            f2 = exp2_int(e2);
            f3 = exp2_int(e - e1 - e2);
        }
        const int quarter = warp & 3, col0 = (warp >> 2) * T::kReaderCols;
        const bool vec = g.n % 4 == 0 && g.split_stride % 4 == 0 && (reinterpret_cast<uintptr_t>(g.out) & 15) == 0;
        float finite = 0.0F;
        uint32_t it = 0, tile_it = 0;
        bool ok = any;
        for (uint32_t u = unit0; ok && u < g.units.n_units; u += unit_step, ++tile_it) {
            const Unit r = decode(u);
            const int acc = tile_it % T::kAccs;
            if (warp == 4 && lane == 0 && rank == 0) {
                ok = mbar_wait(acc_empty(acc), ((tile_it / T::kAccs) & 1) ^ 1, abort_p, g.status);
                tc_fence_after();
                const uint32_t d_main = tmem_base + acc * T::kAccCols;
                const uint32_t d_cross = d_main + BN;
                for (uint32_t kb = r.kb0; ok && kb < r.kb1; ++kb, ++it) {
                    const int s = it % STAGES;
                    ok = mbar_wait(full_bar(s), (it / STAGES) & 1, abort_p, g.status);
                    if (CG == 2) ok = ok && mbar_wait_cluster(peer_bar(s), (it / STAGES) & 1, abort_p, g.status);
                    if (!ok) break;
                    tc_fence_after();
                    const uint32_t stage = base + s * T::kStageBytes;
                    const uint64_t p_hi = h16_desc<P_MN>(stage);
                    const uint64_t p_lo = h16_desc<P_MN>(stage + T::kPBytes);
                    const uint64_t q_hi = h16_desc<Q_MN>(stage + 2 * T::kPBytes);
                    const uint64_t q_lo = h16_desc<Q_MN>(stage + 2 * T::kPBytes + T::kQBytes);
#pragma unroll
                    for (int kk = 0; kk < kBlockK / kStepK; ++kk) {
                        const uint64_t adv_p = static_cast<uint64_t>((P_MN ? kk * kStepK * 128 : kk * kStepK * 2) >> 4);
                        const uint64_t adv_q = static_cast<uint64_t>((Q_MN ? kk * kStepK * 128 : kk * kStepK * 2) >> 4);
                        const uint32_t further = (kb == r.kb0 && kk == 0) ? 0u : 1u;
                        umma_f16<CG>(d_cross, p_lo + adv_p, q_hi + adv_q, kIdesc, further);
                        umma_f16<CG>(d_cross, p_hi + adv_p, q_lo + adv_q, kIdesc, 1u);
                        umma_f16<CG>(d_main, p_hi + adv_p, q_hi + adv_q, kIdesc, further);
                    }
                    commit_all<CG>(empty_bar(s));
                }
                if (ok) commit_all<CG>(acc_full(acc));
            } else if (CG == 2 && warp == 4 && lane == 0) {
                // the odd CTA's stages, passed on by a thread that has no loads under way (an arrival across the pair waits for those)
                for (uint32_t kb = r.kb0; ok && kb < r.kb1; ++kb, ++it) {
                    const int s = it % STAGES;
                    ok = mbar_wait(full_bar(s), (it / STAGES) & 1, abort_p, g.status);
                    if (ok) mbar_arrive_cluster(lead_addr(peer_bar(s)));
                }
            }
            if (warp >= 4 * T::kReaders) continue;
            __syncwarp();
            if (!mbar_wait_parked(acc_full(acc), (tile_it / T::kAccs) & 1, abort_p, g.status)) break;
            tc_fence_after();
            const uint32_t t_acc = tmem_base + (static_cast<uint32_t>(quarter * 32) << 16) + acc * T::kAccCols + col0;
            const int64_t p0 = (int64_t(r.tp) * CG + rank) * kRowsP + quarter * 32, q0 = int64_t(r.tq) * BN + col0;
            const int64_t p_left = (g.swap ? g.n : g.m) - p0, q_extent = g.swap ? g.m : g.n;
            float* out = g.out + int64_t(r.split) * g.split_stride + int64_t(r.batch) * g.m * g.n;
            float* patch = &epi_patch[warp][0][0];
#pragma unroll 1
            for (int c = 0; c < T::kReaderCols; c += 16) {
                const int64_t q_left = q_extent - (q0 + c);
                if (q_left <= 0 || p_left <= 0) break;  // uniform across the warp
                uint32_t v[16], x[16];
                tmem_ld16_two(t_acc + c, t_acc + BN + c, v, x);
#pragma unroll
                for (int j = 0; j < 16; ++j) {
                    const float sum = fmaf(__uint_as_float(x[j]), 0x1p-11F, __uint_as_float(v[j]));
                    finite = fmaf(sum, 0.0F, finite);  // (an overflow among the terms leaves an infinity or a NaN)
                    v[j] = __float_as_uint(sum * f1 * f2 * f3);
                }
                if (g.swap) {
                    // lanes lie along C's rows: 32 columns of one row per store
                    float* to = out + (q0 + c) * g.n + p0 + lane;
#pragma unroll
                    for (int j = 0; j < 16; ++j) {
                        if (j < q_left && lane < p_left) *to = __uint_as_float(v[j]);
                        to += g.n;
                    }
                    continue;
                }
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    *reinterpret_cast<uint4*>(patch + lane * kPatchPitch + 4 * j) = make_uint4(v[4 * j], v[4 * j + 1], v[4 * j + 2], v[4 * j + 3]);
                }
                __syncwarp();
                float* to = out + p0 * g.n + q0 + c;
                if (vec && q_left >= 16) {
                    const int sub = lane >> 2, seg = lane & 3;
#pragma unroll
                    for (int i = 0; i < 4; ++i) {
                        const int rl = i * 8 + sub;
                        if (rl < p_left) {
                            *reinterpret_cast<float4*>(to + int64_t(rl) * g.n + seg * 4) = *reinterpret_cast<const float4*>(patch + rl * kPatchPitch + seg * 4);
                        }
                    }
                } else {
                    // a ragged right edge, or rows that do not begin on 16 bytes: two rows' sixteen columns per store
                    const int sub = lane >> 4, col = lane & 15;
#pragma unroll 4
                    for (int rl = sub; rl < 32; rl += 2) {
                        if (rl < p_left && col < q_left) to[int64_t(rl) * g.n + col] = patch[rl * kPatchPitch + col];
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
        if (finite != 0.0F) g.p.range->spoiled = 1;
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
        tmem_put<CG>(tmem_base, T::kTmemCols);
    }
}

// ---------------------------------------------------------------------------
// TF32 terms
// ---------------------------------------------------------------------------

// The same for products that take TF32 terms (gemm_tc.cu): hi and lo of each float as the planes would hold them, the same three MMAs per K-step, the
// same K-slices, so the result is that of the planes bit for bit -- from one launch instead of two splits and a product, and with no
// plane to write and read.  Neither range nor strays to look for.  One CTA to a 128 x BN tile.
template <int BN>
struct InlineTf32Tile {
    static constexpr int kConverters = (kRowsP + BN) / 16;  // warps
    static constexpr int kThreads = (kFirstConverter + kConverters) * 32;
    static constexpr int kPBytes = kRowsP * kBlockTf32 * 4;
    static constexpr int kQBytes = BN * kBlockTf32 * 4;
    static constexpr int kStageBytes = 2 * (kPBytes + kQBytes);
    static constexpr int kStages = 192 * 1024 / kStageBytes;
    static constexpr int kTmemCols = 2 * BN;  // two accumulators
    static constexpr int kConverterRegs = BN == 128 ? 96 : 112;
    static constexpr int kBars = kStages * kStageBytes;
    static constexpr int kTotal = kBars + 256 + 1024;
};

template <int BN, bool P_MN, bool Q_MN>
__global__ void __launch_bounds__(InlineTf32Tile<BN>::kThreads, 1) gemm_inline_tf32_kernel(const __grid_constant__ InlineArgs g) {
    using T = InlineTf32Tile<BN>;
    constexpr int STAGES = T::kStages;
    constexpr uint32_t kIdesc = make_idesc(kRowsP, BN, P_MN, Q_MN);
    constexpr int kPitch = 36;
    static_assert(8 * (2 * STAGES + 4) <= 256, "barrier block");

    extern __shared__ uint8_t smem_raw[];
    const uint32_t base = (smem_u32(smem_raw) + 1023u) & ~1023u;
    uint8_t* base_ptr = smem_raw + (base - smem_u32(smem_raw));
    const uint32_t bars = base + T::kBars;
    auto full_bar = [&](int s) { return bars + 8u * s; };               // a stage is converted
    auto empty_bar = [&](int s) { return bars + 8u * (STAGES + s); };   // its MMAs are done
    auto acc_full = [&](int a) { return bars + 8u * (2 * STAGES + a); };
    auto acc_empty = [&](int a) { return bars + 8u * (2 * STAGES + 2 + a); };
    __shared__ uint32_t tmem_base_slot;
    __shared__ int abort_flag;
    __shared__ __align__(16) float epi_patch[4][32][kPitch];

    const int warp = threadIdx.x >> 5;
    const int lane = threadIdx.x & 31;
    if (threadIdx.x == 0) {
        abort_flag = 0;
        for (int s = 0; s < STAGES; ++s) {
            mbar_init(full_bar(s), T::kConverters);
            mbar_init(empty_bar(s), 1);
        }
        for (int a = 0; a < 2; ++a) {
            mbar_init(acc_full(a), 1);
            mbar_init(acc_empty(a), 4);
        }
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 4) {
        tmem_alloc(smem_u32(&tmem_base_slot), T::kTmemCols);
        tc_fence_before();
    }
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem_base = tmem_base_slot;
    volatile int* abort_p = &abort_flag;
    pdl_prologue();

    // Registers: a launch of 768 threads has 80 each, one of 640 has 96; 512 x 96 (384 x 112) + 128 x 64 + 128 x 24 are fewer.
    if (warp >= kFirstConverter) {
        // ---------------- converters ----------------
        set_registers<true, T::kConverterRegs>();
        auto convert = [&](auto feed, const int index, const uint32_t tile_at, const uint32_t plane_bytes) {
            using F = decltype(feed);
            const int K = static_cast<int>(g.k);
            // where the loads are, two stages ahead of the conversion; what is left of K there
            uint32_t next_u = blockIdx.x, next_kb = 0, next_end = 0;
            auto place = [&](const Unit& x, uint32_t kb) { feed.place(g.b1, x.batch, index == 0 ? x.tp : x.tq, kb, K); };
            auto enter = [&] {
                const Unit x = unit_of(g.units, next_u);
                next_kb = x.kb0;
                next_end = x.kb1;
                place(x, x.kb0);
            };
            auto request = [&](float4 (&to)[F::kQuads], int& left) {
                left = -1;  // nothing more to convert
                if (next_u >= g.units.n_units) return;
                left = K - static_cast<int>(next_kb) * kBlockTf32;
#pragma unroll
                for (int i = 0; i < F::kQuads; ++i) to[i] = feed.load(i);
                if (++next_kb < next_end) {
                    if (static_cast<int>(next_kb + 1) * kBlockTf32 <= K) feed.next();
                    else place(unit_of(g.units, next_u), next_kb);
                } else if ((next_u += gridDim.x) < g.units.n_units) {
                    enter();
                }
            };
            float4 v0[F::kQuads], v1[F::kQuads];
            int left0, left1;
            enter();
            request(v0, left0);
            request(v1, left1);
            uint32_t it = 0;
            auto step = [&](float4 (&q)[F::kQuads], int& left) {
                const int s = it % STAGES;
                if (!mbar_wait(empty_bar(s), ((it / STAGES) & 1) ^ 1, abort_p, g.status)) return false;
                uint8_t* to = base_ptr + s * T::kStageBytes + tile_at;
                uint32_t top = 0;
#pragma unroll
                for (int i = 0; i < F::kQuads; ++i) {
                    for (float x : {q[i].x, q[i].y, q[i].z, q[i].w}) top = max(top, __float_as_uint(x) << 1);
                }
                if (top < 0xFEFFE000u) {
                    // every value is finite and rounds inside the TF32 range: add half a TF32 ulp, clear 13 bits, lo = tf32(x - hi)
#pragma unroll
                    for (int i = 0; i < F::kQuads; ++i) {
                        uint32_t hi[4], lo[4];
                        const float x[4] = {q[i].x, q[i].y, q[i].z, q[i].w};
#pragma unroll
                        for (int j = 0; j < 4; ++j) {
                            hi[j] = (__float_as_uint(x[j]) + 0x1000u) & 0xFFFFE000u;
                            const float rest = x[j] - __uint_as_float(hi[j]);
                            asm("cvt.rna.tf32.f32 %0, %1;" : "=r"(lo[j]) : "f"(rest));
                        }
                        feed.put(to, i, hi);
                        feed.put(to + plane_bytes, i, lo);
                    }
                } else {
#pragma unroll
                    for (int i = 0; i < F::kQuads; ++i) {
                        uint32_t hi[4], lo[4];
                        const float x[4] = {q[i].x, q[i].y, q[i].z, q[i].w};
#pragma unroll
                        for (int j = 0; j < 4; ++j) split_tf32_select(x[j], hi[j], lo[j]);
                        feed.put(to, i, hi);
                        feed.put(to + plane_bytes, i, lo);
                    }
                }
                if (left < kBlockTf32) {
                    // K past the matrix' end
#pragma unroll 1
                    for (int e = 0; e < 4 * F::kQuads; ++e) {
                        if (feed.k_of(e) < left) continue;
                        *reinterpret_cast<uint32_t*>(to + feed.word(e)) = 0;
                        *reinterpret_cast<uint32_t*>(to + feed.word(e) + plane_bytes) = 0;
                    }
                }
                request(q, left);
                asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
                __syncwarp();
                if (lane == 0) mbar_arrive(full_bar(s));
                ++it;
                return true;
            };
            while (left0 > 0 && step(v0, left0) && left1 > 0 && step(v1, left1)) {
            }
            if (threadIdx.x == kFirstConverter * 32) drain_commits<STAGES>(empty_bar, it, abort_p, g.status);
        };
        constexpr int kPWarps = kRowsP / 16;
        const int t = threadIdx.x - kFirstConverter * 32;
        if (warp < kFirstConverter + kPWarps) {
            if (g.p.quads) convert(Feed<P_MN, kRowsP, true, true>(g.p, t), 0, 0, T::kPBytes);
            else convert(LaneFeed<P_MN, kRowsP>(g.p, t), 0, 0, T::kPBytes);
        } else {
            if (g.q.quads) convert(Feed<Q_MN, BN, true, true>(g.q, t - kPWarps * 32), 1, 2 * T::kPBytes, T::kQBytes);
            else convert(LaneFeed<Q_MN, BN>(g.q, t - kPWarps * 32), 1, 2 * T::kPBytes, T::kQBytes);
        }
    } else if (warp >= 4) {
        // ---------------- MMA issuer ----------------
        set_registers<false, 24>();
        if (warp == 4 && lane == 0) {
            uint32_t it = 0, tile_it = 0;
            bool ok = true;
            for (uint32_t u = blockIdx.x; u < g.units.n_units && ok; u += gridDim.x, ++tile_it) {
                const Unit r = unit_of(g.units, u);
                const int acc = tile_it & 1;
                if (!mbar_wait(acc_empty(acc), ((tile_it >> 1) & 1) ^ 1, abort_p, g.status)) break;
                tc_fence_after();
                const uint32_t d = tmem_base + acc * BN;
                for (uint32_t kb = r.kb0; kb < r.kb1; ++kb, ++it) {
                    const int s = it % STAGES;
                    if (!mbar_wait(full_bar(s), (it / STAGES) & 1, abort_p, g.status)) {
                        ok = false;
                        break;
                    }
                    tc_fence_after();
                    const uint32_t stage = base + s * T::kStageBytes;
                    const uint64_t p_hi = operand_desc<P_MN>(stage);
                    const uint64_t p_lo = operand_desc<P_MN>(stage + T::kPBytes);
                    const uint64_t q_hi = operand_desc<Q_MN>(stage + 2 * T::kPBytes);
                    const uint64_t q_lo = operand_desc<Q_MN>(stage + 2 * T::kPBytes + T::kQBytes);
#pragma unroll
                    for (int kk = 0; kk < kBlockTf32 / 8; ++kk) {
                        const uint64_t adv_p = static_cast<uint64_t>((P_MN ? kk * 1024 : kk * 32) >> 4);
                        const uint64_t adv_q = static_cast<uint64_t>((Q_MN ? kk * 1024 : kk * 32) >> 4);
                        const uint32_t first = (kb == r.kb0 && kk == 0) ? 0u : 1u;
                        umma_tf32(d, p_lo + adv_p, q_hi + adv_q, kIdesc, first);
                        umma_tf32(d, p_hi + adv_p, q_lo + adv_q, kIdesc, 1u);
                        umma_tf32(d, p_hi + adv_p, q_hi + adv_q, kIdesc, 1u);
                    }
                    umma_commit(empty_bar(s));
                }
                if (ok) umma_commit(acc_full(acc));
            }
        }
    } else {
        // ---------------- epilogue ----------------
        set_registers<false, 64>();
        const bool vec = g.n % 4 == 0 && g.split_stride % 4 == 0 && (reinterpret_cast<uintptr_t>(g.out) & 15) == 0;
        uint32_t tile_it = 0;
        for (uint32_t u = blockIdx.x; u < g.units.n_units; u += gridDim.x, ++tile_it) {
            const Unit r = unit_of(g.units, u);
            const int acc = tile_it & 1;
            if (!mbar_wait_parked(acc_full(acc), (tile_it >> 1) & 1, abort_p, g.status)) break;
            tc_fence_after();
            const uint32_t t_acc = tmem_base + (static_cast<uint32_t>(warp * 32) << 16) + acc * BN;
            const int64_t p0 = int64_t(r.tp) * kRowsP + warp * 32, q0 = int64_t(r.tq) * BN;
            const int64_t p_left = g.m - p0;
            float* out = g.out + int64_t(r.split) * g.split_stride + (int64_t(r.batch) * g.m + p0) * g.n + q0;
            float* patch = &epi_patch[warp][0][0];
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
                if (vec && q_left >= 32) {
                    const int sub = lane >> 3, seg = lane & 7;
#pragma unroll
                    for (int i = 0; i < 8; ++i) {
                        const int rl = i * 4 + sub;
                        if (rl < p_left) {
                            *reinterpret_cast<float4*>(out + int64_t(rl) * g.n + c + seg * 4) = *reinterpret_cast<const float4*>(patch + rl * kPitch + seg * 4);
                        }
                    }
                } else if (lane < q_left) {
                    // a ragged right edge, or rows that do not begin on 16 bytes: a row's 32 columns per store
                    const int rows = static_cast<int>(min(int64_t(32), p_left));
#pragma unroll 4
                    for (int rl = 0; rl < rows; ++rl) out[int64_t(rl) * g.n + c + lane] = patch[rl * kPitch + lane];
                }
                __syncwarp();
            }
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(acc_empty(acc));
        }
    }

    __syncwarp();
    __syncthreads();
    if (abort_flag != 0) {
        for (int i = 0; i < 200; ++i) __nanosleep(1000);  // MMAs in flight end before their memory is given up
        __syncthreads();
    }
    if (warp == 4) {
        tc_fence_after();
        tmem_dealloc(tmem_base, T::kTmemCols);
    }
}

// ---------------------------------------------------------------------------
// Host side
// ---------------------------------------------------------------------------

InlineSide side_of(const float* base, const int64_t (&s)[4], int mn_axis, int k_axis, int64_t mn, const GemmProblem& p, bool& is_mn) {
    InlineSide o{};
    const bool one = (s[0] == 0 || p.b0 == 1) && (s[1] == 0 || p.b1 == 1);
    o.base = base;
    o.s_b0 = one ? 0 : s[0];
    o.s_b1 = one ? 0 : s[1];
    o.s_mn = s[mn_axis];
    o.s_k = s[k_axis];
    o.mn = mn;
    o.n_batches = one ? 1 : p.b0 * p.b1;
    o.b1 = p.b1;
    is_mn = s[mn_axis] == 1 && s[k_axis] != 1;  // (as the other tensor-core kernels decide it: strays are noted in that order)
    const int64_t along = is_mn ? o.s_mn : o.s_k, across = is_mn ? o.s_k : o.s_mn;
    o.quads = along == 1 && (is_mn ? mn : p.k) % 4 == 0 && across % 4 == 0 && o.s_b0 % 4 == 0 && o.s_b1 % 4 == 0 && reinterpret_cast<uintptr_t>(base) % 16 == 0;
    return o;
}

// Where the sample of a matrix is taken.
void place_sample(InlineSide& o, const GemmProblem& p, bool is_mn) {
    o.sample_step = static_cast<int>((is_mn ? o.s_mn : o.s_k) * 4);
    const int64_t cols = is_mn ? o.mn : p.k, lines = is_mn ? p.k : o.mn;
    const int64_t per_line = ceil_div(cols, int64_t(128)), total = per_line * lines * o.n_batches, stretch = total / kPieces;
    for (int64_t j = 0; j < kPieces; ++j) {
        // (a piece's place in its stretch varies, so that no pattern of the matrix is in step with it)
        const int64_t piece = total <= kPieces ? std::min(j, total - 1) : j * stretch + (j * 7919) % stretch;
        const int64_t lb = piece / per_line, col = (piece - lb * per_line) * 128, b = lb / lines, line = lb - b * lines;
        o.sample_at[j] = b / p.b1 * o.s_b0 + b % p.b1 * o.s_b1 + line * (is_mn ? o.s_k : o.s_mn) + col * (is_mn ? o.s_mn : o.s_k);
        o.sample_len[j] = static_cast<uint8_t>(std::min<int64_t>(128, cols - col));
    }
}

struct InlinePlan {
    int cg, bn;
    bool swap;
    int64_t tiles_p, tiles_q, k_blocks, splits, kb_per_split, units;
    double cost;
};

// Tile, which operand takes the 128 lanes, and K-slices, by the time of whole waves.
InlinePlan plan_inline(const b200_ctx* ctx, const GemmProblem& p) {
    struct Form { int cg, bn; double block, tail; };  // us of a K-block, and of what is not hidden behind a unit's K-blocks
    static const Form forms[] = {{2, 256, 1.75, 2.5}, {1, 64, 1.15, 1.0}};
    const int sms = ctx->prop.multiProcessorCount;
    InlinePlan best{};
    const int64_t batches = p.b0 * p.b1, k_blocks = ceil_div(p.k, kBlockK);
    bool mn;
    // (operands read one float at a time take a K-block longer)
    const bool quads = side_of(p.a, p.a_s, 2, 3, p.m, p, mn).quads && side_of(p.b, p.b_s, 3, 2, p.n, p, mn).quads;
    bool first = true;
    for (int i = 0; i < 4; ++i) {
        const Form& f = forms[i % 2];
        if (ctx->gemm_inline >= 2 && ctx->gemm_inline != 2 + i) continue;
        InlinePlan c{};
        c.cg = f.cg;
        c.bn = f.bn;
        c.swap = i >= 2;
        c.k_blocks = k_blocks;
        c.tiles_p = ceil_div(c.swap ? p.n : p.m, int64_t(f.cg) * kRowsP);
        c.tiles_q = ceil_div(c.swap ? p.m : p.n, int64_t(f.bn));
        const int64_t tiles = c.tiles_p * c.tiles_q * batches, slots = sms / f.cg;
        c.splits = 1;
        if (tiles < slots && k_blocks >= 4) c.splits = std::max<int64_t>(1, std::min({slots / tiles, k_blocks / 2, int64_t(64)}));
        c.kb_per_split = ceil_div(k_blocks, c.splits);
        c.splits = ceil_div(k_blocks, c.kb_per_split);
        c.units = tiles * c.splits;
        const double waves = double(ceil_div(c.units, slots));
        c.cost = waves * (double(c.kb_per_split) * f.block * (quads ? 1.0 : 1.3) + f.tail) +
                 (c.splits > 1 ? 3.0 + double(c.splits) * double(batches * p.m * p.n) * 1.4e-6 : 0.0);
        if (first || c.cost < best.cost) best = c;
        first = false;
    }
    return best;
}

template <int CG, int BN>
void launch_inline(b200_ctx* ctx, const InlineArgs& g, bool p_mn, bool q_mn, int grid) {
    using T = InlineTile<CG, BN>;
    auto run = [&](auto kernel) {
        B200_CUDA_CHECK(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, T::kTotal));
        if (CG == 2) launch_kernel_clustered(ctx, kernel, grid, T::kThreads, T::kTotal, CG, false, g);
        else launch_kernel(ctx, kernel, grid, T::kThreads, T::kTotal, g);
    };
    if (p_mn && q_mn) run(gemm_inline_kernel<CG, BN, true, true>);
    else if (p_mn) run(gemm_inline_kernel<CG, BN, true, false>);
    else if (q_mn) run(gemm_inline_kernel<CG, BN, false, true>);
    else run(gemm_inline_kernel<CG, BN, false, false>);
}

}  // namespace

// Where the planes would take longer to write and read than this kernel loses in its main loop: a long K beside a small result, a batch of
// thin matrices.  Both times are estimated; this path is taken where its own is 5 % less.  (A K-block of the pair's tile takes 1.75 us here -- converting,
// handing over and multiplying follow one another around a ring of three stages -- and 0.9 us from planes; the passes over the planes take 8 bytes per
// element at 5.8 TB/s.  The whole node, planes / here: 512x65536x512 180 / 120 us, 5 x 3335x2687x174 156 / 129,
// which it takes; 255x29905x606 101 / 90, which its margin leaves to planes; 2048^3 65 / 70, 4096^3 346 / 439, 751x2638x911 55 / 58.  Of 220 products with a long K or many
// thin matrices the rule takes 40, none of them more than 2 % slower than from planes and 1.33 times quicker in the mean.)  Planes that another product of the span reads too are kept.
bool gemm_inline_serves(const b200_ctx* ctx, const GemmProblem& p) {
    if (ctx->gemm_inline == 0 || ctx->gemm_inline >= 8 || ctx->gemm_precision != B200_GEMM_3XTF32 || !ctx->gemm_half_terms || ctx->compared.count(p.out) != 0) {
        return false;
    }
    if (ctx->gemm_inline > 0) return gemm_tc_eligible(ctx, p) && gemm_tc_chain(ctx, p) <= 12288 && gemm_inline_fits(p, false);
    // what takes half terms, and what would if it were not read directly
    if (!gemm_h16_would_serve(ctx, p) || !gemm_inline_fits(p, false) || gemm_h16_shares(ctx, p)) return false;
    // (what is read directly otherwise needs no memory beside its operands, and the planes that stand by take twice theirs: [1048576, 12288] x
    // 64 columns 103 GB beside 52)
    if (ctx->lone_matmul && gemm_tc_plane_bytes(p, true) + gemm_tc_plane_bytes(p, false) > gemm_tc_plane_limit(ctx) && gemm_tc_reads_directly(ctx, p)) return false;
    return (plan_inline(ctx, p).cost + 12.0) * 1.05 < gemm_h16_time(ctx, p) && gemm_tc_eligible(ctx, p);
}

std::string gemm_inline_tile(const b200_ctx* ctx, const GemmProblem& p) {
    const InlinePlan t = plan_inline(ctx, p);
    return std::to_string(t.cg * kRowsP) + "x" + std::to_string(t.bn);
}

void gemm_inline(b200_ctx* ctx, const GemmProblem& p) {
    const InlinePlan t = plan_inline(ctx, p);
    RangeSlot* slots = gemm_h16_slots(ctx, 2);
    if (slots == nullptr) {
        gemm_tc(ctx, p, true);
        return;
    }
    const int64_t out_elems = p.b0 * p.b1 * p.m * p.n;
    const int wide_splits = gemm_tc_slices(ctx, p);
    const int64_t slices = std::max<int64_t>(t.splits, wide_splits);
    const size_t partial_bytes = slices > 1 ? static_cast<size_t>(align_up(out_elems * slices * 4, 1024)) : 0;
    const size_t tf32[2] = {gemm_tc_plane_bytes(p, true), gemm_tc_plane_bytes(p, false)};
    bool mn[2];
    InlineSide side[2] = {side_of(p.a, p.a_s, 2, 3, p.m, p, mn[0]), side_of(p.b, p.b_s, 3, 2, p.n, p, mn[1])};
    Standby standby[2];
    size_t bytes = partial_bytes + 1024;
    for (int i = 0; i < 2; ++i) {
        const int64_t numel = side[i].n_batches * side[i].mn * p.k;
        side[i].limit = std::min(kMaxStrays, kStrayFloor + static_cast<uint32_t>(std::min<int64_t>(numel >> 21, kMaxStrays)));
        side[i].range = slots + i;
        place_sample(side[i], p, mn[i]);
        bytes += tf32[i] + kMaxStrays * 8;
    }
    char* ws = nullptr;
    try {
        ws = static_cast<char*>(ctx->ensure_workspace(bytes));
    } catch (const Error& e) {
        if (e.status != B200_OUT_OF_MEMORY) throw;
        gemm_tc(ctx, p, true);  // (a product that is read directly needs none of it)
        return;
    }
    ws = reinterpret_cast<char*>(align_up(reinterpret_cast<int64_t>(ws), 1024));
    for (int i = 0; i < 2; ++i) {
        standby[i].planes = reinterpret_cast<float*>(ws);
        ws += tf32[i];
        side[i].strays = reinterpret_cast<int64_t*>(ws);
        ws += kMaxStrays * 8;
        standby[i].strays = side[i].strays;
        standby[i].done = nullptr;
    }
    float* partial = reinterpret_cast<float*>(ws);

    InlineArgs g{};
    g.p = t.swap ? side[1] : side[0];
    g.q = t.swap ? side[0] : side[1];
    g.k = p.k;
    g.b1 = p.b1;
    g.out = t.splits > 1 ? partial : p.out;
    g.m = p.m;
    g.n = p.n;
    g.swap = t.swap ? 1 : 0;
    g.units = unit_plan(t.tiles_p, t.tiles_q, p.b0 * p.b1, t.splits, t.k_blocks, t.kb_per_split, 8);
    g.split_stride = out_elems;
    g.status = ctx->d_status;
    int sms = ctx->prop.multiProcessorCount;
    if (ctx->in_grad_sync_span && ctx->comm_pending) sms = std::max(sms - ctx->comm_sms, sms / 2);
    const int grid = static_cast<int>(std::min<int64_t>(t.units, sms / t.cg)) * t.cg;
    {
        ProfScope scope(ctx, "matmul.tcgen05_3xf16");
        const bool p_mn = t.swap ? mn[1] : mn[0], q_mn = t.swap ? mn[0] : mn[1];
        if (t.bn == 256) launch_inline<2, 256>(ctx, g, p_mn, q_mn, grid);
        else launch_inline<1, 64>(ctx, g, p_mn, q_mn, grid);
    }
    ctx->count_launch();
    check_last_launch("matmul (tcgen05, half terms split in the kernel)");
    const RangeGuard guard{side[0].range, side[1].range, side[0].limit, side[1].limit};
    gemm_tc_stand_by(ctx, p, guard, standby[0], standby[1], t.splits > 1 ? partial : p.out, partial);
    gemm_h16_fold(ctx, p, partial, static_cast<int>(t.splits), guard, wide_splits);
}

// TF32 terms split in the kernel: for products that would get TF32 planes, with their K-slices.
void gemm_inline_tf32(b200_ctx* ctx, const GemmProblem& p, float* partial, int64_t splits, int64_t kb_per_split, const char* label) {
    bool mn[2];
    InlineArgs g{};
    g.p = side_of(p.a, p.a_s, 2, 3, p.m, p, mn[0]);
    g.q = side_of(p.b, p.b_s, 3, 2, p.n, p, mn[1]);
    const int bn = p.n > 64 ? 128 : 64;
    g.k = p.k;
    g.b1 = p.b1;
    g.out = splits > 1 ? partial : p.out;
    g.m = p.m;
    g.n = p.n;
    g.units = unit_plan(ceil_div(p.m, int64_t(kRowsP)), ceil_div(p.n, int64_t(bn)), p.b0 * p.b1, splits, ceil_div(p.k, int64_t(kBlockTf32)), kb_per_split, 16);
    g.split_stride = p.b0 * p.b1 * p.m * p.n;
    g.status = ctx->d_status;
    int sms = ctx->prop.multiProcessorCount;
    if (ctx->in_grad_sync_span && ctx->comm_pending) sms = std::max(sms - ctx->comm_sms, sms / 2);
    const int grid = static_cast<int>(std::min<int64_t>(g.units.n_units, sms));
    auto launch = [&](auto tile, auto kernel) {
        using T = decltype(tile);
        B200_CUDA_CHECK(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, T::kTotal));
        launch_kernel(ctx, kernel, grid, T::kThreads, T::kTotal, g);
    };
    auto majors = [&](auto width) {
        constexpr int BN = decltype(width)::value;
        using T = InlineTf32Tile<BN>;
        if (mn[0] && mn[1]) launch(T{}, gemm_inline_tf32_kernel<BN, true, true>);
        else if (mn[0]) launch(T{}, gemm_inline_tf32_kernel<BN, true, false>);
        else if (mn[1]) launch(T{}, gemm_inline_tf32_kernel<BN, false, true>);
        else launch(T{}, gemm_inline_tf32_kernel<BN, false, false>);
    };
    {
        ProfScope scope(ctx, label);
        if (bn == 128) majors(std::integral_constant<int, 128>());
        else majors(std::integral_constant<int, 64>());
    }
    ctx->count_launch();
    check_last_launch("matmul (tcgen05, TF32 terms split in the kernel)");
}

// us of a K-block in the TF32 form.  An operand whose rows along K are no whole quads on 16 bytes is read a float to a lane, each row of a stage from
// two lines: 0.17 us more for either (products of one wave, fitted over 127: both so 1.34 us, one 1.1 to 1.18, quads 0.8 to 0.95 where 1 is taken).
double gemm_inline_tf32_block(const GemmProblem& p) {
    bool mn[2];
    const InlineSide side[2] = {side_of(p.a, p.a_s, 2, 3, p.m, p, mn[0]), side_of(p.b, p.b_s, 3, 2, p.n, p, mn[1])};
    return 1.0 + (mn[0] || side[0].quads ? 0.0 : 0.17) + (mn[1] || side[1].quads ? 0.0 : 0.17);
}

bool gemm_inline_fits(const GemmProblem& p, bool tf32) {
    // (a thread's neighbouring rows are less than 2^31 bytes apart: pitches below 2^25 floats for half terms, 2^24 for TF32 terms; units and
    // lines are counted in 31 bits)
    const int64_t pitch = (int64_t(1) << 31) / (4 * max_row_step(tf32));
    for (int i = 2; i < 4; ++i) {
        if (std::abs(p.a_s[i]) >= pitch || std::abs(p.b_s[i]) >= pitch) return false;
    }
    const int64_t lim = int64_t(1) << 30;
    return p.m < lim && p.n < lim && p.k < lim && p.b0 * p.b1 < lim &&
           double(ceil_div(p.m, int64_t(128))) * double(ceil_div(p.n, int64_t(64))) * double(p.b0 * p.b1) * 64.0 < double(lim);
}

}  // namespace b200
