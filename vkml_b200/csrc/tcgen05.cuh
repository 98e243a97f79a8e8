// What the tensor-core kernels share: mbarrier, TMA and tcgen05 wrappers, shared-memory matrix
// descriptors, bounded waits, and the driver entry point that encodes tensor maps.
#pragma once

#include "gemm.h"

#include <cuda.h>  // CUtensorMap and the cuTensorMapEncodeTiled prototype (types only)

namespace b200 {
namespace {

constexpr uint64_t kWaitLimitNs = 4000000000ULL;  // 4 s


__device__ __forceinline__ uint32_t smem_u32(const void* p) {
    return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}

__device__ __forceinline__ void mbar_init(uint32_t bar, uint32_t count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(count));
}

__device__ __forceinline__ void mbar_arrive_expect_tx(uint32_t bar, uint32_t bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes)
                 : "memory");
}

__device__ __forceinline__ void mbar_arrive(uint32_t bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory");
}

__device__ __forceinline__ bool mbar_try_wait(uint32_t bar, uint32_t parity) {
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok)
        : "r"(bar), "r"(parity)
        : "memory");
    return ok != 0;
}

// The same test, but the hardware may park the thread for up to `hint_ns` while the phase is
// still open (it is woken when the phase completes).  For the many warps that wait for one
// event, a parked warp leaves the issue slots and the shared-memory pipe to the warps that work.
__device__ __forceinline__ bool mbar_try_wait_parked(uint32_t bar, uint32_t parity, uint32_t hint_ns) {
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2, %3;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok)
        : "r"(bar), "r"(parity), "r"(hint_ns)
        : "memory");
    return ok != 0;
}

__device__ __forceinline__ uint64_t global_ns() {
    uint64_t t;
    asm volatile("mov.u64 %0, %globaltimer;" : "=l"(t));
    return t;
}

// Bounded wait. Returns false (and raises the abort flag) when the limit ran out
// or another role already aborted.
__device__ __forceinline__ bool mbar_wait(uint32_t bar, uint32_t parity, volatile int* abort_flag,
                                          uint32_t* status, uint64_t limit_ns = kWaitLimitNs) {
    // The clock is only consulted every 1024 polls (reading %globaltimer costs far more than a
    // poll, and the converter warps wait here once per K-block), so the limit is the stated time
    // plus at most 1024 polls.
    uint64_t start = 0;
    uint32_t spins = 0;
    while (!mbar_try_wait(bar, parity)) {
        if ((++spins & 0x3ff) == 0) {
            if (*abort_flag != 0) {
                return false;
            }
            const uint64_t now = global_ns();
            if (start == 0) {
                start = now;
            } else if (now - start > limit_ns) {
                *abort_flag = 1;
                atomicOr(status, kStatusWaitTimedOut);
                return false;
            }
        }
    }
    return true;
}

// ... for what the other CTA of a pair has written before it arrived.
__device__ __forceinline__ bool mbar_wait_cluster(uint32_t bar, uint32_t parity, volatile int* abort_flag, uint32_t* status) {
    if (!mbar_wait(bar, parity, abort_flag, status)) return false;
    asm volatile("fence.acq_rel.cluster;" ::: "memory");
    return true;
}

// Bounded wait for the warps of a many-waiter role: parked polls, the clock read every 64 of them.
__device__ __forceinline__ bool mbar_wait_parked(uint32_t bar, uint32_t parity, volatile int* abort_flag,
                                                 uint32_t* status) {
    uint64_t start = 0;
    uint32_t spins = 0;
    while (!mbar_try_wait_parked(bar, parity, 2000u)) {
        if ((++spins & 0x3f) == 0) {
            if (*abort_flag != 0) {
                return false;
            }
            const uint64_t now = global_ns();
            if (start == 0) {
                start = now;
            } else if (now - start > kWaitLimitNs) {
                *abort_flag = 1;
                atomicOr(status, kStatusWaitTimedOut);
                return false;
            }
        }
    }
    return true;
}

// The commits of a ring's last round (`used` stages filled in all) have arrived: nobody waits for them otherwise, and one that came
// after the CTA had retired would land on a barrier of whatever CTA has its shared memory then.
template <int STAGES, typename Bar>
__device__ __forceinline__ void drain_commits(Bar empty_bar, uint32_t used, volatile int* abort_flag, uint32_t* status) {
    for (uint32_t i = 0; i < static_cast<uint32_t>(STAGES) && i < used; ++i) {
        const uint32_t last = used - 1 - i;
        if (!mbar_wait(empty_bar(last % STAGES), (last / STAGES) & 1, abort_flag, status)) return;
    }
}

__device__ __forceinline__ void tma_load_2d(uint32_t dst, const CUtensorMap* map, uint32_t bar, int c0,
                                            int c1) {
    asm volatile(
        "cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];"
        ::"r"(dst), "l"(reinterpret_cast<uint64_t>(map)), "r"(bar), "r"(c0), "r"(c1)
        : "memory");
}

__device__ __forceinline__ void tma_load_4d(uint32_t dst, const CUtensorMap* map, uint32_t bar, int c0, int c1,
                                            int c2, int c3) {
    asm volatile(
        "cp.async.bulk.tensor.4d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5, %6}], [%2];"
        ::"r"(dst), "l"(reinterpret_cast<uint64_t>(map)), "r"(bar), "r"(c0), "r"(c1), "r"(c2), "r"(c3)
        : "memory");
}

__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }

// (Instructions marked .aligned want the whole warp at once.  Lanes leave a bounded wait, a role's branch or a ragged store
// each by itself, and nothing makes the compiler bring them together before an asm statement, so every wrapper does.)
__device__ __forceinline__ void tmem_alloc(uint32_t dst_smem, uint32_t cols) {
    __syncwarp();
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(dst_smem), "r"(cols)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
}

__device__ __forceinline__ void tmem_dealloc(uint32_t taddr, uint32_t cols) {
    __syncwarp();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(cols) : "memory");
}

__device__ __forceinline__ void umma_tf32(uint32_t tmem_d, uint64_t adesc, uint64_t bdesc, uint32_t idesc,
                                          uint32_t accumulate) {
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::tf32 [%0], %1, %2, %3, p;\n\t}"
        ::"r"(tmem_d), "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate)
        : "memory");
}

// Arrives on `bar` once every tcgen05.mma issued so far by this thread has finished.
__device__ __forceinline__ void umma_commit(uint32_t bar) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar)
                 : "memory");
}

__device__ __forceinline__ uint32_t cluster_rank() {
    uint32_t r;
    asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
    return r;
}

// The address, in the cluster's shared window, of the even CTA's copy of a shared-memory location.
__device__ __forceinline__ uint32_t lead_addr(uint32_t addr) {
    uint32_t r;
    asm volatile("mapa.shared::cluster.u32 %0, %1, 0;" : "=r"(r) : "r"(addr));
    return r;
}

__device__ __forceinline__ void mbar_arrive_cluster(uint32_t addr) {
    asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];" ::"r"(addr) : "memory");
}

template <int CG>
__device__ __forceinline__ void umma_f16(uint32_t d, uint64_t a, uint64_t b, uint32_t idesc, uint32_t accumulate) {
    if constexpr (CG == 2) {
        asm volatile(
            "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
            "tcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, p;\n\t}"
            ::"r"(d), "l"(a), "l"(b), "r"(idesc), "r"(accumulate) : "memory");
    } else {
        asm volatile(
            "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
            "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}"
            ::"r"(d), "l"(a), "l"(b), "r"(idesc), "r"(accumulate) : "memory");
    }
}

// Arrives on `bar` of every CTA of the tile once the MMAs issued so far are done.
template <int CG>
__device__ __forceinline__ void commit_all(uint32_t bar) {
    if constexpr (CG == 2) {
        asm volatile(
            "tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;"
            ::"r"(bar), "h"(static_cast<uint16_t>(3)) : "memory");
    } else {
        umma_commit(bar);
    }
}

template <int CG>
__device__ __forceinline__ void tmem_get(uint32_t dst_smem, uint32_t cols) {
    __syncwarp();
    if constexpr (CG == 2) {
        asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(dst_smem), "r"(cols) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
    } else {
        tmem_alloc(dst_smem, cols);
    }
}

template <int CG>
__device__ __forceinline__ void tmem_put(uint32_t taddr, uint32_t cols) {
    __syncwarp();
    if constexpr (CG == 2) {
        asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(cols) : "memory");
    } else {
        tmem_dealloc(taddr, cols);
    }
}

__device__ __forceinline__ void tmem_ld32(uint32_t taddr, uint32_t (&r)[32]) {
    __syncwarp();
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x32.b32 "
        "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, "
        "%16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
          "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]),
          "=r"(r[16]), "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]),
          "=r"(r[24]), "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
        : "r"(taddr)
        : "memory");
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
}

// Sixteen columns at each of two places, one wait for both.
__device__ __forceinline__ void tmem_ld16_two(uint32_t t0, uint32_t t1, uint32_t (&a)[16], uint32_t (&b)[16]) {
    __syncwarp();
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 "
        "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%32];\n\t"
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 "
        "{%16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%33];\n\t"
        "tcgen05.wait::ld.sync.aligned;"
        : "=&r"(a[0]), "=&r"(a[1]), "=&r"(a[2]), "=&r"(a[3]), "=&r"(a[4]), "=&r"(a[5]), "=&r"(a[6]), "=&r"(a[7]),
          "=&r"(a[8]), "=&r"(a[9]), "=&r"(a[10]), "=&r"(a[11]), "=&r"(a[12]), "=&r"(a[13]), "=&r"(a[14]), "=&r"(a[15]),
          "=&r"(b[0]), "=&r"(b[1]), "=&r"(b[2]), "=&r"(b[3]), "=&r"(b[4]), "=&r"(b[5]), "=&r"(b[6]), "=&r"(b[7]),
          "=&r"(b[8]), "=&r"(b[9]), "=&r"(b[10]), "=&r"(b[11]), "=&r"(b[12]), "=&r"(b[13]), "=&r"(b[14]), "=&r"(b[15])
        : "r"(t0), "r"(t1)
        : "memory");
}

__device__ __forceinline__ uint64_t smem_desc(uint32_t smem_addr, uint32_t lbo_bytes, uint32_t sbo_bytes,
                                              uint32_t layout_type) {
    uint64_t d = 0;
    d |= static_cast<uint64_t>((smem_addr & 0x3FFFF) >> 4);   // start address, bits 0-13
    d |= static_cast<uint64_t>(lbo_bytes >> 4) << 16;         // leading-dimension byte offset, bits 16-29
    d |= static_cast<uint64_t>(sbo_bytes >> 4) << 32;         // stride-dimension byte offset, bits 32-45
    d |= static_cast<uint64_t>(1) << 46;                      // descriptor version for sm_100
    d |= static_cast<uint64_t>(layout_type) << 61;            // 2: 128-byte swizzle, 1: same with 32-byte atoms
    return d;
}

// Shared-memory matrix descriptors, 128-byte swizzle, 32-bit elements.
//
// K-major tile ([rows][32 floats], one swizzle row per matrix row): 8-row groups are 1024
// bytes apart (stride-dimension offset); the leading-dimension offset is unused because the
// K extent of one instruction (8 floats = 32 bytes) lies inside the swizzle row.  One K step
// advances the start address by 32 bytes.
//
// MN-major tile (the operand is stored with its M or N axis contiguous, as a row-major
// [K][N] matrix is for B): the tile is a row of "atoms", each 32 K-rows of 128 bytes (32
// floats along MN).  32-bit operands must use the 128-byte swizzle with 32-byte atomicity
// here (layout type 1, TMA mode SWIZZLE_128B_ATOM_32B): the pattern repeats every 4 K-rows,
// so the stride-dimension offset is 512 bytes; the next atom along MN starts kMnAtomBytes
// later (leading-dimension offset).  One K step (8 K-rows) advances the start by 1024 bytes.
constexpr uint32_t kMnAtomBytes = 32 * 128;  // 32 K-rows x 128 bytes

template <bool MN_MAJOR>
__device__ __forceinline__ uint64_t operand_desc(uint32_t smem_addr) {
    return MN_MAJOR ? smem_desc(smem_addr, kMnAtomBytes, 512, 1) : smem_desc(smem_addr, 0, 1024, 2);
}

// Instruction descriptor: D = f32, A = B = tf32, M x N tile, operand majors as given.
__host__ __device__ constexpr uint32_t make_idesc(int m, int n, bool a_mn, bool b_mn) {
    return (1u << 4) | (2u << 7) | (2u << 10) | (a_mn ? (1u << 15) : 0u) | (b_mn ? (1u << 16) : 0u) |
           (static_cast<uint32_t>(n >> 3) << 17) | (static_cast<uint32_t>(m >> 4) << 24);
}

// D = f32, A = B = f16.
__host__ __device__ constexpr uint32_t h16_idesc(int m, int n, bool a_mn, bool b_mn) {
    return (1u << 4) | (a_mn ? (1u << 15) : 0u) | (b_mn ? (1u << 16) : 0u) | (static_cast<uint32_t>(n >> 3) << 17) |
           (static_cast<uint32_t>(m >> 4) << 24);
}

// Tiles of 16-bit elements, 128-byte swizzle.  K-major: rows of 64 halves, 8-row groups 1024 bytes apart,
// one K-step is 32 bytes further.  MN-major: atoms of 64 K-rows x 128 bytes (64 elements along MN), 8-row
// groups again 1024 bytes apart, the next atom along MN 8192 bytes further, one K-step 16 rows further.
constexpr uint32_t kAtomBytes = 64 * 128;

template <bool MN>
__device__ __forceinline__ uint64_t h16_desc(uint32_t addr) {
    return smem_desc(addr, MN ? kAtomBytes : 0, 1024, 2);
}

// A float's two TF32 terms without a branch, for warps that convert while the tensor cores run: a few
// warps per scheduler cannot hide a taken-or-not decision per element, and sixteen independent
// elements interleave only if they are one basic block.  hi on the integer pipe (add half a TF32
// ulp, clear 13 bits; where that reaches the infinity exponent -- x is infinite, NaN, or finite
// but rounds past the largest TF32 -- truncate instead, keeping a NaN a NaN), lo = tf32(x - hi)
// on the conversion pipe, forced to zero for a non-finite x.  Same values as split_tf32.
__device__ __forceinline__ void split_tf32_select(float x, uint32_t& hi, uint32_t& lo) {
    const uint32_t b = __float_as_uint(x);
    uint32_t h = (b + 0x1000u) & 0xFFFFE000u;
    const bool nonfinite = (b & 0x7F800000u) == 0x7F800000u;
    const bool over = nonfinite || (h & 0x7F800000u) == 0x7F800000u;  // (a NaN's carry can leave the exponent)
    const bool is_nan = nonfinite && (b & 0x007FFFFFu) != 0u;
    h = over ? (b & 0xFFFFE000u) : h;
    h = is_nan ? (h | 0x00400000u) : h;
    const float rest = x - __uint_as_float(h);  // exact for a finite x
    uint32_t l;
    asm("cvt.rna.tf32.f32 %0, %1;" : "=r"(l) : "f"(rest));
    hi = h;
    lo = nonfinite ? 0u : l;
}

using EncodeTiledFn = CUresult (*)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                   const cuuint64_t*, const cuuint32_t*, const cuuint32_t*,
                                   CUtensorMapInterleave, CUtensorMapSwizzle, CUtensorMapL2promotion,
                                   CUtensorMapFloatOOBfill);

EncodeTiledFn encode_tiled() {
    static EncodeTiledFn fn = [] {
        void* p = nullptr;
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) != cudaSuccess ||
            q != cudaDriverEntryPointSuccess) {
            cudaGetLastError();
            return static_cast<EncodeTiledFn>(nullptr);
        }
        return reinterpret_cast<EncodeTiledFn>(p);
    }();
    return fn;
}

int64_t align_up(int64_t v, int64_t a) { return (v + a - 1) / a * a; }

// ---- ranges (gemm_h16.cu) ----

constexpr float kStrayBelow = 0x1p-13F;   // scaled magnitudes below this keep fewer than 22 bits in two halves
constexpr uint32_t kStrayFloor = 32;      // as many such elements as any matrix may have

// 2^e for -126 <= e <= 127
__device__ __forceinline__ float exp2_int(int e) { return __uint_as_float(static_cast<uint32_t>(e + 127) << 23); }

// The power of two that takes the largest magnitude of a matrix's sample (its bits, finite) into [2^13, 2^14).
__device__ __forceinline__ int range_shift(uint32_t max_bits) {
    if (max_bits == 0) return 0;
    const int e = max_bits >= 0x00800000u ? static_cast<int>(max_bits >> 23) - 127 : -118 - __clz(max_bits);
    return 13 - e;
}

__device__ __forceinline__ bool range_wide(const RangeSlot* s, uint32_t limit) {
    const uint4 v = __ldcg(reinterpret_cast<const uint4*>(s));
    return v.x >= 0x7F800000u || v.y > limit || v.z != 0 || v.w > kStrayFloor;
}

// Whether one of the guard's matrices is wide; every thread of the block calls it.  Two of them ask: all warps of a large grid reading the
// same few words took 4 to 6 us.
__device__ __forceinline__ bool block_wide(const RangeGuard& g) {
    return __syncthreads_or(threadIdx.x < 2 && range_wide(threadIdx.x == 0 ? g.a : g.b, threadIdx.x == 0 ? g.limit_a : g.limit_b)) != 0;
}

}  // namespace
}  // namespace b200
