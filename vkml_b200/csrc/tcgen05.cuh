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
