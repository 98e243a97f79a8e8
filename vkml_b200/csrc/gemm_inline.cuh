// What the kernels share whose own warps bring their operands into shared memory (gemm_inline.cu, gemm_f16_any.cu): units of work and the
// registers' division among the roles.
#pragma once

#include "tcgen05.cuh"

#include <algorithm>
#include <type_traits>

namespace b200 {
namespace {

// How a product is cut: tiles of P (the MMA's rows) and Q, K-slices, batches; P-tiles in groups.
struct UnitPlan {
    uint32_t n_units, tiles_p, tiles_q, group_p, k_blocks, kb_per_split;
    FastDiv by_splits, by_batch, by_group;  // K-slices; tiles of a batch; tiles of a group of P-tiles
};

// A tile and a K-slice of one batch.
struct Unit {
    uint32_t split, batch, tp, tq, kb0, kb1;
};

__device__ __forceinline__ Unit unit_of(const UnitPlan& g, uint32_t u) {
    Unit r;
    uint32_t t, in_batch, group, in_group;
    g.by_splits.divmod(u, t, r.split);
    g.by_batch.divmod(t, r.batch, in_batch);
    g.by_group.divmod(in_batch, group, in_group);
    const uint32_t first = group * g.group_p, rows = min(g.group_p, g.tiles_p - first);
    r.tq = in_group / rows;
    r.tp = first + (in_group - r.tq * rows);
    r.kb0 = r.split * g.kb_per_split;
    r.kb1 = min(r.kb0 + g.kb_per_split, g.k_blocks);
    return r;
}

inline UnitPlan unit_plan(int64_t tiles_p, int64_t tiles_q, int64_t batches, int64_t splits, int64_t k_blocks, int64_t kb_per_split, int group) {
    UnitPlan u{};
    u.n_units = static_cast<uint32_t>(tiles_p * tiles_q * batches * splits);
    u.tiles_p = static_cast<uint32_t>(tiles_p);
    u.tiles_q = static_cast<uint32_t>(tiles_q);
    u.group_p = static_cast<uint32_t>(std::min<int64_t>(tiles_p, group));
    u.k_blocks = static_cast<uint32_t>(k_blocks);
    u.kb_per_split = static_cast<uint32_t>(kb_per_split);
    u.by_splits = FastDiv(static_cast<uint32_t>(splits));
    u.by_batch = FastDiv(u.tiles_p * u.tiles_q);
    u.by_group = FastDiv(u.group_p * u.tiles_q);
    return u;
}

// The calling warps' register count from here on; their group of four warps calls it.
template <bool MORE, int N>
__device__ __forceinline__ void set_registers() {
    __syncwarp();
    if constexpr (MORE) asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(N));
    else asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(N));
}

}  // namespace
}  // namespace b200
