// fp32 GEMM on the CUDA cores: the path for shapes the tensor-core kernel
// does not take (tiny or ragged problems such as the 64x10 logits of the MNIST
// MLP or conv1's K = 27) and for B200_GEMM_FP32.  Two kernels: gemm_small_kernel for products
// that are over in a few microseconds (below), and, for the rest,
//
// 64x64 output tile, K in steps of 16, 256 threads with a 4x4 register block, products
// rounded before they are summed (no fused multiply-add: this is the exactness path);
// operands are read through their element strides, the staging index order is
// picked per operand so the global reads follow whichever axis has unit stride
// (a transposed view is read along its own rows).  A long K with too few tiles
// to fill 148 SMs is split across blockIdx.z into partial sums in the context's
// scratch buffer and folded in split order (deterministic, no atomics), the
// role gemm_split_k_reduce.comp plays in vkML's Vulkan backend.
#include "gemm.h"

namespace b200 {
namespace {

constexpr int BM = 64, BN = 64, BK = 16;

__global__ void __launch_bounds__(256)
gemm_simt_kernel(GemmProblem p, float* __restrict__ dst, int64_t k_chunk, int64_t split_stride) {
    pdl_prologue();
    __shared__ float As[BK][BM + 4];
    __shared__ float Bs[BK][BN + 4];

    const int64_t tiles_n = (p.n + BN - 1) / BN;
    const int64_t tiles_m = (p.m + BM - 1) / BM;
    int64_t t = blockIdx.x;
    const int64_t tn = t % tiles_n;
    t /= tiles_n;
    const int64_t tm = t % tiles_m;
    t /= tiles_m;
    const int64_t i1 = t % p.b1;
    const int64_t i0 = t / p.b1;

    const float* A = p.a + i0 * p.a_s[0] + i1 * p.a_s[1];
    const float* B = p.b + i0 * p.b_s[0] + i1 * p.b_s[1];
    const int64_t m0 = tm * BM, n0 = tn * BN;
    const int64_t k_begin = int64_t(blockIdx.z) * k_chunk;
    const int64_t k_end = min(k_begin + k_chunk, p.k);

    const int tid = threadIdx.x;
    const int tx = tid & 15, ty = tid >> 4;
    const bool a_k_fast = p.a_s[3] == 1 || p.a_s[2] != 1;  // read A along k unless m is the unit axis
    const bool b_n_fast = p.b_s[3] == 1 || p.b_s[2] != 1;  // read B along n unless k is the unit axis

    float acc[4][4] = {};

    // The next K-block travels from global memory to registers while the current one is
    // multiplied out of shared memory, so the load latency is paid once per tile, not per block.
    float ra[4], rb[4];
    auto fetch = [&](int64_t k0) {
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const int e = tid + 256 * j;
            const int mm = a_k_fast ? (e >> 4) : (e & 63);
            const int ka = a_k_fast ? (e & 15) : (e >> 6);
            const int64_t gm = m0 + mm, gka = k0 + ka;
            ra[j] = (gm < p.m && gka < k_end) ? A[gm * p.a_s[2] + gka * p.a_s[3]] : 0.0F;
            const int nn = b_n_fast ? (e & 63) : (e >> 4);
            const int kb = b_n_fast ? (e >> 6) : (e & 15);
            const int64_t gn = n0 + nn, gkb = k0 + kb;
            rb[j] = (gn < p.n && gkb < k_end) ? B[gkb * p.b_s[2] + gn * p.b_s[3]] : 0.0F;
        }
    };
    fetch(k_begin);
    for (int64_t k0 = k_begin; k0 < k_end; k0 += BK) {
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const int e = tid + 256 * j;
            As[a_k_fast ? (e & 15) : (e >> 6)][a_k_fast ? (e >> 4) : (e & 63)] = ra[j];
            Bs[b_n_fast ? (e >> 6) : (e & 15)][b_n_fast ? (e & 63) : (e >> 4)] = rb[j];
        }
        __syncthreads();
        if (k0 + BK < k_end) {
            fetch(k0 + BK);
        }
#pragma unroll
        for (int kk = 0; kk < BK; ++kk) {
            const float4 av = *reinterpret_cast<const float4*>(&As[kk][ty * 4]);
            const float4 bv = *reinterpret_cast<const float4*>(&Bs[kk][tx * 4]);
            const float a[4] = {av.x, av.y, av.z, av.w};
            const float b[4] = {bv.x, bv.y, bv.z, bv.w};
#pragma unroll
            for (int i = 0; i < 4; ++i) {
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    // a rounded product, then a rounded add -- never a fused multiply-add.  vkML's
                    // kernels round every product (shaders/gemm_reg.comp:215 `precise`; the CPU
                    // backend multiplies, then sums), and its adversarial inputs tell the two apart:
                    // alternating +-1e7 sums to exactly zero only if each 1e14 is rounded before it
                    // is added, and an overflowing product must become an infinity of its own sign
                    // so that +inf and -inf meet as NaN (tests/python/test_invariants.py:496-531).
                    acc[i][j] = __fadd_rn(__fmul_rn(a[i], b[j]), acc[i][j]);
                }
            }
        }
        __syncthreads();
    }

    float* C = dst + int64_t(blockIdx.z) * split_stride + ((i0 * p.b1) + i1) * p.m * p.n;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const int64_t gm = m0 + ty * 4 + i;
        if (gm >= p.m) {
            continue;
        }
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const int64_t gn = n0 + tx * 4 + j;
            if (gn < p.n) {
                C[gm * p.n + gn] = acc[i][j];
            }
        }
    }
}

__global__ void __launch_bounds__(256)
split_fold_kernel(float* __restrict__ out, const float* __restrict__ partial, int64_t n, int splits) {
    pdl_prologue();
    const int64_t stride = int64_t(gridDim.x) * blockDim.x;
    for (int64_t i = int64_t(blockIdx.x) * blockDim.x + threadIdx.x; i < n; i += stride) {
        float acc = partial[i];
        for (int s = 1; s < splits; ++s) {
            acc += partial[int64_t(s) * n + i];
        }
        out[i] = acc;
    }
}

// Small products, bound by latency: one launch, no second pass.  A 32x32 tile is computed by a cluster of up to
// eight CTAs, each of which takes an equal stretch of K, brings it into shared memory in as few rounds of loads as
// its length allows (128 of K per round, every load of a round in flight at once) and lets its eight warps take
// every eighth k; the partial tiles are added warp by warp in shared memory, then rank by rank through the cluster's shared
// memory -- a fixed order, no partial planes, no fold kernel.  64x784 . 784x256: 15.0 us on the
// tensor cores, 10.8 here; 128x128 . 128x1024: 9.6 -> 5.6; 256^3: 12.6 -> 7.5.
constexpr int kTile = 32, kRound = 128, kPitch = 36;

// rows x kRound elements of an operand into As[k][row]; `along_k`: k is the axis with unit stride.
__device__ __forceinline__ void load_round(float (*dst)[kPitch], const float* src, int64_t s_row, int64_t s_k, int64_t rows_left,
                                           int64_t k_left, bool along_k, bool quads) {
    const int tid = threadIdx.x;
    if (quads) {
        float4 v[4];
        if (along_k) {  // eight rows x four quads of k to a warp: the transposing stores meet two to a bank
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const int w = (tid >> 5) + 8 * j, row = (w & 3) * 8 + (tid & 7), k = (w >> 2) * 16 + ((tid >> 3) & 3) * 4;
                v[j] = row < rows_left && k < k_left ? __ldg(reinterpret_cast<const float4*>(src + row * s_row + k)) : make_float4(0, 0, 0, 0);
                if (k + 1 >= k_left) v[j].y = 0.0F;
                if (k + 2 >= k_left) v[j].z = 0.0F;
                if (k + 3 >= k_left) v[j].w = 0.0F;
            }
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const int w = (tid >> 5) + 8 * j, row = (w & 3) * 8 + (tid & 7), k = (w >> 2) * 16 + ((tid >> 3) & 3) * 4;
                dst[k][row] = v[j].x;
                dst[k + 1][row] = v[j].y;
                dst[k + 2][row] = v[j].z;
                dst[k + 3][row] = v[j].w;
            }
        } else {
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const int k = (tid >> 3) + 32 * j, row = (tid & 7) * 4;
                v[j] = row < rows_left && k < k_left ? __ldg(reinterpret_cast<const float4*>(src + k * s_k + row)) : make_float4(0, 0, 0, 0);
            }
#pragma unroll
            for (int j = 0; j < 4; ++j) *reinterpret_cast<float4*>(&dst[(tid >> 3) + 32 * j][(tid & 7) * 4]) = v[j];
        }
        return;
    }
    float v[16];
#pragma unroll
    for (int j = 0; j < 16; ++j) {
        const int e = tid + 256 * j;
        const int row = along_k ? (e >> 5 & 31) : (e & 31), k = along_k ? (e & 31) + (e >> 10) * 32 : e >> 5;
        v[j] = row < rows_left && k < k_left ? __ldg(src + row * s_row + k * s_k) : 0.0F;
    }
#pragma unroll
    for (int j = 0; j < 16; ++j) {
        const int e = tid + 256 * j;
        const int row = along_k ? (e >> 5 & 31) : (e & 31), k = along_k ? (e & 31) + (e >> 10) * 32 : e >> 5;
        dst[k][row] = v[j];
    }
}

struct SmallArgs {
    GemmProblem p;
    int64_t tiles_m, tiles_n;
    int64_t k_chunk;       // of K per CTA of a cluster
    int a_quads, b_quads;  // operands that can be read 16 bytes at a time along their unit-stride axis
    int c_quads;
    int with;              // an epilogue
    ProductEpilogue e;
};

template <int CS>
__global__ void __launch_bounds__(256) gemm_small_kernel(SmallArgs g) {
    pdl_prologue();
    __shared__ __align__(16) union {
        struct {
            float a[kRound][kPitch], b[kRound][kPitch];
        };
        float part[8][kTile][kPitch];
    } sm;
    __shared__ __align__(16) float tile_sum[kTile * kTile];
    const GemmProblem& p = g.p;
    const int rank = CS > 1 ? static_cast<int>(blockIdx.x % CS) : 0;  // (the cluster's blocks are neighbours along x)
    int64_t t = blockIdx.x / CS;
    const int64_t tn = t % g.tiles_n;
    t /= g.tiles_n;
    const int64_t tm = t % g.tiles_m, batch = t / g.tiles_m;
    const int64_t i0 = batch / p.b1, i1 = batch - i0 * p.b1;
    const int64_t m0 = tm * kTile, n0 = tn * kTile, k0 = rank * g.k_chunk, k1 = min(k0 + g.k_chunk, p.k);
    const float* A = p.a + i0 * p.a_s[0] + i1 * p.a_s[1] + m0 * p.a_s[2];
    const float* B = p.b + i0 * p.b_s[0] + i1 * p.b_s[1] + n0 * p.b_s[3];
    const int warp = threadIdx.x >> 5, lm = (threadIdx.x & 31) >> 2, ln = threadIdx.x & 3;
    const bool a_along_k = p.a_s[3] == 1 || p.a_s[2] != 1, b_along_k = p.b_s[2] == 1 && p.b_s[3] != 1;
    float acc[4][8] = {};
    for (int64_t k = k0; k < k1; k += kRound) {
        if (k > k0) __syncthreads();
        load_round(sm.a, A + k * p.a_s[3], p.a_s[2], p.a_s[3], p.m - m0, k1 - k, a_along_k, g.a_quads != 0);
        load_round(sm.b, B + k * p.b_s[2], p.b_s[3], p.b_s[2], p.n - n0, k1 - k, b_along_k, g.b_quads != 0);
        __syncthreads();
        const int steps = static_cast<int>(min(int64_t(kRound), k1 - k));
#pragma unroll 4
        for (int kk = warp; kk < steps; kk += 8) {
            const float4 av = *reinterpret_cast<const float4*>(&sm.a[kk][lm * 4]);
            const float4 b0 = *reinterpret_cast<const float4*>(&sm.b[kk][ln * 8]), b1 = *reinterpret_cast<const float4*>(&sm.b[kk][ln * 8 + 4]);
            const float a[4] = {av.x, av.y, av.z, av.w}, b[8] = {b0.x, b0.y, b0.z, b0.w, b1.x, b1.y, b1.z, b1.w};
#pragma unroll
            for (int i = 0; i < 4; ++i) {
#pragma unroll
                for (int j = 0; j < 8; ++j) acc[i][j] = __fadd_rn(__fmul_rn(a[i], b[j]), acc[i][j]);  // two roundings, as below
            }
        }
    }
    __syncthreads();
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        *reinterpret_cast<float4*>(&sm.part[warp][lm * 4 + i][ln * 8]) = make_float4(acc[i][0], acc[i][1], acc[i][2], acc[i][3]);
        *reinterpret_cast<float4*>(&sm.part[warp][lm * 4 + i][ln * 8 + 4]) = make_float4(acc[i][4], acc[i][5], acc[i][6], acc[i][7]);
    }
    __syncthreads();
    auto add4 = [](float4& s, const float4& v) {
        s.x += v.x;
        s.y += v.y;
        s.z += v.z;
        s.w += v.w;
    };
    const int row = threadIdx.x >> 3, col = (threadIdx.x & 7) * 4;
    float4 sum = *reinterpret_cast<const float4*>(&sm.part[0][row][col]);
#pragma unroll
    for (int w = 1; w < 8; ++w) add4(sum, *reinterpret_cast<const float4*>(&sm.part[w][row][col]));
    auto store = [&](int r, int c, const float4& v) {
        if (m0 + r >= p.m || n0 + c >= p.n) return;
        float* dst = p.out + (batch * p.m + m0 + r) * p.n + n0 + c;
        if (g.c_quads) {
            *reinterpret_cast<float4*>(dst) = v;
        } else {
            dst[0] = v.x;
            if (n0 + c + 1 < p.n) dst[1] = v.y;
            if (n0 + c + 2 < p.n) dst[2] = v.z;
            if (n0 + c + 3 < p.n) dst[3] = v.w;
        }
        if (g.with != 0) {
            const int64_t i = dst - p.out;
            const float e[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                if (n0 + c + j < p.n) write_epilogue(g.e, i + j, n0 + c + j, e[j]);
            }
        }
    };
    if constexpr (CS == 1) {
        store(row, col, sum);
    } else {
        *reinterpret_cast<float4*>(&tile_sum[threadIdx.x * 4]) = sum;
        cluster_sync();
        constexpr int kShare = 256 / CS;  // quads of the tile that this CTA adds up
        if (threadIdx.x < kShare) {
            const int q = rank * kShare + threadIdx.x;
            const uint32_t mine = static_cast<uint32_t>(__cvta_generic_to_shared(&tile_sum[q * 4]));
            float4 total = make_float4(0, 0, 0, 0);
#pragma unroll
            for (int r = 0; r < CS; ++r) {
                uint32_t at;
                float4 v;
                asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(at) : "r"(mine), "r"(r));
                asm volatile("ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(at) : "memory");
                if (r == 0) total = v;
                else add4(total, v);
            }
            store(q >> 3, (q & 7) * 4, total);
        }
        cluster_sync();
    }
}

// Reading 16 bytes at a time along the unit-stride axis: every row, batch and stretch of K begins on 16 bytes, and
// what follows the last row or k of a quad is the same row's own (the axis that the quads run along is whole quads, or the rest is masked).
bool quad_operand(const float* base, int64_t unit_extent, int64_t s_other, int64_t s_b0, int64_t s_b1) {
    return reinterpret_cast<uintptr_t>(base) % 16 == 0 && unit_extent % 4 == 0 && s_other % 4 == 0 && s_b0 % 4 == 0 && s_b1 % 4 == 0;
}

struct SmallPlan {
    int64_t tiles;
    int cs;  // CTAs that share a tile's K: one round of loads each, as long as the SMs are not all busy with tiles
};

SmallPlan small_plan(const GemmProblem& p) {
    SmallPlan s{p.b0 * p.b1 * ceil_div(p.m, kTile) * ceil_div(p.n, kTile), 1};
    while (s.cs < 8 && p.k > kRound * s.cs && s.tiles * s.cs * 2 <= 2 * sm_count()) s.cs *= 2;
    return s;
}

bool gemm_small(b200_ctx* ctx, const GemmProblem& p, const ProductEpilogue* epilogue) {
    if (!gemm_small_serves(p)) return false;
    SmallArgs g{};
    g.p = p;
    g.tiles_m = ceil_div(p.m, kTile);
    g.tiles_n = ceil_div(p.n, kTile);
    const auto [tiles, cs] = small_plan(p);
    g.with = epilogue != nullptr ? 1 : 0;
    if (epilogue != nullptr) g.e = *epilogue;
    g.k_chunk = ceil_div(ceil_div(p.k, cs), 4) * 4;
    const bool a_k = p.a_s[3] == 1 || p.a_s[2] != 1, b_k = p.b_s[2] == 1 && p.b_s[3] != 1;
    g.a_quads = a_k ? p.a_s[3] == 1 && quad_operand(p.a, p.k, p.a_s[2], p.a_s[0], p.a_s[1]) : quad_operand(p.a, p.m, p.a_s[3], p.a_s[0], p.a_s[1]);
    g.b_quads = b_k ? quad_operand(p.b, p.k, p.b_s[3], p.b_s[0], p.b_s[1]) : p.b_s[3] == 1 && quad_operand(p.b, p.n, p.b_s[2], p.b_s[0], p.b_s[1]);
    g.c_quads = p.n % 4 == 0 && reinterpret_cast<uintptr_t>(p.out) % 16 == 0;
    const unsigned grid = static_cast<unsigned>(tiles * cs);
    ProfScope scope(ctx, "matmul.fp32_simt");
    if (cs == 1) launch_kernel(ctx, gemm_small_kernel<1>, grid, 256, 0, g);
    else if (cs == 2) launch_kernel_clustered(ctx, gemm_small_kernel<2>, grid, 256, 0, 2, true, g);
    else if (cs == 4) launch_kernel_clustered(ctx, gemm_small_kernel<4>, grid, 256, 0, 4, true, g);
    else launch_kernel_clustered(ctx, gemm_small_kernel<8>, grid, 256, 0, 8, true, g);
    ctx->count_launch();
    check_last_launch("matmul (small)");
    return true;
}

}  // namespace

// Products of up to 2^27 operations: this kernel or the tensor cores?  Up to 2^25 it is this one, in full fp32.  (With more CTAs than are
// resident at once the tensor cores' 22 bits would be had sooner: 32 x 128x32x128 8.1 us against 11.9, 700x33x700 8.5 against 13.8.)
// Above, measured over 55 shapes in three layouts, it wins against operands read directly or through planes while all CTAs are
// resident, two to an SM, a CTA has two rounds of K and the tensor cores no K-slices, which they have from sixteen K-blocks on:
// 264^3 12.5 against 17.2 us, 275x376x276 14.1 against 21.1, 384^3 15.6 against 21.2, 2048x136x68 10.5 against 12.3; but 300x900x100 15.4 against
// 13.4, 400^3 (four rounds) 20.8 against 22.4, 4096x100x100 (512 CTAs) 15.2 against 11.3.  Streamed operands and batches stay on the tensor cores
// there (64x1024x512 14.5 against 17.4; 2 x 300x300x100 would take 13.3 for 18.5).
bool gemm_small_pays(const GemmProblem& p, bool streams) {
    const double flops = 2.0 * double(p.m) * double(p.n) * double(p.k) * double(p.b0 * p.b1);
    if (flops <= double(1 << 25)) return true;
    if (flops > double(1 << 27) || streams || p.b0 * p.b1 != 1) return false;
    const SmallPlan s = small_plan(p);
    return s.tiles * s.cs <= 2 * sm_count() && ceil_div(p.k, s.cs) <= 2 * kRound && p.k <= 480;
}

bool gemm_small_serves(const GemmProblem& p) {
    // (what takes longer than a few microseconds is better off with larger tiles and less traffic per product)
    const double flops = 2.0 * double(p.m) * double(p.n) * double(p.k) * double(p.b0 * p.b1);
    return flops > 0 && (flops <= double(1 << 26) || gemm_small_pays(p, false)) && small_plan(p).tiles <= (int64_t(1) << 28);
}

void gemm_simt(b200_ctx* ctx, const GemmProblem& p, const ProductEpilogue* epilogue) {
    const int64_t batches = p.b0 * p.b1;
    const int64_t out_elems = batches * p.m * p.n;
    if (out_elems == 0) {
        return;
    }
    if (p.k == 0) {
        B200_CUDA_CHECK(cudaMemsetAsync(p.out, 0, sizeof(float) * out_elems, ctx->stream));
        return;
    }
    if (gemm_small(ctx, p, epilogue)) {
        return;
    }
    const int64_t tiles = batches * ceil_div(p.m, BM) * ceil_div(p.n, BN);
    if (tiles > 0x7fffffffLL) {
        fail(B200_NOT_IMPLEMENTED, "matmul: too many output tiles for one launch");
    }
    int64_t splits = 1;
    // few tiles and a long K: spread K over the idle SMs in chunks of at least 48 (three
    // K-blocks, enough for the register prefetch to overlap anything)
    if (tiles < sm_count() && p.k >= 192) {
        splits = std::min<int64_t>(ceil_div(2 * sm_count(), tiles), p.k / 48);
        splits = std::max<int64_t>(1, std::min<int64_t>(splits, 64));
    }
    int64_t k_chunk = ceil_div(ceil_div(p.k, splits), BK) * BK;
    splits = ceil_div(p.k, k_chunk);
    float* dst = p.out;
    if (splits > 1) {
        dst = static_cast<float*>(ctx->ensure_workspace(sizeof(float) * out_elems * splits));
    }
    dim3 grid(static_cast<unsigned>(tiles), 1, static_cast<unsigned>(splits));
    ProfScope scope(ctx, "matmul.fp32_simt");
    launch_kernel(ctx, gemm_simt_kernel, grid, 256, 0, p, dst, k_chunk, out_elems);
    ctx->count_launch();
    if (splits > 1) {
        launch_kernel(ctx, split_fold_kernel, grid_for(out_elems, 256), 256, 0, p.out, dst, out_elems,
                                                                           static_cast<int>(splits));
        ctx->count_launch();
    }
    check_last_launch("matmul (simt)");
}

}  // namespace b200
