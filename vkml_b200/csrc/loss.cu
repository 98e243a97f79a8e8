// The nodes of a cross-entropy loss, in the three runs that vkML's graph and autograd emit them in
// (src/api/ops.cpp:347-354,417-441; src/autograd/autograd.cpp:528-546), each as one pass over the rows:
//
//   head       [[full  full  div]  contiguous(rows)  neg]  contiguous(rows, classes)  cast(labels)  arange  equal  cast  mul
//   backward   log_softmax(x)  exp  sum(g, -1, keepdim)  mul  sub
//   value      mul(logp, onehot)  sum(-1)  neg  mean
//
// and head + backward together where they follow one another.  Every node's value still goes to its own
// buffer, so the passes are bound by writing: 7 planes of floats and one of bytes per element of the logits for
// head + backward.  What is saved is reading those planes back (five of them) and up to twelve launches.
// Values are those of the separate kernels, operation by operation; sums over a row are taken in another
// fixed order.  [1024, 32000]: both spans 495 -> 278 us, 218 of them head and backward
// (1.08 GB, 4.9 TB/s: nearly all of it writes, for which a plain fill reaches 5.6); [65536, 10]: sixteen launches and
// 45.7 us -> two and 15.1.
#include "context.h"
#include "tcgen05.cuh"

namespace b200 {
namespace {

struct LossArgs {
    int64_t rows;
    uint32_t cols;
    FastDiv by_cols;
    // head
    float* scalars[3];       // full, full and their quotient (null: the run starts behind them)
    float scalar_values[3];
    const float* scale;      // one value for the first node, `scale_stride` elements apart per row
    int64_t scale_stride;
    float* spread;           // contiguous(rows) and neg (null: the run starts at the plane)
    float* negated;
    float* plane;
    const int64_t* labels;
    int64_t label_stride;
    float* wanted;
    float* index;
    uint8_t* equal;
    float* onehot;
    float* picked;
    // backward
    const float* x;
    const float* g;          // what is summed: `picked` of a head, or read
    float* logp;
    float* prob;
    float* total;
    float* share;
    float* grad;
    int quads;               // every plane begins on 16 bytes
};

// The row's values of the head's vectors; every thread of the row's group calls it, `first` writes them.
__device__ __forceinline__ void head_row(const LossArgs& a, int64_t r, bool first, float& scale, float& wanted) {
    const float v = a.scalars[0] != nullptr ? a.scalar_values[2] : a.scale[r * a.scale_stride];
    scale = a.negated != nullptr ? -v : v;
    wanted = static_cast<float>(a.labels[r * a.label_stride]);
    if (first) {
        if (r == 0 && a.scalars[0] != nullptr) {
            for (int i = 0; i < 3; ++i) *a.scalars[i] = a.scalar_values[i];
        }
        if (a.negated != nullptr) {
            a.spread[r] = v;
            a.negated[r] = scale;
        }
        a.wanted[r] = wanted;
    }
}

template <int W>
__device__ __forceinline__ void get(const float* p, float (&v)[W]) {
    if constexpr (W == 4) {
        const float4 t = *reinterpret_cast<const float4*>(p);
        v[0] = t.x; v[1] = t.y; v[2] = t.z; v[3] = t.w;
    } else {
        v[0] = *p;
    }
}

template <int W, bool STREAM>
__device__ __forceinline__ void put(float* p, const float (&v)[W]) {
    if constexpr (W == 4) {
        const float4 t = make_float4(v[0], v[1], v[2], v[3]);
        if constexpr (STREAM) __stcs(reinterpret_cast<float4*>(p), t);
        else *reinterpret_cast<float4*>(p) = t;
    } else {
        if constexpr (STREAM) __stcs(p, v[0]);
        else *p = v[0];
    }
}

// What head and backward write for W neighbouring elements of row r from column c on.
template <bool HEAD, bool BACK, int W, bool STREAM>
__device__ __forceinline__ void loss_elements(const LossArgs& a, int64_t at, uint32_t c, float scale, float wanted, const float (&x)[W],
                                              const float (&g_in)[W], float peak, float lg, float total) {
    float g[W];
    if constexpr (HEAD) {
        float plane[W], hot[W];
        uint32_t bits = 0;
#pragma unroll
        for (int w = 0; w < W; ++w) {
            const bool hit = wanted == static_cast<float>(c + w);
            bits |= (hit ? 1u : 0u) << (8 * w);
            plane[w] = scale;
            hot[w] = hit ? 1.0F : 0.0F;
            g[w] = __fmul_rn(scale, hot[w]);
        }
        put<W, STREAM>(a.plane + at, plane);
        put<W, STREAM>(a.onehot + at, hot);
        put<W, STREAM>(a.picked + at, g);
        if constexpr (W == 4) *reinterpret_cast<uint32_t*>(a.equal + at) = bits;
        else a.equal[at] = static_cast<uint8_t>(bits);
    } else {
#pragma unroll
        for (int w = 0; w < W; ++w) g[w] = g_in[w];
    }
    if constexpr (BACK) {
        float l[W], e[W], s[W], d[W];
#pragma unroll
        for (int w = 0; w < W; ++w) {
            l[w] = (x[w] - peak) - lg;
            e[w] = expf(l[w]);
            s[w] = __fmul_rn(e[w], total);
            d[w] = __fsub_rn(g[w], s[w]);
        }
        put<W, STREAM>(a.logp + at, l);
        put<W, STREAM>(a.prob + at, e);
        put<W, STREAM>(a.share + at, s);
        put<W, STREAM>(a.grad + at, d);
    }
}

template <int GROUP>
__device__ __forceinline__ float group_max(float v, float* red) {
#pragma unroll
    for (int o = GROUP < 32 ? GROUP / 2 : 16; o > 0; o >>= 1) v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, o));
    if constexpr (GROUP > 32) {
        if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = v;
        __syncthreads();
        v = red[0];
#pragma unroll
        for (int w = 1; w < GROUP / 32; ++w) v = fmaxf(v, red[w]);
        __syncthreads();
    }
    return v;
}

template <int GROUP>
__device__ __forceinline__ float group_sum(float v, float* red) {
#pragma unroll
    for (int o = GROUP < 32 ? GROUP / 2 : 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    if constexpr (GROUP > 32) {
        if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = v;
        __syncthreads();
        v = red[0];
#pragma unroll
        for (int w = 1; w < GROUP / 32; ++w) v += red[w];
        __syncthreads();
    }
    return v;
}

// Rows begin on any element, so a row is its quads -- from the first element that lies on 16 bytes on -- and
// up to three single elements before and after them, one for each of the group's first lanes.  (All planes
// begin on 16 bytes, so the same quads are aligned in each of them.)
struct RowQuads {
    uint32_t head, quads, edge;  // elements before the quads; quads; this lane's single element (>= cols: none)
    __device__ __forceinline__ RowQuads(int64_t base, uint32_t cols, uint32_t lane) {
        head = static_cast<uint32_t>(-base) & 3u;
        quads = (cols - head) / 4;
        const uint32_t tail = head + 4 * quads;
        edge = lane < head ? lane : (lane >= 4 && lane < 8 && tail + lane - 4 < cols ? tail + lane - 4 : 0xFFFFFFFFu);
    }
};

// A row's sum of `picked`: the scale where the label is a class, and scale x 0 everywhere else -- nothing, or a NaN where the
// scale is not finite.
__device__ __forceinline__ float head_total(const LossArgs& a, float scale, float wanted) {
    const bool hit = wanted >= 0.0F && wanted < static_cast<float>(a.cols);
    const float off = a.cols > (hit ? 1u : 0u) ? __fmul_rn(scale, 0.0F) : 0.0F;
    return __fadd_rn(hit ? scale : 0.0F, off);
}

// A group of threads per row -- a warp up to 1024 classes, a block up to 4096 -- with the row's logits in registers.  Up to 128 classes, where the
// machine's warps would take more than one row each, eight threads: a warp to a row of 47 leaves most of its lanes idle (forward and backward
// with the loss's value, [17795, 47] 25.0 us with a warp, 18.7 with eight threads; [60000, 33] 55.7 and 29.0; [9473, 107] 20.8 and 18.8, where the line
// lies; but 278 rows of 107 9.8 and 14.4).
constexpr int64_t kManyRows = 64;  // per SM: eight blocks of eight warps
template <bool HEAD, bool BACK, int GROUP, int ITEMS>
__global__ void __launch_bounds__(256) loss_rows_kernel(LossArgs a) {
    pdl_prologue();
    constexpr int kRows = 256 / GROUP;
    __shared__ float red[32];
    const uint32_t lane = threadIdx.x % GROUP;
    if (HEAD) {
        for (int64_t c = int64_t(blockIdx.x) * blockDim.x + threadIdx.x; c < a.cols; c += int64_t(gridDim.x) * blockDim.x) {
            a.index[c] = static_cast<float>(c);
        }
    }
    constexpr int kInWarp = GROUP < 32 ? 32 / GROUP : 1;  // rows that a warp has at a time: it goes through them together, past the end over the last one again
    const uint32_t in_warp = GROUP < 32 ? (threadIdx.x & 31) / GROUP : 0;
    for (int64_t first = int64_t(blockIdx.x) * kRows + threadIdx.x / (GROUP * kInWarp) * kInWarp; first < a.rows; first += int64_t(gridDim.x) * kRows) {
        const int64_t r = min(first + in_warp, a.rows - 1);
        const bool live = GROUP >= 32 || first + in_warp < a.rows;
        const int64_t base = r * a.cols;
        const RowQuads q(base, a.cols, lane);
        float scale = 0.0F, wanted = -1.0F, peak = -INFINITY, lg = 0.0F, total = 0.0F;
        if constexpr (HEAD) head_row(a, r, lane == 0, scale, wanted);
        float v[ITEMS * 4], gv[ITEMS * 4], ve[1] = {-INFINITY}, ge[1] = {0.0F};
        if constexpr (BACK) {
            float sum = 0.0F;
            if (q.edge < a.cols) {
                get<1>(a.x + base + q.edge, ve);
                if constexpr (!HEAD) get<1>(a.g + base + q.edge, ge);
            }
            peak = ve[0];
            sum = ge[0];
#pragma unroll
            for (int i = 0; i < ITEMS; ++i) {
                const uint32_t u = lane + i * GROUP;
                float t[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY}, h[4] = {0.0F, 0.0F, 0.0F, 0.0F};
                if (u < q.quads) {
                    get<4>(a.x + base + q.head + u * 4, t);
                    if constexpr (!HEAD) get<4>(a.g + base + q.head + u * 4, h);
                }
#pragma unroll
                for (int w = 0; w < 4; ++w) {
                    v[4 * i + w] = t[w];
                    gv[4 * i + w] = h[w];
                    peak = fmaxf(peak, t[w]);
                    sum += h[w];
                }
            }
            peak = group_max<GROUP>(peak, red);
            float denom = expf(ve[0] - peak);
#pragma unroll
            for (int i = 0; i < ITEMS * 4; ++i) denom += expf(v[i] - peak);
            lg = logf(group_sum<GROUP>(denom, red));
            total = HEAD ? head_total(a, scale, wanted) : group_sum<GROUP>(sum, red);
            if (lane == 0) a.total[r] = total;
        }
        if (!live) continue;
        if (q.edge < a.cols) {
            loss_elements<HEAD, BACK, 1, false>(a, base + q.edge, q.edge, scale, wanted, ve, ge, peak, lg, total);
        }
#pragma unroll
        for (int i = 0; i < ITEMS; ++i) {
            const uint32_t c = q.head + (lane + i * GROUP) * 4;
            if (lane + i * GROUP < q.quads) {
                float t[4], h[4];
#pragma unroll
                for (int w = 0; w < 4; ++w) { t[w] = v[4 * i + w]; h[w] = gv[4 * i + w]; }
                loss_elements<HEAD, BACK, 4, false>(a, base + c, c, scale, wanted, t, h, peak, lg, total);
            }
        }
    }
}

// Longer rows (a vocabulary): one persistent block per SM holds a row in shared memory, and the bulk-copy engine
// brings the next row in behind it, chunk by chunk as this one's are written, so that reading the
// logits never stops the writing.  (Rows re-read from L2 by three smaller blocks per SM took 245 us at [1024, 32000]
// -- 1024 rows make 2.3 waves of those -- against 218 here.)
// Rows of up to 16384 and 8192 classes leave room for more and smaller blocks, so that one block's rows are written while another reduces
// its own (this launch by itself, [689, 6337]: 51 us with one block of 1024 threads, 32 with six of 256, of 64 and 45 for the whole loss; [4000, 4500]
// 222 and 119).  A row's head planes do not depend on
// its logits and are written first: they drain while the row is reduced.
constexpr int kLongThreads = 1024;
constexpr int kLongChunks = 8;
constexpr uint32_t kLongMax = 51200;  // classes: 200 KB of shared memory

template <bool HEAD, bool BACK, int THREADS>
__global__ void __launch_bounds__(THREADS, 1536 / THREADS) loss_long_kernel(LossArgs a, uint32_t* status) {
    extern __shared__ __align__(16) float row[];
    __shared__ uint64_t landed[kLongChunks];
    __shared__ int abort_flag;
    __shared__ float red[32];
    const uint32_t tid = threadIdx.x;
    if (tid == 0) {
        abort_flag = 0;
        for (int c = 0; c < kLongChunks; ++c) mbar_init(smem_u32(&landed[c]), 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    }
    __syncthreads();
    pdl_prologue();
    if (HEAD) {
        for (int64_t c = int64_t(blockIdx.x) * THREADS + tid; c < a.cols; c += int64_t(gridDim.x) * THREADS) {
            a.index[c] = static_cast<float>(c);
        }
    }
    auto chunk = [&](uint32_t quads, int c, uint32_t& q0, uint32_t& q1) {
        const uint32_t per = (quads + kLongChunks - 1) / kLongChunks;
        q0 = min(quads, c * per);
        q1 = min(quads, q0 + per);
    };
    auto fetch = [&](int64_t r, int c) {
        const RowQuads q(r * a.cols, a.cols, 0);
        uint32_t q0, q1;
        chunk(q.quads, c, q0, q1);
        const uint32_t bar = smem_u32(&landed[c]), bytes = (q1 - q0) * 16;
        mbar_arrive_expect_tx(bar, bytes);
        if (bytes > 0) {
            asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
                         ::"r"(smem_u32(row + q0 * 4)), "l"(a.x + r * a.cols + q.head + q0 * 4), "r"(bytes), "r"(bar) : "memory");
        }
    };
    if (tid == 0 && blockIdx.x < a.rows) {
        for (int c = 0; c < kLongChunks; ++c) fetch(blockIdx.x, c);
    }
    uint32_t phase = 0;
    for (int64_t r = blockIdx.x; r < a.rows; r += gridDim.x, phase ^= 1) {
        const int64_t base = r * a.cols;
        const RowQuads q(base, a.cols, tid);
        float scale = 0.0F, wanted = -1.0F, peak, sum = 0.0F, ve[1] = {-INFINITY}, ge[1] = {0.0F};
        if constexpr (HEAD) {
            head_row(a, r, tid == 0, scale, wanted);
            const float none[4] = {}, one[1] = {};
            if (q.edge < a.cols) loss_elements<true, false, 1, true>(a, base + q.edge, q.edge, scale, wanted, one, one, 0.0F, 0.0F, 0.0F);
            for (uint32_t u = tid; u < q.quads; u += THREADS) {
                const uint32_t col = q.head + u * 4;
                loss_elements<true, false, 4, true>(a, base + col, col, scale, wanted, none, none, 0.0F, 0.0F, 0.0F);
            }
        }
        if (q.edge < a.cols) {
            get<1>(a.x + base + q.edge, ve);
            if constexpr (!HEAD) get<1>(a.g + base + q.edge, ge);
        }
        peak = ve[0];
        sum = ge[0];
        bool ok = true;
        for (int c = 0; c < kLongChunks && ok; ++c) {
            ok = mbar_wait_parked(smem_u32(&landed[c]), phase, &abort_flag, status);
            uint32_t q0, q1;
            chunk(q.quads, c, q0, q1);
            for (uint32_t u = q0 + tid; u < q1; u += THREADS) {
                float t[4];
                get<4>(row + u * 4, t);
                peak = fmaxf(fmaxf(fmaxf(peak, t[0]), fmaxf(t[1], t[2])), t[3]);
                if constexpr (!HEAD) {
                    get<4>(a.g + base + q.head + u * 4, t);
                    sum += (t[0] + t[1]) + (t[2] + t[3]);
                }
            }
        }
        if (__syncthreads_or(!ok)) break;
        peak = group_max<THREADS>(peak, red);
        float denom = expf(ve[0] - peak);
        for (uint32_t u = tid; u < q.quads; u += THREADS) {
            float t[4];
            get<4>(row + u * 4, t);
            denom += (expf(t[0] - peak) + expf(t[1] - peak)) + (expf(t[2] - peak) + expf(t[3] - peak));
        }
        const float lg = logf(group_sum<THREADS>(denom, red));
        const float total = HEAD ? head_total(a, scale, wanted) : group_sum<THREADS>(sum, red);
        if (tid == 0) a.total[r] = total;
        if (q.edge < a.cols) {
            if constexpr (HEAD) ge[0] = __fmul_rn(scale, wanted == static_cast<float>(q.edge) ? 1.0F : 0.0F);
            loss_elements<false, BACK, 1, true>(a, base + q.edge, q.edge, scale, wanted, ve, ge, peak, lg, total);
        }
        for (int c = 0; c < kLongChunks; ++c) {
            uint32_t q0, q1;
            chunk(q.quads, c, q0, q1);
            for (uint32_t u = q0 + tid; u < q1; u += THREADS) {
                const uint32_t col = q.head + u * 4;
                float t[4], h[4] = {};
                get<4>(row + u * 4, t);
                if constexpr (!HEAD) get<4>(a.g + base + col, h);
                if constexpr (HEAD) {
#pragma unroll
                    for (int w = 0; w < 4; ++w) h[w] = __fmul_rn(scale, wanted == static_cast<float>(col + w) ? 1.0F : 0.0F);
                }
                loss_elements<false, BACK, 4, true>(a, base + col, col, scale, wanted, t, h, peak, lg, total);
            }
            __syncthreads();
            if (tid == 0 && r + gridDim.x < a.rows) fetch(r + gridDim.x, c);
        }
    }
    if (abort_flag != 0) {
        for (int i = 0; i < 200; ++i) __nanosleep(1000);  // copies in flight land before the block retires
    }
}

// Anything else: rows longer than shared memory, buffers that do not begin on 16 bytes, and a head by
// itself (nothing to reduce, so any split of its elements will do).  Logits are read twice.
template <bool HEAD, bool BACK>
__global__ void __launch_bounds__(256) loss_any_kernel(LossArgs a) {
    pdl_prologue();
    __shared__ float red[32];
    if (HEAD) {
        for (int64_t c = int64_t(blockIdx.x) * 256 + threadIdx.x; c < a.cols; c += int64_t(gridDim.x) * 256) a.index[c] = static_cast<float>(c);
    }
    for (int64_t r = blockIdx.x; r < a.rows; r += gridDim.x) {
        const int64_t base = r * a.cols;
        float scale = 0.0F, wanted = -1.0F, peak = -INFINITY, lg = 0.0F, total = 0.0F;
        if constexpr (HEAD) head_row(a, r, threadIdx.x == 0, scale, wanted);
        if constexpr (BACK) {
            float denom = 0.0F, sum = 0.0F;
#pragma unroll 4
            for (uint32_t c = threadIdx.x; c < a.cols; c += 256) peak = fmaxf(peak, a.x[base + c]);
            peak = group_max<256>(peak, red);
#pragma unroll 4
            for (uint32_t c = threadIdx.x; c < a.cols; c += 256) {
                denom += expf(a.x[base + c] - peak);
                if (!HEAD) sum += a.g[base + c];
            }
            lg = logf(group_sum<256>(denom, red));
            total = HEAD ? head_total(a, scale, wanted) : group_sum<256>(sum, red);
            if (threadIdx.x == 0) a.total[r] = total;
        }
#pragma unroll 2
        for (uint32_t c = threadIdx.x; c < a.cols; c += 256) {
            const float x[1] = {BACK ? a.x[base + c] : 0.0F}, g[1] = {BACK && !HEAD ? a.g[base + c] : 0.0F};
            loss_elements<HEAD, BACK, 1, false>(a, base + c, c, scale, wanted, x, g, peak, lg, total);
        }
    }
}

// Up to 32 classes: a block takes kTileRows whole rows as one run of memory, a thread reduces a row out of
// shared memory, and everything is written in the run's order.
constexpr int kTileRows = 128;
constexpr uint32_t kTileCols = 32;

template <bool HEAD, bool BACK>
__global__ void __launch_bounds__(256) loss_tile_kernel(LossArgs a) {
    pdl_prologue();
    // (rows lie an odd number of words apart: a thread to a row of 32 met 31 others on its bank)
    __shared__ float xs[BACK ? kTileRows * (kTileCols + 1) : 1];
    __shared__ float gs[BACK && !HEAD ? kTileRows * (kTileCols + 1) : 1];
    const uint32_t pitch = a.cols | 1u;
    __shared__ float row_scale[kTileRows], row_wanted[kTileRows], row_peak[kTileRows], row_lg[kTileRows], row_total[kTileRows];
    const int64_t r0 = int64_t(blockIdx.x) * kTileRows;
    const int rows = static_cast<int>(min(int64_t(kTileRows), a.rows - r0));
    const uint32_t n = rows * a.cols;
    const int64_t base = r0 * a.cols;
    if (HEAD && blockIdx.x == 0 && threadIdx.x < a.cols) a.index[threadIdx.x] = static_cast<float>(threadIdx.x);
    // (the block's run of memory begins on 16 bytes; what is no whole quad at its end, or all of it where a plane does not, goes by elements)
    const uint32_t quads = a.quads != 0 ? n / 4 : 0;
    if constexpr (BACK) {
        auto keep = [&](uint32_t i, float x, float g) {
            uint32_t r, c;
            a.by_cols.divmod(i, r, c);
            xs[r * pitch + c] = x;
            if constexpr (!HEAD) gs[r * pitch + c] = g;
        };
        for (uint32_t u = threadIdx.x; u < quads; u += blockDim.x) {
            float x[4], g[4] = {};
            get<4>(a.x + base + 4 * u, x);
            if constexpr (!HEAD) get<4>(a.g + base + 4 * u, g);
#pragma unroll
            for (int w = 0; w < 4; ++w) keep(4 * u + w, x[w], g[w]);
        }
        for (uint32_t i = 4 * quads + threadIdx.x; i < n; i += blockDim.x) keep(i, a.x[base + i], HEAD ? 0.0F : a.g[base + i]);
        __syncthreads();
    }
    if (threadIdx.x < rows) {
        const int t = threadIdx.x;
        float scale = 0.0F, wanted = -1.0F;
        if constexpr (HEAD) head_row(a, r0 + t, true, scale, wanted);
        row_scale[t] = scale;
        row_wanted[t] = wanted;
        if constexpr (BACK) {
            const float* x = xs + t * pitch;
            float peak = -INFINITY, denom = 0.0F, total = 0.0F;
            for (uint32_t c = 0; c < a.cols; ++c) peak = fmaxf(peak, x[c]);
            for (uint32_t c = 0; c < a.cols; ++c) denom += expf(x[c] - peak);
            if constexpr (HEAD) {
                total = head_total(a, scale, wanted);
            } else {
                for (uint32_t c = 0; c < a.cols; ++c) total += gs[t * pitch + c];
            }
            row_peak[t] = peak;
            row_lg[t] = logf(denom);
            row_total[t] = total;
            a.total[r0 + t] = total;
        }
    }
    __syncthreads();
    for (uint32_t u = threadIdx.x; u < quads; u += blockDim.x) {
        // (four elements of one or more rows: the values of loss_elements, element by element)
        float plane[4], hot[4], g[4], l[4], e[4], sh[4], d[4];
        uint32_t bits = 0;
#pragma unroll
        for (int w = 0; w < 4; ++w) {
            uint32_t r, c;
            a.by_cols.divmod(4 * u + w, r, c);
            if constexpr (HEAD) {
                const bool hit = row_wanted[r] == static_cast<float>(c);
                bits |= (hit ? 1u : 0u) << (8 * w);
                plane[w] = row_scale[r];
                hot[w] = hit ? 1.0F : 0.0F;
                g[w] = __fmul_rn(plane[w], hot[w]);
            } else {
                g[w] = gs[r * pitch + c];
            }
            if constexpr (BACK) {
                l[w] = (xs[r * pitch + c] - row_peak[r]) - row_lg[r];
                e[w] = expf(l[w]);
                sh[w] = __fmul_rn(e[w], row_total[r]);
                d[w] = __fsub_rn(g[w], sh[w]);
            }
        }
        const int64_t at = base + 4 * u;
        if constexpr (HEAD) {
            put<4, false>(a.plane + at, plane);
            put<4, false>(a.onehot + at, hot);
            put<4, false>(a.picked + at, g);
            *reinterpret_cast<uint32_t*>(a.equal + at) = bits;
        }
        if constexpr (BACK) {
            put<4, false>(a.logp + at, l);
            put<4, false>(a.prob + at, e);
            put<4, false>(a.share + at, sh);
            put<4, false>(a.grad + at, d);
        }
    }
    for (uint32_t i = 4 * quads + threadIdx.x; i < n; i += blockDim.x) {
        uint32_t r, c;
        a.by_cols.divmod(i, r, c);
        const float x[1] = {BACK ? xs[r * pitch + c] : 0.0F}, g[1] = {BACK && !HEAD ? gs[r * pitch + c] : 0.0F};
        loss_elements<HEAD, BACK, 1, false>(a, base + i, c, row_scale[r], row_wanted[r], x, g, BACK ? row_peak[r] : 0.0F,
                                            BACK ? row_lg[r] : 0.0F, BACK ? row_total[r] : 0.0F);
    }
}

// ---- value: mul, sum, neg, mean ----

struct ValueArgs {
    int64_t rows;
    uint32_t cols;
    FastDiv by_cols;
    const float* a;
    const float* b;
    float* product;
    float* sum;
    float* negated;
    float* mean;
    int quads;           // a, b and product begin on 16 bytes
    float* partial;      // one word per block
    unsigned* arrived;   // counts the blocks; wraps to zero by itself
};

// The block's share of the mean (valid in thread 0) goes to its word; the block that arrives last adds the
// words in block order and writes the mean.
__device__ __forceinline__ void finish_mean(const ValueArgs& v, float mine) {
    __shared__ bool last;
    __shared__ float red[32];
    if (threadIdx.x == 0) {
        v.partial[blockIdx.x] = mine;
        __threadfence();
        last = atomicInc(v.arrived, gridDim.x - 1) == gridDim.x - 1;
        __threadfence();
    }
    __syncthreads();
    if (!last) return;
    float s = 0.0F;
    for (uint32_t i = threadIdx.x; i < gridDim.x; i += blockDim.x) s += __ldcg(v.partial + i);
    s = group_sum<256>(s, red);
    if (threadIdx.x == 0) *v.mean = s / static_cast<float>(v.rows);
}

template <int GROUP, bool QUADS>
__global__ void __launch_bounds__(256) loss_value_kernel(ValueArgs v) {
    pdl_prologue();
    constexpr int kRows = 256 / GROUP;
    __shared__ float red[32];
    const uint32_t lane = threadIdx.x % GROUP;
    float mean = 0.0F;  // of the rows this group's first thread has seen
    constexpr int kInWarp = GROUP < 32 ? 32 / GROUP : 1;  // (as in loss_rows_kernel)
    const uint32_t in_warp = GROUP < 32 ? (threadIdx.x & 31) / GROUP : 0;
    for (int64_t first = int64_t(blockIdx.x) * kRows + threadIdx.x / (GROUP * kInWarp) * kInWarp; first < v.rows; first += int64_t(gridDim.x) * kRows) {
        // (a bound that a group of a warp or more does not need cost its kernel eight registers: [17388, 205] 41.3 us forward and backward, 39.5 without)
        const int64_t r = GROUP >= 32 ? first : min(first + in_warp, v.rows - 1);
        const bool live = GROUP >= 32 || first + in_warp < v.rows;
        const int64_t base = r * v.cols;
        float s = 0.0F;
        auto single = [&](uint32_t c) {
            const float p = __fmul_rn(v.a[base + c], v.b[base + c]);
            v.product[base + c] = p;
            s += p;
        };
        if constexpr (QUADS) {
            const RowQuads q(base, v.cols, lane);
            if (q.edge < v.cols) single(q.edge);
#pragma unroll 4
            for (uint32_t u = lane; u < q.quads; u += GROUP) {
                const int64_t at = base + q.head + u * 4;
                float x[4], y[4];
                get<4>(v.a + at, x);
                get<4>(v.b + at, y);
#pragma unroll
                for (int w = 0; w < 4; ++w) x[w] = __fmul_rn(x[w], y[w]);
                s += (x[0] + x[1]) + (x[2] + x[3]);
                put<4, false>(v.product + at, x);
            }
        } else {
#pragma unroll 4
            for (uint32_t c = lane; c < v.cols; c += GROUP) single(c);
        }
        s = group_sum<GROUP>(s, red);
        if (lane == 0 && live) {
            v.sum[r] = s;
            v.negated[r] = -s;
            mean += -s;
        }
    }
    __syncthreads();
    if constexpr (GROUP < 256) {
        if (lane != 0) mean = 0.0F;
        mean = group_sum<256>(mean, red);
    }
    finish_mean(v, mean);
}

__global__ void __launch_bounds__(256) loss_value_tile_kernel(ValueArgs v) {
    pdl_prologue();
    __shared__ float p[kTileRows * (kTileCols + 1)];
    const uint32_t pitch = v.cols | 1u;
    __shared__ float red[32];
    const int64_t r0 = int64_t(blockIdx.x) * kTileRows;
    const int rows = static_cast<int>(min(int64_t(kTileRows), v.rows - r0));
    const uint32_t n = rows * v.cols;
    const int64_t base = r0 * v.cols;
    auto keep = [&](uint32_t i, float t) {
        uint32_t r, c;
        v.by_cols.divmod(i, r, c);
        p[r * pitch + c] = t;
    };
    const uint32_t quads = v.quads != 0 ? n / 4 : 0;
    for (uint32_t u = threadIdx.x; u < quads; u += 256) {
        float x[4], y[4];
        get<4>(v.a + base + 4 * u, x);
        get<4>(v.b + base + 4 * u, y);
#pragma unroll
        for (int w = 0; w < 4; ++w) {
            x[w] = __fmul_rn(x[w], y[w]);
            keep(4 * u + w, x[w]);
        }
        put<4, false>(v.product + base + 4 * u, x);
    }
    for (uint32_t i = 4 * quads + threadIdx.x; i < n; i += 256) {
        const float t = __fmul_rn(v.a[base + i], v.b[base + i]);
        keep(i, t);
        v.product[base + i] = t;
    }
    __syncthreads();
    float s = 0.0F;
    if (threadIdx.x < rows) {
        for (uint32_t c = 0; c < v.cols; ++c) s += p[threadIdx.x * pitch + c];
        v.sum[r0 + threadIdx.x] = s;
        v.negated[r0 + threadIdx.x] = -s;
    }
    finish_mean(v, group_sum<256>(-s, red));
}

// ---- matching ----

bool aligned16(const void* p) { return reinterpret_cast<uintptr_t>(p) % 16 == 0; }

bool dense_f32(const b200_tensor& t, int64_t rows, int64_t cols) {
    return t.dtype == B200_F32 && t.ndim == 2 && t.data != nullptr && t.dims[0] == rows && t.dims[1] == cols &&
           (rows == 1 || t.strides[0] == cols * 4) && (cols == 1 || t.strides[1] == 4);
}

bool dense_vector(const b200_tensor& t, int64_t n, int dtype) {
    return t.dtype == dtype && t.ndim == 1 && t.data != nullptr && t.dims[0] == n &&
           (n == 1 || t.strides[0] == static_cast<int64_t>(dtype_size(dtype)));
}

// `t` is the [rows, cols] broadcast of the vector at `data`: along the rows (axis 0) or the columns (axis 1).
bool spread_of(const b200_tensor& t, const void* data, int axis, int64_t rows, int64_t cols) {
    if (t.dtype != B200_F32 || t.ndim != 2 || t.data != data || t.dims[0] != rows || t.dims[1] != cols) return false;
    const int64_t extent[2] = {rows, cols};
    for (int d = 0; d < 2; ++d) {
        if (extent[d] != 1 && t.strides[d] != (d == axis ? 4 : 0)) return false;
    }
    return true;
}

uint32_t axes_of(const b200_node& n, bool& keepdim) {
    uint32_t mask = 0;
    uint8_t keep = 0;
    std::memcpy(&mask, n.params, 4);
    std::memcpy(&keep, n.params + 4, 1);
    keepdim = keep != 0;
    return mask;
}

// The head from seq[0] on: how many nodes it has (0: none).
size_t match_head(const b200_node* const* seq, size_t avail, LossArgs& a) {
    size_t at = 0, lead = 0;
    if (seq[0]->op == B200_OP_FULL) {
        if (avail < 11 || seq[1]->op != B200_OP_FULL || seq[2]->op != B200_OP_DIV || seq[3]->op != B200_OP_CONTIGUOUS || seq[3]->out.ndim != 1 ||
            seq[2]->n_src != 2 || seq[2]->src[0].data != seq[0]->out.data || seq[2]->src[1].data != seq[1]->out.data ||
            seq[3]->src[0].data != seq[2]->out.data) {
            return 0;
        }
        for (int i = 0; i < 3; ++i) {
            if (seq[i]->out.dtype != B200_F32 || seq[i]->out.ndim != 0 || seq[i]->out.data == nullptr) return 0;
            a.scalars[i] = static_cast<float*>(seq[i]->out.data);
        }
        for (int i = 0; i < 2; ++i) {
            double v;
            std::memcpy(&v, seq[i]->params, sizeof(v));
            a.scalar_values[i] = static_cast<float>(v);
        }
        a.scalar_values[2] = a.scalar_values[0] / a.scalar_values[1];
        lead = 3;
        seq += 3;
        avail -= 3;
    }
    const b200_node& first = *seq[0];
    if (first.op != B200_OP_CONTIGUOUS) return 0;
    const float* row_value = nullptr;
    if (first.out.ndim == 1) {
        if (avail < 8 || seq[1]->op != B200_OP_NEG || seq[2]->op != B200_OP_CONTIGUOUS) return 0;
        const int64_t rows = first.out.dims[0];
        const b200_tensor& s = first.src[0];
        if (!dense_vector(first.out, rows, B200_F32) || s.dtype != B200_F32 || s.ndim != 1 || s.dims[0] != rows || s.strides[0] % 4 != 0 ||
            s.strides[0] < 0 || !dense_vector(seq[1]->src[0], rows, B200_F32) || seq[1]->src[0].data != first.out.data ||
            !dense_vector(seq[1]->out, rows, B200_F32)) {
            return 0;
        }
        a.scale = static_cast<const float*>(s.data);
        a.scale_stride = s.strides[0] / 4;
        a.spread = static_cast<float*>(first.out.data);
        a.negated = static_cast<float*>(seq[1]->out.data);
        row_value = a.negated;
        at = 2;
    }
    if (avail < at + 6) return 0;
    const b200_node& plane = *seq[at];
    const b200_node& wanted = *seq[at + 1];
    const b200_node& index = *seq[at + 2];
    const b200_node& eq = *seq[at + 3];
    const b200_node& hot = *seq[at + 4];
    const b200_node& mul = *seq[at + 5];
    if (wanted.op != B200_OP_CAST || index.op != B200_OP_ARANGE || eq.op != B200_OP_EQUAL || hot.op != B200_OP_CAST ||
        mul.op != B200_OP_MUL || plane.out.ndim != 2) {
        return 0;
    }
    const int64_t rows = plane.out.dims[0], cols = plane.out.dims[1];
    if (cols >= (int64_t(1) << 24) || !dense_f32(plane.out, rows, cols)) return 0;
    const b200_tensor& ps = plane.src[0];
    if (row_value == nullptr) row_value = static_cast<const float*>(ps.data);
    if (!spread_of(ps, row_value, 0, rows, cols)) return 0;
    if (a.negated == nullptr) {
        a.scale = row_value;
        a.scale_stride = 1;
    }
    const b200_tensor& labels = wanted.src[0];
    if (labels.dtype != B200_I64 || labels.ndim != 1 || labels.dims[0] != rows || labels.strides[0] % 8 != 0 || labels.data == nullptr ||
        !dense_vector(wanted.out, rows, B200_F32) || !dense_vector(index.out, cols, B200_F32)) {
        return 0;
    }
    double range[2];
    std::memcpy(range, index.params, sizeof(range));
    if (range[0] != 0.0 || range[1] != 1.0) return 0;
    if (eq.n_src != 2 || !spread_of(eq.src[0], wanted.out.data, 0, rows, cols) || !spread_of(eq.src[1], index.out.data, 1, rows, cols)) return 0;
    auto dense_bool = [&](const b200_tensor& t) {
        return t.dtype == B200_BOOL && t.ndim == 2 && t.dims[0] == rows && t.dims[1] == cols && (rows == 1 || t.strides[0] == cols) &&
               (cols == 1 || t.strides[1] == 1) && t.data == eq.out.data && t.data != nullptr;
    };
    if (!dense_bool(eq.out) || !dense_bool(hot.src[0]) || !dense_f32(hot.out, rows, cols) || !dense_f32(mul.out, rows, cols) || mul.n_src != 2) return 0;
    const bool plain = mul.src[0].data == plane.out.data && mul.src[1].data == hot.out.data;
    const bool turned = mul.src[1].data == plane.out.data && mul.src[0].data == hot.out.data;
    if ((!plain && !turned) || !dense_f32(mul.src[0], rows, cols) || !dense_f32(mul.src[1], rows, cols)) return 0;
    a.rows = rows;
    a.cols = static_cast<uint32_t>(cols);
    a.plane = static_cast<float*>(plane.out.data);
    a.labels = static_cast<const int64_t*>(labels.data);
    a.label_stride = labels.strides[0] / 8;
    a.wanted = static_cast<float*>(wanted.out.data);
    a.index = static_cast<float*>(index.out.data);
    a.equal = static_cast<uint8_t*>(eq.out.data);
    a.onehot = static_cast<float*>(hot.out.data);
    a.picked = static_cast<float*>(mul.out.data);
    return lead + at + 6;
}

size_t match_backward(const b200_node* const* seq, size_t avail, LossArgs& a) {
    if (avail < 5) return 0;
    const b200_node& lsm = *seq[0];
    const b200_node& ex = *seq[1];
    const b200_node& sum = *seq[2];
    const b200_node& mul = *seq[3];
    const b200_node& sub = *seq[4];
    if (lsm.op != B200_OP_LOG_SOFTMAX || ex.op != B200_OP_EXP || sum.op != B200_OP_SUM || mul.op != B200_OP_MUL || sub.op != B200_OP_SUB) return 0;
    if (lsm.out.ndim != 2) return 0;
    const int64_t rows = lsm.out.dims[0], cols = lsm.out.dims[1];
    int32_t axis = 0;
    std::memcpy(&axis, lsm.params, 4);
    bool keepdim = false;
    const uint32_t mask = axes_of(sum, keepdim);
    if (cols >= (int64_t(1) << 24) || (axis != 1 && axis != -1) || mask != 2u || !keepdim) return 0;
    for (const b200_tensor* t : {&lsm.out, &lsm.src[0], &ex.src[0], &ex.out, &sum.src[0], &mul.src[0], &mul.out, &sub.src[0], &sub.src[1], &sub.out}) {
        if (!dense_f32(*t, rows, cols)) return 0;
    }
    if (!dense_f32(sum.out, rows, 1) || ex.src[0].data != lsm.out.data || mul.n_src != 2 || mul.src[0].data != ex.out.data ||
        !spread_of(mul.src[1], sum.out.data, 0, rows, cols) || sub.n_src != 2 || sub.src[0].data != sum.src[0].data ||
        sub.src[1].data != mul.out.data) {
        return 0;
    }
    if (a.picked != nullptr && (a.rows != rows || a.cols != cols)) return 0;
    a.rows = rows;
    a.cols = static_cast<uint32_t>(cols);
    a.x = static_cast<const float*>(lsm.src[0].data);
    a.g = static_cast<const float*>(sum.src[0].data);
    a.logp = static_cast<float*>(lsm.out.data);
    a.prob = static_cast<float*>(ex.out.data);
    a.total = static_cast<float*>(sum.out.data);
    a.share = static_cast<float*>(mul.out.data);
    a.grad = static_cast<float*>(sub.out.data);
    return 5;
}

template <bool HEAD, bool BACK>
void launch_rows(b200_ctx* ctx, LossArgs a) {
    bool quads = true;
    for (const void* p : {static_cast<const void*>(a.plane), static_cast<const void*>(a.onehot), static_cast<const void*>(a.picked),
                          static_cast<const void*>(a.x), static_cast<const void*>(BACK ? a.g : nullptr), static_cast<const void*>(a.logp),
                          static_cast<const void*>(a.prob), static_cast<const void*>(a.share), static_cast<const void*>(a.grad)}) {
        quads = quads && aligned16(p);
    }
    const bool quads_ok = quads && reinterpret_cast<uintptr_t>(a.equal) % 4 == 0;
    a.quads = quads_ok ? 1 : 0;
    if (a.cols <= kTileCols) {
        a.by_cols = FastDiv(a.cols);
        launch_kernel(ctx, loss_tile_kernel<HEAD, BACK>, static_cast<unsigned>(ceil_div(a.rows, kTileRows)), 256, 0, a);
        return;
    }
    const unsigned warps = static_cast<unsigned>(std::min<int64_t>(ceil_div(a.rows, 8), int64_t(sm_count()) * 8));
    const unsigned eights = static_cast<unsigned>(std::min<int64_t>(ceil_div(a.rows, 32), int64_t(sm_count()) * 8));
    const unsigned blocks = static_cast<unsigned>(std::min<int64_t>(a.rows, int64_t(sm_count()) * 8));
    if (!quads_ok || (BACK ? a.cols > kLongMax : a.cols > 4096)) {
        launch_kernel(ctx, loss_any_kernel<HEAD, BACK>, blocks, 256, 0, a);
        return;
    }
#define B200_LOSS(GROUP, ITEMS, GRID) launch_kernel(ctx, loss_rows_kernel<HEAD, BACK, GROUP, ITEMS>, GRID, 256, 0, a)
    if (a.cols <= 128 && a.rows > kManyRows * sm_count()) B200_LOSS(8, 4, eights);
    else if (a.cols <= 256) B200_LOSS(32, 2, warps);
    else if (a.cols <= 1024) B200_LOSS(32, 8, warps);
    else if (a.cols <= 4096) B200_LOSS(256, 4, blocks);
    else if constexpr (BACK) {
        const size_t smem = (a.cols + 3) / 4 * 16;
        auto launch = [&](auto kernel, int threads, int blocks) {
            B200_CUDA_CHECK(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, 4 * kLongMax));
            launch_kernel(ctx, kernel, static_cast<unsigned>(std::min<int64_t>(a.rows, int64_t(sm_count()) * blocks)), threads, smem, a, ctx->d_status);
        };
        if (a.cols <= 8192) launch(loss_long_kernel<HEAD, BACK, 256>, 256, 6);
        else if (a.cols <= 16384) launch(loss_long_kernel<HEAD, BACK, 512>, 512, 3);
        else launch(loss_long_kernel<HEAD, BACK, kLongThreads>, kLongThreads, 1);
    }
#undef B200_LOSS
}

size_t match_value(const b200_node* const* seq, size_t avail, ValueArgs& v) {
    if (avail < 4) return 0;
    const b200_node& mul = *seq[0];
    const b200_node& sum = *seq[1];
    const b200_node& neg = *seq[2];
    const b200_node& mean = *seq[3];
    if (mul.op != B200_OP_MUL || sum.op != B200_OP_SUM || neg.op != B200_OP_NEG || mean.op != B200_OP_MEAN) return 0;
    if (mul.out.ndim != 2 || mul.n_src != 2) return 0;
    const int64_t rows = mul.out.dims[0], cols = mul.out.dims[1];
    bool keep_sum = false, keep_mean = false;
    const uint32_t sum_axes = axes_of(sum, keep_sum), mean_axes = axes_of(mean, keep_mean);
    if (cols >= (int64_t(1) << 24) || sum_axes != 2u || keep_sum || mean_axes != 1u || keep_mean) return 0;
    if (!dense_f32(mul.out, rows, cols) || !dense_f32(mul.src[0], rows, cols) || !dense_f32(mul.src[1], rows, cols) ||
        !dense_f32(sum.src[0], rows, cols) || sum.src[0].data != mul.out.data || !dense_vector(sum.out, rows, B200_F32) ||
        !dense_vector(neg.src[0], rows, B200_F32) || neg.src[0].data != sum.out.data || !dense_vector(neg.out, rows, B200_F32) ||
        !dense_vector(mean.src[0], rows, B200_F32) || mean.src[0].data != neg.out.data || mean.out.dtype != B200_F32 || mean.out.ndim != 0) {
        return 0;
    }
    v.rows = rows;
    v.cols = static_cast<uint32_t>(cols);
    v.a = static_cast<const float*>(mul.src[0].data);
    v.b = static_cast<const float*>(mul.src[1].data);
    v.product = static_cast<float*>(mul.out.data);
    v.sum = static_cast<float*>(sum.out.data);
    v.negated = static_cast<float*>(neg.out.data);
    v.mean = static_cast<float*>(mean.out.data);
    return 4;
}

void launch_value(b200_ctx* ctx, ValueArgs v) {
    const bool quads = aligned16(v.a) && aligned16(v.b) && aligned16(v.product);
    const bool tile = v.cols <= kTileCols, eight = v.cols <= 128 && v.rows > kManyRows * sm_count(), warp = v.cols <= 1024;
    const unsigned grid = tile ? static_cast<unsigned>(ceil_div(v.rows, kTileRows))
                               : static_cast<unsigned>(std::min<int64_t>(eight ? ceil_div(v.rows, 32) : warp ? ceil_div(v.rows, 8) : v.rows, int64_t(sm_count()) * 8));
    v.by_cols = FastDiv(v.cols);
    v.quads = quads ? 1 : 0;
    v.partial = static_cast<float*>(ctx->ensure_workspace(sizeof(float) * grid));
    v.arrived = ctx->d_counters + kLossCounter;
    if (tile) launch_kernel(ctx, loss_value_tile_kernel, grid, 256, 0, v);
    else if (eight && quads) launch_kernel(ctx, loss_value_kernel<8, true>, grid, 256, 0, v);
    else if (eight) launch_kernel(ctx, loss_value_kernel<8, false>, grid, 256, 0, v);
    else if (warp && quads) launch_kernel(ctx, loss_value_kernel<32, true>, grid, 256, 0, v);
    else if (warp) launch_kernel(ctx, loss_value_kernel<32, false>, grid, 256, 0, v);
    else if (quads) launch_kernel(ctx, loss_value_kernel<256, true>, grid, 256, 0, v);
    else launch_kernel(ctx, loss_value_kernel<256, false>, grid, 256, 0, v);
}

}  // namespace

// How many nodes at the head of `seq` one of the loss's runs covers (0: none); `launch` serves them.
size_t loss_group(b200_ctx* ctx, const b200_node* const* seq, size_t avail, bool launch) {
    LossArgs a{};
    ValueArgs v{};
    size_t n = 0;
    const uint32_t op = seq[0]->op;
    if (op == B200_OP_MUL) {
        n = match_value(seq, avail, v);
        if (n == 0 || !launch) return n;
        ProfScope scope(ctx, "fused.loss_value");
        launch_value(ctx, v);
    } else {
        const size_t head = op == B200_OP_LOG_SOFTMAX ? 0 : match_head(seq, avail, a);
        if (op != B200_OP_LOG_SOFTMAX && head == 0) return 0;
        LossArgs both = a;
        size_t back = avail > head ? match_backward(seq + head, avail - head, both) : 0;
        if (head > 0 && back > 0 && both.g != both.picked) back = 0;  // (the sum is not over this head's rows)
        n = head + back;
        if (n == 0 || !launch) return n;
        if (back > 0) a = both;
        ProfScope scope(ctx, back > 0 ? "fused.log_softmax_backward" : "fused.loss_head");
        if (head > 0 && back > 0) launch_rows<true, true>(ctx, a);
        else if (head > 0) launch_rows<true, false>(ctx, a);
        else launch_rows<false, true>(ctx, a);
    }
    ctx->count_launch();
    check_last_launch("fused loss");
    return n;
}

}  // namespace b200
