// Batched GEMM problem as vkML's matmul node presents it
// (src/backend/cpu/kernels_matmul.cpp:35-87): rank-4 operands
// a[B0,B1,M,K], b[B0,B1,K,N] with arbitrary element strides (stride 0 on a batch
// axis = broadcast, transposed views = swapped inner strides), dense output
// out[B0,B1,M,N].
#pragma once

#include "context.h"

namespace b200 {

struct GemmProblem {
    const float* a;
    const float* b;
    float* out;
    int64_t b0, b1, m, n, k;
    int64_t a_s[4];  // element strides of a over (b0, b1, m, k)
    int64_t b_s[4];  // element strides of b over (b0, b1, k, n)
};

// Whether the product's result lies over memory that an operand is read from (`width`: bytes of an element).
inline bool result_over_operand(const GemmProblem& p, size_t width) {
    const int64_t outer = p.b0 * p.b1 * p.m * p.n;
    auto over = [&](const float* at, const int64_t (&s)[4], int64_t rows, int64_t cols) {
        const int64_t extent[4] = {p.b0, p.b1, rows, cols};
        int64_t lo = 0, hi = 1;
        for (int i = 0; i < 4; ++i) {
            if (extent[i] == 0) return false;
            const int64_t reach = (extent[i] - 1) * s[i];
            (reach < 0 ? lo : hi) += reach;
        }
        const char *base = reinterpret_cast<const char*>(at), *out = reinterpret_cast<const char*>(p.out);
        const int64_t w = static_cast<int64_t>(width);
        return out < base + hi * w && base + lo * w < out + outer * w;
    };
    return over(p.a, p.a_s, p.m, p.k) || over(p.b, p.b_s, p.k, p.n);
}

// The range of one operand matrix, found on the device (gemm_h16.cu): the bits of the largest magnitude in
// a sample of it, how many nonzero elements are too small beside that for the half split, whether one is too large, how many
// of the sample's own elements are too small, and whether the TF32 planes that stand by for it have been written.
struct __align__(16) RangeSlot {
    uint32_t max_bits;
    uint32_t strays;
    uint32_t spoiled;
    uint32_t early;
    uint32_t tf32;
    uint32_t pad[3];
};

// Launches carrying a guard run only if one of the two matrices is wide (see gemm_h16.cu); a == null: always.
struct RangeGuard {
    const RangeSlot* a;
    const RangeSlot* b;
    uint32_t limit_a, limit_b;
};

// What stands by for one operand of a half-term product.  `planes`: its TF32 planes (hi, then lo); `done`: where it is noted that they have
// been written, for an operand that several products of the span share (null: this product alone uses them).  `strays`: the
// positions, in the order of the matrix in memory, of the elements that its half planes leave out.
struct Standby {
    float* planes;
    uint32_t* done;
    const int64_t* strays;
};
constexpr uint32_t kMaxStrays = 512;  // of one matrix; with more it is wide

// What the nodes behind a product make of it, element by element, where the kernel that writes the product can write that too: a bias along the
// columns with ReLU's mask and a ReLU, or where(cond, other, product).  The values are those of the nodes' own kernels.
struct ProductEpilogue {
    const float* bias;  // null: the other form
    float* add;
    float* full_a;      // null: no mask
    uint8_t* mask;
    float* full_b;
    float value_a, value_b;
    float* relu;        // null: none
    const uint8_t* cond;
    const float* other;
    int other_step;     // 0: a buffer that is known to hold one value throughout
    float* chosen;
};
#ifdef __CUDACC__
__device__ __forceinline__ void write_epilogue(const ProductEpilogue& e, int64_t i, int64_t col, float v) {
    if (e.bias == nullptr) {
        e.chosen[i] = e.cond[i] != 0 ? e.other[i * e.other_step] : v;
        return;
    }
    const float y = __fadd_rn(v, e.bias[col]);
    e.add[i] = y;
    if (e.full_a != nullptr) {
        e.full_a[i] = e.value_a;
        e.full_b[i] = e.value_b;
        e.mask[i] = y <= e.value_a ? 1 : 0;  // false for NaN, as the CPU's comparison
    }
    if (e.relu != nullptr) e.relu[i] = y <= 0.0F ? 0.0F : y;
}
#endif

// fp32 FMA on the CUDA cores; any strides, any size. gemm_simt.cu
void gemm_simt(b200_ctx* ctx, const GemmProblem& p, const ProductEpilogue* epilogue = nullptr);
// fuse.cu: how many of the nodes `seq` behind `product` one epilogue serves, and which (`early`: a relu further on, as in launch_fused)
size_t match_product_epilogue(const b200_node& product, const b200_node* const* seq, size_t avail, size_t later, size_t* early, ProductEpilogue& e);
bool gemm_small_serves(const GemmProblem& p);  // its single-launch kernel, which can write an epilogue
// Whether its single-launch kernel beats the tensor cores, which could serve `p` too (`streams`: from a streamed operand).
bool gemm_small_pays(const GemmProblem& p, bool streams);

// tcgen05 tensor-core path (3xTF32 or single-pass TF32). gemm_tc.cu
bool gemm_tc_eligible(const b200_ctx* ctx, const GemmProblem& p);
void gemm_tc(b200_ctx* ctx, const GemmProblem& p, bool three_pass, const ProductEpilogue* epilogue = nullptr);
bool gemm_tc_folds(const b200_ctx* ctx, const GemmProblem& p);  // in K-slices, whose fold can write an epilogue
// What is queued behind gemm_h16's kernel.  Its strays' share of the product is added to `target`, the result or its first partial plane;
// and for the case that an operand turns out wide on the device, the product from TF32 planes: the tiles
// and K-slices that gemm_tc gives the product, so that its results are gemm_tc's bit for bit.  With slices the partial
// planes are left at `partial` for the caller's fold.
void gemm_tc_stand_by(b200_ctx* ctx, const GemmProblem& p, const RangeGuard& guard, const Standby& a, const Standby& b, float* target,
                      float* partial);
int gemm_tc_slices(const b200_ctx* ctx, const GemmProblem& p);
size_t gemm_tc_plane_limit(const b200_ctx* ctx);  // bytes of planes that are held beside the operands without need
size_t gemm_tc_plane_bytes(const GemmProblem& p, bool left);  // of one operand's two planes

// tcgen05 kind::f16: F32 products from two half terms per operand, F16 products directly. gemm_h16.cu
bool gemm_h16_serves(const b200_ctx* ctx, const GemmProblem& p);
void gemm_h16(b200_ctx* ctx, const GemmProblem& p);
void gemm_h16_note_uses(b200_ctx* ctx, const GemmProblem& p);
std::string gemm_h16_tile(const b200_ctx* ctx, const GemmProblem& p);  // "rows x columns" of the tile it gets
// Ranges of `n` matrices, cleared at a span's first use (null: the span has used them up); and the sum of the K-slices' partial planes.
RangeSlot* gemm_h16_slots(b200_ctx* ctx, int n);
void gemm_h16_fold(b200_ctx* ctx, const GemmProblem& p, const float* partial, int splits, const RangeGuard& guard, int wide_splits);
// The same terms, split inside the product's kernel. gemm_inline.cu
bool gemm_inline_serves(const b200_ctx* ctx, const GemmProblem& p);
void gemm_inline_tf32(b200_ctx* ctx, const GemmProblem& p, float* partial, int64_t splits, int64_t kb_per_split, const char* label);
double gemm_inline_tf32_block(const GemmProblem& p);
bool gemm_inline_fits(const GemmProblem& p, bool tf32);  // its index arithmetic, with half or with TF32 terms
std::string gemm_inline_tile(const b200_ctx* ctx, const GemmProblem& p);
bool gemm_h16_would_serve(const b200_ctx* ctx, const GemmProblem& p);  // (whatever else reads the operands without planes)
bool gemm_h16_shares(const b200_ctx* ctx, const GemmProblem& p);       // another product of the span reads the planes of an operand
double gemm_h16_time(const b200_ctx* ctx, const GemmProblem& p);       // estimate in us, its planes included
void gemm_inline(b200_ctx* ctx, const GemmProblem& p);
// Half storage: `p`'s pointers are to halves.  False: not a case for this kernel.  With an epilogue the nodes behind the
// product -- add(y, bias along the rows) and perhaps relu -- are served as well.
struct HalfEpilogue {
    const void* bias;
    void* biased;
    void* rectified;  // may be null
};
bool gemm_f16_storage(b200_ctx* ctx, const GemmProblem& p, const HalfEpilogue* epilogue = nullptr);
bool gemm_f16_any(b200_ctx* ctx, const GemmProblem& p, const HalfEpilogue* epilogue);  // (operands that TMA cannot read, gemm_f16_any.cu)
// True when gemm_tc would serve `p` with the streamed-operand kernel (a small left operand, the
// right operand read once from HBM) rather than from operand planes.
bool gemm_tc_streams(const b200_ctx* ctx, const GemmProblem& p);
int64_t gemm_tc_chain(const b200_ctx* ctx, const GemmProblem& p);  // products that one accumulator of the plane kernel adds up
bool gemm_tc_reads_directly(const b200_ctx* ctx, const GemmProblem& p);  // (taken by itself: no shared planes)
bool gemm_tc_splits_inside(const b200_ctx* ctx, const GemmProblem& p);   // ... or split them into TF32 terms in its converters' registers
// Diagnostic: one block waits `limit_ns` on a barrier nobody arrives on and gives up (gemm_tc.cu).
void gemm_tc_wait_probe(b200_ctx* ctx, uint64_t limit_ns);

// Reuse of split operand planes inside one compute span: count the operands of every
// tensor-core matmul before the span runs, drop planes whose source a node overwrites, and
// release what is left when the span ends.
void gemm_tc_note_uses(b200_ctx* ctx, const GemmProblem& p);
void gemm_tc_invalidate(b200_ctx* ctx, const void* begin, const void* end);
void gemm_tc_end_span(b200_ctx* ctx);

}  // namespace b200
