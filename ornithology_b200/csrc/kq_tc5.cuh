// kq_tc5.cuh — what the two tcgen05 integer projection kernels share (kquant_prefill_tc5.cu: Q4_K, Q6_K; q80_tc5.cu: Q8_0):
// the roles of a CTA, kind::i8 products over operands in core-matrix order, pairs of f32, the walk over the tiles.
#pragma once
#include "kquant.cuh"

namespace kq_tc5 {

using kq::KqGroup;
using kq::QK;

constexpr int NWORK = 16, W_COPY = NWORK, W_MMA = NWORK + 1, X_COPY = NWORK + 2, NTHREADS = (NWORK + 3) * 32, ROWS = 128;
constexpr int PLANE = ROWS * QK;                  // bytes of one int8 plane of a super-block
constexpr int SMS = 148;
constexpr int SMEM_LIMIT = 232448 - 512;          // what a CTA may have, less this kernel's static part

// K-major operand without swizzle: lbo / sbo = bytes between core matrices (8 rows x 16 bytes) along K / along the rows
__device__ __forceinline__ uint64_t desc_plain(uint32_t saddr, uint32_t lbo, uint32_t sbo) {
    return (uint64_t)((saddr >> 4) & 0x3FFF) | ((uint64_t)((lbo >> 4) & 0x3FFF) << 16) | ((uint64_t)((sbo >> 4) & 0x3FFF) << 32) |
           ((uint64_t)1 << 46);
}
// int32 sums, M = 128, both operands signed (or both unsigned) bytes
__device__ __forceinline__ uint32_t idesc_i8(bool is_signed, int n) {
    return (2u << 4) | (is_signed ? (1u << 7) | (1u << 10) : 0u) | ((uint32_t)(n >> 3) << 17) | (8u << 24);
}
__device__ __forceinline__ void mma_i8_ss(uint32_t d_tmem, uint64_t a_desc, uint64_t b_desc, uint32_t id, uint32_t acc) {
    asm volatile("{\n .reg .pred p;\n setp.ne.b32 p, %4, 0;\n tcgen05.mma.cta_group::1.kind::i8 [%0], %1, %2, %3, p;\n}\n"
                 ::"r"(d_tmem), "l"(a_desc), "l"(b_desc), "r"(id), "r"(acc) : "memory");
}

// A product that is then added must be rounded by itself, as the engine rounds it.  A packed multiply and add are contracted
// into one fused operation whatever their rounding is said to be (seen as last-bit differences), so the product is a fused
// multiply-add onto -0, which the compiler does not know to be -0.
__device__ __forceinline__ f32x2 mul2_apart(f32x2 a, f32x2 b, f32x2 minus_zero) { return fma2(a, b, minus_zero); }
// The products of a unit are issued: one arrival when they are complete, and one of the issuing lane itself.  The lane has seen
// the unit's image arrive (the completion of a bulk copy makes it visible to whoever observes it), so its own arrival, a release,
// passes the image on to the workers, which acquire this barrier before they read the activation scales by plain loads.
constexpr int MMA_DONE_ARRIVALS = 2;
__device__ __forceinline__ void mma_issued(uint32_t mma_done) {
    tc5::mbar_arrive(mma_done);
    tc5::mma_commit(mma_done);
}

// A tile is 128 rows of one matrix x H NS tokens; persistent CTAs walk tiles blockIdx.x, + gridDim.x, .. with the token tiles of
// the same rows next to one another (they share the weight bytes in L2).  Every role walks the same tiles with its counters
// running on, so the copies and products of a tile start while the one before it is drained and stored.
struct Tile {
    int pj, n_out, row0, tok0, n_tok, nh;                            // matrix, its rows; first row, first token, tokens, units per super-block
};
template <int NS, int H>
__device__ __forceinline__ Tile tile_of(const KqGroup &grp, int T, int idx) {
    const int ntt = (T + H * NS - 1) / (H * NS), rt = idx / ntt;
    Tile t;
    t.pj = 0;
    while (t.pj + 1 < grp.n && rt >= grp.cta0[t.pj + 1]) t.pj++;
    t.n_out = grp.n_out[t.pj];
    t.row0 = (rt - grp.cta0[t.pj]) * ROWS;
    t.tok0 = (idx - rt * ntt) * (H * NS);
    t.n_tok = min(H * NS, T - t.tok0);
    t.nh = (t.n_tok + NS - 1) / NS;
    return t;
}

}  // namespace kq_tc5
