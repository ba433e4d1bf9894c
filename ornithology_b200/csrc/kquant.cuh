// kquant.cuh — what the integer-projection kernels share (kquant_matmul.cu: mma.sync; kquant_prefill_tc5.cu, q80_tc5.cu: tcgen05):
// the weight formats, the matrices of one launch, the tensor map of a weight matrix.
#pragma once
#include <cuda.h>
#include <cuda_fp16.h>

#include "qproj.cuh"
#include "tcgen05.cuh"          // the tensor-map encoder entry point, bounded mbarrier waits

namespace kq {

constexpr int QK = 256;

enum { T_Q4K = 0, T_Q6K = 1, T_Q80 = 2 };
template <int TYPE> struct Fmt;
template <> struct Fmt<T_Q4K> { static constexpr int BLOCK = 144, BOX = 144; };
template <> struct Fmt<T_Q6K> { static constexpr int BLOCK = 210, BOX = 240; };   // 240: rows 60 words apart, no bank conflicts
template <> struct Fmt<T_Q80> { static constexpr int BLOCK = 272, BOX = 272; };

__device__ __forceinline__ void bulk_copy(uint32_t dst, const void *src, uint32_t bytes, uint32_t bar) {
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];\n"
                 ::"r"(dst), "l"(src), "r"(bytes), "r"(bar) : "memory");
}
__device__ __forceinline__ void tensor_copy_rows(uint32_t dst, const CUtensorMap *map, int word0, int row0, uint32_t bar) {
    asm volatile("cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];\n"
                 ::"r"(dst), "l"(map), "r"(bar), "r"(word0), "r"(row0) : "memory");
}

typedef const unsigned char *smem_ptr;
__device__ __forceinline__ uint32_t lds32(smem_ptr p) { return *reinterpret_cast<const uint32_t *>(p); }
__device__ __forceinline__ float f16_bits_to_f32(uint32_t h) { return __half2float(__ushort_as_half((unsigned short)h)); }

// The weight matrices of one launch: projections that read the same activations (attn_qkv, attn_gate, ssm_alpha and
// ssm_beta of a delta-net layer; attn_q / k / v of a full-attention layer) go as one grid, CTAs cta0[p] .. cta0[p+1]-1
// belonging to matrix p.
constexpr int MAX_GROUP = 8;
struct KqGroup {
    CUtensorMap map[MAX_GROUP];                   // [n_out rows][row bytes / 4 words] of each matrix
    void *y[MAX_GROUP];                           // [T][n_out]
    int n_out[MAX_GROUP];
    int cta0[MAX_GROUP + 1];
    int n;
};

struct KqArgs {
    const unsigned char *img;                     // [token tiles][nseg] Q8_K images
    void *y;                                      // [T][n_out]
    int T, n_out, nseg, out_dtype;
    int nstage, stage_bytes;                      // shared-memory stages of the mma.sync kernel
    unsigned int *status;
    float minus_zero;                             // -0, as a value the compiler cannot see (kquant_prefill_tc5.cu)
};

// what the host knows of a group: the matrices (all of one weight type, one n_in), their outputs
struct HostGroup {
    const void *W[MAX_GROUP];
    void *y[MAX_GROUP];
    int n_out[MAX_GROUP];
    int n;
    int rows_total() const { int r = 0; for (int i = 0; i < n; i++) r += n_out[i]; return r; }
};

// the weight matrix as [n_out rows][row_bytes / 4 words]; one box = box_rows rows x BOX bytes
template <int TYPE>
bool weight_map(CUtensorMap *m, const void *W, int n_in, int n_out, int box_rows) {
    OrnTensorMapEncodeFn enc = orn_tensor_map_encoder();
    const cuuint64_t row_bytes = (cuuint64_t)n_in / QK * Fmt<TYPE>::BLOCK;
    if (!enc || ((uintptr_t)W & 15) != 0 || (row_bytes & 15) != 0) return false;
    cuuint64_t dims[2] = {row_bytes / 4, (cuuint64_t)n_out};
    cuuint64_t strides[1] = {row_bytes};
    cuuint32_t box[2] = {Fmt<TYPE>::BOX / 4, (cuuint32_t)box_rows};
    cuuint32_t es[2] = {1, 1};
    return enc(m, CU_TENSOR_MAP_DATA_TYPE_UINT32, 2, const_cast<void *>(W), dims, strides, box, es, CU_TENSOR_MAP_INTERLEAVE_NONE,
               CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

// the matrices of a launch with cta_rows rows per CTA; false when a map cannot be made
template <int TYPE>
bool fill_group(KqGroup *g, const HostGroup &h, int n_in, int cta_rows) {
    g->n = h.n;
    g->cta0[0] = 0;
    for (int i = 0; i < h.n; i++) {
        if (!weight_map<TYPE>(&g->map[i], h.W[i], n_in, h.n_out[i], cta_rows)) {
            orn_record_error("matmul_q: the weight tensor map could not be made");
            return false;
        }
        g->y[i] = h.y[i]; g->n_out[i] = h.n_out[i];
        g->cta0[i + 1] = g->cta0[i] + (h.n_out[i] + cta_rows - 1) / cta_rows;
    }
    return true;
}

constexpr int TC5_UNIT[3] = {64, 128, 64};        // tokens of a unit of the tcgen05 kernels, by weight type
constexpr float TC5_START[3] = {2.4f, 3.5f, 2.6f};   // microseconds that a launch of them takes beside its super-blocks

// Prompts on the tcgen05 tensor cores (kquant_prefill_tc5.cu, q80_tc5.cu): what the product would take there, in
// microseconds per super-block, and how many units of tokens a CTA should own (0: too large for that kernel); and the launch
template <int TYPE> float kq_tc5_cost(const HostGroup &h, int T, int *units);
template <int TYPE> ornith_status launch_kq_tc5(const HostGroup &h, int n_in, int T, const KqArgs &a, int units, cudaStream_t stream);
template <> float kq_tc5_cost<T_Q80>(const HostGroup &h, int T, int *units);
template <> ornith_status launch_kq_tc5<T_Q80>(const HostGroup &h, int n_in, int T, const KqArgs &a, int units, cudaStream_t stream);

}  // namespace kq
