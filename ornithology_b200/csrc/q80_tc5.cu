// q80_tc5.cu — Q8_0 weights x Q8_K activations on the tcgen05 integer tensor cores, bit for bit the engine's integer path
// (vec_dot_q8_0, reference: src/ornith_qdot.c:144-163, as src/ornith_rforward.c:138-192 drives it).
//
// A Q8_0 block is 32 codes with an f16 scale of its own, and the engine adds scale x (float)(codes . codes) block by block:
// every block is one K = 32 product with an accumulator of its own, read back from tensor memory, converted, scaled and
// added in f32.  That part (about two instructions per row, token and block) is the work; mma.sync adds operand loads and
// the unpacking of weights per 16 x 8 tile to it on the same issue slots, here one thread issues 128 x NS x 32 products and
// the weights are brought into operand form once per 128 rows x NS tokens.
//
// The roles and the walk over the tiles are those of kquant_prefill_tc5.cu.  Per super-block (8 blocks) a worker copies the
// codes of its row group out of the 34-byte blocks into core-matrix order (one plane, two stages: the next super-block is
// unpacked before this one is drained), then drains units of BU blocks, NS tokens wide (BU NS = 256 columns, two slots).
// What bounds it: the drain's issue slots and the latencies between them (a super-block of 128 x 128 takes about 6600 cycles, in
// which a scheduler issues 4700 times; its MMAs take 512 of the tensor pipe).  Measured (us, mma.sync kernel -> this one): 2048 -> 8192, 128
// tokens 24 -> 20, 2048 tokens 319 -> 198; 4096 -> 20608, 777 tokens 625 -> 410, 2048 tokens 1538 -> 951.
#include "kq_tc5.cuh"

namespace {

using namespace kq;
using namespace kq_tc5;

template <int NS> struct Q80Smem {                // byte offsets; every part a multiple of 128
    static constexpr int XB = ORN_Q8K_IMG_LO, XSTAGE = NS / 8 * XB, W = ROWS * Fmt<T_Q80>::BOX;
    static constexpr int O_X = 2 * PLANE, O_W = O_X + 2 * XSTAGE, O_D = O_W + 2 * W;
    static constexpr int BYTES = O_D + 4 * 8 * ROWS * 4 + 128;       // block scales of four super-blocks
    static_assert(XSTAGE % 128 == 0 && W % 128 == 0 && BYTES <= SMEM_LIMIT, "shared memory of one CTA");
};

struct Bars {
    unsigned long long w_full[2], w_free[2], a_full[2], x_full[2], x_free[2], mma_done[2], d_free[2];
};

// 32 codes of each of the 8 blocks of a row: this lane's two words of every block to the k-steps 2 sb and 2 sb + 1
__device__ __forceinline__ void unpack_q80(smem_ptr base, int j, unsigned char *dst) {
    uint32_t w[8][2];
#pragma unroll
    for (int sb = 0; sb < 8; sb++) {
        smem_ptr p = base + 34 * sb + 4 * j;
        if ((sb & 1) == 0) {                                          // 34 sb is a multiple of 4: the codes start mid-word
            w[sb][0] = __byte_perm(lds32(p), lds32(p + 4), 0x5432);
            w[sb][1] = __byte_perm(lds32(p + 16), lds32(p + 20), 0x5432);
        } else {                                                      // 34 sb + 2 is a multiple of 4
            w[sb][0] = lds32(p + 2);
            w[sb][1] = lds32(p + 18);
        }
    }
#pragma unroll
    for (int sb = 0; sb < 8; sb++) {
        *reinterpret_cast<uint32_t *>(dst + (2 * sb) * 128) = w[sb][0];
        *reinterpret_cast<uint32_t *>(dst + (2 * sb + 1) * 128) = w[sb][1];
    }
}

template <int NS>
__global__ void __launch_bounds__(NTHREADS, 1) k_matmul_q80_tc5(KqArgs a, int n_tiles, const __grid_constant__ KqGroup grp) {
    using S = Q80Smem<NS>;
    constexpr int BU = 256 / NS, U = 8 / BU, COLS = NS / 4, BOX = Fmt<T_Q80>::BOX;
    extern __shared__ unsigned char smem_raw[];
    __shared__ __align__(8) Bars bars;
    __shared__ uint32_t tmem_slot;
    unsigned char *smem = smem_raw + ((128 - (tc5::su32(smem_raw) & 127)) & 127);
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, nseg = a.nseg;
    if (tid == 0) {
        for (int i = 0; i < 2; i++) {
            tc5::mbar_init(tc5::su32(&bars.w_full[i]), 1);
            tc5::mbar_init(tc5::su32(&bars.w_free[i]), NWORK);
            tc5::mbar_init(tc5::su32(&bars.a_full[i]), NWORK);
            tc5::mbar_init(tc5::su32(&bars.x_full[i]), 1);
            tc5::mbar_init(tc5::su32(&bars.x_free[i]), NWORK);
            tc5::mbar_init(tc5::su32(&bars.mma_done[i]), MMA_DONE_ARRIVALS);
            tc5::mbar_init(tc5::su32(&bars.d_free[i]), NWORK);
        }
        tc5::mbar_init_fence();
    }
    if (warp == W_MMA) tc5::tmem_alloc(&tmem_slot, 512);
    tc5::fence_before();
    __syncthreads();
    tc5::fence_after();
    const uint32_t tmem = tmem_slot;
    bool ok = true;

    if (warp == W_COPY) {
        // ---- weight bytes, two super-blocks ahead of the workers -------------------------------------------------
        if (tc5::elect_one()) {
            int n = 0;                                                // super-blocks copied
            for (int idx = blockIdx.x; idx < n_tiles && ok; idx += gridDim.x) {
                const Tile t = tile_of<NS, 1>(grp, a.T, idx);
                for (int s = 0; s < nseg; s++, n++) {
                    if (n >= 2) {                                     // the rows that had this stage are unpacked
                        ok = tc5::mbar_wait_parked(tc5::su32(&bars.w_free[n & 1]), (uint32_t)((n - 2) >> 1) & 1u);
                        if (!ok) break;
                        asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory");
                    }
                    const uint32_t bar = tc5::su32(&bars.w_full[n & 1]);          // (rows past n_out are outside the map: zeros)
                    tc5::mbar_expect_tx(bar, (uint32_t)S::W);
                    tensor_copy_rows(tc5::su32(smem + S::O_W + (n & 1) * S::W), &grp.map[t.pj], s * (BOX / 4), t.row0, bar);
                }
            }
            if (!ok) {                                                // leave no copy in flight
                for (int v = n - 1; v >= 0 && v >= n - 2; v--) tc5::mbar_wait(tc5::su32(&bars.w_full[v & 1]), (uint32_t)(v >> 1) & 1u);
                tc5::report_timeout(a.status, ORN_WAIT_DECODE);
            }
        }
    } else if (warp == X_COPY) {
        // ---- activation images ---------------------------------------------------------------------------------------
        if (tc5::elect_one()) {
            asm volatile("griddepcontrol.wait;\n" ::: "memory");     // they come from the kernel in front
            int n = 0;
            for (int idx = blockIdx.x; idx < n_tiles && ok; idx += gridDim.x) {
                const Tile t = tile_of<NS, 1>(grp, a.T, idx);
                const int nt = (t.n_tok + 7) / 8;
                for (int s = 0; s < nseg; s++, n++) {
                    if (n >= 2) {                                     // the super-block that had this stage is drained
                        ok = tc5::mbar_wait_parked(tc5::su32(&bars.x_free[n & 1]), (uint32_t)((n - 2) >> 1) & 1u);
                        if (!ok) break;
                        asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory");
                    }
                    const uint32_t bar = tc5::su32(&bars.x_full[n & 1]), dst = tc5::su32(smem + S::O_X + (n & 1) * S::XSTAGE);
                    tc5::mbar_expect_tx(bar, (uint32_t)(nt * S::XB));
                    for (int i = 0; i < nt; i++)
                        bulk_copy(dst + i * S::XB, a.img + ((size_t)((t.tok0 >> 3) + i) * nseg + s) * ORN_Q8K_IMG_BYTES, S::XB, bar);
                }
            }
            if (!ok) {                                                // leave no copy in flight
                for (int v = n - 1; v >= 0 && v >= n - 2; v--) tc5::mbar_wait(tc5::su32(&bars.x_full[v & 1]), (uint32_t)(v >> 1) & 1u);
                tc5::report_timeout(a.status, ORN_WAIT_DECODE);
            }
        }
    } else if (warp == W_MMA) {
        // ---- MMA issue -----------------------------------------------------------------------------------------------
        if (tc5::elect_one()) {
            int u = 0, n = 0;
            for (int idx = blockIdx.x; idx < n_tiles && ok; idx += gridDim.x) {
                const Tile t = tile_of<NS, 1>(grp, a.T, idx);
                const uint32_t id = idesc_i8(true, (t.n_tok + 15) & ~15);
                for (int s = 0; s < nseg && ok; s++, n++) {
                    ok = tc5::mbar_wait_parked(tc5::su32(&bars.a_full[n & 1]), (uint32_t)(n >> 1) & 1u) &&
                         tc5::mbar_wait(tc5::su32(&bars.x_full[n & 1]), (uint32_t)(n >> 1) & 1u);
                    const uint64_t A = desc_plain(tc5::su32(smem + (n & 1) * PLANE), 128, QK * 8);
                    const uint64_t B = desc_plain(tc5::su32(smem + S::O_X + (n & 1) * S::XSTAGE), 128, S::XB);
                    for (int v = 0; v < U && ok; v++, u++) {
                        const int slot = u & 1;
                        if (u >= 2) ok = tc5::mbar_wait_parked(tc5::su32(&bars.d_free[slot]), (uint32_t)((u >> 1) - 1) & 1u);
                        if (!ok) break;
                        tc5::fence_after();
#pragma unroll
                        for (int i = 0; i < BU; i++)                  // a block is two core matrices along K: 256 bytes
                            mma_i8_ss(tmem + slot * 256 + i * NS, A + 16 * (v * BU + i), B + 16 * (v * BU + i), id, 0);
                        mma_issued(tc5::su32(&bars.mma_done[slot]));
                    }
                }
            }
            if (!ok) {                                                // leave no product in flight
                for (int v = u - 1; v >= 0 && v >= u - 2; v--) tc5::mbar_wait(tc5::su32(&bars.mma_done[v & 1]), (uint32_t)(v >> 1) & 1u);
                tc5::report_timeout(a.status, ORN_WAIT_DECODE);
            }
        }
    } else if (warp < NWORK) {
        // ---- unpack and drain ----------------------------------------------------------------------------------------
        float *scales = reinterpret_cast<float *>(smem + S::O_D);    // [4 super-blocks][8 blocks][128 rows]
        const int q = warp & 3, cg = warp >> 2;                      // tensor-memory lanes 32 q .., columns COLS cg ..
        const uint32_t tq = tmem + ((uint32_t)(q * 32) << 16) + cg * COLS;
        const f32x2 mz = pack2(a.minus_zero, a.minus_zero);
        const int g = lane >> 2, j = lane & 3;
        auto wait_all = [&](unsigned long long *bar, uint32_t parity) {
            if (ok) ok = __all_sync(0xffffffffu, tc5::mbar_wait(tc5::su32(bar), parity));
        };
        // super-block n (counted over all tiles): its plane was that of n - 2, which this warp has drained, so its products
        // are complete.  Its scales were those of n - 4: the products of n - 2 needed their slots back from every warp, so
        // every warp has drained n - 3 and the ones before
        auto unpack = [&](int n) {
            wait_all(&bars.w_full[n & 1], (uint32_t)(n >> 1) & 1u);
            if (!ok) return;
            smem_ptr base = smem + S::O_W + (n & 1) * S::W + (warp * 8 + g) * BOX;
            unpack_q80(base, j, smem + (n & 1) * PLANE + warp * (8 * QK) + lane * 4);
            float *sc = scales + (n & 3) * (8 * ROWS) + warp * 8 + g;
            sc[(2 * j) * ROWS] = f16_bits_to_f32(lds32(base + 68 * j) & 0xFFFFu);             // block 2 j at 68 j, block 2 j + 1 at 68 j + 34
            sc[(2 * j + 1) * ROWS] = f16_bits_to_f32(lds32(base + 68 * j + 32) >> 16);
            asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory");
            __syncwarp();
            if (lane == 0) { tc5::mbar_arrive(tc5::su32(&bars.a_full[n & 1])); tc5::mbar_arrive(tc5::su32(&bars.w_free[n & 1])); }
        };
        int n = 0, du = 0;                                            // super-blocks, units drained
        for (int idx = blockIdx.x; idx < n_tiles; idx += gridDim.x) {
            const int n_tok = tile_of<NS, 1>(grp, a.T, idx).n_tok;
            const bool mine = cg * COLS < n_tok;                      // this warp's columns hold tokens
            f32x2 tot[COLS / 2];
#pragma unroll
            for (int i = 0; i < COLS / 2; i++) tot[i] = 0;
            if (ok) unpack(n);
            for (int s = 0; s < nseg && ok; s++, n++) {
                if (s + 1 < nseg) unpack(n + 1);
                wait_all(&bars.a_full[n & 1], (uint32_t)(n >> 1) & 1u);          // every warp's block scales are in place
                f32x2 blk[COLS / 2];
#pragma unroll
                for (int i = 0; i < COLS / 2; i++) blk[i] = 0;
                for (int v = 0; v < U; v++, du++) {
                    const int slot = du & 1;
                    wait_all(&bars.mma_done[slot], (uint32_t)(du >> 1) & 1u);
                    if (!ok) break;
                    tc5::fence_after();
                    if (mine) {
#pragma unroll
                        for (int i = 0; i < BU; i++) {
                            const float wd1 = scales[(n & 3) * (8 * ROWS) + (v * BU + i) * ROWS + q * 32 + lane];
                            const f32x2 wd = pack2(wd1, wd1);
#pragma unroll
                            for (int c = 0; c < COLS; c += 16) {
                                float d[16];
                                tc5::tmem_ld16_wait(tq + slot * 256 + i * NS + c, d);
#pragma unroll
                                for (int e = 0; e < 8; e++) {
                                    const f32x2 f = pack2((float)__float_as_int(d[2 * e]), (float)__float_as_int(d[2 * e + 1]));
                                    blk[c / 2 + e] = add2(blk[c / 2 + e], mul2_apart(wd, f, mz));
                                }
                            }
                        }
                    }
                    tc5::fence_before();
                    __syncwarp();
                    if (lane == 0) tc5::mbar_arrive(tc5::su32(&bars.d_free[slot]));
                }
                if (!ok) break;
                if (mine) {
                    const unsigned char *xs = smem + S::O_X + (n & 1) * S::XSTAGE + cg * (COLS / 8) * S::XB + ORN_Q8K_IMG_D;
#pragma unroll
                    for (int i = 0; i < COLS / 2; i++) {
                        const float2 y = *reinterpret_cast<const float2 *>(xs + i / 4 * S::XB + (i & 3) * 8);
                        tot[i] = add2(tot[i], mul2_apart(pack2(y.x, y.y), blk[i], mz));
                    }
                }
                __syncwarp();
                if (lane == 0) tc5::mbar_arrive(tc5::su32(&bars.x_free[n & 1]));
            }
            const Tile t = tile_of<NS, 1>(grp, a.T, idx);
            const int row = t.row0 + q * 32 + lane;
            if (row < t.n_out) {
#pragma unroll
                for (int i = 0; i < COLS; i++) {
                    const int c = cg * COLS + i;
                    if (c >= t.n_tok) continue;
                    float v0, v1;
                    unpack2(tot[i / 2], &v0, &v1);
                    const float val = !ok ? NAN : (i & 1) ? v1 : v0;  // NaN once a wait has given up: this tile and the rest of the CTA's
                    if (a.out_dtype == ORNITH_ACT_BF16) act_st((__nv_bfloat16 *)grp.y[t.pj], (size_t)(t.tok0 + c) * t.n_out + row, val);
                    else act_st((float *)grp.y[t.pj], (size_t)(t.tok0 + c) * t.n_out + row, val);
                }
            }
        }
        if (!ok && lane == 0) tc5::report_timeout(a.status, ORN_WAIT_DECODE);
    }
    tc5::fence_before();
    __syncthreads();
    tc5::fence_after();
    if (warp == W_MMA) tc5::tmem_dealloc(tmem, 512);
}

template <int NS>
ornith_status launch_ns(const HostGroup &h, int n_in, int T, const KqArgs &a, cudaStream_t stream) {
    KqGroup g;
    if (!fill_group<T_Q80>(&g, h, n_in, ROWS)) return (ornith_status)ORNITH_ERR_BACKEND;
    static bool opted[ORN_MAX_DEVICES] = {};
    bool &have = opted[orn_device_index()];
    if (!have) {
        ORN_TRY(orn_check(cudaFuncSetAttribute(k_matmul_q80_tc5<NS>, cudaFuncAttributeMaxDynamicSharedMemorySize, Q80Smem<NS>::BYTES), "projection smem opt-in"));
        have = true;
    }
    const int n_tiles = g.cta0[h.n] * ((T + NS - 1) / NS);
    return orn_check(orn_launch_dependent(k_matmul_q80_tc5<NS>, dim3((unsigned)(n_tiles < SMS ? n_tiles : SMS)), dim3(NTHREADS), Q80Smem<NS>::BYTES, stream,
                                          a, n_tiles, g), "k_matmul_q80_tc5");
}

}  // namespace

namespace kq {

// units: tokens of a tile / TC5_UNIT.  Microseconds per super-block and wave, from 8192 -> 4096: 1.9 for 64 tokens, 3.2 for 128.
template <>
float kq_tc5_cost<T_Q80>(const HostGroup &h, int T, int *units) {
    long long row_tiles = 0;
    for (int i = 0; i < h.n; i++) row_tiles += (h.n_out[i] + ROWS - 1) / ROWS;
    *units = 0;
    if (row_tiles * ((T + 63) / 64) > (1 << 30)) return 0.0f;
    const float c64 = 1.9f * (float)((row_tiles * ((T + 63) / 64) + SMS - 1) / SMS);
    const float c128 = 3.2f * (float)((row_tiles * ((T + 127) / 128) + SMS - 1) / SMS);
    *units = c64 <= c128 ? 1 : 2;
    return c64 <= c128 ? c64 : c128;
}
template <>
ornith_status launch_kq_tc5<T_Q80>(const HostGroup &h, int n_in, int T, const KqArgs &a, int units, cudaStream_t stream) {
    return units == 1 ? launch_ns<TC5_UNIT[T_Q80]>(h, n_in, T, a, stream) : launch_ns<2 * TC5_UNIT[T_Q80]>(h, n_in, T, a, stream);
}

}  // namespace kq
