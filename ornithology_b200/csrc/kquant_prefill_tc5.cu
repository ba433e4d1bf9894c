// kquant_prefill_tc5.cu — k-quant weights x Q8_K activations for prompts, on the tcgen05 integer tensor cores, bit for bit
// the engine's integer path (reference: src/ornith_qdot.c:75-141 as src/ornith_rforward.c:138-192 drives it).
//
// Inside a super-block of 256 inputs the engine's dot is whole numbers: code x sub-block scale x activation code.
// The product code x scale of a weight is itself a small integer (Q6_K: -4064 .. 4096, Q4_K: 0 .. 945), so a
// super-block is one dense integer product once that number is split into two int8 planes, w = 128 hi + lo with
// lo = 0 .. 127:  isum = 128 (hi . x) + (lo . x), both with int32 sums in tensor memory (tcgen05.mma kind::i8).
// The sub-block scales, which the mma.sync kernel applies to every int32 tile (4 integer multiply-adds per MMA, its
// bound), cost nothing per token here.  What is left per (row, token, super-block) is the engine's f32 part: one
// conversion, (activation scale x weight scale) x isum, added to the running total, super-blocks in order.  Q4_K's
// minimums x sums of codes are two more MMAs per super-block (low and high bytes of the sums).
//
// A tile is 128 weight rows (the 128 lanes of tensor memory) x H units of NS tokens, one persistent CTA of 19 warps per SM:
//   16 workers    unpack the super-block's rows from the packed bytes into the two planes (one row group of 8 per
//                 warp), then drain finished units: tcgen05.ld, the f32 part, totals in registers (H NS / 4 each);
//   2 copy lanes  weight bytes by tensor copy (two stages), activation images by bulk copy (H + 1 units);
//   1 MMA lane    per unit 8 k-steps x 2 planes.  Two accumulator slots: a unit is multiplied while the one before
//                 it is drained; the unit left over from a super-block is drained after the next one is unpacked.
// What bounds it: the issue slots of the workers.  A super-block of 128 rows x 256 tokens (Q6_K, H = 2) takes about 6100
// cycles, 7800 with its share of a CTA's start and stores in a launch of 16: 2000 to unpack, 2000 for each of two drains; its
// MMAs take 2048 of the tensor pipe.  More tokens per CTA would
// share the unpacking further, but the totals already take half of the register file.
// Measured (us, mma.sync kernel -> this one): Q6_K 4096 tokens 2048 -> 8192 821 -> 224, 777 tokens 4096 -> 20608 806 -> 283 and
// 8192 -> 4096 339 -> 111; Q4_K 602 -> 326, 594 -> 360, 247 -> 167.
// Tried: one weight stage (the copy's latency showed: 262 instead of 224 us); one tile per CTA instead of persistent CTAs (239);
// 16 columns per tensor-memory load (spills); int32 -> float by exponent bias instead of the conversion (no faster).
// The image of 8 tokens x 256 codes holds 8 x 16-byte core matrices in order, so it is a B operand as it lies (K-major,
// no swizzle); the planes are written in the same form (conflict-free 128-byte rows).
#include <type_traits>

#include "kq_tc5.cuh"

namespace {

using namespace kq;
using namespace kq_tc5;

template <int TYPE> struct Tc5Fmt;
// NS tokens per unit; two slots of NACC accumulators of NS columns fill the 512 columns
template <> struct Tc5Fmt<T_Q6K> { static constexpr int NACC = 2, NS = TC5_UNIT[T_Q6K], XB = ORN_Q8K_IMG_LO, AMIN = 0; };
template <> struct Tc5Fmt<T_Q4K> { static constexpr int NACC = 4, NS = TC5_UNIT[T_Q4K], XB = ORN_Q8K_IMG_BYTES, AMIN = ROWS * 32; };

template <int TYPE, int H> struct Tc5Smem {       // byte offsets; every part a multiple of 128
    using F = Tc5Fmt<TYPE>;
    static constexpr int NX = H + 1;                            // units of activation images: the one to come is in flight
    static constexpr int XUNIT = F::NS / 8 * F::XB, W = ROWS * Fmt<TYPE>::BOX;
    static constexpr int O_AMIN = 2 * PLANE, O_X = O_AMIN + F::AMIN, O_W = O_X + NX * XUNIT, O_D = O_W + 2 * W;
    static constexpr int NSCALE = F::AMIN ? 2 : 1;              // weight scales (and minimum scales) of 4 super-blocks
    static constexpr int BYTES = O_D + 4 * NSCALE * ROWS * 4 + 128;
    static_assert(XUNIT % 128 == 0 && W % 128 == 0 && BYTES <= SMEM_LIMIT, "shared memory of one CTA");
};

// four weights as (2 w + 1) mod 2^16 in 16-bit halves (inputs 0, 2 | 1, 3) -> one word of each plane.  A low half that
// is negative borrows from the high one, which only clears the 1 there.
__device__ __forceinline__ void split_planes(uint32_t p02, uint32_t p13, uint32_t *hi, uint32_t *lo) {
    *hi = __byte_perm(p02, p13, 0x7351);                              // 2 w >> 8 = w >> 7
    *lo = (__byte_perm(p02, p13, 0x6240) >> 1) & 0x7F7F7F7Fu;         // w & 127
}
// byte k of w, sign-extended
template <int K> __device__ __forceinline__ int sbyte_of(uint32_t w) {
    int r;
    asm("prmt.b32 %0, %1, 0, %2;" : "=r"(r) : "r"(w), "n"(0x8880 + 0x1111 * K));
    return r;
}

// One row's share of a lane (inputs 4 j .. of every k-step of 16): base = the row's bytes of this super-block, dst = the
// lane's word in k-step 0 of the high plane; k-steps lie 128 bytes apart.
// SKEW: base is 2 past a multiple of 4
template <bool SKEW> __device__ __forceinline__ uint32_t lds32_skew(smem_ptr p) {
    if (!SKEW) return lds32(p);
    return __funnelshift_r(lds32(p - 2), lds32(p + 2), 16);
}
template <bool SKEW>
__device__ __forceinline__ float unpack_q6k(smem_ptr base, int j, unsigned char *dst) {
    uint32_t scw[4];                                                  // 16 signed scales, one per k-step
#pragma unroll
    for (int k = 0; k < 4; k++) scw[k] = lds32_skew<SKEW>(base + 192 + 4 * k);
#pragma unroll
    for (int h = 0; h < 2; h++) {
        uint32_t qlw[2][2], qhw[2];                                   // a half's words before its first store: the compiler keeps loads behind stores
#pragma unroll
        for (int u = 0; u < 2; u++) {
            qlw[u][0] = lds32_skew<SKEW>(base + 64 * h + 16 * u + 4 * j);
            qlw[u][1] = lds32_skew<SKEW>(base + 64 * h + 32 + 16 * u + 4 * j);
            qhw[u] = lds32_skew<SKEW>(base + 128 + 32 * h + 16 * u + 4 * j);
        }
#pragma unroll
        for (int u = 0; u < 2; u++) {
            const uint32_t ql0 = qlw[u][0], ql1 = qlw[u][1], qh = qhw[u];
            auto step = [&](auto C) {                                 // quarter c of the half: twice the 6-bit codes, then k-step 8 h + 2 c + u
                constexpr int c = decltype(C)::value;
                const uint32_t ql = (c & 1) ? ql1 : ql0;
                const uint32_t v = ((c >> 1 ? ql >> 3 : ql << 1) & 0x1E1E1E1Eu) |
                                   ((c == 0 ? qh << 5 : c == 1 ? qh << 3 : c == 2 ? qh << 1 : qh >> 1) & 0x60606060u);
                const int s = 8 * h + 2 * c + u;
                const uint32_t w = scw[2 * h + (c >> 1)];
                const int sc = (c & 1) ? (u ? sbyte_of<3>(w) : sbyte_of<2>(w)) : (u ? sbyte_of<1>(w) : sbyte_of<0>(w));
                const uint32_t bias = (uint32_t)sc * (uint32_t)(-64 * 65537) + 65537u;       // (2 code) sc - 64 sc + 1 in each half
                uint32_t hi, lo;
                split_planes((v & 0x00FF00FFu) * (uint32_t)sc + bias, __byte_perm(v, 0u, 0x4341) * (uint32_t)sc + bias, &hi, &lo);
                *reinterpret_cast<uint32_t *>(dst + s * 128) = hi;
                *reinterpret_cast<uint32_t *>(dst + PLANE + s * 128) = lo;
            };
            step(std::integral_constant<int, 0>{}); step(std::integral_constant<int, 1>{});
            step(std::integral_constant<int, 2>{}); step(std::integral_constant<int, 3>{});
        }
    }
    const uint32_t dbits = SKEW ? lds32(base + 206) >> 16 : lds32(base + 208) & 0xFFFFu;
    return f16_bits_to_f32(dbits);
}
// amin: the lane's word of the row's minimums operand (8 minimums, 8 zeros; the second k-step of 16 stays zero)
__device__ __forceinline__ float2 unpack_q4k(smem_ptr base, int j, unsigned char *dst, unsigned char *amin) {
    const uint32_t hd = lds32(base), w0 = lds32(base + 4), w1 = lds32(base + 8), w2 = lds32(base + 12);
    const uint32_t sc_lo = w0 & 0x3F3F3F3Fu, sc_hi = (w2 & 0x0F0F0F0Fu) | ((w0 >> 2) & 0x30303030u);
    const uint32_t mn_lo = w1 & 0x3F3F3F3Fu, mn_hi = ((w2 >> 4) & 0x0F0F0F0Fu) | ((w1 >> 2) & 0x30303030u);
    uint32_t qw[4][2];                                                // all words before the first store: the compiler keeps loads behind stores
#pragma unroll
    for (int p = 0; p < 4; p++)
#pragma unroll
        for (int half = 0; half < 2; half++) qw[p][half] = lds32(base + 16 + 32 * p + 16 * half + 4 * j);
    *reinterpret_cast<uint32_t *>(amin) = j == 0 ? mn_lo : (j == 1 ? mn_hi : 0u);
#pragma unroll
    for (int p = 0; p < 4; p++)                                       // sub-blocks 2 p (low nibbles) and 2 p + 1 (high)
#pragma unroll
        for (int half = 0; half < 2; half++) {
            const uint32_t q = qw[p][half];
#pragma unroll
            for (int n = 0; n < 2; n++) {
                const int jb = 2 * p + n;
                const uint32_t sc = ((jb < 4 ? sc_lo : sc_hi) >> (8 * (jb & 3))) & 0xFFu;
                uint32_t hi, lo;
                split_planes(((n ? q >> 3 : q << 1) & 0x001E001Eu) * sc, ((n ? q >> 11 : q >> 7) & 0x001E001Eu) * sc, &hi, &lo);
                *reinterpret_cast<uint32_t *>(dst + (2 * jb + half) * 128) = hi;
                *reinterpret_cast<uint32_t *>(dst + PLANE + (2 * jb + half) * 128) = lo;
            }
        }
    return make_float2(f16_bits_to_f32(hd & 0xFFFFu), f16_bits_to_f32(hd >> 16));
}

// (float)(F hi + lo) of two pairs of int32 sums
__device__ __forceinline__ f32x2 sums_to_f32(float h0, float h1, float l0, float l1, int F) {
    return pack2((float)(__float_as_int(h0) * F + __float_as_int(l0)), (float)(__float_as_int(h1) * F + __float_as_int(l1)));
}

constexpr int MAX_NX = 5;
struct Bars {
    unsigned long long w_full[2], w_free[2], a_full, x_full[MAX_NX], x_free[MAX_NX], mma_done[2], d_free[2];
};

template <int TYPE, int H>
__global__ void __launch_bounds__(NTHREADS, 1) k_matmul_kq_tc5(KqArgs a, int n_tiles, const __grid_constant__ KqGroup grp) {
    using F = Tc5Fmt<TYPE>;
    using S = Tc5Smem<TYPE, H>;
    constexpr int BLOCK = Fmt<TYPE>::BLOCK, BOX = Fmt<TYPE>::BOX, NS = F::NS, COLS = NS / 4;
    extern __shared__ unsigned char smem_raw[];
    __shared__ __align__(8) Bars bars;
    __shared__ uint32_t tmem_slot;
    unsigned char *smem = smem_raw + ((128 - (tc5::su32(smem_raw) & 127)) & 127);
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, nseg = a.nseg;
    if (tid == 0) {
        tc5::mbar_init(tc5::su32(&bars.a_full), NWORK);
        for (int i = 0; i < 2; i++) {
            tc5::mbar_init(tc5::su32(&bars.w_full[i]), 1);
            tc5::mbar_init(tc5::su32(&bars.w_free[i]), NWORK);
            tc5::mbar_init(tc5::su32(&bars.mma_done[i]), MMA_DONE_ARRIVALS);
            tc5::mbar_init(tc5::su32(&bars.d_free[i]), NWORK);
        }
        for (int i = 0; i < S::NX; i++) {
            tc5::mbar_init(tc5::su32(&bars.x_full[i]), 1);
            tc5::mbar_init(tc5::su32(&bars.x_free[i]), NWORK);
        }
        tc5::mbar_init_fence();
    }
    if (warp == W_MMA) tc5::tmem_alloc(&tmem_slot, 512);
    if (F::AMIN && tid < 256) *reinterpret_cast<uint4 *>(smem + S::O_AMIN + tid * 16) = make_uint4(0, 0, 0, 0);
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
                const Tile t = tile_of<NS, H>(grp, a.T, idx);
                for (int s = 0; s < nseg; s++, n++) {
                    if (n >= 2) {                                     // the rows that had this stage are unpacked
                        ok = tc5::mbar_wait_parked(tc5::su32(&bars.w_free[n & 1]), (uint32_t)((n - 2) >> 1) & 1u);
                        if (!ok) break;
                        asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory");
                    }
                    // rows past n_out and bytes past a row's end are outside the map: zeros
                    const uint32_t bar = tc5::su32(&bars.w_full[n & 1]);
                    tc5::mbar_expect_tx(bar, (uint32_t)S::W);
                    tensor_copy_rows(tc5::su32(smem + S::O_W + (n & 1) * S::W), &grp.map[t.pj], ((s * BLOCK) & ~15) / 4, t.row0, bar);
                }
            }
            if (!ok) {                                                // leave no copy in flight
                for (int v = n - 1; v >= 0 && v >= n - 2; v--) tc5::mbar_wait(tc5::su32(&bars.w_full[v & 1]), (uint32_t)(v >> 1) & 1u);
                tc5::report_timeout(a.status, ORN_WAIT_DECODE);
            }
        }
    } else if (warp == X_COPY) {
        // ---- activation images, unit by unit ---------------------------------------------------------------------
        if (tc5::elect_one()) {
            asm volatile("griddepcontrol.wait;\n" ::: "memory");     // they come from the kernel in front
            int st = 0, round = 0, issued = 0;
            for (int idx = blockIdx.x; idx < n_tiles && ok; idx += gridDim.x) {
                const Tile t = tile_of<NS, H>(grp, a.T, idx);
                const int nt = (t.n_tok + 7) / 8;
                for (int s = 0; s < nseg && ok; s++)
                    for (int h = 0; h < t.nh; h++) {
                        if (round > 0) {                              // the unit that had this stage is drained
                            ok = tc5::mbar_wait_parked(tc5::su32(&bars.x_free[st]), (uint32_t)(round - 1) & 1u);
                            if (!ok) break;
                            asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory");
                        }
                        const int t0 = h * (NS / 8), n = min(nt - t0, NS / 8);
                        const uint32_t bar = tc5::su32(&bars.x_full[st]), dst = tc5::su32(smem + S::O_X + st * S::XUNIT);
                        tc5::mbar_expect_tx(bar, (uint32_t)(n * F::XB));
                        for (int i = 0; i < n; i++)
                            bulk_copy(dst + i * F::XB, a.img + ((size_t)((t.tok0 >> 3) + t0 + i) * nseg + s) * ORN_Q8K_IMG_BYTES, F::XB, bar);
                        issued++;
                        if (++st == S::NX) { st = 0; round++; }
                    }
            }
            if (!ok) {                                                // leave no copy in flight
                for (int v = issued - 1; v >= 0 && v >= issued - S::NX; v--)
                    tc5::mbar_wait(tc5::su32(&bars.x_full[v % S::NX]), (uint32_t)(v / S::NX) & 1u);
                tc5::report_timeout(a.status, ORN_WAIT_DECODE);
            }
        }
    } else if (warp == W_MMA) {
        // ---- MMA issue ---------------------------------------------------------------------------------------
        // Products follow one another faster behind an election than behind a lane's number.  For Q4_K with two units that is the
        // slower form: 512 tokens 8192 -> 4096 97.1 against 93.6 us, 777 tokens 2048 -> 12352 133 against 128 (one, three and four
        // units 0 to 2 % the other way; Q6_K 0.3 to 1 %).
        constexpr bool ELECT = !(TYPE == T_Q4K && H == 2);
        if (ELECT ? tc5::elect_one() : lane == 0) {
            const uint32_t A = tc5::su32(smem), X = tc5::su32(smem + S::O_X);
            const uint64_t a_hi = desc_plain(A, 128, QK * 8), a_lo = desc_plain(A + PLANE, 128, QK * 8), a_min = desc_plain(A + S::O_AMIN, 128, 256);
            int u = 0, st = 0, round = 0, n_sb = 0;
            for (int idx = blockIdx.x; idx < n_tiles && ok; idx += gridDim.x) {
            const Tile t = tile_of<NS, H>(grp, a.T, idx);
            const int n_last = (t.n_tok - (t.nh - 1) * NS + 15) & ~15;
            for (int s = 0; s < nseg && ok; s++, n_sb++) {
                ok = tc5::mbar_wait_parked(tc5::su32(&bars.a_full), (uint32_t)n_sb & 1u);
                for (int h = 0; h < t.nh && ok; h++, u++) {
                    const int slot = u & 1;
                    ok = tc5::mbar_wait_parked(tc5::su32(&bars.x_full[st]), (uint32_t)round & 1u);
                    if (ok && u >= 2) ok = tc5::mbar_wait_parked(tc5::su32(&bars.d_free[slot]), (uint32_t)((u >> 1) - 1) & 1u);
                    if (!ok) break;
                    tc5::fence_after();
                    const int n = h == t.nh - 1 ? n_last : NS;
                    const uint32_t id = idesc_i8(true, n), d = tmem + slot * (F::NACC * NS), xu = X + st * S::XUNIT;
                    const uint64_t b = desc_plain(xu, 128, F::XB);
#pragma unroll
                    for (int k = 0; k < QK / 32; k++) {               // a k-step is two core matrices: 256 bytes
                        mma_i8_ss(d, a_hi + 16 * k, b + 16 * k, id, k > 0);
                        mma_i8_ss(d + NS, a_lo + 16 * k, b + 16 * k, id, k > 0);
                    }
                    if (F::AMIN) {                                    // the sums' bytes are one core matrix; what lies behind it meets zeros
                        mma_i8_ss(d + 2 * NS, a_min, desc_plain(xu + ORN_Q8K_IMG_LO, 128, F::XB), idesc_i8(false, n), 0);
                        mma_i8_ss(d + 3 * NS, a_min, desc_plain(xu + ORN_Q8K_IMG_HI, 128, F::XB), id, 0);
                    }
                    mma_issued(tc5::su32(&bars.mma_done[slot]));
                    if (++st == S::NX) { st = 0; round++; }
                }
            }
            }
            if (!ok) {                                                // leave no product in flight
                for (int v = u - 1; v >= 0 && v >= u - 2; v--) tc5::mbar_wait(tc5::su32(&bars.mma_done[v & 1]), (uint32_t)(v >> 1) & 1u);
                tc5::report_timeout(a.status, ORN_WAIT_DECODE);
            }
        }
    } else if (warp < NWORK) {
        // ---- unpack and drain --------------------------------------------------------------------------------
        float *scales = reinterpret_cast<float *>(smem + S::O_D);    // [4 super-blocks][NSCALE][128 rows]
        const int q = warp & 3, cg = warp >> 2;                      // tensor-memory lanes 32 q .., columns COLS cg ..
        const uint32_t tq = tmem + ((uint32_t)(q * 32) << 16) + cg * COLS;
        f32x2 tot[H][COLS / 2];
        auto wait_all = [&](unsigned long long *bar, uint32_t parity) {
            if (ok) ok = __all_sync(0xffffffffu, tc5::mbar_wait(tc5::su32(bar), parity));
        };
        const f32x2 mz = pack2(a.minus_zero, a.minus_zero);
        int st = 0, du = 0;                                           // image stage and number of the next unit to drain
        auto drain = [&](auto HI, int n, int n_tok) {                 // a unit of super-block n (counted over all tiles)
            constexpr int h = decltype(HI)::value;
            const int slot = du & 1;
            wait_all(&bars.mma_done[slot], (uint32_t)(du >> 1) & 1u);
            if (!ok) return;
            tc5::fence_after();
            if (h * NS + cg * COLS < n_tok) {
                const float *sc = scales + (n & 3) * (S::NSCALE * ROWS) + q * 32 + lane;
                const f32x2 dw = pack2(sc[0], sc[0]), dmw = F::AMIN ? pack2(-sc[ROWS], -sc[ROWS]) : 0;      // (-yd) dmw = yd (-dmw)
                const unsigned char *xu = smem + S::O_X + st * S::XUNIT + cg * (COLS / 8) * F::XB + ORN_Q8K_IMG_D;
                const uint32_t t0 = tq + slot * (F::NACC * NS);
#pragma unroll
                for (int c = 0; c < COLS; c += 8) {                   // 8 columns = one image tile (16 at a time spill registers)
                    float vh[8], vl[8];
                    f32x2 term[4];
                    tc5::tmem_ld8x2_wait(t0 + c, vh, t0 + NS + c, vl);
                    auto scale_of = [&](int e) {                      // activation scales of columns c + 2 e, + 1
                        const float2 y = *reinterpret_cast<const float2 *>(xu + c / 8 * F::XB + e * 8);
                        return pack2(y.x, y.y);
                    };
#pragma unroll
                    for (int e = 0; e < 4; e++)
                        term[e] = mul2_apart(mul2(scale_of(e), dw), sums_to_f32(vh[2 * e], vh[2 * e + 1], vl[2 * e], vl[2 * e + 1], 128), mz);
                    if (F::AMIN) {
                        tc5::tmem_ld8x2_wait(t0 + 2 * NS + c, vl, t0 + 3 * NS + c, vh);
#pragma unroll
                        for (int e = 0; e < 4; e++)
                            term[e] = add2(term[e], mul2_apart(mul2(scale_of(e), dmw), sums_to_f32(vh[2 * e], vh[2 * e + 1], vl[2 * e], vl[2 * e + 1], 256), mz));
                    }
#pragma unroll
                    for (int e = 0; e < 4; e++) tot[h][c / 2 + e] = add2(tot[h][c / 2 + e], term[e]);
                }
            }
            tc5::fence_before();
            __syncwarp();
            if (lane == 0) {
                tc5::mbar_arrive(tc5::su32(&bars.d_free[slot]));
                tc5::mbar_arrive(tc5::su32(&bars.x_free[st]));
            }
            if (++st == S::NX) st = 0;
            du++;
        };
        auto drain_last = [&](int n, int n_tok) {                     // the last unit of super-block n, which is one of a tile of n_tok tokens
            if (H == 1 || n_tok <= NS) drain(std::integral_constant<int, 0>{}, n, n_tok);
            else if (H == 2 || n_tok <= 2 * NS) drain(std::integral_constant<int, (H >= 2) ? 1 : 0>{}, n, n_tok);
            else if (H == 3 || n_tok <= 3 * NS) drain(std::integral_constant<int, (H >= 3) ? 2 : 0>{}, n, n_tok);
            else drain(std::integral_constant<int, H - 1>{}, n, n_tok);
        };
        auto store = [&](int idx) {
            const Tile t = tile_of<NS, H>(grp, a.T, idx);
            const int row = t.row0 + q * 32 + lane;
            if (row >= t.n_out) return;
#pragma unroll
            for (int h = 0; h < H; h++)
#pragma unroll
                for (int i = 0; i < COLS; i++) {
                    const int c = h * NS + cg * COLS + i;
                    if (c >= t.n_tok) continue;
                    float v0, v1;
                    unpack2(tot[h][i / 2], &v0, &v1);
                    const float val = !ok ? NAN : (i & 1) ? v1 : v0;
                    if (a.out_dtype == ORNITH_ACT_BF16) act_st((__nv_bfloat16 *)grp.y[t.pj], (size_t)(t.tok0 + c) * t.n_out + row, val);
                    else act_st((float *)grp.y[t.pj], (size_t)(t.tok0 + c) * t.n_out + row, val);
                }
        };
        const int g = lane >> 2, j = lane & 3;
        int n = 0;                                                    // super-blocks begun
        for (int idx = blockIdx.x; idx < n_tiles; idx += gridDim.x) {
            const int n_tok = tile_of<NS, H>(grp, a.T, idx).n_tok;
#pragma unroll
            for (int h = 0; h < H; h++)
#pragma unroll
                for (int i = 0; i < COLS / 2; i++) tot[h][i] = 0;
            for (int s = 0; s < nseg; s++, n++) {
                if (s > 0) wait_all(&bars.mma_done[du & 1], (uint32_t)(du >> 1) & 1u);       // the planes are free: the last unit of n - 1 is multiplied
                wait_all(&bars.w_full[n & 1], (uint32_t)(n >> 1) & 1u);
                if (!ok) break;
                const int row = warp * 8 + g;
                smem_ptr base = smem + S::O_W + (n & 1) * S::W + row * BOX + ((s * BLOCK) & 15);
                unsigned char *dst = smem + warp * (8 * QK) + lane * 4;
                float *sc = scales + (n & 3) * (S::NSCALE * ROWS) + row;
                if (TYPE == T_Q6K) {
                    const float d = ((s * BLOCK) & 2) ? unpack_q6k<true>(base, j, dst) : unpack_q6k<false>(base, j, dst);
                    if (j == 0) sc[0] = d;
                } else {
                    const float2 d = unpack_q4k(base, j, dst, smem + S::O_AMIN + warp * 256 + lane * 4);
                    if (j == 0) { sc[0] = d.x; sc[ROWS] = d.y; }
                }
                asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory");
                __syncwarp();
                if (lane == 0) { tc5::mbar_arrive(tc5::su32(&bars.a_full)); tc5::mbar_arrive(tc5::su32(&bars.w_free[n & 1])); }
                if (s > 0) drain_last(n - 1, n_tok);
                wait_all(&bars.a_full, (uint32_t)n & 1u);             // every warp's weight scales are in place
                if (H > 1 && n_tok > NS) drain(std::integral_constant<int, 0>{}, n, n_tok);      // the units of n but its last
                if (H > 2 && n_tok > 2 * NS) drain(std::integral_constant<int, (H > 2) ? 1 : 0>{}, n, n_tok);
                if (H > 3 && n_tok > 3 * NS) drain(std::integral_constant<int, (H > 3) ? 2 : 0>{}, n, n_tok);
            }
            if (ok) drain_last(n - 1, n_tok);
            store(idx);                                               // NaN once a wait has given up: this tile and the rest of the CTA's
        }
        if (!ok && lane == 0) tc5::report_timeout(a.status, ORN_WAIT_DECODE);
    }
    tc5::fence_before();
    __syncthreads();
    tc5::fence_after();
    if (warp == W_MMA) tc5::tmem_dealloc(tmem, 512);
}

template <int TYPE, int H>
ornith_status launch_h(const HostGroup &h, int n_in, int T, const KqArgs &a, cudaStream_t stream) {
    constexpr int TOK = H * Tc5Fmt<TYPE>::NS, SMEM = Tc5Smem<TYPE, H>::BYTES;
    KqGroup g;
    if (!fill_group<TYPE>(&g, h, n_in, ROWS)) return (ornith_status)ORNITH_ERR_BACKEND;
    static bool opted[ORN_MAX_DEVICES] = {};
    bool &have = opted[orn_device_index()];
    if (!have) {
        ORN_TRY(orn_check(cudaFuncSetAttribute(k_matmul_kq_tc5<TYPE, H>, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM), "projection smem opt-in"));
        have = true;
    }
    const int n_tiles = g.cta0[h.n] * ((T + TOK - 1) / TOK);
    return orn_check(orn_launch_dependent(k_matmul_kq_tc5<TYPE, H>, dim3((unsigned)(n_tiles < SMS ? n_tiles : SMS)), dim3(NTHREADS), SMEM, stream,
                                          a, n_tiles, g), "k_matmul_kq_tc5");
}

}  // namespace

namespace kq {

// Microseconds per super-block of a product over all of its waves (fitted to n_in = 8192, n_out = 4096, 777 tokens; H units
// per CTA cost (1 + H) / 2 of one unit, unpacking being shared: measured 1 : 1.5 : 2.1 : 2.7).  *units: the best H.
template <int TYPE>
float kq_tc5_cost(const HostGroup &h, int T, int *units) {
    constexpr int NS = Tc5Fmt<TYPE>::NS, HMAX = TYPE == T_Q6K ? 2 : 4;
    long long row_tiles = 0;
    for (int i = 0; i < h.n; i++) row_tiles += (h.n_out[i] + ROWS - 1) / ROWS;
    float best = 0.0f;
    *units = 0;
    if (row_tiles * ((T + NS - 1) / NS) > (1 << 30)) return best;
    for (int H = 1; H <= HMAX; H++) {
        const long long tiles = row_tiles * ((T + H * NS - 1) / (H * NS));
        const float cost = (float)((tiles + SMS - 1) / SMS * (1 + H)) * (TYPE == T_Q6K ? 1.10f : 0.98f);
        if (*units == 0 || cost < best) { *units = H; best = cost; }
    }
    return best;
}

template <int TYPE>
ornith_status launch_kq_tc5(const HostGroup &h, int n_in, int T, const KqArgs &a, int units, cudaStream_t stream) {
    if (units == 1) return launch_h<TYPE, 1>(h, n_in, T, a, stream);
    if constexpr (TYPE == T_Q4K) {
        if (units == 3) return launch_h<TYPE, 3>(h, n_in, T, a, stream);
        if (units == 4) return launch_h<TYPE, 4>(h, n_in, T, a, stream);
    }
    return launch_h<TYPE, 2>(h, n_in, T, a, stream);
}

template float kq_tc5_cost<T_Q4K>(const HostGroup &, int, int *);
template float kq_tc5_cost<T_Q6K>(const HostGroup &, int, int *);
template ornith_status launch_kq_tc5<T_Q4K>(const HostGroup &, int, int, const KqArgs &, int, cudaStream_t);
template ornith_status launch_kq_tc5<T_Q6K>(const HostGroup &, int, int, const KqArgs &, int, cudaStream_t);

}  // namespace kq
