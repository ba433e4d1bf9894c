// delta_scan_tc5.cu — gated delta-net prefill scan for dk = dv = 128 on the 5th-generation
// tensor cores: operands staged by bulk copies, tcgen05.mma (tf32) with the recurrent state and every
// intermediate of the chunk in tensor memory.
//
// Reference behaviour being replaced: the chunked scan of ornith_delta_prefill
// (src/ornith_attn.c:215-349) inside linear_attn_prefill (src/ornith_rforward.c:563-618), with
// linear_finish (src/ornith_rforward.c:300-314) as the epilogue.
//
// Per chunk of 64 tokens with incoming state S [dv][dk], raw (conv + SiLU) rows k_i, q_i with
// inverse norms rk_i, rq_i, G_i the running sum of the log-decay inside the chunk, p_i = exp(G_i),
// Gamma_ij = exp(G_i - G_j), w_j = Gamma_63,j:
//   M = diag(beta) strictLower(Gamma o Khat Khat^T),  A = (I + M)^-1,  P = lower(Gamma o Qhat Khat^T)
//   T = beta V - diag(beta p rk) (K S^T),  U = A T
//   O = diag(p rq) (Q S^T) + P U
//   S <- p_63 S + sum_j (w_j rk_j u_j) k_j^T
// (Khat, Qhat the normalised rows; the norms are folded into the per-token factors so that the
// tensor cores read the K / Q tiles straight from the conv output; its v channels are stored as beta V, in f32.)  A, P and
// the per-token factors do not depend on the state: k_delta_prep produces them for all chunks at once.
//
// k_delta_scan_tc5, one CTA per (value head, sequence), keeps everything transposed, dv on the
// 128 tensor-memory lanes:
//   (K S^T)^T = S K^T             M128 N64  K128   A operand = the state itself (tensor memory)
//   (Q S^T)^T = S Q^T             M128 N64  K128   the same
//   U^T  = T^T A^T                M128 N64  K64    A operand = T^T, formed in f32 and rounded once
//   S'  = p_63 S + (w rk U)^T K   M128 N128 K64    A operand = (w rk U)^T; B = the K tile, MN-major
//   (PU)^T = U^T P^T              M128 N64  K64    A operand = U^T
// so the fp32 state never leaves tensor memory during a prompt: it is the accumulator of the
// update and, read as tf32 (low mantissa bits ignored), the A operand of the next chunk.
//
// T is a difference, small where the state already holds what is written (keys that come again, slow decay), and its error
// enters the state: it is formed in f32 from f32 terms, rounded to nearest, and meets one rounded A.  As
// U = A (beta V) + A' (K S^T), A' = -A diag(beta p rk), with both matrices and both terms rounded on their own, a token repeated
// 1000 times left the state 3.5e-3 off (largest error over largest value; so 3.1e-4), where independent rows show nothing of it.
#include <cuda.h>
#include <cuda_runtime.h>
#include <math.h>

#include <mutex>
#include <type_traits>

#include "linear_attn.cuh"
#include "tcgen05.cuh"

namespace {
using namespace tc5;

constexpr int C = 64;                                   // tokens per chunk
constexpr float LOG2E_F = 1.4426950408889634f;
// What the preparation leaves for one (value head, chunk), in the layouts the scan's copies need: every part is one
// contiguous bulk copy.
//   A, P    lower triangular: columns 0..31 of 64 rows, then columns 32..63 of rows 32..63; rows of 128 bytes, 128-byte swizzle
//           (a K-major B operand)
//   factors    w rk (64), p rq (64), p_63 and 3 more, -beta p rk (64)
constexpr int REC_A = 0, REC_P = 12288, REC_F = 24576, REC_BYTES = 25600;
constexpr uint32_t TRI_BYTES = 12288, FAC_BYTES = (3 * C + 4) * 4;
constexpr int F_W = 0, F_PQ = C, F_PEND = 2 * C, F_BPK = 2 * C + 4;
static_assert(REC_F + (int)FAC_BYTES <= REC_BYTES && REC_BYTES % 256 == 0 && FAC_BYTES % 16 == 0, "record layout");
// float index of element (i, l) of such a triangle
__device__ __forceinline__ int tri_at(int i, int l) { return (l & 32) * 64 + (i - (l & 32)) * 32 + (((((l & 31) >> 2) ^ (i & 7)) << 2) | (l & 3)); }

__device__ __forceinline__ void tma_load_3d(uint32_t dst, const CUtensorMap *map, int x, int y, int z, uint32_t bar) {
    asm volatile("cp.async.bulk.tensor.3d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5}], [%2];"
                 ::"r"(dst), "l"(map), "r"(bar), "r"(x), "r"(y), "r"(z) : "memory");
}

__device__ __forceinline__ void mma_tf32_sync(float (&d)[4], const float (&a)[4], float b0, float b1) {
    asm("mma.sync.aligned.m16n8k8.row.col.f32.tf32.tf32.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
        : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
        : "r"(__float_as_uint(a[0])), "r"(__float_as_uint(a[1])), "r"(__float_as_uint(a[2])),
          "r"(__float_as_uint(a[3])), "r"(__float_as_uint(b0)), "r"(__float_as_uint(b1)));
}

// =============================================================================
// state-independent part: one CTA per (chunk, key head, sequence), 256 threads
// =============================================================================
//   gates     of up to four value heads, a thread per (head, token), while the K and Q rows are on their way
//   Gram      K K^T and Q K^T, lower triangle, tf32 mma.sync, kept in the accumulators for all value heads
//   M, P      from the accumulators: P to the record, M over the K and Q rows
//   A         blocked inverse, in f32: the 32 x 32 diagonal blocks of all heads by substitution, a warp each (a lane per column), then the
//             block below, four warps to a head, by two products
// What the former kernel spent its 25k to 35k cycles a chunk on was waiting: shared-memory loads behind stores that might alias them,
// a broadcast load to every two multiply-adds, gate inputs and rows fetched one dependent load after the other.  Here the
// loads of a phase are issued together and nothing but M goes through shared memory: 22k to 27k cycles, two CTAs to an SM; 4096 tokens of
// 64 heads 85 -> 68 us.  It is bound by latency and shared memory (issue 0.42, shared-memory pipe 0.77).  Measured and not kept: the products of the
// inverse on the tensor cores in three tf32 terms (60 us, but A then differs in the last places from what f32 gives); three
// CTAs to an SM (75 us, spills); persistent CTAs that request the next item's rows early (71 us).
//
// M has rows of 16-byte pieces; piece c of row r lies at c ^ f(r), f = the three low bits of r in reverse order: a fragment's stores and
// the reads along rows and down columns stay clear of bank conflicts.  Row offsets that are multiples of 8 leave f alone: a lane's
// addresses differ by constants.
__device__ __forceinline__ constexpr int swz(int r) { return ((r & 1) << 2) | (r & 2) | ((r >> 2) & 1); }
__device__ __forceinline__ void ldmatrix_x4(float (&r)[4], uint32_t addr) {
    uint32_t x[4];
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0, %1, %2, %3}, [%4];" : "=r"(x[0]), "=r"(x[1]), "=r"(x[2]), "=r"(x[3]) : "r"(addr) : "memory");
#pragma unroll
    for (int i = 0; i < 4; i++) r[i] = __uint_as_float(x[i]);
}

constexpr int HB = 4;                                   // value heads of a batch
struct PrepSmem {
    union {
        struct { float K[C * 128], Q[C * 128]; } t;     // as copied: 4 slabs of 32 dims x 64 rows of 128 bytes, 128-byte swizzle; dead once the Gram matrices exist
        float M[HB][C * C];
    } u;
    float g[HB][C], be[HB][C], tot[HB], gend[HB], rk[C], rq[C];
};

constexpr int PREP_SMEM = (int)sizeof(PrepSmem) + 1024; // + alignment slack

__device__ __forceinline__ void team_sync(int id) { asm volatile("bar.sync %0, 128;" ::"r"(id) : "memory"); }

// Diagonal block q of (I + M)^-1, 32 x 32, over that of M, by a warp, by forward substitution, lane = column.  M is strictly lower
// triangular inside its 16 x 16 diagonal blocks (zeros elsewhere in them).  Four partial sums per row: the rows form one dependent
// chain, and a single accumulator would make it 496 multiply-adds long.  (A row not yet solved counts as zero.)
__device__ __forceinline__ void invert_diagonal(float *M, int q, int lane) {
    float *B = M + 32 * q * 64 + 32 * q;                  // the block's first piece is number 8 q
    float nx[32];                                         // - the solution
#pragma unroll
    for (int i = 0; i < 32; i++) nx[i] = 0.0f;
#pragma unroll
    for (int i = 0; i < 32; i++) {
        f32x2 a01 = pack2(i == lane ? 1.0f : 0.0f, 0.0f), a23 = 0;
#pragma unroll
        for (int l4 = 0; l4 < (i + 3) / 4; l4++) {
            const float4 m = *reinterpret_cast<const float4 *>(B + i * 64 + ((l4 ^ swz(i)) << 2));
            a01 = fma2(pack2(m.x, m.y), pack2(nx[4 * l4], nx[4 * l4 + 1]), a01);
            if (4 * l4 + 2 < i) a23 = fma2(pack2(m.z, m.w), pack2(nx[4 * l4 + 2], nx[4 * l4 + 3]), a23);
        }
        float s0, s1, s2, s3;
        unpack2(a01, &s0, &s1);
        unpack2(a23, &s2, &s3);
        nx[i] = -((s0 + s1) + (s2 + s3));
    }
    __syncwarp();
#pragma unroll
    for (int i = 0; i < 32; i++) B[i * 64 + (((lane >> 2) ^ swz(i)) << 2) + (lane & 3)] = -nx[i];
}

// rows 8 q .. of the product of the 32 x 32 blocks at L (rows, 16 bytes at a time) and at R (lane = column): y[i] = sum_l L[8 q + i][l] R[l][lane]
__device__ __forceinline__ void block_rows(const float *L, const float *R, int q, int lane, float (&y)[8]) {
    float x[32];
    const int c3 = lane >> 2, c0 = lane & 3;
#pragma unroll
    for (int l = 0; l < 32; l++) x[l] = R[l * 64 + ((c3 ^ swz(l)) << 2) + c0];
#pragma unroll
    for (int i = 0; i < 8; i++) {
        f32x2 a = 0;
#pragma unroll
        for (int l4 = 0; l4 < 8; l4++) {
            const float4 m = *reinterpret_cast<const float4 *>(L + (8 * q + i) * 64 + ((l4 ^ swz(i)) << 2));
            a = fma2(pack2(m.x, m.y), pack2(x[4 * l4], x[4 * l4 + 1]), a);
            a = fma2(pack2(m.z, m.w), pack2(x[4 * l4 + 2], x[4 * l4 + 3]), a);
        }
        float s0, s1;
        unpack2(a, &s0, &s1);
        y[i] = s0 + s1;
    }
}
// The block below the diagonal ones, [[A11, 0], [-A22 M21 A11, A22]], over M21, by the four warps of a team (q = warp of the team, bar = the
// team's barrier), by rows.  The product M21 A11 takes the place above the diagonal blocks, which nothing else uses.
__device__ __forceinline__ void invert_below(float *M, int q, int lane, int bar) {
    float y[8];
    float *M21 = M + 32 * 64, *A22 = M21 + 32, *T = M + 32;
    const int c3 = lane >> 2, c0 = lane & 3;
    block_rows(M21, M, q, lane, y);
#pragma unroll
    for (int i = 0; i < 8; i++) T[(8 * q + i) * 64 + ((c3 ^ swz(i)) << 2) + c0] = y[i];
    team_sync(bar);
    block_rows(A22, T, q, lane, y);
#pragma unroll
    for (int i = 0; i < 8; i++) M21[(8 * q + i) * 64 + ((c3 ^ swz(i)) << 2) + c0] = -y[i];
    team_sync(bar);
}

struct PrepArgs64 {
    const float *Y, *rq, *rk, *la, *be;   // la, be: log-decay and write gate, or nullptr (made here from the layer's inputs)
    unsigned char *rec;                   // records [n_seq * nv][rec_chunks]
    int n_chunks, chunk0, rec_chunks, refresh;
    unsigned int *status;
};

template <typename ACT>
__global__ void __launch_bounds__(256, 2) k_delta_prep(const __grid_constant__ CUtensorMap map_y, LinArgs a, PrepArgs64 p) {
    // A programmatic dependent of the conv in front of it, as the scan is of this kernel (short prompts: three launches of
    // 8 to 40 us, whose latencies showed)
    dependent_entry();
    extern __shared__ __align__(16) unsigned char smraw[];
    __shared__ unsigned long long rows_in;
    PrepSmem &sm = *reinterpret_cast<PrepSmem *>(smraw + ((0u - su32(smraw)) & 1023u));
    const int chunk = p.chunk0 + blockIdx.x, kh = blockIdx.y, b = blockIdx.z, tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
    const int g = lane >> 2, j = lane & 3;
    const int qd = a.nk * 128, Cc = 2 * qd + a.nv * 128, nvk = a.nv / a.nk;
    const int t0 = chunk * C, n = min(C, a.T - t0);
    const size_t tok0 = (size_t)b * a.T + t0;
    auto head_of = [&](int m) { return a.head_map == ORNITH_HEADMAP_GROUPED ? kh * nvk + m : kh + m * a.nk; };

    if (tid == 0) {                                       // (asked for by the threads, 16 bytes each, the requests alone took 2500 cycles)
        mbar_init(su32(&rows_in), 1);
        mbar_init_fence();
        mbar_expect_tx(su32(&rows_in), 65536u);
        for (int sl = 0; sl < 4; sl++) {
            tma_load_3d(su32(sm.u.t.K) + sl * 8192, &map_y, qd + kh * 128 + 32 * sl, t0, b, su32(&rows_in));
            tma_load_3d(su32(sm.u.t.Q) + sl * 8192, &map_y, kh * 128 + 32 * sl, t0, b, su32(&rows_in));
        }
    }
    if (tid < C) {
        sm.rk[tid] = tid < n ? p.rk[(tok0 + tid) * a.nk + kh] : 0.0f;
        sm.rq[tid] = tid < n ? p.rq[(tok0 + tid) * a.nk + kh] : 0.0f;
    }
    // gates of the heads m0 .. m0 + 3: thread (head, token); running sums of the log-decay over the chunk
    const int gh = tid >> 6, pt = tid & 63;
    auto gates = [&](int m0) {
        float gg = 0.0f, bb = 0.0f;
        if (m0 + gh < nvk && pt < n) {
            const int hv = head_of(m0 + gh);
            const size_t i = (tok0 + pt) * a.nv + hv;
            if (p.la) { gg = p.la[i]; bb = p.be[i]; }
            else {                                        // reference: decay_alpha, src/ornith_rforward.c:282-284
                const float xa = act_ld((const ACT *)a.a, i), xb = act_ld((const ACT *)a.b, i), ac = a.a_coef[hv], dt = a.dt_bias[hv];
                gg = ac * softplus_f(xa + dt);
                bb = sigmoid_f(xb);
            }
        }
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const float up = __shfl_up_sync(0xffffffffu, gg, o);
            if (lane >= o) gg += up;
        }
        if (pt == 31) sm.tot[gh] = gg;
        __syncthreads();
        if (pt >= 32) gg += sm.tot[gh];
        if (pt == C - 1) sm.gend[gh] = gg;
        sm.g[gh][pt] = gg;
        sm.be[gh][pt] = bb;
        __syncthreads();
        if (m0 + gh < nvk) {
            float *f = reinterpret_cast<float *>(p.rec + (((size_t)b * a.nv + head_of(m0 + gh)) * p.rec_chunks + blockIdx.x) * REC_BYTES + REC_F);
            const float gend = sm.gend[gh], pp = expf(gg);
            f[F_W + pt] = expf(gend - gg) * sm.rk[pt];
            f[F_PQ + pt] = pp * sm.rq[pt];
            if (pt < 4) f[F_PEND + pt] = expf(gend);
            f[F_BPK + pt] = -bb * pp * sm.rk[pt];
        }
    };
    gates(0);
    // the conv has read the old history for the last time: store the last min(T, conv_k) inputs of the sequence (their own
    // launch took 2.4 us and a gap of a 512-token prompt's 72)
    if (p.refresh && p.chunk0 + (int)gridDim.x == p.n_chunks) {
        const int pos0 = a.pos[b];
        float *ring = a.conv + (size_t)b * a.conv_stride;
        const ACT *X = (const ACT *)a.qkv + (size_t)b * a.T * Cc;
        for (int ch = ((int)blockIdx.x * a.nk + kh) * 256 + tid; ch < Cc; ch += (int)gridDim.x * a.nk * 256) {
            float v[4];                                   // (conv_k is 4 on this path)
#pragma unroll
            for (int i = 0; i < 4; i++) v[i] = a.T - 4 + i >= 0 ? act_ld(X, (size_t)(a.T - 4 + i) * Cc + ch) : 0.0f;
#pragma unroll
            for (int i = 0; i < 4; i++)
                if (a.T - 4 + i >= 0) ring[(size_t)((pos0 + a.T - 4 + i) & 3) * Cc + ch] = v[i];
        }
    }
    if (!mbar_wait_warp(su32(&rows_in), 0u)) {            // A and P become NaN; the copies land before the CTA goes
        report_timeout(p.status, ORN_WAIT_DELTA_SCAN);
        sm.rk[lane] = sm.rk[32 + lane] = NAN;
        (void)mbar_wait_warp(su32(&rows_in), 0u);
    }

    // Gram tiles: warp w has the rows 16 mt .. of K and of Q and up to three groups of 8 columns from nt0 on (20 such groups lie on
    // or below the diagonal)
    const int mt = w < 3 ? 3 : w < 5 ? 2 : w < 7 ? 1 : 0, nt0 = w == 1 || w == 4 ? 3 : w == 2 ? 6 : w == 6 ? 2 : 0,
              cnt = w == 2 || w >= 5 ? 2 : 3;
    float gk[3][4] = {}, gq[3][4] = {};
    {
        const uint32_t ka = su32(sm.u.t.K) + (uint32_t)(16 * mt + (lane & 15)) * 128, kb = su32(sm.u.t.K) + (uint32_t)(8 * nt0 + (lane & 7)) * 128;
        const uint32_t fa = (uint32_t)(((lane >> 4) ^ (lane & 7)) << 4), fb = (uint32_t)(((lane >> 3) ^ (lane & 7)) << 4);
#pragma unroll
        for (int s2 = 0; s2 < 8; s2++) {                  // two k-steps of 8
            float qa[2][4], kf[2][4];
#pragma unroll
            for (int x = 0; x < 2; x++) {
                const uint32_t at = ka + (s2 >> 1) * 8192 + (((4 * (s2 & 1) + 2 * x) << 4) ^ fa);
                ldmatrix_x4(kf[x], at);
                ldmatrix_x4(qa[x], at + C * 128 * 4);
            }
            const uint32_t bt = kb + (s2 >> 1) * 8192 + (((s2 & 1) << 6) ^ fb);
#pragma unroll
            for (int t = 0; t < 3; t++)
                if (t < cnt) {
                    float r[4];
                    ldmatrix_x4(r, bt + t * 1024);
                    mma_tf32_sync(gk[t], kf[0], r[0], r[1]);
                    mma_tf32_sync(gq[t], qa[0], r[0], r[1]);
                    mma_tf32_sync(gk[t], kf[1], r[2], r[3]);
                    mma_tf32_sync(gq[t], qa[1], r[2], r[3]);
                }
        }
        if (n < C) {                                      // rows past the end are zeros, which count for nothing whatever they meet
#pragma unroll
            for (int t = 0; t < 3; t++)
#pragma unroll
                for (int x = 0; x < 4; x++)
                    if (16 * mt + g + 8 * (x >> 1) >= n || 8 * (nt0 + t) + 2 * j + (x & 1) >= n) gk[t][x] = gq[t][x] = 0.0f;
        }
        // the norms of both rows
        const float k0 = sm.rk[16 * mt + g], k1 = sm.rk[16 * mt + g + 8], q0 = sm.rq[16 * mt + g], q1 = sm.rq[16 * mt + g + 8];
#pragma unroll
        for (int t = 0; t < 3; t++)
            if (t < cnt) {
                const float2 rl = *reinterpret_cast<const float2 *>(&sm.rk[8 * (nt0 + t) + 2 * j]);
                gk[t][0] = gk[t][0] * k0 * rl.x; gk[t][1] = gk[t][1] * k0 * rl.y; gk[t][2] = gk[t][2] * k1 * rl.x; gk[t][3] = gk[t][3] * k1 * rl.y;
                gq[t][0] = gq[t][0] * q0 * rl.x; gq[t][1] = gq[t][1] * q0 * rl.y; gq[t][2] = gq[t][2] * q1 * rl.x; gq[t][3] = gq[t][3] * q1 * rl.y;
            }
    }

    for (int m0 = 0; m0 < nvk; m0 += HB) {
        const int heads = min(HB, nvk - m0);
        auto rec_of = [&](int h) { return p.rec + (((size_t)b * a.nv + head_of(m0 + h)) * p.rec_chunks + blockIdx.x) * REC_BYTES; };
        if (m0 > 0) gates(m0);
        __syncthreads();                                  // K and Q, or the A of the heads before, have been read for the last time
        // M and P from the Gram accumulators
        const int i0 = 16 * mt + g, i1 = i0 + 8;
        float *m_at[3];                                   // this lane's elements of M (head 0) and P: rows i0; eight rows on, the swizzle is the same
        int p_at[3];
#pragma unroll
        for (int t = 0; t < 3; t++) {
            const int l = 8 * (nt0 + t) + 2 * j, pc = l >> 2;
            m_at[t] = sm.u.M[0] + i0 * 64 + ((((pc & 7) ^ swz(g)) | (pc & 8)) << 2) + (l & 3);
            p_at[t] = tri_at(i0, l);
        }
#pragma unroll 1
        for (int h = 0; h < heads; h++) {
            const float g0 = sm.g[h][i0], g1 = sm.g[h][i1], b0 = sm.be[h][i0], b1 = sm.be[h][i1];
            float *Pg = reinterpret_cast<float *>(rec_of(h) + REC_P);
            auto tile = [&](int t, auto diag_t) {
                constexpr bool diag = decltype(diag_t)::value;        // a group of columns that meets the diagonal
                const int l = 8 * (nt0 + t) + 2 * j;
                const float2 gl = *reinterpret_cast<const float2 *>(&sm.g[h][l]);
                float e[4] = {(g0 - gl.x) * LOG2E_F, (g0 - gl.y) * LOG2E_F, (g1 - gl.x) * LOG2E_F, (g1 - gl.y) * LOG2E_F}, mm[4], pp[4];
#pragma unroll
                for (int x = 0; x < 4; x++) {
                    const int i = x < 2 ? i0 : i1, c = l + (x & 1);
                    if (diag && c > i) e[x] = -INFINITY;              // (above it the decay would grow)
                    e[x] = ex2_fast(e[x]);
                    mm[x] = (x < 2 ? b0 : b1) * e[x] * gk[t][x];
                    pp[x] = tf32q(e[x] * gq[t][x]);
                    if (diag && c >= i) mm[x] = 0.0f;
                    if (diag && c > i) pp[x] = 0.0f;
                }
                float *m = m_at[t] + h * (C * C), *P = Pg + p_at[t];
                *reinterpret_cast<float2 *>(m) = make_float2(mm[0], mm[1]);
                *reinterpret_cast<float2 *>(m + 512) = make_float2(mm[2], mm[3]);
                *reinterpret_cast<float2 *>(P) = make_float2(pp[0], pp[1]);
                *reinterpret_cast<float2 *>(P + 256) = make_float2(pp[2], pp[3]);
            };
#pragma unroll
            for (int t = 0; t < 3; t++)
                if (t < cnt) {
                    if (((nt0 + t) >> 1) == mt) tile(t, std::true_type{});
                    else tile(t, std::false_type{});
                }
            // the records' rows are whole: zeros right of the diagonal blocks of rows 0..15 (columns 16..31) and 32..47 (48..63)
            if (w == 7 || w == 5) {
                float *P = Pg + (lane >> 1) * 32 + (w == 5 ? 2048 : 0);
#pragma unroll
                for (int x = 0; x < 2; x++) *reinterpret_cast<float4 *>(P + (((4 + 2 * (lane & 1) + x) ^ ((lane >> 1) & 7)) << 2)) = make_float4(0.f, 0.f, 0.f, 0.f);
            }
        }
        __syncthreads();
        if ((w >> 1) < heads) invert_diagonal(sm.u.M[w >> 1], w & 1, lane);
        __syncthreads();
#pragma unroll 1
        for (int h = w >> 2; h < heads; h += 2) {         // two teams of four warps
            float *M = sm.u.M[h];
            invert_below(M, w & 3, lane, 1 + (w >> 2));
            // A, rounded to tf32: columns 0..31 of the rows 16 x .., then columns 32..63 of rows 32 + 16 (x - 4) ..
            const int t = tid & 127, pc = t & 7, r = t >> 3;
            const float *ms = M + r * 64 + ((pc ^ swz(r & 7)) << 2);
            float *Ag = reinterpret_cast<float *>(rec_of(h) + REC_A) + r * 32 + ((pc ^ (r & 7)) << 2);
#pragma unroll
            for (int x = 0; x < 6; x++) {
                const float4 v = *reinterpret_cast<const float4 *>(ms + (x < 4 ? x * 1024 : (x - 2) * 1024 + 32));
                *reinterpret_cast<float4 *>(Ag + x * 512) = make_float4(tf32q(v.x), tf32q(v.y), tf32q(v.z), tf32q(v.w));
            }
        }
    }
}

// =============================================================================
// sequential part: one CTA per (value head, sequence)
// =============================================================================
//   warps 0-7   chain: T from K S^T and beta V, the decayed copy of the state, then U as the operands of the two products behind it;
//               two threads per lane (row of S)
//   warps 8-23  output, off the chain: O, per-token RMSNorm over the head, SiLU(z) gate, store
//   warp 24     one lane issues the copies of the chunk's operands: one buffer each, refilled as soon as the product that reads it is
//               complete, which is most of a chunk before its next use.  K rows that serve as an MN-major operand come in 32-byte swizzle
//               atoms (a K-major tf32 operand must lie in 16-byte atoms, so K is copied twice)
//   warp 25     one lane issues the tcgen05.mma of the chain and Q S^T
//   warp 26     one lane issues those of P U: behind the state update in one stream they kept the issuing lane from the next chunk
//   warp 27     one lane issues the copies of z and of the outputs, and asks L2 for what comes two chunks later (without such
//               copies warp 24 asks: a lane that nothing waits for must not follow the scan by the parity of a barrier, which may
//               go round unseen)
// Tensor memory, 512 columns: two states of 128 (chunk n reads number n & 1; the other takes the decayed copy and then the
// update), K S^T / T / w rk U, the accumulator and then operand U, Q S^T, P U.
// A product that reads what an earlier product of another shape accumulated (the state) is only issued after a wait on that
// one's commit: the pipe does not order them, and issued back to back the read came too early.
// What bounds it: the chain of a chunk, K S^T (530 cycles), its commit, the pass over T (about 500: beta V is in registers by then),
// A T (260), its commit, the pass over U (about 600), the update (530), its commit; Q S^T and P U run beside those waits, and the copies, one
// period ahead, take up to 1.7 us when the passes in front of the next slab share the memory.  5.3k cycles a chunk (64 chunks x 64 heads
// alone 220 -> 180 us; with beta V read from shared memory behind K S^T 5.5k, with z loaded by the output warps 6.2k).
// The output warps have as long for a chunk.  So they read their tiles as 16 x 256-bit fragments, a thread holding 4 rows of 4 tokens
// (the sum of squares over the head is three shuffle levels on 4 values; as one row of 16 tokens it was five levels on 16),
// arithmetic goes in pairs, and z and bf16 outputs pass through shared memory by tensor copies, read and written as transposed
// 8 x 8 matrices (TILE; when z or out is not 16-byte aligned the threads load and store them): loaded by the threads one chunk
// ahead, z held up each chunk's shuffles for 1300 to 2000 cycles.
// Every wait is bounded in time; a wait that gives up is reported through the device status word and poisons the outputs.
constexpr int W_TMA = 24, W_MMA = 25, W_PU = 26, W_IO = 27, NTHREADS = 28 * 32;
constexpr int TM_S = 0, TM_X = 256, TM_U = 320, TM_QS = 384, TM_PU = 448, TM_COLS = 512;   // tensor-memory columns
constexpr int NFAC = 4;
constexpr int SM_K = 0, SM_V = 32768, SM_Q = 65536, SM_KM = 98304;   // (beta V: 64 rows of 128, not swizzled)
// the A tile whole (64 x 64): its upper right quarter is zeroed once and never written again
constexpr int SM_A = 131072, SM_P = SM_A + 16384;
constexpr int SM_F = SM_P + (int)TRI_BYTES;             // NFAC x factors
constexpr int SM_Z = (SM_F + NFAC * (int)FAC_BYTES + 1023) / 1024 * 1024;   // z of a chunk: 64 x 128 activations (bf16 or f32)
constexpr int SM_O = SM_Z + 16384;                      // bf16 outputs of a chunk on their way out (f32 ones are stored by the threads)
constexpr int SCAN_SMEM = SM_Z + 32768 + 1024;          // + alignment slack
static_assert(SCAN_SMEM + 4096 <= 227 * 1024, "with the static part: the shared memory of an SM");

enum { B_K, B_V, B_A, B_Q, B_KM, B_P, NBUF };           // operand buffers
struct ScanBars {
    unsigned long long full[NBUF], empty[NBUF], full_f[NFAC], red[2][4], o_full[4], o_free[4];
    unsigned long long ks_done, t_ready, u_done, wu_ready, u_ready, s_done, pu_done, qs_done, o_read, full_z, empty_z, drained[2];
};

struct ScanArgs {
    const unsigned char *rec;
    float *S;
    long long S_stride;
    const void *z;
    void *out;
    const float *norm_w;
    int nk, nv, head_map, T, n_chunks;
    int c_begin, c_count, rec_chunks;    // the chunks one launch of the sequential form scans (a slab of the prompt); records per head
    float out_scale, eps;
    // Segment-parallel form (n_seg > 1; for few heads): the prompt is cut into n_seg runs of seg_chunks chunks that
    // are scanned at the same time by different CTAs (grid.z = 2 n_seg - 1).  The state enters the recurrence
    // linearly, S_t = S_{t-1} M_t + beta_t v_t k_t^T with M_t = alpha_t (I - beta_t k_t k_t^T) acting on the key
    // index, so a run needs the incoming state only through two things that do not depend on it: the scan of
    // the run from a ZERO state (outputs o0_t, final state S0) and the scan of the run from the IDENTITY with
    // V = 0 (outputs qt_t = Phi_t q_t, final state Phi = prod M_t).  Then o_t = o0_t + S_in qt_t and
    // S_out = S_in Phi + S0; k_delta_seg_carry walks the runs, k_delta_seg_finish adds the correction and
    // applies the output norm and gate.  Run 0 starts from the real state and is final as it is.
    int n_seg, seg_chunks;
    float *seg_state;                    // [n_seq * nv][3 n_seg][128][128]: slot 3j: S0 (j = 0: end state of run 0), 3j+1: Phi, 3j+2: S_in
    float *seg_raw;                      // [2][n_seq * nv][T][128] f32: o0, then qt
    unsigned int *status;
};

// MN-major tf32 operand: rows of 128 bytes along N, groups of 4 k, 32-byte swizzle atoms
// (the only shared-memory layout the tensor core accepts for a transposed 32-bit operand)
__device__ __forceinline__ uint64_t smem_desc_mn32(uint32_t saddr, uint32_t lbo, uint32_t sbo) {
    return (uint64_t)((saddr >> 4) & 0x3FFF) | ((uint64_t)((lbo >> 4) & 0x3FFF) << 16) |
           ((uint64_t)((sbo >> 4) & 0x3FFF) << 32) | ((uint64_t)1 << 46) | ((uint64_t)1 << 61);
}

__device__ __forceinline__ void ld_row32(const float *p, float (&r)[32]) {
#pragma unroll
    for (int i = 0; i < 8; i++) {
        const float4 v = *reinterpret_cast<const float4 *>(p + 4 * i);
        r[4 * i] = v.x; r[4 * i + 1] = v.y; r[4 * i + 2] = v.z; r[4 * i + 3] = v.w;
    }
}

// activation loads whose conversion happens at the point of use (a converted copy made at load time would
// double the registers a batch of loads in flight occupies)
__device__ __forceinline__ uint32_t ld_raw(const float *p, size_t i) { return __float_as_uint(p[i]); }
__device__ __forceinline__ uint32_t ld_raw(const __nv_bfloat16 *p, size_t i) { return reinterpret_cast<const unsigned short *>(p)[i]; }
__device__ __forceinline__ float cvt_raw(const float *, uint32_t r) { return __uint_as_float(r); }
__device__ __forceinline__ float cvt_raw(const __nv_bfloat16 *, uint32_t r) { return __uint_as_float(r << 16); }

// Lanes give up each for itself, by its own reading of the clock, and those that stayed in a loop would miss the others at the warp's next
// collective instruction.  So a chain warp goes on without waiting when a wait gave up, and passes nothing on; an output warp
// leaves with all its lanes.  Votes at the chain's waits took 1.5 %.
__device__ __forceinline__ bool all_lanes(bool ok) { return __all_sync(0xffffffffu, ok); }
// this thread's stores to shared memory, seen by the tensor copy a thread issues after a barrier
__device__ __forceinline__ void fence_async() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }

// four 8 x 8 matrices of 16-bit values, transposed: lane l names row l & 7 of matrix l >> 3 and holds of each the rows 2 (l & 3), + 1 at
// column l >> 2
__device__ __forceinline__ void ldmatrix_x4_trans(uint32_t (&r)[4], uint32_t addr) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0, %1, %2, %3}, [%4];" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr) : "memory");
}
__device__ __forceinline__ void stmatrix_x4_trans(uint32_t addr, const uint32_t (&r)[4]) {
    asm volatile("stmatrix.sync.aligned.m8n8.x4.trans.shared.b16 [%0], {%1, %2, %3, %4};" ::"r"(addr), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]) : "memory");
}

template <typename ACT, bool SEG, bool TILE>
__global__ void __launch_bounds__(NTHREADS, 1) k_delta_scan_tc5(const __grid_constant__ CUtensorMap map_y,
                                                               const __grid_constant__ CUtensorMap map_ym,
                                                               const __grid_constant__ CUtensorMap map_v,
                                                               const __grid_constant__ CUtensorMap map_z,
                                                               const __grid_constant__ CUtensorMap map_o, ScanArgs a) {
    extern __shared__ unsigned char smraw[];
    __shared__ ScanBars bars;
    __shared__ __align__(16) float red[2][4][16][4];                    // [chunk parity][group of 16 tokens][token][lane quarter]
    __shared__ uint32_t tmem_slot;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int hv = blockIdx.x, b = blockIdx.y;
    // what this CTA scans: kind 0 = from the caller's state, final outputs; 1 = from zero, raw outputs;
    // 2 = from the identity with V = 0, raw outputs
    int kind = 0, seg = 0;
    if (SEG && blockIdx.z > 0) { seg = 1 + ((int)blockIdx.z - 1) / 2; kind = 1 + ((int)blockIdx.z - 1) % 2; }
    const int c0 = SEG ? seg * a.seg_chunks : a.c_begin;                       // first chunk
    const int N = SEG ? min(a.seg_chunks, a.n_chunks - c0) : a.c_count;        // chunks of this CTA
    const int kh = a.head_map == ORNITH_HEADMAP_GROUPED ? hv / (a.nv / a.nk) : hv % a.nk;
    const int qd = a.nk * 128, vd = a.nv * 128;
    const uint32_t base = (su32(smraw) + 1023u) & ~1023u; // swizzle atoms are 1 KiB aligned
    unsigned char *gbase = smraw + (base - su32(smraw));

    if (tid == 0) {
        for (int s = 0; s < NBUF; s++) { mbar_init(su32(&bars.full[s]), 1); mbar_init(su32(&bars.empty[s]), s == B_V ? 8 : 1); }
        for (int s = 0; s < NFAC; s++) mbar_init(su32(&bars.full_f[s]), 1);
        for (int s = 0; s < 2; s++)
            for (int g = 0; g < 4; g++) mbar_init(su32(&bars.red[s][g]), 4);
        for (int g = 0; g < 4; g++) { mbar_init(su32(&bars.o_full[g]), 4); mbar_init(su32(&bars.o_free[g]), 1); }
        mbar_init(su32(&bars.ks_done), 1); mbar_init(su32(&bars.t_ready), 8); mbar_init(su32(&bars.u_done), 1);
        mbar_init(su32(&bars.wu_ready), 8); mbar_init(su32(&bars.u_ready), 8); mbar_init(su32(&bars.s_done), 1);
        mbar_init(su32(&bars.pu_done), 1); mbar_init(su32(&bars.qs_done), 1); mbar_init(su32(&bars.o_read), 16);
        for (int s = 0; s < 2; s++) mbar_init(su32(&bars.drained[s]), 1);
        mbar_init(su32(&bars.full_z), 1); mbar_init(su32(&bars.empty_z), 16);
        mbar_init_fence();
    }
    if (warp == W_MMA) tmem_alloc(&tmem_slot, TM_COLS);
    if (tid < 256)                                        // rows 0..31, columns 32..63 of A
        *reinterpret_cast<float4 *>(gbase + SM_A + 8192 + tid * 16) = make_float4(0.f, 0.f, 0.f, 0.f);
    fence_async();
    fence_before();
    __syncthreads();
    fence_after();
    const uint32_t tmem = tmem_slot;
    float *Sg = a.S + (size_t)b * a.S_stride + (size_t)hv * 128 * 128;     // incoming state (kind 0)
    float *Sout = Sg;                                                       // where the final state goes
    float *raw = nullptr;                                                   // raw output rows [T][128] (kinds 1, 2)
    if (SEG) {
        Sout = a.seg_state + (((size_t)b * a.nv + hv) * 3 * a.n_seg + 3 * seg + (kind == 2 ? 1 : 0)) * (128 * 128);
        if (kind) raw = a.seg_raw + ((size_t)(kind - 1) * gridDim.y * a.nv + (size_t)b * a.nv + hv) * (size_t)a.T * 128;
    }
    // lane quarter and token (column) half of a chain thread
    const int qtr = warp & 3, half = (warp >> 2) & 1, row = 32 * qtr + lane;
    const uint32_t lane_t = tmem + ((uint32_t)(32 * qtr) << 16);

    if (warp < 8) {                                       // the state goes to tensor memory: S[r][c] in lane r, column c
#pragma unroll 1
        for (int cc = 0; cc < 2; cc++) {
            float s[32];
            if (kind == 0) ld_row32(Sg + (size_t)row * 128 + 64 * half + 32 * cc, s);
            else {
#pragma unroll
                for (int i = 0; i < 32; i++) s[i] = (SEG && kind == 2 && 64 * half + 32 * cc + i == row) ? 1.0f : 0.0f;
            }
            tmem_st32(lane_t + TM_S + 64 * half + 32 * cc, s);
        }
        tmem_wait_st();
    }
    fence_before();
    __syncthreads();
    bool ok = true;

    constexpr int TZ = (int)sizeof(ACT), CZ = 128 / TZ;   // tiles of z: their number, their channels
    const bool tiles = TILE && !(SEG && kind);            // z and the outputs by tensor copies
    const unsigned char *rec0 = a.rec + (((size_t)b * a.nv + hv) * a.rec_chunks + (SEG ? c0 : 0)) * (size_t)REC_BYTES;
    auto l2_rows = [&](const CUtensorMap *map, int x, int t) {
        asm volatile("cp.async.bulk.prefetch.tensor.3d.L2.global.tile [%0, {%1, %2, %3}];" ::"l"(map), "r"(x), "r"(t), "r"(b) : "memory");
    };
    auto ahead = [&](int n) {                                     // (K and Q rows are shared by the value heads of a key head)
        if (n >= N) return;
        asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(rec0 + (size_t)n * REC_BYTES), "r"((uint32_t)REC_BYTES) : "memory");
        l2_rows(&map_v, 2 * qd + hv * 128, (c0 + n) * C);
        if (tiles)
            for (int t = 0; t < TZ; t++) l2_rows(&map_z, hv * 128 + t * CZ, (c0 + n) * C);
    };

    if (warp == W_TMA) {
        // ================= producer =================
        if (elect_one()) {
            asm volatile("griddepcontrol.wait;\n" ::: "memory");     // everything that comes through here is written by the kernels in front
            int announced = 0, factors = 0;
            if (!tiles) ahead(1);
            for (int n = 0; n < N && ok; n++) {
                if (!tiles) ahead(n + 2);                                 // (behind the waits of the chunk before)
                const unsigned char *r = rec0 + (size_t)n * REC_BYTES;
                const int t0 = (c0 + n) * C;                              // (rows past the sequence's last token arrive as zeros)
                auto refill = [&](int s, uint32_t bytes) {                // the buffer is free: its next contents are announced
                    if (n >= 1) ok = ok && mbar_wait_parked(su32(&bars.empty[s]), (uint32_t)(n - 1) & 1u);
                    if (ok) { mbar_expect_tx(su32(&bars.full[s]), bytes); announced++; }
                    return ok;
                };
                auto rows = [&](int dst, const CUtensorMap *map, int x, int s) {
                    for (int sl = 0; sl < 4; sl++) tma_load_3d(base + dst + sl * 8192, map, x + 32 * sl, t0, b, su32(&bars.full[s]));
                };
                auto part = [&](int dst, int off, uint32_t bytes, int s) { bulk_load(base + dst, r + off, bytes, su32(&bars.full[s])); };
                if (!refill(B_K, 32768u)) break;
                rows(SM_K, &map_y, qd + kh * 128, B_K);
                // (the readers of the factors of chunk n - 4 are done: K S^T of chunk n - 1 was behind them)
                mbar_expect_tx(su32(&bars.full_f[n % NFAC]), FAC_BYTES);
                bulk_load(base + SM_F + n % NFAC * FAC_BYTES, r + REC_F, FAC_BYTES, su32(&bars.full_f[n % NFAC]));
                factors++;
                if (!refill(B_V, 32768u)) break;
                tma_load_3d(base + SM_V, &map_v, 2 * qd + hv * 128, t0, b, su32(&bars.full[B_V]));
                if (!refill(B_A, TRI_BYTES)) break;
                part(SM_A, REC_A, 8192u, B_A);
                part(SM_A + 8192 + 4096, REC_A + 8192, 4096u, B_A);
                if (!refill(B_Q, 32768u)) break;
                rows(SM_Q, &map_y, kh * 128, B_Q);
                if (!refill(B_KM, 32768u)) break;
                rows(SM_KM, &map_ym, qd + kh * 128, B_KM);
                if (!refill(B_P, TRI_BYTES)) break;
                part(SM_P, REC_P, TRI_BYTES, B_P);
            }
            if (!ok) {                                                    // the copies asked for land before the CTA goes
                for (int s = 0; s < NBUF && s < announced; s++) (void)mbar_wait(su32(&bars.full[s]), (uint32_t)((announced + NBUF - 1 - s) / NBUF - 1) & 1u);
                for (int s = 0; s < NFAC && s < factors; s++) (void)mbar_wait(su32(&bars.full_f[s]), (uint32_t)((factors + NFAC - 1 - s) / NFAC - 1) & 1u);
            }
        }
    } else if (warp == W_MMA) {
        // ================= every tcgen05.mma =================
        if (elect_one()) {
            constexpr uint32_t ID_64 = idesc(2, 64, false), ID_SU = idesc(2, 128, true);
            auto full = [&](int s, int n) { return mbar_wait(su32(&bars.full[s]), (uint32_t)n & 1u); };
            auto empty = [&](int s) { mma_commit(su32(&bars.empty[s])); };
            auto times_state = [&](uint32_t d, uint32_t S, uint32_t tile) {       // D[dv][token] = sum_dk S[dv][dk] tile[token][dk]
#pragma unroll
                for (int ks = 0; ks < 16; ks++) mma_tf32_ts(d, S + 8 * ks, smem_desc(tile + (ks >> 2) * 8192 + (ks & 3) * 32, 16, 1024), ID_64, ks > 0);
            };
            // what a product needs beside the result it follows is waited for ahead of that result
            for (int n = 0; n < N; n++) {
                const uint32_t S = tmem + TM_S + 128 * (n & 1), S2 = tmem + TM_S + 128 * ((n & 1) ^ 1);
                ok = full(B_K, n) && (n == 0 || mbar_wait(su32(&bars.s_done), (uint32_t)(n - 1) & 1u));
                if (!ok) break;
                fence_after();
                times_state(tmem + TM_X, S, base + SM_K);                         // (K S^T)^T
                mma_commit(su32(&bars.ks_done));
                empty(B_K);
                // U^T = T^T A^T; U of the chunk before is an operand no more
                ok = full(B_A, n) && (n == 0 || mbar_wait(su32(&bars.pu_done), (uint32_t)(n - 1) & 1u)) && mbar_wait(su32(&bars.t_ready), (uint32_t)n & 1u);
                if (!ok) break;
                fence_after();
#pragma unroll
                for (int ks = 0; ks < 8; ks++)
                    mma_tf32_ts(tmem + TM_U, tmem + TM_X + 8 * ks, smem_desc(base + SM_A + (ks >> 2) * 8192 + (ks & 3) * 32, 16, 1024), ID_64, ks > 0);
                mma_commit(su32(&bars.u_done));
                empty(B_A);
                // the tiles Q S^T and P U of the chunk before have been read
                ok = full(B_Q, n) && (n == 0 || mbar_wait(su32(&bars.o_read), (uint32_t)(n - 1) & 1u));
                if (!ok) break;
                fence_after();
                times_state(tmem + TM_QS, S, base + SM_Q);                        // (Q S^T)^T, while the chain warps work on U
                mma_commit(su32(&bars.qs_done));
                empty(B_Q);
                ok = full(B_KM, n) && mbar_wait(su32(&bars.wu_ready), (uint32_t)n & 1u);
                if (!ok) break;
                fence_after();
#pragma unroll
                for (int ks = 0; ks < 8; ks++)            // S' += (w rk U)^T K, the K tile read MN-major
                    mma_tf32_ts(S2, tmem + TM_X + 8 * ks, smem_desc_mn32(base + SM_KM + ks * 1024, 8192, 512), ID_SU, 1u);
                mma_commit(su32(&bars.s_done));
                empty(B_KM);
            }
            if (!ok) {                                                    // nothing may be multiplied when the tensor memory goes back
                mma_commit(su32(&bars.drained[0]));
                (void)mbar_wait(su32(&bars.drained[0]), 0u);
            }
        }
    } else if (warp == W_PU) {
        // ================= (P U)^T =================
        // P is lower triangular (layout: tri_at), rows 0..31 need tokens j < 32 only
        if (elect_one()) {
            constexpr uint32_t ID_32 = idesc(2, 32, false);
            for (int n = 0; n < N; n++) {
                ok = mbar_wait_parked(su32(&bars.full[B_P]), (uint32_t)n & 1u) && (n == 0 || mbar_wait_parked(su32(&bars.o_read), (uint32_t)(n - 1) & 1u)) &&
                     mbar_wait_parked(su32(&bars.u_ready), (uint32_t)n & 1u);
                if (!ok) break;
                fence_after();
#pragma unroll
                for (int ks = 0; ks < 4; ks++) mma_tf32_ts(tmem + TM_PU, tmem + TM_U + 8 * ks, smem_desc(base + SM_P + ks * 32, 16, 1024), ID_32, ks > 0);
#pragma unroll
                for (int ks = 0; ks < 8; ks++)
                    mma_tf32_ts(tmem + TM_PU + 32, tmem + TM_U + 8 * ks,
                                smem_desc(base + SM_P + (ks < 4 ? 4096 + ks * 32 : 8192 + (ks - 4) * 32), 16, 1024), ID_32, ks > 0);
                mma_commit(su32(&bars.pu_done));
                mma_commit(su32(&bars.empty[B_P]));
            }
            if (!ok) {
                mma_commit(su32(&bars.drained[1]));
                (void)mbar_wait(su32(&bars.drained[1]), 0u);
            }
        }
    } else if (warp < 8) {
        // ================= chain: T, the decayed state, U =================
        const uint32_t X = lane_t + TM_X + 32 * half, U = lane_t + TM_U + 32 * half;
        const float *bv = reinterpret_cast<const float *>(gbase + SM_V) + 32 * half * 128 + row;     // beta V of token 32 half + i: bv[128 i]
        const float quiet_nan = __int_as_float(0x7fc00000);              // (as tf32, too)
        for (int n = 0; n < N; n++) {
            const float *fac = reinterpret_cast<const float *>(gbase + SM_F + (n % NFAC) * FAC_BYTES);
            const uint32_t S = lane_t + TM_S + 128 * (n & 1) + 64 * half, S2 = lane_t + TM_S + 128 * ((n & 1) ^ 1) + 64 * half;
            ok = ok && mbar_wait(su32(&bars.full_f[n % NFAC]), (uint32_t)(n / NFAC) & 1u) && (n == 0 || mbar_wait(su32(&bars.s_done), (uint32_t)(n - 1) & 1u));
            fence_after();
            float x[32], v[32];
            // the other state = p_63 S, while the tensor core reads S (the update is accumulated onto it): a half beside K S^T, a half
            // beside A T
            const float pend = fac[F_PEND];
            auto decay = [&](int cc) {
                const f32x2 p2 = pack2(pend, pend);
                tmem_ld32_wait(S + 32 * cc, x);
#pragma unroll
                for (int i = 0; i < 32; i += 2) { const f32x2 y = mul2(p2, pack2(x[i], x[i + 1])); unpack2(y, &x[i], &x[i + 1]); }
                tmem_st32(S2 + 32 * cc, x);
            };
            decay(0);
            ok = ok && mbar_wait(su32(&bars.full[B_V]), (uint32_t)n & 1u);
#pragma unroll
            for (int i = 0; i < 32; i++) v[i] = SEG && kind == 2 ? 0.0f : bv[128 * i];
            // A beta v or a factor that is no finite number makes this row's U NaN.  The roundings below would hide it (-0 for NaN, see
            // tf32q; a minimum for each of the 96 took 4 % of the prefill), so it is looked for here, beside K S^T, and written
            // below.  What is no number in the state or in A shows in Q S^T or in P U anyway.
            bool bad = __any_sync(0xffffffffu, 0.0f * fac[F_BPK + 32 * half + lane] != 0.0f);
            {
                f32x2 z = 0;
                float z0, z1;
#pragma unroll
                for (int i = 0; i < 32; i += 2) z = fma2(pack2(v[i], v[i + 1]), 0, z);
                unpack2(z, &z0, &z1);
                bad = bad || z0 + z1 != 0.0f;
            }
            ok = ok && mbar_wait(su32(&bars.ks_done), (uint32_t)n & 1u);
            fence_after();
            tmem_ld32_wait(X, x);                                        // (K S^T)^T
#pragma unroll
            for (int i = 0; i < 32; i += 4) {                            // T^T over it
                const float4 b4 = *reinterpret_cast<const float4 *>(fac + F_BPK + 32 * half + i);    // -beta p rk
                unpack2(fma2(pack2(b4.x, b4.y), pack2(x[i], x[i + 1]), pack2(v[i], v[i + 1])), &x[i], &x[i + 1]);
                unpack2(fma2(pack2(b4.z, b4.w), pack2(x[i + 2], x[i + 3]), pack2(v[i + 2], v[i + 3])), &x[i + 2], &x[i + 3]);
            }
#pragma unroll
            for (int i = 0; i < 32; i++) x[i] = tf32q_finite(x[i]);
            tmem_st32(X, x);
            tmem_wait_st();
            fence_before();
            if (all_lanes(ok) && lane == 0) { mbar_arrive(su32(&bars.t_ready)); mbar_arrive(su32(&bars.empty[B_V])); }
            decay(1);
            ok = ok && mbar_wait(su32(&bars.u_done), (uint32_t)n & 1u);
            fence_after();
            tmem_ld32_wait(U, x);                                        // U^T
            // (w rk U)^T over T^T first: the state update waits for it
#pragma unroll
            for (int hh = 0; hh < 4; hh++) {                             // 8 tokens at a time
                float f[8];
#pragma unroll
                for (int i = 0; i < 2; i++) {
                    const float4 w4 = *reinterpret_cast<const float4 *>(fac + F_W + 32 * half + 8 * hh + 4 * i);   // w rk
                    const float *t = x + 8 * hh + 4 * i;
                    const f32x2 t0 = mul2(pack2(w4.x, w4.y), pack2(t[0], t[1])), t1 = mul2(pack2(w4.z, w4.w), pack2(t[2], t[3]));
                    unpack2(t0, f + 4 * i, f + 4 * i + 1);
                    unpack2(t1, f + 4 * i + 2, f + 4 * i + 3);
                }
#pragma unroll
                for (int i = 0; i < 8; i++) f[i] = tf32q_finite(f[i]);
                if (hh == 0 && bad) f[0] = quiet_nan;
                tmem_st8(X + 8 * hh, f);
            }
            tmem_wait_st();
            fence_before();
            if (all_lanes(ok) && lane == 0) mbar_arrive(su32(&bars.wu_ready));
#pragma unroll
            for (int i = 0; i < 32; i++) x[i] = tf32q_finite(x[i]);
            if (bad) x[0] = quiet_nan;
            tmem_st32(U, x);                                             // tf32 U^T over the accumulator
            tmem_wait_st();
            fence_before();
            if (all_lanes(ok) && lane == 0) mbar_arrive(su32(&bars.u_ready));
        }
        ok = ok && mbar_wait(su32(&bars.s_done), (uint32_t)(N - 1) & 1u);
        fence_after();
#pragma unroll 1
        for (int cc = 0; cc < 2; cc++) {                                 // the state goes home
            float x[32];
            tmem_ld32_wait(lane_t + TM_S + 128 * (N & 1) + 64 * half + 32 * cc, x);
            float4 *dst = reinterpret_cast<float4 *>(Sout + (size_t)row * 128 + 64 * half + 32 * cc);
#pragma unroll
            for (int i = 0; i < 8; i++)
                dst[i] = ok ? make_float4(x[4 * i], x[4 * i + 1], x[4 * i + 2], x[4 * i + 3]) : make_float4(NAN, NAN, NAN, NAN);
        }
    } else if (warp < W_TMA) {
        // ================= output =================
        // 16 warps: lane quarter qtr, group grp of 16 tokens.  A thread (g, j) has the rows 8 k + g of the quarter (k = 0..3) and the
        // tokens 8 m + 2 j + c of the group (m, c = 0, 1): value 8 m + 2 k + c
        constexpr bool TILE_O = TILE && sizeof(ACT) == 2;
        const int grp = (warp - 8) >> 2, g = lane >> 2, j = lane & 3;
        float nw[4];
#pragma unroll
        for (int k = 0; k < 4; k++) nw[k] = a.norm_w[32 * qtr + 8 * k + g];
        const ACT *zp = (const ACT *)a.z;
        ACT *op = (ACT *)a.out;
        const size_t gofs = ((size_t)b * a.T + 2 * j) * vd + (size_t)hv * 128 + 32 * qtr + g;       // + (token of the group's first) vd + 8 k + ..
        const uint32_t t_qs = lane_t + TM_QS + 16 * grp, t_pu = lane_t + TM_PU + 16 * grp;
        // z and the outputs in shared memory: rows of 128 bytes per token, 128-byte swizzle, 64 (bf16) or 32 (f32) channels to a
        // tile of 8 KiB: the 16-byte pieces of a row change places by its number modulo 8.  bf16: the address of the 8 x 8 matrix row
        // this lane names (matrix lane >> 3 = channels 8 (lane >> 3) .., row = token lane & 7); f32: this thread's element, k = c = 0
        const uint32_t zoff = sizeof(ACT) == 2
            ? (qtr >> 1) * 8192 + (16 * grp + (lane & 7)) * 128 + (((4 * (qtr & 1) + (lane >> 3)) ^ (lane & 7)) * 16)
            : qtr * 8192 + (16 * grp + 2 * j) * 128 + ((g >> 2) ^ (2 * j)) * 16 + (g & 3) * 4;
        int n = 0;
        for (; n < N; n++) {
            const int s = n & 1, tok = (c0 + n) * C + 16 * grp;
            float zr[16];
            if (!(SEG && kind)) {
                // the gate factors of this chunk, while the tensor core still works on it: norm weight x SiLU(z)
                if (TILE) {
                    ok = mbar_wait_parked(su32(&bars.full_z), (uint32_t)n & 1u);
#pragma unroll
                    for (int m = 0; m < 2; m++) {
                        if (sizeof(ACT) == 2) {
                            uint32_t r[4];
                            ldmatrix_x4_trans(r, base + SM_Z + zoff + m * 1024);
#pragma unroll
                            for (int k = 0; k < 4; k++) { zr[8 * m + 2 * k] = __uint_as_float(r[k] << 16); zr[8 * m + 2 * k + 1] = __uint_as_float(r[k] & 0xFFFF0000u); }
                        } else {
#pragma unroll
                            for (int i = 0; i < 8; i++)
                                zr[8 * m + i] = *reinterpret_cast<const float *>(gbase + SM_Z + ((zoff ^ ((i >> 1) * 32)) ^ ((i & 1) * 16)) + (i & 1) * 128 + m * 1024);
                        }
                    }
                    __syncwarp();
                    if (lane == 0) mbar_arrive(su32(&bars.empty_z));
                } else {
#pragma unroll
                    for (int i = 0; i < 16; i++) {
                        const int k = (i >> 1) & 3, t = tok + 8 * (i >> 3) + (i & 1);
                        zr[i] = t + 2 * j < a.T ? cvt_raw(zp, ld_raw(zp, gofs + (size_t)t * vd + 8 * k)) : 0.0f;
                    }
                }
#pragma unroll
                for (int i = 0; i < 16; i += 2) {
                    const f32x2 z2 = pack2(zr[i], zr[i + 1]), e2 = mul2(z2, pack2(-LOG2E_F, -LOG2E_F));
                    float e0, e1;
                    unpack2(e2, &e0, &e1);
                    unpack2(add2(pack2(ex2_fast(e0), ex2_fast(e1)), pack2(1.0f, 1.0f)), &e0, &e1);
                    const float w = nw[(i >> 1) & 3];
                    unpack2(mul2(mul2(z2, pack2(w, w)), pack2(rcp_fast(e0), rcp_fast(e1))), &zr[i], &zr[i + 1]);
                }
            }
            ok = all_lanes(ok && mbar_wait_parked(su32(&bars.full_f[n % NFAC]), (uint32_t)(n / NFAC) & 1u) && mbar_wait_parked(su32(&bars.qs_done), (uint32_t)n & 1u) &&
                           mbar_wait_parked(su32(&bars.pu_done), (uint32_t)n & 1u));
            if (!ok) break;
            fence_after();
            float x[16];                                                 // O = p rq QS + P U
            {
                const float *pq = reinterpret_cast<const float *>(gbase + SM_F + (n % NFAC) * FAC_BYTES) + F_PQ + 16 * grp + 2 * j;
                float q[16];
                tmem_ld_16x256_wait(t_qs, q, t_pu, x);
                const float2 pa = *reinterpret_cast<const float2 *>(pq), pb = *reinterpret_cast<const float2 *>(pq + 8);
                const f32x2 p2[2] = {pack2(pa.x, pa.y), pack2(pb.x, pb.y)};
#pragma unroll
                for (int i = 0; i < 16; i += 2) unpack2(fma2(p2[i >> 3], pack2(q[i], q[i + 1]), pack2(x[i], x[i + 1])), &x[i], &x[i + 1]);
            }
            fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(su32(&bars.o_read));              // the tensor core may overwrite both tiles
            if (SEG && kind) {                                           // raw outputs of a run scanned from zero / from the identity: no norm, no gate
#pragma unroll
                for (int i = 0; i < 16; i++) {
                    const int k = (i >> 1) & 3, t = tok + 8 * (i >> 3) + 2 * j + (i & 1);
                    if (t < a.T) raw[(size_t)t * 128 + 32 * qtr + 8 * k + g] = x[i];
                }
                continue;
            }
            {
                // sum of squares: over the thread's rows, then over the 8 lanes of a j; lane (bit 4 = m, bit 3 = c, j) ends up with token
                // 8 m + 2 j + c of the group
                f32x2 s0 = 0, s1 = 0;
#pragma unroll
                for (int k = 0; k < 4; k++) {
                    const f32x2 a0 = pack2(x[2 * k], x[2 * k + 1]), a1 = pack2(x[8 + 2 * k], x[8 + 2 * k + 1]);
                    s0 = fma2(a0, a0, s0);
                    s1 = fma2(a1, a1, s1);
                }
                float v00, v01, v10, v11;
                unpack2(s0, &v00, &v01);
                unpack2(s1, &v10, &v11);
                const bool hm = lane & 16, hc = lane & 8;
                float a0 = hm ? v10 : v00, a1 = hm ? v11 : v01;
                a0 += __shfl_xor_sync(0xffffffffu, hm ? v00 : v10, 16);
                a1 += __shfl_xor_sync(0xffffffffu, hm ? v01 : v11, 16);
                float b0 = hc ? a1 : a0;
                b0 += __shfl_xor_sync(0xffffffffu, hc ? a0 : a1, 8);
                b0 += __shfl_xor_sync(0xffffffffu, b0, 4);
                if ((lane & 4) == 0) red[s][grp][8 * (lane >> 4) + 2 * j + ((lane >> 3) & 1)][qtr] = b0;
            }
            __syncwarp();
            if (lane == 0) mbar_arrive(su32(&bars.red[s][grp]));
            if (TILE_O && n >= 1) ok = mbar_wait_parked(su32(&bars.o_free[grp]), (uint32_t)(n - 1) & 1u);      // the group's rows of the chunk before have left
            ok = all_lanes(ok && mbar_wait_parked(su32(&bars.red[s][grp]), (uint32_t)(n >> 1) & 1u));
            if (!ok) break;
            const float4 r4 = *reinterpret_cast<const float4 *>(&red[s][grp][8 * (lane >> 4) + 2 * j + ((lane >> 3) & 1)][0]);
            const float ss = a.out_scale * a.out_scale * ((r4.x + r4.y) + (r4.z + r4.w));
            const float inv = rsqrtf(ss * (1.0f / 128.0f) + a.eps) * a.out_scale;   // of this lane's token
            f32x2 i2[2];
#pragma unroll
            for (int m = 0; m < 2; m++) i2[m] = pack2(__shfl_sync(0xffffffffu, inv, 16 * m + j), __shfl_sync(0xffffffffu, inv, 16 * m + 8 + j));
#pragma unroll
            for (int i = 0; i < 16; i += 2) unpack2(mul2(mul2(pack2(x[i], x[i + 1]), i2[i >> 3]), pack2(zr[i], zr[i + 1])), &x[i], &x[i + 1]);
            if (TILE_O) {
#pragma unroll
                for (int m = 0; m < 2; m++) {
                    uint32_t r[4];
#pragma unroll
                    for (int k = 0; k < 4; k++) {
                        const __nv_bfloat162 o2 = __floats2bfloat162_rn(x[8 * m + 2 * k], x[8 * m + 2 * k + 1]);
                        r[k] = *reinterpret_cast<const uint32_t *>(&o2);
                    }
                    stmatrix_x4_trans(base + SM_O + zoff + m * 1024, r);
                }
                fence_async();
                __syncwarp();
                if (lane == 0) mbar_arrive(su32(&bars.o_full[grp]));
            } else {
#pragma unroll
                for (int i = 0; i < 16; i++) {
                    const int k = (i >> 1) & 3, t = tok + 8 * (i >> 3) + (i & 1);
                    if (t + 2 * j < a.T) act_st(op, gofs + (size_t)t * vd + 8 * k, x[i]);
                }
            }
        }
        for (; n < N && !(SEG && kind); n++) {                           // a wait gave up: poison what was not written
            const int tok = (c0 + n) * C + 16 * grp;
            for (int i = 0; i < 16; i++) {
                const int kk = (i >> 1) & 3, t = tok + 8 * (i >> 3) + (i & 1);
                if (t + 2 * j < a.T) act_st(op, gofs + (size_t)t * vd + 8 * kk, NAN);
            }
        }
    }
    if (warp == W_IO) {
        // ================= z, outputs, L2 =================
        if (tiles && elect_one()) {
            asm volatile("griddepcontrol.wait;\n" ::: "memory");
            auto load_z = [&](int n) {
                mbar_expect_tx(su32(&bars.full_z), (uint32_t)(C * 128 * TZ));
                for (int t = 0; t < TZ; t++)
                    tma_load_3d(base + SM_Z + t * 8192, &map_z, hv * 128 + t * CZ, (c0 + n) * C, b, su32(&bars.full_z));
            };
            ahead(1);
            load_z(0);
            int loads = 1;
            for (int n = 0; n < N && ok; n++) {
                ahead(n + 2);
                ok = mbar_wait_parked(su32(&bars.empty_z), (uint32_t)n & 1u);
                if (ok && n + 1 < N) { load_z(n + 1); loads++; }
                if (TZ == 2 && ok) {
                    for (int g = 0; g < 4 && ok; g++) {
                        ok = mbar_wait_parked(su32(&bars.o_full[g]), (uint32_t)n & 1u);
                        const int tok = (c0 + n) * C + 16 * g;
                        if (ok && tok < a.T) {                           // (rows past T are left out by the copy)
#pragma unroll
                            for (int hf = 0; hf < 2; hf++)
                                asm volatile("cp.async.bulk.tensor.3d.global.shared::cta.tile.bulk_group [%0, {%2, %3, %4}], [%1];"
                                             ::"l"(&map_o), "r"(base + SM_O + hf * 8192 + g * 2048), "r"(hv * 128 + hf * 64), "r"(tok), "r"(b) : "memory");
                        }
                        asm volatile("cp.async.bulk.commit_group;" ::: "memory");
                    }
                    asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory");
                    for (int g = 0; g < 4; g++) mbar_arrive(su32(&bars.o_free[g]));
                }
            }
            if (!ok) (void)mbar_wait(su32(&bars.full_z), (uint32_t)(loads - 1) & 1u);
            asm volatile("cp.async.bulk.wait_group 0;" ::: "memory");    // shared memory outlives the copies
        }
    }
    if (!ok) report_timeout(a.status, ORN_WAIT_DELTA_SCAN);
    fence_before();
    __syncthreads();
    if (warp == W_MMA) tmem_dealloc(tmem, TM_COLS);
}


// =============================================================================
// segment-parallel form: carrying the state over the runs, and the finishing pass
// =============================================================================
// S_in of run j+1 = S_in of run j x Phi_j + S0_j, rows of the state independent of one another: one CTA per
// (sequence, head, group of 8 rows), 128 threads = the 128 columns.  Leaves S_in of every run j >= 1 in its slot
// of seg_state and the final state in the caller's S.
__global__ void __launch_bounds__(128) k_delta_seg_carry(ScanArgs a) {
    __shared__ float srow[8][128];
    __shared__ __align__(16) float phi[32][128];                                  // 32 rows of Phi at a time
    const int hv = blockIdx.x, b = blockIdx.y, r0 = 8 * blockIdx.z, c = threadIdx.x;
    float *slots = a.seg_state + ((size_t)b * a.nv + hv) * 3 * a.n_seg * (128 * 128);
    float s[8];
#pragma unroll
    for (int r = 0; r < 8; r++) s[r] = slots[(size_t)(r0 + r) * 128 + c];          // end state of run 0
    for (int j = 1; j < a.n_seg; j++) {
        const float *S0 = slots + (size_t)(3 * j) * (128 * 128), *Phi = S0 + 128 * 128;
        float *Sin = slots + (size_t)(3 * j + 2) * (128 * 128);
        float acc[8];
#pragma unroll
        for (int r = 0; r < 8; r++) { Sin[(size_t)(r0 + r) * 128 + c] = s[r]; srow[r][c] = s[r]; acc[r] = S0[(size_t)(r0 + r) * 128 + c]; }
        for (int l0 = 0; l0 < 128; l0 += 32) {
            __syncthreads();                                                      // srow written / phi free again
            float4 v[8];
#pragma unroll
            for (int i = 0; i < 8; i++) v[i] = reinterpret_cast<const float4 *>(Phi + (size_t)l0 * 128)[i * 128 + c];
#pragma unroll
            for (int i = 0; i < 8; i++) reinterpret_cast<float4 *>(&phi[0][0])[i * 128 + c] = v[i];
            __syncthreads();
#pragma unroll 8
            for (int l = 0; l < 32; l++) {
                const float p = phi[l][c];
#pragma unroll
                for (int r = 0; r < 8; r++) acc[r] = fmaf(srow[r][l0 + l], p, acc[r]);
            }
        }
        __syncthreads();
#pragma unroll
        for (int r = 0; r < 8; r++) s[r] = acc[r];
    }
    float *Sg = a.S + (size_t)b * a.S_stride + (size_t)hv * 128 * 128;
#pragma unroll
    for (int r = 0; r < 8; r++) Sg[(size_t)(r0 + r) * 128 + c] = s[r];
}

// o_t = o0_t + S_in qt_t for the tokens of the runs j >= 1, then the output scale, the per-head RMSNorm and the
// SiLU(z) gate (reference: linear_finish, src/ornith_rforward.c:300-314).  One CTA per (256 tokens, head, sequence)
// walks four tiles of 64 tokens with S_in of its run in shared memory: a 64 x 128 x 128 product on tf32 mma.sync
// (A = the qt rows, B = S_in, both rounded to tf32), four warps of 16 tokens; the normalised tile then goes through
// shared memory so that z is read and the output written in whole rows.
constexpr int FIN_LD = 132, FIN_TOK = 256;
struct FinSmem { float Sin[128 * FIN_LD]; float Qt[64 * FIN_LD]; };
template <typename ACT>
__global__ void __launch_bounds__(128, 2) k_delta_seg_finish(ScanArgs a) {
    extern __shared__ __align__(16) unsigned char smraw[];
    FinSmem &sm = *reinterpret_cast<FinSmem *>(smraw);
    const int hv = blockIdx.y, b = blockIdx.z, tid = threadIdx.x, lane = tid & 31, w = tid >> 5, g = lane >> 2, j4 = lane & 3;
    const int seg_tokens = a.seg_chunks * C;                                       // a multiple of FIN_TOK? no: of 64
    const int tiles_per_seg = (seg_tokens + FIN_TOK - 1) / FIN_TOK;
    const int seg = 1 + (int)blockIdx.x / tiles_per_seg;                           // run 0 is final already
    const int tbeg = seg * seg_tokens + ((int)blockIdx.x % tiles_per_seg) * FIN_TOK;
    const int tend = min(min(tbeg + FIN_TOK, (seg + 1) * seg_tokens), a.T);
    if (tbeg >= tend) return;
    const size_t hb = (size_t)b * a.nv + hv, planes = (size_t)gridDim.z * a.nv;
    const float *Sin = a.seg_state + (hb * 3 * a.n_seg + 3 * seg + 2) * (128 * 128);
    const float *o0 = a.seg_raw + hb * (size_t)a.T * 128, *qt = a.seg_raw + (planes + hb) * (size_t)a.T * 128;
    const int vd = a.nv * 128;
    const ACT *zp = (const ACT *)a.z;
    ACT *op = (ACT *)a.out;
    for (int e = tid; e < 128 * 32; e += 128) {
        const int r = e >> 5, c4 = (e & 31) * 4;
        float4 v = *reinterpret_cast<const float4 *>(Sin + (size_t)r * 128 + c4);
        v.x = tf32r(v.x); v.y = tf32r(v.y); v.z = tf32r(v.z); v.w = tf32r(v.w);
        *reinterpret_cast<float4 *>(&sm.Sin[r * FIN_LD + c4]) = v;
    }
    const float4 nw4 = *reinterpret_cast<const float4 *>(a.norm_w + 4 * lane);     // channels 4 lane .. of the store pass
    for (int t0 = tbeg; t0 < tend; t0 += 64) {
        __syncthreads();                                                          // the tile buffer is free (and S_in is in place)
        for (int e = tid; e < 64 * 32; e += 128) {
            const int i = e >> 5, c4 = (e & 31) * 4;
            float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
            if (t0 + i < tend) v = *reinterpret_cast<const float4 *>(qt + (size_t)(t0 + i) * 128 + c4);
            v.x = tf32r(v.x); v.y = tf32r(v.y); v.z = tf32r(v.z); v.w = tf32r(v.w);
            *reinterpret_cast<float4 *>(&sm.Qt[i * FIN_LD + c4]) = v;
        }
        __syncthreads();
        // acc[nt][x]: token 16 w + g + 8 (x >> 1), value row 8 nt + 2 j4 + (x & 1)
        float acc[16][4];
#pragma unroll
        for (int nt = 0; nt < 16; nt++)
#pragma unroll
            for (int x = 0; x < 4; x++) acc[nt][x] = 0.0f;
        const float *A0 = sm.Qt + (16 * w) * FIN_LD;
#pragma unroll 2
        for (int k0 = 0; k0 < 128; k0 += 8) {
            float af[4];
            af[0] = A0[g * FIN_LD + k0 + j4];
            af[1] = A0[(g + 8) * FIN_LD + k0 + j4];
            af[2] = A0[g * FIN_LD + k0 + j4 + 4];
            af[3] = A0[(g + 8) * FIN_LD + k0 + j4 + 4];
#pragma unroll
            for (int nt = 0; nt < 16; nt++) {
                const float *br = sm.Sin + (8 * nt + g) * FIN_LD + k0 + j4;         // B[k][n] = S_in[n][k]
                mma_tf32_sync(acc[nt], af, br[0], br[4]);
            }
        }
        __syncthreads();                                                          // every warp is done reading the qt tile
        // the correction goes over the qt tile (own rows only), then whole rows: + o0, scale, norm, gate, store
#pragma unroll
        for (int nt = 0; nt < 16; nt++) {
            const int r = 8 * nt + 2 * j4;
            *reinterpret_cast<float2 *>(&sm.Qt[(16 * w + g) * FIN_LD + r]) = make_float2(acc[nt][0], acc[nt][1]);
            *reinterpret_cast<float2 *>(&sm.Qt[(16 * w + g + 8) * FIN_LD + r]) = make_float2(acc[nt][2], acc[nt][3]);
        }
        __syncwarp();
        // whole rows, 4 channels per lane; the loads of 8 tokens are issued together (memory latency, not arithmetic,
        // bounds this pass)
#pragma unroll
        for (int i0 = 0; i0 < 16; i0 += 8) {
            float4 b4[8], z4[8];
#pragma unroll
            for (int i = 0; i < 8; i++) {
                const int t = min(t0 + 16 * w + i0 + i, tend - 1);               // rows past the end repeat the last row (never stored)
                b4[i] = *reinterpret_cast<const float4 *>(o0 + (size_t)t * 128 + 4 * lane);
                z4[i] = act_ld4(zp, ((size_t)b * a.T + t) * vd + (size_t)hv * 128 + 4 * lane);
            }
#pragma unroll
            for (int i = 0; i < 8; i++) {
                const int t = t0 + 16 * w + i0 + i;
                const float4 c4 = *reinterpret_cast<const float4 *>(&sm.Qt[(16 * w + i0 + i) * FIN_LD + 4 * lane]);
                float4 o = make_float4((c4.x + b4[i].x) * a.out_scale, (c4.y + b4[i].y) * a.out_scale,
                                       (c4.z + b4[i].z) * a.out_scale, (c4.w + b4[i].w) * a.out_scale);
                float ss = (o.x * o.x + o.y * o.y) + (o.z * o.z + o.w * o.w);
                ss = warp_sum(ss);
                const float inv = rsqrtf(ss * (1.0f / 128.0f) + a.eps);
                if (t < tend)
                    act_st4(op, ((size_t)b * a.T + t) * vd + (size_t)hv * 128 + 4 * lane,
                            make_float4(o.x * inv * nw4.x * silu_fast(z4[i].x), o.y * inv * nw4.y * silu_fast(z4[i].y),
                                        o.z * inv * nw4.z * silu_fast(z4[i].z), o.w * inv * nw4.w * silu_fast(z4[i].w)));
            }
        }
    }
}

// How many runs the prompt is cut into: only when the heads alone would leave most SMs idle (2 P - 1 CTAs per head), with at least 16
// chunks per run, and not into two: every run but the first is scanned twice and finished by two more kernels.  us, one run | the
// best cut: 32 heads x 4096 tokens 239 | 272, 8192 458 | 491; 16 heads x 1024 tokens 66 | 105, 4096 221 | 215, 8192 420 | 354;
// 8 heads x 2048 101 | 117, 4096 192 | 166, 32768 1397 | 653.  ORNITH_CUDA_DELTA_SEGMENTS=<n> forces a count (1 = off).
int delta_seg_plan(int nv, int n_seq, int n_chunks, int *seg_chunks) {
    int p = 1;
    const char *e = getenv("ORNITH_CUDA_DELTA_SEGMENTS");
    if (e && e[0]) {
        p = atoi(e);
        if (p > n_chunks / 8) p = n_chunks / 8;
    } else {
        const int heads = nv * n_seq;
        if (heads <= 29) p = (148 / heads + 1) / 2;                  // 2 p - 1 <= 148 / heads
        if (p > 16) p = 16;
        if (p > n_chunks / 16) p = n_chunks / 16;
        if (p == 2) p = 1;
    }
    if (p < 1) p = 1;
    int sc = (n_chunks + p - 1) / p;
    p = (n_chunks + sc - 1) / sc;                                     // no empty run
    *seg_chunks = sc;
    return p;
}

// [n_seq][T][width] values: boxes of 128 bytes of channels (or `channels`) x `rows` tokens of one sequence, 128-byte swizzle.  The sequences are a
// dimension of their own: rows of a box behind a sequence's last token arrive as zeros and not as the next one's first tokens, whose
// infinities the products would spread over the chunk (0 x Inf).
ornith_status rows_map(CUtensorMap *m, const void *basep, bool bf, uint64_t width, uint64_t T, uint64_t n_seq, uint32_t rows,
                       CUtensorMapSwizzle swizzle = CU_TENSOR_MAP_SWIZZLE_128B, uint32_t channels = 0) {
    OrnTensorMapEncodeFn enc = orn_tensor_map_encoder();
    if (!enc) { orn_record_error("delta scan: cuTensorMapEncodeTiled is not available"); return (ornith_status)ORNITH_ERR_BACKEND; }
    const uint64_t row = width * (bf ? 2 : 4);
    cuuint64_t dims[3] = {(cuuint64_t)width, (cuuint64_t)T, (cuuint64_t)n_seq};
    cuuint64_t strides[2] = {(cuuint64_t)row, (cuuint64_t)(row * T)};
    cuuint32_t box[3] = {channels ? channels : bf ? 64u : 32u, rows, 1};
    cuuint32_t es[3] = {1, 1, 1};
    const CUresult r = enc(m, bf ? CU_TENSOR_MAP_DATA_TYPE_BFLOAT16 : CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 3, const_cast<void *>(basep), dims, strides, box, es,
                           CU_TENSOR_MAP_INTERLEAVE_NONE, swizzle, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
                           CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS) { orn_record_error("delta scan: cuTensorMapEncodeTiled failed (%d)", (int)r); return (ornith_status)ORNITH_ERR_BACKEND; }
    return ORNITH_OK;
}

}  // namespace

// How a prompt is cut: into runs scanned side by side (n_seg > 1), or into slabs of `per` chunks, whose records take `slots`
// places in turn.
struct DeltaPlan { int n_chunks, n_seg, seg_chunks, per, slots; };

static int slab_plan(int heads, int n_chunks, int n_seg);

static DeltaPlan delta_plan(int nv, int n_seq, int T) {
    DeltaPlan p;
    p.n_chunks = (T + C - 1) / C;
    const int units = nv * n_seq;
    p.n_seg = delta_seg_plan(nv, n_seq, p.n_chunks, &p.seg_chunks);
    p.per = p.n_chunks;
    p.slots = 1;
    if (p.n_seg > 1) return p;
    const int n = slab_plan(units, p.n_chunks, p.n_seg);
    if (n > 1) {                                                      // the pipeline: one slab is scanned while the next is prepared
        p.per = (p.n_chunks + n - 1) / n;
        p.slots = 2;
    }
    return p;
}

static size_t rec_part(const DeltaPlan &p, int units) { return align_up((size_t)p.slots * units * p.per * REC_BYTES, 256); }
static size_t seg_state_part(int units, int n_seg) { return n_seg > 1 ? align_up((size_t)units * 3 * n_seg * 128 * 128 * 4, 256) : 0; }
static size_t seg_raw_part(int units, int T, int n_seg) { return n_seg > 1 ? align_up((size_t)2 * units * T * 128 * 4, 256) : 0; }

size_t linear_prefill_tc5_work_bytes(int nk, int nv, int n_seq, int T) {
    (void)nk;
    const DeltaPlan p = delta_plan(nv, n_seq, T);
    const int units = nv * n_seq;
    return rec_part(p, units) + seg_state_part(units, p.n_seg) + seg_raw_part(units, T, p.n_seg);
}

// The second stream and the events of the slab pipeline, one set per device.  The lock covers one call's
// launches: a wait takes the event's state at the moment it is enqueued, so the next call may re-record.
static constexpr int MAX_SLABS = 16;
namespace {
struct SlabPipe {
    std::mutex lock;
    cudaStream_t scan_stream = nullptr;
    cudaEvent_t front_done[MAX_SLABS] = {}, scan_done[MAX_SLABS] = {};
};
SlabPipe g_slab_pipe[ORN_MAX_DEVICES];

ornith_status slab_pipe_ready(SlabPipe &p) {
    if (p.scan_stream) return ORNITH_OK;
    int least = 0, greatest = 0;
    ORN_TRY(orn_check(cudaDeviceGetStreamPriorityRange(&least, &greatest), "stream priority range"));
    cudaStream_t st = nullptr;
    ORN_TRY(orn_check(cudaStreamCreateWithPriority(&st, cudaStreamNonBlocking, greatest), "delta scan stream"));
    for (int i = 0; i < MAX_SLABS; i++) {
        ORN_TRY(orn_check(cudaEventCreateWithFlags(&p.front_done[i], cudaEventDisableTiming), "slab event"));
        ORN_TRY(orn_check(cudaEventCreateWithFlags(&p.scan_done[i], cudaEventDisableTiming), "slab event"));
    }
    p.scan_stream = st;
    return ORNITH_OK;
}
}  // namespace

// Slabs of the prompt; 1 = no pipeline (ORNITH_CUDA_DELTA_SLABS overrides).  The scan of up to half as many heads as SMs leaves the
// passes in front of it room; each slab costs a start of the scan.  us at 1 | 2 | 3 | 4 | 8 slabs: 64 heads x 4096 tokens 281 | 275 | 286 |
// 286 | 322, 8192 546 | 499 | 490 | 496 | 525, 16384 1062 | 944 | 908 | 898 | 932, 32768 2155 | 1848 | 1810 | 1772 | 1813; 32 heads x 8192
// 493 | 462 | 457 | 488, 16384 885 | 809 | 796 | 810; 128 heads x 8192 749 | 737 | 794 | 833 | 956.
static int slab_plan(int heads, int n_chunks, int n_seg) {
    if (n_seg > 1 || heads > 148) return 1;
    int n = heads <= 74 ? min(4, 1 + n_chunks / 128) : 1;
    const char *e = getenv("ORNITH_CUDA_DELTA_SLABS");
    if (e && e[0]) n = atoi(e);
    if (n > MAX_SLABS) n = MAX_SLABS;
    if (n > n_chunks) n = n_chunks;
    return n < 1 ? 1 : n;
}

// frees the current device's scan stream and events (the next long prefill makes new ones); the device is idle
ornith_status release_delta_slab_pipe() {
    SlabPipe &p = g_slab_pipe[orn_device_index()];
    std::lock_guard<std::mutex> hold(p.lock);
    if (!p.scan_stream) return ORNITH_OK;
    for (int i = 0; i < MAX_SLABS; i++) {
        for (cudaEvent_t *e : {&p.front_done[i], &p.scan_done[i]}) { if (*e) (void)cudaEventDestroy(*e); *e = nullptr; }
    }
    const cudaError_t e = cudaStreamDestroy(p.scan_stream);
    p.scan_stream = nullptr;
    return orn_check(e, "delta scan stream destroy");
}

using ScanKernel = void (*)(CUtensorMap, CUtensorMap, CUtensorMap, CUtensorMap, CUtensorMap, ScanArgs);
static ScanKernel scan_kernel(bool bf, bool seg, bool tile) {
    static const ScanKernel k[8] = {k_delta_scan_tc5<float, false, false>, k_delta_scan_tc5<__nv_bfloat16, false, false>,
                                    k_delta_scan_tc5<float, true, false>,  k_delta_scan_tc5<__nv_bfloat16, true, false>,
                                    k_delta_scan_tc5<float, false, true>,  k_delta_scan_tc5<__nv_bfloat16, false, true>,
                                    k_delta_scan_tc5<float, true, true>,   k_delta_scan_tc5<__nv_bfloat16, true, true>};
    return k[bf + 2 * seg + 4 * tile];
}

ornith_status launch_linear_prefill_tc5(const LinArgs &x, int n_seq, int act_dtype, const float *Y, const float *rq,
                                        const float *rk, const float *la, const float *be, const TC5Front *front,
                                        float *work, cudaStream_t s) {
    const int Cc = 2 * x.nk * 128 + x.nv * 128, units = x.nv * n_seq;
    if ((size_t)n_seq * x.T >= (1u << 31)) {
        orn_record_error("delta scan: %d sequences x %d tokens exceed the tensor-map coordinates", n_seq, x.T);
        return ORNITH_ERR_UNSUPPORTED;
    }
    DeltaPlan p = delta_plan(x.nv, n_seq, x.T);
    // the finishing pass behind several runs reads z and the norm's weights and writes the outputs four values at a time: a call
    // with any of them off that grid is one run, whose records take no more scratch
    const uintptr_t four = act_dtype == ORNITH_ACT_BF16 ? 8 : 16;
    if (p.n_seg > 1 && (((uintptr_t)x.z | (uintptr_t)x.out) % four || (uintptr_t)x.norm_w % 16)) p.n_seg = 1;
    static bool configured_dev[ORN_MAX_DEVICES] = {};
    bool &configured = configured_dev[orn_device_index()];
    if (!configured) {
        const auto opt_in = [](auto *k, size_t smem, const char *what) {
            return orn_check(cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem), what);
        };
        ORN_TRY(opt_in(k_delta_prep<float>, PREP_SMEM, "delta prep smem opt-in"));
        ORN_TRY(opt_in(k_delta_prep<__nv_bfloat16>, PREP_SMEM, "delta prep smem opt-in"));
        for (int v = 0; v < 8; v++) ORN_TRY(opt_in(scan_kernel(v & 1, v & 2, v & 4), SCAN_SMEM, "delta scan smem opt-in"));
        ORN_TRY(opt_in(k_delta_seg_finish<float>, sizeof(FinSmem), "delta finish smem opt-in"));
        ORN_TRY(opt_in(k_delta_seg_finish<__nv_bfloat16>, sizeof(FinSmem), "delta finish smem opt-in"));
        configured = true;
    }
    const bool bf = act_dtype == ORNITH_ACT_BF16;
    // z and the outputs travel by tensor copies where their rows lie on 16-byte boundaries (the row length always is a multiple)
    const bool tile = ((uintptr_t)x.z % 16) == 0 && ((uintptr_t)x.out % 16) == 0;
    CUtensorMap my, mym, mv, mz, mo;
    ORN_TRY(rows_map(&my, Y, false, (uint64_t)Cc, (uint64_t)x.T, (uint64_t)n_seq, C));
    ORN_TRY(rows_map(&mym, Y, false, (uint64_t)Cc, (uint64_t)x.T, (uint64_t)n_seq, C, CU_TENSOR_MAP_SWIZZLE_128B_ATOM_32B));
    ORN_TRY(rows_map(&mv, Y, false, (uint64_t)Cc, (uint64_t)x.T, (uint64_t)n_seq, C, CU_TENSOR_MAP_SWIZZLE_NONE, 128));
    mz = mo = my;
    if (tile) {
        ORN_TRY(rows_map(&mz, x.z, bf, (uint64_t)x.nv * 128, (uint64_t)x.T, (uint64_t)n_seq, C));
        ORN_TRY(rows_map(&mo, x.out, bf, (uint64_t)x.nv * 128, (uint64_t)x.T, (uint64_t)n_seq, 16));
    }
    unsigned char *rec = (unsigned char *)work;
    const size_t slot_bytes = (size_t)units * p.per * REC_BYTES;
    ScanArgs a;
    a.rec = rec; a.S = x.S; a.S_stride = x.S_stride; a.z = x.z; a.out = x.out; a.norm_w = x.norm_w;
    a.nk = x.nk; a.nv = x.nv; a.head_map = x.head_map; a.T = x.T; a.n_chunks = p.n_chunks;
    a.c_begin = 0; a.c_count = p.n_chunks; a.rec_chunks = p.per;
    a.out_scale = x.out_scale; a.eps = x.eps; a.status = orn_status_word();
    a.n_seg = p.n_seg; a.seg_chunks = p.seg_chunks;
    a.seg_state = (float *)((char *)work + rec_part(p, units));
    a.seg_raw = (float *)((char *)a.seg_state + seg_state_part(units, p.n_seg));

    // the records of the chunks cb .. cb + cn - 1, into a slot.  With a front the launch that ends the prompt also stores the
    // new history (without one the caller has done that)
    auto prep = [&](int cb, int cn, int slot, bool chained) {
        PrepArgs64 pa;
        pa.Y = Y; pa.rq = rq; pa.rk = rk; pa.la = la; pa.be = be;
        pa.rec = rec + slot * slot_bytes;
        pa.n_chunks = p.n_chunks; pa.chunk0 = cb; pa.rec_chunks = p.per; pa.refresh = front != nullptr; pa.status = orn_status_word();
        const dim3 pgrid((unsigned)cn, (unsigned)x.nk, (unsigned)n_seq);
        if (chained)
            return orn_check(bf ? orn_launch_dependent(k_delta_prep<__nv_bfloat16>, pgrid, dim3(256), PREP_SMEM, s, my, x, pa)
                                : orn_launch_dependent(k_delta_prep<float>, pgrid, dim3(256), PREP_SMEM, s, my, x, pa), "k_delta_prep");
        if (bf) k_delta_prep<__nv_bfloat16><<<pgrid, 256, PREP_SMEM, s>>>(my, x, pa);
        else    k_delta_prep<float><<<pgrid, 256, PREP_SMEM, s>>>(my, x, pa);
        return orn_check_launch("k_delta_prep");
    };
    auto scan = [&](int cb, int cn, int slot, cudaStream_t ss, bool chained) {
        ScanArgs sa = a;
        sa.rec = rec + slot * slot_bytes; sa.c_begin = cb; sa.c_count = cn;
        dim3 grid((unsigned)x.nv, (unsigned)n_seq);
        if (chained)
            return orn_check(orn_launch_dependent(scan_kernel(bf, false, tile), grid, dim3(NTHREADS), SCAN_SMEM, ss, my, mym, mv, mz, mo, sa), "k_delta_scan_tc5");
        scan_kernel(bf, false, tile)<<<grid, NTHREADS, SCAN_SMEM, ss>>>(my, mym, mv, mz, mo, sa);
        return orn_check_launch("k_delta_scan_tc5");
    };

    if (front && p.slots == 2) {
        // front of slab k + 1 on the caller's stream beside the scan of slab k on the scan stream
        SlabPipe &pipe = g_slab_pipe[orn_device_index()];
        std::lock_guard<std::mutex> hold(pipe.lock);
        ORN_TRY(slab_pipe_ready(pipe));
        int k = 0, forked = -1;                                       // forked: the last slab whose scan was enqueued
        auto slab = [&](int cb, int cn) -> ornith_status {
            ORN_TRY(front->conv(cb * C, min(x.T, (cb + cn) * C), s));
            if (k >= 2) ORN_TRY(orn_check(cudaStreamWaitEvent(s, pipe.scan_done[k - 2], 0), "slab event wait"));     // its records' place is free
            ORN_TRY(prep(cb, cn, k & 1, false));
            ORN_TRY(orn_check(cudaEventRecord(pipe.front_done[k], s), "slab event record"));
            ORN_TRY(orn_check(cudaStreamWaitEvent(pipe.scan_stream, pipe.front_done[k], 0), "slab event wait"));
            forked = k;
            ORN_TRY(scan(cb, cn, k & 1, pipe.scan_stream, false));
            return orn_check(cudaEventRecord(pipe.scan_done[k], pipe.scan_stream), "slab event record");
        };
        ornith_status st = ORNITH_OK;
        for (int cb = 0; cb < p.n_chunks && st == ORNITH_OK; cb += p.per, k++) st = slab(cb, min(p.per, p.n_chunks - cb));
        // the caller's stream always rejoins the scan stream, also when a launch failed on the way
        ornith_status join = ORNITH_OK;
        if (forked >= 0) {
            if (st != ORNITH_OK) join = orn_check(cudaEventRecord(pipe.scan_done[forked], pipe.scan_stream), "slab event record");
            if (join == ORNITH_OK) join = orn_check(cudaStreamWaitEvent(s, pipe.scan_done[forked], 0), "slab event wait");
        }
        return st != ORNITH_OK ? st : join;
    }
    if (front) ORN_TRY(front->conv(0, x.T, s));
    if (p.n_seg <= 1) {
        for (int cb = 0; cb < p.n_chunks; cb += p.per) {              // (more than one slab: the scan of one before the preparation of the next)
            const int cn = min(p.per, p.n_chunks - cb);
            ORN_TRY(prep(cb, cn, 0, front != nullptr && cb == 0));
            ORN_TRY(scan(cb, cn, 0, s, true));
        }
        return ORNITH_OK;
    }
    // few heads: the runs of the prompt side by side, then the carry over the runs and the finishing pass
    ORN_TRY(prep(0, p.n_chunks, 0, front != nullptr));
    dim3 grid((unsigned)x.nv, (unsigned)n_seq, (unsigned)(2 * a.n_seg - 1));
    scan_kernel(bf, true, tile)<<<grid, NTHREADS, SCAN_SMEM, s>>>(my, mym, mv, mz, mo, a);
    ORN_TRY(orn_check_launch("k_delta_scan_tc5 (runs)"));
    k_delta_seg_carry<<<dim3((unsigned)x.nv, (unsigned)n_seq, 16), 128, 0, s>>>(a);
    ORN_TRY(orn_check_launch("k_delta_seg_carry"));
    const int fin_tiles = (a.n_seg - 1) * ((a.seg_chunks * C + FIN_TOK - 1) / FIN_TOK);
    dim3 fgrid((unsigned)fin_tiles, (unsigned)x.nv, (unsigned)n_seq);
    if (bf) k_delta_seg_finish<__nv_bfloat16><<<fgrid, 128, sizeof(FinSmem), s>>>(a);
    else    k_delta_seg_finish<float><<<fgrid, 128, sizeof(FinSmem), s>>>(a);
    return orn_check_launch("k_delta_seg_finish");
}
