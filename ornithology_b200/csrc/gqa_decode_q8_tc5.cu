// gqa_decode_q8_tc5.cu — split-K GQA decode over Q8_0 rows on the 5th-generation tensor cores, groups of up to 16 query heads,
// head_dim 256.
//
// Replaces the attend half of ornith_gqa_step (reference: src/ornith_attn.c:111-148), its normalisation (src/ornith_attn.c:131-148) and
// the output gate (src/ornith_rforward.c:450).
//
// What bounds it: the rows from memory on long contexts, a piece's fixed chain (queries, first rows, products, partial, merge) on short
// ones.  A warp that builds mma.sync fragments from the raw rows (the kernel that ran here before) issues a dozen
// instructions per 16-byte piece for every 8 heads and was bound by that: 0.72 of the memory rate with 8 heads to a KV head, 0.43 with
// 16, whose rows it converted twice.  Here a row is converted once, whatever the number of heads, and the products cost no issue
// slots.  One CTA per SM walks a range of the batch's rows, 128 tokens (a tile) at a time:
//   S^T[token][head] = K Q^T    M128 N16 K256   A = K rows in tensor memory (a thread's row is its lane), B = Q in shared memory
//   O^T[dim][head] += V^T P^T   M128 N16 K128, twice   A = V rows, B = P, both in shared memory and MN-major
//   warps 0-7    K: half a row per thread to f16, tcgen05.st
//   warps 8-15   V: half a row per thread to f16 in a 128-byte-swizzled buffer, two buffers of 64 tokens
//   warps 16-19  softmax, a thread per token: probabilities against a reference maximum that only moves when exceeded by 2^6 (O is then
//                rescaled in tensor memory); at the end of a piece its partial
//   warps 20,21  copy the raw rows of K and of V, 32 to a slot: one tensor copy, or a row per lane where fewer are left
//   warp 22      one lane issues the products
//   all warps, at the end: the merge of the sequences whose last partial was written here
// Time of one decode step's attention with its preparation, us, raw-fragment kernel -> this one: 16 query / 2 KV heads (35B), 1 sequence
// of 16384 tokens 33.5 -> 25.8, 8 of 256 36 -> 18.8, 32 of 1024 42.6 -> 26.8, 64 of 16384 218 -> 194 (5.8 TB/s, 0.88 of the copy rate), 256 of
// 256 56 -> 56; 32 query heads (397B), 1 of 4096 25.3 -> 23.0, 16 of 16384 117 -> 75, 256 of 4096 432 -> 259, 256 of 8192 790 -> 488.
// What it took, at 256 x 8192: the roles' unrolled code within the instruction caches (730 -> 605: one code for both halves of a row); a
// loader of its own for V (issue and waits of one warp came to 4200 cycles a tile, 605 -> 541); P with the heads contiguous, two
// 16-byte stores in place of sixteen of 2 bytes (541 -> 496).
// Shared-memory traffic is the next bound: raw rows in and out (K's read with two lanes to a bank), V as f16 in and out: 2.6k of the 3.0k
// cycles in which a tile's rows arrive at the memory rate.  K goes from registers to tensor memory for that reason.
// Precision as in the other kernels: q scaled per head by a power of two and rounded to f16, decoded K/V elements with one f16
// rounding, probabilities times 2^8 rounded to f16, f32 accumulation.
// Every wait is bounded; one that gives up poisons the partials from there on and is reported through the status word.
//
// Schedule: the 16-token units of all sequences, laid end to end with a.piece_cost extra ones in front of every sequence (the fixed work of a
// piece), are cut into gridDim.y ranges of equal length, found on the device from kv_len: the host never learns the contexts.  A CTA walks
// the pieces of the sequences that fall into its range, one partial per piece.  Every CTA is resident at once and all of them stream
// about the same number of rows; the CTAs of the KV heads (blockIdx.x) walk the same range side by side, their rows interleave in memory.
#include <cuda.h>

#include <string.h>

#include "full_attn.cuh"
#include "tcgen05.cuh"

namespace {
using namespace tc5;

constexpr int HD = 256, ROWB = 272, UNIT = 16, TILE = 128, SLOT = 32, NSLOT = 16;
constexpr int SLOT_BYTES = SLOT * ROWB;                 // 8704
constexpr int SM_V = 0, SM_Q = 65536, SM_P = SM_Q + 8192, SM_RAW = SM_P + 8192;      // P: 2 tiles of 4 KiB
constexpr int SMEM = SM_RAW + NSLOT * SLOT_BYTES + 1024;     // + alignment slack
constexpr int TM_K = 0, TM_S = 256, TM_O = 288, TM_COLS = 512;   // tensor-memory columns: K 2 x 128, S 2 x 16, O 2 halves x 16
constexpr int W_V = 8, W_SM = 16, W_LD = 20, W_MMA = 22, NT = 23 * 32;
constexpr int NMERGE = 32;
constexpr float LOG2E = 1.4426950408889634f, LN2 = 0.6931471805599453f;

struct __align__(16) Bars {
    unsigned long long raw_full[NSLOT], raw_empty[NSLOT];
    unsigned long long k_full[2], k_empty[2], v_full[2], v_empty[2], s_full[2], s_empty[2], p_full[2], p_empty[2];
    unsigned long long q_full, o_free, drained;
};

// Units a step reads for sequence b: its context and the token being appended; none for a sequence whose cache is full (it is left alone).
__device__ __forceinline__ int seq_units(const DecodeArgs &a, int b) {
    const int len0 = a.kv_len[b];
    const int cap = (int)(a.kv.seq_off[b + 1] - a.kv.seq_off[b]);
    return len0 >= cap ? 0 : (len0 + UNIT) / UNIT;
}

// The walk over the pieces of a range, the same for every warp.  (range, sequence) pairs in walking order: range + sequence is unique, the
// slot of the piece's partial.
struct Walk { int b, first, pos, end, W; };
struct Piece { int b, t0, t1, slot, slot0, nlive; };    // tokens t0 .. t1 - 1 of sequence b; its partial's slot, the sequence's first slot and count
__device__ __forceinline__ bool next_piece(const DecodeArgs &a, Walk &w, int range, Piece &p) {
    if (w.pos >= w.end) return false;
    const int pad = a.piece_cost;
    int nb = seq_units(a, w.b);
    while (nb == 0 || w.first + pad + nb <= w.pos) { w.first += nb ? nb + pad : 0; w.b++; nb = seq_units(a, w.b); }
    const int real0 = w.first + pad, lo = max(w.pos - real0, 0), hi = min(nb, w.end - real0);
    if (hi <= lo) return false;                          // the range ends inside the charge in front of the sequence
    const int c_first = real0 / w.W;
    p.b = w.b;
    p.t0 = lo * UNIT;
    p.t1 = min(a.kv_len[w.b] + 1, hi * UNIT);
    p.slot = range + w.b;
    p.slot0 = c_first + w.b;
    p.nlive = (real0 + nb - 1) / w.W - c_first + 1;
    w.pos = real0 + hi;
    return true;
}

__device__ __forceinline__ uint32_t h2_mul_sub(uint32_t biased, uint32_t scale) {   // (x - 1152) * scale
    const __half2 bias = __floats2half2_rn(1152.0f, 1152.0f);
    __half2 v = __hmul2(__hsub2(*reinterpret_cast<__half2 *>(&biased), bias), *reinterpret_cast<__half2 *>(&scale));
    return *reinterpret_cast<uint32_t *>(&v);
}
__device__ __forceinline__ uint2 lds64u(uint32_t addr) {
    uint2 v;
    asm volatile("ld.shared.v2.u32 {%0, %1}, [%2];" : "=r"(v.x), "=r"(v.y) : "r"(addr));
    return v;
}
// The 64 f16 pairs of the raw half row at `half`, in order: sink(i, pair).  A row is a stream of 16-bit elements, per block (4 of them) one
// f16 scale and 16 pairs of codes; every position is a constant, and a pair never straddles a word.  One code for both halves, with
// 8-byte reads (two to a bank) because of it: the roles' code has to fit the instruction caches.
template <typename SINK>
__device__ __forceinline__ void decode_half(uint32_t half, uint32_t keep, SINK sink) {
    uint32_t scale = 0;
#pragma unroll
    for (int c = 0; c < 17; c++) {
        const uint2 v = lds64u(half + 8 * c);
        const uint32_t w[2] = {v.x, v.y};
#pragma unroll
        for (int i = 0; i < 4; i++) {
            const int e = 4 * c + i, b = e / 17, k = e % 17;
            if (k == 0) scale = __byte_perm(w[i >> 1], 0u, (i & 1) ? 0x3232 : 0x1010) & keep;
            else sink(16 * b + k - 1, h2_mul_sub(__byte_perm(w[i >> 1] ^ 0x80808080u, 0x64646464u, (i & 1) ? 0x4342 : 0x4140), scale));
        }
    }
}

// (the parked wait starts with the clock, 160 cycles that most waits here do not need)
__device__ __forceinline__ bool wait_for(uint32_t bar, uint32_t parity) { return mbar_try(bar, parity) || mbar_wait_parked(bar, parity); }
// Lanes give up each for itself, by its own reading of the clock.  So no lane leaves its warp when a wait did: those that stayed would
// miss it at the next collective instruction.  The warp goes on without waiting and passes nothing on (the loaders, who must not copy
// over a slot in use, leave together).  Votes at the waits themselves took 1 % of the batches of 256 x 8192 tokens.
__device__ __forceinline__ bool all_lanes(bool ok) { return __all_sync(0xffffffffu, ok); }
// Operand B with the heads contiguous: rows of 16 heads (32 bytes) a token, 32-byte swizzle (16-byte piece c of row r at c ^ (r >> 2 & 1))
__device__ __forceinline__ uint64_t p_desc(uint32_t saddr) {
    return (uint64_t)((saddr >> 4) & 0x3FFF) | ((uint64_t)1 << 16) | ((uint64_t)(256 >> 4) << 32) | ((uint64_t)1 << 46) | ((uint64_t)6 << 61);
}
__device__ __forceinline__ void sm_sync(int id) { asm volatile("bar.sync %0, 128;" ::"r"(id) : "memory"); }     // the softmax warps
__device__ __forceinline__ bool sm_any(int id, bool x) {
    uint32_t r;
    asm volatile("{\n .reg .pred p, q;\n setp.ne.u32 p, %1, 0;\n barrier.cta.red.or.pred.aligned q, %2, 128, p;\n selp.u32 %0, 1, 0, q;\n}\n"
                 : "=r"(r) : "r"((uint32_t)x), "r"(id) : "memory");
    return r != 0;
}
__device__ __forceinline__ void fence_async() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }
__device__ __forceinline__ void tensor_copy(uint32_t dst, const CUtensorMap *map, int head, int token, uint32_t bar) {
    asm volatile("cp.async.bulk.tensor.3d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5}], [%2];\n"
                 ::"r"(dst), "l"(map), "r"(bar), "r"(0), "r"(head), "r"(token) : "memory");
}

// One head of a sequence from its partials, by one warp: lane owns the float2 columns lane + 32 k; four partials' rows in flight
__device__ __forceinline__ void merge_head(const DecodeArgs &a, int b, int head, int slot0, int nlive, int lane) {
    const float *ph = a.part + ((size_t)head * a.nsplit + slot0) * (HD + 2);
    const size_t row = (size_t)b * a.nh + head;
    float2 gate[4];
#pragma unroll
    for (int k = 0; k < 4; k++) {
        const size_t at = row * HD * 2 + HD + 2 * (lane + 32 * k);
        gate[k] = make_float2(0.0f, 0.0f);
        if (a.gated)
            gate[k] = a.act_dtype == ORNITH_ACT_BF16 ? make_float2(act_ld((const __nv_bfloat16 *)a.qproj, at), act_ld((const __nv_bfloat16 *)a.qproj, at + 1))
                                                     : make_float2(act_ld((const float *)a.qproj, at), act_ld((const float *)a.qproj, at + 1));
    }
    float M = -INFINITY;
    for (int s = lane; s < nlive; s += 32) {
        const float2 ml = __ldcg(reinterpret_cast<const float2 *>(ph + (size_t)s * (HD + 2)));
        if (ml.y > 0.0f) M = fmaxf(M, ml.x);
    }
    M = warp_max(M);
    float lsum = 0.0f;
    float2 acc[4];
#pragma unroll
    for (int k = 0; k < 4; k++) acc[k] = make_float2(0.0f, 0.0f);
    for (int s = 0; s < nlive; s += 4) {
        float2 v[4][4], ml[4];
#pragma unroll
        for (int x = 0; x < 4; x++) {
            const float2 *r = reinterpret_cast<const float2 *>(ph + (size_t)min(s + x, nlive - 1) * (HD + 2));
            ml[x] = __ldcg(r);
#pragma unroll
            for (int k = 0; k < 4; k++) v[x][k] = __ldcg(r + 1 + lane + 32 * k);
        }
#pragma unroll
        for (int x = 0; x < 4; x++) {
            const float wt = s + x < nlive && ml[x].y > 0.0f ? expf(ml[x].x - M) : 0.0f;
            if (wt != 0.0f) {
                lsum += ml[x].y * wt;
#pragma unroll
                for (int k = 0; k < 4; k++) { acc[k].x += v[x][k].x * wt; acc[k].y += v[x][k].y * wt; }
            }
        }
    }
    const float inv = 1.0f / lsum;
#pragma unroll
    for (int k = 0; k < 4; k++) {
        float2 o = make_float2(acc[k].x * inv, acc[k].y * inv);
        if (a.gated) { o.x *= sigmoid_f(gate[k].x); o.y *= sigmoid_f(gate[k].y); }
        const size_t at = row * HD + 2 * (lane + 32 * k);
        if (a.act_dtype == ORNITH_ACT_BF16) { act_st((__nv_bfloat16 *)a.out, at, o.x); act_st((__nv_bfloat16 *)a.out, at + 1, o.y); }
        else { act_st((float *)a.out, at, o.x); act_st((float *)a.out, at + 1, o.y); }
    }
}

// NH = columns of scores worked on: 8 or 16
template <int NH>
__global__ void __launch_bounds__(NT, 1) k_gqa_decode_q8_tc5(DecodeArgs a, const __grid_constant__ CUtensorMap map_k,
                                                             const __grid_constant__ CUtensorMap map_v, int tensor_copies) {
    extern __shared__ unsigned char smraw[];
    __shared__ Bars bars;
    __shared__ Walk walk_s;
    __shared__ uint32_t tmem_slot;
    __shared__ __align__(16) float rs_s[16], m_s[16], l_s[4][16], cm_s[4][16];
    __shared__ int3 merge_s[NMERGE];                     // sequences whose last partial this CTA wrote: sequence, first slot, partials
    __shared__ int merge_n, last_s;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int nkv = a.kv.nkv, G = a.nh / nkv, kvh = blockIdx.x, range = blockIdx.y;
    // the next layer's front-end kernel may become resident now; it waits for this grid before it does anything
    asm volatile("griddepcontrol.launch_dependents;\n" ::: "memory");
    const uint32_t base = (su32(smraw) + 1023u) & ~1023u;
    unsigned char *gbase = smraw + (base - su32(smraw));

    // range length and this CTA's first sequence (kv_len and seq_off are not written by the kernel in front)
    if (warp == 0) {
        const int pad = a.piece_cost;
        int total = 0;
        for (int b0 = 0; b0 < a.n_seq; b0 += 32) {
            const int n = b0 + lane < a.n_seq ? seq_units(a, b0 + lane) : 0;
            total += __reduce_add_sync(0xffffffffu, n ? n + pad : 0);
        }
        Walk w;
        w.W = max((total + (int)gridDim.y - 1) / (int)gridDim.y, a.range_floor);
        w.pos = range * w.W;
        w.end = min(total, w.pos + w.W);
        w.b = 0; w.first = 0;
        int running = 0;
        for (int b0 = 0; b0 < a.n_seq && w.pos < total; b0 += 32) {
            const int n = b0 + lane < a.n_seq ? seq_units(a, b0 + lane) : 0, cost = n ? n + pad : 0;
            int incl = cost;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) { const int t = __shfl_up_sync(0xffffffffu, incl, o); if (lane >= o) incl += t; }
            const int lo = running + incl - cost;
            const unsigned hit = __ballot_sync(0xffffffffu, cost && lo <= w.pos && w.pos < lo + cost);
            if (hit) {
                const int src = __ffs(hit) - 1;
                w.b = b0 + src;
                w.first = __shfl_sync(0xffffffffu, lo, src);
                break;
            }
            running += __shfl_sync(0xffffffffu, incl, 31);
        }
        if (lane == 0) walk_s = w;
    }
    if (tid == 0) {
        for (int s = 0; s < NSLOT; s++) { mbar_init(su32(&bars.raw_full[s]), 1); mbar_init(su32(&bars.raw_empty[s]), 2); }
        for (int s = 0; s < 2; s++) {
            mbar_init(su32(&bars.k_full[s]), 8); mbar_init(su32(&bars.k_empty[s]), 1);
            mbar_init(su32(&bars.v_full[s]), 4); mbar_init(su32(&bars.v_empty[s]), 1);
            mbar_init(su32(&bars.s_full[s]), 1); mbar_init(su32(&bars.s_empty[s]), 4);
            mbar_init(su32(&bars.p_full[s]), 4); mbar_init(su32(&bars.p_empty[s]), 1);
        }
        mbar_init(su32(&bars.q_full), 4); mbar_init(su32(&bars.o_free), 4); mbar_init(su32(&bars.drained), 1);
        mbar_init_fence();
        merge_n = 0;
    }
    __syncthreads();
    Walk w = walk_s;
    if (w.pos >= w.end) { asm volatile("griddepcontrol.wait;\n" ::: "memory"); return; }
    if (warp == W_MMA) tmem_alloc(&tmem_slot, TM_COLS);
    fence_before();
    __syncthreads();
    fence_after();
    const uint32_t tmem = tmem_slot;
    bool ok = true;
    Piece p;

    if (warp == W_LD || warp == W_LD + 1) {
        // ================= raw rows: K, V =================
        asm volatile("griddepcontrol.wait;\n" ::: "memory");         // the row the step appends
        const int kv = warp - W_LD;
        const CUtensorMap *map = kv ? &map_v : &map_k;
        const uint8_t *rows = kv ? a.kv.V : a.kv.K;
        int T = 0, n = 0;
        while (ok && next_piece(a, w, range, p)) {
            const int64_t row0 = a.kv.seq_off[p.b];
            for (int t = p.t0; t < p.t1 && ok; t += TILE, T++)
                for (int i = 0; i < 4 && ok; i++) {
                    const int s = 8 * kv + (T & 1) * 4 + i, tok = t + i * SLOT, valid = max(0, min(SLOT, p.t1 - tok));
                    if (T >= 2) ok = all_lanes(wait_for(su32(&bars.raw_empty[s]), (uint32_t)((T >> 1) - 1) & 1u));
                    if (!ok) break;
                    const uint32_t bar = su32(&bars.raw_full[s]), dst = base + SM_RAW + s * SLOT_BYTES;
                    if (valid == SLOT && tensor_copies) {
                        if (elect_one()) {
                            mbar_expect_tx(bar, SLOT_BYTES);
                            tensor_copy(dst, map, kvh, (int)row0 + tok, bar);
                        }
                    } else {
                        if (lane == 0) { if (valid) mbar_expect_tx(bar, (uint32_t)(valid * ROWB)); else mbar_arrive(bar); }
                        __syncwarp();
                        if (lane < valid) bulk_load(dst + lane * ROWB, rows + ((size_t)(row0 + tok + lane) * nkv + kvh) * ROWB, ROWB, bar);
                    }
                    n++;
                }
        }
        // n slots were filled, in turn: none of the copies may outlive the CTA, whatever happened to those that wait for them
        for (int s = 0; s < 8 && s < n; s++) ok = wait_for(su32(&bars.raw_full[8 * kv + s]), (uint32_t)((n + 7 - s) / 8 - 1) & 1u) && ok;
    } else if (warp < W_V) {
        // ================= K rows to f16, in tensor memory =================
        // Warps 0-3 have dims 0..127 of 32 rows each, warps 4-7 dims 128..255.
        const int q = warp & 3, hf = warp >> 2;
        int T = 0;
        while (next_piece(a, w, range, p)) {
            for (int t = p.t0; t < p.t1; t += TILE, T++) {
                const int g = T & 1, slot = 4 * g + q;
                const uint32_t kt = tmem + ((uint32_t)(32 * q) << 16) + TM_K + 128 * g + 64 * hf;
                if (T >= 2) ok = ok && wait_for(su32(&bars.k_empty[g]), (uint32_t)((T >> 1) - 1) & 1u);
                ok = ok && wait_for(su32(&bars.raw_full[slot]), (uint32_t)(T >> 1) & 1u);
                fence_after();
                if (t + 32 * q < p.t1) {                             // (rows past the end: whatever their scores are, they are masked)
                    float o[32];
                    decode_half(base + SM_RAW + slot * SLOT_BYTES + lane * ROWB + hf * (ROWB / 2), 0xffffffffu, [&](int i, uint32_t h2) {
                        o[i & 31] = __uint_as_float(h2);
                        if ((i & 31) == 31) tmem_st32(kt + (i & ~31), o);
                    });
                    tmem_wait_st();
                }
                fence_before();
                if (all_lanes(ok) && lane == 0) { mbar_arrive(su32(&bars.k_full[g])); mbar_arrive(su32(&bars.raw_empty[slot])); }
            }
        }
    } else if (warp < W_SM) {
        // ================= V rows to f16 =================
        constexpr int NST = 32;
        // Four warps have tokens 0..63 of a tile, four tokens 64..127, each half in an f16 buffer and value products of its own: while
        // one half is multiplied the other is decoded.  A thread has 128 dims of a row.
        const int th = (warp - W_V) >> 2, r = 2 * th + ((warp >> 1) & 1), hf = (lane >> 3) & 1, row = (warp & 1) * 16 + (lane >> 4) * 8 + (lane & 7), token = 32 * r + row;
        const uint32_t vt = base + SM_V + th * 32768 + hf * 16384 + (token & 63) * 128;
        int T = 0;
        while (next_piece(a, w, range, p)) {
            for (int t = p.t0; t < p.t1; t += TILE, T++) {
                const int slot = 8 + (T & 1) * 4 + r;
                ok = ok && wait_for(su32(&bars.raw_full[slot]), (uint32_t)(T >> 1) & 1u);
                // the first 64 dims stay in registers while the value product of the tile before still reads the buffer
                // a row past the end becomes zeros (a probability of zero must not meet anything but a number)
                uint32_t o[NST];
                auto put = [&](int c, const uint32_t *v) {           // 8 dims: piece c & 7 of slab c >> 3
                    asm volatile("st.shared.v4.u32 [%0], {%1, %2, %3, %4};"
                                 ::"r"(vt + (c >> 3) * 8192 + (((c & 7) ^ (lane & 7)) << 4)), "r"(v[0]), "r"(v[1]), "r"(v[2]), "r"(v[3]) : "memory");
                };
                decode_half(base + SM_RAW + slot * SLOT_BYTES + row * ROWB + hf * (ROWB / 2), t + token < p.t1 ? 0xffffffffu : 0u, [&](int i, uint32_t h2) {
                    if (i < NST) {
                        o[i] = h2;
                        if (i == NST - 1) {
#pragma unroll
                            for (int k = 0; k < NST; k++) asm volatile("" : "+r"(o[k]));     // (decoded here, not after the wait)
                            if (T >= 1) ok = ok && wait_for(su32(&bars.v_empty[th]), (uint32_t)(T - 1) & 1u);
#pragma unroll
                            for (int c = 0; c < NST / 4; c++) put(c, o + 4 * c);
                        }
                        return;
                    }
                    o[i & 3] = h2;
                    if ((i & 3) == 3) put(i >> 2, o);
                });
                fence_async();
                if (all_lanes(ok) && lane == 0) { mbar_arrive(su32(&bars.raw_empty[slot])); mbar_arrive(su32(&bars.v_full[th])); }
            }
        }
    } else if (warp == W_MMA) {
        // ================= products =================
        if (elect_one()) {
            constexpr uint32_t ID_S = idesc(0, 16, false), ID_O = ID_S | (3u << 15);     // O: A and B MN-major
            int T = 0, n = 0;
            auto values = [&](int t, bool first) {                   // O^T += V^T P^T of tile t
                const int g = t & 1;
                ok = ok && wait_for(su32(&bars.p_full[g]), (uint32_t)(t >> 1) & 1u);
                if (ok && first && n > 0) ok = wait_for(su32(&bars.o_free), (uint32_t)(n - 1) & 1u);
#pragma unroll
                for (int th = 0; th < 2; th++) {
                    ok = ok && wait_for(su32(&bars.v_full[th]), (uint32_t)t & 1u);
                    if (!ok) return;
                    fence_after();
#pragma unroll
                    for (int hf = 0; hf < 2; hf++)
#pragma unroll
                        for (int ks = 0; ks < 4; ks++)
                            mma_f16_ss(tmem + TM_O + 16 * hf, smem_desc(base + SM_V + th * 32768 + hf * 16384 + ks * 2048, 8192, 1024),
                                       p_desc(base + SM_P + g * 4096 + th * 2048 + ks * 512), ID_O, !first || th > 0 || ks > 0);
                    mma_commit(su32(&bars.v_empty[th]));
                }
                mma_commit(su32(&bars.p_empty[g]));
            };
            while (ok && next_piece(a, w, range, p)) {
                ok = wait_for(su32(&bars.q_full), (uint32_t)n & 1u);
                const int T0 = T;
                for (int t = p.t0; t < p.t1 && ok; t += TILE, T++) {
                    const int g = T & 1;
                    ok = wait_for(su32(&bars.k_full[g]), (uint32_t)(T >> 1) & 1u) &&
                         (T < 2 || wait_for(su32(&bars.s_empty[g]), (uint32_t)((T >> 1) - 1) & 1u));
                    if (!ok) break;
                    fence_after();
#pragma unroll
                    for (int ks = 0; ks < 16; ks++)
                        mma_f16_ts(tmem + TM_S + 16 * g, tmem + TM_K + 128 * g + 8 * ks, smem_desc(base + SM_Q + (ks >> 2) * 2048 + (ks & 3) * 32, 16, 1024),
                                   ID_S, ks > 0);
                    mma_commit(su32(&bars.s_full[g]));
                    mma_commit(su32(&bars.k_empty[g]));
                    if (T > T0) values(T - 1, T - 1 == T0);
                }
                if (ok) values(T - 1, T - 1 == T0);                  // ahead of the wait for the next piece's queries
                n++;
            }
            if (!ok) {                                               // nothing may be multiplied when the tensor memory goes back
                mma_commit(su32(&bars.drained));
                (void)wait_for(su32(&bars.drained), 0u);
            }
        }
    } else {
        // ================= softmax, partials, merge =================
        asm volatile("griddepcontrol.wait;\n" ::: "memory");         // query rows, zeroed counters
        const int q = warp & 3, st = tid - W_SM * 32, token = 32 * q + lane;
        const uint32_t lane_t = tmem + ((uint32_t)(32 * q) << 16);
        const size_t part_stride = (size_t)a.nsplit * (HD + 2);      // next head
        const int head0 = kvh * G;
        for (int e = st; e < 512; e += 128)                          // both tiles of P: the rows of heads that do not exist stay zero
            *reinterpret_cast<uint4 *>(gbase + SM_P + 16 * e) = make_uint4(0u, 0u, 0u, 0u);
        int T = 0;
        while (next_piece(a, w, range, p)) {
            // ---- queries: eight threads to a head, 32 dims each (the scores of the piece before have all been made)
            {
                const int h = st >> 3, part = st & 7;
                const float *qr = a.q_prep + ((size_t)p.b * a.nh + head0 + (h < G ? h : 0)) * HD + 32 * part;
                float x[32], mx = 0.0f;
#pragma unroll
                for (int i = 0; i < 8; i++) {
                    const float4 v = reinterpret_cast<const float4 *>(qr)[i];
                    x[4 * i] = v.x; x[4 * i + 1] = v.y; x[4 * i + 2] = v.z; x[4 * i + 3] = v.w;
                    mx = fmaxf(mx, fmaxf(fmaxf(fabsf(v.x), fabsf(v.y)), fmaxf(fabsf(v.z), fabsf(v.w))));
                }
#pragma unroll
                for (int o = 1; o < 8; o <<= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
                int e = 0;
                if (mx > 0.0f && mx < INFINITY) (void)frexpf(mx, &e);
                const float down = h < G ? exp2f((float)-e) : 0.0f;
#pragma unroll
                for (int i = 0; i < 4; i++) {
                    uint32_t v[4];
#pragma unroll
                    for (int k = 0; k < 4; k++) {
                        const __half2 h2 = __floats2half2_rn(x[8 * i + 2 * k] * down, x[8 * i + 2 * k + 1] * down);
                        v[k] = *reinterpret_cast<const uint32_t *>(&h2);
                    }
                    // dims 32 part + 8 i ..: slab part >> 1, piece 4 (part & 1) + i
                    *reinterpret_cast<uint4 *>(gbase + SM_Q + (part >> 1) * 2048 + h * 128 + (((4 * (part & 1) + i) ^ (h & 7)) << 4)) = make_uint4(v[0], v[1], v[2], v[3]);
                }
                if (part == 0) { rs_s[h] = h < G ? a.scale * exp2f((float)e) * LOG2E : 0.0f; m_s[h] = -INFINITY; }
                fence_async();
                sm_sync(1);
                if (lane == 0) mbar_arrive(su32(&bars.q_full));
            }
            // (a wait that gave up leaves the loop running: the four warps share its barriers)
            float l[NH];
#pragma unroll
            for (int h = 0; h < NH; h++) l[h] = 0.0f;
            for (int t = p.t0; t < p.t1; t += TILE, T++) {
                const int g = T & 1;
                ok = ok && wait_for(su32(&bars.s_full[g]), (uint32_t)(T >> 1) & 1u);
                fence_after();
                float x[16];
                tmem_ld16_wait(lane_t + TM_S + 16 * g, x);
                // x: scores in logs, over 2^-8 of the reference maximum (m_s)
                const bool live = t + token < p.t1;
                float top = -INFINITY;
#pragma unroll
                for (int h = 0; h < NH; h += 4) {
                    const float4 r4 = *reinterpret_cast<const float4 *>(&rs_s[h]), m4 = *reinterpret_cast<const float4 *>(&m_s[h]);
                    x[h] = fmaf(x[h], r4.x, -m4.x); x[h + 1] = fmaf(x[h + 1], r4.y, -m4.y);
                    x[h + 2] = fmaf(x[h + 2], r4.z, -m4.z); x[h + 3] = fmaf(x[h + 3], r4.w, -m4.w);
                    top = fmaxf(top, fmaxf(fmaxf(x[h], x[h + 1]), fmaxf(x[h + 2], x[h + 3])));
                }
                ok = ok && (T < 2 || wait_for(su32(&bars.p_empty[g]), (uint32_t)((T >> 1) - 1) & 1u));
                if (sm_any(2, live && !(top <= 14.0f))) {
                    // a score above 2^6 times a reference maximum, or no maximum yet: move it (all threads agree)
                    fence_after();
                    tmem_ld16_wait(lane_t + TM_S + 16 * g, x);
                    float corr[NH];
#pragma unroll
                    for (int h = 0; h < NH; h++) {
                        x[h] = live ? x[h] * rs_s[h] : -INFINITY;
                        const float c = warp_max(x[h]);
                        if (lane == 0) cm_s[q][h] = c;
                    }
                    sm_sync(1);
#pragma unroll
                    for (int h = 0; h < NH; h++) {
                        const float c = fmaxf(fmaxf(cm_s[0][h], cm_s[1][h]), fmaxf(cm_s[2][h], cm_s[3][h])) - 8.0f, m = m_s[h], nm = c > m + 6.0f ? c : m;
                        corr[h] = exp2f(m - nm);                     // 0 on the first tile
                        l[h] = t == p.t0 ? 0.0f : l[h] * corr[h];
                        x[h] -= nm;
                    }
                    sm_sync(1);
                    if (st < NH) {
                        const float c = fmaxf(fmaxf(cm_s[0][st], cm_s[1][st]), fmaxf(cm_s[2][st], cm_s[3][st])) - 8.0f;
                        if (c > m_s[st] + 6.0f) m_s[st] = c;
                    }
                    if (t > p.t0) {                                  // O between two value products: the last one is done, the next waits for us
                        ok = ok && wait_for(su32(&bars.p_empty[(T - 1) & 1]), (uint32_t)((T - 1) >> 1) & 1u);
                        fence_after();
                        float o0[16], o1[16];
                        tmem_ld16x2_wait(lane_t + TM_O, o0, lane_t + TM_O + 16, o1);
#pragma unroll
                        for (int h = 0; h < NH; h++) { o0[h] *= corr[h]; o1[h] *= corr[h]; }
                        tmem_st16(lane_t + TM_O, o0);
                        tmem_st16(lane_t + TM_O + 16, o1);
                        tmem_wait_st();
                    }
                    sm_sync(1);
                }
                fence_before();
                __syncwarp();
                if (lane == 0) mbar_arrive(su32(&bars.s_empty[g]));
                if (t + TILE > p.t1 && !live) {
#pragma unroll
                    for (int h = 0; h < NH; h++) x[h] = -INFINITY;
                }
#pragma unroll
                for (int h = 0; h < NH; h += 8) {
                    uint32_t e2[4];
#pragma unroll
                    for (int i = 0; i < 8; i += 2) {
                        const float e0 = ex2_fast(x[h + i]), e1 = ex2_fast(x[h + i + 1]);
                        l[h + i] += e0;
                        l[h + i + 1] += e1;
                        const __half2 v = __floats2half2_rn(e0, e1);
                        e2[i >> 1] = *reinterpret_cast<const uint32_t *>(&v);
                    }
                    *reinterpret_cast<uint4 *>(gbase + SM_P + g * 4096 + token * 32 + (((h >> 3) ^ ((token >> 2) & 1)) << 4)) = make_uint4(e2[0], e2[1], e2[2], e2[3]);
                }
                fence_before();
                fence_async();
                __syncwarp();
                if (lane == 0) mbar_arrive(su32(&bars.p_full[g]));
            }
            // ---- the piece's partial: lane = dim
            ok = ok && wait_for(su32(&bars.p_empty[(T - 1) & 1]), (uint32_t)((T - 1) >> 1) & 1u);
            float o0[16], o1[16];
            fence_after();
            tmem_ld16x2_wait(lane_t + TM_O, o0, lane_t + TM_O + 16, o1);
            fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(su32(&bars.o_free));
#pragma unroll
            for (int h = 0; h < NH; h++) {
                const float sum = warp_sum(l[h]);
                if (lane == 0) l_s[q][h] = sum;
            }
            float *part_g = a.part + (size_t)head0 * a.nsplit * (HD + 2);
            float *part = part_g + (size_t)p.slot * (HD + 2);
#pragma unroll
            for (int h = 0; h < NH; h++)
                if (h < G) {
                    float *d = part + h * part_stride + 2 + token;
                    d[0] = ok ? o0[h] * (1.0f / 256.0f) : NAN;
                    d[128] = ok ? o1[h] * (1.0f / 256.0f) : NAN;
                }
            sm_sync(1);
            if (st < G) {
                part[st * part_stride] = (m_s[st] + 8.0f) * LN2;
                part[st * part_stride + 1] = ok ? ((l_s[0][st] + l_s[1][st]) + (l_s[2][st] + l_s[3][st])) * (1.0f / 256.0f) : 1.0f;
            }
            // ---- the last CTA of this (sequence, KV head) to get here merges (nobody waits), at the end and
            // with all its warps; four warps between two pieces, where the pipeline stands still meanwhile, once the list is full
            __threadfence();
            sm_sync(1);
            if (st == 0) {
                last_s = atomicAdd(a.group_ctr + (size_t)p.b * gridDim.x + blockIdx.x, 1) == p.nlive - 1;
                if (last_s && merge_n < NMERGE) {
                    merge_s[merge_n++] = make_int3(p.b, p.slot0, p.nlive);
                    last_s = 0;
                }
            }
            sm_sync(1);
            if (!last_s) continue;
            __threadfence();
            for (int h = q; h < G; h += 4) merge_head(a, p.b, head0 + h, p.slot0, p.nlive, lane);
        }
    }
    if (!ok) report_timeout(a.status, ORN_WAIT_DECODE);
    fence_before();
    __syncthreads();
    if (warp == W_MMA) tmem_dealloc(tmem, TM_COLS);
    asm volatile("griddepcontrol.wait;\n" ::: "memory");             // the gates (over long since)
    __threadfence();
    for (int i = warp; i < merge_n * G; i += NT / 32) {
        const int3 m = merge_s[i / G];
        merge_head(a, m.x, kvh * G + i % G, m.y, m.z, lane);
    }
}

// [token][KV head][68 words]: a box is the 32 rows of one head for 32 tokens; only whole boxes of valid tokens are asked for, so the
// token extent is left open
bool rows_map(CUtensorMap *m, const void *pool, int nkv) {
    OrnTensorMapEncodeFn enc = orn_tensor_map_encoder();
    if (!enc || ((uintptr_t)pool & 15) != 0) return false;
    cuuint64_t dims[3] = {(cuuint64_t)(ROWB / 4), (cuuint64_t)nkv, (cuuint64_t)1 << 31};
    cuuint64_t strides[2] = {(cuuint64_t)ROWB, (cuuint64_t)nkv * ROWB};
    cuuint32_t box[3] = {(cuuint32_t)(ROWB / 4), 1, (cuuint32_t)SLOT};
    cuuint32_t es[3] = {1, 1, 1};
    return enc(m, CU_TENSOR_MAP_DATA_TYPE_UINT32, 3, const_cast<void *>(pool), dims, strides, box, es, CU_TENSOR_MAP_INTERLEAVE_NONE,
               CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

}  // namespace

// Ranges the scratch is made for: four to an SM and 8 heads (what an earlier kernel had resident), fewer when the batch is too small for ranges
// of at least floor_w units (same rule as in the kernel).  This kernel has one CTA per SM and uses at most a quarter of them on
// large batches; callers hold scratch of this size, and the rule below counts in it.
static int balanced_ranges(int nkv, int nh, int n_seq, int max_len, int floor_w) {
    const int X = nkv * ((nh / nkv + 7) / 8);
    const long long tiles = (max_len + UNIT - 1) / UNIT;
    const long long by_work = ((long long)n_seq * tiles + floor_w - 1) / floor_w, cap = 592 / X > 0 ? 592 / X : 1;
    return (int)(by_work < cap ? (by_work > 0 ? by_work : 1) : cap);
}
// By the longest context the call allows: ranges of at least 16 units (two tiles) and at most ~32 partials to a sequence, which the last CTA
// merges alone.  Short ranges (one tile, at most 16 partials) only while the long ones are fewer than 100: beyond that the SMs are busy.
// us of a step's attention, this rule | long ranges only | short ones always: 35B, 1 sequence of 256 tokens 13.0 | 13.8 | 13.0, of 2048 17.0 | 16.0 |
// 17.0, of 4096 17.8 | 17.8 | 18.3, of 32768 30.1 | 30.1 | 39.0; 2 of 1024 15.3 | 19.5 | 15.2; 4 of 256 18.9 | 21.0 | 19.0, of 16384 29.2 |
// 29.3 | 33.4; 8 of 1024 20.1 | 21.2 | 20.1, of 2048 23.4 | 23.3 | 19.4 (the line of 100 is not the best there), of 8192 28.8 | 28.7 | 28.6;
// 397B, 1 of 32768 35.8 | 35.7 | 43.5, 2 of 1024 18.3 | 23.8 | 18.3, 8 of 2048 29.9 | 29.8 | 24.0.
int gqa_decode_range_floor(int nkv, int nh, int n_seq, int max_len, bool short_ranges) {
    const int tiles = (max_len + UNIT - 1) / UNIT, w16 = (tiles + 15) / 16, w32 = (tiles + 31) / 32, w_long = w32 > 16 ? w32 : 16;
    const int X = nkv * ((nh / nkv + 7) / 8);
    if (!short_ranges || w16 > 16 || X * balanced_ranges(nkv, nh, n_seq, max_len, w_long) >= 100) return w_long;
    return w16 < 8 ? 8 : w16;
}
int gqa_decode_q8_slots(int nkv, int nh, int n_seq, int max_len, int range_floor) {
    return balanced_ranges(nkv, nh, n_seq, max_len, range_floor) + n_seq;
}

bool gqa_decode_q8_supported(const KvView &kv, int nh) {
    return kv.mode == ORNITH_KV_Q8_0 && kv.hd == HD && nh % kv.nkv == 0 && nh / kv.nkv <= 16 &&
           ((uintptr_t)kv.K % 16) == 0 && ((uintptr_t)kv.V % 16) == 0;
}

ornith_status launch_gqa_decode_q8_tc5(const DecodeArgs &a_in, int n_seq, cudaStream_t st) {
    DecodeArgs a = a_in;
    const int G = a.nh / a.kv.nkv;
    static bool configured_dev[ORN_MAX_DEVICES] = {};
    bool &configured = configured_dev[orn_device_index()];
    if (!configured) {
        ORN_TRY(orn_check(cudaFuncSetAttribute(k_gqa_decode_q8_tc5<8>, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM), "gqa decode smem opt-in"));
        ORN_TRY(orn_check(cudaFuncSetAttribute(k_gqa_decode_q8_tc5<16>, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM), "gqa decode smem opt-in"));
        configured = true;
    }
    // without the tensor maps (driver entry point missing) every slot is filled with row copies
    CUtensorMap mk, mv;
    memset(&mk, 0, sizeof mk);
    memset(&mv, 0, sizeof mv);
    const char *env = getenv("ORNITH_CUDA_DECODE_ROW_COPIES");
    const int tensor_copies = !(env && env[0] == '1') && rows_map(&mk, a.kv.K, a.kv.nkv) && rows_map(&mv, a.kv.V, a.kv.nkv);
    a.n_seq = n_seq;
    a.status = orn_status_word();
    // one CTA per SM, fewer where the ranges would be shorter than the floor
    const int all = 148 / a.kv.nkv > 0 ? 148 / a.kv.nkv : 1, have = balanced_ranges(a.kv.nkv, a.nh, n_seq, a.max_len, a.range_floor);
    // What a piece costs beside its rows, in units of 16 tokens: 24 (three tiles' time: queries, the pipeline's start, the partial) where
    // every SM has a range, so that a range with several sequences gets fewer rows.  4 / 24, us: 64 sequences of 1024 to 32768 tokens, 35B
    // 205 / 200, 40 of 1 to 3000 35.8 / 30.7, 200 of 1 to 600 of the 397B 88 / 70.  With fewer ranges than SMs a range is a piece or
    // part of one, and ranges would fall into the charge in front of a sequence (3 of 1 to 1000 tokens: 17.4 / 18.5).
    static int piece_cost = -1;                                   // ORNITH_CUDA_DECODE_PIECE_COST=<units> overrides it
    if (piece_cost < 0) { const char *e = getenv("ORNITH_CUDA_DECODE_PIECE_COST"); piece_cost = e ? atoi(e) : 99; if (piece_cost < 0 || piece_cost > 15) piece_cost = 99; }
    a.piece_cost = piece_cost < 99 ? piece_cost : have < all ? 4 : 24;
    const dim3 grid((unsigned)a.kv.nkv, (unsigned)(have < all ? have : all));
    return orn_check(G <= 8 ? orn_launch_dependent(k_gqa_decode_q8_tc5<8>, grid, dim3(NT), SMEM, st, a, mk, mv, tensor_copies)
                            : orn_launch_dependent(k_gqa_decode_q8_tc5<16>, grid, dim3(NT), SMEM, st, a, mk, mv, tensor_copies), "k_gqa_decode_q8_tc5");
}
