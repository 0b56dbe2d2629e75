/*
 * router_select.cuh — top-k selection on the BF16 codes of logits (c/moe.h:321-371): intervals
 * of them in the one-kernel decode path (exact_sum.cuh), known ones in the many-token router,
 * where a token has more candidates than a warp has lanes, and in the few-token router.
 *
 * The engine takes the top-k of its softmax PROBABILITIES.  exp and the division keep
 * the order of the BF16 logits whenever the logits near the top differ by 2^-18 or
 * more: two different BF16 values do unless both are smaller than 2^-10 in magnitude
 * (the spacing below 2^-10 is 2^-18, and 2^-10 itself is that far from the next smaller
 * one); probabilities above exp(-80) do not underflow.  So one small competitor is in
 * its place among the others, and what does not compete is below the top_k-th as long as
 * that one is not small itself.  Where order cannot be shown (`odd`), the caller runs the
 * engine's softmax on exact logits.
 */
#pragma once
#include "common.cuh"
#include "exact_dense.cuh"
#include "exact_sum.cuh"
#include "router.cuh"

namespace apus {

/* Order-preserving 16-bit key of a BF16 code (-0 counts as +0), and back. */
__device__ __forceinline__ uint32_t code_key(uint32_t code) {
    code &= 0xffffu;
    if (code == 0x8000u) code = 0;
    return code ^ ((code & 0x8000u) ? 0xffffu : 0x8000u);
}
__device__ __forceinline__ float key_value(uint32_t key) {
    return __uint_as_float((key ^ ((key & 0x8000u) ? 0x8000u : 0xffffu)) << 16);
}
constexpr uint32_t CODE_NEVER = 0xff80ff80u;         /* known to be -inf: out of the race */

struct Choice {
    uint32_t kkey;       /* key of the top_k-th low code */
    bool open;           /* the set depends on an interval */
    bool odd;            /* code order may not decide */
    bool any;            /* some competitor (or the shared gate) is not known */
};
/* One warp: sel[0 .. TK-1] = the TK experts with the largest low codes cd[0 .. E-1]
 * (lowest index first on ties).  Anything else whose high code reaches the TK-th low
 * code may belong there instead.  cd[E]: the shared gate's. */
__device__ __forceinline__ Choice rt_select(const uint32_t *cd, int E, int TK, int lane,
                                            int *sel) {
    /* keys: low code, then lowest index first; all different.  Up to 256 experts
     * they stay in registers. */
    constexpr int R = 8;
    uint32_t kr[R], best = 0, kth = 0;
    const bool regs = E <= 32 * R;
    auto key_of = [&](int e) { return (code_key(cd[e]) << 16) | (0xffffu - (uint32_t)e); };
    if (regs) {
#pragma unroll
        for (int i = 0; i < R; i++) {
            kr[i] = lane + 32 * i < E ? key_of(lane + 32 * i) : 0u;
            best = max(best, kr[i]);
        }
    } else {
#pragma unroll 1
        for (int e = lane; e < E; e += 32) best = max(best, key_of(e));
    }
#pragma unroll 1
    for (int i = 0; i < TK; i++) {
        kth = __reduce_max_sync(0xffffffffu, best);
        if (lane == 0) sel[i] = (int)(0xffffu - (kth & 0xffffu));
        if (regs) {
            best = 0;
#pragma unroll
            for (int j = 0; j < R; j++)
                if (kr[j] < kth) best = max(best, kr[j]);
        } else if (best == kth) {                        /* this lane's next one */
            best = 0;
            for (int e = lane; e < E; e += 32) {
                const uint32_t k = key_of(e);
                if (k < kth) best = max(best, k);
            }
        }
    }
    Choice c;
    c.kkey = kth >> 16;
    bool open = false, odd = false, any = false;
    int small = 0, zeros = 0;                            /* below 2^-10: nonzero, zero */
    float top = -INFINITY;
    uint32_t reach = 0;                                  /* bit i: expert lane + 32 i competes */
    if (regs) {
#pragma unroll
        for (int i = 0; i < R; i++)
            if (lane + 32 * i < E && code_key(cd[lane + 32 * i] >> 16) >= c.kkey) reach |= 1u << i;
    } else {
        for (int e = lane, i = 0; e < E; e += 32, i++)
            if (code_key(cd[e] >> 16) >= c.kkey) reach |= 1u << i;
    }
    for (; reach; reach &= reach - 1) {
        const int e = lane + 32 * (__ffs(reach) - 1);
        const uint32_t v = cd[e];
        const bool known = code_known(v);
        any |= !known;
        if (!known && key_of(e) < kth) open = true;      /* not among the chosen */
        const float lo = bf16lo(v), hi = bf16hi(v);
        const bool plain = fabsf(lo) >= 9.765625e-4f && fabsf(hi) >= 9.765625e-4f &&
                           (lo < 0.0f) == (hi < 0.0f);
        if (!(fabsf(lo) <= 32.0f && fabsf(hi) <= 32.0f)) odd = true;      /* or a NaN */
        if (known && (v & 0x7fffu) == 0)
            zeros++;
        else if (!plain)                                 /* an interval around zero counts */
            small++;
        top = fmaxf(top, hi);
    }
    __syncwarp();
    /* order-preserving integer of a float, for the integer reduction */
    const int ti = __float_as_int(top);
    const int tm = __reduce_max_sync(0xffffffffu, ti >= 0 ? ti : ti ^ 0x7fffffff);
    top = __int_as_float(tm >= 0 ? tm : tm ^ 0x7fffffff);
    const float kval = key_value(c.kkey);
    if (!(kval - top >= -80.0f) || fabsf(kval) < 9.765625e-4f) odd = true;
    /* equal zeros tie, as their probabilities do; beside another small one they may not */
    small = (int)__reduce_add_sync(0xffffffffu, (unsigned)small);
    zeros = (int)__reduce_add_sync(0xffffffffu, (unsigned)zeros);
    if (small > 1 || (small > 0 && zeros > 0)) odd = true;
    c.odd = __any_sync(0xffffffffu, odd);
    c.open = __any_sync(0xffffffffu, open);
    c.any = __any_sync(0xffffffffu, any) || c.odd || !code_known(cd[E]);
    return c;
}
/* the logits that need their chain: competitors whose code is open (all of them if
 * probabilities have to decide), and the shared gate */
__device__ __forceinline__ bool rt_needs(const uint32_t *cd, int e, int E, uint32_t kkey,
                                         bool odd) {
    return e <= E && !code_known(cd[e]) && (odd || e == E || code_key(cd[e] >> 16) >= kkey);
}
/* One warp, all codes of the selection known: its order and the renormalised weights
 * q_i / sum q in that order (c/moe.h:363-370).  The engine divides by the softmax
 * denominator S first, p_i = q_i / S, and S cancels only up to the rounding of the p_i and
 * of their sum: the quotients are within (2 TK + 2) 2^-24 of each other, and their BF16
 * codes can differ by a step where one of them lies that near a midpoint (5e-4 of the
 * weights for TK 8; 1.5e-5 do differ).  Returned: some quotient does.
 * A caller that knows every logit of the token runs the engine's steps then. */
__device__ __forceinline__ bool rt_weights(const uint32_t *cd, const int *sel, int TK, int lane,
                                           int32_t *idx_out, uint16_t *w_out) {
    const bool on = lane < TK;
    const int e = on ? sel[lane] : 0;
    const uint32_t c = cd[e] & 0xffffu;
    const uint32_t key = on ? (code_key(c) << 16) | (0xffffu - (uint32_t)e) : 0u;
    int rank = 0;
    for (int i = 0; i < TK; i++) rank += __shfl_sync(0xffffffffu, key, i) > key;
    const float m = key_value(__reduce_max_sync(0xffffffffu, key) >> 16);
    const float q = on ? (float)exp((double)__fsub_rn(bf16lo(c), m)) : 0.0f;
    float sw = 0.0f;
    for (int i = 0; i < TK; i++) {
        const int src = __ffs(__ballot_sync(0xffffffffu, on && rank == i)) - 1;
        sw = __fadd_rn(sw, __shfl_sync(0xffffffffu, q, src));
    }
    const float w = on ? __fdiv_rn(q, sw) : 0.0f;
    if (on) {
        idx_out[rank] = e;
        if (w_out) w_out[rank] = bf16_bits(w);
    }
    const int off = (int)(__float_as_uint(w) & 0xffffu) - 0x8000;
    return __any_sync(0xffffffffu, on && abs(off) <= 2 * TK + 2) != 0;
}

/* n <= G exact chains by one warp, chain c's result in lane c.  The dependent add per
 * step is the floor (4.6 cycles: 4.8 us for 2048 steps), and a full SM is bound by
 * issue: unpacking both operands in the chain's lane takes four slots a step for a
 * handful of busy lanes.  So the warp first multiplies together, a lane eight products
 * at a time, into G rows of 256 (256 elements of each chain, or 256 G of one), then a
 * chain's lane only loads and adds, while the next segment's operands are under way.  A
 * product rounded to fp32 and then added IS the engine's step, whether it is exact or
 * not.
 * wrow(c): weight row of chain c < n (called by all lanes together); xpiece(p): 16-byte
 * piece p of the token; buf: CH_ROW * G floats of shared memory, 16-byte aligned. */
constexpr int CH_ROW = 256 + 4;          /* the rows of eight lanes in different banks */
constexpr int CH_CHAINS = 4;             /* G of the one-kernel path */
constexpr int CH_BYTES = CH_CHAINS * CH_ROW * 4;
template <int G, typename WRow, typename XPiece>
__device__ __forceinline__ float warp_chains(int n, int K, int lane, float *buf, WRow wrow,
                                             XPiece xpiece) {
    const bool one = n == 1;
    const int seg = one ? 256 * G : 256;
    uint4 wq[G], xq[G];
    auto load = [&](int k0) {
#pragma unroll
        for (int g = 0; g < G; g++) {
            if (!one && g >= n) break;
            const uint16_t *w = wrow(one ? 0 : g);
            const int k = k0 + (one ? g * 256 : 0) + lane * 8;
            wq[g] = k < K ? ldg16(w + k) : make_uint4(0, 0, 0, 0);
            if (one || g == 0) xq[g] = k < K ? xpiece(k / 8) : make_uint4(0, 0, 0, 0);
        }
    };
    float acc = 0.0f;
    load(0);
#pragma unroll 1
    for (int k0 = 0; k0 < K; k0 += seg) {
        float xf[8];
#pragma unroll
        for (int g = 0; g < G; g++) {
            if (!one && g >= n) break;
            if (one || g == 0) unpack8(xq[g], xf);
            float wf[8];
            unpack8(wq[g], wf);
            /* the first four of every eight, then the second four: consecutive lanes
             * write consecutive pieces */
            float4 *d = reinterpret_cast<float4 *>(buf + g * CH_ROW) + lane;
            d[0] = make_float4(__fmul_rn(wf[0], xf[0]), __fmul_rn(wf[1], xf[1]),
                               __fmul_rn(wf[2], xf[2]), __fmul_rn(wf[3], xf[3]));
            d[32] = make_float4(__fmul_rn(wf[4], xf[4]), __fmul_rn(wf[5], xf[5]),
                                __fmul_rn(wf[6], xf[6]), __fmul_rn(wf[7], xf[7]));
        }
        __syncwarp();
        if (k0 + seg < K) load(k0 + seg);
        if (lane < n) {
#pragma unroll 1
            for (int r = 0, left = min(seg, K - k0) / 8; left > 0; r++, left -= 32) {
                const float4 *s = reinterpret_cast<const float4 *>(buf + (lane + r) * CH_ROW);
                const int last = min(left, 32) - 1;
                float4 a0 = s[0], b0 = s[32], a1 = s[min(1, last)], b1 = s[32 + min(1, last)];
#pragma unroll 4
                for (int i = 0; i <= last; i++) {        /* two eights (75 cycles) ahead */
                    const float4 a = a0, b = b0;
                    a0 = a1;
                    b0 = b1;
                    a1 = s[min(i + 2, last)];
                    b1 = s[32 + min(i + 2, last)];
                    acc = __fadd_rn(__fadd_rn(__fadd_rn(__fadd_rn(acc, a.x), a.y), a.z), a.w);
                    acc = __fadd_rn(__fadd_rn(__fadd_rn(__fadd_rn(acc, b.x), b.y), b.z), b.w);
                }
            }
        }
        __syncwarp();
    }
    return acc;
}
/* One chain per lane: weight row in global memory (16-byte pieces, sixteen of them under
 * way), token in fp32 in shared memory; K % 128 == 0.  Eight steps are 37 cycles of
 * dependent adds and 19 instructions for the warp, whatever its lanes are doing; no barrier
 * on the way, and up to 32 chains at once.  The better form where the SM has issue slots to
 * spare; warp_chains where it is full. */
template <bool FMA>
__device__ __forceinline__ float lane_chain(const uint16_t *w, const float *xs, int K) {
    constexpr int AHEAD = 16;
    uint4 q[AHEAD];
#pragma unroll
    for (int c = 0; c < AHEAD; c++) q[c] = ldg16(w + c * 8);
    float acc = 0.0f;
#pragma unroll 1
    for (int k = 0; k < K; k += AHEAD * 8) {
        const int next = k + AHEAD * 8 < K ? AHEAD * 8 : 0;
        const float4 *x4 = reinterpret_cast<const float4 *>(xs + k);
#pragma unroll
        for (int c = 0; c < AHEAD; c++) {
            float wf[8];
            unpack8(q[c], wf);
            q[c] = ldg16(w + k + next + c * 8);
            const float4 a = x4[2 * c], b = x4[2 * c + 1];
            const float xf[8] = {a.x, a.y, a.z, a.w, b.x, b.y, b.z, b.w};
#pragma unroll
            for (int j = 0; j < 8; j++) acc = exact_step<FMA>(wf[j], xf[j], acc);
        }
    }
    return acc;
}

}  // namespace apus
