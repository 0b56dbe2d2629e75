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
    uint32_t kr[R], best = 0, kth = 0, mine = 0;
    uint32_t far = 0;                       /* largest high key of those that are not known */
    const bool regs = E <= 32 * R;
    auto key_of = [&](uint32_t c, int e) { return (code_key(c) << 16) | (0xffffu - (uint32_t)e); };
    auto far_of = [&](uint32_t c) { return code_known(c) ? 0u : code_key(c >> 16) + 1u; };
    if (regs) {
#pragma unroll
        for (int i = 0; i < R; i++) {
            const uint32_t c = lane + 32 * i < E ? cd[lane + 32 * i] : CODE_NEVER;
            kr[i] = lane + 32 * i < E ? key_of(c, lane + 32 * i) : 0u;
            best = max(best, kr[i]);
            far = max(far, far_of(c));
        }
    } else {
#pragma unroll 1
        for (int e = lane; e < E; e += 32) {
            best = max(best, key_of(cd[e], e));
            far = max(far, far_of(cd[e]));
        }
    }
    uint32_t first = 0;
#pragma unroll 1
    for (int i = 0; i < TK; i++) {
        kth = __reduce_max_sync(0xffffffffu, best);
        if (lane == (i & 31)) mine = kth;
        if ((i & 31) == 31) {
            if (i == 31) first = __shfl_sync(0xffffffffu, mine, 0);
            sel[i - 31 + lane] = (int)(0xffffu - (mine & 0xffffu));
        }
        if (regs) {
            uint32_t b[R];
#pragma unroll
            for (int j = 0; j < R; j++) b[j] = kr[j] < kth ? kr[j] : 0u;
            best = max(max(max(b[0], b[1]), max(b[2], b[3])), max(max(b[4], b[5]), max(b[6], b[7])));
        } else if (best == kth) {                        /* this lane's next one */
            best = 0;
#pragma unroll 1
            for (int e = lane; e < E; e += 32) {
                const uint32_t k = key_of(cd[e], e);
                if (k < kth) best = max(best, k);
            }
        }
    }
    if (lane < (TK & 31)) sel[(TK & ~31) + lane] = (int)(0xffffu - (mine & 0xffffu));
    if (TK < 32) first = __shfl_sync(0xffffffffu, mine, 0);
    Choice c;
    c.kkey = kth >> 16;
    const float kval = key_value(c.kkey);
    /* Nearly always: every logit that reaches that far is known, so the chosen ones alone do,
     * and they lie between two values that leave nothing to doubt. */
    if (!__any_sync(0xffffffffu, far > c.kkey) && kval >= 9.765625e-4f &&
        key_value(first >> 16) <= 32.0f) {
        c.open = c.odd = false;
        c.any = !code_known(cd[E]);
        return c;
    }
    /* every expert whose high code reaches that far, without a branch: a lane's last one would
     * keep the others waiting */
    constexpr uint32_t SMALL = 0x3a80u, FAR = 0x4200u;   /* 2^-10 and 32 */
    uint32_t flags = 0, count = 0, topk = 0;     /* 1 any, 2 open, 4 odd; small ones, zeros << 16 */
    auto judge = [&](uint32_t w, uint32_t key) {
        const uint32_t hk = code_key(w >> 16), lm = w & 0x7fffu, hm = (w >> 16) & 0x7fffu;
        const bool in = hk >= c.kkey, known = code_known(w);
        topk = max(topk, hk);
        if (in && !known) flags |= key < kth ? 3u : 1u;  /* open: not among the chosen */
        if (in && max(lm, hm) > FAR) flags |= 4u;        /* or a NaN */
        const bool plain = min(lm, hm) >= SMALL && !((w ^ (w >> 16)) & 0x8000u);
        /* (an interval around zero counts as small) */
        if (in && !plain) count += known && lm == 0 ? 0x10000u : 1u;
    };
#pragma unroll 1
    for (int e = lane; e < E; e += 32) judge(cd[e], key_of(cd[e], e));
    __syncwarp();
    flags = __reduce_or_sync(0xffffffffu, flags);
    count = __reduce_add_sync(0xffffffffu, count);
    const float top = key_value(__reduce_max_sync(0xffffffffu, topk));
    if (!(kval - top >= -80.0f) || fabsf(kval) < 9.765625e-4f) flags |= 4u;
    /* equal zeros tie, as their probabilities do; beside another small one they may not */
    const uint32_t small = count & 0xffffu, zeros = count >> 16;
    if (small > 1 || (small > 0 && zeros > 0)) flags |= 4u;
    c.odd = flags & 4u;
    c.open = flags & 2u;
    c.any = (flags & 5u) || !code_known(cd[E]);
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
#pragma unroll 1
    for (int i = 0; i < TK; i++) rank += __shfl_sync(0xffffffffu, key, i) > key;
    const float m = key_value(__reduce_max_sync(0xffffffffu, key) >> 16);
    const float q = on ? (float)exp((double)__fsub_rn(bf16lo(c), m)) : 0.0f;
    float sw = 0.0f;
#pragma unroll 1
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
