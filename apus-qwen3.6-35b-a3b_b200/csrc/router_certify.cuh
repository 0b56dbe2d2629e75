/*
 * router_certify.cuh — exact expert selection for many tokens at a fraction of the
 * exact router's cost (c/moe.h:321-371 decides with BF16-rounded logits whose every
 * bit depends on a 2048-step sequential fp32 chain per expert, c/moe.h:289-291).
 *
 * Only the top_k experts of a token matter, and an expert far below the
 * top_k-th cannot become one because of rounding.  So:
 *
 *   1. fast logits a[t][e] for all experts come from the tensor cores (any
 *      summation order, prefill_gemm.cuh MODE 2);
 *   2. TokenCandidates bounds how far the fast and the exact value of a pair can
 *      be apart:  |a - z| <= B(t,e) = cbound * ||x_t||_2 * ||w_e||_2
 *      (both are fp32 summations of the same exactly representable products;
 *      a summation of n terms in any order errs by at most about n*u times the
 *      sum of their magnitudes, which Cauchy-Schwarz bounds by the norms;
 *      cbound leaves the tensor cores eight times the worst case of the
 *      sequential chain);
 *   3. with a8 the top_k-th largest fast logit, every expert with
 *          a + B(t,e)  >=  a8 - Bmax(t) - spacing
 *      is a CANDIDATE (spacing = one BF16 step at that magnitude, so that two
 *      values further apart than it cannot round to the same code).  Any
 *      other expert's exact rounded logit is strictly below those of top_k
 *      experts, whatever the rounding did: it cannot be selected;
 *   4. every candidate (10.6 of 256 at the real dimensions, 12.7 with a skewed router) and
 *      the shared-gate row get their exact chain, and |a - z| <= B is checked on
 *      every pair: ST_BOUND_VIOLATED is recorded if the assumption ever fails;
 *   5. selection and weights follow from the codes (router_select.cuh).
 *
 * Few tokens do 2-5 in one kernel, a warp per token (router_direct_kernel); many put the
 * tokens on lists, one per candidate expert, whose chains a second kernel walks 32 to a
 * warp before a third selects.
 */
#pragma once
#include <climits>

#include "common.cuh"
#include "decode_gemv.cuh"
#include "router_select.cuh"

namespace apus {

constexpr int RC_WARPS = 8;         /* tokens of a CTA: candidates and choice */
constexpr int ST_BOUND_VIOLATED = 5;
constexpr int RC_MAX_SLABS = 4;     /* K slices of the fast-logit GEMM */

struct CertifyArgs {
    const float *approx;            /* [nslab][T, E]: the fast logits are the sum */
    int nslab;
    const uint16_t *x, *w;          /* [T, K], [E, K] */
    const uint16_t *extra_row;      /* [K] shared-gate row (optional) */
    const float *wnorm;             /* [E + 1]: ||w_e||_2 rounded up; [E] = their max */
    int T, E, K, topk;
    float wmin, wmax;               /* smallest nonzero and largest |w| (0: unknown) */
    float wmin_extra, wmax_extra;
    float cbound;                   /* see above */
    /* between the three kernels */
    float *xnorm;                   /* [T] ||x_t||_2 rounded up; sign set: products round or
                                     * sums may overflow */
    int32_t *ncand;                 /* [T] candidates without the gate */
    uint16_t *cand;                 /* [T, RC_NARROW] */
    /* [T, code_pitch] codes of the candidates, then of the shared gate.  A token with at most
     * RC_NARROW of both has them side by side, the experts' numbers in `cand`; a token with
     * more has them at the experts' places, CODE_NEVER elsewhere. */
    uint32_t *codes;
    int code_pitch;
    uint32_t *lists;                /* [E, T] of each candidate expert: token << RC_SLOT_BITS |
                                     * place of the code in the token's row */
    int32_t *counts;                /* [E] at steps of RC_COUNT_STEP, cleared */
    int32_t *idx_out;               /* [T, topk] selection */
    uint16_t *w_out;                /* [T, topk] renormalised weights (optional) */
    uint16_t *extra_out;            /* [T] */
    int32_t *unit_hist;             /* [T / 256][E] += the selection (optional, place.cuh) */
    int *status;
    unsigned int *stats;            /* [0] += chains walked (optional) */
};
constexpr int RC_NARROW = 32;
constexpr int RC_SLOT_BITS = 11;    /* a slot is at most E <= 1024 */
constexpr size_t RC_MAX_T = (size_t)1 << (32 - RC_SLOT_BITS);
/* Counters that many tokens add to at once, one to a cache line: side by side, 87,000
 * additions to 256 counters took 10 of the candidates kernel's 38 us (8192 tokens). */
constexpr int RC_COUNT_STEP = 32;
inline int rc_code_pitch(int E) { return (E + 4) & ~3; }
/* the kernels' workspace behind the slabs, in 32-bit words */
inline size_t rc_list_words(size_t T, size_t E) {
    const size_t Tp = (T + 3) & ~(size_t)3;
    return 2 * Tp + T * (RC_NARROW / 2 + (size_t)rc_code_pitch((int)E) + E) + E * RC_COUNT_STEP;
}
inline void rc_carve(CertifyArgs &a, float *ws) {
    const size_t Tp = ((size_t)a.T + 3) & ~(size_t)3;
    a.xnorm = ws;
    a.ncand = reinterpret_cast<int32_t *>(ws + Tp);
    a.cand = reinterpret_cast<uint16_t *>(ws + 2 * Tp);
    a.code_pitch = rc_code_pitch(a.E);
    a.codes = reinterpret_cast<uint32_t *>(ws + 2 * Tp) + (size_t)a.T * (RC_NARROW / 2);
    a.lists = a.codes + (size_t)a.T * a.code_pitch;
    a.counts = reinterpret_cast<int32_t *>(a.lists + (size_t)a.E * a.T);
}

/* order-preserving integer key of a float (larger float -> larger int) */
__device__ __forceinline__ int rc_float_key(float f) {
    const int b = __float_as_int(f);
    return b >= 0 ? b : (b ^ 0x7fffffff);
}
__device__ __forceinline__ float rc_approx(const CertifyArgs &a, int t, int e) {
    float p[RC_MAX_SLABS];
#pragma unroll
    for (int sl = 0; sl < RC_MAX_SLABS; sl++)
        p[sl] = sl < a.nslab ? __ldg(&a.approx[((size_t)sl * a.T + t) * a.E + e]) : 0.0f;
    return (p[0] + p[1]) + (p[2] + p[3]);
}
/* phase boundaries of the first CTA (global timer, ns) for the profiling notes */
__device__ __forceinline__ void rc_mark(const CertifyArgs &a, int k) {
    if (a.stats && blockIdx.x == 0 && threadIdx.x == 0) {
        unsigned long long tm;
        asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(tm));
        a.stats[2 + k] = (unsigned int)tm;
    }
}

/* What is known of a token before its chains: one warp per token, E % 32 == 0, K % 256 == 0.
 * R: experts per lane, at least E / 32. */
template <int R>
struct TokenCandidates {
    unsigned in[R];                 /* bit l of in[i]: expert l + 32 i is a candidate */
    float av[R], wn[R];             /* this lane's fast logits and row norms */
    float xnorm, cb;
    int n;
    bool plain;                     /* no product rounds, no sum overflows */
    __device__ __forceinline__ void find(const CertifyArgs &a, int t, int lane) {
        /* ---- the token: norm, range of its values ---- */
        const int E = a.E, K = a.K, TK = a.topk;
        float ss = 0.0f;
        PackedRange range;
        const uint16_t *xr = a.x + (size_t)t * K + lane * 8;
#pragma unroll 8
        for (int k = 0; k < K; k += 256) {
            const uint4 v = ldg16(xr + k);
            float f[8], q[8];
            unpack8(v, f);
#pragma unroll
            for (int j = 0; j < 8; j++) q[j] = f[j] * f[j];
            ss += ((q[0] + q[1]) + (q[2] + q[3])) + ((q[4] + q[5]) + (q[6] + q[7]));
            range.fold8(v);
        }
        xnorm = norm_above(warp_sum(ss), K);
        const unsigned xlo = __reduce_min_sync(0xffffffffu, range.low()),
                       xhi = __reduce_max_sync(0xffffffffu, range.high());
        const float wn_max = __ldg(&a.wnorm[E]);
#pragma unroll
        for (int i = 0; i < R; i++)
            wn[i] = lane + 32 * i < E ? __ldg(&a.wnorm[lane + 32 * i]) : 0.0f;
        asm volatile("griddepcontrol.wait;" ::: "memory");

        /* ---- fast logits, the top_k-th of them, the candidates ---- */
#pragma unroll
        for (int i = 0; i < R; i++)
            av[i] = lane + 32 * i < E ? rc_approx(a, t, lane + 32 * i) : 0.0f;
        /* Keys of the values with their lowest bits replaced by the index: all different,
         * and the top_k-th of them, those bits cleared, is at most the top_k-th value. */
        constexpr unsigned IDX = R > 8 ? 1023u : 255u;
        unsigned kr[R], best = 0, kth = 0;
#pragma unroll
        for (int i = 0; i < R; i++) {
            const int e = lane + 32 * i;
            kr[i] = e < E ? (((unsigned)rc_float_key(av[i]) ^ 0x80000000u) & ~IDX) | (unsigned)e
                          : 0u;
            best = max(best, kr[i]);
        }
#pragma unroll 1
        for (int m = 0; m < TK; m++) {
            kth = __reduce_max_sync(0xffffffffu, best);
            best = 0;
#pragma unroll
            for (int i = 0; i < R; i++)
                if (kr[i] < kth) best = max(best, kr[i]);
        }
        const int wk = (int)((kth & ~IDX) ^ 0x80000000u);
        const float a8 = __int_as_float(wk >= 0 ? wk : wk ^ 0x7fffffff);
        cb = a.cbound * xnorm;
        const float bmax = cb * wn_max;
        /* one BF16 step at the magnitude of the values compared, rounded up */
        const float spacing = (fabsf(a8) + bmax) * (1.0f / 64.0f) + 1e-30f;
        const float thr = a8 - bmax - spacing;
        n = 0;
#pragma unroll
        for (int i = 0; i < R; i++) {
            in[i] = __ballot_sync(0xffffffffu, lane + 32 * i < E && av[i] + cb * wn[i] >= thr);
            n += __popc(in[i]);
        }
        plain = products_exact(a.wmin, a.wmax, xlo, xhi) && bmax < 1e30f &&
                (!a.extra_row || products_exact(a.wmin_extra, a.wmax_extra, xlo, xhi));
        if (a.stats && lane == 0) {
            const unsigned chains = (unsigned)n + (a.extra_row ? 1u : 0u);
            atomicAdd(&a.stats[0], chains);
            if (t == 0) a.stats[6] = chains;
        }
    }
};

/* grid = ceil(T / RC_WARPS) */
template <int R>
__global__ void __launch_bounds__(RC_WARPS * 32)
router_candidates_kernel(const __grid_constant__ CertifyArgs a) {
    /* the next kernel may be scheduled; this kernel's own wait for the fast-logit
     * GEMM comes after the token is read (it is the GEMM's input, complete
     * before it lets this kernel start) */
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    const int E = a.E, lane = threadIdx.x & 31, t = blockIdx.x * RC_WARPS + (threadIdx.x >> 5);
    rc_mark(a, 0);
    if (t >= a.T) {
        asm volatile("griddepcontrol.wait;" ::: "memory");
        return;
    }
    TokenCandidates<R> c;
    c.find(a, t, lane);
    int at[R];
#pragma unroll
    for (int i = 0; i < R; i++)
        at[i] = (c.in[i] >> lane) & 1u ? atomicAdd(&a.counts[(lane + 32 * i) * RC_COUNT_STEP], 1)
                                       : 0;
    const int gate = a.extra_row ? 1 : 0;
    const bool narrow = c.n + gate <= RC_NARROW;
    uint32_t *cd = a.codes + (size_t)t * a.code_pitch;
    int before = 0;
#pragma unroll
    for (int i = 0; i < R; i++) {
        const int e = lane + 32 * i;
        if ((c.in[i] >> lane) & 1u) {
            const int slot = narrow ? before + __popc(c.in[i] & ((1u << lane) - 1u)) : e;
            a.lists[(size_t)e * a.T + at[i]] = ((uint32_t)t << RC_SLOT_BITS) | (uint32_t)slot;
            if (narrow) a.cand[(size_t)t * RC_NARROW + slot] = (uint16_t)e;
        } else if (!narrow && e < E) {
            cd[e] = CODE_NEVER;
        }
        before += __popc(c.in[i]);
    }
    if (lane == 0) {
        a.xnorm[t] = c.plain ? c.xnorm : -c.xnorm;
        a.ncand[t] = c.n;
        if (!gate && !narrow) cd[E] = CODE_NEVER;
    }
    rc_mark(a, 1);
}

/* ---- chains --------------------------------------------------------------------------
 * A warp takes 32 tokens of one list, a chain to a lane, all on one weight row.  Rows
 * arrive 64 k at a time (cp.async, eight lanes per row, pitch 144 bytes: a lane reads its
 * own row without bank conflicts, the weights as a broadcast), CW_STAGES - 1 blocks ahead.
 *
 * Bound: the rows' way from L2, 4 KB per chain (8192 tokens, gate included: 95,424 chains and
 * 391 MB with an even router, 111,979 and 459 with a skewed one): 54 and 61 us by ncu, 7.2 and
 * 7.5 TB/s, issue slots 57-60 % taken, and much the same with 8, 11, 12 and 15 warps of
 * 5, 4, 4 and 3 blocks each; blocks of 32 k 10-20 % slower.  Routing of 8192 tokens, even
 * and skewed: 92 and 100 us; with one warp per token, an interval around each chain (the same
 * rows) and a chain only where the interval left a code open: 126 and 174 (1999 tokens: 45 and
 * 46, 49 and 62). */
constexpr int CW_WARPS = 15, CW_STAGES = 3, CW_BK = 64;
constexpr int CW_PITCH = CW_BK * 2 + 16;
constexpr int CW_STAGE = 33 * CW_PITCH;
constexpr int CW_LANES = CW_BK / 8, CW_ROWS = 32 / CW_LANES;   /* of a row; rows side by side */
inline size_t router_chains_smem(int E) {
    return (size_t)CW_WARPS * CW_STAGES * CW_STAGE + (size_t)(2 * E + 3) * 4;
}

template <bool FMA>
__device__ __forceinline__ float chain_tile(const uint16_t *const (&src)[CW_LANES], int n,
                                            const uint16_t *w, int K, unsigned char *ring,
                                            int lane) {
    const uint32_t dst =
        smem_u32(ring) + (uint32_t)(lane / CW_LANES * CW_PITCH + lane % CW_LANES * 16);
    const int nkb = K / CW_BK;
    int f_s = 0, s = 0;
    auto fetch = [&](int kb) {
        if (kb < nkb) {
            const uint32_t d = dst + (uint32_t)(f_s * CW_STAGE);
#pragma unroll
            for (int j = 0; j < CW_LANES; j++)
                if (lane / CW_LANES + CW_ROWS * j < n)
                    cp_async16_to(d + (uint32_t)(j * CW_ROWS * CW_PITCH), src[j] + kb * CW_BK);
            if (lane < CW_LANES) cp_async16_to(d + 32 * CW_PITCH, w + kb * CW_BK + lane * 8);
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
        if (++f_s == CW_STAGES) f_s = 0;
    };
    float acc = 0.0f;
#pragma unroll
    for (int kb = 0; kb < CW_STAGES - 1; kb++) fetch(kb);
#pragma unroll 1
    for (int kb = 0; kb < nkb; kb++) {
        asm volatile("cp.async.wait_group %0;" ::"n"(CW_STAGES - 2) : "memory");
        __syncwarp();                       /* block kb landed, block kb - 1 is used up */
        fetch(kb + CW_STAGES - 1);
        const unsigned char *b = ring + s * CW_STAGE, *xl = b + lane * CW_PITCH,
                            *wl = b + 32 * CW_PITCH;
        if (++s == CW_STAGES) s = 0;
#pragma unroll
        for (int c = 0; c < CW_BK / 8; c++) {
            float xf[8], wf[8];
            unpack8(*reinterpret_cast<const uint4 *>(xl + c * 16), xf);
            unpack8(*reinterpret_cast<const uint4 *>(wl + c * 16), wf);
#pragma unroll
            for (int j = 0; j < 8; j++) acc = exact_step<FMA>(wf[j], xf[j], acc);
        }
    }
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    __syncwarp();
    return acc;
}

/* persistent: one CTA per SM */
__global__ void __launch_bounds__(CW_WARPS * 32, 1)
router_chains_kernel(const __grid_constant__ CertifyArgs a) {
    extern __shared__ __align__(16) unsigned char cw_smem[];
    const int E = a.E, K = a.K, T = a.T;
    int *s_cnt = reinterpret_cast<int *>(cw_smem + (size_t)CW_WARPS * CW_STAGES * CW_STAGE),
        *s_first = s_cnt + E + 1;           /* [E + 1] tokens of a list, [E + 2] its first tile */
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    pdl_enter();
    for (int e = tid; e <= E; e += CW_WARPS * 32)
        s_cnt[e] = e < E ? min(__ldcg(&a.counts[e * RC_COUNT_STEP]), T) : a.extra_row ? T : 0;
    __syncthreads();
    if (warp == 0) {
        const int per = (E + 32) / 32, lo = min(lane * per, E + 1), hi = min(lo + per, E + 1);
        int n = 0;
        for (int e = lo; e < hi; e++) n += (s_cnt[e] + 31) / 32;
        int inc = n;
#pragma unroll
        for (int d = 1; d < 32; d <<= 1) {
            const int v = __shfl_up_sync(0xffffffffu, inc, d);
            if (lane >= d) inc += v;
        }
        int at = inc - n;
        for (int e = lo; e < hi; e++) {
            s_first[e] = at;
            at += (s_cnt[e] + 31) / 32;
        }
        if (lane == 31) s_first[E + 1] = inc;
    }
    __syncthreads();
    unsigned char *ring = cw_smem + (size_t)warp * CW_STAGES * CW_STAGE;
    const int n_tiles = s_first[E + 1];
#pragma unroll 1
    for (int tile = warp * gridDim.x + blockIdx.x; tile < n_tiles;
         tile += CW_WARPS * gridDim.x) {
        int e = 0;                          /* the last with s_first[e] <= tile */
        for (int hi = E; e < hi;) {
            const int mid = (e + hi + 1) >> 1;
            if (s_first[mid] <= tile) e = mid; else hi = mid - 1;
        }
        const int first = (tile - s_first[e]) * 32, n = min(32, s_cnt[e] - first);
        /* lanes beyond the list have no row of their own: their sums are not used */
        const int i = first + (lane < n ? lane : 0);
        const uint32_t entry = e == E ? 0u : __ldcg(&a.lists[(size_t)e * T + i]);
        const int t = e == E ? i : (int)(entry >> RC_SLOT_BITS);
        const int n_gate = e == E ? __ldcg(&a.ncand[t]) : 0;
        const uint16_t *src[CW_LANES];
#pragma unroll
        for (int j = 0; j < CW_LANES; j++)
            src[j] = a.x + (size_t)__shfl_sync(0xffffffffu, t, lane / CW_LANES + CW_ROWS * j) * K +
                     lane % CW_LANES * 8;
        const uint16_t *w = e == E ? a.extra_row : a.w + (size_t)e * K;
        const float xn = __ldcg(&a.xnorm[t]);
        const float fast = e < E ? rc_approx(a, t, e) : 0.0f;
        const float bound = e < E ? a.cbound * fabsf(xn) * __ldg(&a.wnorm[e]) : 0.0f;
        const bool odd = __float_as_int(xn) < 0;
        const float z = __any_sync(0xffffffffu, odd) ? chain_tile<false>(src, n, w, K, ring, lane)
                                                     : chain_tile<true>(src, n, w, K, ring, lane);
        if (lane < n) {
            /* (values that may overflow on the way are outside the bound's derivation) */
            if (e < E && bound < 1e30f && !(fabsf(z - fast) <= bound))
                set_status(a.status, ST_BOUND_VIOLATED);
            const int slot = e < E ? (int)(entry & ((1u << RC_SLOT_BITS) - 1u))
                                   : n_gate < RC_NARROW ? n_gate : E;
            a.codes[(size_t)t * a.code_pitch + slot] = 0x10001u * bf16_bits(z);
        }
    }
}

/* ---- selection and weights: one warp per token ----------------------------------------
 * A narrow token has a candidate to a lane: expert e and code, n of them.  What rt_select and
 * rt_weights do, with every code known, without shared memory.  Returned: code order decides,
 * and chosen is this lane's expert, if any.
 *
 * Code order decides (router_select.cuh) where every two different neighbours are 2^-18 apart
 * as the engine's exp takes them (less the largest logit, rounded), from the largest down to
 * the first below the top_k-th code: any of its equals may be the chosen one, and what comes
 * behind them must not have their probability.  What is no candidate is far enough below if the
 * top_k-th is not small, or by the margin that it was left out with: 2^-6 bmax less the two
 * roundings to BF16, 2^-17 and more.  (Softmax for every token with a small top_k-th made
 * a skewed batch wait 7 us for a few of them.) */
__device__ __forceinline__ bool choose_narrow(int n, int e, uint32_t code, float bmax, int TK,
                                              int lane, int32_t *idx, uint16_t *wo,
                                              int &chosen) {
    const bool on = lane < n;
    const uint32_t key = on ? (code_key(code) << 16) | (0xffffu - (uint32_t)e) : 0u;
    int rank = 0;
    uint32_t next = 0;                                   /* the key behind this one */
#pragma unroll 1
    for (int i = 0; i < n; i++) {
        const uint32_t k = __shfl_sync(0xffffffffu, key, i);
        rank += k > key;
        if (k < key) next = max(next, k);
    }
    const unsigned last = __ballot_sync(0xffffffffu, on && rank == TK - 1);
    const uint32_t kkey = __shfl_sync(0xffffffffu, key, last ? __ffs(last) - 1 : 0) >> 16;
    const float top = key_value(__reduce_max_sync(0xffffffffu, key) >> 16),
                kval = key_value(kkey), v = bf16lo(code);
    const bool sel = on && rank < TK;
    const bool close = next && (next >> 16) != (key >> 16) &&
                       !(__fsub_rn(v, top) - __fsub_rn(key_value(next >> 16), top) >=
                         3.814697265625e-6f);
    const bool odd = !last || !(kval - top >= -80.0f) ||
                     (fabsf(kval) < 9.765625e-4f && bmax < 9.765625e-4f) ||
                     (on && (key >> 16) >= kkey && (close || !(fabsf(v) <= 32.0f)));
    if (__any_sync(0xffffffffu, odd)) return false;
    const float q = sel ? (float)exp((double)__fsub_rn(v, top)) : 0.0f;
    float sw = 0.0f;
#pragma unroll 1
    for (int i = 0; i < TK; i++) {
        const int src = __ffs(__ballot_sync(0xffffffffu, sel && rank == i)) - 1;
        sw = __fadd_rn(sw, __shfl_sync(0xffffffffu, q, src));
    }
    if (sel) {
        idx[rank] = chosen = e;
        if (wo) wo[rank] = bf16_bits(__fdiv_rn(q, sw));
    }
    return true;
}
/* Of all experts: cd[0 .. E] as rt_select has them, in shared memory. */
__device__ __forceinline__ bool choose_wide(const uint32_t *cd, int E, int TK, int lane, int *sel,
                                            int32_t *idx, uint16_t *wo, int &chosen) {
    if (rt_select(cd, E, TK, lane, sel).odd) return false;
    __syncwarp();
    rt_weights(cd, sel, TK, lane, idx, wo);
    if (lane < TK) chosen = sel[lane];
    return true;
}
/* The engine's softmax on the exact logits of the candidates and the rounded fast ones of the
 * rest, which only enter its denominator.  cd: E words of shared memory; of a wide token, its
 * codes. */
__device__ __forceinline__ void choose_softmax(const CertifyArgs &a, int t, uint32_t *cd,
                                               bool narrow, int n, int e, uint32_t code, int lane,
                                               int32_t *idx, uint16_t *wo, int &chosen) {
    float *p = reinterpret_cast<float *>(cd);
#pragma unroll 4
    for (int i = lane; i < a.E; i += 32)
        p[i] = narrow || cd[i] == CODE_NEVER ? bf16_round(rc_approx(a, t, i)) : bf16lo(cd[i]);
    __syncwarp();
    if (narrow && lane < n) p[e] = bf16lo(code);
    __syncwarp();
    router_softmax_topk(p, a.E, a.topk, lane, idx, wo);
    __syncwarp();
    if (lane < a.topk) chosen = idx[lane];
}
__device__ __forceinline__ void count_choice(const CertifyArgs &a, int t, int chosen) {
    if (a.unit_hist && chosen >= 0)
        atomicAdd(&a.unit_hist[(size_t)(t / 256) * a.E + chosen], 1);
}

/* Dynamic shared memory: one row of codes per warp. */
inline size_t router_choose_smem(int E) { return (size_t)RC_WARPS * rc_code_pitch(E) * 4; }
__global__ void __launch_bounds__(RC_WARPS * 32)
router_choose_kernel(const __grid_constant__ CertifyArgs a) {
    extern __shared__ __align__(16) unsigned char ch_smem[];
    __shared__ int s_sel[RC_WARPS][32];
    const int E = a.E, TK = a.topk, lane = threadIdx.x & 31, warp = threadIdx.x >> 5,
              t = blockIdx.x * RC_WARPS + warp;
    pdl_enter();
    if (t >= a.T) return;
    rc_mark(a, 2);
    const uint32_t *codes = a.codes + (size_t)t * a.code_pitch;
    const int n = __ldcg(&a.ncand[t]), gate = a.extra_row ? 1 : 0;
    uint32_t code = __ldcg(codes + lane) & 0xffffu;
    const int e = __ldcg(&a.cand[(size_t)t * RC_NARROW + lane]);
    const float xnorm = __ldcg(&a.xnorm[t]), bmax = a.cbound * xnorm * __ldg(&a.wnorm[E]);
    const bool plain = __float_as_int(xnorm) >= 0, narrow = n + gate <= RC_NARROW;
    int32_t *idx = a.idx_out + (size_t)t * TK;
    uint16_t *wo = a.w_out ? a.w_out + (size_t)t * TK : nullptr;
    uint32_t *cd = reinterpret_cast<uint32_t *>(ch_smem) + warp * a.code_pitch;
    int chosen = -1;
    bool done = false;
    if (narrow) {
        if (gate && lane == n) a.extra_out[t] = (uint16_t)code;
        if (plain) done = choose_narrow(n, e, code, bmax, TK, lane, idx, wo, chosen);
    } else {
        for (int i = lane; i <= E; i += 32) cd[i] = __ldcg(codes + i);
        __syncwarp();
        if (gate && lane == 0) a.extra_out[t] = (uint16_t)cd[E];
        if (plain) done = choose_wide(cd, E, TK, lane, s_sel[warp], idx, wo, chosen);
    }
    if (!done) choose_softmax(a, t, cd, narrow, n, e, code, lane, idx, wo, chosen);
    count_choice(a, t, chosen);
    rc_mark(a, 3);
}

/* ---- few tokens: all three steps in one kernel -----------------------------------------
 * One warp, and one CTA, per token; its candidates' chains one to a lane, rows straight from
 * L2.  The longest chain and four round trips bound it, whatever runs beside it: there is
 * nothing to share yet between the tokens of an expert.  Dynamic shared memory: the token in
 * fp32, codes, candidates. */
inline size_t router_direct_smem(int E, int K) {
    return (size_t)K * 4 + (size_t)rc_code_pitch(E) * 6 + 16;
}
template <int R>
__global__ void __launch_bounds__(32)
router_direct_kernel(const __grid_constant__ CertifyArgs a) {
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");   /* as above */
    extern __shared__ __align__(16) unsigned char rd_smem[];
    __shared__ int s_sel[32];
    const int E = a.E, K = a.K, TK = a.topk, lane = threadIdx.x, t = blockIdx.x;
    float *xs = reinterpret_cast<float *>(rd_smem);
    uint32_t *cd = reinterpret_cast<uint32_t *>(xs + K);
    uint16_t *cand = reinterpret_cast<uint16_t *>(cd + a.code_pitch);
    rc_mark(a, 0);
    TokenCandidates<R> c;
    c.find(a, t, lane);
    int before = 0;
#pragma unroll
    for (int i = 0; i < R; i++) {
        const int e = lane + 32 * i;
        if ((c.in[i] >> lane) & 1u)
            cand[before + __popc(c.in[i] & ((1u << lane) - 1u))] = (uint16_t)e;
        if (e < E) cd[e] = CODE_NEVER;
        before += __popc(c.in[i]);
    }
    const int gate = a.extra_row ? 1 : 0;
    if (lane == 0) {
        cd[E] = CODE_NEVER;
        if (gate) cand[c.n] = (uint16_t)E;
    }
    for (int k = lane * 8; k < K; k += 256) {
        float f[8];
        unpack8(ldg16(a.x + (size_t)t * K + k), f);
        float4 *d4 = reinterpret_cast<float4 *>(xs + k);
        d4[0] = make_float4(f[0], f[1], f[2], f[3]);
        d4[1] = make_float4(f[4], f[5], f[6], f[7]);
    }
    __syncwarp();
    rc_mark(a, 1);
    const int n_eval = c.n + gate;
    const bool narrow = n_eval <= RC_NARROW;
    uint32_t code = 0;
    int mine = 0;
#pragma unroll 1
    for (int c0 = 0; c0 < n_eval; c0 += 32) {
        const bool on = c0 + lane < n_eval;
        mine = cand[on ? c0 + lane : c0];                /* the others read along */
        const uint16_t *w = mine == E ? a.extra_row : a.w + (size_t)mine * K;
        const float z = c.plain ? lane_chain<true>(w, xs, K) : lane_chain<false>(w, xs, K);
        code = bf16_bits(z);
        if (on) {
            const float bound = mine < E ? c.cb * __ldg(&a.wnorm[mine]) : 0.0f;
            if (mine < E && bound < 1e30f && !(fabsf(z - rc_approx(a, t, mine)) <= bound))
                set_status(a.status, ST_BOUND_VIOLATED);
            cd[mine] = 0x10001u * code;
        }
    }
    __syncwarp();
    rc_mark(a, 2);
    if (gate && lane == 0) a.extra_out[t] = (uint16_t)cd[E];
    int32_t *idx = a.idx_out + (size_t)t * TK;
    uint16_t *wo = a.w_out ? a.w_out + (size_t)t * TK : nullptr;
    int chosen = -1;
    const bool done =
        c.plain && (narrow ? choose_narrow(c.n, mine, code, c.cb * __ldg(&a.wnorm[E]), TK, lane,
                                           idx, wo, chosen)
                           : choose_wide(cd, E, TK, lane, s_sel, idx, wo, chosen));
    if (!done) choose_softmax(a, t, cd, false, 0, 0, 0, lane, idx, wo, chosen);
    count_choice(a, t, chosen);
    rc_mark(a, 3);
}

/* ||w_e||_2 per row, rounded up; out[E] = the largest.  One warp per row. */
__global__ void __launch_bounds__(256)
row_norm_kernel(const uint16_t *__restrict__ w, int E, int K, float *__restrict__ out) {
    const int warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31;
    if (warp >= E) return;
    float ss = 0.f;
    for (int k = lane; k < K; k += 32) {
        const float v = bf16_f32(w[(size_t)warp * K + k]);
        ss = fmaf(v, v, ss);
    }
    ss = warp_sum(ss);
    const float n = norm_above(ss, K);
    if (lane == 0) {
        out[warp] = n;
        atomicMax(reinterpret_cast<unsigned int *>(out + E), __float_as_uint(n));
    }
}

}  // namespace apus
