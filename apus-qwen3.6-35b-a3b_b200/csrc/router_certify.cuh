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
 *   2. this kernel bounds how far the fast and the exact value of a pair can
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
 *   4. candidates (about top_k + 2 of 256 at the real dimensions) and the
 *      shared-gate row get an interval that nearly always pins the BF16 code of
 *      their exact chain (exact_sum.cuh), the few that it does not and that matter
 *      get the chain itself;
 *   5. the kernel checks |a - z| <= B on every pair it evaluates and
 *      records ST_BOUND_VIOLATED if the assumption ever fails.
 *
 * Selection and weights then follow from the codes (router_select.cuh).
 *
 * One warp per token from end to end.  Bound: instruction issue for many tokens
 * (about 200 per candidate and warp), latency for few; so a lane keeps its 64 values
 * of the token as fp32 in registers, the eights of a row are independent, and the
 * lanes' partial results meet in shared memory, where one lane per candidate adds
 * them up.  Candidate rows (4 KB each, from L2) arrive through a ring of D slots per
 * warp.  (A chain per candidate, one per lane, took 33 us at 512 tokens, 55 at 1999
 * and 148 at 8192; up to two tokens an SM it is what runs, one chain to a lane, since
 * an interval costs more than the chains it saves there.)
 */
#pragma once
#include <climits>

#include "common.cuh"
#include "decode_gemv.cuh"
#include "router_select.cuh"

namespace apus {

constexpr int RC_WARPS = 2;         /* tokens of a CTA at most: a token with chains to walk takes
                                     * twice as long as one without, and holds up its CTA's slot */
constexpr int RC_MAX_E = 1024;
constexpr int ST_BOUND_VIOLATED = 5;
constexpr int RC_MAX_SLABS = 4;     /* K slices of the fast-logit GEMM */

struct CertifyArgs {
    const float *approx;            /* [nslab][T, E]: the fast logits are the sum */
    int nslab;
    const uint16_t *x, *w;          /* [T, K], [E, K] */
    const uint16_t *extra_row;      /* [K] shared-gate row (optional) */
    const float *wnorm;             /* [E + 1]: ||w_e||_2 rounded up; [E] = their max */
    float wnorm_extra;              /* the same of extra_row */
    int T, E, K, topk;
    float wmin, wmax;               /* smallest nonzero and largest |w| (0: unknown) */
    float wmin_extra, wmax_extra;
    float cbound;                   /* see above */
    int32_t *idx_out;               /* [T, topk] selection */
    uint16_t *w_out;                /* [T, topk] renormalised weights (optional) */
    uint16_t *extra_out;            /* [T] */
    int32_t *unit_hist;             /* [T / 256][E] += the selection (optional, place.cuh) */
    int *status;
    unsigned int *stats;            /* [0] += logits resolved exactly (optional) */
    int direct;                     /* every candidate's chain, no intervals (LANES) */
    LaneRow lr;
};

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

constexpr int RC_BATCH = 12;        /* candidates whose partial results meet at once */
/* Dynamic shared memory, per warp: D row slots, partial sums, codes [E + 1],
 * candidates [E + 1]. */
inline size_t router_certify_smem(int E, int K, int slots) {
    const size_t ring = (size_t)slots * LaneRow(K).bytes();   /* later the chains' products */
    return (ring > CH_BYTES ? ring : CH_BYTES) + RC_BATCH * 33 * 2 * 4 +
           (size_t)((E + 4) & ~3) * 4 + (size_t)((E + 8) & ~7) * 2;
}

/* grid = ceil(T / warps); E % 32 == 0, K % 256 == 0.  R: experts per lane, at least
 * E / 32; NU: 16-byte pieces of a lane's chunk that are kept in registers (K / 256),
 * 0: any K, the token is read again for each candidate; D: ring slots; LANES: chains one to
 * a lane (lane_chain) and not with the warp's help (warp_chains). */
template <int R, int NU, int D, bool LANES>
__global__ void __launch_bounds__(RC_WARPS * 32, 16 / RC_WARPS)
router_certify_kernel(const __grid_constant__ CertifyArgs a) {
    /* the next kernel may be scheduled; this kernel's own wait for the fast-logit
     * GEMM comes after the token is staged (it is the GEMM's input, complete
     * before it lets this kernel start) */
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    extern __shared__ __align__(16) unsigned char rc_smem[];
    __shared__ int s_sel[RC_WARPS][32];
    const int E = a.E, K = a.K, TK = a.topk;
    const LaneRow lr = a.lr;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
    const int t = blockIdx.x * nw + warp;
    const int row_bytes = lr.bytes(), ring_bytes = max(D * row_bytes, CH_BYTES);
    const int cd_n = (E + 4) & ~3, cand_n = (E + 8) & ~7;
    unsigned char *slots = rc_smem + (size_t)warp * ring_bytes;
    float *part = reinterpret_cast<float *>(rc_smem + (size_t)nw * ring_bytes) +
                  warp * (RC_BATCH * 33 * 2);
    uint32_t *cd = reinterpret_cast<uint32_t *>(rc_smem + (size_t)nw * ring_bytes) +
                   nw * (RC_BATCH * 33 * 2) + warp * cd_n;
    uint16_t *cand = reinterpret_cast<uint16_t *>(rc_smem + (size_t)nw * ring_bytes +
                                                  (size_t)nw * (RC_BATCH * 33 * 2 + cd_n) * 4) +
                     warp * cand_n;
    auto mark = [&](int k) {
        /* phase boundaries of the first warp (global timer, ns) for the profiling notes */
        if (a.stats && blockIdx.x == 0 && threadIdx.x == 0) {
            unsigned long long tm;
            asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(tm));
            a.stats[2 + k] = (unsigned int)tm;
        }
    };
    mark(0);
    if (t >= a.T) {
        asm volatile("griddepcontrol.wait;" ::: "memory");
        return;
    }
    /* ---- the token: norm, range of its values ---- */
    const uint32_t slot0 = smem_u32(slots);
    const unsigned char *x_lane = slots + lane * lr.pitch;
    lane_row_fetch(slot0, a.x + (size_t)t * K, lr, K, lane);
    cp_async_done();
    __syncwarp();
    unsigned long long xp[NU > 0 ? NU * 4 : 1];          /* pairs of values */
    float ss = 0.0f;
    unsigned int xlo = 0x7f800000u, xhi = 0;
    auto square = [&](const uint4 v, float (&f)[8]) {
        unpack8(v, f);
        float q[8];
#pragma unroll
        for (int j = 0; j < 8; j++) q[j] = f[j] * f[j];
        ss += ((q[0] + q[1]) + (q[2] + q[3])) + ((q[4] + q[5]) + (q[6] + q[7]));
        fold_range8(v, xlo, xhi);
    };
    if (NU > 0) {
#pragma unroll
        for (int u = 0; u < NU; u++) {
            float f[8];
            square(*reinterpret_cast<const uint4 *>(x_lane + u * 16), f);
#pragma unroll
            for (int j = 0; j < 4; j++) xp[u * 4 + j] = pack_f32x2(f[2 * j], f[2 * j + 1]);
        }
    } else {
        for (int u = 0; u < lr.nu; u++) {
            float f[8];
            square(*reinterpret_cast<const uint4 *>(x_lane + u * 16), f);
        }
    }
    const float xnorm = norm_above(warp_sum(ss), K);
    xlo = __reduce_min_sync(0xffffffffu, xlo);
    xhi = __reduce_max_sync(0xffffffffu, xhi);
    const bool ok = products_exact(a.wmin, a.wmax, xlo, xhi),
               ok_extra = products_exact(a.wmin_extra, a.wmax_extra, xlo, xhi);
    const float wn_max = __ldg(&a.wnorm[E]);
    float av[R], wn[R];
#pragma unroll
    for (int i = 0; i < R; i++) wn[i] = lane + 32 * i < E ? __ldg(&a.wnorm[lane + 32 * i]) : 0.0f;
    asm volatile("griddepcontrol.wait;" ::: "memory");

    /* ---- fast logits, the top_k-th of them, the candidates ---- */
#pragma unroll
    for (int i = 0; i < R; i++) av[i] = lane + 32 * i < E ? rc_approx(a, t, lane + 32 * i) : 0.0f;
    /* Keys of the values with their lowest bits replaced by the index: all different,
     * and the top_k-th of them, those bits cleared, is at most the top_k-th value. */
    constexpr unsigned IDX = R > 8 ? 1023u : 255u;
    unsigned kr[R], best = 0, kth = 0;
#pragma unroll
    for (int i = 0; i < R; i++) {
        const int e = lane + 32 * i;
        kr[i] = e < E ? (((unsigned)rc_float_key(av[i]) ^ 0x80000000u) & ~IDX) | (unsigned)e : 0u;
        best = max(best, kr[i]);
    }
#pragma unroll 1
    for (int n = 0; n < TK; n++) {
        kth = __reduce_max_sync(0xffffffffu, best);
        best = 0;
#pragma unroll
        for (int i = 0; i < R; i++)
            if (kr[i] < kth) best = max(best, kr[i]);
    }
    const int wk = (int)((kth & ~IDX) ^ 0x80000000u);
    const float a8 = __int_as_float(wk >= 0 ? wk : wk ^ 0x7fffffff);
    const float cb = a.cbound * xnorm;
    const float bmax = cb * wn_max;
    /* one BF16 step at the magnitude of the values compared, rounded up */
    const float spacing = (fabsf(a8) + bmax) * (1.0f / 64.0f) + 1e-30f;
    const float thr = a8 - bmax - spacing;
    int n_cand = 0;
#pragma unroll
    for (int i = 0; i < R; i++) {
        const int e = lane + 32 * i;
        const bool in = e < E && av[i] + cb * wn[i] >= thr;
        const unsigned m = __ballot_sync(0xffffffffu, in);
        if (in) cand[n_cand + __popc(m & ((1u << lane) - 1u))] = (uint16_t)e;
        /* a candidate's fast logit waits in its code's place */
        if (e < E) cd[e] = in ? __float_as_uint(av[i]) : CODE_NEVER;
        n_cand += __popc(m);
    }
    if (lane == 0) {
        if (a.extra_row) cand[n_cand] = (uint16_t)E;
        cd[E] = a.extra_row ? 0u : CODE_NEVER;
    }
    const int n_eval = n_cand + (a.extra_row ? 1 : 0);
    __syncwarp();
    mark(1);

    /* ---- their chains, or intervals ---- */
    auto row_of = [&](int e) { return e == E ? a.extra_row : a.w + (size_t)e * K; };
    auto xpiece = [&](int p) { return ldg16(a.x + (size_t)t * K + p * 8); };
    auto token_f32 = [&](float *d) {
        for (int p = lane; p < K / 8; p += 32) {
            float f[8];
            unpack8(xpiece(p), f);
            float4 *d4 = reinterpret_cast<float4 *>(d + p * 8);
            d4[0] = make_float4(f[0], f[1], f[2], f[3]);
            d4[1] = make_float4(f[4], f[5], f[6], f[7]);
        }
        __syncwarp();
    };
    int f_slot = 0;
    /* Few tokens: a chain for every candidate at once, no intervals.  (Values large enough
     * to overflow, or NaN, take the intervals, which leave those open.) */
    const bool direct = LANES && a.direct && ok && (ok_extra || !a.extra_row) && bmax < 1e30f;
    if (direct) {
        float *xs = reinterpret_cast<float *>(slots);
        token_f32(xs);
#pragma unroll 1
        for (int c0 = 0; c0 < n_eval; c0 += 32) {
            const bool mine = c0 + lane < n_eval;
            const int e = cand[mine ? c0 + lane : c0];       /* the others read along */
            const float z = lane_chain<true>(row_of(e), xs, K);
            if (mine) {
                if (e < E && !(fabsf(z - __uint_as_float(cd[e])) <= cb * __ldg(&a.wnorm[e])))
                    set_status(a.status, ST_BOUND_VIOLATED);
                cd[e] = 0x10001u * bf16_bits(z);
            }
        }
        __syncwarp();
    }
    auto fetch = [&](int c) {
        if (c < n_eval)
            lane_row_fetch(slot0 + (uint32_t)(f_slot * row_bytes), row_of(cand[c]), lr, K, lane);
        if (++f_slot == D) f_slot = 0;
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    const uint16_t *xg = a.x + (size_t)t * K + (size_t)lane * lr.nu * 8;   /* NU == 0 */
    if (!direct)
#pragma unroll 1
        for (int c = 0; c < D; c++) fetch(c);
    int slot = 0;
#pragma unroll 1
    for (int c0 = direct ? n_eval : 0; c0 < n_eval; c0 += RC_BATCH) {
        const int n = min(RC_BATCH, n_eval - c0);
#pragma unroll 1
        for (int c = 0; c < n; c++) {
            asm volatile("cp.async.wait_group %0;" ::"n"(D - 1) : "memory");
            __syncwarp();
            const unsigned char *wl = slots + slot * row_bytes + lane * lr.pitch;
            if (++slot == D) slot = 0;
            float run = 0.0f, runs = 0.0f;
            auto eight = [&](const uint4 v, const unsigned long long *f) {
                float wf[8];
                unpack8(v, wf);
                unsigned long long q;                    /* even elements, odd elements */
                asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(q) : "l"(pack_f32x2(wf[0], wf[1])), "l"(f[0]));
#pragma unroll
                for (int j = 1; j < 4; j++)
                    asm("fma.rn.f32x2 %0, %1, %2, %0;"
                        : "+l"(q) : "l"(pack_f32x2(wf[2 * j], wf[2 * j + 1])), "l"(f[j]));
                runs += fabsf(run);
                run += __uint_as_float((unsigned)q) + __uint_as_float((unsigned)(q >> 32));
            };
            if (NU > 0) {
#pragma unroll
                for (int u = 0; u < NU; u++)
                    eight(*reinterpret_cast<const uint4 *>(wl + u * 16), xp + u * 4);
            } else {
#pragma unroll 1
                for (int u = 0; u < lr.nu; u++) {
                    float f[8];
                    unsigned long long fp[4];
                    unpack8(ldg16(xg + u * 8), f);
#pragma unroll
                    for (int j = 0; j < 4; j++) fp[j] = pack_f32x2(f[2 * j], f[2 * j + 1]);
                    eight(*reinterpret_cast<const uint4 *>(wl + u * 16), fp);
                }
            }
            part[c * 33 + lane] = run;
            part[(RC_BATCH + c) * 33 + lane] = runs;
            __syncwarp();                      /* the slot is read out */
            fetch(c0 + c + D);
        }
        /* Lane c: the interval of candidate c.  Error terms as in exact_sum.cuh, the
         * lanes' sums added in order: 8 nu |sum before the lane| (+ 1 for the add)
         * and 8 (+ 1) |running sum| per eight, 8 (+ 4: two chains of four and their
         * sum) of the magnitudes, which Cauchy-Schwarz bounds by the norms. */
        if (lane < n) {
            const int e = cand[c0 + lane];
            const float wn_e = e == E ? a.wnorm_extra : __ldg(&a.wnorm[e]);
            float s = 0.0f, starts = 0.0f, runs = 0.0f;
#pragma unroll 8
            for (int l = 0; l < 32; l++) {
                starts += fabsf(s);
                s += part[lane * 33 + l];
                runs += part[(RC_BATCH + lane) * 33 + l];
            }
            const float err = (starts * (8.0f * lr.nu + 1.0f) + 9.0f * runs +
                               12.0f * wn_e * xnorm) * (1.05f * 5.9604645e-8f);
            if (e < E && !(fabsf(s - __uint_as_float(cd[e])) <= cb * wn_e))
                set_status(a.status, ST_BOUND_VIOLATED);
            const float lo = __fadd_rd(s, -err), hi = __fadd_ru(s, err);
            cd[e] = (e == E ? ok_extra : ok) && lo <= hi
                        ? (uint32_t)bf16_bits(lo) | ((uint32_t)bf16_bits(hi) << 16)
                        : CODE_UNKNOWN;
        }
        __syncwarp();
    }
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    __syncwarp();

    /* ---- selection; chains where an interval leaves something open ---- */
    int *sel = s_sel[warp];
    Choice ch = rt_select(cd, E, TK, lane, sel);
    if (ch.any) {
        float *buf = reinterpret_cast<float *>(slots);
        if (LANES) {
            token_f32(buf);
            resolve_lanes(cd, cand, n_eval, E, K, ch.kkey, ch.odd, lane, buf,
                          ok && (ok_extra || !a.extra_row), row_of);
        } else {
            resolve_chains(cd, cand, n_eval, E, K, ch.kkey, ch.odd, lane, buf, row_of, xpiece);
        }
        if (ch.open && !ch.odd) rt_select(cd, E, TK, lane, sel);
        __syncwarp();
    }
    mark(2);
    if (a.stats && lane == 0) {
        atomicAdd(&a.stats[0], (unsigned)n_eval);
        if (blockIdx.x == 0 && warp == 0) a.stats[6] = (unsigned)n_eval;
    }
    if (a.extra_row && lane == 0) a.extra_out[t] = (uint16_t)cd[E];
    int32_t *idx = a.idx_out + (size_t)t * TK;
    uint16_t *wo = a.w_out ? a.w_out + (size_t)t * TK : nullptr;
    if (ch.odd) {
        /* the engine's softmax on the exact logits of the candidates and the rounded
         * fast ones of the rest, which only enter its denominator */
        float *p = reinterpret_cast<float *>(cd);
#pragma unroll
        for (int i = 0; i < R; i++) {
            const int e = lane + 32 * i;
            if (e < E) p[e] = cd[e] == CODE_NEVER ? bf16_round(av[i]) : bf16lo(cd[e]);
        }
        __syncwarp();
        router_softmax_topk(p, E, TK, lane, idx, wo);
    } else {
        rt_weights(cd, sel, TK, lane, idx, wo);
    }
    if (a.unit_hist) {
        __syncwarp();
        if (lane < TK) atomicAdd(&a.unit_hist[(size_t)(t / 256) * E + idx[lane]], 1);
    }
    mark(3);
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
