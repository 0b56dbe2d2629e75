/*
 * place.cuh — the block's dispatch and the permuted copy of its input in one kernel:
 * perm (the stable counting sort of dispatch.cuh), the grouped GEMMs' tile lists and
 * xg[p] = x[perm[p] / top_k] (c/layer.h:599-606).
 *
 * Where the router has counted its selections per unit of 256 tokens, every CTA finds
 * the first position of its own tokens' assignments by itself: totals and prefixes from
 * the counts, plus the selections of the unit's tokens before its own.  So no CTA waits
 * for a scan in another one, a token's row is read once and written to its top_k places
 * (the sorted copy read it top_k times), and the first CTA builds the tile lists beside
 * the others.  Up to one unit of tokens every CTA counts all selections itself.
 *
 * Bound: the top_k row writes (268 MB at 8192 tokens).  At 8192 tokens histogram, scan,
 * permutation, tile lists and copy took 49 + 69 us and five launches; this 67 (512 tokens
 * 28 and 12, up to 128 tokens 17 and 10).
 */
#pragma once
#include "common.cuh"
#include "dispatch.cuh"
#include "pair_gemm.cuh"

namespace apus {

constexpr int PL_THREADS = 1024;
constexpr int PL_UNIT = 256;             /* tokens of a unit of the router's counts */

struct PlaceArgs {
    const int32_t *idx;                  /* [T, TK] */
    const int32_t *unit_hist;            /* [ceil(T / PL_UNIT)][E], null: count here */
    const uint16_t *x;                   /* [T, H] */
    uint16_t *xg;                        /* [T TK, H], null: no copy */
    int32_t *perm;                       /* [T TK] */
    int T, TK, E, H;
    int tb;                              /* tokens of a CTA; tb TK <= 1024 */
    int *status;
};

__device__ __forceinline__ void build_lists(int cnt, int off, int E, const TilePlan &tp) {
    build_tiles_body(cnt, off, E, tp.T, tp.m_gu, tp.m_gu_sh, tp.m_dn, tp.bn_gu, tp.bn_dn,
                     tp.bn_sh_gu, tp.bn_sh_dn, tp.tl);
}
__device__ __forceinline__ void build_lists(int cnt, int off, int E, const PairPlan &hp) {
    build_pair_body(cnt, off, E, hp);
}

/* grid = 1 + ceil(T / tb); thread e speaks for expert e (E <= 1024).  PER_SM: resident
 * CTAs; two (and 32 registers) pay where the row writes dominate, not where the lists do. */
template <typename Plan, int PER_SM>
__global__ void __launch_bounds__(PL_THREADS, PER_SM)
place_kernel(const __grid_constant__ PlaceArgs a, const __grid_constant__ Plan plan) {
    __shared__ int s_tot[PL_THREADS], s_bef[PL_THREADS];     /* [parts][E padded] */
    __shared__ int s_first[PL_THREADS];
    __shared__ __align__(16) int s_key[PL_THREADS];
    __shared__ int s_pos[PL_THREADS], s_warp[32];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int E = a.E, TK = a.TK, A = a.T * TK;
    const bool lists = blockIdx.x == 0;
    const int t0 = lists ? 0 : ((int)blockIdx.x - 1) * a.tb, nt = lists ? 0 : min(a.tb, a.T - t0);
    const int u0 = t0 / PL_UNIT, n = nt * TK;
    const int Ep = (E + 31) & ~31, parts = a.unit_hist ? PL_THREADS / Ep : 1;
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    s_tot[tid] = s_bef[tid] = 0;
    __syncthreads();
    asm volatile("griddepcontrol.wait;" ::: "memory");
    auto key_at = [&](int i) {
        const int e = __ldcg(&a.idx[i]);       /* L2: the previous kernels may share the SM */
        if ((unsigned)e >= (unsigned)E) set_status(a.status, ST_BAD_INDEX);
        return (unsigned)e < (unsigned)E ? e : -1;
    };
    if (tid < n) s_key[tid] = key_at(t0 * TK + tid);
    if (a.unit_hist) {
        const int part = tid / Ep, e = tid - part * Ep, units = (a.T + PL_UNIT - 1) / PL_UNIT;
        int tot = 0, bef = 0;
        if (part < parts && e < E) {
#pragma unroll 8
            for (int u = part; u < units; u += parts) {
                const int v = __ldcg(&a.unit_hist[(size_t)u * E + e]);
                tot += v;
                bef += u < u0 ? v : 0;
            }
            s_tot[tid] = tot;
            atomicAdd(&s_bef[tid], bef);
        }
        for (int i = u0 * PL_UNIT * TK + tid; i < t0 * TK; i += PL_THREADS) {
            const int k = key_at(i);
            if (k >= 0) atomicAdd(&s_bef[k], 1);             /* into part 0 */
        }
    } else {
        for (int i = tid; i < A; i += PL_THREADS) {
            const int k = key_at(i);
            if (k >= 0) {
                atomicAdd(&s_tot[k], 1);
                if (i < t0 * TK) atomicAdd(&s_bef[k], 1);
            }
        }
    }
    __syncthreads();
    int total = 0, before = 0;
    if (tid < E)
        for (int q = 0; q < parts; q++) {
            total += s_tot[q * Ep + tid];
            before += s_bef[q * Ep + tid];
        }
    int inc = total;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
        const int v = __shfl_up_sync(0xffffffffu, inc, d);
        if (lane >= d) inc += v;
    }
    if (lane == 31) s_warp[warp] = inc;
    __syncthreads();
    const int off =
        inc - total + __reduce_add_sync(0xffffffffu, lane < warp ? s_warp[lane] : 0);
    if (lists) {
        build_lists(total, off, E, plan);
        return;
    }
    s_first[tid] = off + before;
    __syncthreads();
    if (tid < n) {
        /* rank among the CTA's earlier assignments of the same expert */
        const int e = s_key[tid];
        int rank = 0;
        const int4 *k4 = reinterpret_cast<const int4 *>(s_key);
        for (int q = 0; q < tid / 4; q++) {
            const int4 k = k4[q];
            rank += (k.x == e) + (k.y == e) + (k.z == e) + (k.w == e);
        }
        for (int i = tid & ~3; i < tid; i++) rank += s_key[i] == e;
        const int p = e >= 0 ? s_first[e] + rank : -1;
        const bool in = p >= 0 && p < A;
        s_pos[tid] = in ? p : -1;
        if (in) a.perm[p] = t0 * TK + tid;
    }
    if (!a.xg) return;
    __syncthreads();
    const int c8 = a.H / 8, items = nt * c8;
    const uint4 *src = reinterpret_cast<const uint4 *>(a.x) + (size_t)t0 * c8;
    uint4 *dst = reinterpret_cast<uint4 *>(a.xg);
    for (int i0 = tid; i0 < items; i0 += 2 * PL_THREADS) {
        const int i1 = i0 + PL_THREADS;
        const uint4 v0 = __ldg(src + i0), v1 = i1 < items ? __ldg(src + i1) : v0;
#pragma unroll
        for (int h = 0; h < 2; h++) {
            const int i = h ? i1 : i0;
            if (i >= items) break;
            const int t = i / c8, c = i - t * c8;
            for (int j = 0; j < TK; j++) {
                const int p = s_pos[t * TK + j];
                if (p >= 0) dst[(size_t)p * c8 + c] = h ? v1 : v0;
            }
        }
    }
}

/* tokens of a CTA: all CTAs resident at once; without a copy as few CTAs as the rank
 * loop allows */
inline int place_tokens(int T, int TK, int ctas, bool copy) {
    const int others = ctas > 1 ? ctas - 1 : 1;      /* beside the lists' (none waits for another) */
    const int most = PL_THREADS / TK, want = copy ? (T + others - 1) / others : T;
    return want < most ? want : most;
}

}  // namespace apus
