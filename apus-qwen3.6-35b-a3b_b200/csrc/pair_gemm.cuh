/*
 * pair_gemm.cuh — the expert products for thousands of tokens: a grouped BF16
 * GEMM in which TWO SMs work on one tile (tcgen05.mma.cta_group::2).
 *
 * Replaces, like prefill_gemm.cuh, the per-expert loop of the CPU engine's
 * batched body (c/layer.h:599-621) and its shared-expert GEMMs
 * (c/layer.h:593-596); this is the form for many rows per expert, where the
 * one-SM kernel is held back by the operand bytes every SM has to pull through
 * L2 (48 KB per 64-deep k-block for a 128 x 128(x2) tile).
 *
 * Orientation: the expert's TOKEN rows are the MMA's M dimension, 256 per pair
 * of CTAs (128 per CTA, one TMEM lane each), the WEIGHT rows are N = 256, of
 * which each CTA of the pair loads one half into its own shared memory; the
 * pair's MMA reads both halves.  Per k-block a CTA pulls 16 KB of tokens and
 * 16 KB of weights for 128 x 256 outputs: two thirds of the bytes per flop of
 * the one-SM kernel, and an expert with up to 256 rows reads its weights once.
 *
 *   gate_up:  a CTA's half is 64 gate rows and the 64 matching up rows, so every
 *             thread finds g and u of the same (token, i) in its own TMEM lane:
 *             act = rnd(rnd(silu(rnd g)) * rnd u)   routed  (c/moe.h:387-395)
 *             sa  = rnd(silu(rnd g) * rnd u)        shared  (c/moe.h:438-445)
 *   down:     N = 256 output columns h0..h0+255 (128 per CTA);
 *             y = rnd(D) stored at row perm[r] of the flat assignment-ordered
 *             buffer (the engine's eo, c/layer.h:618) or row t of sy.
 *
 * That MMA costs the same however few of its 256 rows are tokens.  So an expert's last
 * rows, or all of them where they are few, are multiplied the other way round: the
 * weights are M and the token rows N (a multiple of 32), which costs what the rows
 * cost.  In that orientation g and u of a pair (token, i) sit 64 lanes apart; the
 * epilogue warps hand u over through shared memory.  Rows behind full chunks are taken
 * right after those, while the expert's weights are in L2; half of the pairs start with
 * the few-row experts, half end with them, so that these, bound by memory, run beside
 * tiles bound by the tensor cores.  (Both ran in the one-SM kernels before, after the
 * pair kernel: weights of experts with a remainder were fetched twice.  As a second MMA
 * beside the chunk's own, the remainder took both accumulators, and the wait for the
 * epilogue cost more than the extra tile.)
 *
 * Bound: at 64 experts of 256 rows gate_up takes 98 us, its loads alone 87, MMAs and
 * epilogue alone 68.  What held it back before (108) was the issuing lane: flag check,
 * barrier, descriptors, 4 MMAs and commit took 900 cycles for 512 of tensor work; now
 * the whole warp stays together and elects a lane (pg_elect).
 *
 * A CTA fetches a token box just tall enough for its share (32, 64, 96 or 128 rows).
 * Rows past a CTA's share hold stale data whose results are not stored.
 *
 * One persistent cluster of two CTAs per SM pair, 10 warps per CTA: warp 0
 * issues TMA loads (no multicast: each CTA loads its own operands; the
 * completion bytes of both CTAs are counted on the leader's barrier), warp 1 of
 * the leader CTA issues the MMAs and both warps 1 own their CTA's 512 TMEM
 * columns (two accumulators), warps 2-9 drain the accumulators.  Stage and accumulator
 * hand-backs from the MMA to both CTAs are tcgen05.commit with a cluster mask.  Every
 * wait is bounded; a wait that runs out raises the CTA's abort flag and records a status
 * code, and every role falls through to the common exit (cluster barrier, TMEM release).
 */
#pragma once
#include <cuda.h>
#include <cuda_runtime.h>

#include "common.cuh"
#include "dispatch.cuh"
#include "prefill_gemm.cuh"

namespace apus {

constexpr int PP_BM = 128;          /* token rows per CTA (256 per pair) */
constexpr int PP_BN = 256;          /* weight rows per tile (128 per CTA) */
constexpr int PP_BK = 64;
constexpr int PP_HALF_BYTES = 128 * PP_BK * 2;       /* 16 KB */
constexpr int PP_STAGE_BYTES = 2 * PP_HALF_BYTES;    /* tokens | weights */
constexpr int PP_STAGES = 6;
constexpr int PP_EPI_WARPS = 8;
constexpr int PP_THREADS = 64 + PP_EPI_WARPS * 32;
constexpr int PP_TMEM_COLS = 512;
constexpr uint32_t PP_PEER_MASK = 0xFEFFFFFFu;      /* cluster address of CTA 0's copy */

/* Behind the stages and the barriers.  gate_up: u of 32 columns x 64 rows, per half of
 * the epilogue warps.  down with outputs stored into peers' memory: a 32-row x 128-byte
 * staging tile per epilogue warp, so that a row leaves as 128 contiguous bytes. */
constexpr int PP_EXCH_BYTES = 2 * 32 * 64 * 2;
constexpr int PP_STAGING_BYTES = PP_EPI_WARPS * 4096;
inline int pp_smem_bytes(bool staging = false) {
    return PP_STAGES * PP_STAGE_BYTES + (staging ? PP_STAGING_BYTES : PP_EXCH_BYTES) + 1024 + 256;
}

/* token-side tensor maps: the same tensor with boxes of 32, 64, 96, 128 rows */
struct PairMaps {
    CUtensorMap m[4];
};
/* rows of a c-row tile that CTA `rank` owns: the first ceil(c/2) or the rest */
__host__ __device__ __forceinline__ int pp_rows_of(int c, int rank) {
    const int n0 = (c + 1) >> 1;
    return rank ? c - n0 : n0;
}

struct PairParams {
    /* {expert or E, n-tile, first row, rows: up to 256, negative where they are N} */
    const int4 *tiles, *few;           /* few: those of the few-row experts */
    const int *n_tiles, *n_few;
    int K;
    int E, e_begin;
    int rows_per_expert;     /* weight rows per expert in the routed tensor */
    int up_off;              /* gate_up: offset of the up rows (I) */
    uint16_t *out_routed, *out_shared;
    int ld_routed, ld_shared;
    const int32_t *perm;     /* down: sorted position -> flat assignment */
    /* down, expert parallelism: routed output row a is row a % peer_cap of the
     * buffer at peer_dst[a / peer_cap], in another GPU's memory (null: off) */
    const unsigned long long *peer_dst;
    int peer_cap;
    int *status;
};

/* The tiles of a pair: every npairs-th of both lists, the second one dealt from the
 * other end (so that the same pairs do not get one more of both). */
struct PairTiles {
    const int4 *tiles, *few;
    int pair, npairs, n_main, n_few;
    bool few_first;
    int4 ahead;
    __device__ __forceinline__ PairTiles(const PairParams &p, int pair_, int npairs_)
        : tiles(p.tiles), few(p.few), pair(pair_), npairs(npairs_) {
        auto mine = [&](int n, int at) { return at < n ? (n - at + npairs - 1) / npairs : 0; };
        n_main = mine(*p.n_tiles, pair);
        n_few = mine(*p.n_few, npairs - 1 - pair);
        few_first = pair >= npairs / 2;
    }
    __device__ __forceinline__ int n() const { return n_main + n_few; }
    __device__ __forceinline__ int4 load(int k) const {
        if (k >= n()) return make_int4(0, 0, 0, 0);
        const bool f = few_first ? k < n_few : k >= n_main;
        const int i = f == few_first ? k : k - (few_first ? n_few : n_main);
        return __ldg(f ? &few[npairs - 1 - pair + i * npairs] : &tiles[pair + i * npairs]);
    }
    /* k-th tile (asked for in order): its rows as M or as N.  The next one's load is
     * under way meanwhile. */
    __device__ __forceinline__ int4 get(int k, int &rows_m, int &rows_n) {
        const int4 t = k ? ahead : load(0);
        ahead = load(k + 1);
        rows_m = max(t.w, 0);
        rows_n = max(-t.w, 0);
        return t;
    }
};
/* columns of the MMA that has the rows as N */
__device__ __forceinline__ int pp_cols(int rows_n) { return (rows_n + 31) & ~31; }

__device__ __forceinline__ uint32_t pp_cta_rank() {
    uint32_t r;
    asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
    return r;
}
__device__ __forceinline__ void pp_cluster_sync() {
    asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
    asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
}
/* TMA tile load into this CTA's shared memory; completion bytes counted on the
 * LEADER CTA's barrier at the same offset (no multicast) */
__device__ __forceinline__ void pp_tma_load(void *dst, const CUtensorMap *map, int x, int y,
                                            uint64_t *bar) {
    asm volatile(
        "cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.mbarrier::"
        "complete_tx::bytes [%0], [%1, {%3, %4}], [%2];" ::"r"(smem_u32(dst)),
        "l"(reinterpret_cast<uint64_t>(map)), "r"(smem_u32(bar) & PP_PEER_MASK), "r"(x),
        "r"(y)
        : "memory");
}
__device__ __forceinline__ void pp_tmem_alloc(uint32_t *holder, uint32_t cols) {
    asm volatile(
        "tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(
            smem_u32(holder)),
        "r"(cols)
        : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void pp_tmem_dealloc(uint32_t taddr, uint32_t cols) {
    asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(taddr),
                 "r"(cols)
                 : "memory");
}
__device__ __forceinline__ void pp_mma(uint32_t d_tmem, uint64_t adesc, uint64_t bdesc,
                                       uint32_t idesc, uint32_t accumulate) {
    asm volatile(
        "{\n\t"
        ".reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, p;\n\t"
        "}\n" ::"r"(d_tmem),
        "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate)
        : "memory");
}
/* arrive, once every MMA issued so far is done, on the barrier at this offset
 * in BOTH CTAs of the pair */
__device__ __forceinline__ void pp_commit_both(uint64_t *bar) {
    const uint16_t mask = 3;
    asm volatile(
        "tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster."
        "multicast::cluster.b64 [%0], %1;" ::"r"(smem_u32(bar)),
        "h"(mask)
        : "memory");
}
/* arrive on the leader CTA's copy of a barrier */
__device__ __forceinline__ void pp_arrive_leader(uint64_t *bar) {
    asm volatile(
        "{\n\t"
        ".reg .b32 ra;\n\t"
        "mapa.shared::cluster.u32 ra, %0, 0;\n\t"
        "mbarrier.arrive.release.cluster.shared::cluster.b64 _, [ra];\n\t"
        "}\n" ::"r"(smem_u32(bar))
        : "memory");
}
/* kind::f16 instruction descriptor: D fp32, A/B BF16, both K-major, M x N */
__device__ __forceinline__ uint32_t pp_idesc(int m, int n) {
    return (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(n >> 3) << 17) |
           ((uint32_t)(m >> 4) << 24);
}
/* 32 bytes (one whole sector) per store: a thread owns a row, so a warp's store
 * touches 32 rows whatever its width; half as many, complete sectors */
__device__ __forceinline__ void st32(uint16_t *p, const uint32_t (&v)[8]) {
    asm volatile("st.global.v8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};" ::"l"(p),
                 "r"(v[0]), "r"(v[1]), "r"(v[2]), "r"(v[3]), "r"(v[4]), "r"(v[5]), "r"(v[6]),
                 "r"(v[7])
                 : "memory");
}

/* MODE 0: gate_up + SwiGLU;  MODE 1: down */
template <int MODE>
__global__ void __launch_bounds__(PP_THREADS, 1)
pair_gemm_kernel(const __grid_constant__ PairMaps mapA,        /* xg | act   (tokens) */
                 const __grid_constant__ PairMaps mapAs,       /* x  | sa */
                 const __grid_constant__ CUtensorMap mapB,     /* routed weights */
                 const __grid_constant__ CUtensorMap mapBs,    /* shared g | d */
                 const __grid_constant__ CUtensorMap mapBs2,   /* shared u */
                 PairParams p) {
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    extern __shared__ unsigned char pp_smem_raw[];
    unsigned char *smem = reinterpret_cast<unsigned char *>(
        (reinterpret_cast<uintptr_t>(pp_smem_raw) + 1023) & ~(uintptr_t)1023);
    uint64_t *bars = reinterpret_cast<uint64_t *>(smem + (size_t)PP_STAGES * PP_STAGE_BYTES);
    unsigned char *behind = reinterpret_cast<unsigned char *>(bars) + 256;
    uint64_t *full = bars, *empty = bars + PP_STAGES;
    uint64_t *tfull = bars + 2 * PP_STAGES, *tempty = tfull + 2;
    uint32_t *tmem_holder = reinterpret_cast<uint32_t *>(tempty + 2);
    volatile int *abort_flag = reinterpret_cast<volatile int *>(tmem_holder + 1);

    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const uint32_t rank = pp_cta_rank();
    if (tid == 0) {
        for (int s = 0; s < PP_STAGES; s++) {
            mbar_init(&full[s], 1);
            mbar_init(&empty[s], 1);
        }
        for (int a = 0; a < 2; a++) {
            mbar_init(&tfull[a], 1);
            mbar_init(&tempty[a], 2 * PP_EPI_WARPS);   /* the epilogue warps of both CTAs */
        }
        *abort_flag = 0;
        mbar_fence_init();
    }
    __syncthreads();
    if (warp == 1) pp_tmem_alloc(tmem_holder, PP_TMEM_COLS);
    tc_fence_before();
    __syncthreads();
    pp_cluster_sync();       /* the peer's barriers exist before anything signals them */
    tc_fence_after();
    const uint32_t tmem_base = *tmem_holder;
    asm volatile("griddepcontrol.wait;" ::: "memory");
    PairTiles tiles(p, blockIdx.x >> 1, gridDim.x >> 1);
    const int n_tiles = tiles.n(), num_kb = p.K / PP_BK;

    if (warp == 0) {
        /* ---------------- TMA producer (both CTAs) ---------------- */
        int s = 0;
        uint32_t ph = 0;
        bool alive = true;
        for (int k = 0; alive && k < n_tiles; k++) {
            int rows_m, rows_n;
            const int4 t = tiles.get(k, rows_m, rows_n);
            const bool shared = t.x == p.E;
            const PairMaps &ma = shared ? mapAs : mapA;
            /* this CTA's share of the rows, and the box that covers it */
            const int r0 = rows_n ? pp_cols(rows_n) / 2 : pp_rows_of(rows_m, 0),
                      r1 = rows_n ? r0 : rows_m - r0;
            const int h0 = (r0 + 31) >> 5, h1 = (r1 + 31) >> 5, h = rank ? h1 : h0;
            const int arow = t.z + (rank ? r0 : 0);
            const CUtensorMap *map_a = &ma.m[h ? h - 1 : 0];
            const CUtensorMap *mb = shared ? &mapBs : &mapB,
                              *mb2 = shared ? &mapBs2 : &mapB;
            const int wrow = shared ? 0 : (t.x - p.e_begin) * p.rows_per_expert;
            const int brow = MODE == 0 ? wrow + t.y * 128 + (int)rank * 64
                                       : wrow + t.y * PP_BN + (int)rank * 128;
            const int brow2 = brow + (shared ? 0 : p.up_off);
            const uint32_t bytes = (uint32_t)(2 * PP_HALF_BYTES) +
                                   (uint32_t)(h0 + h1) * 32u * PP_BK * 2u;
            for (int kb = 0; kb < num_kb; kb++) {
                if (!pg_wait_warp(&empty[s], ph ^ 1u, abort_flag, p.status, ST_MBAR_TIMEOUT)) {
                    alive = false;
                    break;
                }
                unsigned char *st = smem + (size_t)s * PP_STAGE_BYTES;
                if (pg_elect()) {
                    if (rank == 0) mbar_expect_tx(&full[s], bytes);
                    /* a CTA without a row of the tile skips the token load */
                    if (h) pp_tma_load(st, map_a, kb * PP_BK, arow, &full[s]);
                    pp_tma_load(st + PP_HALF_BYTES, mb, kb * PP_BK, brow, &full[s]);
                    if (MODE == 0)
                        pp_tma_load(st + PP_HALF_BYTES + PP_HALF_BYTES / 2, mb2, kb * PP_BK,
                                    brow2, &full[s]);
                }
                if (++s == PP_STAGES) {
                    s = 0;
                    ph ^= 1u;
                }
            }
        }
    } else if (warp == 1) {
        /* ---------------- MMA issuer (leader CTA only) ---------------- */
        if (rank == 0) {
            int s = 0;
            uint32_t ph = 0;
            bool alive = true;
            const uint64_t desc0 = umma_smem_desc(smem_u32(smem));   /* + offset / 16 */
            for (int k = 0; k < n_tiles; k++) {
                int rows_m, rows_n;
                tiles.get(k, rows_m, rows_n);
                const uint32_t idesc = pp_idesc(2 * PP_BM, rows_n ? pp_cols(rows_n) : PP_BN);
                /* what is M and what is N of a stage */
                const uint64_t off_m = rows_n ? PP_HALF_BYTES >> 4 : 0,
                               off_n = rows_n ? 0 : PP_HALF_BYTES >> 4;
                const uint32_t acc = (uint32_t)k & 1u, d = tmem_base + acc * 256u;
                if (!pg_wait_warp(&tempty[acc], (((uint32_t)k >> 1) & 1u) ^ 1u, abort_flag,
                                  p.status, ST_TMEM_TIMEOUT))
                    break;
                tc_fence_after();
                for (int kb = 0; kb < num_kb; kb++) {
                    if (!pg_wait_warp(&full[s], ph, abort_flag, p.status, ST_MBAR_TIMEOUT)) {
                        alive = false;
                        break;
                    }
                    tc_fence_after();
                    const uint64_t at = desc0 + (uint64_t)(s * (PP_STAGE_BYTES >> 4)),
                                   dm = at + off_m, dn = at + off_n;
                    if (pg_elect()) {
#pragma unroll
                        for (int j = 0; j < PP_BK / 16; j++)
                            pp_mma(d, dm + 2u * j, dn + 2u * j, idesc, (kb | j) ? 1u : 0u);
                        pp_commit_both(&empty[s]);   /* frees the stage in both CTAs */
                    }
                    if (++s == PP_STAGES) {
                        s = 0;
                        ph ^= 1u;
                    }
                }
                if (!alive) break;
                if (pg_elect()) pp_commit_both(&tfull[acc]);
            }
        }
    } else {
        /* ---------------- epilogue (warps 2..9, both CTAs) ---------------- */
        const int q = warp & 3;                 /* TMEM lane quarter of this warp */
        const int half = (warp - 2) >> 2;       /* which columns of the tile */
        const int rl = q * 32 + lane;           /* this thread's TMEM lane */
        /* a warp that gave up goes on through the tiles without reading: the others may
         * still meet it at the barriers below */
        bool alive = true;
        for (int k = 0; k < n_tiles; k++) {
            int rows_m, rows_n;
            const int4 t = tiles.get(k, rows_m, rows_n);
            const bool shared = t.x == p.E;
            uint16_t *out = shared ? p.out_shared : p.out_routed;
            const int ld = shared ? p.ld_shared : p.ld_routed;
            const uint32_t acc = (uint32_t)k & 1u, aph = ((uint32_t)k >> 1) & 1u;
            const uint32_t taddr = tmem_base + acc * 256u + ((uint32_t)(q * 32) << 16);
            if (rows_m) {
                /* ---- tokens as M: a thread owns a token row ---- */
                const int n_mine = pp_rows_of(rows_m, (int)rank);
                const bool valid = rl < n_mine;
                int orow = t.z + (rank ? pp_rows_of(rows_m, 0) : 0) + rl;
                if (MODE == 1 && !shared && valid) orow = __ldg(&p.perm[orow]);
                alive = alive && pg_wait_warp(&tfull[acc], aph, abort_flag, p.status,
                                              ST_TMEM_TIMEOUT);
                tc_fence_after();
                /* a warp whose rows are all past the tile's end has nothing to read */
                const bool any = alive && q * 32 < n_mine;
                if (MODE == 0) {
                    /* columns of a CTA's half: 64 g, 64 u */
                    for (int c0 = 0; any && c0 < 64; c0 += 32) {
                        uint32_t g[32], u[32];
                        tmem_ld32(taddr + (uint32_t)(half * 128 + c0), g);
                        tmem_ld32(taddr + (uint32_t)(half * 128 + 64 + c0), u);
                        tmem_ld_wait();
                        if (valid) {
                            uint16_t *dst = out + (size_t)orow * ld + t.y * 128 + half * 64 + c0;
#pragma unroll
                            for (int j = 0; j < 32; j += 16) {
                                uint32_t pk[8];
#pragma unroll
                                for (int h = 0; h < 8; h++) {
                                    float g0 = __uint_as_float(g[j + 2 * h]),
                                          g1 = __uint_as_float(g[j + 2 * h + 1]),
                                          u0 = __uint_as_float(u[j + 2 * h]),
                                          u1 = __uint_as_float(u[j + 2 * h + 1]);
                                    bf16_round2(g0, g1);
                                    bf16_round2(u0, u1);
                                    pk[h] = shared ? silu_mul_pack2(g0, u0, g1, u1)
                                                   : silu_act_pack2(g0, u0, g1, u1);
                                }
                                st32(dst + j, pk);
                            }
                        }
                    }
                } else if (p.peer_dst && !shared) {
                    /* A thread owns a row, so a warp's store would touch 32 rows
                     * with 32 bytes each: fine for local memory, where L2 merges
                     * sectors, poor as NVLink packets.  The warp turns its 32 x 64
                     * chunk round in shared memory (16-byte units, XOR-swizzled by
                     * row) and stores it as 128 contiguous bytes per row, four
                     * rows an instruction. */
                    unsigned char *stg = behind + (size_t)(warp - 2) * 4096;
                    unsigned long long my_row = 0;
                    if (valid) {
                        const int sr = orow / p.peer_cap;
                        my_row = __ldg(p.peer_dst + sr) +
                                 (unsigned long long)(orow - sr * p.peer_cap) * ld * 2ull;
                    }
                    for (int c0 = half * 128; any && c0 < half * 128 + 128; c0 += 64) {
                        uint32_t v[32], v2[32];
                        tmem_ld32(taddr + (uint32_t)c0, v);
                        tmem_ld32(taddr + (uint32_t)c0 + 32u, v2);
                        tmem_ld_wait();
#pragma unroll
                        for (int h8 = 0; h8 < 8; h8++) {
                            const uint32_t *f = h8 < 4 ? v + 8 * h8 : v2 + 8 * (h8 - 4);
                            uint4 q4;
                            q4.x = pack_bf16_rn(__uint_as_float(f[0]), __uint_as_float(f[1]));
                            q4.y = pack_bf16_rn(__uint_as_float(f[2]), __uint_as_float(f[3]));
                            q4.z = pack_bf16_rn(__uint_as_float(f[4]), __uint_as_float(f[5]));
                            q4.w = pack_bf16_rn(__uint_as_float(f[6]), __uint_as_float(f[7]));
                            *reinterpret_cast<uint4 *>(stg + lane * 128 +
                                                       ((h8 ^ (lane & 7)) << 4)) = q4;
                        }
                        __syncwarp();
#pragma unroll
                        for (int i = 0; i < 8; i++) {
                            const int rr = i * 4 + (lane >> 3), ch = lane & 7;
                            const unsigned long long rp = __shfl_sync(0xffffffffu, my_row, rr);
                            const uint4 q4 = *reinterpret_cast<const uint4 *>(
                                stg + rr * 128 + ((ch ^ (rr & 7)) << 4));
                            if (rp)
                                *reinterpret_cast<uint4 *>(
                                    reinterpret_cast<unsigned char *>((uintptr_t)rp) +
                                    (size_t)(t.y * PP_BN + c0) * 2 + (ch << 4)) = q4;
                        }
                        __syncwarp();
                    }
                } else {
                    for (int c0 = half * 128; any && c0 < half * 128 + 128; c0 += 32) {
                        uint32_t v[32];
                        tmem_ld32(taddr + (uint32_t)c0, v);
                        tmem_ld_wait();
                        if (valid) {
                            uint16_t *dst = out + (size_t)orow * ld + t.y * PP_BN + c0;
#pragma unroll
                            for (int j = 0; j < 32; j += 16) {
                                uint32_t pk[8];
#pragma unroll
                                for (int h = 0; h < 8; h++)
                                    pk[h] = pack_bf16_rn(__uint_as_float(v[j + 2 * h]),
                                                         __uint_as_float(v[j + 2 * h + 1]));
                                st32(dst + j, pk);
                            }
                        }
                    }
                }
            } else {
                /* ---- weights as M: a thread owns a weight row, a column is a token ---- */
                alive = alive && pg_wait_warp(&tfull[acc], aph, abort_flag, p.status,
                                              ST_TMEM_TIMEOUT);
                tc_fence_after();
                for (int c0 = half * 32; c0 < rows_n; c0 += 64) {
                    uint32_t v[32];
                    if (alive) {
                        tmem_ld32(taddr + (uint32_t)c0, v);
                        tmem_ld_wait();
                    }
                    if (MODE == 0) {
                        /* lanes 0..63: g of 64 rows, 64..127: u of the same */
                        uint32_t *ex = reinterpret_cast<uint32_t *>(behind) + half * (16 * 64) +
                                       (q & 1) * 32 + lane;
                        if (alive && q >= 2) {
#pragma unroll
                            for (int j = 0; j < 16; j++)
                                ex[j * 64] = pack_bf16_rn(__uint_as_float(v[2 * j]),
                                                          __uint_as_float(v[2 * j + 1]));
                        }
                        asm volatile("bar.sync %0, 128;" ::"r"(1 + half) : "memory");
                        if (alive && q < 2) {
                            uint16_t *dst = out + (size_t)(t.z + c0) * ld + t.y * 128 +
                                            (int)rank * 64 + rl;
#pragma unroll
                            for (int j = 0; j < 16; j++) {
                                const int n = c0 + 2 * j;
                                if (n < rows_n) {
                                    const uint32_t uu = ex[j * 64];
                                    float g0 = __uint_as_float(v[2 * j]),
                                          g1 = __uint_as_float(v[2 * j + 1]);
                                    bf16_round2(g0, g1);
                                    const uint32_t pk =
                                        shared ? silu_mul_pack2(g0, bf16lo(uu), g1, bf16hi(uu))
                                               : silu_act_pack2(g0, bf16lo(uu), g1, bf16hi(uu));
                                    dst[(size_t)(2 * j) * ld] = (uint16_t)pk;
                                    if (n + 1 < rows_n)
                                        dst[(size_t)(2 * j + 1) * ld] = (uint16_t)(pk >> 16);
                                }
                            }
                        }
                        asm volatile("bar.sync %0, 128;" ::"r"(1 + half) : "memory");
                    } else {
                        /* output row of each of the 32 columns: one load per lane,
                         * handed round by shuffle */
                        unsigned long long my_row = 0;
                        if (c0 + lane < rows_n) {
                            int orow = t.z + c0 + lane;
                            if (!shared) orow = __ldg(&p.perm[orow]);
                            if (p.peer_dst && !shared) {
                                const int sr = orow / p.peer_cap;
                                my_row = __ldg(p.peer_dst + sr) +
                                         (unsigned long long)(orow - sr * p.peer_cap) * ld * 2ull;
                            } else {
                                my_row = (unsigned long long)reinterpret_cast<uintptr_t>(
                                    out + (size_t)orow * ld);
                            }
                        }
                        const int col = t.y * PP_BN + (int)rank * 128 + rl;
#pragma unroll
                        for (int j = 0; j < 32; j += 2) {
                            uint16_t *r0 = reinterpret_cast<uint16_t *>(
                                (uintptr_t)__shfl_sync(0xffffffffu, my_row, j));
                            uint16_t *r1 = reinterpret_cast<uint16_t *>(
                                (uintptr_t)__shfl_sync(0xffffffffu, my_row, j + 1));
                            const uint32_t pk = pack_bf16_rn(__uint_as_float(v[j]),
                                                             __uint_as_float(v[j + 1]));
                            if (alive && r0) r0[col] = (uint16_t)pk;
                            if (alive && r1) r1[col] = (uint16_t)(pk >> 16);
                        }
                    }
                }
            }
            tc_fence_before();
            __syncwarp();
            if (lane == 0) pp_arrive_leader(&tempty[acc]);
        }
    }
    /* neither CTA may leave (or free its tensor memory) while the other can
     * still signal its barriers or have MMAs in flight into its TMEM */
    tc_fence_before();
    __syncthreads();
    pp_cluster_sync();
    if (warp == 1) {
        tc_fence_after();
        pp_tmem_dealloc(tmem_base, PP_TMEM_COLS);
    }
}

/* ---- host side ---------------------------------------------------------------- */
inline int g_pp_enable = 1;          /* APUS_CUDA_PAIR=0: never take this path */
/* Mean rows per resident expert from which it is taken.  us of the block with the one-SM
 * kernels against these, even router: 104 rows 453, 463; 112 479, 490; 120 500, 500; 128
 * 529, 512; 136 551, 533; 144 615, 565.  Skewed: 96 481, 482; 104 510, 499; 112 540, 523;
 * 120 551, 536; 128 580, 564.  Hidden 4096, width 768, even: 112 833, 825; 128 865, 816; 160
 * 1017, 894.  (The experts alone, as in expert parallelism, even: 112 397, 404; 128 431, 436;
 * 144 488, 456.) */
inline int g_pp_min_rows = 120;
/* Last chunks of fewer rows are taken as N (APUS_CUDA_PAIR_SWAP_BELOW).  8192 skewed tokens:
 * never 912 us, below 64 911, 128 896, 160 891, 192 869, 224 860, 256 (always) 886; 144 rows
 * an expert, skewed: 655, 589, 571, 618, 603, 586, 625. */
inline int g_pp_swap_below = 192;

inline bool pair_supported(const ApusCudaMoeCfg &c, int sm_count, int smem_optin) {
    return g_pp_enable && prefill_supported(c) && c.hidden % PP_BN == 0 &&
           sm_count >= 2 && pp_smem_bytes() <= smem_optin;
}

/* ---- tile lists ---------------------------------------------------------------
 * An expert's rows are cut into chunks of 256, one tile per chunk and 256 weight rows
 * (128 gate, 128 up).  A remainder of fewer than `swap_below` rows is taken as N; behind
 * full chunks it follows them in the list, without a full chunk it goes to the list of
 * few-row experts.  Chunks of one expert are adjacent, so its weights come from HBM
 * once and from L2 afterwards; the shared expert's (dense over the tokens) come first.
 * One CTA of 1024 threads, thread e = expert e, which holds its row count and first
 * sorted position. */
struct PairLists {
    int4 *gu, *dn, *few_gu, *few_dn;
    int *n_gu, *n_dn, *n_few_gu, *n_few_dn;
};
struct PairPlan {
    int T;                   /* tokens of the shared expert (0: none) */
    int m_gu, m_dn;          /* weight tiles per chunk: gate_up, down */
    int swap_below;
    PairLists l;
};
struct PairCut {
    int chunks, few;                     /* of either list */
    __device__ __forceinline__ PairCut(int cnt, int swap_below) {
        few = cnt > 0 && cnt < swap_below;
        chunks = few ? 0 : (cnt + 2 * PP_BM - 1) / (2 * PP_BM);
    }
};

__device__ __forceinline__ void build_pair_body(int cnt, int off, int E, const PairPlan &pp) {
    __shared__ int wt[2][32];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const PairCut cut(cnt, pp.swap_below), sh(pp.T, pp.swap_below);
    int inc[2] = {cut.chunks, cut.few};
#pragma unroll
    for (int d = 1; d < 32; d <<= 1)
#pragma unroll
        for (int q = 0; q < 2; q++) {
            const int v = __shfl_up_sync(0xffffffffu, inc[q], d);
            if (lane >= d) inc[q] += v;
        }
    if (lane == 31)
        for (int q = 0; q < 2; q++) wt[q][warp] = inc[q];
    __syncthreads();
    int base[2], total[2];
#pragma unroll
    for (int q = 0; q < 2; q++) {
        const int v = wt[q][lane];
        base[q] = __reduce_add_sync(0xffffffffu, lane < warp ? v : 0);
        total[q] = __reduce_add_sync(0xffffffffu, v);
    }
    const PairLists &l = pp.l;
    /* chunk n of `rows` rows that start at `o`: entry `at` of the list */
    auto put = [&](int4 *gu, int4 *dn, int at, int e, int o, int rows, int n) {
        const int left = min(rows - n * 2 * PP_BM, 2 * PP_BM),
                  w = left < pp.swap_below ? -left : left;
        for (int m = 0; m < pp.m_gu; m++)
            gu[at * pp.m_gu + m] = make_int4(e, m, o + n * 2 * PP_BM, w);
        for (int m = 0; m < pp.m_dn; m++)
            dn[at * pp.m_dn + m] = make_int4(e, m, o + n * 2 * PP_BM, w);
    };
    if (tid < E) {
        const int first = sh.chunks + base[0] + inc[0] - cut.chunks;
        for (int n = 0; n < cut.chunks; n++) put(l.gu, l.dn, first + n, tid, off, cnt, n);
        if (cut.few) put(l.few_gu, l.few_dn, sh.few + base[1] + inc[1] - 1, tid, off, cnt, 0);
    }
    for (int n = tid; n < sh.chunks; n += blockDim.x) put(l.gu, l.dn, n, E, 0, pp.T, n);
    if (tid == 0) {
        if (sh.few) put(l.few_gu, l.few_dn, 0, E, 0, pp.T, 0);
        *l.n_gu = (sh.chunks + total[0]) * pp.m_gu;
        *l.n_dn = (sh.chunks + total[0]) * pp.m_dn;
        *l.n_few_gu = (sh.few + total[1]) * pp.m_gu;
        *l.n_few_dn = (sh.few + total[1]) * pp.m_dn;
    }
}

__global__ void __launch_bounds__(1024)
build_pair_tiles_kernel(const int32_t *__restrict__ counts,
                        const int32_t *__restrict__ offsets, int E, PairPlan pp) {
    pdl_enter();
    const int tid = threadIdx.x;
    build_pair_body(tid < E ? counts[tid] : 0, tid < E ? offsets[tid] : 0, E, pp);
}

/* list storage inside the block's tile workspace (prefill_tiles_bytes_for) */
inline bool pair_plan(const ApusCudaMoeCfg &c, int T, bool do_shared, int A, void *ws,
                      size_t ws_bytes, PairPlan *out) {
    const int E = (int)c.experts;
    PairPlan p;
    memset(&p, 0, sizeof p);
    p.T = do_shared ? T : 0;
    p.m_gu = (int)c.moe_inter / 128;
    p.m_dn = (int)c.hidden / PP_BN;
    p.swap_below = g_pp_swap_below < 2 * PP_BM ? g_pp_swap_below : 2 * PP_BM;
    const size_t chunks = (size_t)A / (2 * PP_BM) + E + (size_t)T / (2 * PP_BM) + 1,
                 few = (size_t)E + 1;
    const size_t n_gu = chunks * p.m_gu, n_dn = chunks * p.m_dn, n_fg = few * p.m_gu,
                 n_fd = few * p.m_dn;
    if ((n_gu + n_dn + n_fg + n_fd) * sizeof(int4) + 64 > ws_bytes) return false;
    p.l.gu = reinterpret_cast<int4 *>(ws);
    p.l.dn = p.l.gu + n_gu;
    p.l.few_gu = p.l.dn + n_dn;
    p.l.few_dn = p.l.few_gu + n_fg;
    p.l.n_gu = reinterpret_cast<int *>(p.l.few_dn + n_fd);
    p.l.n_dn = p.l.n_gu + 1;
    p.l.n_few_gu = p.l.n_gu + 2;
    p.l.n_few_dn = p.l.n_gu + 3;
    *out = p;
    return true;
}

template <typename... KArgs, typename... Args>
inline cudaError_t launch_pair(void (*kernel)(KArgs...), int grid, int threads, size_t smem,
                               cudaStream_t st, Args... args) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(grid);
    cfg.blockDim = dim3(threads);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = 2;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[1].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = g_apus_use_pdl ? 2 : 1;
    return cudaLaunchKernelEx(&cfg, kernel, static_cast<KArgs>(args)...);
}

/* Routed + shared experts through the two-SM kernels.  Same contract as
 * run_prefill_experts.  placed: tile lists and the permuted copy are made already
 * (place.cuh). */
inline int run_pair_experts(int sm_count, int smem_optin, PrefillMaps *maps,
                            const ApusCudaMoeCfg &c, int e_begin, const uint16_t *x, int T,
                            int A, int TK, bool do_shared, const DispatchOut &d,
                            uint16_t *xg, uint16_t *act, uint16_t *sa, uint16_t *eo,
                            uint16_t *sy, void *tiles_ws, int *status, cudaStream_t st,
                            int *launches, void (*mark)(int stage),
                            const PeerRows *peer = nullptr, const PairPlan *placed = nullptr) {
    const int H = (int)c.hidden, I = (int)c.moe_inter, Is = (int)c.shared_inter,
              E = (int)c.experts;
    if (!maps) {
        snprintf(g_prefill_err, sizeof g_prefill_err, "tensor maps missing");
        return 1;
    }
    const int smem = pp_smem_bytes(), smem_dn = pp_smem_bytes(peer != nullptr);
    if (smem_dn > smem_optin || Is != I) {
        snprintf(g_prefill_err, sizeof g_prefill_err,
                 "two-SM grouped GEMM: %d B shared memory, shared_inter == moe_inter", smem);
        return 1;
    }
    PairPlan plan;
    if (placed) {
        plan = *placed;
    } else {
        if (!pair_plan(c, T, do_shared, A, tiles_ws,
                       prefill_tiles_bytes_for(c, (size_t)A, (size_t)T), &plan)) {
            snprintf(g_prefill_err, sizeof g_prefill_err, "tile workspace too small");
            return 1;
        }
        launch_k(build_pair_tiles_kernel, dim3(1), dim3(1024), 0, st,
                 (const int32_t *)d.counts, (const int32_t *)d.offsets, E, plan);
        (*launches)++;
    }
    const PairLists &tl = plan.l;
    if (A > 0 && !placed) {
        long total = (long)A * (H / 8);
        int blocks = (int)((total + 255) / 256);
        if (blocks > sm_count * 16) blocks = sm_count * 16;
        if (peer)
            launch_k(gather_rows_peer_kernel, dim3(blocks), dim3(256), 0, st, peer->src,
                     peer->cap, (const int32_t *)d.perm, A, H, TK, xg,
                     (const int32_t *)(d.offsets + E));
        else
            launch_k(gather_rows_kernel, dim3(blocks), dim3(256), 0, st, x, d.perm, A, H, TK,
                     xg, (const int32_t *)(d.offsets + E));
        (*launches)++;
    }
    if (mark) mark(APUS_CUDA_STAGE_GATHER);
    PairMaps m_xg, m_x, m_act, m_sa;
    int bad = 0;
    for (int h = 0; h < 4; h++) {
        const int box = 32 * (h + 1);
        bad |= encode_2d(maps->encode, &m_xg.m[h], A > 0 ? (const void *)xg : (const void *)x,
                         (size_t)(A > 0 ? A : (T > 0 ? T : 1)), H, box);
        bad |= encode_2d(maps->encode, &m_x.m[h], x, (size_t)(T > 0 ? T : 1), H, box);
        bad |= encode_2d(maps->encode, &m_act.m[h],
                         A > 0 ? (const void *)act : (const void *)sa, (size_t)(A > 0 ? A : 1),
                         I, box);
        bad |= encode_2d(maps->encode, &m_sa.m[h],
                         do_shared ? (const void *)sa : (const void *)x,
                         (size_t)(do_shared && T > 0 ? T : 1), Is, box);
    }
    if (bad) return 1;
    static bool attr_set = false;
    if (!attr_set) {
        cudaFuncSetAttribute(pair_gemm_kernel<0>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             smem);
        cudaFuncSetAttribute(pair_gemm_kernel<1>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             pp_smem_bytes(true) <= smem_optin ? pp_smem_bytes(true) : smem);
        attr_set = true;
    }
    const int grid = sm_count & ~1;
    PairParams p1;
    memset(&p1, 0, sizeof p1);
    p1.tiles = tl.gu;
    p1.n_tiles = tl.n_gu;
    p1.few = tl.few_gu;
    p1.n_few = tl.n_few_gu;
    p1.K = H;
    p1.E = E;
    p1.e_begin = e_begin;
    p1.rows_per_expert = 2 * I;
    p1.up_off = I;
    p1.out_routed = act;
    p1.out_shared = sa;
    p1.ld_routed = I;
    p1.ld_shared = Is;
    p1.perm = d.perm;
    p1.status = status;
    launch_pair(pair_gemm_kernel<0>, grid, PP_THREADS, (size_t)smem, st, m_xg, m_x, maps->w_gu64,
                maps->sh_g64, maps->sh_u64, p1);
    (*launches)++;
    if (mark) mark(APUS_CUDA_STAGE_GATE_UP);
    PairParams p2 = p1;
    p2.tiles = tl.dn;
    p2.n_tiles = tl.n_dn;
    p2.few = tl.few_dn;
    p2.n_few = tl.n_few_dn;
    p2.K = I;
    p2.rows_per_expert = H;
    p2.up_off = 0;
    p2.out_routed = eo;
    p2.out_shared = sy;
    p2.ld_routed = H;
    p2.ld_shared = H;
    p2.peer_dst = peer ? peer->dst : nullptr;
    p2.peer_cap = peer ? peer->cap : 0;
    launch_pair(pair_gemm_kernel<1>, grid, PP_THREADS, (size_t)smem_dn, st, m_act, m_sa,
                maps->w_d, maps->sh_d, maps->sh_d, p2);
    (*launches)++;
    if (mark) mark(APUS_CUDA_STAGE_DOWN);
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) {
        snprintf(g_prefill_err, sizeof g_prefill_err, "two-SM grouped GEMM launch: %s",
                 cudaGetErrorString(e));
        return 1;
    }
    return 0;
}

}  // namespace apus
