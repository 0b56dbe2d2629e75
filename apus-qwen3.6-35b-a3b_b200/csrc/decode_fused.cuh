/*
 * decode_fused.cuh — the whole MoE block for one to eight tokens in ONE
 * cooperative kernel (c/layer.h:333-370 end to end, and through
 * apus_cuda_moe_layer_dev the norm before and the residual add after,
 * c/layer.h:386-388): router, softmax / top-k, the routed and shared experts'
 * gate/up rows with SwiGLU, one grid-wide barrier, the down rows, and the weighted
 * combine + shared gate + add.
 *
 * At one token the block is a 57 MB weight stream that should take 9 us; what it
 * takes instead is dependent latencies, so the kernel is built around those:
 *
 *  - one launch; one CTA per SM; sixteen compute warps and one helper warp;
 *  - no sequential chain on the path (exact_sum.cuh): the norm's sum of squares by
 *    parity functions, the router's logits as intervals that nearly always pin
 *    their BF16 code.  The experts whose rank the intervals decide are streamed at
 *    once; the helper warps walk the few chains that are left (one token needs one
 *    in five times) beside the stream, since only the order and the weights of the
 *    selected experts can still depend on them.  Only when the SET is open does
 *    everyone wait for the chains.  (A chain for every logit, then softmax over
 *    all of them, put 21 of 47 us in front of the first expert weight.)
 *  - selection looks at BF16 logits, not at probabilities (router_select.cuh);
 *  - weight rows are multiplied by mma.sync m16n8k16 with the tokens as the eight
 *    columns, so eight tokens cost the instructions of one (scalar multiply-adds
 *    held the gate/up phase at 27 us for 15 us of bytes at three tokens).  Each
 *    warp owns a sixteenth of K: it fetches exactly what it multiplies, into a
 *    ring of its own (cp.async), and keeps its token fragments in registers; the
 *    sixteen partial sums of a row meet in shared memory;
 *  - the ring never drains between phases: shared gate/up rows are requested
 *    before anything is known, down rows as soon as the last gate/up row has been,
 *    i.e. before the grid barrier they come after;
 *  - the down phase gives each CTA a slice of the output columns across ALL
 *    selected experts, so the combine is local and no second barrier is needed.
 *
 * CTAs wait on one another (router counter, chain counter, barrier), which is only
 * legal because the launch is cooperative (all CTAs co-resident).  Every wait is
 * bounded: on a timeout the CTA records a status code and drains to the exit.
 * The counters only ever grow, the two that count CTAs by DF_ROUND per launch (CTA 0
 * adds what the others leave to it), so that a CTA finds its launch's target in the
 * value it reads at its start, nobody has to reset anything on the way out, and the
 * kernel can be replayed from a CUDA graph.
 */
#pragma once
#include <climits>
#include <type_traits>

#include "common.cuh"
#include "decode_gemv.cuh"
#include "decode_tags.h"
#include "exact_dense.cuh"
#include "exact_sum.cuh"
#include "router_select.cuh"

namespace apus {

constexpr int DF_CW = 16;               /* compute warps */
constexpr int DF_THREADS = (DF_CW + 1) * 32;
constexpr int DF_MAX_T = 8;
constexpr int DF_MAX_A = 64;            /* T * top_k */
constexpr int DF_ROWS = 16;             /* weight rows of a tile: 8 gate + 8 up, or down rows */
constexpr int DF_PAIRS = DF_ROWS / 2;
constexpr int DF_KS = 8;                /* 16-wide k steps of a tile, at most */
constexpr int DF_MAX_K_DOWN = 4 * DF_KS * 16;   /* half of it is at most two tiles */
constexpr int DF_DEPTH = 2;             /* tiles of a warp's ring */
constexpr int DF_MAX_COLS = 16;         /* output columns of a CTA, at most */

/* ---- shared memory ------------------------------------------------------------ */
struct FusedLayout {
    int per;                 /* gate/up: k steps per warp */
    int pitch;               /* bytes of a tile row */
    int slot;                /* bytes of a ring slot */
    LaneRow lr;
    int xrow;                /* bytes of a token row (LaneRow) */
    int act_pitch, sact_pitch;
    int rrows;               /* router rows of a CTA, at most */
    int off_x, off_rr, off_code, off_tmask, off_amb, off_act, off_sact, off_red, total;
    FusedLayout() = default;
    FusedLayout(int T, int H, int I, int Is, int E, int TK, int G) {
        const int A = T * TK;
        per = (H / 16 + DF_CW - 1) / DF_CW;
        pitch = DF_KS * 32 + 16;
        slot = DF_ROWS * pitch;
        lr = LaneRow(H);
        xrow = lr.bytes();
        act_pitch = I * 2 + 16;
        sact_pitch = Is * 2 + 16;
        rrows = (E + 1 + G - 1) / G;
        int p = DF_CW * DF_DEPTH * slot;
        /* tokens, router rows, logits, open pairs; later the activations */
        off_x = p;
        off_rr = off_x + T * xrow;
        off_code = off_rr + (rrows * xrow > CH_BYTES ? rrows * xrow : CH_BYTES);
        off_tmask = off_code + T * (E + 1) * 4;
        off_amb = off_tmask + 1024;
        const int end1 = off_amb + T * (E + 1) * 2;
        off_act = p;
        off_sact = off_act + A * act_pitch;
        const int end2 = off_sact + T * sact_pitch;
        p = ((end1 > end2 ? end1 : end2) + 127) & ~127;
        /* partial sums of a tile [2][warps][rows][8]; before them the norm's gains,
         * after them the down outputs [2 halves][A + T][columns] */
        off_red = p;
        const int r1 = 2 * DF_CW * DF_ROWS * 8 * 4, r2 = 2 * (A + T) * DF_MAX_COLS * 4;
        total = p + (r1 > r2 ? r1 : r2);
    }
};

struct FusedArgs {
    int T, H, I, Is, E, TK;
    float wmin, wmax;                   /* smallest nonzero and largest |w|: router matrix */
    float wmin_gate, wmax_gate;         /* ... shared-gate row */
    const float *wnorm;                 /* [E] row norms, rounded up */
    float wnorm_gate;
    const uint16_t *x;                  /* [T, H] block input; or, with res set, unused */
    /* the two steps either side of the block folded in: res [T,H] is the residual
     * stream, the block input is rmsnorm(res, 1 + ln_w) (every CTA computes it for
     * itself: 4 KB per token, no exchange), and res_out = rnd(res + moe_out) */
    const uint16_t *res, *ln_w;
    uint16_t *res_out;
    const uint16_t *rtr_w, *exp_gu, *exp_d, *sh_g, *sh_u, *sh_d, *sh_gate;
    /* global scratch owned by the backend */
    uint32_t *code_ws;                  /* [DF_MAX_T][E + 1] logit code intervals */
    uint16_t *chain_ws;                 /* [DF_MAX_T * (E + 1)] codes of the walked chains */
    uint16_t *act_ws;                   /* [DF_MAX_A][I] */
    uint16_t *sa_ws;                    /* [DF_MAX_T][Is] */
    unsigned int *sync;                 /* [0] router, [1] barrier, [2] chains */
    /* outputs */
    uint16_t *out;                      /* [T, H] */
    int32_t *idx_out;                   /* [T, TK] (optional) */
    uint16_t *w_out;                    /* [T, TK] (optional) */
    uint16_t *tr_routed, *tr_shared, *tr_out;
    int *status;
    unsigned int *stats;                /* [0] += chains walked */
    /* optional phase timeline: [grid][DF_MARKS] global-timer nanoseconds */
    unsigned long long *timeline;
    FusedLayout L;
};
constexpr int DF_MARKS = 8;
__device__ __forceinline__ void df_mark(const FusedArgs &a, int k) {
    if (a.timeline && threadIdx.x == 0) {
        unsigned long long t;
        asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
        a.timeline[(size_t)blockIdx.x * DF_MARKS + k] = t;
    }
}

__device__ __forceinline__ unsigned int ld_acquire(const unsigned int *p) {
    unsigned int v;
    asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
    return v;
}
__device__ __forceinline__ void red_release_add(unsigned int *p, unsigned int v) {
    asm volatile("red.release.gpu.global.add.u32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}
/* the value a round counter reaches when every CTA of this launch has arrived; v was
 * read before this CTA arrived */
__device__ __forceinline__ unsigned int round_target(unsigned int v) {
    return (v & ~(DF_ROUND - 1)) + DF_ROUND;
}
__device__ __forceinline__ void round_arrive(unsigned int *p) {
    red_release_add(p, blockIdx.x == 0 ? DF_ROUND - gridDim.x + 1u : 1u);
}
/* one thread: wait until *p has reached the target (modulo 2^32); false on timeout */
__device__ __forceinline__ bool spin_until(const unsigned int *p, unsigned int target) {
    for (uint32_t i = 0; i < (1u << 21); i++) {
        if ((int)(ld_acquire(p) - target) >= 0) return true;
        if (i > 64) __nanosleep(40);
    }
    return false;
}
__device__ __forceinline__ void df_bar_compute() {
    asm volatile("bar.sync 1, %0;" ::"n"(DF_CW * 32) : "memory");
}
/* the helper warp has finished with the token rows and the logits */
__device__ __forceinline__ void df_bar_helper_arrive() {
    asm volatile("bar.arrive 2, %0;" ::"n"(DF_THREADS) : "memory");
}
__device__ __forceinline__ void df_bar_helper_wait() {
    asm volatile("bar.sync 2, %0;" ::"n"(DF_THREADS) : "memory");
}
__global__ void __launch_bounds__(DF_THREADS, 1)
decode_fused_kernel(const __grid_constant__ FusedArgs a) {
    extern __shared__ __align__(128) unsigned char df_smem[];
    const int T = a.T, H = a.H, I = a.I, Is = a.Is, E = a.E, TK = a.TK;
    const int A = T * TK, G = gridDim.x;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const FusedLayout &L = a.L;
    const LaneRow lr = L.lr;
    unsigned char *xs = df_smem + L.off_x, *rr = df_smem + L.off_rr;
    uint32_t *codes = reinterpret_cast<uint32_t *>(df_smem + L.off_code);   /* [T][E + 1] */
    uint16_t *amb = reinterpret_cast<uint16_t *>(df_smem + L.off_amb);      /* t << 11 | e */
    unsigned char *act = df_smem + L.off_act, *sact = df_smem + L.off_sact;
    uint32_t *s_tmask = reinterpret_cast<uint32_t *>(df_smem + L.off_tmask);   /* [256]: tokens of
                                                        * each expert, a byte each */
    float *red = reinterpret_cast<float *>(df_smem + L.off_red);
    __shared__ int s_sel[DF_MAX_A];                /* selected experts, in provisional order */
    __shared__ int s_idx[DF_MAX_A], s_row[DF_MAX_A];   /* final order; down output of each */
    __shared__ uint16_t s_w[DF_MAX_A];
    __shared__ float s_gate[DF_MAX_T], s_sum[DF_MAX_T], s_rs[DF_MAX_T], s_sq[2][DF_MAX_T];
    __shared__ unsigned int s_xlo[DF_MAX_T], s_xhi[DF_MAX_T];
    __shared__ int s_namb[DF_MAX_T], s_full[DF_MAX_T], s_open;
    __shared__ int s_wu[DF_CW], s_wa[DF_CW];       /* per warp: experts, assignments before it */
    __shared__ int s_uexp[DF_MAX_A], s_ubase[DF_MAX_A];
    __shared__ uint8_t s_umask[DF_MAX_A];
    __shared__ int s_U;
    __shared__ volatile int s_dead;
    __shared__ unsigned int s_chain0;              /* chain counter before this launch */

    df_mark(a, 0);                          /* start */
    /* ---- this CTA's shares ---- */
    const int r_first = blockIdx.x, n_rr = r_first <= E ? (E - r_first) / G + 1 : 0;
    /* (in 32 bits, which the sizes that fused_supported admits leave room for: a 64-bit
     * division takes half a microsecond) */
    const unsigned b = blockIdx.x, g = gridDim.x;
    const int sh_lo = (int)((unsigned)Is * b / g), sh_n = (int)((unsigned)Is * (b + 1) / g) - sh_lo;
    const int nS = (sh_n + DF_PAIRS - 1) / DF_PAIRS;   /* shared gate/up tiles */
    const int h_lo = (int)((unsigned)H * b / g);
    const int ncols = (int)((unsigned)H * (b + 1) / g) - h_lo;
    /* routed gate/up pairs and tiles, distinct experts: known after the selection */
    int gu_lo = 0, gu_n = 0, nR = 0, U = 0;

    /* ---- tokens, router rows and gains: requested first of all ---- */
    const int cph = H / 8;
    const uint4 *xsrc = reinterpret_cast<const uint4 *>(a.res ? a.res : a.x);
    auto rsrc = [&](int c) {
        const int r = c / cph, e = r_first + r * G;
        return (e == E ? a.sh_gate : a.rtr_w + (size_t)e * H) + (size_t)(c - r * cph) * 8;
    };
    uint4 rv = make_uint4(0, 0, 0, 0), xv = rv;
    if (tid < T * cph) xv = __ldcg(xsrc + tid);
    if (tid < n_rr * cph) rv = ldg16(rsrc(tid));
    uint4 gv = make_uint4(0, 0, 0, 0);       /* gain offsets; H / 8 <= the thread count */
    if (a.res && a.ln_w && tid < cph) gv = ldg16(a.ln_w + tid * 8);
    uint4 *gains = reinterpret_cast<uint4 *>(red);   /* the partial sums come later */

    /* ---- ring of this warp ---- */
    const uint32_t ring = smem_u32(df_smem + (size_t)warp * DF_DEPTH * L.slot);
    const int ks_lo = min(warp * L.per, H / 16), nks = min(L.per, H / 16 - ks_lo);
    /* fetch: a lane takes the same 16 bytes of every other row where a row slice is
     * 256 bytes (gate rows by the lower lanes, up rows by the upper ones) */
    const uint32_t f_dst = (uint32_t)((lane >> 4) * L.pitch + (lane & 15) * 16);
    const size_t f_col = (size_t)ks_lo * 16 + (lane & 15) * 8;
    const uint16_t *f_src = ((lane >> 4) ? a.sh_u : a.sh_g) + (size_t)sh_lo * H + f_col;
    int f_left = 1 << 30;                   /* pairs of the expert from f_src on */
    auto pair_row = [&](bool sh, int pi, int up) {   /* row `up` (0 gate, 1 up) of pair pi */
        if (sh) return (up ? a.sh_u : a.sh_g) + (size_t)(sh_lo + pi) * H;
        const int it = gu_lo + pi, u = it / I;
        return a.exp_gu + ((size_t)s_uexp[u] * 2 * I + (size_t)(it - u * I + (up ? I : 0))) * H;
    };
    auto fetch_pairs = [&](uint32_t slot, bool sh, int p0, int np) {
        if (nks == DF_KS && np == DF_PAIRS && f_left >= DF_PAIRS) {
#pragma unroll
            for (int q = 0; q < DF_PAIRS; q++)
                cp_async16_to(slot + f_dst + (uint32_t)(2 * q * L.pitch), f_src + (size_t)q * H);
        } else if (nks > 0) {
            /* ragged: the slice is narrower, or the tile ends or changes expert */
            const int cpr = nks * 2;
#pragma unroll 1
            for (int c = lane; c < 2 * np * cpr; c += 32) {
                const int r = c / cpr, ch = c - r * cpr;
                cp_async16_to(slot + (uint32_t)(r * L.pitch + ch * 16),
                              pair_row(sh, p0 + (r >> 1), r & 1) + ks_lo * 16 + ch * 8);
            }
        }
        f_src += (size_t)DF_PAIRS * H;
        f_left -= DF_PAIRS;
        if (!sh && f_left <= 0 && p0 + DF_PAIRS < gu_n) {      /* the next tile's expert */
            const int it = gu_lo + p0 + DF_PAIRS, u = it / I;
            f_src = pair_row(false, p0 + DF_PAIRS, lane >> 4) + f_col;
            f_left = (u + 1) * I - it;
        }
    };
    /* Down: warp w takes (item, half of K) = w, w + 16, ...; items are the distinct
     * experts and, last, the shared expert.  A unit is one or two tiles of at most
     * 128 k, all of this CTA's columns high. */
    struct DownUnit {
        const uint16_t *src;
        int K, k0, nk;                      /* first k step, k steps */
    };
    auto down_unit = [&](int j) {
        const int v = j * DF_CW + warp, item = v >> 1;
        DownUnit d;
        d.K = item == U ? Is : I;
        const int half = (d.K / 16 + 1) / 2;
        d.k0 = (v & 1) * half;
        d.nk = min(half, d.K / 16 - d.k0);
        d.src = (item == U ? a.sh_d : a.exp_d + (size_t)s_uexp[item] * H * I) +
                (size_t)h_lo * d.K + d.k0 * 16;
        return d;
    };
    auto fetch_down = [&](uint32_t slot, const DownUnit &d, int ks0) {
        const int cpr = 2 * min(DF_KS, d.nk - ks0);
        const uint16_t *src = d.src + ks0 * 16;
        if (cpr == 16) {
            src += (size_t)(lane >> 4) * d.K + (lane & 15) * 8;
#pragma unroll
            for (int q = 0; q < DF_ROWS / 2; q++)
                if (2 * q + (lane >> 4) < ncols)
                    cp_async16_to(slot + f_dst + (uint32_t)(2 * q * L.pitch),
                                  src + (size_t)(2 * q) * d.K);
        } else {
#pragma unroll 1
            for (int c = lane; c < ncols * cpr; c += 32) {
                const int r = c / cpr, ch = c - r * cpr;
                cp_async16_to(slot + (uint32_t)(r * L.pitch + ch * 16),
                              src + (size_t)r * d.K + ch * 8);
            }
        }
    };
    int i_tile = 0, i_slot = 0;             /* next gate/up tile of the phase, next slot */
    int i_unit = 0, i_ks = 0, n_unit = 0;   /* next down unit and k step in it */
    /* requests this warp's next tile if it is known; one commit group per call, so
     * that a fixed number of groups stays ahead of the tile in use.  The callers say what it
     * can be: the kernel waits for its instructions wherever they are new, so none of what a
     * phase never requests lies in its way (a stack of four layers at 1 / 3 / 8 tokens 138 /
     * 210 / 368 -> 136 / 202 / 361 us). */
    constexpr int SHARED = 0, ROUTED = 1, DOWN = 2;
    auto issue = [&](auto phase) {
        constexpr int PHASE = decltype(phase)::value;
        const uint32_t slot = ring + (uint32_t)(i_slot * L.slot);
        bool some = false;
        if (PHASE != DOWN && i_tile < (PHASE == SHARED ? nS : nR)) {
            const int p0 = i_tile++ * DF_PAIRS;
            fetch_pairs(slot, PHASE == SHARED, p0,
                        min(DF_PAIRS, (PHASE == SHARED ? sh_n : gu_n) - p0));
            some = true;
        } else if (PHASE != SHARED && i_unit < n_unit) {
            const DownUnit d = down_unit(i_unit);
            fetch_down(slot, d, i_ks);
            i_ks += DF_KS;
            if (i_ks >= d.nk) {
                i_ks = 0;
                i_unit++;
            }
            some = true;
        }
        if (some && ++i_slot == DF_DEPTH) i_slot = 0;
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    if (warp < DF_CW)
#pragma unroll 1
        for (int j = 0; j < DF_DEPTH; j++)   /* constants: nothing to wait for */
            issue(std::integral_constant<int, SHARED>());

    unsigned int sync_at[2] = {0, 0};
    if (tid == 0) {
        s_dead = 0;
        s_open = 0;
        s_U = 0;
        /* one round trip: nothing is read on the strength of these */
        const uint4 v = __ldcg(reinterpret_cast<const uint4 *>(a.sync));
        sync_at[0] = round_target(v.x);
        sync_at[1] = round_target(v.y);
        s_chain0 = v.z;
    }
    if (tid < DF_MAX_T) {
        s_xlo[tid] = 0x7f800000u;
        s_xhi[tid] = 0;
    }
    if (tid < cph) gains[tid] = gv;
#pragma unroll 1
    for (int c = tid, t = tid / cph; c < T * cph; c += DF_THREADS, t = c / cph) {
        if (c != tid) xv = __ldcg(xsrc + c);
        *reinterpret_cast<uint4 *>(xs + t * L.xrow + lr.at(c - t * cph)) = xv;
    }
#pragma unroll 1
    for (int c = tid, r = tid / cph; c < n_rr * cph; c += DF_THREADS, r = c / cph) {
        if (c != tid) rv = ldg16(rsrc(c));
        *reinterpret_cast<uint4 *>(rr + r * L.xrow + lr.at(c - r * cph)) = rv;
    }
    __syncthreads();
    /* Norm (bit for bit the engine's) and the range of the tokens' values: warps t
     * and 8 + t have a half of token t each, where its lane chunks can be halved. */
    {
        const int t = warp & 7, part = warp >> 3, parts = lr.nu % 2 == 0 ? 2 : 1;
        if (t < T && part < parts) {
            unsigned char *row = xs + t * L.xrow;
            float rs = 1.0f;
            auto meet = [&] { asm volatile("bar.sync %0, 64;" ::"r"(3 + t) : "memory"); };
            if (a.res) {
                const float ss =
                    lr.nu / parts <= 4
                        ? exact_sumsq<4, false>(row, lr, lane, part, parts, &s_sum[t], meet)
                        : exact_sumsq<0, false>(row, lr, lane, part, parts, &s_sum[t], meet);
                if (part) s_rs[t] = norm_scale(ss, H);
                if (parts == 2) {
                    meet();
                    rs = s_rs[t];
                } else {
                    rs = norm_scale(ss, H);
                }
            }
            PackedRange range;
            float sq = 0.0f;
            /* (rolled: unrolled twice, a layer waited 1.2 us longer for instructions) */
#pragma unroll 1
            for (int c = part * 32 + lane; c < cph; c += 32 * parts) {
                uint4 *p = reinterpret_cast<uint4 *>(row + lr.at(c));
                uint4 v = *p;
                if (a.res) *p = v = norm8(v, gains[c], rs);
                range.fold8(v);
                float f[8];
                unpack8(v, f);
#pragma unroll
                for (int j = 0; j < 8; j++) sq = fmaf(f[j], f[j], sq);
            }
            sq = warp_sum(sq);
            const unsigned lo = __reduce_min_sync(0xffffffffu, range.low()),
                           hi = __reduce_max_sync(0xffffffffu, range.high());
            if (lane == 0) {
                s_sq[part][t] = sq;
                atomicMin(&s_xlo[t], lo);
                atomicMax(&s_xhi[t], hi);
            }
        }
    }
    __syncthreads();

    /* ---- router logits of this CTA's rows ---- */
    if (warp < DF_CW)
        for (int p = warp; p < n_rr * T; p += DF_CW) {
            const int r = p / T, t = p - r * T, e = r_first + r * G;
            const bool exact =
                e == E ? products_exact(a.wmin_gate, a.wmax_gate, s_xlo[t], s_xhi[t])
                       : products_exact(a.wmin, a.wmax, s_xlo[t], s_xhi[t]);
            uint32_t v = CODE_UNKNOWN;
            if (exact) {
                const float sq = s_sq[0][t] + (lr.nu % 2 == 0 ? s_sq[1][t] : 0.0f),
                            wn = e == E ? a.wnorm_gate : __ldg(&a.wnorm[e]);
                v = certified_logit(rr + r * L.xrow, xs + t * L.xrow, lr, lane,
                                    wn * norm_above(sq, H));
            }
            if (lane == 0) a.code_ws[(size_t)t * (E + 1) + e] = v;
        }
    __syncthreads();
    if (tid == 0) round_arrive(&a.sync[0]);          /* cumulative over the barrier */
    df_mark(a, 1);                          /* own logits published */

    /* ---- token fragments of this warp's k slice (all tokens are columns) ---- */
    uint32_t bf[DF_KS][2];
    {
        const int t = lane >> 2, q = (lane & 3) * 2;
#pragma unroll
        for (int s = 0; s < DF_KS; s++) {
            bf[s][0] = bf[s][1] = 0;
            if (warp < DF_CW && s < nks && t < T) {
                const unsigned char *row = xs + t * L.xrow;
                const int c = (ks_lo + s) * 2;
                bf[s][0] = *reinterpret_cast<const uint32_t *>(row + lr.at(c) + q * 2);
                bf[s][1] = *reinterpret_cast<const uint32_t *>(row + lr.at(c + 1) + q * 2);
            }
        }
    }
    int c_slot = 0;
    /* where ldmatrix finds this lane's row of the tile in use: matrices are (rows
     * 0-7, k 0-7), (rows 8-15, k 0-7), (rows 0-7, k 8-15), (rows 8-15, k 8-15) */
    const uint32_t m_off = (uint32_t)((lane & 15) * L.pitch + (lane >> 4) * 16);
    auto next_tile = [&]() {
        asm volatile("cp.async.wait_group %0;" ::"n"(DF_DEPTH - 1) : "memory");
        __syncwarp();
        const uint32_t t = ring + (uint32_t)(c_slot * L.slot) + m_off;
        if (++c_slot == DF_DEPTH) c_slot = 0;
        return t;
    };
    /* gate/up tiles [0, n): the warps' partial sums meet in shared memory, four
     * warps in turn finish a tile while the others go on */
    auto run_tiles = [&](int n, auto phase) {
        constexpr bool sh = decltype(phase)::value == SHARED;
#pragma unroll 1
        for (int j = 0; j < n; j++) {
            float *buf = red + (j & 1) * (DF_CW * DF_ROWS * 8);
            const uint32_t t = next_tile();
            float c0[4] = {0.f, 0.f, 0.f, 0.f}, c1[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
            for (int s = 0; s < DF_KS; s++)
                if (s < nks) {
                    uint32_t r[4];
                    ldmatrix_x4(r, t + (uint32_t)(s * 32));
                    mma_16x8((s & 1) ? c1 : c0, r, bf[s][0], bf[s][1]);
                }
            float *dst = buf + (warp * DF_ROWS + (lane >> 2)) * 8 + (lane & 3) * 2;
            *reinterpret_cast<float2 *>(dst) = make_float2(c0[0] + c1[0], c0[1] + c1[1]);
            *reinterpret_cast<float2 *>(dst + 64) = make_float2(c0[2] + c1[2], c0[3] + c1[3]);
            __syncwarp();                       /* the slot is read out */
            issue(phase);
            df_bar_compute();
            if ((warp >> 2) == (j & 3)) {
                /* thread = row (2p gate, 2p + 1 up) x column */
                const int i = (warp & 3) * 32 + lane, col = i & 7, pi = j * DF_PAIRS + (i >> 4);
                float v = 0.0f;
#pragma unroll
                for (int w = 0; w < DF_CW; w++) v += buf[w * (DF_ROWS * 8) + i];
                const float up = __shfl_xor_sync(0xffffffffu, v, 8);
                if (!(i & 8) && pi < (sh ? sh_n : gu_n)) {
                    const float g = bf16_round(v), u = bf16_round(up);
                    if (sh) {
                        if (col < T)
                            a.sa_ws[(size_t)col * Is + sh_lo + pi] = silu_mul_bits(g, u);
                    } else {
                        const int it = gu_lo + pi, uu = it / I;
                        const unsigned m = s_umask[uu];
                        if ((m >> col) & 1u)
                            a.act_ws[(size_t)(s_ubase[uu] + __popc(m & ((1u << col) - 1u))) * I +
                                     (it - uu * I)] = silu_act_bits(g, u);
                    }
                }
            }
        }
    };
    if (warp < DF_CW) run_tiles(nS, std::integral_constant<int, SHARED>());
    df_mark(a, 2);                          /* shared gate/up done */
    /* ---- routing ---- */
    if (tid == 0 && !spin_until(&a.sync[0], sync_at[0])) {
        set_status(a.status, ST_SCHED_TIMEOUT);
        s_dead = 1;
    }
    if (tid < 256) s_tmask[tid] = 0;
    __syncthreads();
    bool dead = s_dead != 0;
    /* four requested before the first is stored: eight tokens' are four to a thread */
#pragma unroll 1
    for (int i0 = tid; i0 < T * (E + 1); i0 += 4 * DF_THREADS) {
        uint32_t v[4];
#pragma unroll
        for (int q = 0; q < 4; q++) {
            const int i = i0 + q * DF_THREADS;
            v[q] = i < T * (E + 1) && !dead ? __ldcg(&a.code_ws[i]) : 0u;
        }
#pragma unroll
        for (int q = 0; q < 4; q++)
            if (i0 + q * DF_THREADS < T * (E + 1)) codes[i0 + q * DF_THREADS] = v[q];
    }
    __syncthreads();
    uint32_t kkey = 0;
    if (warp < T && !dead) {
        const uint32_t *cd = codes + warp * (E + 1);
        const Choice c = rt_select(cd, E, TK, lane, s_sel + warp * TK);
        kkey = c.kkey;
        int n = 0;
        if (c.any)
#pragma unroll 1
            for (int e0 = 0; e0 <= E; e0 += 32)
                n += __popc(__ballot_sync(0xffffffffu, rt_needs(cd, e0 + lane, E, kkey, c.odd)));
        if (lane == 0) {
            s_namb[warp] = n;
            s_full[warp] = c.odd;
            if (c.open || c.odd) s_open = 1;
        }
    }
    __syncthreads();
    int n_amb = 0;
    if (!dead)
        for (int t = 0; t < T; t++) n_amb += s_namb[t];
    if (n_amb > 0) {
        if (warp < T) {
            /* the same list in every CTA: by token, then by expert */
            int at = 0;
            for (int t = 0; t < warp; t++) at += s_namb[t];
            const uint32_t *cd = codes + warp * (E + 1);
            for (int e0 = 0; e0 <= E; e0 += 32) {
                const int e = e0 + lane;
                const bool need = rt_needs(cd, e, E, kkey, s_full[warp] != 0);
                const unsigned m = __ballot_sync(0xffffffffu, need);
                if (need) amb[at + __popc(m & ((1u << lane) - 1u))] = (uint16_t)((warp << 11) | e);
                at += __popc(m);
            }
        }
        __syncthreads();
    }
    const bool open = s_open != 0;           /* the set itself waits for the chains */
    /* Pair i of the list is CTA i % G's; its helper warp walks it, the products in the
     * place of the router rows. */
    auto walk_chains = [&]() {
        if ((int)blockIdx.x >= n_amb) return;
        for (int i = blockIdx.x; i < n_amb; i += G) {
            const int t = amb[i] >> 11, e = amb[i] & 0x7ff;
            const uint16_t *w = e == E ? a.sh_gate : a.rtr_w + (size_t)e * H;
            const unsigned char *xr = xs + t * L.xrow;
            const float z = warp_chains<CH_CHAINS>(
                1, H, lane, reinterpret_cast<float *>(rr),
                [&](int) { return w; },
                [&](int p) { return *reinterpret_cast<const uint4 *>(xr + lr.at(p)); });
            if (lane == 0) a.chain_ws[i] = bf16_bits(z);
        }
        if (lane == 0) {
            if (a.stats && blockIdx.x == 0) atomicAdd(&a.stats[0], (unsigned)n_amb);
            red_release_add(&a.sync[2], 1u);
        }
    };
    const unsigned chain_target = s_chain0 + (unsigned)min(n_amb, G);
    if (open) {
        if (warp == DF_CW) walk_chains();
        if (tid == 0 && !spin_until(&a.sync[2], chain_target)) {
            set_status(a.status, ST_SCHED_TIMEOUT);
            s_dead = 1;
        }
        __syncthreads();
        dead = s_dead != 0;
        for (int i = tid; i < n_amb && !dead; i += DF_THREADS) {
            const uint32_t c = __ldcg(&a.chain_ws[i]);
            codes[(amb[i] >> 11) * (E + 1) + (amb[i] & 0x7ff)] = c | (c << 16);
        }
        __syncthreads();
        if (warp < T && !dead) {
            if (s_full[warp]) {
                /* the engine's softmax and selection on exact logits */
                float *p = reinterpret_cast<float *>(codes + warp * (E + 1));
                for (int e = lane; e < E; e += 32) p[e] = bf16lo(codes[warp * (E + 1) + e]);
                __syncwarp();
                router_softmax_topk(p, E, TK, lane, s_idx + warp * TK, s_w + warp * TK);
                __syncwarp();
                for (int i = lane; i < TK; i += 32) s_sel[warp * TK + i] = s_idx[warp * TK + i];
            } else {
                rt_select(codes + warp * (E + 1), E, TK, lane, s_sel + warp * TK);
            }
        }
        __syncthreads();
    }
    /* ---- the distinct experts, ascending, and who uses them ---- */
    if (tid < A && !dead)
        atomicOr(&s_tmask[s_sel[tid] >> 2], (1u << (tid / TK)) << ((s_sel[tid] & 3) * 8));
    __syncthreads();
    if (warp < DF_CW) {
        /* warp w looks at experts 64 w .. 64 w + 63 */
        unsigned m0 = 0, m1 = 0;
        const int e0 = warp * 64 + lane, e1 = e0 + 32;
        const unsigned b0 = (s_tmask[e0 >> 2] >> ((e0 & 3) * 8)) & 0xffu,
                       b1 = (s_tmask[e1 >> 2] >> ((e1 & 3) * 8)) & 0xffu;
        m0 = __ballot_sync(0xffffffffu, b0 != 0);
        m1 = __ballot_sync(0xffffffffu, b1 != 0);
        int c0 = __popc(b0), c1 = __popc(b1), i0 = c0, i1 = c1;
#pragma unroll
        for (int d = 1; d < 32; d <<= 1) {
            const int v0 = __shfl_up_sync(0xffffffffu, i0, d),
                      v1 = __shfl_up_sync(0xffffffffu, i1, d);
            if (lane >= d) { i0 += v0; i1 += v1; }
        }
        const int t0 = __shfl_sync(0xffffffffu, i0, 31), t1 = __shfl_sync(0xffffffffu, i1, 31);
        if (lane == 0) {
            s_wu[warp] = __popc(m0) + __popc(m1);
            s_wa[warp] = t0 + t1;
        }
        df_bar_compute();
        int ub = 0, ab = 0;
        const int nw = (E + 63) / 64;
        for (int w = 0; w < min(warp, nw); w++) {
            ub += s_wu[w];
            ab += s_wa[w];
        }
        const unsigned below = (1u << lane) - 1u;
        if (b0) {
            const int u = ub + __popc(m0 & below);
            s_uexp[u] = e0; s_umask[u] = (uint8_t)b0; s_ubase[u] = ab + i0 - c0;
        }
        if (b1) {
            const int u = ub + __popc(m0) + __popc(m1 & below);
            s_uexp[u] = e1; s_umask[u] = (uint8_t)b1; s_ubase[u] = ab + t0 + i1 - c1;
        }
        if (warp == nw - 1 && lane == 0) s_U = ub + s_wu[warp];
    }
    __syncthreads();
    U = dead ? 0 : s_U;
    df_mark(a, 3);                          /* selection known */

    if (warp == DF_CW) {
        /* ---- helper warp: chains, final order, weights, shared gate ---- */
        if (!open && n_amb > 0) {
            walk_chains();
            bool ok = true;
            if (lane == 0) ok = spin_until(&a.sync[2], chain_target);
            ok = __shfl_sync(0xffffffffu, (int)ok, 0) != 0;
            if (!ok) set_status(a.status, ST_SCHED_TIMEOUT);
            for (int i = lane; i < n_amb && ok; i += 32) {
                const uint32_t c = __ldcg(&a.chain_ws[i]);
                codes[(amb[i] >> 11) * (E + 1) + (amb[i] & 0x7ff)] = c | (c << 16);
            }
            __syncwarp();
        }
        for (int t = 0; t < T && !dead; t++) {
            if (!s_full[t])
                rt_weights(codes + t * (E + 1), s_sel + t * TK, TK, lane, s_idx + t * TK,
                           s_w + t * TK);
            if (lane == 0)
                s_gate[t] = bf16_round(sigmoid_f32(bf16lo(codes[t * (E + 1) + E])));
        }
        __syncwarp();
        /* where the down output of each slot will be */
        for (int i = lane; i < A && !dead; i += 32) {
            const int t = i / TK, e = s_idx[i];
            int lo = 0, hi = U - 1;
            while (lo < hi) {
                const int mid = (lo + hi) >> 1;
                if (s_uexp[mid] < e) lo = mid + 1; else hi = mid;
            }
            s_row[i] = s_ubase[lo] + __popc(s_umask[lo] & ((1u << t) - 1u));
            if (blockIdx.x == 0) {
                if (a.idx_out) a.idx_out[i] = e;
                if (a.w_out) a.w_out[i] = s_w[i];
            }
        }
        __syncwarp();
        df_bar_helper_arrive();
        return;
    }

    /* ---- routed gate/up ---- */
    if (!dead) {
        gu_lo = (int)((unsigned)(U * I) * b / g);
        gu_n = (int)((unsigned)(U * I) * (b + 1) / g) - gu_lo;
        nR = (gu_n + DF_PAIRS - 1) / DF_PAIRS;
        const int units = 2 * (U + 1);
        n_unit = warp < units ? (units - warp + DF_CW - 1) / DF_CW : 0;
        if (gu_n > 0) {
            f_src = pair_row(false, 0, lane >> 4) + f_col;
            f_left = (gu_lo / I + 1) * I - gu_lo;
        }
    }
    i_tile = 0;
#pragma unroll 1
    for (int j = 0; j < DF_DEPTH; j++) issue(std::integral_constant<int, ROUTED>());
    run_tiles(nR, std::integral_constant<int, ROUTED>());
    df_mark(a, 4);                      /* routed gate/up done */
    df_bar_compute();
    if (tid == 0) {
        round_arrive(&a.sync[1]);
        if (!spin_until(&a.sync[1], sync_at[1])) {
            set_status(a.status, ST_SCHED_TIMEOUT);
            s_dead = 1;
        }
    }
    df_bar_helper_wait();               /* token rows and logits make room */
    dead = s_dead != 0;
    df_mark(a, 5);                      /* barrier passed */
    {
        /* routed activations, then the shared ones: four pieces requested before
         * the first is stored */
        const int ci = I / 8, cs = Is / 8, na = A * ci, n = na + T * cs;
#pragma unroll 1
        for (int c0 = tid; c0 < n; c0 += 4 * DF_CW * 32) {
            uint4 v[4];
            uint32_t dst[4];
#pragma unroll
            for (int q = 0; q < 4; q++) {
                const int c = c0 + q * DF_CW * 32;
                if (c < n) {
                    const bool sh = c >= na;
                    const int k = sh ? c - na : c, w = sh ? cs : ci, r = k / w;
                    v[q] = __ldcg(reinterpret_cast<const uint4 *>(sh ? a.sa_ws : a.act_ws) + k);
                    dst[q] = (uint32_t)((sh ? L.off_sact + r * L.sact_pitch
                                            : L.off_act + r * L.act_pitch) + (k - r * w) * 16);
                }
            }
#pragma unroll
            for (int q = 0; q < 4; q++)
                if (c0 + q * DF_CW * 32 < n) *reinterpret_cast<uint4 *>(df_smem + dst[q]) = v[q];
        }
    }
    df_bar_compute();
    /* ---- down rows of this CTA's columns ---- */
#pragma unroll 1
    for (int j = 0; j < n_unit; j++) {
        const DownUnit d = down_unit(j);
        const int v = j * DF_CW + warp, item = v >> 1;
        const bool sh = item == U;
        const int cnt = sh ? T : __popc(s_umask[item]), row0 = sh ? 0 : s_ubase[item];
        const int n = min(lane & 7, cnt - 1);            /* extra columns are not used */
        uint32_t ba = (sh ? smem_u32(sact) + (uint32_t)(n * L.sact_pitch)
                          : smem_u32(act) + (uint32_t)((row0 + n) * L.act_pitch)) +
                      (uint32_t)(d.k0 * 32 + (lane >> 3) * 16);
        float c0[4] = {0.f, 0.f, 0.f, 0.f}, c1[4] = {0.f, 0.f, 0.f, 0.f};
        /* a second half without a k step (16 values in all) is a turn and a slot of the
         * ring like any other, as in issue() */
        int ks0 = 0;
#pragma unroll 1
        do {
            const uint32_t t = next_tile();
            const int nk = min(DF_KS, d.nk - ks0);
            /* mma.sync cuts off what its accumulator cannot hold: two steps on one that
             * starts at zero, sums of those rounded to nearest.  Eight steps on one
             * narrowed 1.02e-4 of the outputs to another BF16 value than 64-bit sums
             * do (K 512), this 0.79e-4, as scalar multiply-adds did (0.78e-4).  The
             * gate/up tiles end in a sum of sixteen warps and need no more than that
             * (0.98e-4 of K 2048; scalar 1.04e-4). */
#pragma unroll
            for (int s = 0; s < DF_KS; s += 2)
                if (s < nk) {
                    uint32_t br[4], r[4];
                    float p[4] = {0.f, 0.f, 0.f, 0.f};
                    ldmatrix_x4(br, ba + (uint32_t)(s * 32));
                    ldmatrix_x4(r, t + (uint32_t)(s * 32));
                    mma_16x8(p, r, br[0], br[1]);
                    if (s + 1 < nk) {
                        ldmatrix_x4(r, t + (uint32_t)(s * 32 + 32));
                        mma_16x8(p, r, br[2], br[3]);
                    }
#pragma unroll
                    for (int q = 0; q < 4; q++) ((s & 2) ? c1 : c0)[q] += p[q];
                }
            __syncwarp();
            issue(std::integral_constant<int, DOWN>());
            ks0 += DF_KS;
            ba += DF_KS * 32;
        } while (ks0 < d.nk);
        const int r = lane >> 2, col = (lane & 3) * 2;
        float *dst = red + ((size_t)(v & 1) * (A + T) + (sh ? A : row0) + col) * DF_MAX_COLS + r;
        if (col < cnt) {
            dst[0] = c0[0] + c1[0];
            dst[8] = c0[2] + c1[2];
        }
        if (col + 1 < cnt) {
            dst[DF_MAX_COLS] = c0[1] + c1[1];
            dst[DF_MAX_COLS + 8] = c0[3] + c1[3];
        }
    }
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    df_bar_compute();
    df_mark(a, 6);                      /* down rows done */

    /* ---- combine (c/layer.h:350,356-361), this CTA's columns ---- */
    if (!dead && tid < T * ncols) {
        const int t = tid / ncols, h = tid - t * ncols;
        const float *y0 = red, *y1 = red + (size_t)(A + T) * DF_MAX_COLS;
        float acc = 0.0f;
        for (int s = 0; s < TK; s++) {
            const int o = s_row[t * TK + s] * DF_MAX_COLS + h;
            acc = __fadd_rn(acc, __fmul_rn(bf16_f32(s_w[t * TK + s]), bf16_round(y0[o] + y1[o])));
        }
        const float routed = bf16_round(acc);
        const int o = (A + t) * DF_MAX_COLS + h;
        const float shared = bf16_round(__fmul_rn(bf16_round(y0[o] + y1[o]), s_gate[t]));
        const uint16_t v = bf16_bits(__fadd_rn(routed, shared));
        const size_t at = (size_t)t * H + h_lo + h;
        if (a.out) a.out[at] = v;
        if (a.res_out)                          /* c/layer.h:230-234,388 */
            a.res_out[at] = bf16_bits(__fadd_rn(bf16_f32(a.res[at]), bf16_f32(v)));
        if (a.tr_out) a.tr_out[at] = v;
        if (a.tr_routed) a.tr_routed[at] = bf16_bits(routed);
        if (a.tr_shared) a.tr_shared[at] = bf16_bits(shared);
    }
    df_mark(a, 7);                      /* combine done */
}

}  // namespace apus
