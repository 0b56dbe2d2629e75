/*
 * decode_stack.cuh — the MoE block for one to eight tokens, and stacks of layers of it, in ONE
 * cooperative kernel, for rows of 2048 values (decode_fused.cuh has the same steps for other
 * shapes, one layer per launch; its head comment explains them: intervals for the logits, the
 * selection on BF16 codes, mma.sync with the tokens as columns, one grid barrier).
 *
 * What bounds a layer at few tokens is not the 58 MB of weights (9 us) but instructions: each is
 * fetched for the first time when it is needed, at about 8 cycles an instruction out of L2, 2.7
 * once it is in the 128 KB that an SM keeps, 1 in the innermost 28 KB.  (decode_fused_kernel:
 * 176 KB of code; 25 % of the warps' time waiting for instructions.  Here: 111 KB, and 29 in
 * functions beside a layer's way.)  So
 *  - a stack of layers is a loop in the kernel: from the second layer on, the code is there, and
 *    no launch lies between two layers, only a grid barrier;
 *  - there is little code: the row length is a constant, loops are rolled where a phase runs once,
 *    the shared and the routed gate/up rows go through the same loop, and so does a tile of down
 *    rows through the same fragments;
 *  - weights come by bulk copies that one warp requests (a tile of eight gate and eight up rows
 *    is two requests of 32 KB, an expert's down rows one): the multiplying warps carry no
 *    addresses.  (A request costs the copy engine 60 cycles, so rows of 1 KB one by one stream
 *    at 4.4 TB/s and pieces of 2 KB and more at 7.0.)
 *  - what a warp waits for comes with its own validity where it is small: logits and chains are
 *    64-bit words that hold the layer's tag (decode_tags.h), so no counter, fence and second
 *    look.
 *
 * Copies are dense, so the rows of a fragment lie on the same banks; a lane's 16 bytes are four
 * k steps of its row, and odd rows read the two halves of a 128-byte line the other way round.
 */
#pragma once
#include "decode_fused.cuh"

namespace apus {

constexpr int DS_H = 2048;              /* values of a row */
constexpr int DS_CW = 16;               /* multiplying warps; each has 128 k of a row */
constexpr int DS_THREADS = (DS_CW + 2) * 32;    /* a requesting warp and a helper more */
constexpr int DS_PAIRS = 8;             /* gate/up pairs of a tile */
constexpr int DS_CELL = 16 * 1024;      /* down rows of an expert: at most 16 of 1 KB */
constexpr int DS_CELLS = 8;
constexpr int DS_TILE = 2 * DS_PAIRS * DS_H * 2;        /* 64 KB: four cells */
constexpr int DS_WORDS = DF_MAX_T * 1025;       /* tagged words of logits, and of chains */
static_assert(CH_BYTES <= 8 * sizeof(SumShare), "a chain's products in the place of the sums'");
static_assert(DS_CELL * DS_CELLS == 2 * DS_TILE, "two tiles or eight cells");

struct StackLayout {
    int xrow, rrows;
    int off_x, off_rr, off_gain, off_share, off_code, off_tmask, off_amb, off_red, total;
    StackLayout() = default;
    StackLayout(int T, int I, int E, int TK, int G) {
        const int A = T * TK;
        xrow = LaneRow(DS_H).bytes();
        rrows = (E + 1 + G - 1) / G;
        off_x = 2 * DS_TILE;
        off_rr = off_x + T * xrow;
        off_gain = off_rr + rrows * xrow;
        off_share = off_gain + DS_H * 2;
        off_code = off_share + 8 * (int)sizeof(SumShare);
        off_tmask = (off_code + T * (E + 1) * 4 + 7) & ~7;
        off_amb = off_tmask + 1024;
        off_red = (off_amb + T * (E + 1) * 2 + 127) & ~127;
        /* partial sums of a tile [2][warps][rows][8]; later the down outputs
         * [128-k slices][A + T][columns] */
        const int r1 = 2 * DS_CW * 2 * DS_PAIRS * 8 * 4,
                  r2 = I / 128 * (A + T) * DF_MAX_COLS * 4;
        total = off_red + (r1 > r2 ? r1 : r2);
    }
};

struct StackLayer {
    float wmin, wmax;                   /* smallest nonzero and largest |w|: router matrix */
    float wmin_gate, wmax_gate;         /* ... shared-gate row */
    float wnorm_gate;
    const float *wnorm;                 /* [E] row norms, rounded up */
    const uint16_t *ln_w;
    const uint16_t *rtr_w, *exp_gu, *exp_d, *sh_g, *sh_u, *sh_d, *sh_gate;
};
struct StackArgs {
    int T, I, E, TK;
    int slices_log2;                    /* 128-k slices of a down row: I = 128 << this, 1 or 2 */
    int n_layers;                       /* > 1: in place on res_out == res */
    const uint16_t *x;                  /* as in FusedArgs */
    const uint16_t *res;
    uint16_t *res_out;
    uint64_t *code_ws;                  /* [T][E + 1] logit code intervals, tag above */
    uint64_t *chain_ws;                 /* [T * (E + 1)] codes of the walked chains, tag; both
                                         * of DS_WORDS */
    uint16_t *act_ws;                   /* [DF_MAX_A + DF_MAX_T][I] */
    unsigned int *sync;                 /* barrier */
    int absent;                         /* a CTA that leaves at once (a test's), or -1 */
    uint16_t *out;
    int32_t *idx_out;
    uint16_t *w_out;
    uint16_t *tr_routed, *tr_shared, *tr_out;
    int *status;
    unsigned int *stats;                /* [0] += chains walked */
    unsigned long long *timeline;       /* of the last layer */
    StackLayout L;
    StackLayer layer[DS_LAYERS];
};

/* a word that carries its own validity: 64 bits are stored and loaded as one */
__device__ __forceinline__ void st_tagged(uint64_t *p, uint32_t v, uint32_t tag) {
    asm volatile("st.relaxed.gpu.global.u64 [%0], %1;" ::"l"(p), "l"(v | ((uint64_t)tag << 32))
                 : "memory");
}
__device__ __forceinline__ uint64_t ld_tagged(const uint64_t *p) {
    uint64_t v;
    asm volatile("ld.relaxed.gpu.global.u64 %0, [%1];" : "=l"(v) : "l"(p) : "memory");
    return v;
}

/* both codes of an interval, a zero always the positive one (the order of the codes as integers
 * is then that of the values, but for the sign) */
__device__ __forceinline__ uint32_t no_negative_zero(uint32_t v) {
    if ((v & 0xffffu) == 0x8000u) v &= 0xffff0000u;
    if ((v >> 16) == 0x8000u) v &= 0xffffu;
    return v;
}
/* Waits end when what they wait for is there, at their limit, or when the CTA has given up
 * elsewhere (`dead`), so that one limit is waited for and not one for every piece that is missing.
 * (rolled: the compiler's unrolling of the waits alone was 40 KB) */
__device__ __forceinline__ bool ds_wait(uint64_t *bar, uint32_t parity, const volatile int &dead) {
#pragma unroll 1
    for (uint32_t i = 0; i < APUS_WAIT_LIMIT; i++) {
        if (mbar_try_wait(bar, parity)) return true;
        if (i > 64) {
            if (dead) return false;
            __nanosleep(64);
        }
    }
    return false;
}
__device__ __forceinline__ bool ds_spin(const unsigned int *p, unsigned int target,
                                        const volatile int &dead) {
#pragma unroll 1
    for (uint32_t i = 0; i < (1u << 21); i++) {
        if ((int)(ld_acquire(p) - target) >= 0) return true;
        if (i > 64) {
            if (dead) return false;
            __nanosleep(40);
        }
    }
    return false;
}

__device__ __forceinline__ bool mbar_test(uint64_t *bar, uint32_t parity) {
    uint32_t ok;
    asm volatile(
        "{\n"
        ".reg .pred p;\n"
        "mbarrier.test_wait.parity.shared::cta.b64 p, [%1], %2;\n"
        "selp.u32 %0, 1, 0, p;\n"
        "}\n"
        : "=r"(ok)
        : "r"(smem_u32(bar)), "r"(parity)
        : "memory");
    return ok != 0;
}

/* A lane's share of a row's 128-k slice: 16 bytes of each of its four 64-byte windows, which
 * are the operands of two k steps each.  p: the row's slice + (lane & 3) * 16. */
__device__ __forceinline__ void slice_pieces(const unsigned char *p, bool odd, uint4 (&f)[4]) {
#pragma unroll
    for (int l = 0; l < 2; l++) {
        const uint4 a = *reinterpret_cast<const uint4 *>(p + l * 128 + (odd ? 64 : 0)),
                    b = *reinterpret_cast<const uint4 *>(p + l * 128 + (odd ? 0 : 64));
        f[2 * l] = odd ? b : a;
        f[2 * l + 1] = odd ? a : b;
    }
}

struct StackShared {
    uint64_t tile_full[2], tile_free[2], cell_full[DS_CELLS], cell_free[DS_CELLS];
    float gate[DF_MAX_T], sq[4][DF_MAX_T];
    float part[2][DS_CW];               /* a logit's parts: sums, error terms */
    unsigned int xlo[DF_MAX_T], xhi[DF_MAX_T];
    int sel[DF_MAX_A];                  /* selected experts, in provisional order */
    int idx[DF_MAX_A], row[DF_MAX_A];   /* final order; down output of each */
    int uexp[DF_MAX_A], ubase[DF_MAX_A];
    int namb[DF_MAX_T], full[DF_MAX_T], open;
    int asked[2 + DS_CELLS];            /* copies requested of each place of tiles, of cells */
    volatile int dead;                  /* this CTA has given up: a wait ran out */
    unsigned int tag;                   /* of this launch and layer */
    uint16_t w[DF_MAX_A];
    uint8_t umask[DF_MAX_A];
};

/* Parts of a layer that most CTAs or warps never run, or that nobody waits for, as functions:
 * their code and registers stay out of the others' way. */

/* All words lose their tags, before any CTA writes this launch's first ones; target: thread 0's
 * of a round of its own. */
__device__ __noinline__ void stack_clear_words(const StackArgs &a, StackShared &S,
                                               unsigned int target) {
#pragma unroll 1
    for (int i = blockIdx.x * DS_THREADS + threadIdx.x; i < DS_WORDS; i += gridDim.x * DS_THREADS) {
        st_tagged(&a.code_ws[i], 0, 0);
        st_tagged(&a.chain_ws[i], 0, 0);
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        round_arrive(a.sync);
        if (!ds_spin(a.sync, target, S.dead)) {
            set_status(a.status, ST_SCHED_TIMEOUT);
            S.dead = 1;
        }
    }
}
/* The first warp of a CTA that has given up, the others being through: its copies must have landed
 * before the shared memory is another's. */
__device__ __noinline__ void stack_drain(StackShared &S) {
    const volatile int never = 0;
    const int i = threadIdx.x;
    if (i < 2 + DS_CELLS && S.asked[i] > 0)
        ds_wait(i < 2 ? &S.tile_full[i] : &S.cell_full[i - 2], (unsigned)(S.asked[i] - 1) & 1u,
                never);
    __syncwarp();
}

/* The open logits of token t are experts amb[t][0 .. namb[t]); counted through all tokens, pair i
 * is walked by CTA i % G.  This waits for that of pair k of token t, and puts it among the codes. */
__device__ __forceinline__ bool take_chain(const StackArgs &a, StackShared &S, uint32_t *codes,
                                           const uint16_t *amb, int t, int k) {
    const int at = t * (a.E + 1);
    uint64_t c = 0;
    bool there = false;
#pragma unroll 1
    for (uint32_t n = 0; !there && n < (1u << 21); n++) {
        c = ld_tagged(&a.chain_ws[at + k]);
        there = (unsigned)(c >> 32) == S.tag;
        if (!there && n > 64) {
            if (S.dead) break;
            __nanosleep(40);
        }
    }
    codes[at + amb[at + k]] = (uint32_t)c | ((uint32_t)c << 16);
    if (!there) set_status(a.status, ST_SCHED_TIMEOUT);
    return there;
}
/* The helper warp; buf: CH_BYTES of shared memory for the products. */
__device__ __noinline__ void stack_walk_chains(const StackArgs &a, int layer, StackShared &S,
                                               const uint16_t *amb, const unsigned char *xs,
                                               unsigned char *buf) {
    const StackLayer &W = a.layer[layer];
    const LaneRow lr(DS_H);
    const int lane = threadIdx.x & 31, E = a.E, G = gridDim.x;
    int next = blockIdx.x, n = 0;       /* this CTA's next pair; pairs of the tokens so far */
#pragma unroll 1
    for (int t = 0; t < a.T; t++) {
        const int at = t * (E + 1);
#pragma unroll 1
        for (; next < n + S.namb[t]; next += G) {
            const int e = amb[at + next - n];
            const uint16_t *w = e == E ? W.sh_gate : W.rtr_w + (size_t)e * DS_H;
            const unsigned char *xr = xs + t * a.L.xrow;
            const float z = warp_chains<CH_CHAINS>(
                1, DS_H, lane, reinterpret_cast<float *>(buf), [&](int) { return w; },
                [&](int p) { return *reinterpret_cast<const uint4 *>(xr + lr.at(p)); });
            if (lane == 0)
                st_tagged(&a.chain_ws[at + next - n], no_negative_zero(bf16_bits(z)), S.tag);
        }
        n += S.namb[t];
    }
    if (lane == 0 && n > 0 && a.stats && blockIdx.x == 0) atomicAdd(&a.stats[0], (unsigned)n);
}
/* The selection where stack_select leaves something to look at: the whole of rt_select, and the
 * list of what is open.  Returned: open | odd << 1 | entries of the list << 2. */
__device__ __noinline__ int stack_select_slow(const uint32_t *cd, int E, int TK, int *sel,
                                              uint16_t *amb) {
    const int lane = threadIdx.x & 31;
    const Choice c = rt_select(cd, E, TK, lane, sel);
    int n = 0;
    if (c.any)
#pragma unroll 1
        for (int e = lane; e - lane <= E; e += 32) {
            const bool need = rt_needs(cd, e, E, c.kkey, c.odd);
            const unsigned m = __ballot_sync(0xffffffffu, need);
            if (need) amb[n + __popc(m & ((1u << lane) - 1u))] = (uint16_t)e;
            n += __popc(m);
        }
    return (c.open ? 1 : 0) | (c.odd ? 2 : 0) | (n << 2);
}
/* rt_select on the codes as they arrive (v[q]: expert lane + 32 q; no negative zeros; E <= 256),
 * and the list of what is open, the same one in every CTA.  What is left out of it is what hardly
 * ever is: a chosen logit, or one that may be, below 2^-10 or above 32.  A warp alone waits for
 * each of its instructions, so the keys are made two at a time and the competitors that are not
 * known are all that is looked at again.  (Four layers at one token:
 * 112 us -> 107.5.) */
__device__ __forceinline__ int stack_select(const uint64_t (&v)[9], const uint32_t *cd, int E,
                                            int TK, int lane, int *sel, uint16_t *amb) {
    constexpr uint32_t SMALL = 0x3a80u | 0x8000u, FAR = 0x4200u | 0x8000u;  /* keys of 2^-10, 32 */
    auto keys_of = [](uint32_t w) {                      /* code_key of both halves */
        return w ^ (((w >> 15) & 0x00010001u) * 0xffffu | 0x80008000u);
    };
    uint32_t kr[8], unk = 0, kth = 0, mine = 0;
#pragma unroll
    for (int q = 0; q < 8; q++) {
        const int e = lane + 32 * q;
        const uint32_t k = keys_of((uint32_t)v[q]);
        kr[q] = e < E ? (k << 16) | (0xffffu - (uint32_t)e) : 0u;
        if (e < E && (k & 0xffffu) != k >> 16) unk |= 1u << q;
    }
    uint32_t best = max(max(max(kr[0], kr[1]), max(kr[2], kr[3])),
                        max(max(kr[4], kr[5]), max(kr[6], kr[7])));
#pragma unroll 1
    for (int i = 0; i < TK; i++) {
        kth = __reduce_max_sync(0xffffffffu, best);
        if (lane == (i & 31)) mine = kth;
        if (i == 31) sel[lane] = (int)(0xffffu - (mine & 0xffffu));
        uint32_t b[8];
#pragma unroll
        for (int j = 0; j < 8; j++) b[j] = kr[j] < kth ? kr[j] : 0u;
        best = max(max(max(b[0], b[1]), max(b[2], b[3])), max(max(b[4], b[5]), max(b[6], b[7])));
    }
    if (lane < (TK & 31)) sel[(TK & ~31) + lane] = (int)(0xffffu - (mine & 0xffffu));
    const uint32_t kkey = kth >> 16;
    bool open = false, other = false;
    int n = 0;
#pragma unroll 1
    while (__any_sync(0xffffffffu, unk != 0)) {
        const int e = lane + 32 * (__ffs(unk) - 1);
        bool need = false;
        if (unk) {
            const uint32_t k = keys_of(cd[e]);
            need = k >> 16 >= kkey;
            open |= need && ((k << 16) | (0xffffu - (uint32_t)e)) < kth;
            other |= need && ((k & 0xffffu) < SMALL || k >> 16 > FAR);
            unk &= unk - 1;
        }
        const unsigned m = __ballot_sync(0xffffffffu, need);
        if (need) amb[n + __popc(m & ((1u << lane) - 1u))] = (uint16_t)e;
        n += __popc(m);
    }
    /* the largest: the first one's low code, or what the loop looked at */
    other |= kkey < SMALL || (lane == 0 && (TK < 32 ? mine >> 16 > FAR : true));
    if (__any_sync(0xffffffffu, other)) return stack_select_slow(cd, E, TK, sel, amb);
    if (!code_known(cd[E])) {
        if (lane == 0) amb[n] = (uint16_t)E;
        n++;
    }
    return (__any_sync(0xffffffffu, open) ? 1 : 0) | (n << 2);
}
/* A warp to a token, its chains known: the selection again, or the engine's softmax. */
__device__ __forceinline__ void stack_select_again(const StackArgs &a, StackShared &S,
                                                   uint32_t *cd, int t) {
    const int lane = threadIdx.x & 31, E = a.E, TK = a.TK;
    if (S.full[t]) {
        float *p = reinterpret_cast<float *>(cd);
#pragma unroll 1
        for (int e = lane; e < E; e += 32) p[e] = bf16lo(cd[e]);
        __syncwarp();
        router_softmax_topk(p, E, TK, lane, S.idx + t * TK, S.w + t * TK);
        __syncwarp();
#pragma unroll 1
        for (int i = lane; i < TK; i += 32) S.sel[t * TK + i] = S.idx[t * TK + i];
    } else {
        rt_select(cd, E, TK, lane, S.sel + t * TK);
    }
}
/* The helper warp: final order, weights, shared gate, and where the down output of each slot
 * will be. */
__device__ __noinline__ void stack_weights(const StackArgs &a, StackShared &S, uint32_t *codes,
                                           const uint16_t *amb, int U) {
    const int lane = threadIdx.x & 31, T = a.T, E = a.E, TK = a.TK;
    if (!S.open)
#pragma unroll 1
        for (int t = 0; t < T; t++)
#pragma unroll 1
            for (int k = lane; k < S.namb[t]; k += 32)
                if (!take_chain(a, S, codes, amb, t, k)) S.dead = 1;
    __syncwarp();
#pragma unroll 1
    for (int t = 0; t < T; t++) {
        if (!S.full[t])
            rt_weights(codes + t * (E + 1), S.sel + t * TK, TK, lane, S.idx + t * TK, S.w + t * TK);
        if (lane == 0) S.gate[t] = bf16_round(sigmoid_f32(bf16lo(codes[t * (E + 1) + E])));
    }
    __syncwarp();
#pragma unroll 1
    for (int i = lane; i < T * TK; i += 32) {
        const int t = i / TK, e = S.idx[i];
        int lo = 0, hi = U - 1;
#pragma unroll 1
        while (lo < hi) {
            const int mid = (lo + hi) >> 1;
            if (S.uexp[mid] < e) lo = mid + 1; else hi = mid;
        }
        S.row[i] = S.ubase[lo] + __popc(S.umask[lo] & ((1u << t) - 1u));
        if (blockIdx.x == 0) {
            if (a.idx_out) a.idx_out[i] = e;
            if (a.w_out) a.w_out[i] = S.w[i];
        }
    }
    __syncwarp();
}

/* A CTA that has given up leaves the launch before a layer's first barrier: the others' rounds, and
 * the launches to come, count on its arrivals. */
__device__ __noinline__ bool stack_leave(const StackArgs &a, int layer) {
    if (threadIdx.x == 0) {
        set_status(a.status, ST_SCHED_TIMEOUT);
        red_release_add(a.sync, (2u * (a.n_layers - layer) - 1u) *
                                    (blockIdx.x == 0 ? DF_ROUND - gridDim.x + 1u : 1u));
    }
    return false;
}

/* One layer; tile0, item0: gate/up tiles and down items before it; sync_at: thread 0's target
 * of the barrier.  False: given up, in all warps.
 *
 * Where a wait runs out, S.dead is set and the status recorded.  The CTA's own barriers need all of
 * its warps, so it goes on without waiting for anything, on whatever is there, to where the next
 * selection would be, and leaves.  (There S.dead is read anyway; asking where a layer begins cost
 * a quarter of a microsecond a layer.)  It is read between two barriers, between which nobody can
 * be who may set it, so all warps agree. */
__device__ __forceinline__ bool stack_layer(const StackArgs &a, StackShared &S, int layer,
                                            unsigned int &sync_at, int &tile0, int &item0) {
    extern __shared__ __align__(128) unsigned char ds_smem[];

    const bool first = layer == 0;
    /* What is computed from these is computed again in every layer, and below in both phases,
     * instead of being kept in registers over the loops: 96 of them are all that eighteen warps
     * can have (four layers at 1 / 3 / 8 tokens 114 / 178 / 341 us without any of it). */
    int wl = layer;
    asm volatile("" : "+r"(wl));
    const StackLayer &W = a.layer[wl];
    int tid = threadIdx.x;
    const int T = a.T, G = gridDim.x, cta = blockIdx.x;
    asm volatile("" : "+r"(tid));
    const int I = a.I, E = a.E, TK = a.TK, A = T * TK;
    const int lane = tid & 31, warp = tid >> 5;
    const StackLayout &L = a.L;
    const LaneRow lr(DS_H);
    constexpr int PIECES = DS_H / 8;
    unsigned char *xs = ds_smem + L.off_x, *rr = ds_smem + L.off_rr;
    uint4 *gains = reinterpret_cast<uint4 *>(ds_smem + L.off_gain);
    uint32_t *codes = reinterpret_cast<uint32_t *>(ds_smem + L.off_code);   /* [T][E + 1] */
    uint16_t *amb = reinterpret_cast<uint16_t *>(ds_smem + L.off_amb);      /* [T][E + 1]: a
                                                        * token's open logits, S.namb of them */
    uint32_t *s_tmask = reinterpret_cast<uint32_t *>(ds_smem + L.off_tmask);   /* tokens of each
                                                        * expert, a byte each (64 words in use) */
    float *red = reinterpret_cast<float *>(ds_smem + L.off_red);
    const uint16_t *res = first ? a.res : a.res_out;

    auto mark = [&](int k) {
        if (a.timeline && tid == 0) {
            unsigned long long t;
            asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
            a.timeline[(size_t)cta * DF_MARKS + k] = t;
        }
    };
    auto give_up = [&] {
        set_status(a.status, ST_SCHED_TIMEOUT);
        S.dead = 1;
    };
    /* the k-th use of a place in the ring: copies landed, or warps done with it (both within
     * this CTA, so that nothing is left in flight when another CTA's part never came) */
    /* (by parity: whoever waits for the k-th has seen the one before it, or knows it to be over) */
    auto landed = [&](uint64_t *bar, int k) {
        const bool ok = ds_wait(bar, (unsigned)k & 1u, S.dead);
        if (!ok) give_up();
        return ok;
    };
    mark(0);
    /* ---- this CTA's shares ---- */
    const int n_rr = cta <= E ? (E - cta) / G + 1 : 0;
    const unsigned b = cta, g = G;
    const int sh_lo = (int)((unsigned)I * b / g), sh_n = (int)((unsigned)I * (b + 1) / g) - sh_lo;
    const int h_lo = (int)((unsigned)DS_H * b / g);
    const int ncols = (int)((unsigned)DS_H * (b + 1) / g) - h_lo;

    /* ---- what does not depend on the layer before: router rows, gains, first weights ---- */
    if (first) {
        if (tid == 0) {
            S.dead = 0;
            S.tag = sync_at = round_target(__ldcg(a.sync));
#pragma unroll 1
            for (int i = 0; i < DS_CELLS; i++) {
                S.asked[i] = S.asked[2 + i] = 0;
                mbar_init(&S.cell_full[i], 1);
                mbar_init(&S.cell_free[i], 1u << a.slices_log2);
                if (i < 2) {
                    mbar_init(&S.tile_full[i], 1);
                    mbar_init(&S.tile_free[i], DS_CW);
                }
            }
            mbar_fence_init();
        }
        __syncthreads();
        if (stack_clears(S.tag)) {
            stack_clear_words(a, S, sync_at);
            sync_at += DF_ROUND;
        }
        if (cta == a.absent) return stack_leave(a, layer);
    }
    /* a tile of n pairs, the first k of one expert and the others of the next: lanes 0-3
     * request a piece each */
    auto request_tile = [&](int tile, const uint16_t *gate, const uint16_t *up, int k,
                            const uint16_t *gate2, const uint16_t *up2, int n) {
        const bool free = tile < 2 || landed(&S.tile_free[tile & 1], (tile >> 1) + 1);
        if (!__all_sync(0xffffffffu, free)) return;
        uint64_t *bar = &S.tile_full[tile & 1];
        unsigned char *dst = ds_smem + (tile & 1) * DS_TILE;
        if (lane == 0) {
            S.asked[tile & 1] = (tile >> 1) + 1;
            mbar_expect_tx(bar, (uint32_t)(2 * n * DS_H * 2));
        }
        __syncwarp();
        const int rows = lane & 2 ? n - k : k;
        if (lane < 4 && rows > 0)
            bulk_g2s(dst + ((lane & 1) * DS_PAIRS + (lane & 2 ? k : 0)) * DS_H * 2,
                     lane & 2 ? (lane & 1 ? up2 : gate2) : lane & 1 ? up : gate,
                     (uint32_t)(rows * DS_H * 2), bar);
    };
    const int n_sh = (sh_n + DS_PAIRS - 1) / DS_PAIRS;
    if (warp == DS_CW)
#pragma unroll 1
        for (int j = 0; j < n_sh; j++) {        /* (two at most) */
            const int n = min(DS_PAIRS, sh_n - j * DS_PAIRS);
            const size_t at = (size_t)(sh_lo + j * DS_PAIRS) * DS_H;
            request_tile(tile0 + j, W.sh_g + at, W.sh_u + at, n, nullptr, nullptr, n);
        }
    /* (the requesting warp has asked for a later layer's in the layer before) */
    auto fetch_rows = [&](const StackLayer &w, int at, int step) {
#pragma unroll 1
        for (int c = at; c < (n_rr + 1) * PIECES; c += step) {
            const int r = c / PIECES, e = cta + r * G, p = c % PIECES;
            if (r < n_rr)
                cp_async16_to(smem_u32(rr + r * L.xrow + lr.at(p)),
                              (e == E ? w.sh_gate : w.rtr_w + (size_t)e * DS_H) + p * 8);
            else if (a.res && w.ln_w)
                cp_async16_to(smem_u32(gains + p), w.ln_w + p * 8);
            else
                gains[p] = make_uint4(0, 0, 0, 0);
        }
    };
    if (first && warp < DS_CW) fetch_rows(W, tid, DS_CW * 32);
    if (tid < 256) s_tmask[tid] = 0;
    if (tid < DF_MAX_T) {
        S.xlo[tid] = 0x7f800000u;
        S.xhi[tid] = 0;
    }
    if (tid == 0) {
        S.open = 0;
        /* the rows that the other CTAs' combines left: the end of the layer before */
        if (!first) {
            if (!S.dead && !ds_spin(a.sync, sync_at, S.dead)) give_up();
            sync_at += DF_ROUND;
        }
        S.tag = stack_tag(sync_at);
    }
    asm volatile("cp.async.wait_all;" ::: "memory");
    __syncthreads();
    {
        const uint4 *src = reinterpret_cast<const uint4 *>(res ? res : a.x);
#pragma unroll 1
        for (int c = tid; c < T * PIECES; c += DS_THREADS)
            *reinterpret_cast<uint4 *>(xs + c / PIECES * L.xrow + lr.at(c % PIECES)) =
                __ldcg(src + c);
    }
    __syncthreads();
    /* ---- norm (bit for bit the engine's) and the range of the tokens' values: four warps to a
     * token, or two ---- */
    const int parts = T <= 4 ? 4 : 2, t_norm = T <= 4 ? warp & 3 : warp & 7;
    if (t_norm < T && warp < DS_CW) {
        const int t = t_norm, part = T <= 4 ? warp >> 2 : warp >> 3;
        unsigned char *row = xs + t * L.xrow;
        float rs = 1.0f;
        if (res) {
            SumShare &share = reinterpret_cast<SumShare *>(ds_smem + L.off_share)[t];
            auto meet = [&] {
                asm volatile("bar.sync %0, %1;" ::"r"(3 + t), "r"(32 * parts) : "memory");
            };
            const float sum = parts == 4 ? exact_sumsq_wide<4>(row, lr, lane, part, share, meet)
                                         : exact_sumsq_wide<2>(row, lr, lane, part, share, meet);
            /* norm_scale; a quotient by a power of two is the product */
            rs = __fdiv_rn(1.0f, __fsqrt_rn(__fadd_rn(__fmul_rn(sum, 1.0f / DS_H), 1e-6f)));
        }
        PackedRange range;
        float sq = 0.0f;
#pragma unroll 1
        for (int c = part * 32 + lane; c < PIECES; c += 32 * parts) {
            uint4 *p = reinterpret_cast<uint4 *>(row + lr.at(c));
            uint4 v = *p;
            if (res) *p = v = norm8(v, gains[c], rs);
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
            S.sq[part][t] = sq;
            atomicMin(&S.xlo[t], lo);
            atomicMax(&S.xhi[t], hi);
        }
    }
    __syncthreads();

    /* ---- router logits of this CTA's rows: up to two tokens four warps to one, up to four two
     * (certified_logit, the rows cut across the warps like the norm's).  Its error terms hold
     * with one factor larger: of u |lane sum| there are one for the lane's last addition, five for
     * the scan and, where four warps share a row, up to three more, two in `before` and one in
     * `tot`: nine, and ten are taken. ---- */
    const int lg = L.rrows > 2 || T > 4 ? 0 : T > 2 ? 1 : 2, per = 1 << lg;
    if (warp < DS_CW)
#pragma unroll 1
        for (int p = warp >> lg; p < n_rr * T; p += DS_CW >> lg) {
            const int r = p >= T ? p / T : 0, t = p - r * T, e = cta + r * G,
                      part = warp & (per - 1);
            const bool gate = e == E;
            const bool exact = products_exact(gate ? W.wmin_gate : W.wmin,
                                              gate ? W.wmax_gate : W.wmax, S.xlo[t], S.xhi[t]);
            const int chunk = part * 32 + lane, nu = 8 >> lg;
            const int off = (chunk >> lg) * lr.pitch + (chunk & (per - 1)) * nu * 16;
            const unsigned char *wp = rr + r * L.xrow + off, *xp = xs + t * L.xrow + off;
            float run = 0.0f, err = 0.0f;
#pragma unroll 2
            for (int i = 0; i < nu; i++) {
                float wf[8], xf[8];
                unpack8(*reinterpret_cast<const uint4 *>(wp + i * 16), wf);
                unpack8(*reinterpret_cast<const uint4 *>(xp + i * 16), xf);
                float s0 = __fmul_rn(wf[0], xf[0]), s1 = __fmul_rn(wf[4], xf[4]);
#pragma unroll
                for (int j = 1; j < 4; j++) {
                    s0 = __fmaf_rn(wf[j], xf[j], s0);
                    s1 = __fmaf_rn(wf[4 + j], xf[4 + j], s1);
                }
                err += fabsf(run);
                run += s0 + s1;
            }
            float sum = run;
#pragma unroll
            for (int d = 1; d < 32; d <<= 1) {
                const float v = __shfl_up_sync(0xffffffffu, sum, d);
                if (lane >= d) sum += v;
            }
            float tot = __shfl_sync(0xffffffffu, sum, 31);
            auto meet = [&] {
                asm volatile("bar.sync %0, %1;" ::"r"(3 + (warp >> lg)), "r"(32 << lg) : "memory");
            };
            if (per > 1) {
                if (lane == 0) S.part[0][warp] = tot;
                meet();
                float before = 0.0f;
                for (int i = 0; i < part; i++) before += S.part[0][warp - part + i];
                sum += before;
                tot += before;              /* (the last part's: the whole) */
            }
            err = warp_sum(8.0f * nu * fabsf(sum - run) + 9.0f * err + 10.0f * fabsf(run));
            if (per > 1) {
                if (lane == 0) S.part[1][warp] = err;
                meet();
                err = 0.0f;
                for (int i = 0; i < per; i++) err += S.part[1][warp - part + i];
            }
            if (part == per - 1 && lane == 0) {
                const float sq = T <= 4 ? (S.sq[0][t] + S.sq[1][t]) + (S.sq[2][t] + S.sq[3][t])
                                        : S.sq[0][t] + S.sq[1][t];
                const float cs = (gate ? W.wnorm_gate : __ldg(&W.wnorm[e])) * norm_above(sq, DS_H);
                err = (err + 12.0f * cs) * (1.05f * 5.9604645e-8f);
                const float lo = __fadd_rd(tot, -err), hi = __fadd_ru(tot, err);
                const uint32_t v = exact && lo <= hi
                                       ? (uint32_t)bf16_bits(lo) | ((uint32_t)bf16_bits(hi) << 16)
                                       : CODE_UNKNOWN;
                st_tagged(&a.code_ws[(size_t)t * (E + 1) + e], no_negative_zero(v), S.tag);
            }
        }
    mark(1);                                /* own logits published */

    const int fr = lane >> 2, fq = lane & 3;        /* row and piece of a fragment */
    const bool odd = fr & 1;
    int U = 0, gu_lo = 0, gu_n = 0, n_tiles = n_sh;
    /* the shared expert's gate/up rows, for which nobody waits; then the routed ones */
#pragma unroll 1
    for (int phase = 0; phase < 2; phase++) {
        int lane = tid & 31, warp = tid >> 5;
        asm volatile("" : "+r"(lane), "+r"(warp));
        const int fr = lane >> 2, fq = lane & 3;
        const bool odd = fr & 1;
        if (phase == 1) {
            mark(2);                        /* shared gate/up done */
            /* ---- routing: a warp to a token; the others wait for all of them ---- */
            auto mark_chosen = [&] {        /* the token's bit at its experts */
                __syncwarp();
#pragma unroll 1
                for (int i = lane; i < TK; i += 32) {
                    const int e = S.sel[warp * TK + i];
                    atomicOr(&s_tmask[e >> 2], (1u << warp) << ((e & 3) * 8));
                }
            };
            uint32_t *cd = codes + warp * (E + 1);
            if (warp < T) {
                /* its logits, as soon as this launch's are there, all under way at once */
                constexpr int R = 9;
                const uint64_t *src = a.code_ws + (size_t)warp * (E + 1) + lane;
                const unsigned tag = S.tag;
                uint64_t v[R];
                bool all = false;
#pragma unroll 1
                for (uint32_t i = 0; !all && i < (1u << 21); i++) {
                    all = true;
#pragma unroll
                    for (int q = 0; q < R; q++)
                        v[q] = lane + q * 32 < E + 1 ? ld_tagged(src + q * 32)
                                                     : (uint64_t)tag << 32;
#pragma unroll
                    for (int q = 0; q < R; q++) all &= (unsigned)(v[q] >> 32) == tag;
                    all = __all_sync(0xffffffffu, all);
                    if (!all && i > 64) {
                        if (__any_sync(0xffffffffu, S.dead)) break;
                        __nanosleep(40);
                    }
                }
#pragma unroll
                for (int q = 0; q < R; q++)
                    if (lane + q * 32 < E + 1) cd[lane + q * 32] = (uint32_t)v[q];
                __syncwarp();
                if (all) {
                    const int r = stack_select(v, cd, E, TK, lane, S.sel + warp * TK,
                                               amb + warp * (E + 1));
                    if (lane == 0) {
                        S.namb[warp] = r >> 2;
                        S.full[warp] = (r >> 1) & 1;
                        if (r & 3) S.open = 1;
                    }
                    mark_chosen();
                } else if (lane == 0) {
                    give_up();
                }
            }
            __syncthreads();
            if (S.dead) return stack_leave(a, layer);
            if (warp == DS_CW + 1)
                stack_walk_chains(a, layer, S, amb, xs, ds_smem + L.off_share);
            if (S.open) {                   /* the set itself waits for the chains */
                if (tid < 256) s_tmask[tid] = 0;
                __syncthreads();            /* (all have seen that S.dead is not set) */
#pragma unroll 1
                for (int t = warp; t < T; t += DS_THREADS / 32)
#pragma unroll 1
                    for (int k = lane; k < S.namb[t]; k += 32)
                        if (!take_chain(a, S, codes, amb, t, k)) S.dead = 1;
                __syncthreads();
                if (S.dead) return stack_leave(a, layer);
                if (warp < T) {
                    stack_select_again(a, S, cd, warp);
                    mark_chosen();
                }
                __syncthreads();
            }
            /* ---- the distinct experts, ascending, and who uses them: every warp writes the
             * whole list, and waits for nobody's ---- */
            {
                /* a lane has eight experts (E <= 256) */
                const uint2 m = reinterpret_cast<const uint2 *>(s_tmask)[lane];
                auto used = [](uint32_t v) {        /* 0x80 in each byte that is not zero */
                    return (((v & 0x7f7f7f7fu) + 0x7f7f7f7fu) | v) & 0x80808080u;
                };
                const int mine = __popc(used(m.x)) + __popc(used(m.y)) +
                                 ((__popc(m.x) + __popc(m.y)) << 16);
                int incl = mine;                    /* experts | assignments << 16 */
#pragma unroll
                for (int d = 1; d < 32; d <<= 1) {
                    const int v = __shfl_up_sync(0xffffffffu, incl, d);
                    if (lane >= d) incl += v;
                }
                int p = incl - mine;
                U = __shfl_sync(0xffffffffu, incl, 31) & 0xffff;
                /* bit i: expert 8 lane + i */
                uint32_t r = (((used(m.x) >> 7) * 0x01020408u) >> 24 & 15u) |
                             (((used(m.y) >> 7) * 0x01020408u) >> 20 & 0xf0u);
#pragma unroll 1
                for (; r; r &= r - 1) {
                    const int k = __ffs(r) - 1;
                    const uint32_t who = ((k & 4 ? m.y : m.x) >> ((k & 3) * 8)) & 0xffu;
                    const int u = p & 0xffff;
                    S.uexp[u] = lane * 8 + k;
                    S.umask[u] = (uint8_t)who;
                    S.ubase[u] = p >> 16;
                    p += 1 + (__popc(who) << 16);
                }
                __syncwarp();
            }
            mark(3);                        /* selection known */
            gu_lo = (int)((unsigned)(U * I) * b / g);
            gu_n = (int)((unsigned)(U * I) * (b + 1) / g) - gu_lo;
            n_tiles = (gu_n + DS_PAIRS - 1) / DS_PAIRS;
            tile0 += n_sh;

            if (warp == DS_CW) {
                /* ---- the requesting warp: routed gate/up rows, then the down rows of this
                 * CTA's columns (the shared expert's last), each as its place comes free ---- */
#pragma unroll 1
                for (int j = 0; j < n_tiles; j++) {
                    const int it = gu_lo + j * DS_PAIRS, u = it / I, i = it - u * I;
                    const int n = min(DS_PAIRS, gu_n - j * DS_PAIRS), k = min(n, I - i);
                    const size_t half = (size_t)I * DS_H;
                    const uint16_t *w = W.exp_gu + S.uexp[u] * 2 * half + (size_t)i * DS_H,
                                   *w2 = W.exp_gu + S.uexp[k < n ? u + 1 : u] * 2 * half;
                    request_tile(tile0 + j, w, w + half, k, w2, w2 + half, n);
                }
                tile0 += n_tiles;
                /* (nobody looks at this layer's any more) */
                if (layer + 1 < a.n_layers) fetch_rows(a.layer[layer + 1], lane, 32);
                /* a lane to a cell: it asks again as soon as its cell is free (one after another
                 * they kept each other waiting: 25 us for the down rows of eight tokens) */
                const uint32_t bytes = (uint32_t)(ncols * I * 2);
                bool busy = lane < DS_CELLS && lane <= U;
                int d = lane;
                /* ... when the tile that lies there has been read, then its item before this */
                uint64_t *free_bar = &S.tile_free[(tile0 + (lane >> 2)) & 1];
                int use = (tile0 - 2 + (lane >> 2)) >> 1;
                /* (a limit behind the barrier's: what frees a cell may wait for that) */
#pragma unroll 1
                for (uint32_t n = 0; __any_sync(0xffffffffu, busy); n++) {
                    if (n > 256) {
                        if (n > 8 * APUS_WAIT_LIMIT) give_up();
                        if (__any_sync(0xffffffffu, S.dead)) break;
                        __nanosleep(20);
                    }
                    if (busy && mbar_test(free_bar, (unsigned)use & 1u)) {
                        if (d <= U) {
                            const int c = (item0 + d) & (DS_CELLS - 1);
                            uint64_t *bar = &S.cell_full[c];
                            S.asked[2 + c] = ((item0 + d) >> 3) + 1;
                            mbar_expect_tx(bar, bytes);
                            bulk_g2s(ds_smem + (((tile0 & 1) * 4 + d) & (DS_CELLS - 1)) * DS_CELL,
                                     (d == U ? W.sh_d : W.exp_d + (size_t)S.uexp[d] * DS_H * I) +
                                         (size_t)h_lo * I,
                                     bytes, bar);
                            free_bar = &S.cell_free[c];
                            use = (item0 + d) >> 3;
                            d += DS_CELLS;
                        } else {
                            busy = false;   /* and nothing is left in it: the next layer's first
                                             * tiles may lie anywhere */
                        }
                    }
                }
                __syncwarp();
                item0 += U + 1;
                return true;
            }
            if (warp > DS_CW) {
                stack_weights(a, S, codes, amb, U);
                asm volatile("bar.arrive 2, %0;" ::"n"(DS_CW * 32 + 32) : "memory");
                tile0 += n_tiles;
                item0 += U + 1;
                return true;
            }
        }
        /* ---- gate/up tiles: the warps' partial sums meet in shared memory, four warps in
         * turn finish a tile while the others go on ---- */
        /* a warp's share of the tokens: column fr, 128 k */
        uint4 xf[4];
#pragma unroll
        for (int w = 0; w < 4; w++)
            xf[w] = *reinterpret_cast<const uint4 *>(xs + min(fr, T - 1) * L.xrow +
                                                     lr.at((warp & 15) * 16 + w * 4 + fq));
        if (warp < DS_CW)
#pragma unroll 1
            for (int j = 0; j < n_tiles; j++) {
                const int tile = tile0 + j;
                float *buf = red + (j & 1) * (DS_CW * 2 * DS_PAIRS * 8);
                const unsigned char *p = ds_smem + (tile & 1) * DS_TILE + fr * (DS_H * 2) +
                                         warp * 256 + fq * 16;
                landed(&S.tile_full[tile & 1], tile >> 1);
                uint4 gr[4], ur[4];
                slice_pieces(p, odd, gr);
                slice_pieces(p + DS_PAIRS * DS_H * 2, odd, ur);
                float c0[4] = {0.f, 0.f, 0.f, 0.f}, c1[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
                for (int w = 0; w < 4; w++) {
                    const uint32_t r0[4] = {gr[w].x, ur[w].x, gr[w].y, ur[w].y},
                                   r1[4] = {gr[w].z, ur[w].z, gr[w].w, ur[w].w};
                    mma_16x8(c0, r0, xf[w].x, xf[w].y);
                    mma_16x8(c1, r1, xf[w].z, xf[w].w);
                }
                __syncwarp();
                if (lane == 0) mbar_arrive(&S.tile_free[tile & 1]);
                /* (gate and up of a pair side by side) */
                float *dst = buf + (warp * 2 * DS_PAIRS + 2 * fr) * 8 + fq * 2;
                *reinterpret_cast<float2 *>(dst) = make_float2(c0[0] + c1[0], c0[1] + c1[1]);
                *reinterpret_cast<float2 *>(dst + 8) = make_float2(c0[2] + c1[2], c0[3] + c1[3]);
                df_bar_compute();
                if ((warp >> 2) == (j & 3)) {
                    /* thread = row (2p gate, 2p + 1 up) x column */
                    const int i = (warp & 3) * 32 + lane, col = i & 7,
                              pi = j * DS_PAIRS + (i >> 4);
                    float v = 0.0f;
#pragma unroll
                    for (int w = 0; w < DS_CW; w++) v += buf[w * (2 * DS_PAIRS * 8) + i];
                    const float up = bf16_round(__shfl_xor_sync(0xffffffffu, v, 8));
                    const float gate = bf16_round(v);
                    if (!(i & 8) && pi < (phase ? gu_n : sh_n)) {
                        int row = A + col, at = sh_lo + pi;
                        bool mine = col < T;
                        if (phase) {
                            const int it = gu_lo + pi, u = it / I;
                            const unsigned m = S.umask[u];
                            mine = (m >> col) & 1u;
                            row = S.ubase[u] + __popc(m & ((1u << col) - 1u));
                            at = it - u * I;
                        }
                        /* silu_act_bits, silu_mul_bits */
                        float y = __fmul_rn(gate, sigmoid_f32(gate));
                        if (phase) y = bf16_round(y);
                        if (mine) a.act_ws[(size_t)row * I + at] = bf16_bits(__fmul_rn(y, up));
                    }
                }
            }
    }
    if (warp >= DS_CW) return true;         /* (not reached: for the compiler) */
    tile0 += n_tiles;
    mark(4);                                /* routed gate/up done */
    df_bar_compute();
    if (tid == 0) {
        round_arrive(a.sync);
        if (!S.dead && !ds_spin(a.sync, sync_at, S.dead)) give_up();
        sync_at += DF_ROUND;                /* the layer's end */
    }
    df_bar_compute();
    const bool dead = S.dead != 0;
    mark(5);                                /* barrier passed */
    /* ---- down rows of this CTA's columns: a warp to 128 k of an expert.  Its activations are
     * nobody else's here: they come straight from L2, beside the wait for the rows (all of them
     * through shared memory first: 1.7 kcycles at one token, 6.6 at eight; those of the next unit
     * while this one is at work cost sixteen registers, and with what they spilled 3 to 5 % of
     * four layers). ---- */
    auto unit_rows = [&](int v, int &cnt, int &row0) {
        const int d = v >> a.slices_log2;
        cnt = d == U ? T : __popc(S.umask[d]);
        row0 = d == U ? A : S.ubase[d];
    };
    auto unit_acts = [&](int v, uint4 (&x)[4]) {
        int cnt, row0;
        unit_rows(v, cnt, row0);
        const uint4 *q = reinterpret_cast<const uint4 *>(
            a.act_ws + (size_t)(row0 + min(fr, cnt - 1)) * I +   /* (extra columns are not used) */
            (v & ((1 << a.slices_log2) - 1)) * 128 + fq * 8);
#pragma unroll
        for (int w = 0; w < 4; w++) x[w] = __ldcg(q + w * 4);
    };
    const int n_units = (U + 1) << a.slices_log2;
    /* the combine's output of this thread, and what it is added to */
    const int out_t = tid / ncols, out_at = out_t * DS_H + h_lo + (tid - out_t * ncols);
    uint16_t out_res = 0;
    if (a.res_out && out_t < T) out_res = __ldcg(res + out_at);
#pragma unroll 1
    for (int v = warp; v < n_units; v += DS_CW) {
        uint4 xv[4];
        unit_acts(v, xv);
        const int d = v >> a.slices_log2, slice = v & ((1 << a.slices_log2) - 1);
        int cnt, row0;
        unit_rows(v, cnt, row0);
        const int item = item0 + d, cell = ((tile0 & 1) * 4 + d) & (DS_CELLS - 1);
        const unsigned char *p = ds_smem + cell * DS_CELL + fr * (I * 2) + slice * 256 + fq * 16;
        landed(&S.cell_full[item & (DS_CELLS - 1)], item >> 3);
        uint4 lo[4], hi[4];
        slice_pieces(p, odd, lo);
        slice_pieces(p + 8 * I * 2, odd, hi);
        __syncwarp();
        if (lane == 0) mbar_arrive(&S.cell_free[item & (DS_CELLS - 1)]);
        /* mma.sync cuts off what its accumulator cannot hold: two steps on one that starts at
         * zero, sums of those rounded to nearest (decode_fused.cuh has the figures; the gate/up
         * tiles end in a sum of sixteen warps and need no more than that). */
        float c0[4] = {0.f, 0.f, 0.f, 0.f}, c1[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
        for (int w = 0; w < 4; w++) {
            const uint4 x = xv[w];
            const uint32_t r0[4] = {lo[w].x, hi[w].x, lo[w].y, hi[w].y},
                           r1[4] = {lo[w].z, hi[w].z, lo[w].w, hi[w].w};
            float t[4] = {0.f, 0.f, 0.f, 0.f};
            mma_16x8(t, r0, x.x, x.y);
            mma_16x8(t, r1, x.z, x.w);
#pragma unroll
            for (int k = 0; k < 4; k++) ((w & 1) ? c1 : c0)[k] += t[k];
        }
        const int col = fq * 2;
        float *dst = red + ((size_t)slice * (A + T) + row0 + col) * DF_MAX_COLS + fr;
        if (col < cnt) {
            dst[0] = c0[0] + c1[0];
            dst[8] = c0[2] + c1[2];
        }
        if (col + 1 < cnt) {
            dst[DF_MAX_COLS] = c0[1] + c1[1];
            dst[DF_MAX_COLS + 8] = c0[3] + c1[3];
        }
    }
    item0 += U + 1;
    df_bar_compute();
    mark(6);                                /* down rows done */

    /* ---- combine (c/layer.h:350,356-361), this CTA's columns: the slices' sums, then a thread
     * to an output ---- */
#pragma unroll 1
    for (int i = tid; i < (A + T) * DF_MAX_COLS; i += DS_CW * 32) {
        const int n = (A + T) * DF_MAX_COLS;
        float y = red[i];
        y += red[n + i];
        if (a.slices_log2 > 1) y += red[2 * n + i] + red[3 * n + i];
        red[i] = bf16_round(y);
    }
    /* the helper warp has been through as well */
    asm volatile("bar.sync 2, %0;" ::"n"(DS_CW * 32 + 32) : "memory");
    if (!dead && out_t < T) {
        const int t = out_t, h = out_at - t * DS_H - h_lo;
        float acc = 0.0f;
#pragma unroll 2
        for (int s = 0; s < TK; s++)
            acc = __fadd_rn(acc, __fmul_rn(bf16_f32(S.w[t * TK + s]),
                                           red[S.row[t * TK + s] * DF_MAX_COLS + h]));
        const float routed = bf16_round(acc);
        const float shared = bf16_round(__fmul_rn(red[(A + t) * DF_MAX_COLS + h], S.gate[t]));
        const uint16_t v = bf16_bits(__fadd_rn(routed, shared));
        const size_t at = out_at;
        if (a.out) a.out[at] = v;
        if (a.res_out)                          /* c/layer.h:230-234,388 */
            a.res_out[at] = bf16_bits(__fadd_rn(bf16_f32(out_res), bf16_f32(v)));
        if (a.tr_out) a.tr_out[at] = v;
        if (a.tr_routed) a.tr_routed[at] = bf16_bits(routed);
        if (a.tr_shared) a.tr_shared[at] = bf16_bits(shared);
    }
    mark(7);                                /* combine done */
    if (layer + 1 < a.n_layers) {
        df_bar_compute();
        if (tid == 0) round_arrive(a.sync);
    }
    return true;
}

__global__ void __launch_bounds__(DS_THREADS, 1)
decode_stack_kernel(const __grid_constant__ StackArgs a) {
    __shared__ StackShared S;
    unsigned int sync_at = 0;
    int tile0 = 0, item0 = 0;
#pragma unroll 1
    for (int layer = 0; layer < a.n_layers; layer++)
        if (!stack_layer(a, S, layer, sync_at, tile0, item0)) break;
    __syncthreads();                        /* nobody requests or waits any more */
    if (S.dead && threadIdx.x < 32) stack_drain(S);
}

}  // namespace apus
