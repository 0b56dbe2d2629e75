/*
 * exact_sum.cuh — results of the engine's sequential fp32 sums without walking
 * the whole chain.
 *
 * The engine's sums are chains of 2048 dependent fp32 adds (4.6 cycles each on
 * this GPU: 4.8 us), and their last bits matter.  Two observations:
 *
 * 1. Sum of squares (RMSNorm, c/attn.h:175-186).  All terms are >= 0, so the sum
 *    only grows, and while it stays inside one binade [2^k, 2^(k+1)) it is an
 *    integer number of units u = 2^(k-23) to which every step adds an integer:
 *    the term rounded to units, ties decided by whether the sum is even.  A step
 *    is therefore a function of the sum's parity, such functions compose, and
 *    composition is associative.  Each of 32 lanes finds the function of its 64
 *    terms by adding them to the binade's smallest even and smallest odd sum, and
 *    a segmented scan joins the lanes.  Only where the sum crosses into the next
 *    binade (about six lanes, lane 0 among them) are the additions done one after
 *    another.  Every run is verified (it must start and end inside the binade it
 *    was composed for) and redone sequentially otherwise, so the result is the
 *    chain's, bit for bit, whatever the data.
 *
 * 2. Router logits (c/moe.h:289-291) are rounded to BF16 before anything looks at
 *    them.  With exact products, chain and true sum differ by at most
 *    u * sum |partial sum| (each add errs by half an ulp of its result), so a
 *    tree sum with that bound, evaluated from the data, usually pins the BF16
 *    code (97-99 % of the logits that compete for the top-k at the real
 *    dimensions); only the others need their chain.
 */
#pragma once
#include "common.cuh"
#include "decode_gemv.cuh"

namespace apus {

/* A row of H values as BF16 in shared memory, cut into nl lane chunks of nu 16-byte
 * pieces, each followed by 16 bytes, so that 32 lanes reading 16 bytes of their
 * chunks meet no bank conflict.  nl = the largest power of two <= 32 with 8 nl | H. */
struct LaneRow {
    int nl, nu, pitch;                /* lanes, 16-byte pieces per lane, bytes per chunk */
    uint32_t inv;                     /* piece / nu == piece * inv >> 20 below 4096 pieces */
    LaneRow() = default;
    __host__ __device__ explicit LaneRow(int H) {
        nl = 32;
        while (nl > 1 && H % (8 * nl)) nl >>= 1;
        nu = H / (8 * nl);
        pitch = nu * 16 + 16;
        inv = (1u << 20) / (uint32_t)(nu > 0 ? nu : 1) + 1;
    }
    __host__ __device__ int bytes() const { return nl * pitch; }
    /* byte offset of piece c (values 8 c .. 8 c + 7) */
    __device__ __forceinline__ int at(int c) const {
        const int l = (int)(((uint32_t)c * inv) >> 20);
        return l * 16 + c * 16;       /* l * pitch + (c - l * nu) * 16 */
    }
};

/* what a run of additions does to a sum in units, by the parity it starts from */
struct ParityFn {
    int i0, i1;
};
__device__ __forceinline__ ParityFn compose(ParityFn f, ParityFn g) {
    ParityFn r;
    r.i0 = f.i0 + ((f.i0 & 1) ? g.i1 : g.i0);
    r.i1 = f.i1 + ((f.i1 & 1) ? g.i0 : g.i1);
    return r;
}
__device__ __forceinline__ int binade(float s) { return (int)(__float_as_uint(s) >> 23); }

/* eight additions, as the engine does them */
__device__ __forceinline__ float add8(float s, const float (&q)[8]) {
#pragma unroll
    for (int j = 0; j < 8; j++) s = __fadd_rn(s, q[j]);
    return s;
}
__device__ __forceinline__ void square8(const unsigned char *p, float (&q)[8]) {
    float f[8];
    unpack8(*reinterpret_cast<const uint4 *>(p), f);
#pragma unroll
    for (int j = 0; j < 8; j++) q[j] = __fmul_rn(f[j], f[j]);
}

/* Sum of squares of a LaneRow; the chain's value in every lane.  One warp (parts
 * == 1), or two with half of the row each (parts == 2, an even lr.nu): the second
 * prepares everything while the first walks, then takes the sum over from
 * `hand_over` in shared memory and goes on, `meet` being a barrier of the two.
 *
 * P > 0: a lane's chunk is at most P pieces, and its squares stay in registers.  What bounds
 * a row is the walk over the lanes that leave a binade (about seven of 32 or 64), one
 * addition after another: out of registers 150 cycles for 32 of them, out of shared memory
 * twice that.  (P == 0: any chunk, rolled loops over shared memory; ALONE: the walking lane
 * reads alone, which an SM full of rows asks for.) */
template <int P, bool ALONE, typename Meet>
__device__ __forceinline__ float exact_sumsq(const unsigned char *row, const LaneRow lr, int lane,
                                             int part, int parts, float *hand_over, Meet meet) {
    /* chunk of this lane: of lr.nl * parts chunks in row order */
    const int per = lr.nu / parts, nl = lr.nl;           /* pieces of a chunk; lanes at work */
    const bool active = lane < nl;
    const int chunk = part * nl + (active ? lane : 0), l = chunk / parts;
    const unsigned char *mine = row + l * lr.pitch + (chunk - l * parts) * per * 16;
    const int nu = active ? per : 0;
    float qr[P > 0 ? P : 1][8];
    if (P > 0)
#pragma unroll
        for (int u = 0; u < P; u++) {
            /* (adding zeros changes nothing) */
            if (u < nu) square8(mine + u * 16, qr[u]);
            else
#pragma unroll
                for (int j = 0; j < 8; j++) qr[u][j] = 0.0f;
        }
    auto each = [&](auto use) {                          /* use(eight squares), in order */
        if (P > 0) {
#pragma unroll
            for (int u = 0; u < P; u++) use(qr[u]);
        } else {
#pragma unroll 1
            for (int u = 0; u < nu; u++) {
                float q[8];
                square8(mine + u * 16, q);
                use(q);
            }
        }
    };
    /* where the sum will be, roughly: tree sums and a scan over the lanes */
    auto tree8 = [](const float (&q)[8]) {
        return ((q[0] + q[1]) + (q[2] + q[3])) + ((q[4] + q[5]) + (q[6] + q[7]));
    };
    float tot = 0.0f;
    each([&](const float (&q)[8]) { tot += tree8(q); });
    float before = 0.0f;
    if (part) {                                          /* the first half's */
        const int c0 = active ? lane : 0, l0 = c0 / parts;
        const unsigned char *p = row + l0 * lr.pitch + (c0 - l0 * parts) * per * 16;
#pragma unroll 1
        for (int u = 0; u < nu; u++) {
            float q[8];
            square8(p + u * 16, q);
            before += tree8(q);
        }
        before = warp_sum(before);
    }
    float incl = tot;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
        const float v = __shfl_up_sync(0xffffffffu, incl, d);
        if (lane >= d) incl += v;
    }
    /* the binade this lane's terms are expected to be added in (key < 0: more than
     * one, or unsure) and what they do there, found by adding them to the binade's
     * smallest even and odd sum */
    const int b0 = binade((before + (incl - tot)) * 0.9998f),
              b1 = binade((before + incl) * 1.0002f);
    const int key = active && b0 == b1 && b0 > 0 && b0 < 255 ? b0 : -1 - lane;
    const float even = __uint_as_float((uint32_t)b0 << 23),
                odd = __uint_as_float(((uint32_t)b0 << 23) + 1u);
    float fe = even, fo = odd;
    each([&](const float (&q)[8]) {
        fe = add8(fe, q);
        fo = add8(fo, q);
    });
    ParityFn f;
    f.i0 = __float_as_int(fe) - __float_as_int(even);
    f.i1 = __float_as_int(fo) - __float_as_int(odd);
    /* joined over runs of lanes in the same binade */
    const int prev = __shfl_up_sync(0xffffffffu, key, 1);
    const unsigned heads = __ballot_sync(0xffffffffu, lane == 0 || key != prev);
    const int head = 31 - __clz(heads & (0xffffffffu >> (31 - lane)));
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
        ParityFn g;
        g.i0 = __shfl_up_sync(0xffffffffu, f.i0, d);
        g.i1 = __shfl_up_sync(0xffffffffu, f.i1, d);
        if (lane - d >= head) f = compose(g, f);
    }
    float s = 0.0f;
    if (part) {
        meet();
        s = *hand_over;
    }
    /* walk the runs in order; a run must start and end in its binade (then it never
     * left it), otherwise its lanes add one by one */
#pragma unroll 1
    for (int cur = 0; cur < nl;) {
        const unsigned rest = cur == 31 ? 0u : heads & (0xffffffffu << (cur + 1));
        const int end = min(rest ? __ffs(rest) - 1 : 32, nl);
        const int kb = __shfl_sync(0xffffffffu, key, cur);
        if (kb >= 0) {
            const int i0 = __shfl_sync(0xffffffffu, f.i0, end - 1),
                      i1 = __shfl_sync(0xffffffffu, f.i1, end - 1);
            const int bits = __float_as_int(s);
            const float s2 = __int_as_float(bits + ((bits & 1) ? i1 : i0));
            if (binade(s) == kb && binade(s2) == kb && s2 >= s) {
                s = s2;
                cur = end;
                continue;
            }
        }
#pragma unroll 1
        for (; cur < end; cur++) {
            float t = s;
            if (!ALONE) {                                    /* its own lane's counts */
                each([&](const float (&q)[8]) { t = add8(t, q); });
            } else if (lane == cur) {
#pragma unroll 2
                for (int u = 0; u < nu; u++) {
                    float q[8];
                    square8(mine + u * 16, q);
                    t = add8(t, q);
                }
            }
            s = __shfl_sync(0xffffffffu, t, cur);
        }
    }
    if (parts == 2 && part == 0) {
        if (lane == 0) *hand_over = s;
        meet();
    }
    return s;
}

/* The same sum of a row of 2048 values by W warps, four or two: what the one-kernel path waits
 * for before anything else.  A lane has 64 / W terms, and a binade's end costs
 * one addition instead of a chunk's: the tree sums say at which term the sum passes it, so a lane
 * there has a parity function for the terms before, the term itself with the neighbour that
 * lies nearer to the edge (the chain's sum may pass one term earlier or later than the tree's),
 * and a function for the terms behind.  The functions are joined from one such place to the
 * next, and every lane of the W warps walks the few joined runs and the terms between them.  A run must start
 * and end in the binade it was composed for, as above; otherwise everything is added in order.
 * Cycles of a row, instructions at hand: 2590 by four warps, 3310 by two, against 4000 to 4900
 * by two of the form above. */
constexpr int SUM_RUNS = 16;             /* runs of a warp, at most; one more ends them */
struct SumShare {
    float total[4];                      /* the warps' tree sums */
    float start;                         /* the sum of the row's first chunks */
    int n[4];                            /* runs of each warp; < 0: add in order */
    /* x: function of an even sum | binade << 24, y: of an odd one; z, w: the terms behind it */
    int4 run[4][SUM_RUNS];
};
template <int W, typename Meet>
__device__ __forceinline__ float exact_sumsq_wide(const unsigned char *row, const LaneRow lr,
                                                  int lane, int part, SumShare &sh, Meet meet) {
    constexpr int P = 8 / W, N = P * 8;         /* 16-byte pieces and terms of a lane */
    /* The row's first chunks, where a chunk may pass two edges, are simply added up: with two of
     * 16 terms 11 of 1600 normal rows had to be added in order, with three none. */
    constexpr int HEAD = W == 4 ? 3 : 2;
    const int chunk = part * 32 + lane, l = chunk / W;
    const unsigned char *mine = row + l * lr.pitch + (chunk - l * W) * P * 16;
    float q[N];
#pragma unroll
    for (int u = 0; u < P; u++) {
        float f[8];
        unpack8(*reinterpret_cast<const uint4 *>(mine + u * 16), f);
#pragma unroll
        for (int j = 0; j < 8; j++) q[u * 8 + j] = __fmul_rn(f[j], f[j]);
    }
    /* tree sums: of the lane, of the lanes before it, of the warps before that */
    float tot = 0.0f;
#pragma unroll
    for (int u = 0; u < P; u++)
        tot += ((q[u * 8] + q[u * 8 + 1]) + (q[u * 8 + 2] + q[u * 8 + 3])) +
               ((q[u * 8 + 4] + q[u * 8 + 5]) + (q[u * 8 + 6] + q[u * 8 + 7]));
    float incl = tot;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
        const float v = __shfl_up_sync(0xffffffffu, incl, d);
        if (lane >= d) incl += v;
    }
    if (lane == 31) sh.total[part] = incl;
    meet();
    float before = 0.0f;
#pragma unroll
    for (int w = 0; w < W - 1; w++)
        if (w < part) before += sh.total[w];
    const float first = before + (incl - tot);
    /* Binades, taken from the sums at the lanes' ends so that neighbours agree on them. */
    const bool head = chunk < HEAD;
    const int b1 = binade(before + incl);
    int b0 = __shfl_up_sync(0xffffffffu, b1, 1);
    if (lane == 0) b0 = binade(before);
    const bool cross = !head && b1 != b0;
    bool bad = b1 < b0 || b0 > 250;
    /* terms [0, j0) before the edge, j0 and j1 on it */
    const float edge = __uint_as_float((uint32_t)(b0 + 1) << 23);
    int j0 = N, j1 = N;
    if (cross) {
        float p = first, below = first, above = INFINITY;
        j0 = 0;
#pragma unroll
        for (int i = 0; i < N; i++) {
            p += q[i];
            const bool under = p < edge;
            j0 += under;
            if (under) below = p;
            else above = fminf(above, p);
        }
        j0 = min(j0, N - 1);
        j1 = j0;
        if (edge - below < above - edge) j0 = max(j0 - 1, 0);
        else j1 = min(j1 + 1, N - 1);
    }
    /* what the terms do to the smallest even and odd sum of their binade */
    const int e0 = head ? 0 : b0 << 23, e1 = b1 << 23;
    float fe = __int_as_float(e0), fo = __int_as_float(e0 + 1);
    float q0 = 0.0f, q1 = 0.0f;
#pragma unroll
    for (int i = 0; i < N; i++) {
        const float t = i < j0 ? q[i] : 0.0f;
        fe = __fadd_rn(fe, t);
        fo = __fadd_rn(fo, t);
    }
    auto square_at = [&](int i) {
        const float v = bf16_f32(reinterpret_cast<const uint16_t *>(mine)[i]);
        return __fmul_rn(v, v);
    };
    if (cross) {
        q0 = square_at(j0);
        if (j1 > j0) q1 = square_at(j1);
    }
    ParityFn pre;
    pre.i0 = __float_as_int(fe) - e0;
    pre.i1 = __float_as_int(fo) - (e0 + 1);
    if (part == 0) {
        float s = fe;
#pragma unroll
        for (int c = 1; c < HEAD; c++) {
            s = __shfl_sync(0xffffffffu, s, c - 1);
#pragma unroll
            for (int i = 0; i < N; i++) s = __fadd_rn(s, q[i]);
        }
        if (lane == HEAD - 1) sh.start = s;
        if (head) pre.i0 = pre.i1 = 0;
    }
    ParityFn f = pre;
    if (__any_sync(0xffffffffu, cross)) {
        fe = __int_as_float(e1);
        fo = __int_as_float(e1 + 1);
#pragma unroll
        for (int i = 0; i < N; i++) {
            const float t = i > j1 ? q[i] : 0.0f;
            fe = __fadd_rn(fe, t);
            fo = __fadd_rn(fo, t);
        }
        if (cross) {
            f.i0 = __float_as_int(fe) - e1;
            f.i1 = __float_as_int(fo) - (e1 + 1);
        }
    }
    /* joined from one edge to the next; the run that ends at a lane's edge is what the lanes
     * before it left and its own terms before the edge */
    const unsigned edges = __ballot_sync(0xffffffffu, cross);
    const int from = 31 - __clz((edges | 1u) & (0xffffffffu >> (31 - lane)));
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
        ParityFn g;
        g.i0 = __shfl_up_sync(0xffffffffu, f.i0, d);
        g.i1 = __shfl_up_sync(0xffffffffu, f.i1, d);
        if (lane - d >= from) f = compose(g, f);
    }
    ParityFn run;
    run.i0 = __shfl_up_sync(0xffffffffu, f.i0, 1);
    run.i1 = __shfl_up_sync(0xffffffffu, f.i1, 1);
    run = lane > 0 ? compose(run, pre) : pre;
    bad = __any_sync(0xffffffffu, bad) || __popc(edges) >= SUM_RUNS;
    if (cross && !bad)
        sh.run[part][__popc(edges & ((1u << lane) - 1u))] =
            make_int4(run.i0 | (b0 << 24), run.i1, __float_as_int(q0), __float_as_int(q1));
    if (lane == 31) {
        const int n = __popc(edges);
        if (!bad) sh.run[part][n] = make_int4(f.i0 | (b1 << 24), f.i1, 0, 0);
        sh.n[part] = bad ? -1 : n + 1;
    }
    meet();
    float s = sh.start;
    int n[W];
    int4 r[W];
#pragma unroll
    for (int w = 0; w < W; w++) {
        n[w] = sh.n[w];
        r[w] = sh.run[w][0];
    }
    bool ok = true;
#pragma unroll
    for (int w = 0; w < W; w++) {
        ok &= n[w] > 0;
#pragma unroll 1
        for (int i = 1;; i++) {
            const int4 next = sh.run[w][min(i, SUM_RUNS - 1)];
            const int at = __float_as_int(s), to = at + ((at & 1) ? r[w].y : r[w].x & 0xffffff);
            ok &= (at >> 23) == (int)((unsigned)r[w].x >> 24) && (to >> 23) == (at >> 23);
            s = __fadd_rn(__fadd_rn(__int_as_float(to), __int_as_float(r[w].z)),
                          __int_as_float(r[w].w));
            if (i >= n[w]) break;
            r[w] = next;
        }
    }
    if (!ok) {                               /* (inline: a call cost 1 % of a decode layer) */
        s = 0.0f;
#pragma unroll 1
        for (int c = 0; c < lr.nl * lr.nu; c++) {
            float t[8];
            square8(row + lr.at(c), t);
            s = add8(s, t);
        }
        meet();                              /* the caller may write over the row */
    }
    return s;
}

/* y = rnd((x * rs) * (1 + w)), eight values; w: the gain offsets */
__device__ __forceinline__ uint4 norm8(const uint4 v, const uint4 g, float rs) {
    const uint32_t xw[4] = {v.x, v.y, v.z, v.w}, gw[4] = {g.x, g.y, g.z, g.w};
    uint32_t o[4];
#pragma unroll
    for (int q = 0; q < 4; q++) {
        const float g0 = __fadd_rn(1.0f, bf16lo(gw[q])), g1 = __fadd_rn(1.0f, bf16hi(gw[q]));
        o[q] = pack_bf16_rn(__fmul_rn(__fmul_rn(bf16lo(xw[q]), rs), g0),
                            __fmul_rn(__fmul_rn(bf16hi(xw[q]), rs), g1));
    }
    return make_uint4(o[0], o[1], o[2], o[3]);
}
__device__ __forceinline__ float norm_scale(float ss, int H) {
    return __fdiv_rn(1.0f, __fsqrt_rn(__fadd_rn(__fdiv_rn(ss, (float)H), 1e-6f)));
}

/* RMSNorm with (1+w) gain (c/attn.h:175-186), rows of N % 8 == 0 values, 16-byte
 * aligned; one warp per row.  Bound: the latency of one row for few rows, and instruction issue
 * for many.  P as above, the smallest that holds lr.nu pieces (a lane adds the zeros of the
 * others too, and every piece takes registers from the rows beside it): 2 from N 512, 4, 8 up
 * to 2048; 0: longer rows and those of few lanes.  us, squares in shared memory -> as now (P 8
 * or 0 for all): 8192 rows of N 512 21.1 -> 17.9 (24.2), 1024 26.2 -> 20.0 (26.9), 2048 35.7 ->
 * 31.1, 2560 42.4 -> 42.5 (52.8), 4096 60.3 -> 61.2 (73.6); 33 rows of 2048 11.7 -> 10.3. */
constexpr int RN_WARPS = 4;
template <int P>
__global__ void __launch_bounds__(RN_WARPS * 32)
rmsnorm_rows_kernel(const uint16_t *__restrict__ x, const uint16_t *__restrict__ w,
                    uint16_t *__restrict__ y, int T, int N, LaneRow lr) {
    extern __shared__ __align__(16) unsigned char rn_smem[];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int t = blockIdx.x * RN_WARPS + warp;
    pdl_enter();
    if (t >= T) return;
    unsigned char *row = rn_smem + warp * lr.bytes();
    const uint4 *src = reinterpret_cast<const uint4 *>(x + (size_t)t * N);
    const uint4 *gsrc = reinterpret_cast<const uint4 *>(w);
    constexpr int R = 8;                /* pieces a lane holds: rows of up to 2048 values */
    uint4 g[R];
    if (N <= R * 256) {
        uint4 v[R];
#pragma unroll
        for (int i = 0; i < R; i++) {
            const int c = lane + 32 * i;
            v[i] = c < N / 8 ? __ldg(src + c) : make_uint4(0, 0, 0, 0);
            g[i] = w && c < N / 8 ? __ldg(gsrc + c) : make_uint4(0, 0, 0, 0);
        }
#pragma unroll
        for (int i = 0; i < R; i++) {
            const int c = lane + 32 * i;
            if (c < N / 8) *reinterpret_cast<uint4 *>(row + lr.at(c)) = v[i];
        }
    } else {
        for (int c = lane; c < N / 8; c += 32)
            *reinterpret_cast<uint4 *>(row + lr.at(c)) = __ldg(src + c);
    }
    __syncwarp();
    const float rs =
        norm_scale(exact_sumsq<P, P == 0>(row, lr, lane, 0, 1, nullptr, [] {}), N);
    uint4 *dst = reinterpret_cast<uint4 *>(y + (size_t)t * N);
    if (N <= R * 256) {
#pragma unroll
        for (int i = 0; i < R; i++) {
            const int c = lane + 32 * i;
            if (c < N / 8)
                dst[c] = norm8(*reinterpret_cast<const uint4 *>(row + lr.at(c)), g[i], rs);
        }
    } else {
        for (int c = lane; c < N / 8; c += 32)
            dst[c] = norm8(*reinterpret_cast<const uint4 *>(row + lr.at(c)),
                           w ? __ldg(gsrc + c) : make_uint4(0, 0, 0, 0), rs);
    }
}

/* The same for rows of 2048 values, at most one to an SM: the latency of one row is all that is
 * waited for, so four warps share it.  One CTA per row.  Back to back, us, the form above -> this:
 * 9 rows 4.8 -> 2.3, 61 rows 4.9 -> 2.4, 148 rows 4.9 -> 2.4; four layers of 9 tokens 389 -> 376,
 * of 32 731 -> 718, of 148 1101 -> 1097.  From 300 rows on one of them often needs the sum in
 * order (9.3 against 5.5): those stay with the form above. */
__global__ void __launch_bounds__(128)
rmsnorm_wide_kernel(const uint16_t *__restrict__ x, const uint16_t *__restrict__ w,
                    uint16_t *__restrict__ y) {
    constexpr int N = 2048;
    __shared__ __align__(16) unsigned char row[32 * (N / 16 + 16)];
    __shared__ SumShare share;
    const LaneRow lr(N);
    const int tid = threadIdx.x;
    const uint4 *src = reinterpret_cast<const uint4 *>(x + (size_t)blockIdx.x * N),
                *gsrc = reinterpret_cast<const uint4 *>(w);
    uint4 g[2] = {make_uint4(0, 0, 0, 0), make_uint4(0, 0, 0, 0)}, v[2];
    pdl_enter();                             /* the gains too may be the kernel's before */
    if (w)
#pragma unroll
        for (int i = 0; i < 2; i++) g[i] = __ldg(gsrc + tid + 128 * i);
#pragma unroll
    for (int i = 0; i < 2; i++) v[i] = __ldg(src + tid + 128 * i);
#pragma unroll
    for (int i = 0; i < 2; i++) *reinterpret_cast<uint4 *>(row + lr.at(tid + 128 * i)) = v[i];
    __syncthreads();
    const float rs = norm_scale(
        exact_sumsq_wide<4>(row, lr, tid & 31, tid >> 5, share, [] { __syncthreads(); }), N);
    uint4 *dst = reinterpret_cast<uint4 *>(y + (size_t)blockIdx.x * N);
#pragma unroll
    for (int i = 0; i < 2; i++) dst[tid + 128 * i] = norm8(v[i], g[i], rs);
}

/* A logit as far as it is known: the BF16 codes between which the chain's rounded
 * result must lie, low code in the low half.  Equal halves: known. */
__device__ __forceinline__ bool code_known(uint32_t lohi) {
    return (lohi & 0xffffu) == (lohi >> 16);
}
constexpr uint32_t CODE_UNKNOWN = 0x7f80ff80u;       /* [-inf, +inf] */

/* At least the 2-norm of n values whose squares an fp32 sum (any order) gave as ss: the
 * sum is within a relative n 2^-23 and, where squares underflow, n 2^-149. */
__device__ __forceinline__ float norm_above(float ss, int n) {
    return sqrtf(ss + (float)n * 1.4e-45f) * 1.001f;
}

/* The logit of one weight row and one token by a warp: LaneRows, every product exact
 * (the caller has checked the operands' ranges).  A lane adds its terms in eights (two
 * chains of four and their sum) onto a running sum; the lanes' sums are scanned.  The
 * error terms, with u = 2^-24:
 *   chain against true sum:  u * sum over its adds of |result|; a result inside an
 *     eight is at most |sum before the lane| + |running sum before the eight| + the
 *     eight's sum of magnitudes;
 *   this sum against the true one:  4 u of the magnitudes, u |running sum| per eight,
 *     u |lane sum| per level of the scan (five; six with the lane's last running sum, and
 *     eight are taken).
 * The magnitudes of all eights together are at most cs = ||w|| ||x|| (Cauchy-Schwarz).
 * The factors below round up (second-order terms, and the fp32 sums that the bound
 * itself is built from). */
__device__ __forceinline__ uint32_t certified_logit(const unsigned char *w, const unsigned char *x,
                                                    const LaneRow lr, int lane, float cs) {
    const bool active = lane < lr.nl;
    const int nu = active ? lr.nu : 0;
    const unsigned char *wp = w + (active ? lane : 0) * lr.pitch,
                        *xp = x + (active ? lane : 0) * lr.pitch;
    float run = 0.0f, e = 0.0f;
#pragma unroll 2
    for (int g = 0; g < nu; g++) {
        float wf[8], xf[8];
        unpack8(*reinterpret_cast<const uint4 *>(wp + g * 16), wf);
        unpack8(*reinterpret_cast<const uint4 *>(xp + g * 16), xf);
        float s0 = __fmul_rn(wf[0], xf[0]), s1 = __fmul_rn(wf[4], xf[4]);
#pragma unroll
        for (int j = 1; j < 4; j++) {
            s0 = __fmaf_rn(wf[j], xf[j], s0);
            s1 = __fmaf_rn(wf[4 + j], xf[4 + j], s1);
        }
        e += fabsf(run);
        run += s0 + s1;
    }
    float sum = run;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
        const float v = __shfl_up_sync(0xffffffffu, sum, d);
        if (lane >= d) sum += v;
    }
    e = warp_sum(8.0f * nu * fabsf(sum - run) + 9.0f * e + 8.0f * fabsf(run));
    const float tot = __shfl_sync(0xffffffffu, sum, 31),
                err = (e + 12.0f * cs) * (1.05f * 5.9604645e-8f);
    const float lo = __fadd_rd(tot, -err), hi = __fadd_ru(tot, err);
    return lo <= hi ? (uint32_t)bf16_bits(lo) | ((uint32_t)bf16_bits(hi) << 16)
                    : CODE_UNKNOWN;                              /* NaN */
}

}  // namespace apus
