/*
 * exact_dense.cuh — the engine's dense products in its normative order, at the
 * speed of the weight stream (few rows) or of the fp32 pipes (many rows).
 *
 * y[m,o] is one fp32 chain per output, k strictly ascending, product and sum
 * each rounded once (c/bf16.h:285-294).  A product of two BF16 values has at
 * most 16 significant bits, so it is exact in fp32 unless it underflows or
 * overflows; then fma(w, x, acc) is the same number as rn(rn(w*x) + acc).  Each
 * CTA checks (smallest nonzero |w|, largest |w|: found once when the weights
 * become resident) against those of its own rows of x and otherwise runs the
 * literal multiply-then-add chain.
 *
 * The chain fixes the order inside an output, so the parallelism is outputs:
 *   exact_rows_kernel   up to four rows of x: one weight row per lane, weights
 *                       streamed through shared memory
 *   exact_tile_kernel   more rows: tiles of 8 x 32 to 32 x 128 (rows x outputs)
 * Both want K % 8 == 0 (16-byte pieces of a row); other K keep exact_gemm_kernel.
 */
#pragma once
#include "common.cuh"
#include "decode_gemv.cuh"

namespace apus {

struct ExactArgs {
    const uint16_t *w, *x;      /* [O, K], [M, K] */
    void *y;                    /* [M, O] BF16, or fp32 with f32_out */
    int M, K;
    long O;
    float wmin, wmax;           /* smallest nonzero |w| (0: unknown), largest |w| */
    int f32_out;
};

/* |code| range of n BF16 values: out[0] = min over the nonzero ones, out[1] =
 * max, as fp32 bits (the host initialises them to +inf and 0) */
__global__ void __launch_bounds__(256)
bf16_range_kernel(const uint16_t *__restrict__ w, size_t n, unsigned int *out) {
    unsigned int lo = 0x7f800000u, hi = 0;
    for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < n;
         i += (size_t)gridDim.x * blockDim.x) {
        const unsigned int a = ((unsigned int)w[i] << 16) & 0x7fffffffu;
        if (a != 0 && a < lo) lo = a;
        if (a > hi) hi = a;
    }
    lo = __reduce_min_sync(0xffffffffu, lo);
    hi = __reduce_max_sync(0xffffffffu, hi);
    if ((threadIdx.x & 31) == 0) {
        atomicMin(out, lo);
        atomicMax(out + 1, hi);
    }
}

/* range of eight packed codes, folded into lo / hi */
__device__ __forceinline__ void fold_range8(const uint4 &v, unsigned int &lo, unsigned int &hi) {
    const uint32_t w[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
    for (int q = 0; q < 4; q++) {
        const unsigned int a = (w[q] << 16) & 0x7fffffffu, b = w[q] & 0x7fff0000u;
        if (a != 0) lo = min(lo, a);
        if (b != 0) lo = min(lo, b);
        hi = max(hi, max(a, b));
    }
}
/* the same of many, two codes to an instruction: |code| - 1, where a zero is the largest */
struct PackedRange {
    uint32_t lo = 0xffffffffu, hi = 0;
    __device__ __forceinline__ void fold8(const uint4 &v) {
        const uint32_t w[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
        for (int q = 0; q < 4; q++) {
            const uint32_t m = w[q] & 0x7fff7fffu;
            uint32_t less;
            asm("add.u16x2 %0, %1, %2;" : "=r"(less) : "r"(m), "r"(0xffffffffu));
            asm("min.u16x2 %0, %0, %1;" : "+r"(lo) : "r"(less));
            asm("max.u16x2 %0, %0, %1;" : "+r"(hi) : "r"(m));
        }
    }
    /* as fold_range8 has them */
    __device__ __forceinline__ unsigned low() const {
        const unsigned m = min(lo & 0xffffu, lo >> 16);
        return m == 0xffffu ? 0x7f800000u : (m + 1u) << 16;
    }
    __device__ __forceinline__ unsigned high() const { return max(hi & 0xffffu, hi >> 16) << 16; }
};
/* every product of the two ranges is exact in fp32 (a NaN or an infinity on
 * either side fails the second test) */
__device__ __forceinline__ bool products_exact(float wmin, float wmax, unsigned int xlo,
                                               unsigned int xhi) {
    return wmin > 0.0f &&
           (double)wmin * (double)__uint_as_float(xlo) >= 7.52316384526264e-37 && /* 2^-120 */
           (double)wmax * (double)__uint_as_float(xhi) < 1.7e38;                  /* < 2^127 */
}
__device__ __forceinline__ void cp_async16_zfill(uint32_t dst, const void *src, bool valid) {
    const int bytes = valid ? 16 : 0;
    asm volatile("cp.async.ca.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(bytes)
                 : "memory");
}

template <bool FMA>
__device__ __forceinline__ float exact_step(float w, float x, float acc) {
    return FMA ? __fmaf_rn(w, x, acc) : __fadd_rn(acc, __fmul_rn(w, x));
}

/* ---- few rows ------------------------------------------------------------------
 * Bound: the weight stream.  A warp owns 32 consecutive weight rows, one per
 * lane, so a lane's chain needs its own row while HBM wants whole lines: the
 * warp copies 64 k of its 32 rows at a time (eight lanes per row, 128 bytes
 * each) into a private ring of shared memory with cp.async, several blocks ahead,
 * and every lane reads its row back from there (pitch 144 bytes: conflict-free).
 * Steps of one block cost about 350 cycles for 4 KB, so the eight warps of an SM
 * could take in 90 bytes per clock; HBM delivers 22.  O 248320, K 2048 (1 GB):
 * 162 us = 6.3 TB/s of measured 6.5 (one thread per row from global memory: 260). */
constexpr int ER_BK = 64;
constexpr int ER_PITCH = ER_BK * 2 + 16;
constexpr int ER_BUF = 32 * ER_PITCH;
constexpr int ER_MAX_M = 4;
/* blocks in flight per warp: what shared memory holds for eight warps; a CTA of
 * one to four warps has room for the whole memory latency of its only chain */
__host__ __device__ constexpr int er_stages(bool few) { return few ? 10 : 5; }
constexpr int ER_FEW_WARPS = 4;
inline size_t exact_rows_smem(int M, int K, int warps) {
    const size_t kp = ((size_t)K + ER_BK - 1) / ER_BK * ER_BK;
    return (size_t)M * kp * 4 + (size_t)warps * er_stages(warps <= ER_FEW_WARPS) * ER_BUF;
}

template <int M, int ER_STAGES, bool FMA>
__device__ __forceinline__ void exact_rows_walk(const ExactArgs &a, const float *xs, int kp,
                                                unsigned char *ring, long warp, long nwarps) {
    const int lane = threadIdx.x & 31;
    const int nkb = kp / ER_BK;
    const long groups = (a.O + 31) / 32;
    const long mine = warp < groups ? (groups - warp + nwarps - 1) / nwarps : 0;
    const long total = mine * nkb;
    const int pc = lane & 7, pr = lane >> 3;           /* piece of a row, row of four */
    const uint32_t dst0 = smem_u32(ring) + (uint32_t)(pr * ER_PITCH + pc * 16);
    /* the copy side runs ER_STAGES - 1 blocks ahead with its own position */
    long i_g = warp;
    int i_kb = 0, i_s = 0;
    long issued = 0;
    auto issue = [&]() {
        if (issued < total) {
            const int k = i_kb * ER_BK + pc * 8;
            const uint32_t dst = dst0 + (uint32_t)(i_s * ER_BUF);
#pragma unroll
            for (int j = 0; j < 8; j++) {
                const long o = i_g * 32 + j * 4 + pr;
                const bool ok = o < a.O && k < a.K;
                cp_async16_zfill(dst + (uint32_t)(j * 4 * ER_PITCH),
                                 a.w + (ok ? o * a.K + k : 0), ok);
            }
            if (++i_kb == nkb) {
                i_kb = 0;
                i_g += nwarps;
            }
            if (++i_s == ER_STAGES) i_s = 0;
            issued++;
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    for (int s = 0; s < ER_STAGES - 1; s++) issue();
    int s = 0;
    for (long g = warp; g < groups; g += nwarps) {
        float acc[M];
#pragma unroll
        for (int m = 0; m < M; m++) acc[m] = 0.0f;
#pragma unroll 1
        for (int kb = 0; kb < nkb; kb++) {
            asm volatile("cp.async.wait_group %0;" ::"n"(ER_STAGES - 2) : "memory");
            __syncwarp();      /* everyone's pieces landed; the oldest block is read out */
            issue();
            const unsigned char *wl = ring + (size_t)s * ER_BUF + (size_t)lane * ER_PITCH;
            const float *xk = xs + kb * ER_BK;
#pragma unroll
            for (int c = 0; c < ER_BK / 8; c++) {
                float wf[8];
                unpack8(*reinterpret_cast<const uint4 *>(wl + c * 16), wf);
#pragma unroll
                for (int m = 0; m < M; m++) {
                    const float4 xa = *reinterpret_cast<const float4 *>(xk + (size_t)m * kp + c * 8);
                    const float4 xb =
                        *reinterpret_cast<const float4 *>(xk + (size_t)m * kp + c * 8 + 4);
                    const float xf[8] = {xa.x, xa.y, xa.z, xa.w, xb.x, xb.y, xb.z, xb.w};
#pragma unroll
                    for (int j = 0; j < 8; j++) acc[m] = exact_step<FMA>(wf[j], xf[j], acc[m]);
                }
            }
            if (++s == ER_STAGES) s = 0;
        }
        const long o = g * 32 + lane;
        if (o < a.O) {
#pragma unroll
            for (int m = 0; m < M; m++) {
                if (a.f32_out)
                    reinterpret_cast<float *>(a.y)[(size_t)m * a.O + o] = acc[m];
                else
                    reinterpret_cast<uint16_t *>(a.y)[(size_t)m * a.O + o] = bf16_bits(acc[m]);
            }
        }
    }
    asm volatile("cp.async.wait_group 0;" ::: "memory");
}

template <int M, bool FEW>
__global__ void __launch_bounds__(256)
exact_rows_kernel(ExactArgs a) {
    constexpr int ER_STAGES = er_stages(FEW);
    extern __shared__ __align__(16) unsigned char er_smem[];
    __shared__ unsigned int s_lo, s_hi;
    const int kp = (a.K + ER_BK - 1) / ER_BK * ER_BK;
    float *xs = reinterpret_cast<float *>(er_smem);
    if (threadIdx.x == 0) {
        s_lo = 0x7f800000u;
        s_hi = 0;
    }
    __syncthreads();
    unsigned int lo = 0x7f800000u, hi = 0;
    for (int i = threadIdx.x; i < M * (kp / 8); i += blockDim.x) {
        const int m = i / (kp / 8), k = (i - m * (kp / 8)) * 8;
        const uint4 v = k < a.K ? ldg16(a.x + (size_t)m * a.K + k) : make_uint4(0, 0, 0, 0);
        float f[8];
        unpack8(v, f);
        fold_range8(v, lo, hi);
        float4 *d = reinterpret_cast<float4 *>(xs + (size_t)m * kp + k);
        d[0] = make_float4(f[0], f[1], f[2], f[3]);
        d[1] = make_float4(f[4], f[5], f[6], f[7]);
    }
    lo = __reduce_min_sync(0xffffffffu, lo);
    hi = __reduce_max_sync(0xffffffffu, hi);
    if ((threadIdx.x & 31) == 0) {
        atomicMin(&s_lo, lo);
        atomicMax(&s_hi, hi);
    }
    __syncthreads();
    const int warps = blockDim.x >> 5;
    unsigned char *ring = er_smem + (size_t)M * kp * 4 +
                          (size_t)(threadIdx.x >> 5) * ER_STAGES * ER_BUF;
    const long warp = (long)blockIdx.x * warps + (threadIdx.x >> 5),
               nwarps = (long)gridDim.x * warps;
    if (products_exact(a.wmin, a.wmax, s_lo, s_hi))
        exact_rows_walk<M, ER_STAGES, true>(a, xs, kp, ring, warp, nwarps);
    else
        exact_rows_walk<M, ER_STAGES, false>(a, xs, kp, ring, warp, nwarps);
}

/* ---- more rows -----------------------------------------------------------------
 * Bound: instruction issue.  A warp owns 32 * NO outputs (NO weight rows per lane)
 * x RM rows of x; the four warps of a CTA share the weight rows.
 * What the layout is for:
 *  - a shared-memory load delivers 128 bytes per cycle to the SM, broadcast or
 *    not.  fp32 operands under a 4 x 4 register tile cost 64 load cycles per k
 *    against 32 of multiply-adds (89 us at M 512, O 1024, K 2048), so operands
 *    stay BF16: a lane's 16 bytes are 8 k of its own weight row, or 8 k of one x
 *    row for the whole warp;
 *  - two chains per instruction (fma.rn.f32x2: the same fp32 pipes, half the issue
 *    slots) leave room for the shifts and masks that widen the operands.  The pair
 *    runs over two x rows; a weight is widened once and used for all RM of them.
 * M 512, O 1024, K 2048: 570 us as one thread per output reading global memory,
 * now 74 (fp32 pipes alone: 29; what is left is the widening, which the same pipes
 * do half of); M 64: 28, M 8, O 512: 28.
 * Rows arrive in blocks of 64 k (cp.async, eight lanes per row, pitch 144 bytes as
 * above), ET_STAGES - 1 blocks ahead; one barrier per block. */
constexpr int ET_STAGES = 4;
template <int RM, int NO>
struct ExactTile {
    static constexpr int M = 4 * RM, O = 32 * NO, THREADS = 128;
    static constexpr int SMEM = ET_STAGES * (O + M) * ER_PITCH;
};

__device__ __forceinline__ unsigned long long pack_f32x2(float lo, float hi) {
    unsigned long long r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
    return r;
}
template <bool FMA>
__device__ __forceinline__ void exact_step2(unsigned long long w, unsigned long long x,
                                            unsigned long long &acc) {
    if (FMA) {
        asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(acc) : "l"(w), "l"(x));
    } else {
        auto lo = [](unsigned long long v) { return __uint_as_float((uint32_t)v); };
        auto hi = [](unsigned long long v) { return __uint_as_float((uint32_t)(v >> 32)); };
        acc = pack_f32x2(__fadd_rn(lo(acc), __fmul_rn(lo(w), lo(x))),
                         __fadd_rn(hi(acc), __fmul_rn(hi(w), hi(x))));
    }
}

template <int RM, int NO, bool FMA>
__device__ __forceinline__ void exact_tile_body(const ExactArgs &a, unsigned char *smem, long o0,
                                                int m0) {
    using Tile = ExactTile<RM, NO>;
    constexpr int WROWS = Tile::O, ROWS = WROWS + Tile::M, BUF = ROWS * ER_PITCH;
    constexpr int STEP = Tile::THREADS / 8;             /* rows fetched side by side */
    constexpr int NP = (ROWS + STEP - 1) / STEP;        /* 16-byte pieces per thread */
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int nkb = (a.K + ER_BK - 1) / ER_BK;
    /* fetch side: piece fc of rows fr, fr + STEP, ... (rows of w, then rows of x) */
    const int fc = tid & 7, fr = tid >> 3;
    const uint16_t *src[NP];
    uint32_t rok = 0;
#pragma unroll
    for (int i = 0; i < NP; i++) {
        const int r = fr + i * STEP;
        const bool ok = r < WROWS ? o0 + r < a.O : r < ROWS && m0 + r - WROWS < a.M;
        src[i] = (r < WROWS ? a.w + (ok ? (o0 + r) * a.K : 0)
                            : a.x + (ok ? (long)(m0 + r - WROWS) * a.K : 0)) + fc * 8;
        rok |= (ok ? 1u : 0u) << i;
    }
    const uint32_t dst0 = smem_u32(smem) + (uint32_t)(fr * ER_PITCH + fc * 16);
    int f_s = 0;
    auto fetch = [&](int kb) {
        if (kb < nkb) {
            const bool kok = kb * ER_BK + fc * 8 < a.K;
#pragma unroll
            for (int i = 0; i < NP; i++) {
                const bool ok = kok && ((rok >> i) & 1u);
                if (fr + i * STEP < ROWS)
                    cp_async16_zfill(dst0 + (uint32_t)(f_s * BUF + i * STEP * ER_PITCH),
                                     ok ? src[i] + (size_t)kb * ER_BK : a.w, ok);
            }
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
        if (++f_s == ET_STAGES) f_s = 0;
    };
    unsigned long long acc[NO][RM / 2];
#pragma unroll
    for (int i = 0; i < NO; i++)
#pragma unroll
        for (int j = 0; j < RM / 2; j++) acc[i][j] = 0ull;
    for (int kb = 0; kb < ET_STAGES - 1; kb++) fetch(kb);
    int s = 0;
#pragma unroll 1
    for (int kb = 0; kb < nkb; kb++) {
        asm volatile("cp.async.wait_group %0;" ::"n"(ET_STAGES - 2) : "memory");
        __syncthreads();       /* block kb landed everywhere, block kb - 1 is used up */
        fetch(kb + ET_STAGES - 1);
        const unsigned char *wb = smem + (size_t)s * BUF + (size_t)lane * ER_PITCH;
        const unsigned char *xb = smem + (size_t)s * BUF + (size_t)(WROWS + warp * RM) * ER_PITCH;
        uint4 wv[2][NO], xv[2][RM];
        auto load = [&](int c, uint4 (&wq)[NO], uint4 (&xq)[RM]) {
#pragma unroll
            for (int i = 0; i < NO; i++)
                wq[i] = *reinterpret_cast<const uint4 *>(wb + i * 32 * ER_PITCH + c * 16);
#pragma unroll
            for (int m = 0; m < RM; m++)
                xq[m] = *reinterpret_cast<const uint4 *>(xb + m * ER_PITCH + c * 16);
        };
        auto use = [&](const uint4 (&wq)[NO], const uint4 (&xq)[RM]) {
#pragma unroll
            for (int h = 0; h < 8; h++) {
                auto word = [&](const uint4 &v) {
                    const uint32_t q = h < 2 ? v.x : h < 4 ? v.y : h < 6 ? v.z : v.w;
                    return (h & 1) ? bf16hi(q) : bf16lo(q);
                };
                unsigned long long wp[NO];
#pragma unroll
                for (int i = 0; i < NO; i++) {
                    const float f = word(wq[i]);
                    wp[i] = pack_f32x2(f, f);
                }
#pragma unroll
                for (int j = 0; j < RM / 2; j++) {
                    const unsigned long long xp = pack_f32x2(word(xq[2 * j]), word(xq[2 * j + 1]));
#pragma unroll
                    for (int i = 0; i < NO; i++) exact_step2<FMA>(wp[i], xp, acc[i][j]);
                }
            }
        };
        if (m0 + warp * RM < a.M) {
            load(0, wv[0], xv[0]);
#pragma unroll 1
            for (int c = 0; c < ER_BK / 8; c += 2) {
                load(c + 1, wv[1], xv[1]);
                use(wv[0], xv[0]);
                load(c + 2 < ER_BK / 8 ? c + 2 : 0, wv[0], xv[0]);
                use(wv[1], xv[1]);
            }
        }
        if (++s == ET_STAGES) s = 0;
    }
    __syncthreads();
#pragma unroll
    for (int i = 0; i < NO; i++) {
        const long o = o0 + i * 32 + lane;
        if (o >= a.O) continue;
#pragma unroll
        for (int j = 0; j < RM; j++) {
            const int m = m0 + warp * RM + j;
            if (m >= a.M) continue;
            const float v =
                __uint_as_float((uint32_t)(acc[i][j >> 1] >> ((j & 1) * 32)));
            if (a.f32_out)
                reinterpret_cast<float *>(a.y)[(size_t)m * a.O + o] = v;
            else
                reinterpret_cast<uint16_t *>(a.y)[(size_t)m * a.O + o] = bf16_bits(v);
        }
    }
}

/* grid: x over the row blocks (tiles that share weights run together), y over
 * the output blocks, taken in steps of gridDim.y */
template <int RM, int NO>
__global__ void __launch_bounds__(128)
exact_tile_kernel(ExactArgs a) {
    using Tile = ExactTile<RM, NO>;
    extern __shared__ __align__(16) unsigned char et_smem[];
    __shared__ unsigned int s_lo, s_hi;
    const int m0 = blockIdx.x * Tile::M, rows = min(Tile::M, a.M - m0);
    if (threadIdx.x == 0) {
        s_lo = 0x7f800000u;
        s_hi = 0;
    }
    __syncthreads();
    unsigned int lo = 0x7f800000u, hi = 0;
    const uint16_t *x0 = a.x + (size_t)m0 * a.K;
#pragma unroll 8
    for (long i = threadIdx.x; i < (long)rows * (a.K / 8); i += Tile::THREADS)
        fold_range8(ldg16(x0 + i * 8), lo, hi);
    lo = __reduce_min_sync(0xffffffffu, lo);
    hi = __reduce_max_sync(0xffffffffu, hi);
    if ((threadIdx.x & 31) == 0) {
        atomicMin(&s_lo, lo);
        atomicMax(&s_hi, hi);
    }
    __syncthreads();
    const bool fma = products_exact(a.wmin, a.wmax, s_lo, s_hi);
    for (long o0 = (long)blockIdx.y * Tile::O; o0 < a.O; o0 += (long)gridDim.y * Tile::O) {
        if (fma)
            exact_tile_body<RM, NO, true>(a, et_smem, o0, m0);
        else
            exact_tile_body<RM, NO, false>(a, et_smem, o0, m0);
    }
}

}  // namespace apus
