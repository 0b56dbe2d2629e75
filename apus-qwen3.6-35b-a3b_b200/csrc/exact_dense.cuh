/*
 * exact_dense.cuh — the engine's dense products in its normative order, at the
 * speed of the weight stream (few rows) or of the fp32 pipes (many rows).
 *
 * y[m,o] is one fp32 chain per output, k strictly ascending, product and sum
 * each rounded once (c/bf16.h:285-294).  A product of two BF16 values has at
 * most 16 significant bits, so it is exact in fp32 unless it underflows or
 * overflows; then fma(w, x, acc) is the same number as rn(rn(w*x) + acc).  Each
 * CTA checks (smallest nonzero |w|, largest |w|: found once when the weights
 * become resident) against those of its own rows of x, the kernel of many rows block by
 * block, and otherwise runs the literal multiply-then-add chain.
 *
 * The chain fixes the order inside an output, so the parallelism is outputs:
 *   exact_rows_kernel   up to four rows of x: one weight row per lane, weights
 *                       streamed through shared memory
 *   exact_tile_kernel   more rows: tiles of 2 x 128 to 32 x 128 (rows x outputs)
 * Both want K % 8 == 0 (16-byte pieces of a row); other K keep exact_gemm_kernel.
 */
#pragma once
#include <type_traits>

#include "common.cuh"
#include "decode_gemv.cuh"
#include "exact_codes.h"

namespace apus {

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
struct ExactArgs {
    const uint16_t *w, *x;      /* [O, K], [M, K] */
    void *y;                    /* [M, O] BF16, or fp32 with f32_out */
    int M, K;
    long O;
    float wmin, wmax;           /* smallest nonzero |w| (0: unknown), largest |w| */
    ExactCodes codes;           /* of x, for exact_tile_kernel */
    int f32_out;
};

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
 * Bound: the fp32 pipes and the issue slots beside them.  A warp owns 32 * NO outputs (NO
 * weight rows per lane) x RM rows of x; a CTA's four warps stand WM over rows of x and 4 / WM
 * over outputs, and share what they read.  What the layout is for:
 *  - two chains per instruction (fma.rn.f32x2: the same fp32 pipes, half the issue slots);
 *    the pair runs over two x rows;
 *  - widening takes as many instructions as multiplying if every operand is widened where it
 *    is used.  x is the same for all lanes, so the CTA widens a block of it once, into pairs
 *    of rows that a broadcast load puts where the multiply-add wants them; weights are a
 *    lane's own, stay BF16 (sixteen bytes are eight k) and are widened once for all RM rows.
 * Rows arrive in blocks of 64 k (cp.async, eight lanes per row; weights at pitch 144 bytes as
 * above), ET_STAGES - 1 blocks ahead; one barrier per block.  Whether a block's products are
 * exact is known when its x has been widened, a block ahead: up to the first that holds one
 * that may not be, both forms of the chain are the same, and from there on it is literal.
 * (A weight of 1e-38 among 512 rows, K 2048, O 1024 / 4096: calls of 192 / 481 us; the whole
 * chain again where it turns out inexact at its end 279 / 712, x read twice to know it before
 * 258 / 514.)
 * K 2048, a tile alone on its SM: 2 x 128 (rows x outputs) 24.3 us, 8 x 64 24.7, 16 x 64 29.9,
 * 32 x 128 70.  (Both operands widened in the lanes, 32 x 128: 74, 8 x 32: 28.) */
constexpr int ET_STAGES = 4;
constexpr int ET_WARPS = 4;
template <int RM, int NO, int WM>
struct ExactTile {
    static constexpr int WO = ET_WARPS / WM, M = RM * WM, O = WO * 32 * NO,
                         THREADS = ET_WARPS * 32;
    static constexpr int W_STAGE = O * ER_PITCH, R_STAGE = M * ER_BK * 2, X_BUF = ER_BK * M * 4;
    static constexpr int SMEM = ET_STAGES * (W_STAGE + R_STAGE) + 2 * X_BUF;
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

/* literal: two words of shared memory: products of an even, an odd block widened so far may
 * round */
template <int RM, int NO, int WM>
__device__ __forceinline__ void exact_tile_body(const ExactArgs &a, unsigned char *smem, long o0,
                                                int m0, volatile int *literal) {
    using Tile = ExactTile<RM, NO, WM>;
    constexpr int STEP = Tile::THREADS / 8;
    constexpr int XR = Tile::M * ER_BK / Tile::THREADS;  /* x rows that a thread widens */
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int wm = warp % WM, wo = warp / WM;
    const int nkb = (a.K + ER_BK - 1) / ER_BK;
    unsigned char *raw = smem + (size_t)ET_STAGES * Tile::W_STAGE;       /* x as it comes */
    float *xs = reinterpret_cast<float *>(raw + ET_STAGES * Tile::R_STAGE);   /* [2][WM][k][RM] */
    /* piece fc of rows fr, fr + STEP, ... */
    const int fc = tid & 7, fr = tid >> 3;
    const uint16_t *wsrc = a.w + (size_t)(o0 + fr) * a.K + fc * 8,
                   *xsrc = a.x + (size_t)(m0 + fr) * a.K + fc * 8;
    const uint32_t wdst = smem_u32(smem) + (uint32_t)(fr * ER_PITCH + fc * 16),
                   xdst = smem_u32(raw) + (uint32_t)(tid * 16);
    int f_s = 0;
    auto fetch = [&](int kb) {
        if (kb < nkb) {
            const bool kok = kb * ER_BK + fc * 8 < a.K;
#pragma unroll
            for (int i = 0; i < Tile::O / STEP; i++) {
                const bool ok = kok && o0 + fr + i * STEP < a.O;
                cp_async16_zfill(wdst + (uint32_t)(f_s * Tile::W_STAGE + i * STEP * ER_PITCH),
                                 ok ? wsrc + (size_t)(i * STEP) * a.K + kb * ER_BK : a.w, ok);
            }
#pragma unroll
            for (int i = 0; i < (Tile::M + STEP - 1) / STEP; i++)
                if (fr + i * STEP < Tile::M) {
                    const bool ok = kok && m0 + fr + i * STEP < a.M;
                    cp_async16_zfill(
                        xdst + (uint32_t)(f_s * Tile::R_STAGE + i * STEP * ER_BK * 2),
                        ok ? xsrc + (size_t)(i * STEP) * a.K + kb * ER_BK : a.x, ok);
                }
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
        if (++f_s == ET_STAGES) f_s = 0;
    };
    /* x: one k of XR rows */
    const int xk = tid & (ER_BK - 1), xr0 = (tid / ER_BK) * XR;
    int x_s = 0;
    auto widen_x = [&](int kb) {
        const uint16_t *src = reinterpret_cast<const uint16_t *>(raw + x_s * Tile::R_STAGE) +
                              xr0 * ER_BK + xk;
        if (++x_s == ET_STAGES) x_s = 0;
        float f[XR];
        unsigned lo = 0xffffffffu, hi = 0;
#pragma unroll
        for (int r = 0; r < XR; r++) {
            const unsigned v = src[r * ER_BK], m = v & 0x7fffu;
            lo = min(lo, m - 1u);
            hi = max(hi, m);
            f[r] = __uint_as_float(v << 16);
        }
        if (!a.codes.hold(lo, hi)) literal[kb & 1] = 1;
        float *d = xs + (kb & 1) * (ER_BK * Tile::M);
        constexpr int V = XR < RM ? XR : RM < 4 ? RM : 4;    /* rows to a store, of one group */
        static_assert(XR % V == 0 && RM % V == 0, "");
#pragma unroll
        for (int r = 0; r < XR; r += V) {
            const int row = xr0 + r;
            float *at = d + (row / RM * ER_BK + xk) * RM + row % RM;
            if (V == 4)
                *reinterpret_cast<float4 *>(at) =
                    make_float4(f[r], f[(r + 1) % XR], f[(r + 2) % XR], f[(r + 3) % XR]);
            else if (V == 2)
                *reinterpret_cast<float2 *>(at) = make_float2(f[r], f[(r + 1) % XR]);
            else
                at[0] = f[r];
        }
    };
    unsigned long long acc[NO][RM / 2];
#pragma unroll
    for (int i = 0; i < NO; i++)
#pragma unroll
        for (int j = 0; j < RM / 2; j++) acc[i][j] = 0ull;
    if (tid < 2) literal[tid] = 0;
    for (int kb = 0; kb < ET_STAGES - 1; kb++) fetch(kb);
    asm volatile("cp.async.wait_group %0;" ::"n"(ET_STAGES - 2) : "memory");
    __syncthreads();
    widen_x(0);
    int s = 0;
    auto landed = [&] {        /* block kb + 1 everywhere; block kb - 1 is used up */
        asm volatile("cp.async.wait_group %0;" ::"n"(ET_STAGES - 3) : "memory");
        __syncthreads();
    };
    /* four k of x, eight of the weights: the next ones are requested before these are used */
    uint4 wq[2][NO];
    unsigned long long xp[2][4][RM / 2];
    const unsigned char *wb;
    const float *xb;
    auto load_w = [&](int c, uint4 (&q)[NO]) {
#pragma unroll
        for (int i = 0; i < NO; i++)
            q[i] = *reinterpret_cast<const uint4 *>(wb + i * 32 * ER_PITCH + c * 16);
    };
    auto load_p = [&](int c4, unsigned long long (&q)[4][RM / 2]) {
        const float *at = xb + c4 * 4 * RM;
        if (RM >= 4) {
#pragma unroll
            for (int h = 0; h < 4; h++)
#pragma unroll
                for (int j = 0; j < RM / 4; j++) {
                    const ulonglong2 v = reinterpret_cast<const ulonglong2 *>(at + h * RM)[j];
                    q[h][2 * j] = v.x;
                    q[h][(2 * j + 1) % (RM / 2)] = v.y;
                }
        } else {                       /* two k to a load */
#pragma unroll
            for (int h = 0; h < 2; h++) {
                const ulonglong2 v = reinterpret_cast<const ulonglong2 *>(at)[h];
                q[2 * h][0] = v.x;
                q[2 * h + 1][0] = v.y;
            }
        }
    };
    /* requested before it is known which form the block takes (2 x 128 25.7 -> 24.6 us), where
     * the registers that this holds are no matter (32 x 128: 165 and 128 of them, 130.5 us for
     * 125.7) */
    constexpr bool EARLY = RM * NO <= 8;
    auto first = [&] {
        load_w(0, wq[0]);
        load_p(0, xp[0]);
    };
    auto start = [&](int kb) {
        wb = smem + (size_t)s * Tile::W_STAGE + (size_t)(wo * 32 * NO + lane) * ER_PITCH;
        xb = xs + (kb & 1) * (ER_BK * Tile::M) + wm * (ER_BK * RM);
        if (++s == ET_STAGES) s = 0;
        fetch(kb + ET_STAGES - 1);
        if (kb + 1 < nkb) widen_x(kb + 1);
        if (EARLY) first();
    };
    auto multiply = [&](auto fma) {
        if (!EARLY) first();
        auto use = [&](const uint4 (&wv)[NO], int half, const unsigned long long (&q)[4][RM / 2]) {
#pragma unroll
            for (int h = 0; h < 4; h++)
#pragma unroll
                for (int i = 0; i < NO; i++) {
                    const uint32_t v = half ? (h < 2 ? wv[i].z : wv[i].w)
                                            : (h < 2 ? wv[i].x : wv[i].y);
                    const float f = (h & 1) ? bf16hi(v) : bf16lo(v);
                    const unsigned long long wp = pack_f32x2(f, f);
#pragma unroll
                    for (int j = 0; j < RM / 2; j++)
                        exact_step2<decltype(fma)::value>(wp, q[h][j], acc[i][j]);
                }
        };
        /* Unrolled, the products of a whole block are scheduled together: 16 x 64 31.6 -> 29.9 us,
         * two of them on an SM 66.2 -> 62.4, 2 x 128 24.6 -> 24.3.  32 x 128 gains nothing (69.8,
         * 70.0), and its literal form outgrows the instruction cache (calls of 512 x 4096 481 ->
         * 600). */
        constexpr int TURNS = RM * NO <= 8 ? ER_BK / 16 : 1;
#pragma unroll TURNS
        for (int c = 0; c < ER_BK / 8; c += 2) {
            const int next = c + 2 < ER_BK / 8 ? c + 2 : 0;
            load_p(2 * c + 1, xp[1]);
            load_w(c + 1, wq[1]);
            use(wq[0], 0, xp[0]);
            load_p(2 * c + 2, xp[0]);
            use(wq[0], 1, xp[1]);
            load_p(2 * c + 3, xp[1]);
            load_w(next, wq[0]);
            use(wq[1], 0, xp[0]);
            load_p(2 * next, xp[0]);
            use(wq[1], 1, xp[1]);
        }
    };
    int kb = 0;
    bool lit = false;
#pragma unroll 1
    for (; kb < nkb; kb++) {
        landed();
        lit = literal[kb & 1] != 0;
        start(kb);
        if (lit) break;
        multiply(std::true_type());
    }
    if (lit)
#pragma unroll 1
        for (;;) {
            multiply(std::false_type());
            if (++kb == nkb) break;
            landed();
            start(kb);
        }
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    __syncthreads();
#pragma unroll
    for (int i = 0; i < NO; i++) {
        const long o = o0 + (wo * NO + i) * 32 + lane;
        if (o >= a.O) continue;
#pragma unroll
        for (int j = 0; j < RM; j++) {
            const int m = m0 + wm * RM + j;
            if (m >= a.M) continue;
            const float v = __uint_as_float((uint32_t)(acc[i][j >> 1] >> ((j & 1) * 32)));
            const size_t at = (size_t)m * a.O + o;
            if (a.f32_out)
                reinterpret_cast<float *>(a.y)[at] = v;
            else
                reinterpret_cast<uint16_t *>(a.y)[at] = bf16_bits(v);
        }
    }
}

/* grid: one CTA per tile, or any number of them; tiles that share weights side by side */
template <int RM, int NO, int WM>
__global__ void __launch_bounds__(ET_WARPS * 32)
exact_tile_kernel(ExactArgs a) {
    using Tile = ExactTile<RM, NO, WM>;
    extern __shared__ __align__(16) unsigned char et_smem[];
    __shared__ int s_literal[2];
    const long mt = (a.M + Tile::M - 1) / Tile::M, tiles = mt * ((a.O + Tile::O - 1) / Tile::O);
#pragma unroll 1
    for (long tile = blockIdx.x; tile < tiles; tile += gridDim.x) {
        const long ot = tile / mt;
        exact_tile_body<RM, NO, WM>(a, et_smem, ot * Tile::O, (int)(tile - ot * mt) * Tile::M,
                                    s_literal);
    }
}

}  // namespace apus
