/*
 * misc_kernels.cuh — the engine's per-matmul hooks in its normative
 * accumulation order, the two steps either side of the MoE block, and the
 * synthetic-tensor fill.
 */
#pragma once
#include "common.cuh"
#include "synth.h"

namespace apus {

/* One fp32 chain per output, k strictly ascending, product and sum each
 * rounded once (c/bf16.h:285-294).  The product of two BF16 values is exact
 * in fp32 unless it underflows; the literal multiply-then-add is kept here.  This
 * form serves rows that are not made of aligned 16-byte pieces (K % 8 != 0); the
 * others run exact_dense.cuh. */
__device__ __forceinline__ float exact_dot(const uint16_t *__restrict__ wrow,
                                           const uint16_t *__restrict__ xrow,
                                           int K) {
    float acc = 0.0f;
    /* a lane's row and its own sequence of steps: the next sixteen operands are under way
     * during the adds of these (M 40, O 333, K 1001, with both copies: 88 -> 66 us) */
    constexpr int B = 16;
    uint16_t wv[B], xv[B];
#pragma unroll
    for (int j = 0; j < B; j++) {
        wv[j] = j < K ? __ldg(wrow + j) : (uint16_t)0;
        xv[j] = j < K ? __ldg(xrow + j) : (uint16_t)0;
    }
    int k = 0;
#pragma unroll 1
    for (; k + B <= K; k += B) {
#pragma unroll
        for (int j = 0; j < B; j++) {
            acc = __fadd_rn(acc, __fmul_rn(bf16_f32(wv[j]), bf16_f32(xv[j])));
            const int n = k + B + j;
            wv[j] = n < K ? __ldg(wrow + n) : (uint16_t)0;
            xv[j] = n < K ? __ldg(xrow + n) : (uint16_t)0;
        }
    }
#pragma unroll
    for (int j = 0; j < B; j++)
        if (k + j < K) acc = __fadd_rn(acc, __fmul_rn(bf16_f32(wv[j]), bf16_f32(xv[j])));
    return acc;
}

/* y[m,o] = rnd(chain) — apus_bf16_gemv_hot / apus_bf16_gemm_hot
 * (c/bf16.h:199-231), row m of a GEMM bitwise its GEMV. */
__global__ void __launch_bounds__(128)
exact_gemm_kernel(const uint16_t *__restrict__ w, const uint16_t *__restrict__ x,
                  uint16_t *__restrict__ y, long M, long O, int K) {
    for (long i = (long)blockIdx.x * blockDim.x + threadIdx.x; i < M * O;
         i += (long)gridDim.x * blockDim.x) {
        long m = i / O, o = i - m * O;
        y[i] = bf16_bits(exact_dot(w + o * K, x + m * K, K));
    }
}
/* fp32-out matvec, no narrowing — apus_moe_matvec_f32_hot (c/moe.h:284-310) */
__global__ void __launch_bounds__(128)
exact_matvec_f32_kernel(const uint16_t *__restrict__ w,
                        const uint16_t *__restrict__ x, float *__restrict__ y,
                        long O, int K) {
    for (long o = (long)blockIdx.x * blockDim.x + threadIdx.x; o < O;
         o += (long)gridDim.x * blockDim.x)
        y[o] = exact_dot(w + o * K, x, K);
}

/* y[m,o] = rnd(sum_k W[o,k] x[m,k]) as a weight STREAM (the engine's largest
 * dense product per token is the output head, 248320 x 2048 = 1 GB of weights,
 * c/model.h:667-688): device pointers, M <= 8 rows of x, K % 256 == 0.
 *
 * Bound: the weight stream.  A warp owns 16 weight rows at a time and copies 128 k of
 * them per slot into a ring of its own (cp.async, whole 256-byte pieces of a row), four
 * slots ahead; mma.sync m16n8k16 multiplies them with all rows of x at once (columns past
 * M repeat the last row and are not stored), so eight rows cost what one does.  Scalar
 * multiply-adds on rows loaded straight into registers took 174 us for one row and 780 for
 * eight (O 248320, K 2048); this 168 and 174 (6.0 of 6.5 TB/s).
 * mma.sync cuts off what its accumulator cannot hold, so two steps share one that starts
 * at zero and the rest is a tree: at K 2048 1.0e-4 of the results narrow to another BF16
 * value than 64-bit sums do, as in the scalar form (6e-4 with all 64 steps on one); at
 * K 8192 1.1e-4 (scalar 1.7e-4, 23e-4).
 * The summation order differs from the engine's sequential chain, so the result
 * agrees to BF16 tolerance, not bitwise; the exact-order form is exact_dense.cuh
 * behind the host-pointer hooks. */
constexpr int GV_BK = 128;
constexpr int GV_PITCH = GV_BK * 2 + 16;         /* ldmatrix rows in different banks */
constexpr int GV_SLOT = 16 * GV_PITCH;
constexpr int GV_STAGES = 5;
/* Too few rows for all warps: `split` of them (a power of two) share sixteen rows, each
 * with a part of K, and add up in shared memory; one warp alone is bound by the latency of
 * its four slots (2048 rows of 2048: 8.4 us for one row of x and 12.3 for eight; shared 3.9
 * and 6.3, the scalar form 4.5 and 19). */
constexpr int GV_PART = 16 * 8 * 4;
inline size_t gemv_stream_smem(int M, int K, int warps, int split) {
    return (size_t)M * (2 * (size_t)K + 16) +
           (size_t)warps * (GV_STAGES * GV_SLOT + (split > 1 ? GV_PART : 0));
}

__global__ void __launch_bounds__(256)
gemv_stream_kernel(const uint16_t *__restrict__ w, const uint16_t *__restrict__ x,
                   uint16_t *__restrict__ y, int M, long O, int K, int split, long rounds) {
    extern __shared__ __align__(16) unsigned char gv_smem[];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, warps = blockDim.x >> 5;
    const int team = warp / split, part = warp - team * split, teams = warps / split;
    const int x_pitch = 2 * K + 16;
    const uint32_t ring = smem_u32(gv_smem) + (uint32_t)(M * x_pitch + warp * GV_STAGES * GV_SLOT);
    float *sums = reinterpret_cast<float *>(gv_smem + (size_t)M * x_pitch +
                                            (size_t)warps * GV_STAGES * GV_SLOT) +
                  (size_t)warp * (GV_PART / 4);
    /* As many rounds as sixteen rows per team ask for, the teams side by side, all rows
     * dealt evenly (of a piece of fewer than sixteen those missing are not fetched, what lies
     * in their place is not stored).  Whole rounds and a short last one left a team alone
     * with a row or two, at the latency of its slots: O 20000, K 8192 92 us against 62. */
    const unsigned nw = gridDim.x * teams, id = team * gridDim.x + blockIdx.x;
    const long per = O / rounds, extra = O - per * rounds;       /* a round's rows (+ 1) */
    auto piece = [&](long i, long &o, long &end) {
        const unsigned n = (unsigned)per + (i < extra), q = n / nw, r = n - q * nw;
        o = i * per + min(i, extra) + id * q + min(id, r);
        end = o + q + (id < r);
    };
    const int kb0 = K / GV_BK * part / split, kb1 = K / GV_BK * (part + 1) / split;
    long i_i = 0, i_o, i_end;
    int i_kb = kb0, i_s = 0;
    piece(0, i_o, i_end);
    auto issue = [&]() {
        if (i_i < rounds) {
            const int c = lane & 15;
            const uint32_t dst = ring + (uint32_t)(i_s * GV_SLOT + c * 16);
#pragma unroll
            for (int j = 0; j < 8; j++) {
                const int r = j * 2 + (lane >> 4);
                const long o = i_o + r;
                if (o < i_end)
                    cp_async16_to(dst + (uint32_t)(r * GV_PITCH),
                                  w + o * K + i_kb * GV_BK + c * 8);
            }
            if (++i_kb == kb1) {
                i_kb = kb0;
                if (++i_i < rounds) piece(i_i, i_o, i_end);
            }
            if (++i_s == GV_STAGES) i_s = 0;
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    for (int s = 0; s < GV_STAGES - 1; s++) issue();
    if ((reinterpret_cast<uintptr_t>(x) & 15) == 0) {
        for (int m = 0; m < M; m++)
            for (int p = threadIdx.x; p < K / 8; p += blockDim.x)
                *reinterpret_cast<uint4 *>(gv_smem + (size_t)m * x_pitch + p * 16) =
                    ldg16(x + (size_t)m * K + p * 8);
    } else {
        for (int m = 0; m < M; m++)
            for (int k = threadIdx.x; k < K; k += blockDim.x)
                *reinterpret_cast<uint16_t *>(gv_smem + (size_t)m * x_pitch + k * 2) =
                    x[(size_t)m * K + k];
    }
    __syncthreads();
    /* ldmatrix: weights (rows 0-7, k 0-7), (rows 8-15, k 0-7), (rows 0-7, k 8-15), ..;
     * x: eight k of the eight columns per matrix, 32 k at a time */
    const uint32_t a_off = (uint32_t)((lane & 15) * GV_PITCH + (lane >> 4) * 16);
    const uint32_t b_at = smem_u32(gv_smem) + (uint32_t)(min(lane & 7, M - 1) * x_pitch +
                                                         (lane >> 3) * 16);
    int s = 0;
    for (long i = 0; i < rounds; i++) {
        long o0, o_end;
        piece(i, o0, o_end);
        float c0[4] = {0, 0, 0, 0}, c1[4] = {0, 0, 0, 0};
#pragma unroll 1
        for (int kb = kb0; kb < kb1; kb++) {
            asm volatile("cp.async.wait_group %0;" ::"n"(GV_STAGES - 2) : "memory");
            __syncwarp();      /* everyone's pieces landed; the oldest slot is read out */
            issue();
            const uint32_t at = ring + (uint32_t)(s * GV_SLOT) + a_off;
            /* everything is read before the first product, and no product waits for the one
             * before it (the warp issues in order) */
            uint32_t a0[4][4], a1[4][4], b[4][4];
            float p[4][4];
#pragma unroll
            for (int j = 0; j < 4; j++) {
                ldmatrix_x4(b[j], b_at + (uint32_t)((kb * GV_BK + j * 32) * 2));
                ldmatrix_x4(a0[j], at + (uint32_t)(j * 64));
                ldmatrix_x4(a1[j], at + (uint32_t)(j * 64 + 32));
            }
#pragma unroll
            for (int j = 0; j < 4; j++) mma_16x8_first(p[j], a0[j], b[j][0], b[j][1]);
#pragma unroll
            for (int j = 0; j < 4; j++) mma_16x8(p[j], a1[j], b[j][2], b[j][3]);
            const bool fold = (kb & 3) == 3;
#pragma unroll
            for (int q = 0; q < 4; q++) {
                c0[q] += (p[0][q] + p[1][q]) + (p[2][q] + p[3][q]);
                if (fold) {
                    c1[q] += c0[q];
                    c0[q] = 0.0f;
                }
            }
            if (++s == GV_STAGES) s = 0;
        }
#pragma unroll
        for (int q = 0; q < 4; q++) c0[q] += c1[q];
        if (split > 1) {
            *reinterpret_cast<float4 *>(sums + lane * 4) = make_float4(c0[0], c0[1], c0[2], c0[3]);
            asm volatile("bar.sync %0, %1;" ::"r"(1 + team), "r"(split * 32) : "memory");
            if (part == 0)
                for (int p = 1; p < split; p++) {
                    const float4 v =
                        *reinterpret_cast<const float4 *>(sums + p * (GV_PART / 4) + lane * 4);
                    c0[0] += v.x;
                    c0[1] += v.y;
                    c0[2] += v.z;
                    c0[3] += v.w;
                }
            asm volatile("bar.sync %0, %1;" ::"r"(1 + team), "r"(split * 32) : "memory");
            if (part) continue;
        }
#pragma unroll
        for (int q = 0; q < 4; q++) {
            const long o = o0 + (lane >> 2) + (q >> 1) * 8;
            const int m = (lane & 3) * 2 + (q & 1);
            if (o < o_end && m < M) y[(size_t)m * O + o] = bf16_bits(c0[q]);
        }
    }
    asm volatile("cp.async.wait_group 0;" ::: "memory");
}

/* RMSNorm with (1+w) gain, single rounding (c/attn.h:175-186): the sum of
 * squares is the ascending sequential fp32 chain; one warp per row, lane 0
 * walks the chain over the row staged in shared memory. */
__global__ void __launch_bounds__(128)
rmsnorm_kernel(const uint16_t *__restrict__ x, const uint16_t *__restrict__ w,
               uint16_t *__restrict__ y, int T, int N) {
    extern __shared__ float rs_smem[];   /* [4][N] */
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int t = blockIdx.x * 4 + warp;
    if (t >= T) return;
    float *row = rs_smem + (size_t)warp * N;
    for (int i = lane; i < N; i += 32)
        row[i] = bf16_f32(x[(size_t)t * N + i]);
    __syncwarp();
    /* the reference's sum of squares is one ascending fp32 chain; the dependent
     * add is the critical path, so operands come in vectors, sixteen steps per
     * iteration, and the next iteration's loads are hoisted above the adds */
    float ss = 0.0f;
    if (lane == 0) {
        int i = 0;
        const float4 *r4 = reinterpret_cast<const float4 *>(row);
#pragma unroll 2
        for (; (N & 3) == 0 && i + 16 <= N; i += 16) {   /* rows stay 16-byte aligned */
            const float4 v[4] = {r4[i / 4], r4[i / 4 + 1], r4[i / 4 + 2], r4[i / 4 + 3]};
#pragma unroll
            for (int q = 0; q < 4; q++) {
                ss = __fadd_rn(ss, __fmul_rn(v[q].x, v[q].x));
                ss = __fadd_rn(ss, __fmul_rn(v[q].y, v[q].y));
                ss = __fadd_rn(ss, __fmul_rn(v[q].z, v[q].z));
                ss = __fadd_rn(ss, __fmul_rn(v[q].w, v[q].w));
            }
        }
        for (; i < N; i++) ss = __fadd_rn(ss, __fmul_rn(row[i], row[i]));
    }
    ss = __shfl_sync(0xffffffffu, ss, 0);
    const float rs = __fdiv_rn(
        1.0f, __fsqrt_rn(__fadd_rn(__fdiv_rn(ss, (float)N), 1e-6f)));
    for (int i = lane; i < N; i += 32) {
        float g = __fadd_rn(1.0f, w ? bf16_f32(w[i]) : 0.0f);
        y[(size_t)t * N + i] = bf16_bits(__fmul_rn(__fmul_rn(row[i], rs), g));
    }
}

/* out = rnd(f32(a) + f32(b))  (c/layer.h:230-234) */
__global__ void __launch_bounds__(256)
resadd_kernel(const uint16_t *__restrict__ a, const uint16_t *__restrict__ b,
              uint16_t *__restrict__ out, size_t n) {
    for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < n;
         i += (size_t)gridDim.x * blockDim.x)
        out[i] = bf16_bits(__fadd_rn(bf16_f32(a[i]), bf16_f32(b[i])));
}

__global__ void __launch_bounds__(256)
synth_fill_kernel(uint16_t *__restrict__ dst, size_t n, uint64_t key,
                  uint64_t first, double sigma) {
    for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < n;
         i += (size_t)gridDim.x * blockDim.x)
        dst[i] = apus_synth_bf16(key, first + i, sigma);
}

}  // namespace apus
