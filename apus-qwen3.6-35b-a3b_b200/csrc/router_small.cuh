/*
 * router_small.cuh — the router for few tokens of the multi-kernel paths: every logit's
 * exact chain, latency first (c/moe.h:321-371).
 */
#pragma once
#include "common.cuh"
#include "decode_gemv.cuh"
#include "router.cuh"
#include "router_select.cuh"

namespace apus {

/*
 * Latency path for few tokens.  grid = (ceil(rows / ROWS), ceil(T / 4)), block
 * = 128: a CTA pulls ROWS router rows into shared memory with one bulk copy
 * each (all in flight at once, so the 1 MiB router matrix arrives spread over
 * many SMs instead of trickling through one) and stages four tokens as fp32;
 * the lanes of ROWS/8 warps walk one exact chain each (lane = row * 4 + token),
 * and the BF16 logits go to global memory.  ROWS is 8 while all CTAs are resident at
 * once, three to an SM (up to 52 tokens here), and 16 above, two to an SM: a second
 * wave costs a whole chain (61 tokens: 31 -> 24 us).  The CTA that arrives last for a
 * token (one atomic counter per token, which it resets for the next call) runs
 * that token's softmax / top-k on one of its warps.  No CTA ever waits on
 * another.  It decides on the BF16 codes of the logits and only where code order may
 * not decide, or a weight might narrow differently, runs the engine's softmax
 * (router_select.cuh; softmax for all took 2 us more).  Requires K % 8 == 0 and a
 * 16-byte-aligned router matrix.
 * Dynamic shared memory: ROWS * (K*2 + 16) + 4 * ((K + 4) + (E + 1)) * 4 bytes.
 */
constexpr int ROUTER_SMALL_TOK = 4;
constexpr int ROUTER_SMALL_THREADS = 128;

inline size_t router_small_smem(int E, int K, int rows) {
    return (size_t)rows * (K * 2 + 16) + (size_t)ROUTER_SMALL_TOK * (K + 4) * 4 +
           (size_t)ROUTER_SMALL_TOK * (E + 1) * 4;
}

template <int ROUTER_SMALL_ROWS>
__global__ void __launch_bounds__(ROUTER_SMALL_THREADS)
router_small_kernel(const uint16_t *__restrict__ x,
                    const uint16_t *__restrict__ wr, int T, int E, int K,
                    int topk, float wmin, float wmin_extra,
                    int32_t *__restrict__ idx_out,
                    uint16_t *__restrict__ w_out,
                    uint16_t *__restrict__ logits_out,
                    const uint16_t *__restrict__ extra_row,
                    uint16_t *__restrict__ extra_out,
                    float *__restrict__ logits_ws,     /* [T][E] fp32 */
                    unsigned int *__restrict__ counters, /* [T], zero between calls */
                    int *status) {
    /* the next kernel may be scheduled; the wait for the previous one comes
     * after the router rows (constants) have been requested */
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    extern __shared__ __align__(128) unsigned char smem_raw[];
    const int pitch = K * 2 + 16;                 /* bytes; de-conflicts banks */
    const int xpitch = K + 4;                     /* floats; likewise for the tokens */
    unsigned char *rows_s = smem_raw;
    float *xs = reinterpret_cast<float *>(smem_raw + ROUTER_SMALL_ROWS * pitch);
    uint32_t *codes = reinterpret_cast<uint32_t *>(xs + (size_t)ROUTER_SMALL_TOK * xpitch);
    __shared__ __align__(8) uint64_t bar;
    __shared__ unsigned int s_xmin;
    __shared__ int s_last[ROUTER_SMALL_TOK];
    __shared__ int s_sel[ROUTER_SMALL_TOK][32];

    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int t0 = blockIdx.y * ROUTER_SMALL_TOK;
    const int nt = min(ROUTER_SMALL_TOK, T - t0);
    const int rows_total = E + (extra_row ? 1 : 0);
    const int r0 = blockIdx.x * ROUTER_SMALL_ROWS;
    const int nrows = min(ROUTER_SMALL_ROWS, rows_total - r0);

    if (tid == 0) {
        mbar_init(&bar, 1);
        mbar_fence_init();
        s_xmin = 0x7f800000u;
        mbar_expect_tx(&bar, (uint32_t)nrows * (uint32_t)K * 2u);
        for (int r = 0; r < nrows; r++) {
            const uint16_t *src = (r0 + r == E) ? extra_row
                                                : wr + (size_t)(r0 + r) * K;
            bulk_g2s(rows_s + (size_t)r * pitch, src, (uint32_t)K * 2u, &bar);
        }
    }
    if (tid < ROUTER_SMALL_TOK) s_last[tid] = 0;
    asm volatile("griddepcontrol.wait;" ::: "memory");   /* the tokens may be its output */
    __syncthreads();
    unsigned int xmin = 0x7f800000u;
    const int c8 = K / 8;
    for (int c = tid; c < nt * c8; c += ROUTER_SMALL_THREADS) {
        const int tt = c / c8, cc = c - tt * c8;
        const uint4 v = ldg16(x + (size_t)(t0 + tt) * K + (size_t)cc * 8);
        const uint32_t wds[4] = {v.x, v.y, v.z, v.w};
        float4 *d = reinterpret_cast<float4 *>(xs + (size_t)tt * xpitch + cc * 8);
        d[0] = make_float4(bf16lo(v.x), bf16hi(v.x), bf16lo(v.y), bf16hi(v.y));
        d[1] = make_float4(bf16lo(v.z), bf16hi(v.z), bf16lo(v.w), bf16hi(v.w));
#pragma unroll
        for (int q = 0; q < 4; q++) {
            unsigned int a = (wds[q] << 16) & 0x7fffffffu;
            unsigned int b = wds[q] & 0x7fff0000u;
            if (a != 0 && a < xmin) xmin = a;
            if (b != 0 && b < xmin) xmin = b;
        }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1)
        xmin = min(xmin, __shfl_xor_sync(0xffffffffu, xmin, o));
    if (lane == 0) atomicMin(&s_xmin, xmin);
    __syncthreads();
    constexpr int CHAIN_WARPS = ROUTER_SMALL_ROWS / 8;
    if (warp < CHAIN_WARPS) {
        const double xmn = (double)__uint_as_float(s_xmin);
        const bool use_fma = (wmin > 0.0f) && ((double)wmin * xmn >= 7.52316384526264e-37);
        const bool use_fma_x =
            (wmin_extra > 0.0f) && ((double)wmin_extra * xmn >= 7.52316384526264e-37);
        const bool arrived = mbar_wait(&bar, 0);
        if (!arrived) set_status(status, ST_MBAR_TIMEOUT);
        const int r = warp * 8 + (lane >> 2), tt = lane & 3;
        if (arrived && r < nrows && tt < nt) {
            const uint16_t *wrow =
                reinterpret_cast<const uint16_t *>(rows_s + (size_t)r * pitch);
            const float *xr = xs + (size_t)tt * xpitch;
            const bool fma_row = (r0 + r != E) ? use_fma : use_fma_x;
            const float acc = fma_row ? small_chain<true>(wrow, xr, K)
                                      : small_chain<false>(wrow, xr, K);
            const uint16_t code = bf16_bits(acc);
            const int t = t0 + tt;
            if (r0 + r == E) {
                extra_out[t] = code;
            } else {
                logits_ws[(size_t)t * E + r0 + r] = bf16_f32(code);
                if (logits_out) logits_out[(size_t)t * E + r0 + r] = code;
            }
        }
        /* the last CTA of a token finishes that token */
        __threadfence();
        __syncwarp();
        if (lane < nt &&
            atomicAdd(&counters[t0 + lane], 1u) == gridDim.x * CHAIN_WARPS - 1)
            s_last[lane] = 1;
    }
    __syncthreads();
    for (int tt = warp; tt < nt; tt += ROUTER_SMALL_THREADS / 32) {
        if (!s_last[tt]) continue;
        const int t = t0 + tt;
        uint32_t *cd = codes + (size_t)tt * (E + 1);
        __threadfence();
        bool nan = false;
        for (int e = lane; e < E; e += 32) {
            const uint32_t c = __float_as_uint(__ldcg(&logits_ws[(size_t)t * E + e])) >> 16;
            nan |= (c & 0x7fffu) > 0x7f80u;
            cd[e] = c * 0x10001u;
        }
        if (lane == 0) {
            cd[E] = CODE_NEVER;
            counters[t] = 0;
        }
        __syncwarp();
        int32_t *idx = idx_out + (size_t)t * topk;
        uint16_t *wo = w_out ? w_out + (size_t)t * topk : nullptr;
        const Choice c = rt_select(cd, E, topk, lane, s_sel[tt]);
        if (c.odd || __any_sync(0xffffffffu, nan) ||
            (rt_weights(cd, s_sel[tt], topk, lane, idx, wo) && wo)) {
            __syncwarp();
            float *p = reinterpret_cast<float *>(cd);
            for (int e = lane; e < E; e += 32) p[e] = bf16lo(cd[e]);
            __syncwarp();
            router_softmax_topk(p, E, topk, lane, idx, wo);
        }
    }
}

}  // namespace apus
