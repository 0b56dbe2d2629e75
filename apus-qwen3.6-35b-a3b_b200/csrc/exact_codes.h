/*
 * exact_codes.h — which BF16 codes make exact fp32 products with a given range of others.  Found
 * on the host, once per launch: the products that decide it, taken in every block of a tile, cost
 * 2 us of its 24.  Plain C++, so that a test without a GPU can go through all codes.
 */
#pragma once
#include <cmath>
#include <cstring>

#ifdef __CUDACC__
#define APUS_HD __host__ __device__ __forceinline__
#else
#define APUS_HD inline
#endif

namespace apus {

/* The magnitudes of one side with which products_exact (exact_dense.cuh) holds, given the
 * smallest nonzero and the largest magnitude wmin, wmax of the other: |code| - 1 from `below` (a
 * zero is the largest) and |code| up to `high`. */
struct ExactCodes {
    unsigned below;
    int high;                   /* -1: no product is known to be exact */
    ExactCodes() = default;
    ExactCodes(float wmin, float wmax) {
        const double lo = wmin, hi = wmax;
        auto value = [](int code) {
            float f;
            const unsigned bits = (unsigned)code << 16;
            memcpy(&f, &bits, 4);
            return (double)f;
        };
        auto first = [](auto holds) {               /* code in 1 .. 0x7f80 */
            int a = 1, b = 0x7f80;
            while (a < b) {
                const int mid = (a + b) / 2;
                if (holds(mid)) b = mid; else a = mid + 1;
            }
            return a;
        };
        below = (unsigned)first([&](int c) { return lo * value(c) >= 7.52316384526264e-37; }) - 1u;
        high = first([&](int c) { return !(hi * value(c) < 1.7e38); }) - 1;
        if (!(lo > 0.0) || !(hi < INFINITY)) high = -1;
    }
    APUS_HD bool hold(unsigned lo, unsigned hi) const {
        return lo >= below && (int)hi <= high;
    }
};

}  // namespace apus
