/* ExactCodes against the rule it stands for, every code of x against weight ranges that include
 * subnormals, the largest values, infinities, NaN, none known (0) and none at all (inf, 0). */
#include <cstdio>
#include <cstring>
#include <initializer_list>

#include "exact_codes.h"

static float value(unsigned code) {
    const unsigned bits = code << 16;
    float f;
    memcpy(&f, &bits, 4);
    return f;
}
/* products_exact of exact_dense.cuh; lo: smallest nonzero |code| (0: there is none), hi: largest */
static bool exact(float wmin, float wmax, unsigned lo, unsigned hi) {
    return wmin > 0.0f &&
           (double)wmin * (double)value(lo ? lo : 0x7f80) >= 7.52316384526264e-37 &&
           (double)wmax * (double)value(hi) < 1.7e38;
}

int main() {
    const unsigned w[] = {0,      1,      2,      0x7f,   0x80,   0x81,   0x200,  0x380,  0x381,
                          0x382,  0x383,  0x384,  0x400,  0x1000, 0x2000, 0x3c00, 0x3f80, 0x4000,
                          0x7000, 0x7e00, 0x7f00, 0x7f7f, 0x7f80, 0x7fc0, 0x7fff};
    long n = 0, wrong = 0;
    for (unsigned a : w)
        for (unsigned b : w) {
            if (b < a && !(a == 0x7f80 && b == 0)) continue;
            const apus::ExactCodes codes(value(a), value(b));
            for (unsigned c = 0; c <= 0x7fff; c++)
                for (unsigned lo : {c, c ? 1 + c * 7919u % c : 0u, 0u}) {
                    if (lo == 0 && c != 0) continue;         /* a largest one is a nonzero one */
                    n++;
                    wrong += codes.hold(lo ? lo - 1 : 0xffffffffu, c) !=
                             exact(value(a), value(b), lo, c);
                }
        }
    printf("%ld ranges, %ld wrong\n", n, wrong);
    return wrong || n < 1000000;
}
