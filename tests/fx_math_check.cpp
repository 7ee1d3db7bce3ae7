// Prints the host side of the fixed-point arithmetic (fx_math.cuh) for the CPU
// test tests/test_fx_math_host.py: cosines and sines against long double, the
// two-limb form of values, and the split of constants.
#include "fx_math.cuh"

#include <cmath>
#include <cstdio>

using namespace kfft;

int main() {
    const uint64_t ns[] = {1, 2, 3, 4, 7, 8, 12, 16, 360, 4096, 59049, 1000003, 8589934591ull};
    for (uint64_t n : ns) {
        long double worst = 0;
        for (uint64_t i = 0; i < 4000; ++i) {
            const uint64_t e = n <= 4000 ? i % n : (i * 2654435761ull + i) % n;
            const FxCosSin v = fx_cossin(e, n);
            const long double a = 2 * acosl(-1.0L) * (long double)e / n;
            worst = fmaxl(worst, fabsl(cosl(a) * kFxOne - v.c));
            worst = fmaxl(worst, fabsl(sinl(a) * kFxOne - v.s));
        }
        std::printf("cossin %llu %.3Lf\n", (unsigned long long)n, worst);
    }
    // limbs: h * 2^32 + l is the value, or one unit beside it where l would be -2^31
    long long off = 0;
    uint64_t x = 88172645463325252ull;
    for (int i = 0; i < 100000; ++i) {
        x ^= x << 13, x ^= x >> 7, x ^= x << 17;
        const fx_t v = i % 3 == 0 ? fx_t(x >> 2) - (fx_t(1) << 61) : (fx_t(x >> 34) << 32) + fx_t(INT32_MIN) * (i % 2);
        const fx_t back = fx_t(fx_hi(v)) * (fx_t(1) << 32) + fx_lo(v);
        if (fx_lo(v) == INT32_MIN) off = 1 << 20;
        off = std::max<long long>(off, std::llabs(back - v));
    }
    std::printf("limbs %lld\n", off);
    // constants: n + f / 2^64, the halves exact
    for (long P : {3l, 5l, 6l, 7l, 8l, 9l, 11l, 12l, 13l, 16l})
        for (long m = 0; m < P; ++m)
            for (bool s : {false, true}) {
                const fx_t c = fx_const62(m, P, s);
                const long double a = 2 * acosl(-1.0L) * m / P;
                const long double v = fx_const_n(c) + (long double)fx_const_f(c) / 18446744073709551616.0L;
                std::printf("const %ld %ld %d %.3Lf\n", P, m, int(s), fabsl((s ? sinl(a) : cosl(a)) - v) * kFxOne);
            }
    std::printf("half %d %lld %d %lld\n", fx_const_n(fx_const62(1, 6, false)),
                (long long)fx_const_f(fx_const62(1, 6, false)), fx_const_n(fx_const62(1, 3, false)),
                (long long)fx_const_f(fx_const62(1, 3, false)));
    return 0;
}
