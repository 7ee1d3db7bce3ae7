// Checks, for the CPU test tests/test_fx_rule_host.py, the rule by which a lane
// stays in fixed point (fx_math.cuh): random lanes of zeros, tiny and large
// parts in many arrangements; in every lane that stays, each part of each
// output takes in an input part near the largest, or nothing at all.
#include "fx_math.cuh"

#include <cmath>
#include <cstdio>
#include <cstring>
#include <random>
#include <vector>

using namespace kfft;

static uint32_t mag(double v) {
    uint64_t u;
    std::memcpy(&u, &v, 8);
    return uint32_t(u >> 32) & 0x7fffffffu;
}

int main() {
    std::mt19937_64 rng(1);
    auto uni = [&] { return double(rng() >> 11) * 0x1p-53; };
    const int lengths[] = {3, 5, 6, 7, 8, 9, 10, 12, 15, 16, 20, 24, 32, 48, 64};
    const double kPi = 3.14159265358979323846;
    long stay = 0, leave = 0, wrong = 0, exact_lost = 0;
    for (int trial = 0; trial < 40000; ++trial) {
        const int n = lengths[rng() % 15], mode = int(rng() % 5), step = 2 + int(rng() % 7);
        const double p0 = uni(), p1 = uni() * (1 - p0);
        auto part = [&] {
            const double u = uni(), s = (rng() & 1) ? 1.0 : -1.0;
            return u < p0 ? 0.0 : s * (0.5 + 0.5 * uni()) * (u < p0 + p1 ? 1e-6 : 1.0);
        };
        std::vector<double> re(n), im(n);
        const int off = int(rng() % step);
        for (int i = 0; i < n; ++i) {
            re[i] = part();
            im[i] = mode == 0 ? 0.0 : part();
            if (mode == 1) im[i] *= 1e-7;                          // nearly real
            if (mode == 2 && uni() < 0.7) re[i] = im[i] = 0;       // few values
            if (mode == 3 && i % step != off) re[i] *= 1e-6, im[i] *= 1e-6;  // a comb over tiny ones
            if (mode == 4 && i != off) re[i] *= 1e-9, im[i] *= 1e-9;         // one value
        }
        uint32_t most = 0, holds = 0;
        for (int i = 0; i < n; ++i) most = std::max(most, std::max(mag(re[i]), mag(im[i])));
        if (!most) continue;
        const int span = fx_span(n % 16 == 0 ? 4 : 16);
        const uint32_t near = fx_near(most, span);
        for (int i = 0; i < n; ++i) {
            const int k = (i + 1) % n;
            holds |= fx_holds(mag(re[i]), mag(im[i]), re[i] != 0, im[i] != 0, near);
            if (std::max(mag(re[i]), mag(im[i])) >= near && std::max(mag(re[k]), mag(im[k])) >= near) holds |= FX_PAIR;
        }
        if (fx_apart(holds)) {
            ++leave;
            continue;
        }
        ++stay;
        double top = 0;
        for (int i = 0; i < n; ++i) top = std::max(top, std::max(std::fabs(re[i]), std::fabs(im[i])));
        const double low = std::ldexp(top, -span - 8);  // a term near the largest, at any angle but an axis
        for (int k = 0; k < n; ++k) {
            double tr = 0, ti = 0;
            for (int i = 0; i < n; ++i) {
                const int e = k * i % n;
                const double c = 4 * e == n || 4 * e == 3 * n ? 0 : std::cos(2 * kPi * e / n);
                const double s = e == 0 || 2 * e == n ? 0 : std::sin(2 * kPi * e / n);
                tr = std::max(tr, std::max(std::fabs(re[i] * c), std::fabs(im[i] * s)));
                ti = std::max(ti, std::max(std::fabs(im[i] * c), std::fabs(re[i] * s)));
            }
            if ((tr > 0 && tr < low) || (ti > 0 && ti < low)) {
                ++wrong;
                break;
            }
        }
    }
    // a part within the span of the largest keeps all its 53 bits
    for (int P = 2; P <= 16; ++P)
        if (59 - fx_room(P) - fx_span(P) < 52) ++exact_lost;
    std::printf("%ld %ld %ld %ld\n", stay, leave, wrong, exact_lost);
    return 0;
}
