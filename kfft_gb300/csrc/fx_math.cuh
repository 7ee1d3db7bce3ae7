// fx_math.cuh -- 64-bit block fixed-point arithmetic of the double build's
// transform tiles.
//
// GB300 issues about 2 FP64 operations a clock and SM but 60 32x32+64-bit
// integer multiply-adds (mad.wide.s32) and 60 64-bit additions (measured:
// 0.60 T/s DFMA, 18.9 T/s mad.wide, 19.0 T/s add.s64), so the double build
// computes its butterflies in 64-bit integers: the values of one lane (one
// sub-FFT of a tile) share a power-of-two scale that follows the lane's
// largest value from stage to stage.  Inputs and outputs stay doubles.
//
// What is kept, in units of the lane's scale: an input's leading bit lies at 59
// for the lane's largest part (58 before a first stage of radix 5 to 8, 57
// before one of 9 to 16), and what falls below one unit is cut off; behind a
// chirp or an outer twiddle it lies at 61 (60, 59) and the product, a quarter of
// the true one, is whole units.  Later stages shift the lane's largest part up
// to 60 or 61 (less the radix's room) before their twiddles, whose products
// again are quarters in whole units.  Additions are exact.  So the largest part
// has 57 to 60 significant bits against the 53 of a double, and a smaller one
// as many fewer as it is smaller: the error is a few units whatever a value's
// size, below a double's in the norm of the lane but not for a part that
// nothing large is added to.  Lanes with such parts are found and left to
// arithmetic in doubles (fx_apart below).
//
// A real number x in [-1, 1] that multiplies data (a twiddle's part) is held
// as x * 2^62 in two signed 32-bit limbs, hi * 2^32 + lo with lo in
// (-2^31, 2^31), so that every partial product is one signed mad.wide.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

#include <type_traits>

#include "engine.cuh"

namespace kfft {

typedef long long fx_t;

struct cfx_t {
    fx_t x, y;
};

// ---------------------------------------------------------------------------
// cos and sin of 2 pi e / n to within a few 2^-62, in integers: exact octant
// reduction of e / n, then the Taylor series on [0, pi/4]
// ---------------------------------------------------------------------------
constexpr fx_t kFxOne = fx_t(1) << 62;
constexpr fx_t kFxQuarterPi = 0x3243F6A8885A308DLL;  // pi/4 * 2^62

__host__ __device__ constexpr fx_t fx_mul62(fx_t a, fx_t b) {
    return fx_t((static_cast<__int128>(a) * b + (static_cast<__int128>(1) << 61)) >> 62);
}

struct FxCosSin {
    fx_t c, s;
};

// angle u * pi/4, u in [0, 1] scaled by 2^62 (the first terms left out, x^21 / 21!
// and x^20 / 20!, are below 2^-68)
__host__ __device__ constexpr FxCosSin fx_taylor(fx_t u) {
    const fx_t x = fx_mul62(u, kFxQuarterPi);
    const fx_t x2 = fx_mul62(x, x);
    fx_t term = x, s = x;
    for (int k = 1; k < 10; ++k) {
        term = -(fx_mul62(term, x2) / fx_t((2 * k) * (2 * k + 1)));
        s += term;
    }
    term = kFxOne;
    fx_t c = kFxOne;
    for (int k = 1; k < 10; ++k) {
        term = -(fx_mul62(term, x2) / fx_t((2 * k - 1) * (2 * k)));
        c += term;
    }
    return {c, s};
}

// cos and sin of 2 pi e / n, 0 <= e < n < 2^33
__host__ __device__ constexpr FxCosSin fx_cossin(uint64_t e, uint64_t n) {
    const uint64_t t = (8 * e) / n;
    uint64_t r = 8 * e - t * n;  // the angle is (t + r / n) pi / 4
    if (t & 1) r = n - r;        // odd octants from their far end
    const uint64_t q1 = (r << 30) / n, r1 = (r << 30) % n;
    const uint64_t q2 = (r1 << 30) / n, r2 = (r1 << 30) % n;
    const uint64_t q3 = (r2 << 2) / n;
    const FxCosSin b = fx_taylor(fx_t((q1 << 32) + (q2 << 2) + q3));
    const uint64_t q = ((t + 1) / 2) & 3;  // quarter turns to add
    const fx_t c = b.c, s = (t & 1) ? -b.s : b.s;
    if (q == 0) return {c, s};
    if (q == 1) return {-s, c};
    if (q == 2) return {-c, -s};
    return {s, -c};
}

// ---------------------------------------------------------------------------
// parts that arithmetic in doubles keeps apart
// ---------------------------------------------------------------------------
// One scale a lane cuts off what lies far below the lane's largest part.  Where
// every part of every output takes in something near the largest, nothing is
// lost that doubles would keep: they round there too.  That is so as soon as
// one element has both parts near the largest, however it is rotated, and
// nearly every lane has one.  The others: values on an axis times twiddles on
// an axis stay on one, so large real inputs never reach the imaginary part of
// bin 0, and a single large real input at position 0 those of no bin at all.
// With all values real (or all imaginary) two large neighbours reach every part
// that is not zero; otherwise the lane stays in fixed point only if it holds
// nothing small, and the FP64 body takes it if it does.  (An impulse of 1.3 over
// noise of 2^-40, 4096 points: the imaginary parts were 3e-6 off, in FP64 2e-16.)

// headroom bits a radix-P butterfly needs beyond a factor 4
constexpr __host__ __device__ int fx_room(int P) { return P <= 4 ? 0 : (P <= 8 ? 1 : 2); }

// How many bits below the largest a part may lie and still count as near it:
// up to 7 it is held to its last bit (the leading bit at 59, 53 bits), less the
// room of the first radix.
__host__ __device__ constexpr int fx_span(int P) { return 7 - fx_room(P); }
// magnitude words (the high word of a double without its sign) from this one
// on are near the largest, `most`
__host__ __device__ constexpr uint32_t fx_near(uint32_t most, int span) {
    const int e = int(most >> 20) - span;
    return uint32_t(e > 1 ? e : 1) << 20;
}
// what a lane holds: nonzero real parts, nonzero imaginary ones, nonzero parts
// that are not near the largest, an element with both parts near it, two
// neighbours (the last and the first among them) with a part each near it
enum : uint32_t { FX_HAS_RE = 1, FX_HAS_IM = 2, FX_HAS_SMALL = 4, FX_BOTH = 8, FX_PAIR = 16 };
// all but the last for an element of magnitude words a and b, nonzero if re and im
__host__ __device__ constexpr uint32_t fx_holds(uint32_t a, uint32_t b, bool re, bool im, uint32_t near) {
    return (re ? uint32_t(FX_HAS_RE) : 0u) | (im ? uint32_t(FX_HAS_IM) : 0u) |
           ((re && a < near) || (im && b < near) ? uint32_t(FX_HAS_SMALL) : 0u) |
           (a >= near && b >= near ? uint32_t(FX_BOTH) : 0u);
}
// true when the lane needs the FP64 body
__host__ __device__ constexpr bool fx_apart(uint32_t holds) {
    const bool one_axis = (holds & (FX_HAS_RE | FX_HAS_IM)) != (FX_HAS_RE | FX_HAS_IM);
    return (holds & FX_HAS_SMALL) && !(holds & FX_BOTH) && !(one_axis && (holds & FX_PAIR));
}

// the two limbs of v, the low one never -2^31 (its negation has to fit)
__host__ __device__ constexpr int32_t fx_lo(fx_t v) {
    const int32_t l = int32_t(uint32_t(uint64_t(v)));
    return l == INT32_MIN ? l + 1 : l;
}
__host__ __device__ constexpr int32_t fx_hi(fx_t v) {
    const int32_t l = int32_t(uint32_t(uint64_t(v)));
    return int32_t((v - fx_t(l)) >> 32);
}

// cos or sin of 2 pi m / P as N + F / 2^64
constexpr fx_t fx_const62(long m, long P, bool want_sin) {
    m %= P;
    if (m < 0) m += P;
    const FxCosSin p = fx_cossin(uint64_t(m), uint64_t(P));
    const fx_t v = want_sin ? p.s : p.c, h = kFxOne / 2;
    // the halves, exactly
    if (v - h > -64 && v - h < 64) return h;
    if (v + h > -64 && v + h < 64) return -h;
    return v;
}
// v = N + F / 2^64 with F in [-2^63, 2^63)
constexpr int fx_const_n(fx_t v) { return v >= kFxOne / 2 ? 1 : (v < -(kFxOne / 2) ? -1 : 0); }
constexpr fx_t fx_const_f(fx_t v) { return (v - fx_t(fx_const_n(v)) * kFxOne) * 4; }

#if defined(__CUDACC__)
// ---------------------------------------------------------------------------
// products
// ---------------------------------------------------------------------------
__device__ __forceinline__ fx_t fx_mad(int32_t a, int32_t b, fx_t c) {
    fx_t r;
    asm("mad.wide.s32 %0, %1, %2, %3;" : "=l"(r) : "r"(a), "r"(b), "l"(c));
    return r;
}
__device__ __forceinline__ fx_t fx_mul(int32_t a, int32_t b) {
    fx_t r;
    asm("mul.wide.s32 %0, %1, %2;" : "=l"(r) : "r"(a), "r"(b));
    return r;
}
// the same with an immediate (a register copy of every constant would be
// hoisted out of the stage loop and spilled)
template <int32_t B>
__device__ __forceinline__ fx_t fx_madc(int32_t a, fx_t c) {
    fx_t r;
    asm("mad.wide.s32 %0, %1, %2, %3;" : "=l"(r) : "r"(a), "n"(B), "l"(c));
    return r;
}
template <int32_t B>
__device__ __forceinline__ fx_t fx_mulcc(int32_t a) {
    fx_t r;
    asm("mul.wide.s32 %0, %1, %2;" : "=l"(r) : "r"(a), "n"(B));
    return r;
}
// c + the high word of v, sign extended: one mad.wide by `one`, a 1 that the
// compiler does not know (PassDesc::fx_one; a known 1 becomes three
// instructions on the ALU pipe, the busiest one here)
__device__ __forceinline__ fx_t fx_add_high(fx_t v, fx_t c, int32_t one) {
    return fx_mad(int32_t(v >> 32), one, c);
}
// signed limbs of a value: v = h * 2^32 + l, l as a signed word
struct FxLimbs {
    int32_t h, l;
};
__device__ __forceinline__ FxLimbs fx_limbs(fx_t v) {
    FxLimbs r;
    r.l = int32_t(v);
    r.h = int32_t(v >> 32) + int32_t(uint32_t(r.l) >> 31);
    return r;
}

// a * w / 4 for a twiddle w (|w| <= 1), |a| <= 2^62.5
__device__ __forceinline__ cfx_t fx_cmul(cfx_t a, const FxTw& w, int32_t one) {
    const FxLimbs x = fx_limbs(a.x), y = fx_limbs(a.y);
    const int32_t nih = -w.ih, nil = -w.il;
    fx_t cr = fx_mul(x.h, w.rl);
    cr = fx_mad(x.l, w.rh, cr);
    cr = fx_mad(y.h, nil, cr);
    cr = fx_mad(y.l, nih, cr);
    fx_t ci = fx_mul(x.h, w.il);
    ci = fx_mad(x.l, w.ih, ci);
    ci = fx_mad(y.h, w.rl, ci);
    ci = fx_mad(y.l, w.rh, ci);
    cfx_t r;
    r.x = fx_add_high(cr, fx_mad(y.h, nih, fx_mul(x.h, w.rh)), one);
    r.y = fx_add_high(ci, fx_mad(y.h, w.rh, fx_mul(x.h, w.ih)), one);
    return r;
}

// the twiddle a * w of two twiddles
__device__ __forceinline__ FxTw fx_tw_mul(const FxTw& a, const FxTw& w, int32_t one) {
    const int32_t nih = -w.ih, nil = -w.il;
    fx_t cr = fx_mul(a.rh, w.rl);
    cr = fx_mad(a.rl, w.rh, cr);
    cr = fx_mad(a.ih, nil, cr);
    cr = fx_mad(a.il, nih, cr);
    fx_t ci = fx_mul(a.rh, w.il);
    ci = fx_mad(a.rl, w.ih, ci);
    ci = fx_mad(a.ih, w.rl, ci);
    ci = fx_mad(a.il, w.rh, ci);
    const fx_t re = fx_add_high(cr, fx_mad(a.ih, nih, fx_mul(a.rh, w.rh)), one) << 2;
    const fx_t im = fx_add_high(ci, fx_mad(a.ih, w.rh, fx_mul(a.rh, w.ih)), one) << 2;
    FxTw r;
    const FxLimbs p = fx_limbs(re), q = fx_limbs(im);
    r.rh = p.h;
    r.rl = p.l;
    r.ih = q.h;
    r.il = max(q.l, -INT32_MAX);
    return r;
}

// x times the constant N + F / 2^64 (|F| <= 2^63, N in -1, 0, 1), or with
// ACC that added to `acc`: exact to about one unit, no rescaling
template <int N, fx_t F, bool ACC = false>
__device__ __forceinline__ fx_t fx_mulc(fx_t x, FxLimbs l, int32_t one, fx_t acc = 0) {
    if (N == 1) acc = ACC ? acc + x : x;
    if (N == -1) acc = ACC ? acc - x : -x;
    if constexpr (F == 0) {
        return acc;
    } else if constexpr (F == INT64_MIN) {
        return acc - (x >> 1);
    } else {
        constexpr int32_t fl = fx_lo(F), fh = fx_hi(F);
        const fx_t cross = fx_madc<fh>(l.l, fx_mulcc<fl>(l.h));
        if constexpr (N == 0 && !ACC) acc = fx_mulcc<fh>(l.h);
        else acc = fx_madc<fh>(l.h, acc);
        return fx_add_high(cross, acc, one);
    }
}

// ---------------------------------------------------------------------------
// butterflies (forward; an inverse transform swaps the parts of its inputs
// and outputs).  Each grows a value's modulus by at most its radix.
// ---------------------------------------------------------------------------
__device__ __forceinline__ cfx_t fx_add(cfx_t a, cfx_t b) { return {a.x + b.x, a.y + b.y}; }
__device__ __forceinline__ cfx_t fx_sub(cfx_t a, cfx_t b) { return {a.x - b.x, a.y - b.y}; }

// a * W_P^E (W = exp(-2 pi i / P)), E modulo P
template <int P, int E>
__device__ __forceinline__ cfx_t fx_wmul(cfx_t a, int32_t one) {
    constexpr int e = ((E % P) + P) % P;
    if constexpr (e == 0) {
        return a;
    } else if constexpr ((4 * e) % P == 0) {
        constexpr int q = (4 * e) / P;
        if constexpr (q == 1) return cfx_t{a.y, -a.x};
        else if constexpr (q == 2) return cfx_t{-a.x, -a.y};
        else return cfx_t{-a.y, a.x};
    } else if constexpr ((8 * e) % P == 0) {
        // odd eighths: (+-1 -+ i) / sqrt 2
        constexpr fx_t r = fx_const62(1, 8, false);
        constexpr int rn = fx_const_n(r);
        constexpr fx_t rf = fx_const_f(r);
        const fx_t s = a.x + a.y, t = a.y - a.x;
        const fx_t p = fx_mulc<rn, rf>(s, fx_limbs(s), one), m = fx_mulc<rn, rf>(t, fx_limbs(t), one);
        constexpr int o = (8 * e) / P;
        if constexpr (o == 1) return cfx_t{p, m};
        else if constexpr (o == 3) return cfx_t{m, -p};
        else if constexpr (o == 5) return cfx_t{-p, -m};
        else return cfx_t{-m, p};
    } else {
        constexpr fx_t c = fx_const62(e, P, false), s = fx_const62(e, P, true);
        constexpr int cn = fx_const_n(c), sn = fx_const_n(s), nsn = fx_const_n(-s);
        constexpr fx_t cf = fx_const_f(c), sf = fx_const_f(s), nsf = fx_const_f(-s);
        const FxLimbs x = fx_limbs(a.x), y = fx_limbs(a.y);
        // (x + i y)(c - i s)
        return {fx_mulc<sn, sf, true>(a.y, y, one, fx_mulc<cn, cf>(a.x, x, one)),
                fx_mulc<nsn, nsf, true>(a.x, x, one, fx_mulc<cn, cf>(a.y, y, one))};
    }
}

__device__ __forceinline__ void fx_dft4(cfx_t& a0, cfx_t& a1, cfx_t& a2, cfx_t& a3) {
    const cfx_t s0 = fx_add(a0, a2), s1 = fx_sub(a0, a2);
    const cfx_t s2 = fx_add(a1, a3), d = fx_sub(a1, a3);
    a0 = fx_add(s0, s2);
    a2 = fx_sub(s0, s2);
    a1 = {s1.x + d.y, s1.y - d.x};
    a3 = {s1.x - d.y, s1.y + d.x};
}

template <int I, int N, class F>
__device__ __forceinline__ void fx_for(F&& f) {
    if constexpr (I < N) {
        f(std::integral_constant<int, I>{});
        fx_for<I + 1, N>(f);
    }
}

template <int P>
__device__ __forceinline__ void fx_dft_odd(cfx_t* v, int32_t one) {
    constexpr int H = (P - 1) / 2;
    cfx_t s[H], d[H];
    const cfx_t x0 = v[0];
    cfx_t sum = v[0];
#pragma unroll
    for (int n = 1; n <= H; ++n) {
        s[n - 1] = fx_add(v[n], v[P - n]);
        d[n - 1] = fx_sub(v[n], v[P - n]);
        sum = fx_add(sum, s[n - 1]);
    }
    fx_for<1, H + 1>([&](auto kc) {
        constexpr int K = decltype(kc)::value;
        cfx_t a = x0, b = {0, 0};
        fx_for<1, H + 1>([&](auto nc) {
            constexpr int n = decltype(nc)::value;
            constexpr fx_t c = fx_const62(long(n) * K, P, false), si = fx_const62(long(n) * K, P, true);
            constexpr int cn = fx_const_n(c), sn = fx_const_n(si);
            constexpr fx_t cf = fx_const_f(c), sf = fx_const_f(si);
            a.x = fx_mulc<cn, cf, true>(s[n - 1].x, fx_limbs(s[n - 1].x), one, a.x);
            a.y = fx_mulc<cn, cf, true>(s[n - 1].y, fx_limbs(s[n - 1].y), one, a.y);
            b.x = fx_mulc<sn, sf, true>(d[n - 1].x, fx_limbs(d[n - 1].x), one, b.x);
            b.y = fx_mulc<sn, sf, true>(d[n - 1].y, fx_limbs(d[n - 1].y), one, b.y);
        });
        v[K] = {a.x + b.y, a.y - b.x};      // a - i b
        v[P - K] = {a.x - b.y, a.y + b.x};  // a + i b
    });
    v[0] = sum;
}

constexpr int fx_gcd(int a, int b) { return b == 0 ? a : fx_gcd(b, a % b); }
constexpr int fx_modinv(int a, int m) {
    for (int x = 1; x < m; ++x)
        if ((a * x) % m == 1) return x;
    return 1 % m;
}

template <int P>
__device__ __forceinline__ void fx_dft(cfx_t* v, int32_t one);

// P = A * B: Good-Thomas for coprime factors, else Cooley-Tukey
template <int A, int B>
__device__ __forceinline__ void fx_dft_composite(cfx_t* v, int32_t one) {
    constexpr int P = A * B;
    constexpr bool kPfa = fx_gcd(A, B) == 1;
    cfx_t t[P];
    fx_for<0, B>([&](auto n2c) {
        constexpr int n2 = decltype(n2c)::value;
        cfx_t a[A];
        fx_for<0, A>([&](auto n1c) {
            constexpr int n1 = decltype(n1c)::value;
            a[n1] = v[kPfa ? (B * n1 + A * n2) % P : B * n1 + n2];
        });
        fx_dft<A>(a, one);
        fx_for<0, A>([&](auto k1c) {
            constexpr int k1 = decltype(k1c)::value;
            if constexpr (kPfa) t[n2 * A + k1] = a[k1];
            else t[n2 * A + k1] = fx_wmul<P, n2 * k1>(a[k1], one);
        });
    });
    fx_for<0, A>([&](auto k1c) {
        constexpr int k1 = decltype(k1c)::value;
        cfx_t b[B];
        fx_for<0, B>([&](auto n2c) {
            constexpr int n2 = decltype(n2c)::value;
            b[n2] = t[n2 * A + k1];
        });
        fx_dft<B>(b, one);
        fx_for<0, B>([&](auto k2c) {
            constexpr int k2 = decltype(k2c)::value;
            v[kPfa ? (B * fx_modinv(B % A, A) * k1 + A * fx_modinv(A % B, B) * k2) % P : k1 + A * k2] =
                b[k2];
        });
    });
}

template <int P>
__device__ __forceinline__ void fx_dft(cfx_t* v, int32_t one) {
    if constexpr (P == 2) {
        const cfx_t t = v[0];
        v[0] = fx_add(t, v[1]);
        v[1] = fx_sub(t, v[1]);
    } else if constexpr (P == 4) fx_dft4(v[0], v[1], v[2], v[3]);
    else if constexpr (P == 8) fx_dft_composite<2, 4>(v, one);
    else if constexpr (P == 16) fx_dft_composite<4, 4>(v, one);
    else if constexpr (P == 6) fx_dft_composite<2, 3>(v, one);
    else if constexpr (P == 9) fx_dft_composite<3, 3>(v, one);
    else if constexpr (P == 10) fx_dft_composite<2, 5>(v, one);
    else if constexpr (P == 12) fx_dft_composite<4, 3>(v, one);
    else if constexpr (P == 14) fx_dft_composite<2, 7>(v, one);
    else if constexpr (P == 15) fx_dft_composite<3, 5>(v, one);
    else fx_dft_odd<P>(v, one);
}

// ---------------------------------------------------------------------------
// doubles
// ---------------------------------------------------------------------------
// A finite d with exponent field at most `emax` as fixed point: exponent
// field emax has its leading bit at `top`.  (Subnormals read as numbers of
// about 2^-1022: the lane's emax is far above, they shift out.)
__device__ __forceinline__ fx_t fx_from_double(double d, int emax, int top) {
    const uint32_t hi = uint32_t(__double2hiint(d)), lo = uint32_t(__double2loint(d));
    const int e = int((hi >> 20) & 0x7ffu);
    // the significand, leading bit at 63
    const uint64_t m = (uint64_t(__funnelshift_l(lo, hi, 11) | 0x80000000u) << 32) | (lo << 11);
    fx_t v;  // (shr clamps: a shift of 64 or more leaves zero)
    asm("shr.u64 %0, %1, %2;" : "=l"(v) : "l"(m), "r"(emax + (63 - top) - e));
    const fx_t s = fx_t(int32_t(hi) >> 31);
    return (v ^ s) - s;
}

// v * 2^(eb - 1085) rounded to a double (|v| < 2^63; the result is normal or zero)
__device__ __forceinline__ double fx_to_double(fx_t v, int eb) {
    const uint32_t sgn = uint32_t(uint64_t(v) >> 32) & 0x80000000u;
    uint64_t a = uint64_t(v < 0 ? -v : v);
    if (uint32_t(a >> 32) == 0) {  // a value far below its lane's largest
        if (a == 0) return 0.0;
        if (uint32_t(a) >> 31) {  // keep the leading bit below 63
            a <<= 31;
            eb -= 31;
        } else {
            a <<= 32;
            eb -= 32;
        }
    }
    const int lz = __clz(int(uint32_t(a >> 32)));
    // the leading bit at 62, half a unit of the 53 bits added
    const uint64_t r = ((a << (lz - 1)) + 0x200u) >> 10;
    return __hiloint2double(int((uint32_t(r >> 32) + (uint32_t(eb - lz) << 20)) | sgn),
                            int(uint32_t(r)));
}
#endif

}  // namespace kfft
