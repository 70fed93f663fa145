// pp_exact64.cuh -- correctly rounded binary64 square root and quotients on
// the integer and FP32 pipes.
//
// GB300 issues a binary64 instruction of a warp once in 16 clocks per SM
// (measured: 1.99 FMA lanes/clk/SM; a correctly rounded division 0.23 and a
// square root 0.22 lanes/clk/SM, i.e. 140 clocks a warp).  The integer
// multiply-add runs at 62 lanes/clk/SM, additions and logic at 89, FP32 at
// 128.  So the roots and quotients of the step are formed here from an FP32
// approximation, exact integer residuals (64-bit arithmetic modulo 2^64: the
// residuals are small, so their low 64 bits determine them) and one exact
// comparison that settles the rounding.  The result is the IEEE
// round-to-nearest-even value, bit for bit; no operation of the binary64
// pipe is used.
//
// Everything is elementary: Newton's iteration for 1/sqrt and 1/x, schoolbook
// division with two 30-bit digits, and the midpoint tests
//   sqrt:     Y is right iff (Y - 1/2)^2 < N < (Y + 1/2)^2
//   quotient: Q is right iff |2 (N - Q D)| < D
// (neither can be an equality: the root of an integer is not a half-integer,
// and N 2^53 = (2 Q + 1) D has no solution with D < 2^53).
//
// The code also compiles for the host (seeds from 1/sqrtf and 1/x there), so
// the rounding is tested on the CPU as well.
#pragma once

#include <cstdint>
#include <cstring>

#ifdef __CUDACC__
#define PP_HD __host__ __device__ __forceinline__
#else
#include <cmath>
#define PP_HD inline
#endif

namespace pp {
namespace exact64 {

PP_HD uint32_t mulhi(uint32_t a, uint32_t b) {
#ifdef __CUDA_ARCH__
    return __umulhi(a, b);
#else
    return (uint32_t)(((uint64_t)a * b) >> 32);
#endif
}

PP_HD uint32_t float_bits(float x) {
#ifdef __CUDA_ARCH__
    return __float_as_uint(x);
#else
    uint32_t u;
    std::memcpy(&u, &x, 4);
    return u;
#endif
}

PP_HD float bits_float(uint32_t u) {
#ifdef __CUDA_ARCH__
    return __uint_as_float(u);
#else
    float x;
    std::memcpy(&x, &u, 4);
    return x;
#endif
}

PP_HD uint64_t double_bits(double x) {
#ifdef __CUDA_ARCH__
    return (uint64_t)__double_as_longlong(x);
#else
    uint64_t u;
    std::memcpy(&u, &x, 8);
    return u;
#endif
}

PP_HD double bits_double(uint64_t u) {
#ifdef __CUDA_ARCH__
    return __longlong_as_double((long long)u);
#else
    double x;
    std::memcpy(&x, &u, 8);
    return x;
#endif
}

// Seeds: relative error at most 2^-22.9 (sqrt) and 2^-22.9 (reciprocal).
#ifndef __CUDA_ARCH__
// the tests shift the host's seeds within the bound
inline float& seed_shift() {
    static float s = 0.0f;
    return s;
}
#endif

PP_HD float seed_rsqrt(float x) {
#ifdef __CUDA_ARCH__
    float y;
    asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
#else
    return (float)((1.0 / std::sqrt((double)x)) * (1.0 + (double)seed_shift()));
#endif
}

PP_HD float seed_rcp(float x) {
#ifdef __CUDA_ARCH__
    float y;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
#else
    return (float)((1.0 / (double)x) * (1.0 + (double)seed_shift()));
#endif
}

PP_HD float fma32(float a, float b, float c) {
#ifdef __CUDA_ARCH__
    return __fmaf_rn(a, b, c);
#else
    return std::fma(a, b, c);
#endif
}

// rint(x) for |x| < 2^22, given fma(.., .., kMagic) = x + 1.5 * 2^23.
constexpr float kMagic = 12582912.0f;
constexpr uint32_t kMagicBits = 0x4B400000u;
PP_HD int32_t magic_int(float m) { return (int32_t)(float_bits(m) - kMagicBits); }
// float(v) for |v| < 2^22, exactly.  (An integer-to-float conversion runs on
// GB300's binary64 pipe, 16 clocks a warp: four of them took a seventh of the
// fused step.)
PP_HD float small_float(int32_t v) { return bits_float(kMagicBits + (uint32_t)v) - kMagic; }

// The low 32 bits of v >> s (0 < s < 32).
PP_HD uint32_t shift_word(uint64_t v, int s) {
#ifdef __CUDA_ARCH__
    return __funnelshift_r((uint32_t)v, (uint32_t)(v >> 32), s);
#else
    return (uint32_t)(v >> s);
#endif
}

// A positive normal binary64 number m 2^(e - 1023 - 52): m its 53-bit
// significand, e its biased exponent.
struct Num {
    uint64_t m;
    int32_t e;
};

constexpr uint64_t kHidden = 1ull << 52;

PP_HD Num unpack(uint64_t bits) {
    const uint32_t hi = (uint32_t)(bits >> 32);
    const uint32_t mh = (hi & 0xFFFFFu) | 0x100000u;
    return Num{((uint64_t)mh << 32) | (uint32_t)bits, (int32_t)((hi >> 20) & 0x7FFu)};
}

// A divisor: significand, biased exponent and v = 2^32 2^52 / m, rounded
// down with an error below 3.6.
struct Divisor {
    uint64_t m;
    uint32_t v;
    int32_t e;
};

// v from the 53-bit significand m and an approximation r of 2^52 / m with a
// relative error of at most 2^-21.8.  One Newton step in integers:
// v1 = v0 + v0 (2^63 - v0 t) / 2^63 with t the leading 32 bits of m; the
// rounding of t, of the correction and the square of r's error leave
// v1 - 2^84/m in (-0.6, 2.6).
PP_HD uint32_t reciprocal_word(uint64_t m, float r) {
    r = r < 0.99999994f ? r : 0.99999994f;
    const uint32_t v0 = (float_bits(r) - 0x3E800000u) << 8;
    const uint32_t t = shift_word(m, 21);
    const uint64_t prod = (uint64_t)v0 * t;
    const int32_t n = (int32_t)shift_word(prod, 20);  // (prod - 2^63) >> 20
    const float c = fma32(small_float(n), r * -0x1p-11f, kMagic);
    return v0 + (uint32_t)magic_int(c) - 3u;
}

// sqrt of a positive normal number as a divisor of its own (its bits are
// pack(d)).  S = (mm 2^-52) 4^h with mm in [2^52, 2^54), Y = sqrt(mm 2^52).
PP_HD Divisor sqrt_rn(uint64_t bits) {
    const Num s = unpack(bits);
    const uint32_t odd = ~(uint32_t)s.e & 1u;  // odd unbiased exponent
    const uint64_t mm = s.m << odd;
    const float f = bits_float((shift_word(bits, 29) & 0x7FFFFFu) + (odd ? 0x40000000u : 0x3F800000u));
    const float r = seed_rsqrt(f);
    // g = sqrt(mm 2^-52) within 2^-21.9, as a 24-bit integer yh = g 2^23
    float g = f * r;
    g = g > 1.0f ? g : 1.0f;
    g = g < 1.99999988f ? g : 1.99999988f;
    const uint32_t yh = float_bits(g) - 0x3F000000u;
    // first residual mm - (8 yh)^2, |.| < 2^33.2; correction in 2^10 ulp, 3.2
    // of which are its error (2 from the dropped bits of the residual)
    const uint32_t y8 = yh << 3;
    const uint64_t r1 = mm - (uint64_t)y8 * y8;
    const int32_t p1 = (int32_t)shift_word(r1, 12);
    const int32_t t1 = magic_int(fma32(small_float(p1), r * 2.0f, kMagic));
    const uint64_t z = ((uint64_t)yh << 19) + (uint64_t)(int64_t)t1;
    // second residual mm 2^32 - z^2, |.| < 2^45.8; correction in ulp, then
    // |Y - sqrt| < 0.5 + 2^-8
    const uint64_t r2 = (mm << 32) - z * z;
    const int32_t p2 = (int32_t)shift_word(r2, 24);
    const int32_t t2 = magic_int(fma32(small_float(p2), r * 0x1p-9f, kMagic));
    uint64_t y = (z << 10) + (uint64_t)(int64_t)t2;
    // exact rounding: r3 = mm 2^52 - Y^2 must lie in (-Y, Y]
    const int64_t r3 = (int64_t)((mm << 52) - y * y);
    y += (uint64_t)(int64_t)(r3 > (int64_t)y) - (uint64_t)(int64_t)(r3 <= -(int64_t)y);
    return Divisor{y, reciprocal_word(y, r), (s.e + 1023 - (int32_t)odd) >> 1};
}

PP_HD Divisor divisor(uint64_t bits) {
    const Num d = unpack(bits);
    const float f = bits_float((shift_word(bits, 29) & 0x7FFFFFu) + 0x3F800000u);
    return Divisor{d.m, reciprocal_word(d.m, seed_rcp(f)), d.e};
}

PP_HD uint64_t pack(uint64_t m, int32_t e) {
    return m + ((uint64_t)(uint32_t)(e - 1) << 52);
}

// +0 or -0, from the two words: the compiler turns a test of the whole into
// a comparison on the binary64 pipe.
PP_HD bool is_zero(uint64_t bits) {
    uint32_t hi = (uint32_t)(bits >> 32) << 1, lo = (uint32_t)bits;
#ifdef __CUDA_ARCH__
    asm("" : "+r"(hi), "+r"(lo));
#endif
    return (hi | lo) == 0;
}

// Rounds hi 2^64 + lo (a product of two 53-bit significands, the first shifted
// up by 11: 2^115 .. 2^117) to 53 bits, ties to even; e is the product's
// exponent when hi >= 2^52.  A significand of 2^53 is left as it is: pack()
// carries it into the exponent.
PP_HD Num round_product(uint64_t hi, uint64_t lo, int32_t e) {
    const bool small = (uint32_t)(hi >> 52) == 0;
    const uint32_t l1 = (uint32_t)(lo >> 32), l0 = (uint32_t)lo;
    const uint64_t m = small ? (hi << 1) | (l1 >> 31) : hi;
    const uint32_t f1 = small ? (l1 << 1) | (l0 >> 31) : l1;
    const uint32_t f0 = small ? l0 << 1 : l0;
    const uint32_t f = f1 | (uint32_t)(f0 != 0);
    const uint32_t odd = (uint32_t)m & 1u;
    return Num{m + (uint64_t)(f > 0x80000000u - odd), e - (int32_t)small};
}

PP_HD uint64_t wide(uint32_t a, uint32_t b) { return (uint64_t)a * b; }

// a a, correctly rounded.
PP_HD Num square_rn(const Num& a) {
    const uint64_t s = a.m << 11;
    const uint32_t a1 = (uint32_t)(s >> 32), a0 = (uint32_t)s;
    const uint32_t b1 = (uint32_t)(a.m >> 32), b0 = (uint32_t)a.m;
    const uint64_t p0 = wide(a0, b0);
    const uint64_t p1 = wide(a1, b0) + (p0 >> 32);
    const uint64_t p2 = wide(a0, b1) + (uint32_t)p1;
    const uint64_t hi = wide(a1, b1) + (p1 >> 32) + (p2 >> 32);
    return round_product(hi, (p2 << 32) | (uint32_t)p0, 2 * a.e - 1022);
}

// Significand and biased exponent of (a.m 2^a.e) / d, correctly rounded.
PP_HD Num div_rn(const Num& a, const Divisor& d) {
    const bool lt = a.m < d.m;
    const uint64_t n = a.m + (lt ? a.m : 0ull);  // n / d.m in [1, 2)
    // first digit: q1 = n 2^30 / d.m - eps, 0 <= eps < 5.6
    const uint32_t q1 = mulhi(shift_word(n, 22), d.v);
    const uint64_t r1 = (n << 30) - (uint64_t)q1 * d.m;  // eps d.m < 2^56
    // second digit: (r1 / d.m) 2^28 within 4.6, in units of 2^-6 ulp
    const uint32_t q2 = (mulhi(shift_word(r1, 24), d.v) + 34u) >> 6;
    uint64_t q = ((uint64_t)q1 << 22) + q2;
    // exact rounding: |2 rem| < d.m
    const int64_t r2 = (int64_t)((r1 << 23) - ((uint64_t)q2 * d.m << 1));  // 2 rem
    q += (uint64_t)(int64_t)(r2 > (int64_t)d.m) - (uint64_t)(int64_t)(r2 < -(int64_t)d.m);
    return Num{q, a.e - d.e + 1023 - (int32_t)lt};
}

// a / d for a of either sign, zero included.  Neither NaN nor infinite; a
// nonzero a is normal, and so is the quotient (the caller checks).
PP_HD uint64_t div_bits(uint64_t a, const Divisor& d) {
    const Num q = div_rn(unpack(a), d);
    const uint64_t sign = a & 0x8000000000000000ull;
    const uint64_t bits = sign | pack(q.m, q.e);
    return is_zero(a) ? a : bits;
}

// bits of a a (+0 for a zero).  A nonzero a is within 2^+-500, so that the
// square is normal and its exponent stays inside its field: beyond, an infinity
// or a NaN among it, the result is some other finite number.
PP_HD uint64_t square_bits(uint64_t a) {
    const Num q = square_rn(unpack(a));
    return is_zero(a) ? 0 : pack(q.m, q.e);
}

PP_HD double div_signed(uint64_t a, const Divisor& d) { return bits_double(div_bits(a, d)); }

PP_HD int leading_zeros(uint64_t v) {
#ifdef __CUDA_ARCH__
    const uint32_t hi = (uint32_t)(v >> 32);
    return hi ? __clz(hi) : 32 + __clz((uint32_t)v);
#else
    return v ? __builtin_clzll(v) : 64;
#endif
}

// bits of a positive integer as a binary64 number.
PP_HD uint64_t int_bits(int v) {
    const int up = leading_zeros((uint64_t)(uint32_t)v) - 11;
    return ((uint64_t)(uint32_t)v << up) + ((uint64_t)(1023 + 51 - up) << 52);
}

// bits of (y - x) / x, both positive and normal.  False when the exponents
// differ by more than one or the difference takes more than 53 bits (its
// rounding is then the caller's): otherwise y - x is exact.
PP_HD bool relative_difference(const Divisor& y, const Divisor& x, uint64_t& bits) {
    const int32_t de = y.e - x.e;
    const int64_t diff = (int64_t)(y.m << (de > 0)) - (int64_t)(x.m << (de < 0));
    const uint64_t m = (uint64_t)(diff < 0 ? -diff : diff);
    const int up = leading_zeros(m) - 11;
    const Num q = div_rn(Num{m << (up & 63), (de > 0 ? x.e : y.e) - up}, x);
    bits = m == 0 ? 0 : ((uint64_t)diff & 0x8000000000000000ull) | pack(q.m, q.e);
    return (uint32_t)(de + 1) <= 2u && (m >> 53) == 0;
}

// Zero, or a number of either sign whose exponent field is at least lo.
PP_HD bool zero_or_above(uint64_t bits, uint32_t lo) {
    return ((uint32_t)(bits >> 32) << 1) >= (lo << 21) || is_zero(bits);
}

// Are the exponent fields of all three at most hi?  Neither an infinity nor a NaN
// is among them while hi is below 2047.
PP_HD bool all_below(uint64_t a, uint64_t b, uint64_t c, uint32_t hi) {
    const uint32_t x = (uint32_t)(a >> 32) << 1, y = (uint32_t)(b >> 32) << 1;
    const uint32_t z = (uint32_t)(c >> 32) << 1, xy = x > y ? x : y;
    return (xy > z ? xy : z) < ((hi + 1) << 21);
}

// Is `bits` a positive number of exponent field lo .. hi (0 < lo)?
PP_HD bool positive_in(uint64_t bits, uint32_t lo, uint32_t hi) {
    return (uint32_t)(bits >> 52) - lo <= hi - lo;
}

// Stretch and direction cosines of a bond, s = (y - xi) / xi and q = p / y with
// y = |p|.  Kept as bits: where two paths join, the compiler merges doubles with
// an instruction of the binary64 pipe each.
struct Stretch {
    uint64_t s, qx, qy, qz;
};

// The stretch of the bond with deformed vector p and reference length xi, without a
// binary64 operation for the root, the difference and the four quotients; op adds
// (and multiplies, without kIntSquares).  It takes lengths within 2^+-200 (squares
// 2^+-400) that differ by less than a factor of two, and components that are zero
// or within 2^-500 .. 2^201, so that no intermediate is subnormal or overflows;
// any(x, y, z, xi, r) fills r for everything else (NaN and infinities among it).
// The upper limit of the components has to be tested before kIntSquares squares
// them: the sum of wrapped squares can be in range.
//
// The fallback is called from here, not by the caller upon a flag: with the flag
// the plain kernel's rows of 128 slots took 2.32 ms a step instead of 2.09 (in 56
// registers instead of 64).
template <bool kIntSquares, class Ops, class Vec, class Any>
PP_HD Stretch stretch(const Ops& op, const Vec& p, double xi, Any any) {
    const uint64_t xb = double_bits(p.x), yb = double_bits(p.y), zb = double_bits(p.z);
    const uint64_t lb = double_bits(xi);
    Stretch r{0, 0, 0, 0};
    bool ok = positive_in(lb, 1023 - 200, 1023 + 200) && zero_or_above(xb, 1023 - 500) &&
              zero_or_above(yb, 1023 - 500) && zero_or_above(zb, 1023 - 500) &&
              all_below(xb, yb, zb, 1023 + 200);
    if (ok) {
        const double x2 = kIntSquares ? bits_double(square_bits(xb)) : op.mul(p.x, p.x);
        const double y2 = kIntSquares ? bits_double(square_bits(yb)) : op.mul(p.y, p.y);
        const double z2 = kIntSquares ? bits_double(square_bits(zb)) : op.mul(p.z, p.z);
        const uint64_t sb = double_bits(op.add(op.add(x2, y2), z2));
        ok = positive_in(sb, 1023 - 400, 1023 + 400);
        const Divisor len = sqrt_rn(sb);
        ok = relative_difference(len, divisor(lb), r.s) && ok;
        r.qx = div_bits(xb, len);
        r.qy = div_bits(yb, len);
        r.qz = div_bits(zb, len);
    }
    if (!ok) {
        Stretch t;
        any(p.x, p.y, p.z, xi, &t);
        r = t;
    }
    return r;
}

}  // namespace exact64
}  // namespace pp
