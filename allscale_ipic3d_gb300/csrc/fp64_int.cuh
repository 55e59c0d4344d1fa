// Correctly rounded FP64 arithmetic on the integer pipe.
//
// GB300 issues one FP64 warp instruction per 64 cycles and SM sub-partition
// (measured: 64 for a DFMA, 76 for a DADD or DMUL), but a 32 x 32 -> 64-bit
// multiply-add per 3, a 32-bit shift per 2 and a logic or add per 1. The
// kernels that must round as the reference's host build does (FP64 dipole
// mover, tracer) are bound by that FP64 pipe alone, so the operations below
// run beside it, on significands: a product costs about 45 cycles, a sum of
// positive terms about 35, a^2.5 about 190 (about 1300 in double-double
// FP64), a quotient about 65 (about 700, the compiler's).
//
// Every function returns the IEEE round-to-nearest-even result of the exact
// value for regular operands; callers test with `regular` that operands are
// normal numbers whose results stay normal, and take the FP64 instructions
// otherwise. The functions are plain C++ (host and device): the host tests
// run them against the host's own FP64 arithmetic.
//
// Methods: school-book products with a rounded cut; long division by
// reciprocal estimates with an exact remainder (Brent & Zimmermann, Modern
// Computer Arithmetic, 1.4 and 3.4); Newton's iteration for the square root
// with exact residuals (same, 1.5 and 4.2.3).
#pragma once

#include <cmath>
#include <cstdint>
#include <cstring>

#ifdef __CUDACC__
#define IPG_HD __host__ __device__ __forceinline__
#else
#define IPG_HD inline
#endif

namespace ipg {
namespace soft {

// A regular number: (-1)^sign * m * 2^(e - 1075), 2^52 <= m <= 2^53 (a
// rounding may leave m = 2^53; `pack` carries it into the exponent, and the
// functions accept it as an operand). sign: the double's top bit in place.
struct Num {
    uint64_t m;
    int e;
    uint32_t sign;
};

// A double's bits. The move hides them from the compiler, which turns masks
// and zero tests of bits that it knows to be a double's back into FP64
// instructions (absolute value: an addition; x == 0: a comparison).
IPG_HD uint64_t bits_of(double x) {
#ifdef __CUDA_ARCH__
    uint64_t b;
    asm("mov.b64 %0, %1;" : "=l"(b) : "d"(x));
    return b;
#else
    uint64_t b;
    std::memcpy(&b, &x, 8);
    return b;
#endif
}
IPG_HD double from_bits(uint64_t b) {
#ifdef __CUDA_ARCH__
    return __longlong_as_double((long long)b);
#else
    double x;
    std::memcpy(&x, &b, 8);
    return x;
#endif
}

// biased exponent of x (0: zero or subnormal, 2047: infinity or NaN)
IPG_HD int exponent_of(double x) { return (int)((uint32_t)(bits_of(x) >> 52) & 0x7ff); }

// |x| in [2^-range, 2^(range + 1))
IPG_HD bool regular(double x, int range) {
    return (uint32_t)(exponent_of(x) - (1023 - range)) <= (uint32_t)(2 * range);
}

// An integer that orders doubles by their high words as their values do
// (negative ones below positive ones, NaN outside every finite value).
IPG_HD int32_t order_key_hi(double x) {
    const int32_t h = (int32_t)(uint32_t)(bits_of(x) >> 32);
    return h ^ ((h >> 31) & 0x7fffffff);
}

// The keys strictly between those of low and high, both finite: doubles of
// such a key lie within [low, high]. The keys of one box can be more than 2^31
// apart (any box around +-2): the differences are unsigned.
struct KeyBox {
    uint32_t first, count;
};
IPG_HD KeyBox key_box(double low, double high) {
    KeyBox b;
    const int64_t first = (int64_t)order_key_hi(low) + 1, count = order_key_hi(high) - first;
    b.first = (uint32_t)first;
    b.count = count > 0 ? (uint32_t)count : 0u;
    return b;
}
IPG_HD bool in_key_box(double x, const KeyBox& b) { return (uint32_t)order_key_hi(x) - b.first < b.count; }

IPG_HD Num unpack(double x) {
    const uint64_t b = bits_of(x);
    const uint32_t h = (uint32_t)(b >> 32);
    Num r;
    r.m = ((uint64_t)((h & 0xfffffu) | 0x100000u) << 32) | (uint32_t)b;
    r.e = (int)((h >> 20) & 0x7ff);
    r.sign = h & 0x80000000u;
    return r;
}

// e - 1 in the exponent field, plus m with its leading bit: m = 2^53 carries
IPG_HD double pack(const Num& a) {
    const uint64_t hi = (uint64_t)(a.sign + ((uint32_t)(a.e - 1) << 20)) << 32;
    return from_bits(hi + a.m);
}

// r + 1 if the fraction x / 2^32 (its last bit sticky) rounds up
IPG_HD uint64_t round_even(uint64_t r, uint32_t x) {
    const uint64_t t = (uint64_t)x + (0x7fffffffu + ((uint32_t)r & 1u));
    return r + (t >> 32);
}

// The product of two significands p = ma mb in [2^104, 2^106], rounded.
IPG_HD Num round_product(uint64_t hi, uint32_t w1, uint32_t w0, int e, uint32_t sign) {
    // hi = floor(p / 2^52); w1:w0 the rest, left-aligned
    uint32_t x = w1 | (w0 != 0);
    const bool big = (uint32_t)(hi >> 32) >= (1u << 21);
    uint64_t r = hi;
    if (big) {
        x = ((uint32_t)hi << 31) | (x >> 1) | (x & 1u);
        r = hi >> 1;
    }
    Num o;
    o.m = round_even(r, x);
    o.e = e + (big ? 1 : 0);
    o.sign = sign;
    return o;
}

IPG_HD Num mul(const Num& a, const Num& b) {
    const uint64_t A = a.m << 10, B = b.m << 2;
    const uint32_t a0 = (uint32_t)A, a1 = (uint32_t)(A >> 32), b0 = (uint32_t)B, b1 = (uint32_t)(B >> 32);
    const uint64_t p00 = (uint64_t)a0 * b0;
    const uint64_t p01 = (uint64_t)a0 * b1 + (p00 >> 32);
    const uint64_t p10 = (uint64_t)a1 * b0 + (uint32_t)p01;
    const uint64_t hi = (uint64_t)a1 * b1 + (p01 >> 32) + (p10 >> 32);
    return round_product(hi, (uint32_t)p10, (uint32_t)p00, a.e + b.e - 1023, a.sign ^ b.sign);
}

IPG_HD Num sqr(const Num& a) {
    // p 2^12 = (m 2^6)^2
    const uint64_t A = a.m << 6;
    const uint32_t a0 = (uint32_t)A, a1 = (uint32_t)(A >> 32);
    const uint64_t p00 = (uint64_t)a0 * a0;
    const uint64_t x = (uint64_t)a0 * a1;                        // the cross product, twice
    const uint64_t mid = (x << 1) + (p00 >> 32);                 // a1 < 2^28: x < 2^60
    const uint64_t hi = (uint64_t)a1 * a1 + (mid >> 32);
    return round_product(hi, (uint32_t)mid, (uint32_t)p00, 2 * a.e - 1023, 0);
}

// 3 a
IPG_HD Num triple(const Num& a) {
    const uint64_t p = 3 * a.m;  // [3 2^52, 3 2^53]
    const int sh = p >= (1ull << 54) ? 2 : 1;
    Num o;
    o.m = round_even(p >> sh, (uint32_t)p << (32 - sh));
    o.e = a.e + sh;
    o.sign = a.sign;
    return o;
}

// |a| + |b|
IPG_HD Num add_positive(const Num& a, const Num& b) {
    // with b.m = 2^53 the value may exceed a's although the exponent is
    // lower: the sum is symmetric, only the alignment follows the exponents
    const bool ge = a.e >= b.e;
    const uint64_t big = ge ? a.m : b.m;
    const uint64_t small = ge ? b.m : a.m;
    const int d = ge ? a.e - b.e : b.e - a.e;
    // 9 more bits, and what is shifted out of the smaller term as a sticky bit
    uint64_t s = 0;
    uint32_t sticky = 1;
    if (d < 64) {
        const uint64_t t = small << 9;
        s = t >> d;
        sticky = (s << d) != t;
    }
    const uint64_t sum = (big << 9) + s;  // [2^61, 2^63]
    const int sh = (uint32_t)(sum >> 32) >= (1u << 30) ? 10 : 9;
    Num o;
    o.m = round_even(sum >> sh, ((uint32_t)sum << (32 - sh)) | sticky);
    o.e = (ge ? a.e : b.e) + (sh - 9);
    o.sign = 0;
    return o;
}

// w = 2^k within a range where 1 / w is exact and normal
IPG_HD bool power_of_two(double w) { return regular(w, 900) && w > 0 && (bits_of(w) & 0xfffffffffffffull) == 0; }

// 0.0 + x: x, except that -0 becomes +0
IPG_HD double plus_zero(double x) { return bits_of(x) == 0x8000000000000000ull ? 0.0 : x; }

IPG_HD double fused(double a, double b, double c) {
#ifdef __CUDA_ARCH__
    return __fma_rn(a, b, c);
#else
    return std::fma(a, b, c);
#endif
}

// a / w in FP64 without the compiler's division (about 10 FP64 instructions
// and a branch): a product where 1 / w = inv is exact, else two corrections
// of a * inv by its residual -- the first brings it within a unit in the
// last place, the second, with an exact residual, rounds it correctly
// (Markstein, IBM J. R&D 34, 1990) -- and the division itself at the ends of
// the range.
IPG_HD double quotient(double a, double w, double inv, int exact) {
    if (exact) return a * inv;
    if (!regular(a, 900) || !regular(w, 100)) {
        if ((bits_of(a) << 1) == 0 && regular(w, 100)) return a * inv;  // a zero of a's and w's signs
        return a / w;
    }
    double q = a * inv;
    q = fused(fused(-w, q, a), inv, q);
    return fused(fused(-w, q, a), inv, q);
}

// 1 / d to an ulp from y with relative error e = 1 - d y below 2^-20: two terms
// of the geometric series 1 / d = y (1 + e + e^2 + ...), the third-order Newton
// iteration (Brent & Zimmermann, 4.2).
IPG_HD double refine_reciprocal(double d, double y) {
    const double e = fused(-d, y, 1.0);
    return fused(y, fused(e, e, e), y);
}

// FP32 estimates (relative error at most 2^-22 for the functions below)
IPG_HD float estimate_rcp(float x) {
#ifdef __CUDA_ARCH__
    float r;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
    return r;
#else
    extern float soft_host_rcp(float);
    return soft_host_rcp(x);
#endif
}
IPG_HD float estimate_rsqrt(float x) {
#ifdef __CUDA_ARCH__
    float r;
    asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
    return r;
#else
    extern float soft_host_rsqrt(float);
    return soft_host_rsqrt(x);
#endif
}
IPG_HD uint32_t float_bits(float x) {
#ifdef __CUDA_ARCH__
    return __float_as_uint(x);
#else
    uint32_t b;
    std::memcpy(&b, &x, 4);
    return b;
#endif
}
IPG_HD float float_from(uint32_t b) {
#ifdef __CUDA_ARCH__
    return __uint_as_float(b);
#else
    float x;
    std::memcpy(&x, &b, 4);
    return x;
#endif
}
IPG_HD uint32_t mul_hi(uint32_t a, uint32_t b) { return (uint32_t)(((uint64_t)a * b) >> 32); }

// A divisor with its reciprocal: R / 2^84 = 1 / D to 2^-31 relative.
struct Divisor {
    uint64_t D;  // [2^52, 2^53)
    int e;
    uint32_t sign, R;
};

IPG_HD Divisor divisor(const Num& a) {
    Divisor d;
    const int c = (int)(a.m >> 53);
    d.D = a.m >> c;
    d.e = a.e + c;
    d.sign = a.sign;
    const uint32_t d32 = (uint32_t)(d.D >> 21);
    // 1 / (D / 2^52) in (1/2, 1] from the significand's top 24 bits
    const float f = estimate_rcp(float_from((127u << 23) | ((d32 >> 8) & 0x7fffffu)));
    const uint32_t fb = float_bits(f);
    // r0 = f 2^32 - (0 or 1): f 2^32 reaches 2^32 for D = 2^52
    const uint64_t r64 = (uint64_t)((fb & 0x7fffffu) | 0x800000u) << ((fb >> 23) - 118);
    const uint32_t r0 = r64 > 0xffffffffull ? 0xffffffffu : (uint32_t)r64;
    // Newton: r0 + r0 (2^63 - d32 r0) / 2^63
    const int64_t err = (int64_t)((1ull << 63) - (uint64_t)d32 * r0);
    const int64_t r1 = (int64_t)r0 + (((int64_t)(int32_t)(err >> 11) * (int64_t)r0) >> 52);
    d.R = r1 > 0xffffffffll ? 0xffffffffu : (uint32_t)r1;
    return d;
}

// a / d
IPG_HD Num div(const Num& a, const Divisor& d) {
    const int c = (int)(a.m >> 53);
    const uint64_t N0 = a.m >> c;
    const bool less = N0 < d.D;
    const uint64_t N = N0 << (less ? 1 : 0);  // N / D in [1, 2)
    // q = floor(N 2^53 / D), 54 bits: q1 2^26 + q2, each estimated from R,
    // with exact remainders modulo 2^64. R is within 2^-31 relative, N >> 22
    // within 2^-30, so the estimate of q1 lies in (true - 1.4, true + 0.13];
    // one less leaves rem1 in (0.8 D, 2.4 D), and q2 in (true - 1.2, true +
    // 0.1]: the remainder is off by at most one D either way
    const uint32_t q1 = (mul_hi((uint32_t)(N >> 22), d.R) >> 3) - 1;
    const uint64_t rem1 = (N << 27) - (uint64_t)q1 * d.D;
    const uint32_t q2 = mul_hi((uint32_t)(rem1 >> 23), d.R) >> 3;
    uint64_t q = ((uint64_t)q1 << 26) + q2;
    int64_t rem = (int64_t)((rem1 << 26) - (uint64_t)q2 * d.D);
    if (rem < 0) {
        rem += (int64_t)d.D;
        --q;
    }
    if (rem >= (int64_t)d.D) {
        rem -= (int64_t)d.D;
        ++q;
    }
    Num o;
    o.m = round_even(q >> 1, ((uint32_t)q << 31) | (rem != 0));
    o.e = a.e + c - d.e + (less ? 1022 : 1023);
    o.sign = a.sign ^ d.sign;
    return o;
}

// a^2.5 for a > 0, correctly rounded where `sure` is set: the exact value is
// then further from a rounding boundary than the evaluation's error; unset
// for one argument in 2000 and for exact midpoints, which the caller
// evaluates in FP64.
//
// a = M 2^(2k), M in [1, 4): M^2.5 = M^2 sqrt(M). f = 1/sqrt(M) to 2^-22.3
// (the FP32 estimate's 2^-22.9, its argument cut to 24 bits); s1 = M f;
// s0 = s1 + (M - s1^2) f / 2, to 1.5 f's error squared = 2^-43.9; s = s0 +
// (M - s0^2) f / 2, to 2^-43.9 2^-22.3 = 2^-66.2; both residuals are exact,
// and so is the 128-bit M^2, whose product with s keeps 128 bits.
IPG_HD Num pow25(const Num& a, bool& sure) {
    const int c = (int)(a.m >> 53);
    const uint64_t m = a.m >> c;
    const int E = a.e + c - 1023;
    const int odd = E & 1, k = (E - odd) / 2;
    const uint64_t X = m << (10 + odd);  // M 2^62
    const float f = estimate_rsqrt(float_from(((uint32_t)(127 + odd) << 23) | ((uint32_t)(m >> 29) & 0x7fffffu)));
    const uint32_t fb = float_bits(f);
    const uint32_t F = ((fb & 0x7fffffu) | 0x800000u) << ((fb >> 23) - 119);  // f 2^31
    const uint32_t S1 = mul_hi((uint32_t)(X >> 32), F);                       // s1 2^29
    const int64_t e1 = (int64_t)((X >> 4) - (uint64_t)S1 * S1);               // (M - s1^2) 2^58
    // s0 2^48
    const uint64_t S0 = ((uint64_t)S1 << 19) + (uint64_t)(((int64_t)(int32_t)(e1 >> 9) * (int64_t)F) >> 33);
    // (M - s0^2) 2^96, small: exact modulo 2^64
    const uint32_t s0l = (uint32_t)S0, s0h = (uint32_t)(S0 >> 32);
    const uint64_t sq = (uint64_t)s0l * s0l + ((uint64_t)(2 * s0l * s0h) << 32);
    const int64_t e2 = (int64_t)((X << 34) - sq);
    const int64_t ds = ((int64_t)(int32_t)(e2 >> 26) * (int64_t)F) >> 23;  // 2^79
    const uint64_t S = (S0 << 15) + (uint64_t)(ds >> 16);                  // s 2^63
    const uint32_t Sl = (uint32_t)ds & 0xffffu;                            // and 16 bits more
    // M^2 2^124 = P1:P0
    const uint32_t x0 = (uint32_t)X, x1 = (uint32_t)(X >> 32);
    const uint64_t q00 = (uint64_t)x0 * x0, q01 = (uint64_t)x0 * x1, q11 = (uint64_t)x1 * x1;
    const uint64_t mid = q01 + (q00 >> 33);  // x0's low bits are zero: no carry out (x0 x1 + 2^31 < 2^64)
    const uint64_t P1 = q11 + (mid >> 31);
    const uint32_t P0h = (uint32_t)(mid << 1) | (uint32_t)((q00 >> 32) & 1);
    // Y = M^2.5 2^123 = P1 S + P0 S / 2^64 + P1 Sl / 2^16, 128 bits
    const uint32_t u0 = (uint32_t)P1, u1 = (uint32_t)(P1 >> 32), v0 = (uint32_t)S, v1 = (uint32_t)(S >> 32);
    const uint64_t y00 = (uint64_t)u0 * v0;
    const uint64_t y01 = (uint64_t)u0 * v1 + (y00 >> 32);
    const uint64_t y10 = (uint64_t)u1 * v0 + (uint32_t)y01;
    uint64_t Yh = (uint64_t)u1 * v1 + (y01 >> 32) + (y10 >> 32);
    uint64_t Yl = (y10 << 32) | (uint32_t)y00;
    const uint64_t more = (uint64_t)P0h * v1;        // P0 S / 2^64
    const uint64_t more2 = ((uint64_t)u1 * Sl) << 16;  // P1 Sl / 2^16 (u1 Sl < 2^48)
    uint64_t t = Yl + more;
    Yh += t < more;
    Yl = t + more2;
    Yh += Yl < more2;
    // Y in [2^123, 2^128): normalise
    const uint32_t top = (uint32_t)(Yh >> 32);
    int lz = top >= (1u << 31) ? 0 : top >= (1u << 30) ? 1 : top >= (1u << 29) ? 2 : top >= (1u << 28) ? 3 : 4;
    const uint64_t Z = (Yh << lz) | ((Yl >> 32) >> (32 - lz));
    // fraction of the significand's last place, in 2^-32: 11 bits of Z, 21 below
    const uint32_t x = ((uint32_t)Z << 21) | ((uint32_t)((Yl << lz) >> 32) >> 11);
    // the error, 2^-66 relative, is at most 2^-66 2^53 2^32 = 2^19 units of
    // x; 2^20 units on either side of the midpoint are left to the caller
    sure = (uint32_t)(x - 0x80000000u + (1u << 20)) > (1u << 21);
    Num o;
    o.m = (Z >> 11) + (x >> 31);
    o.e = 1027 - lz + 5 * k;
    o.sign = 0;
    return o;
}

}  // namespace soft
}  // namespace ipg
