// Exact FP64 helpers that run on the integer pipes.
//
// GB300 executes FP64 arithmetic, FP64 compares (DSETP) and float<->double
// conversions (F2F) on one narrow FP64 pipe: about 2 lanes per clock per SM,
// against 128 for 32-bit integer and FP32 work.  The step kernels are bound by
// that pipe, so every FP64-pipe instruction whose result can be formed exactly
// from the bit pattern moves here.  Each function returns bit-for-bit what the
// FP64 instruction it replaces returns, for every input (zeros, subnormals,
// infinities and NaNs included: the rare cases fall back to that
// instruction).  The functions compile for the host as well, where
// tests/fp64_int_check.cpp compares them with the host's IEEE arithmetic.
#pragma once
#include <cstdint>
#include <cstring>

#if defined(__CUDACC__)
#define GVX_FP64I __host__ __device__ __forceinline__
#else
#define GVX_FP64I static inline
#endif

namespace gvx {
namespace fp64i {

// On the device the bit pattern moves through an opaque register move, so that the
// compiler cannot fold the integer tests below back into FP64 compares.
GVX_FP64I uint64_t bits(double x) {
#ifdef __CUDA_ARCH__
    uint64_t u;
    asm("mov.b64 %0, %1;" : "=l"(u) : "d"(x));
    return u;
#else
    uint64_t u; std::memcpy(&u, &x, 8); return u;
#endif
}
GVX_FP64I double from_bits(uint64_t u) {
#ifdef __CUDA_ARCH__
    double x;
    asm("mov.b64 %0, %1;" : "=d"(x) : "l"(u));
    return x;
#else
    double x; std::memcpy(&x, &u, 8); return x;
#endif
}
// The FP64 instructions of the rare cases, in a form the compiler does not move out
// of their branch (a speculated copy would run on the FP64 pipe for every call).
GVX_FP64I double rare_mul(double a, double b) {
#ifdef __CUDA_ARCH__
    double r;
    asm volatile("mul.rn.f64 %0, %1, %2;" : "=d"(r) : "d"(a), "d"(b));
    return r;
#else
    return a * b;
#endif
}
GVX_FP64I double rare_f2d(float f) {
#ifdef __CUDA_ARCH__
    double r;
    asm volatile("cvt.f64.f32 %0, %1;" : "=d"(r) : "f"(f));
    return r;
#else
    return (double)f;
#endif
}
GVX_FP64I float rare_d2f(double x) {
#ifdef __CUDA_ARCH__
    float r;
    asm volatile("cvt.rn.f32.f64 %0, %1;" : "=f"(r) : "d"(x));
    return r;
#else
    return (float)x;
#endif
}
GVX_FP64I uint32_t fbits(float x) {
#ifdef __CUDA_ARCH__
    return __float_as_uint(x);
#else
    uint32_t u; std::memcpy(&u, &x, 4); return u;
#endif
}
GVX_FP64I float from_fbits(uint32_t u) {
#ifdef __CUDA_ARCH__
    return __uint_as_float(u);
#else
    float x; std::memcpy(&x, &u, 4); return x;
#endif
}

constexpr uint64_t kSign = 0x8000000000000000ull, kAbs = 0x7FFFFFFFFFFFFFFFull;
constexpr uint64_t kFrac = 0x000FFFFFFFFFFFFFull, kInf = 0x7FF0000000000000ull;

// x * 2 (exponent + 1 for normal x that stays finite; subnormals shift left)
GVX_FP64I double mul2(double x) {
    const uint64_t b = bits(x);
    const uint32_t e = (uint32_t)(b >> 52) & 0x7FFu;
    if (e - 1u < 0x7FDu) return from_bits(b + (1ull << 52));
    if (e == 0u) return from_bits((b & kSign) | ((b & kAbs) << 1));
    return rare_mul(x, 2.0);
}
// x * 0.5 (exponent - 1 while the result stays normal; +-0 unchanged)
GVX_FP64I double half(double x) {
    const uint64_t b = bits(x);
    const uint32_t e = (uint32_t)(b >> 52) & 0x7FFu;
    if (e - 2u < 0x7FDu) return from_bits(b - (1ull << 52));
    if ((b & kAbs) == 0) return x;
    return rare_mul(x, 0.5);
}

// (double)f: exact; normal floats and zeros on the integer pipes
GVX_FP64I double f2d(float f) {
    const uint32_t u = fbits(f);
    const uint32_t e = (u >> 23) & 0xFFu;
    if (e - 1u >= 254u) {
        if ((u & 0x7FFFFFFFu) == 0) return from_bits((uint64_t)u << 32);
        return rare_f2d(f);
    }
    const uint32_t hi = (u & 0x80000000u) | (((u & 0x7FFFFFFFu) >> 3) + (896u << 20));
    return from_bits(((uint64_t)hi << 32) | (((uint64_t)u << 29) & 0xFFFFFFFFull));
}
// (float)x, round to nearest even; results that are normal floats, and zeros, on the integer pipes
GVX_FP64I float d2f(double x) {
    const uint64_t u = bits(x);
    const uint32_t e = (uint32_t)(u >> 52) & 0x7FFu;
    if (e - 897u >= 254u) {
        if ((u & kAbs) == 0) return from_fbits((uint32_t)(u >> 32));
        return rare_d2f(x);
    }
    uint32_t m = (uint32_t)((u & kFrac) >> 29);
    const uint32_t rest = (uint32_t)u & 0x1FFFFFFFu;
    m += (uint32_t)((rest > 0x10000000u) | ((rest == 0x10000000u) & (m & 1u)));
    return from_fbits(((uint32_t)(u >> 32) & 0x80000000u) + ((e - 896u) << 23) + m);
}

// Ordered comparisons with IEEE semantics: false when either operand is NaN, -0 == +0.
GVX_FP64I int64_t order_key(uint64_t u) { return (int64_t)u >= 0 ? (int64_t)u : (int64_t)(kSign - u); }
GVX_FP64I bool is_nan_bits(uint64_t u) { return (u & kAbs) > kInf; }
GVX_FP64I bool lt(double a, double b) {
    const uint64_t ua = bits(a), ub = bits(b);
    return !(is_nan_bits(ua) | is_nan_bits(ub)) & (order_key(ua) < order_key(ub));
}
GVX_FP64I bool gt(double a, double b) { return lt(b, a); }
GVX_FP64I bool le(double a, double b) {
    const uint64_t ua = bits(a), ub = bits(b);
    return !(is_nan_bits(ua) | is_nan_bits(ub)) & (order_key(ua) <= order_key(ub));
}
GVX_FP64I bool ge(double a, double b) { return le(b, a); }
// x > 0 and x >= 0 (false for NaN and for -0 in the strict form)
GVX_FP64I bool gt0(double x) { const int64_t b = (int64_t)bits(x); return b > 0 && (uint64_t)b <= kInf; }
GVX_FP64I bool ge0(double x) { const uint64_t b = bits(x); return (b == kSign) | ((int64_t)b >= 0 && b <= kInf); }
// x == 0 (either sign)
GVX_FP64I bool eq0(double x) { return (bits(x) & kAbs) == 0; }

// x + 0.0 with x possibly -0: IEEE gives +0 for -0 and x otherwise (NaN stays NaN)
GVX_FP64I double plus_zero(double x) { const uint64_t b = bits(x); return from_bits(b == kSign ? 0ull : b); }

// Sums, differences and products with an operand z that the algorithm makes an
// exact zero (either sign), for any non-NaN y and finite k: IEEE gives the other
// operand, except that a sum of two zeros is -0 only when both are -0 (a difference
// a - b is a + (-b)), and a finite k times a zero is a zero with the XOR of the signs.
GVX_FP64I double zero_plus(double z, double y) {    // z + y, equally y + z
    const uint64_t uz = bits(z), uy = bits(y);
    return from_bits((uy & kAbs) == 0 ? (uz & uy) : uy);
}
GVX_FP64I double zero_minus(double z, double y) {   // z - y
    const uint64_t uz = bits(z), uy = bits(y);
    return from_bits((uy & kAbs) == 0 ? (uz & ~uy & kSign) : (uy ^ kSign));
}
GVX_FP64I double minus_zero(double y, double z) {   // y - z
    const uint64_t uz = bits(z), uy = bits(y);
    return from_bits((uy & kAbs) == 0 ? (uy & ~uz & kSign) : uy);
}
GVX_FP64I double times_zero(double k, double z) {   // k * z
    return from_bits((bits(k) ^ bits(z)) & kSign);
}

// ------------------------------------------------------------ products, quotients, roots
// Exact FP64 multiplication, division and square root in 32-bit integer arithmetic, for
// operands whose magnitude lies in [2^-255, 2^257) ("in band": biased exponents 768..1279, so
// that no zero, subnormal, infinity or NaN enters and no result leaves the normal range).
// Within the band each returns what the FP64 instruction returns, rounded to nearest even; an
// operand outside it leaves one of kOutOfBand's bits in `rare`, and the caller, which looks at
// `rare` once for a whole group of operations, then discards the results and forms them with
// the FP64 instructions.  (A branch per operation would end the instruction-level parallelism
// these sequences live on; a predicated FP64 instruction costs the pipe the same cycles with
// no lane active as with 32.)
//
// Why: measured on GB300 (2 blocks of 256 threads an SM, four independent chains a thread), a
// warp's DADD or DMUL takes about 80 cycles of its quarter of the SM (77 in this probe, 80 in the one of
// Add in links_int.cuh), a division 548, a square root 572, and the integer pipes run beside it: a product formed here takes 42-50 cycles of issue,
// and product-and-add pairs (product here, sum on the FP64 pipe) 82 cycles a pair against 154,
// two products and an add 97 against 231.
constexpr uint32_t kOutOfBand = 0xC0000000u;

GVX_FP64I uint32_t hi32(double x) {
#ifdef __CUDA_ARCH__
    return (uint32_t)__double2hiint(x);
#else
    return (uint32_t)(bits(x) >> 32);
#endif
}
GVX_FP64I uint32_t lo32(double x) {
#ifdef __CUDA_ARCH__
    return (uint32_t)__double2loint(x);
#else
    return (uint32_t)bits(x);
#endif
}
GVX_FP64I double from_words(uint32_t hi, uint32_t lo) {
#ifdef __CUDA_ARCH__
    return __hiloint2double((int)hi, (int)lo);
#else
    return from_bits(((uint64_t)hi << 32) | lo);
#endif
}
// The high word of (hi:lo) << s, 0 < s < 32.
GVX_FP64I uint32_t shl_words(uint32_t lo, uint32_t hi, uint32_t s) {
#ifdef __CUDA_ARCH__
    return __funnelshift_l(lo, hi, s);
#else
    return (hi << s) | (lo >> (32 - s));
#endif
}
GVX_FP64I uint32_t mul_hi(uint32_t a, uint32_t b) {
#ifdef __CUDA_ARCH__
    return __umulhi(a, b);
#else
    return (uint32_t)(((uint64_t)a * b) >> 32);
#endif
}
GVX_FP64I uint64_t mul_wide(uint32_t a, uint32_t b) { return (uint64_t)a * b; }
GVX_FP64I uint32_t max_u(uint32_t a, uint32_t b) { return a > b ? a : b; }
GVX_FP64I uint32_t min_u(uint32_t a, uint32_t b) { return a < b ? a : b; }

// Top two bits clear exactly when the exponent field of high word h is in 768..1279 (either sign).
GVX_FP64I uint32_t band(uint32_t h) { return h + h - 0x60000000u; }

// About 1/f and 1/sqrt(f) for a float given by its bits (f in [1, 2) and [1, 4)); the callers
// need a relative error of at most 2^-22.  On the host GVX_SEED_ERROR stands in for the hardware's.
#ifndef GVX_SEED_ERROR
#define GVX_SEED_ERROR 0.0
#endif
GVX_FP64I uint32_t seed_rcp(uint32_t fb) {
#ifdef __CUDA_ARCH__
    float r;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(__uint_as_float(fb)));
    return __float_as_uint(r);
#else
    return fbits((float)((1.0 / from_fbits(fb)) * (1.0 + GVX_SEED_ERROR)));
#endif
}
GVX_FP64I uint32_t seed_rsqrt(uint32_t fb) {
#ifdef __CUDA_ARCH__
    float r;
    asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(__uint_as_float(fb)));
    return __float_as_uint(r);
#else
    return fbits((float)((1.0 / __builtin_sqrt((double)from_fbits(fb))) * (1.0 + GVX_SEED_ERROR)));
#endif
}

// x * y.  The 53-bit significands (21 and 32 bits a word) multiply into h : lo(m) : lo(t), 105 or
// 106 bits; one funnel shift by 11 or 12 aligns the top 53 of them, and the rest, with every bit
// below folded into its lowest, carries into them when it is over half, or half and the last bit odd.
GVX_FP64I double mul_band(double x, double y, uint32_t& rare) {
    const uint32_t hx = hi32(x), x0 = lo32(x), hy = hi32(y), y0 = lo32(y);
    rare |= band(hx) | band(hy);
    const uint32_t x1 = (hx & 0xFFFFFu) | 0x100000u, y1 = (hy & 0xFFFFFu) | 0x100000u;
    const uint64_t t = mul_wide(x0, y0);
    uint64_t m = mul_wide(x1, y0) + (t >> 32);
    m += mul_wide(x0, y1);
    const uint64_t h = mul_wide(x1, y1) + (m >> 32);
    const uint32_t hh = (uint32_t)(h >> 32), hl = (uint32_t)h, ml = (uint32_t)m, tl = (uint32_t)t;
    const uint32_t c = hh >> 9, s = 12u - c;   // c: 106 bits
    const uint32_t rh = shl_words(hl, hh, s), rl = shl_words(ml, hl, s);
    const uint32_t rest = shl_words(tl, ml, s) | min_u(tl, 1u);
    // sign and exponent: the signs add modulo 2 in bit 31, the exponents in bits 20..30 (in band
    // their sum stays within 11 bits); less the implicit bit that rh brings
    const uint32_t E = (hx - x1) + (hy - y1) - 0x3FE00000u + (c << 20);
    const uint32_t bump = 0x7FFFFFFFu + (rl & 1u);
#ifdef __CUDA_ARCH__
    uint32_t lo, hi;
    asm("{.reg .u32 d; add.cc.u32 d, %2, %3; addc.cc.u32 %0, %4, 0; addc.u32 %1, %5, %6;}"
        : "=r"(lo), "=r"(hi) : "r"(rest), "r"(bump), "r"(rl), "r"(rh), "r"(E));
    return from_words(hi, lo);
#else
    const uint64_t r = (((uint64_t)rh << 32) | rl) + (((uint64_t)rest + bump) >> 32);
    return from_bits(r + ((uint64_t)E << 32));
#endif
}

// n / d.  A 32-bit reciprocal of d's significand (hardware seed, one Newton step, kept below the
// true value) gives the quotient's top 32 bits and then 23 more from the exact remainder; the last
// remainder says whether that is the floor or one less.  The floor at one bit more than 53 decides
// the rounding: a quotient of two 53-bit numbers is never halfway between two of them.
GVX_FP64I double div_band(double n, double d, uint32_t& rare) {
    const uint32_t hn = hi32(n), n0 = lo32(n), hd = hi32(d), d0 = lo32(d);
    rare |= band(hn) | band(hd);
    const uint32_t n1 = (hn & 0xFFFFFu) | 0x100000u, d1 = (hd & 0xFFFFFu) | 0x100000u;
    const uint32_t n32 = shl_words(n0, n1, 11), d32 = shl_words(d0, d1, 11);
    const uint32_t f = max_u(seed_rcp(0x3F800000u | ((d32 >> 8) & 0x7FFFFFu)) - 10u, 0x3F000000u);
    const uint32_t r0 = (f << 8) | 0x80000000u;                       // 1/d * 2^32, below it by at most 2^-20
    const uint64_t e = 0x8000000000000000ull - mul_wide(d32, r0);     // (1 - d r0) * 2^63
    const uint32_t r = r0 + (mul_hi(r0, (uint32_t)(e >> 12)) >> 19);  // r0 + r0 (1 - d r0)
    const uint64_t N = ((uint64_t)n1 << 32) | n0, D = ((uint64_t)d1 << 32) | d0;
    const uint32_t q1 = mul_hi(n32, r) - 8u;                          // n/d * 2^31, from below
    const uint64_t R1 = (N << 31) - (uint64_t)q1 * D;                 // its remainder, below 16 D
    const uint32_t q2 = (mul_hi((uint32_t)(R1 >> 26), r) - 2u) >> 3;  // R1/D * 2^23, from below
    const uint64_t R2 = (R1 << 23) - (uint64_t)q2 * D;
    uint64_t Q = ((uint64_t)q1 << 23) + q2;                           // floor(n/d * 2^54) or one less
    Q += R2 >= D ? 1 : 0;
    const uint32_t c = (uint32_t)(Q >> 54);                           // the quotient of the significands is >= 1
    const uint64_t q = (Q + 1 + c) >> (1 + c);
    const uint32_t E = ((hn - n1) - (hd - d1)) + 0x3FD00000u + (c << 20);
    return from_words((uint32_t)(q >> 32) + E, (uint32_t)q);
}

// sqrt(x).  A 30-bit reciprocal root (hardware seed, one Newton step, from below) gives the root's
// top 30 bits and then 24 more from the exact remainder; the remainder of the 54-bit root says
// whether it is the floor or one less, and its last bit decides the rounding (a root of a 53-bit
// number is never halfway).  A negative x is out of band.
GVX_FP64I double sqrt_band(double x, uint32_t& rare) {
    const uint32_t hx = hi32(x), x0 = lo32(x);
    rare |= band(hx) | (hx & 0x80000000u);
    const uint32_t x1 = (hx & 0xFFFFFu) | 0x100000u;
    const uint32_t odd = ((hx >> 20) & 1u) ^ 1u;                      // m in [2, 4): the true exponent is odd
    const uint64_t M = (((uint64_t)x1 << 32) | x0) << odd;            // m * 2^52
    const uint32_t m32 = (uint32_t)(M >> 22);                         // m * 2^30
    const uint32_t f = max_u(seed_rsqrt(((127u + odd) << 23) + (shl_words(x0, x1, 3) & 0x7FFFFFu)) - 10u, 0x3F000000u);
    const uint32_t r0 = (f << 8) | 0x80000000u;                       // 1/sqrt(m) * 2^32, below it by at most 2^-20
    const uint32_t u = 0x40000000u - mul_hi(m32, mul_hi(r0, r0));     // (1 - m r0^2) * 2^30
    const uint32_t r = r0 + mul_hi(r0, u + u);                        // r0 + r0 (1 - m r0^2) / 2
    const uint32_t s1 = mul_hi(m32, r) - 8u;                          // sqrt(m) * 2^30, from below
    const uint64_t R = (M << 8) - (uint64_t)s1 * s1;
    const uint32_t q2 = mul_hi((uint32_t)(R >> 6), r) >> 1;           // R / (2 sqrt(m)) * 2^24
    uint64_t S = (((uint64_t)s1 << 24) + q2) >> 1;                    // floor(sqrt(m) * 2^53) or one less
    const uint64_t rem = (M << 54) - S * S;                           // modulo 2^64: it is below 2^58
    S += rem > 2 * S ? 1 : 0;
    const uint64_t q = (S + 1) >> 1;
    const uint32_t E = ((((hx >> 20) + 1023u - odd) >> 1) - 1u) << 20;
    return from_words((uint32_t)(q >> 32) + E, (uint32_t)q);
}

// n / d and sqrt(x) for any operands: the forms above, and the FP64 instructions for the rare rest.
GVX_FP64I double div_any(double n, double d) {
    uint32_t rare = 0;
    double q = div_band(n, d, rare);
    if (rare & kOutOfBand) {
#ifdef __CUDA_ARCH__
        asm volatile("div.rn.f64 %0, %1, %2;" : "=d"(q) : "d"(n), "d"(d));
#else
        q = n / d;
#endif
    }
    return q;
}
GVX_FP64I double sqrt_any(double x) {
    uint32_t rare = 0;
    double q = sqrt_band(x, rare);
    if (rare & kOutOfBand) {
#ifdef __CUDA_ARCH__
        asm volatile("sqrt.rn.f64 %0, %1;" : "=d"(q) : "d"(x));
#else
        q = __builtin_sqrt(x);
#endif
    }
    return q;
}

// x/2 and 2x for an x that mul_band, div_band or sqrt_band checks afterwards (in band: the
// exponent steps; a zero, infinity or NaN stays out of band).
GVX_FP64I double half_band(double x) { return from_words(hi32(x) - 0x100000u, lo32(x)); }
GVX_FP64I double mul2_band(double x) { return from_words(hi32(x) + 0x100000u, lo32(x)); }

// (double)f for a normal f or a zero.
GVX_FP64I double f2d_band(float f, uint32_t& rare) {
    const uint32_t u = fbits(f), a = u & 0x7FFFFFFFu;
    rare = (a - 0x00800000u >= 0x7F000000u && a != 0) ? kOutOfBand : rare;
    const uint32_t hi = (u & 0x80000000u) | (a != 0 ? (a >> 3) + (896u << 20) : 0u);
    return from_words(hi, u << 29);
}
// (float)x, rounded to nearest even, for an x within the normal floats (up to half of the largest).
GVX_FP64I float d2f_band(double x, uint32_t& rare) {
    const uint32_t h = hi32(x), l = lo32(x);
    rare = (h & 0x7FFFFFFFu) - (897u << 20) >= (253u << 20) ? kOutOfBand : rare;
    const uint64_t u = (((uint64_t)h << 32) | l) + 0x0FFFFFFFu + ((l >> 29) & 1u);
    const uint32_t m = (uint32_t)(u >> 29) + 0x40000000u;             // exponent less 896, fraction
    return from_fbits((h & 0x80000000u) | m);
}
// x cut to a float (relative error below 2^-23), for an x within the normal floats.
GVX_FP64I float cut_band(double x, uint32_t& rare) {
    const uint32_t h = hi32(x), l = lo32(x);
    rare = (h & 0x7FFFFFFFu) - (897u << 20) >= (254u << 20) ? kOutOfBand : rare;
    return from_fbits((h & 0x80000000u) | ((shl_words(l, h, 3) + 0x40000000u) & 0x7FFFFFFFu));
}
// a < b for two positive numbers.
GVX_FP64I bool lt_pos(double a, double b) {
    return (((uint64_t)hi32(a) << 32) | lo32(a)) < (((uint64_t)hi32(b) << 32) | lo32(b));
}

}  // namespace fp64i
}  // namespace gvx
