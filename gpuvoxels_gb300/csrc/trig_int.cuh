// The sine of the actuation temperature on the integer pipes.
//
// The library's double-precision sin costs a warp 1,340 cycles of its SM quarter, nearly all of them
// on GB300's narrow FP64 pipe, and its result is rounded to a float in the end.  This one reduces the
// argument and sums the Taylor series in 64-bit fixed point through 32-bit multiplications (absolute
// error below 2^-61).  Only the float is used, and only where no double within a few units in the
// last place of the product could round to another one, so the float is the library's.
#pragma once
#include "fp64_int.cuh"

namespace gvx {
namespace fp64i {

GVX_FP64I uint64_t mul_hi64(uint64_t a, uint64_t b) {
#ifdef __CUDA_ARCH__
    return __umul64hi(a, b);
#else
    return (uint64_t)(((unsigned __int128)a * b) >> 64);
#endif
}
GVX_FP64I int clz64(uint64_t x) {
#ifdef __CUDA_ARCH__
    return __clzll((long long)x);
#else
    return __builtin_clzll(x);
#endif
}
// V * 2^e for V in [2^62, 2^64), rounded to 53 bits; e such that the result is normal.
GVX_FP64I double round64(uint64_t V, int e) {
    const int s = 10 + (int)(V >> 63);
    const uint64_t r = (V >> s) + ((V >> (s - 1)) & 1u);   // 2^52..2^53 (V + half could pass 2^64)
    return from_bits(r + ((uint64_t)(uint32_t)(e + s + 1023 + 51) << 52));
}
// sin(y) for |y| in [2^-10, 2^20): y/(2 pi) to 2^-64 of a turn, folded into a quarter turn R, and
// sin(pi/2 R) = R (c0 - c1 R^2 + ...), c_n = (pi/2)^(2n+1) / (2n+1)!.  Absolute error below 2^-61.
GVX_FP64I double sin_band(double y, uint32_t& rare) {
    const uint32_t h = hi32(y), y0 = lo32(y), y1 = (h & 0xFFFFFu) | 0x100000u;
    const int E = (int)((h >> 20) & 0x7FFu) - 1023;
    rare = (uint32_t)(E + 10) >= 30u ? kOutOfBand : rare;
    // y1:y0 times 1/(2 pi) 2^96 = i2:i1:i0; the turn's fraction starts at bit 84 - E
    constexpr uint32_t i0 = 0x7F09D5F4u, i1 = 0x9391054Au, i2 = 0x28BE60DBu;
    uint64_t a = mul_wide(y0, i0) >> 32;
    uint64_t b = mul_wide(y0, i1) + a;
    uint64_t c = mul_wide(y1, i0) + (uint32_t)b;
    uint64_t d = mul_wide(y0, i2) + (b >> 32);
    uint64_t f = mul_wide(y1, i1) + (c >> 32);
    d += (uint32_t)f;                               // d < 2^64 - 2^32 + 2^32: no carry is lost (i2 < 2^30)
    const uint64_t g = mul_wide(y1, i2) + (f >> 32) + (d >> 32);
    const uint32_t w2 = (uint32_t)d, w3 = (uint32_t)g, w4 = (uint32_t)(g >> 32);
    const uint32_t s = (uint32_t)(E + 12) & 31u;    // 32 - (20 - E)
    const uint64_t F = ((uint64_t)shl_words(w3, w4, s) << 32) | shl_words(w2, w3, s);   // fraction of a turn, times 2^64
    uint64_t R = F << 2;
    if (F & (1ull << 62)) R = ~R;                   // second and fourth quarters
    const uint64_t r2 = mul_hi64(R, R);
    const uint32_t r32 = (uint32_t)(r2 >> 32);
    uint32_t p = 0x944u - mul_hi(r32, 0xCu);        // c_n 2^63, n = 10..8
    p = 0x62901u - mul_hi(r32, p);
    p = 0x355D865u - mul_hi(r32, p);
    uint64_t q = 0x16FADB9F1ull - mul_hi(r32, p);   // n = 7..0
    q = 0x7A3D0D3406ull - mul_hi64(r2, q);
    q = 0x1E3074FDE887ull - mul_hi64(r2, q);
    q = 0x541E0D21FB9E0ull - mul_hi64(r2, q);
    q = 0x9969667315EC2Eull - mul_hi64(r2, q);
    q = 0xA335E33BAD570E9ull - mul_hi64(r2, q);
    q = 0x52AEF39896F94AFBull - mul_hi64(r2, q);
    q = 0xC90FDAA22168C235ull - mul_hi64(r2, q);
    const uint64_t v = mul_hi64(R, q);              // |sin| 2^63
    rare = v < (1ull << 54) ? kOutOfBand : rare;    // near a multiple of pi its relative precision is spent
    const int z = clz64(v | 1u) & 63;
    const double r = round64(v << z, -63 - z);
    return from_words(hi32(r) | ((h ^ (uint32_t)(F >> 32)) & 0x80000000u), lo32(r));
}

// (float)(amp * sin(y)) as the library's sin gives it: the product here and there differ by less
// than 2^5 units of 2^-53 (sin: 2 units in the last place there, below 1 here for results over 2^-9),
// so they round to the same float unless the 29 bits that the rounding drops are that close to half.
GVX_FP64I float sin_times_band(double amp, double y, uint32_t& rare) {
    const double T = amp * sin_band(y, rare);
    rare = ((lo32(T) & 0x1FFFFFFFu) - 0x0FFFFFE0u) < 0x40u ? kOutOfBand : rare;
    return d2f_band(T, rare);
}

}  // namespace fp64i
}  // namespace gvx
