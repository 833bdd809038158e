// Check of the in-band operations of gpuvoxels_gb300/csrc/fp64_int.cuh (mul_band, div_band,
// sqrt_band, d2f_band, cut_band, f2d_band) against IEEE-754 arithmetic, and of trig_int.cuh's
// sin_times_band against (float)(amp * sin(y)) with the library's sin: compiled as C++ it runs on
// the host, with errors of up to 2^-22 put into the division's and the root's seeds; compiled as
// CUDA (-x cu) it runs on the device against the FP64 instructions.  Inputs: random patterns in
// and around the band, short significands, significands ending in ones, products and squares an
// ulp or two from exact ones (the quotients and roots nearest to halfway).
// Usage: fp64_band_check [cases]; exit status 0 when no result differs.
#include <cstdint>
#ifndef __CUDACC__
static double g_seed_error = 0.0;
#define GVX_SEED_ERROR g_seed_error
#endif
#include "../gpuvoxels_gb300/csrc/trig_int.cuh"

#include <cmath>
#include <cstdio>
#include <cstdlib>

using namespace gvx::fp64i;

GVX_FP64I uint64_t next(uint64_t& s) {   // splitmix64
    uint64_t z = (s += 0x9E3779B97F4A7C15ull);
    z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
    z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
    return z ^ (z >> 31);
}
GVX_FP64I uint64_t with_exponent(uint64_t u, uint32_t e) { return (u & 0x800FFFFFFFFFFFFFull) | ((uint64_t)e << 52); }

// One case: the number of results that differ, and (bit k) which operations were in band.
GVX_FP64I int one_case(uint64_t i, uint32_t* in_band) {
    uint64_t s = i * 0x2545F4914F6CDD1Dull + 77;
    uint64_t a = next(s), b = next(s);
    const uint64_t t = next(s);
    const int mode = (int)(i & 15);
    if (mode != 0) {
        a = with_exponent(a, 760 + (uint32_t)(next(s) % 528));
        b = with_exponent(b, 760 + (uint32_t)(next(s) % 528));
    }
    if (mode & 1) { a &= ~0ull << (t % 53); b &= ~0ull << ((t >> 8) % 53); }
    if (mode & 2) { a |= (1ull << ((t >> 16) % 53)) - 1; b |= (1ull << ((t >> 24) % 53)) - 1; }
    double x = from_bits(a), y = from_bits(b), z = fabs(x);
    if ((mode & 12) == 12) {   // close to exact quotients and roots
        const double w = 1.0 + ((int)((t >> 32) % 5) - 2) * 0x1p-53;
        x = (x * y) * w;
        z = (z * z) * w;
    }
#ifndef __CUDACC__
    g_seed_error = ((double)((t >> 40) % 2001) - 1000.0) / 1000.0 * 0x1p-22;
#endif
    int bad = 0;
    uint32_t r = 0;
    auto check = [&](int k, bool same) {
        if (r & kOutOfBand) { r = 0; return; }
        *in_band |= 1u << k;
        if (!same) bad++;
        r = 0;
    };
    double q = mul_band(x, y, r);
    check(0, bits(q) == bits(x * y));
    q = div_band(x, y, r);
    check(1, bits(q) == bits(x / y));
    q = sqrt_band(z, r);
    check(2, bits(q) == bits(sqrt(z)));
    double v = (mode & 4) ? x : from_bits(with_exponent(a, 890 + (uint32_t)((t >> 44) % 270)));
    if (mode & 8) v = from_bits((bits(v) & ~((1ull << 29) - 1)) | (1ull << 28));   // float rounding ties
    float f = d2f_band(v, r);
    check(3, fbits(f) == fbits((float)v));
    f = cut_band(v, r);
    check(4, fabs((double)f - v) <= fabs(v) * 0x1p-23);
    f = from_fbits(mode == 0 ? (uint32_t)t & 0x80000000u : (uint32_t)t);
    q = f2d_band(f, r);
    check(5, bits(q) == bits((double)f));
    const double amp = ldexp(1.0 + (double)(t & 0xFFFFF) * 0x1p-20, (int)(t % 17) - 8) * ((t >> 20) & 1 ? 1.0 : -1.0);
    double turn = from_bits(with_exponent(a, 1023 - 14 + (uint32_t)((t >> 21) % 36)));
    if (mode & 4)   // within 2^-20..2^-50 of a multiple of pi/2: results next to 0 and to +-1
        turn = (double)(int)((t >> 26) % 4096 + 1) * 1.5707963267948966 * (1.0 + ldexp((double)(int)(t % 7) - 3.0, -20 - (int)((t >> 40) % 34)));
    f = sin_times_band(amp, turn, r);
    check(6, fbits(f) == fbits((float)(amp * sin(turn))));
    // an operand that is zero, subnormal, infinite or NaN is always found
    const uint64_t odd[] = {0, kSign, 1, kInf, kInf | kSign, 0x7FF8000000000000ull};
    const double o = from_bits(odd[t % 6]);
    // any operands
    auto same = [](double p, double w) { return bits(p) == bits(w) || (p != p && w != w); };
    if (!same(div_any(x, y), x / y) || !same(div_any(o, y), o / y) || !same(div_any(y, o), y / o)) bad++;
    if (!same(sqrt_any(z), sqrt(z)) || !same(sqrt_any(x), sqrt(x)) || !same(sqrt_any(o), sqrt(o))) bad++;
    auto missed = [&]() { const bool m = (r & kOutOfBand) == 0; r = 0; return m; };
    (void)mul_band(o, y, r); if (missed()) bad++;
    (void)mul_band(y, half_band(o), r); if (missed()) bad++;
    (void)div_band(o, y, r); if (missed()) bad++;
    (void)div_band(y, o, r); if (missed()) bad++;
    (void)sqrt_band(o, r); if (missed()) bad++;
    (void)sqrt_band(-z, r); if (missed()) bad++;
    return bad;
}

#ifdef __CUDACC__
__global__ void cases(uint64_t n, unsigned long long* bad, unsigned* seen) {
    unsigned long long k = 0;
    uint32_t in = 0;
    for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < n; i += (uint64_t)gridDim.x * blockDim.x) k += one_case(i, &in);
    if (k) atomicAdd(bad, k);
    atomicOr(seen, in);
}
#endif

int main(int argc, char** argv) {
    const uint64_t n = argc > 1 ? std::strtoull(argv[1], nullptr, 10) : 3000000ull;
    unsigned long long bad = 0;
    unsigned seen = 0;
#ifdef __CUDACC__
    unsigned long long* d;
    if (cudaMalloc(&d, 16) != cudaSuccess || cudaMemset(d, 0, 16) != cudaSuccess) return 2;
    cases<<<608, 256>>>(n, d, (unsigned*)(d + 1));
    unsigned long long h[2];
    if (cudaMemcpy(h, d, 16, cudaMemcpyDeviceToHost) != cudaSuccess) return 2;
    bad = h[0];
    seen = (unsigned)h[1];
#else
    for (uint64_t i = 0; i < n; i++) bad += one_case(i, &seen);
#endif
    std::printf("%llu cases, %llu mismatches, operations seen in band %x\n", (unsigned long long)n, bad, seen);
    return bad || seen != 0x7Fu ? 1 : 0;
}
