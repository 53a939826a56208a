// The cloud-in-cell weights (sx sy) sz of FP64 positions, every product rounded to
// nearest even as the FP64 multiplier rounds it, on the integer pipe.
//
// Why.  GB300 issues an FP64 instruction of a warp every 77 cycles per SM quarter, so the
// FP64 pipe bounds the kick (57 of them per particle: 9 for the position within its cell,
// 12 products, 24 for the interpolation, 12 for the update) and the deposit (21 and the
// additions).  The fractions, their complements and the twelve products below, and six of
// the update's (mul_on_int), are integer instructions that run beside the rest: 24 of the
// 57 and 18 of the 21.  Measured at 256^3, one particle per cell: k_kick 1843 -> 1172 us
// (1290 without the update's six); k_deposit_keys 1409 -> 908 us, 1227 by the weights, the
// others by what is said there.
//
// How.  For l in [1/2, 2^31) the bits of l below the point, shifted to the top of a
// 64-bit word X, are frac(l) = X 2^-64 exactly, and 1 - frac(l) = -X 2^-64 (modulo 2^64).
// Normalised (leading bit at bit 63) they have at most 53 bits, as doubles do; a product
// of two is 128 bits, rounded at bit 11 of its upper word by the bits below.  Where a
// fraction or its complement is below 2^-32 (a position on a cell face, say), l is
// outside the range, or a rounded product sx sy is a power of two, the FP64 products
// stand in.
#pragma once

#include "pm_common.cuh"

namespace nyxpm {

struct CicAxis {
    unsigned long long m[2];   // 1 - frac, frac: bit 63 set
    unsigned e[2];             // their biased exponents
};

// i = floor(l); false where the integer form does not hold
__device__ __forceinline__ bool cic_axis(double l, int* i, CicAxis& a)
{
    const unsigned long long u = (unsigned long long)__double_as_longlong(l);
    const unsigned e = (unsigned)(u >> 52);
    const unsigned up = e - 1011u;   // 11 .. 42: the point to the top of the word
    const unsigned long long m = (u & 0xfffffffffffffULL) | (1ULL << 52);
    const unsigned long long X = m << (up & 63u), Y = 0ULL - X;
    *i = (int)(m >> ((64u - up) & 63u));
    const unsigned xh = (unsigned)(X >> 32), yh = (unsigned)(Y >> 32);
    const unsigned cx = (unsigned)__clz((int)xh), cy = (unsigned)__clz((int)yh);
    a.m[0] = Y << (cy & 31u);
    a.m[1] = X << (cx & 31u);
    a.e[0] = 1022u - cy;
    a.e[1] = 1022u - cx;
    return up - 11u < 32u && xh != 0u && yh != 0u;
}

// the 128-bit product of two normalised mantissas, normalised: its upper word with
// bit 0 set if any bit below is; e += its leading bit's place
__device__ __forceinline__ unsigned long long cic_product(unsigned long long a, unsigned long long b, unsigned& e)
{
    const unsigned ah = (unsigned)(a >> 32), al = (unsigned)a, bh = (unsigned)(b >> 32), bl = (unsigned)b;
    const unsigned long long p0 = (unsigned long long)al * bl;
    const unsigned long long p1 = (unsigned long long)al * bh + (p0 >> 32);
    const unsigned long long p2 = (unsigned long long)ah * bl + (unsigned)p1;
    unsigned long long hi = (unsigned long long)ah * bh + (p1 >> 32) + (p2 >> 32);
    const unsigned lo = (unsigned)p2;
    const unsigned top = (unsigned)(hi >> 63), sh = 1u - top;
    hi = (hi << sh) | ((lo >> 31) & sh);
    // (the product is a multiple of 2^22, so what is left below is not 0 if lo or p0 is not)
    const unsigned rest = (lo << sh) | (unsigned)p0;
    e += top;
    return hi | (rest != 0u ? 1ULL : 0ULL);
}

// 0 or 1: what rounding to nearest even adds at bit 11
__device__ __forceinline__ unsigned cic_up(unsigned long long hi)
{
    const unsigned w = (unsigned)hi;
    return ((w & 0x7ffu) + 0x3ffu + ((w >> 11) & 1u)) >> 11;
}

// a b
__device__ __forceinline__ double mul_on_int(double a, double b)
{
    const unsigned long long ua = (unsigned long long)__double_as_longlong(a);
    const unsigned long long ub = (unsigned long long)__double_as_longlong(b);
    const unsigned ea = (unsigned)(ua >> 52) & 0x7ffu, eb = (unsigned)(ub >> 52) & 0x7ffu;
    unsigned e = ea + eb - 1023u;
    if (ea - 1u >= 2046u || eb - 1u >= 2046u || e - 2u >= 2043u) return a * b;   // 0, subnormal, out of range, NaN
    const unsigned long long h = cic_product((ua << 11) | (1ULL << 63), (ub << 11) | (1ULL << 63), e);
    // the leading one adds 1 to the exponent field
    const unsigned long long bits = (h >> 11) + cic_up(h) + ((unsigned long long)(e - 1u) << 52);
    return __longlong_as_double((long long)(bits | ((ua ^ ub) & (1ULL << 63))));
}

// w[cx + 2 cy + 4 cz] = (sx[cx] sy[cy]) sz[cz], s[0] = 1 - frac, s[1] = frac, of the
// positions l in cells (l + 1/2); cell = floor(l)
__device__ __forceinline__ void cic_weights(double lx, double ly, double lz, int (&cell)[3], double (&w)[8])
{
    CicAxis x, y, z;
    bool ok = cic_axis(lx, cell, x);
    ok = cic_axis(ly, cell + 1, y) && ok;
    ok = cic_axis(lz, cell + 2, z) && ok;
    if (ok) {
#pragma unroll
        for (int t = 0; t < 4; ++t) {
            unsigned e = x.e[t & 1] + y.e[t >> 1] - 1023u;
            const unsigned long long hi = cic_product(x.m[t & 1], y.m[t >> 1], e);
            const unsigned long long xy = ((hi >> 11) + cic_up(hi)) << 11;
            ok = ok && xy != 0ULL;   // rounded up to the next power of two
#pragma unroll
            for (int cz = 0; cz < 2; ++cz) {
                unsigned ez = e + z.e[cz] - 1023u;
                const unsigned long long h = cic_product(xy, z.m[cz], ez);
                // the leading one adds 1 to the exponent field
                const unsigned long long bits = (h >> 11) + cic_up(h) + ((unsigned long long)(ez - 1u) << 52);
                w[t + 4 * cz] = __longlong_as_double((long long)bits);
            }
        }
    }
    if (!ok) {
        const double fx = floor_int(lx, cell), fy = floor_int(ly, cell + 1), fz = floor_int(lz, cell + 2);
        const double px = lx - fx, py = ly - fy, pz = lz - fz;
        const double sx[2] = {1.0 - px, px}, sy[2] = {1.0 - py, py}, sz[2] = {1.0 - pz, pz};
#pragma unroll
        for (int t = 0; t < 8; ++t) w[t] = (sx[t & 1] * sy[t >> 1 & 1]) * sz[t >> 2];
    }
}

}  // namespace nyxpm
