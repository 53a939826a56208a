// The FP64 neighbour sum ((((v0 + v1) + v2) + v3) + v4) + v5, every addition rounded
// to nearest even as the FP64 adder rounds it, on the integer and FP32 pipes.
//
// Why.  GB300 issues an FP64 addition of a warp every 77 cycles per SM quarter
// (measured; 0.53 T additions/s on the chip), an integer or FP32 one every 1 to 2.
// A Gauss-Seidel update is five additions and one fused multiply-add, 460 cycles of
// the FP64 pipe per warp, and the two kinds of pipe run side by side (64 FP32 or
// integer instructions beside 4 FP64 additions take the time of the FP64 ones
// alone).  The sum below is about 140 integer and FP32 instructions and gives the
// same bits, so the smoother leaves the FP64 pipe its multiply-add only.  Measured at
// 256^3 on GB300, a half sweep (k_gsrb2): 104.5 us with FP64 additions in every warp,
// 69.6 us with integer sums in every warp, 59.4 us with FP64 additions in one warp of
// four, 59.5 us in three of eight, 68 us in half; the memory traffic alone is 30 us.
// The same for the trilinear prolongation (weights in the aligning product) gains
// nothing: its eight weighted terms leave room for 2^3 between the values, and in a
// warp some lane's coarse corrections, which change sign every few cells, are further
// apart.
//
// How.  The six values become two's complement integers in one unit, half a last
// place of the smallest one, by a 32 x 32 -> 64 bit product of the mantissa with
// +-2^shift.  Values at most 2^6 apart keep every partial sum below 2^63.  A partial
// sum is an exact 64-bit addition; rounding it to 53 bits drops its k lowest bits,
// 0 <= k <= 11, with k from the position of its leading bit.  The drop is made by an
// FP32 addition: the 13 lowest bits t as the float 2^23 + t (an OR of its bit
// pattern), plus 2^(23+k), whose last place is 2^k: the FP32 adder rounds to nearest
// even, and its tie looks at bit k, which is the parity the FP64 adder looks at.
// Subtracting 2^(23+k) again is exact.  (k = 0 rounds at bit 1, where the lowest bit
// is 0: the unit is half a last place.  k < 0 changes nothing.)  The float's bit
// pattern less that of 2^23 is the rounded integer, so the next addition takes the
// pattern and the constant is taken off with the next value.
// Zeros, subnormals, infinities, NaNs, values further apart than 2^6 and sums whose
// leading bit falls below 2^32 units go to the FP64 additions (a call, so that the
// others branch around it).
#pragma once

#include "pm_common.cuh"

namespace nyxpm {

static __device__ __noinline__ double sum6_fp64(double a, double b, double c, double d, double e, double f)
{
    double s = a + b;
    s = s + c;
    s = s + d;
    s = s + e;
    return s + f;
}

// bit pattern of 2^23 as a float: the 13 bits below it hold an integer
constexpr unsigned kSum6One = 0x4B000000u;
constexpr unsigned kSum6Low = 0x1fffu;

// The 13 lowest bits of a partial sum (its low word lo, its high word hi) rounded to
// a multiple of 2^k, as the bits of 2^23 + result.  bfind gives the leading bit's
// position f below the sign bits of hi (-1: none); k = f - 20.
__device__ __forceinline__ unsigned sum6_round(unsigned lo, int hi)
{
    int f;
    asm("bfind.s32 %0, %1;" : "=r"(f) : "r"(hi));
    const float c = __int_as_float(f * 0x800000 + (130 << 23));   // 2^(23 + k)
    const float x = __uint_as_float((lo & kSum6Low) | kSum6One);
    return __float_as_uint(__fsub_rn(__fadd_rn(x, c), c));
}

// v as a two's complement integer in units of half a last place of the least exponent
// 1 - E1, plus off, modulo 2^64: (h 2^32 + lo) p with p = +-2^s; p < 0 read as unsigned
// is 2^32 too large.
__device__ __forceinline__ unsigned long long sum6_term(double v, unsigned E1, unsigned long long off)
{
    const unsigned hi = (unsigned)__double2hiint(v), lo = (unsigned)__double2loint(v);
    const unsigned s = (hi >> 20) + E1;   // 1 .. 7, modulo 32 (the sign bit of hi is a multiple of it)
    const unsigned h = (hi & 0xfffffu) | 0x100000u;
    const unsigned sg = (unsigned)((int)hi >> 31);
    unsigned p;
    asm("shf.l.wrap.b32 %0, 0, %1, %2;" : "=r"(p) : "r"(2u * sg + 1u), "r"(s));
    unsigned long long t;
    asm("mad.wide.u32 %0, %1, %2, %3;" : "=l"(t) : "r"(lo), "r"(p), "l"(off));
    const unsigned th = h * p + (unsigned)(t >> 32) + sg * lo;
    return ((unsigned long long)th << 32) | (unsigned)t;
}

// a rounded sum, in those units, as a double; false if its leading bit is below 2^32
__device__ __forceinline__ bool sum6_finish(unsigned long long acc, unsigned E, double& out)
{
    const unsigned sg = (unsigned)((int)(acc >> 32) >> 31);
    acc = (acc ^ (((unsigned long long)sg << 32) | sg)) + (unsigned long long)(sg & 1u);
    const unsigned uh = (unsigned)(acc >> 32), ul = (unsigned)acc;
    const unsigned c = (unsigned)__clz((int)uh);
    unsigned nh, nl;   // leading bit to bit 63
    asm("shf.l.wrap.b32 %0, %1, %2, %3;" : "=r"(nh) : "r"(ul), "r"(uh), "r"(c));
    asm("shf.l.wrap.b32 %0, 0, %1, %2;" : "=r"(nl) : "r"(ul), "r"(c));
    // biased exponent E + 10 - c; the leading one adds 1 to the field
    const unsigned H = (nh >> 11) + ((E + 9u - c) << 20) + (sg & 0x80000000u);
    out = __hiloint2double((int)H, (int)__funnelshift_r(nl, nh, 11));
    return uh != 0u;
}

constexpr unsigned long long kSum6Keep = ~(unsigned long long)kSum6Low;

__device__ __forceinline__ double sum6_int(const double (&v)[6])
{
    unsigned a[6];   // bit patterns without the sign
#pragma unroll
    for (int i = 0; i < 6; ++i) a[i] = 2u * (unsigned)__double2hiint(v[i]);
    const unsigned mn = min(__vimin3_u32(a[0], a[1], a[2]), __vimin3_u32(a[3], a[4], a[5]));
    const unsigned mx = max(__vimax3_u32(a[0], a[1], a[2]), __vimax3_u32(a[3], a[4], a[5]));
    const unsigned E = mn >> 21, X = mx >> 21;   // least and greatest biased exponent
    // E >= 64 keeps the result's exponent (at least E - 21) normal; the upper end is
    // far from overflow
    if (X - E <= 6u && E - 64u < 1900u) {
        unsigned long long acc = sum6_term(v[0], 1u - E, 0ULL) + sum6_term(v[1], 1u - E, 0ULL);
#pragma unroll
        for (int i = 2; i < 6; ++i) {
            const unsigned u = sum6_round((unsigned)acc, (int)(acc >> 32));
            acc = (acc & kSum6Keep) + u + sum6_term(v[i], 1u - E, 0ULL - kSum6One);
        }
        const unsigned u = sum6_round((unsigned)acc, (int)(acc >> 32));
        double r;
        if (sum6_finish((acc & kSum6Keep) + (unsigned long long)(u - kSum6One), E, r)) return r;
    }
    return sum6_fp64(v[0], v[1], v[2], v[3], v[4], v[5]);
}

// Whether this warp sums on the integer pipes.  One warp in four keeps the FP64
// additions, so that both kinds of pipe are busy; which one moves with the block, as a
// warp's number modulo 4 is the SM quarter it runs on.
__device__ __forceinline__ bool sum6_on_int()
{
    const unsigned w = (threadIdx.x + blockDim.x * (threadIdx.y + blockDim.y * threadIdx.z)) >> 5;
    return ((w + blockIdx.x + blockIdx.y + blockIdx.z) & 3u) != 3u;
}

__device__ __forceinline__ double sum6(const double (&v)[6], bool on_int)
{
    if (on_int) return sum6_int(v);
    double s = v[0] + v[1];
    s = s + v[2];
    s = s + v[3];
    s = s + v[4];
    return s + v[5];
}

}  // namespace nyxpm
