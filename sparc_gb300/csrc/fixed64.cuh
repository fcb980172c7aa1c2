// FP64-accurate arithmetic in 32-bit integer instructions ("block fixed point").
//
// GB300 issues two FP64 lanes per clock and SM (measured: DFMA 2.05, DADD 1.73) but 64
// 32 x 32 + 64-bit integer multiply-adds (mad.wide, measured 63) and about 128 integer adds.
// A linear operator whose operands share a scale therefore runs faster on integers than on
// doubles: with E the largest biased exponent of a block of values, each value becomes the
// fixed-point integer U = x 2^(56 - (E - 1023)), |U| < 2^57, rounded to nearest (exact for every
// value within 2^-4 of the largest), held as two signed digits, U = h 2^29 + l with
// |h|, |l| <= 2^28. The quantum is 2^-56 of the largest value's binade, an eighth of its last
// FP64 bit and a sixteenth of the rounding that FP64 applies to a partial sum, so a sum formed
// this way is at least as accurate, in the norm of the block, as the FP64 one. What repeats in
// every application has to be finer, as it adds up over the degrees of a filter: values cut
// toward zero and coefficients of two digits each made a filter of 20 degrees 1.5 to 2 times less
// accurate than FP64, and ties rounded to one side (values and results away from zero, a potential's
// products up) 1.4 to 1.6 times for columns that fall off from a point, as their errors then have one
// sign. With ties to even and a third coefficient digit the error of a filter with projectors, in
// the norm of a column and against extended precision, is 0.5 to 0.65 of FP64's for uniform and
// smooth columns and for those that fall off by exp(-0.9 r) (Bohr) from a point. What is lost is
// accuracy at a single point whose values are far below their block's largest.
// Sums of six digits fit 32 bits; products with coefficient digits accumulate exactly in 64 bits.
#pragma once

#include <cuda_runtime.h>

namespace sgpu {
namespace fx {

constexpr int kDigit = 29;                       // bits per digit
constexpr int kBits = 57;                        // |U| < 2^kBits
constexpr int kDrop = 26;                        // bits of the middle sum below a result's unit
// biased exponents that a block scale may have: below, U 2^(...) or a product could leave the
// normal range of a double on the way back, above it could overflow; such blocks (and those
// with an infinity or a NaN, exponent 2047) take the FP64 path
constexpr int kMinExp = 256, kMaxExp = 1800;

// the exponent key of a value: ordered as |x| is, key >> 20 its biased exponent
__device__ __forceinline__ unsigned exp_key(double x)
{
    return (unsigned)__double2hiint(x) & 0x7fffffffu;
}

// digits (h, l) of x at block exponent E >= the exponent of x (kMinExp <= E)
__device__ __forceinline__ int2 to_digits(double x, int E)
{
    const unsigned hi = (unsigned)__double2hiint(x), lo = (unsigned)__double2loint(x);
    const int ex = (int)((hi >> 20) & 0x7ffu);
    const int d = min(E - ex, 63);  // ex = 0 (zero, denormal): everything is shifted out
    unsigned long long M = ((unsigned long long)((hi & 0xfffffu) | 0x100000u) << 32) | lo;
    // 8 U, so that h is the upper word; then a half for the rounding, ties to even, and the half digit
    // that rounds h. Values 2^-5 to 2^-7 below the scale lose one to three bits and end in a tie that
    // often; further down ties are rare, and the bits below 8 U make them look like ones.
    M = (M << (kBits + 3 - 53)) >> d;
    const unsigned odd = (((unsigned)M >> 3) | ((unsigned)(d + 120) >> 7)) & 1u;  // or d > 7
    M += (1ull << 31) + 3u + odd;
    const int sg = 1 | ((int)hi >> 31);
    const int l = (int)((unsigned)M ^ 0x80000000u) >> (32 - kDigit);
    const int h = (int)(M >> 32);
    return make_int2(h * sg, l * sg);
}

// hh += h Wh, mid += h Wl + l Wh (l Wl is below 2^-58 of the product's scale). The plain C product of
// widened operands is not safe here: with a loop-invariant operand the compiler hoists its sign
// extension and multiplies 64 by 64 bits (a nonlocal apply of 27 products took 119 multiply-pipe
// instructions per entry).
__device__ __forceinline__ long long mad_wide(int a, int b, long long c)
{
    long long d;
    asm("mul.wide.s32 %0, %1, %2;" : "=l"(d) : "r"(a), "r"(b));
    return c + d;
}
__device__ __forceinline__ void mac(long long &hh, long long &mid, int h, int l, int Wh, int Wl)
{
    hh = mad_wide(h, Wh, hh);
    mid = mad_wide(h, Wl, mid);
    mid = mad_wide(l, Wh, mid);
}

// the sum hh 2^58 + mid 2^29 in units of 2^(29 + kDrop)
__device__ __forceinline__ long long total(long long hh, long long mid)
{
    return (hh << (kDigit - kDrop)) + ((mid + (1ll << (kDrop - 1))) >> kDrop);
}

// The same with a coefficient's third digit, Wr 2^-30 of Wl's unit: lo += h Wr in units of 4 of mid's
__device__ __forceinline__ void mac(long long &hh, long long &mid, int &lo, int h, int l, int Wh, int Wl,
                                    int Wr)
{
    mac(hh, mid, h, l, Wh, Wl);
    lo += __mulhi(h, Wr);
}
__device__ __forceinline__ long long total(long long hh, long long mid, int lo)
{
    return total(hh, mid + (long long)lo * 4);
}

// T 2^K as a double, rounded to nearest, ties to even; the result's exponent must be normal
__device__ __forceinline__ double to_double(long long T, int K)
{
    const int sg = (int)(T >> 63);
    unsigned long long A = (unsigned long long)((T ^ (long long)sg) - (long long)sg);
    const unsigned ah = (unsigned)(A >> 32);
    const int n = __clz((int)(ah ? ah : (unsigned)A)) + (ah ? 0 : 32);
    const int sh = n - 1;  // |T| < 2^63: n >= 1
    A <<= sh;  // leading one at bit 62; rounded at bit 10, ties to even
    A += 0x1ffull + (((unsigned)A >> 10) & 1u);
    const unsigned be1 = (unsigned)(1023 + 62 - sh + K - 1);  // the leading one adds 1
    const unsigned long long b = (A >> 10) + ((unsigned long long)be1 << 52);
    const unsigned rh = (unsigned)(b >> 32) | ((unsigned)sg & 0x80000000u);
    return n >= 64 ? 0.0 : __hiloint2double((int)rh, (int)(unsigned)b);
}

}  // namespace fx
}  // namespace sgpu
