// nsp_fx.cuh -- 64-bit fixed point for the FP64 form's transforms.
//
// GB300 issues one FP64 warp instruction per 64 cycles and SM sub-partition, a 32-bit
// integer one per 2: an FP64 transform is bound by that pipe alone.  A transform is a
// sum of its inputs with coefficients of modulus 1, so with the inputs of one line
// (all of them, one scale) held as 64-bit integers no partial sum overflows and every
// addition is exact: two integer instructions instead of 64 cycles.  Only the
// twiddle products round, at one unit of the last place.
//
//   scale     a line's values are multiplied by 2^(61 - E), E the exponent of an upper
//             bound of sum |Re| + |Im| over the line (two-sided for a real field's half
//             spectrum), so the unit is 2^-61 of that sum and everything stays below 2^62
//             with two real fields packed into one complex transform;
//   error     a white line of n values has a sum of sqrt(n) times its norm, so the unit is
//             2^-57 of the result's norm at n = 257 and less elsewhere; the products' rounding
//             leaves 2^-55 .. 2^-58 of the norm where an FP64 transform leaves 2^-53;
//   products  x w with w = 2^62 times a twiddle, both split into 32-bit halves with a signed
//             low part: 3 of the 4 half products (the low-low one is below one unit), the
//             middle ones rounded to nearest: 6 wide multiply-adds per real output.
//             Measured against 64-bit long-double arithmetic (N at one level, norm-wise):
//             1.2e-16 .. 3.3e-16 for decaying and 1.5e-16 .. 4.0e-16 for white spectra of
//             32 x 65 to 128 x 257 modes, 2.7e-16 .. 6.4e-16 and 1.3e-15 .. 3.6e-15 with the
//             FP64 transforms it replaced;
//   range     FP64's: the unit goes down to 2^-1075 and results to subnormal numbers (the field of
//             0 at both conversions costs 0.3 .. 0.8% of a step of this form);
//   Inf, NaN  a line that holds one, or whose bound passes 2^1023, gives NaN (its E is FX_BAD), as
//             its FP64 transform would with Inf.
#pragma once
#include <cuda_runtime.h>

#include "nsp_fft.cuh"

namespace nsp {

constexpr int FX_BITS = 61;      // a line's sum of magnitudes stays below 2^FX_BITS
constexpr int FX_BAD = 1 << 20;  // exponent of a line that holds Inf or NaN

// Upper 31 bits of |x|: orders like the value (as an unsigned integer).
__device__ __forceinline__ unsigned fx_key(double x) { return (unsigned)__double2hiint(x) & 0x7FFFFFFFu; }

// |x| of key k in units of 2^(emax - 20), rounded up, for keys with exponents up to emax.
__device__ __forceinline__ unsigned fx_mag(unsigned k, unsigned emax) {
  return (((k & 0xFFFFFu) | 0x100000u) >> min(emax - (k >> 20), 31u)) + 1u;
}

// The line's exponent E from its largest exponent field and its sum of magnitudes (fx_mag
// units): the sum is below 2^E.  Clamped at a unit of 2^-1075, below the smallest FP64 number's,
// so that a line follows its values down to subnormal ones; a line whose bound exceeds 2^1023
// (results up to 2^1024) counts as infinite.
__device__ __forceinline__ int fx_exponent(int emax, unsigned sum) {
  const int E = max(emax - 1043 + (32 - __clz((int)sum)), -1014);
  return emax >= 0x7FF || E > 1023 ? FX_BAD : E;
}

// Largest exponent field and sum of magnitudes of a line in one pass: the sum is kept in units
// of the largest value so far (rounded up each time the unit grows).
struct FxSum {
  int e = 0;
  unsigned s = 0u;
  // two values by their keys
  __device__ __forceinline__ void add(unsigned kx, unsigned ky) {
    const int n = max(e, (int)(max(kx, ky) >> 20));
    s = (s >> min(n - e, 31)) + fx_mag(kx, (unsigned)n) + fx_mag(ky, (unsigned)n) + 1u;
    e = n;
  }
  // ... and over the warp; returns the exponent
  __device__ __forceinline__ int warp_exponent() const {
    const int n = __reduce_max_sync(0xFFFFFFFFu, e);
    return fx_exponent(n, __reduce_add_sync(0xFFFFFFFFu, (s >> min(n - e, 31)) + 1u));
  }
};

// x 2^(FX_BITS - E) rounded to the nearest integer; |x| < 2^E.  (Truncation would stop every
// coefficient below one unit; rounded, the units of the others carry it on average as the
// roundings of a floating-point sum do.)
__device__ __forceinline__ fx fx_from(double x, int E) {
  const unsigned hi = (unsigned)__double2hiint(x), lo = (unsigned)__double2loint(x);
  const unsigned e = (hi >> 20) & 0x7FFu, nz = min(e, 1u);  // (zero and subnormal: 0.m at exponent 1)
  const unsigned mh = (hi & 0xFFFFFu) + (nz << 20);
  // 1.m left-aligned below the sign bit, then shifted right by r >= 2
  const unsigned long long m = ((unsigned long long)__funnelshift_l(lo, mh, 10) << 32) | (lo << 10);
  const int r = E + 1084 - FX_BITS - (int)e + (int)nz;
  const fx v = (fx)(((m >> min(r - 1, 63)) + 1) >> 1);
  const fx s = (fx)((int)hi >> 31);
  return (v ^ s) - s;
}
// The same for x q, q < 2^9 a whole number: the product is formed exactly.
__device__ __forceinline__ fx fx_from_times(double x, unsigned q, int E) {
  const unsigned hi = (unsigned)__double2hiint(x), lo = (unsigned)__double2loint(x);
  const unsigned e = (hi >> 20) & 0x7FFu, nz = min(e, 1u);
  const unsigned mh = (hi & 0xFFFFFu) + (nz << 20);
  const int z = __clz((int)q) - 22;  // q 2^z in [2^9, 2^10): the product in [2^61, 2^63)
  const unsigned qz = q << z;
  const unsigned long long m = (unsigned long long)lo * qz + ((unsigned long long)(mh * qz) << 32);
  const int r = E + 1074 - FX_BITS - (int)e + (int)nz + z;
  const fx v = q ? (fx)(((m >> min(r - 1, 63)) + 1) >> 1) : 0;
  const fx s = (fx)((int)hi >> 31);
  return (v ^ s) - s;
}

// v 2^e rounded to nearest, |v| < 2^62, e = E - FX_BITS of a line (or one less: a halved result).
// The leading bit goes to 62, or to where a result below 2^-1022 has it with an exponent field of 0.
__device__ __forceinline__ double fx_to(fx v, int e) {
  const int s = (int)(v >> 63);
  const unsigned long long a = (unsigned long long)((v ^ (fx)s) - (fx)s);
  const int z = min(__clzll((long long)a) - 1, e + 1084);  // (rounding carries into 63 at most)
  const unsigned long long q = ((a << (z & 63)) + 0x200u) >> 10;
  const unsigned hi = (unsigned)(q >> 32) + ((unsigned)(1084 + e - z) << 20);
  return __hiloint2double((int)(a ? hi | ((unsigned)s & 0x80000000u) : 0u), (int)q);
}

__device__ __forceinline__ double fx_nan() { return __hiloint2double(0x7FF80000, 0); }

// Signed halves: x = h 2^32 + l.
__device__ __forceinline__ void fx_split(fx x, int& h, int& l) {
  l = (int)x;
  h = (int)(x >> 32) - (l >> 31);
}
__device__ __forceinline__ long long fx_mad(int a, int b, long long c) { return (long long)a * b + c; }
// Products are summed as hi 2^64 + mid 2^32, mid first (from the rounding constant); its upper
// word then starts hi, so that the two words shifted out of (hi, low word of mid) are the
// result / 2^62.
constexpr long long FX_HALF = 1ll << 29;
__device__ __forceinline__ fx fx_out(long long hi, long long mid) {
  const unsigned h0 = (unsigned)hi, h1 = (unsigned)(hi >> 32);
  return (fx)(((unsigned long long)__funnelshift_l(h0, h1, 2) << 32) | __funnelshift_l((unsigned)mid, h0, 2));
}

// x c / 2^62 for c = (ch, cl) in signed halves.
__device__ __forceinline__ fx fx_mulc(fx x, int ch, int cl) {
  int h, l;
  fx_split(x, h, l);
  const long long mid = fx_mad(l, ch, fx_mad(h, cl, FX_HALF));
  return fx_out(fx_mad(h, ch, mid >> 32), mid);
}

// v (re + i im), the factor's parts in signed halves.
__device__ __forceinline__ cpx<fx> fx_cmul(const cpx<fx>& v, int rh, int rl, int ih, int il) {
  int xh, xl, yh, yl;
  fx_split(v.x, xh, xl);
  fx_split(v.y, yh, yl);
  const int nh = -ih, nl = -il;
  const long long mx = fx_mad(yl, nh, fx_mad(yh, nl, fx_mad(xl, rh, fx_mad(xh, rl, FX_HALF))));
  const long long my = fx_mad(xl, ih, fx_mad(xh, il, fx_mad(yl, rh, fx_mad(yh, rl, FX_HALF))));
  return mk<fx>(fx_out(fx_mad(yh, nh, fx_mad(xh, rh, mx >> 32)), mx),
                fx_out(fx_mad(xh, ih, fx_mad(yh, rh, my >> 32)), my));
}
// w = exp(-2 pi i e / n) of the table; the inverse takes its conjugate.
template <> __device__ __forceinline__ cpx<fx> twmul<fx, +1>(const cpx<fx>& v, const int4& w) {
  return fx_cmul(v, w.x, w.y, -w.z, -w.w);
}
template <> __device__ __forceinline__ cpx<fx> twmul<fx, -1>(const cpx<fx>& v, const int4& w) {
  return fx_cmul(v, w.x, w.y, w.z, w.w);
}

// Constants exp(2 pi i e / n) of the register transforms as 2^62 fractions in signed halves
// (Re h, Re l, Im h, Im l): n = 16 for e = 1, 2 and n = 9 for e = 1, 2, 4.
struct FxConst { int rh, rl, ih, il; };
constexpr FxConst FX_W16_1{992008094, 1696238673, 410903207, -1364630830};
constexpr FxConst FX_W16_2{759250125, -25716447, 759250125, -25716447};
constexpr FxConst FX_W9_1{822533958, -1633652124, 690187940, 2016164183};
constexpr FxConst FX_W9_2{186453311, 96060625, 1057429273, 37236404};
constexpr FxConst FX_W9_4{-1008987269, 1537591498, 367241333, -1978927779};
template <int SIGN> __device__ __forceinline__ cpx<fx> fx_rot(const cpx<fx>& v, FxConst c) {
  return fx_cmul(v, c.rh, c.rl, SIGN * c.ih, SIGN * c.il);
}

// s / 2, an odd s rounded to the even neighbour (no bias).
__device__ __forceinline__ fx fx_half(fx s) {
  const fx t = s >> 1;
  return t + (s & t & 1);
}

// 2^62 sin(pi/3) = 0x376CF5D0B09954E7 rounded, in signed halves.
constexpr int FX_S3_H = 0x376CF5D1, FX_S3_L = (int)0xB09954E7;
template <int SIGN> __device__ __forceinline__ void dft3_fx(cpx<fx>* v) {
  const cpx<fx> s = cadd(v[1], v[2]), id = muli<fx, SIGN>(csub(v[1], v[2])), a = v[0];
  v[0] = cadd(a, s);
  const cpx<fx> m = mk<fx>(a.x - fx_half(s.x), a.y - fx_half(s.y));
  const cpx<fx> e = mk<fx>(fx_mulc(id.x, FX_S3_H, FX_S3_L), fx_mulc(id.y, FX_S3_H, FX_S3_L));
  v[1] = cadd(m, e);
  v[2] = csub(m, e);
}


template <> struct Rot<fx> {
  template <int SIGN, int N, int E> static __device__ __forceinline__ cpx<fx> by(const cpx<fx>& v) {
    if constexpr (N == 9) {
      return fx_rot<SIGN>(v, E == 1 ? FX_W9_1 : E == 2 ? FX_W9_2 : FX_W9_4);
    } else {
      constexpr int e = N == 8 ? 2 * E : E;
      if constexpr (e == 4) return muli<fx, SIGN>(v);
      else if constexpr (e == 2 || e == 6) {  // (+-1 + SIGN i) sqrt(1/2)
        const cpx<fx> i = muli<fx, SIGN>(v), a = e == 2 ? cadd(v, i) : csub(i, v);
        return mk<fx>(fx_mulc(a.x, FX_W16_2.rh, FX_W16_2.rl), fx_mulc(a.y, FX_W16_2.rh, FX_W16_2.rl));
      } else if constexpr (e == 1) return fx_rot<SIGN>(v, FX_W16_1);
      else if constexpr (e == 3) return fx_cmul(v, FX_W16_1.ih, FX_W16_1.il, SIGN * FX_W16_1.rh, SIGN * FX_W16_1.rl);
      else return fx_cmul(v, -FX_W16_1.rh, -FX_W16_1.rl, -SIGN * FX_W16_1.ih, -SIGN * FX_W16_1.il);  // e == 9
    }
  }
};

__device__ __forceinline__ double2 fx_value(const cpx<fx>& v, int E) {
  if (E == FX_BAD) return make_double2(fx_nan(), fx_nan());
  return make_double2(fx_to(v.x, E - FX_BITS), fx_to(v.y, E - FX_BITS));
}

// ---- kernels along z (the z stage, the cross sections)
constexpr int MAXRZ = 6;  // register rounds of the run-time FFT
// Threads of the z kernels, about the butterflies of a pass over their 6 RPB lines, and the
// blocks per SM that the registers are limited for.  Measured per length, one z-stage launch of
// NR=48 x 32 x n/3 modes, ns per member and mode against three blocks of 192 threads (two of
// 288 from 576 points): 72: 800 (905), 96: 811 (1020), 144: 809 (936), 162: 1053 (1232),
// 192: 665 (733), 216: 922 (931), 288: 775, 384: 734 (788), 432: 863 (912), 576: 943 (989),
// 768: 855 (930): many small blocks cover the barriers between the passes, where the radix
// leaves them the registers.
constexpr int z_threads(int n) { return n == 432 ? 288 : n == 0 || n >= 96 ? 192 : n >= 54 ? 128 : 96; }
constexpr int z_blocks(int n) {
  return n == 0 ? 1 : n >= 576 ? 2 : n == 288 || n == 432 ? 3 : n >= 216 ? 4 : n >= 162 ? 5 : n >= 96 ? 6 : 8;
}

// Values per line in shared memory: the gaps between passes, at least two behind the line.
constexpr int line_pitch(int n) { return line_pad(n - 1) + 1 > n + 2 ? line_pad(n - 1) + 1 : n + 2; }
// Theta rows per block: two (three packed forward transforms for both) while the six lines of
// each leave three blocks on an SM.
constexpr int z_rows(int n) { return n == 0 || n >= 384 ? 1 : 2; }
static_assert(MAXRZ * z_threads(0) >= RT_TASKS, "register rounds of the run-time FFT");
// Threads of a run-time length: a thread's 255 registers leave an SM one block of 192, and six
// lines of up to 18 points are 18 to 54 butterflies, so those take blocks of 64 (64 members of
// NR=48 x 4 x 2 modes, z stage: 867 -> 291 us, FP64 transforms 797; 64 of 18 x 6: 5185 -> 1767,
// 5245; the cross sections of 64 of NR=96 x 4 x 2: 658 -> 300, direct sums 229).
constexpr int RT_SHORT = 18;
constexpr int rt_z_threads(int n) { return n <= RT_SHORT ? 64 : z_threads(0); }
static_assert(MAXRZ * rt_z_threads(RT_SHORT) >= 6 * RT_SHORT / 2, "register rounds of the short run-time lengths");

}  // namespace nsp
