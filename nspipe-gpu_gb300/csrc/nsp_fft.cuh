// nsp_fft.cuh -- batched mixed-radix (4/2/3) complex FFTs in shared memory.
//
// In-place Stockham autosort: every stage loads each thread's butterfly inputs
// into registers, synchronises the block, and writes the outputs to their
// Stockham positions, so no ping-pong buffer is needed.  A stage of radix P
// with sub-transform size Ns reads x[j + q n/P], twiddles by w^(q (j mod Ns) n/(Ns P)),
// applies the P-point DFT and writes x[(j/Ns) Ns P + j mod Ns + q Ns]; the result
// is in natural order.  Twiddles come from a table tw[e] = exp(-2 pi i e / n)
// (conjugated for the inverse), computed on the host from long-double sin/cos.
#pragma once
#include <cuda_runtime.h>

#include <type_traits>

#include "nsp_internal.h"

namespace nsp {

// Aligned to its full size so that loads and stores of a complex value are single vector accesses.
template <typename T> struct alignas(2 * sizeof(T)) cpx { T x, y; };
template <typename T> struct vec2;
template <> struct vec2<double> { using type = double2; };
template <> struct vec2<float> { using type = float2; };

template <typename T> __device__ __forceinline__ cpx<T> mk(T x, T y) { cpx<T> r; r.x = x; r.y = y; return r; }
template <typename T> __device__ __forceinline__ cpx<T> cadd(cpx<T> a, cpx<T> b) { return mk<T>(a.x + b.x, a.y + b.y); }
template <typename T> __device__ __forceinline__ cpx<T> csub(cpx<T> a, cpx<T> b) { return mk<T>(a.x - b.x, a.y - b.y); }
template <typename T> __device__ __forceinline__ cpx<T> cmulv(cpx<T> a, cpx<T> b) {
  return mk<T>(a.x * b.x - a.y * b.y, a.x * b.y + a.y * b.x);
}
// multiply by sign*i
template <typename T, int SIGN> __device__ __forceinline__ cpx<T> muli(cpx<T> a) {
  return SIGN > 0 ? mk<T>(-a.y, a.x) : mk<T>(a.y, -a.x);
}

// 64-bit fixed point (nsp_fx.cuh): the value type of the FP64 form's transforms.
using fx = long long;
template <> struct vec2<fx> { using type = int4; };  // a twiddle as two split 62-bit fractions

// v times the table's twiddle w = exp(-2 pi i e / n), conjugated for the inverse (SIGN > 0).
template <typename T, int SIGN>
__device__ __forceinline__ cpx<T> twmul(const cpx<T>& v, const typename vec2<T>::type& w) {
  return cmulv(v, mk<T>(w.x, SIGN > 0 ? -w.y : w.y));
}
template <int SIGN> __device__ __forceinline__ void dft3_fx(cpx<fx>* v);  // nsp_fx.cuh

template <typename T, int SIGN, int P> __device__ __forceinline__ void dft(cpx<T>* v) {
  if (P == 2) {
    cpx<T> a = v[0], b = v[1];
    v[0] = cadd(a, b);
    v[1] = csub(a, b);
  } else if (P == 4) {
    cpx<T> t0 = cadd(v[0], v[2]), t1 = csub(v[0], v[2]);
    cpx<T> t2 = cadd(v[1], v[3]), t3 = muli<T, SIGN>(csub(v[1], v[3]));
    v[0] = cadd(t0, t2);
    v[2] = csub(t0, t2);
    v[1] = cadd(t1, t3);
    v[3] = csub(t1, t3);
  } else if constexpr (std::is_same<T, fx>::value) {  // P == 3
    dft3_fx<SIGN>(v);
  } else {
    const T s3 = (T)0.8660254037844386;  // sin(pi/3)
    cpx<T> s = cadd(v[1], v[2]), d = csub(v[1], v[2]);
    cpx<T> a = v[0];
    v[0] = cadd(a, s);
    cpx<T> m = mk<T>(a.x - (T)0.5 * s.x, a.y - (T)0.5 * s.y);
    cpx<T> id = muli<T, SIGN>(d);
    v[1] = mk<T>(m.x + s3 * id.x, m.y + s3 * id.y);
    v[2] = mk<T>(m.x - s3 * id.x, m.y - s3 * id.y);
  }
}

// 16-byte asynchronous copies global -> shared (cp.async), groups of copies and their waits.
__device__ __forceinline__ void cp_async16(void* dst, const void* src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"((unsigned)__cvta_generic_to_shared(dst)), "l"(src)
               : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;\n" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_async_wait() { asm volatile("cp.async.wait_group %0;\n" ::"n"(N) : "memory"); }

// One Stockham stage over nb transforms of length n.  Element e of transform t
// lives at buf[t*bs + e*es].  TFAST: consecutive threads take consecutive
// transforms (for element-strided layouts), else consecutive butterflies.
template <typename T, int SIGN, int P, int MAXR, bool TFAST>
__device__ __forceinline__ void fft_stage(cpx<T>* buf, int n, int nb, int es, int bs, int Ns,
                                          const typename vec2<T>::type* __restrict__ tw) {
  const int nbf = n / P;
  const int total = nb * nbf;
  const int tstride = n / (Ns * P);
  cpx<T> v[MAXR][P];
#pragma unroll
  for (int rr = 0; rr < MAXR; rr++) {
    int b = threadIdx.x + rr * blockDim.x;
    if (b < total) {
      int t = TFAST ? b % nb : b / nbf;
      int j = TFAST ? b / nb : b - t * nbf;
      const cpx<T>* x = buf + (size_t)t * bs;
#pragma unroll
      for (int q = 0; q < P; q++) v[rr][q] = x[(j + q * nbf) * es];
    }
  }
  __syncthreads();
#pragma unroll
  for (int rr = 0; rr < MAXR; rr++) {
    int b = threadIdx.x + rr * blockDim.x;
    if (b < total) {
      int t = TFAST ? b % nb : b / nbf;
      int j = TFAST ? b / nb : b - t * nbf;
      int k = j % Ns;
      if (k) {
#pragma unroll
        for (int q = 1; q < P; q++) {
          v[rr][q] = twmul<T, SIGN>(v[rr][q], __ldg(tw + (q * k * tstride) % n));
        }
      }
      dft<T, SIGN, P>(v[rr]);
      cpx<T>* x = buf + (size_t)t * bs;
      int base = (j / Ns) * Ns * P + k;
#pragma unroll
      for (int q = 0; q < P; q++) x[(base + q * Ns) * es] = v[rr][q];
    }
  }
  __syncthreads();
}

// Full transform (SIGN -1 forward, +1 inverse, unnormalised).  The caller
// synchronises before the call (data written) and may read right after.
template <typename T, int SIGN, int MAXR, bool TFAST>
__device__ void fft_batch(cpx<T>* buf, const FftPlan& pl, int nb, int es, int bs,
                          const typename vec2<T>::type* __restrict__ tw) {
  int Ns = 1;
  for (int s = 0; s < pl.nst; s++) {
    int P = pl.rad[s];
    if (P == 4) fft_stage<T, SIGN, 4, MAXR, TFAST>(buf, pl.n, nb, es, bs, Ns, tw);
    else if (P == 2) fft_stage<T, SIGN, 2, MAXR, TFAST>(buf, pl.n, nb, es, bs, Ns, tw);
    else fft_stage<T, SIGN, 3, MAXR, TFAST>(buf, pl.n, nb, es, bs, Ns, tw);
    Ns *= P;
  }
}

// ---------------------------------------------------------------------------
// Radices (4, 2, 3) of the compiled register transforms (reg_fft), stage by stage.
__host__ __device__ constexpr int ct_radix(int n, int s) {
  int k = 0;
  while (n % 4 == 0) { if (k == s) return 4; n /= 4; k++; }
  while (n % 2 == 0) { if (k == s) return 2; n /= 2; k++; }
  while (n % 3 == 0) { if (k == s) return 3; n /= 3; k++; }
  return 0;
}
__host__ __device__ constexpr int ct_nstages(int n) {
  int k = 0;
  while (ct_radix(n, k)) k++;
  return k;
}

// ---------------------------------------------------------------------------
// Transforms of few passes: radices up to 16 with the butterflies in registers.

// v exp(SIGN 2 pi i E / N) for the constants of the register transforms, N = 8, 9 or 16
// (nsp_fx.cuh: fixed point).
template <typename T> struct Rot {
  template <int SIGN, int N, int E> static __device__ __forceinline__ cpx<T> by(const cpx<T>& v) {
    constexpr T h = (T)0.70710678118654752440, c = (T)0.92387953251128675613, s = (T)0.38268343236508977173;
    constexpr T c9[5] = {1, (T)0.76604444311897803520, (T)0.17364817766693034885, 0, (T)-0.93969262078590838405};
    constexpr T s9[5] = {0, (T)0.64278760968653932632, (T)0.98480775301220805937, 0, (T)0.34202014332566873304};
    constexpr int e = N == 8 ? 2 * E : E;
    if constexpr (N == 9) return cmulv(v, mk<T>(c9[E], SIGN * s9[E]));
    else if constexpr (e == 4) return muli<T, SIGN>(v);
    else if constexpr (e == 2 || e == 6) {  // (+-1 + SIGN i) sqrt(1/2)
      const cpx<T> i = muli<T, SIGN>(v), a = e == 2 ? cadd(v, i) : csub(i, v);
      return mk<T>(h * a.x, h * a.y);
    } else if constexpr (e == 1) return cmulv(v, mk<T>(c, SIGN * s));
    else if constexpr (e == 3) return cmulv(v, mk<T>(s, SIGN * c));
    else return cmulv(v, mk<T>(-c, -SIGN * s));  // e == 9
  }
};

// P-point transform in registers, natural order: 2, 3, 4 (dft), 8 = 2 x 4, 9 = 3 x 3 and
// 16 = 4 x 4 with constant twiddles, 6 = 2 x 3 and 12 = 3 x 4 by Good and Thomas without any.
template <typename T, int SIGN, int P> __device__ __forceinline__ void reg_dft(cpx<T>* v) {
  if constexpr (P <= 4) {
    dft<T, SIGN, P>(v);
  } else if constexpr (P == 6 || P == 12) {
    constexpr int A = P / 3;  // 3 x A, coprime; input (A a + 3 b) mod P, output (KA a + KB b) mod P
    constexpr int KA = 4, KB = A == 4 ? 9 : 3;
    cpx<T> t[P];
#pragma unroll
    for (int b = 0; b < A; b++) {
      cpx<T> x[3] = {v[(3 * b) % P], v[(A + 3 * b) % P], v[(2 * A + 3 * b) % P]};
      dft<T, SIGN, 3>(x);
#pragma unroll
      for (int a = 0; a < 3; a++) t[a * A + b] = x[a];
    }
#pragma unroll
    for (int a = 0; a < 3; a++) {
      dft<T, SIGN, A>(t + a * A);
#pragma unroll
      for (int b = 0; b < A; b++) v[(KA * a + KB * b) % P] = t[a * A + b];
    }
  } else {
    constexpr int B = P == 8 ? 2 : P == 9 ? 3 : 4, A = P / B;  // input B a + b, output a + A b
    cpx<T> t[B][A];
#pragma unroll
    for (int b = 0; b < B; b++) {
#pragma unroll
      for (int a = 0; a < A; a++) t[b][a] = v[B * a + b];
      dft<T, SIGN, A>(t[b]);
    }
    if constexpr (P == 8) {
      t[1][1] = Rot<T>::template by<SIGN, 8, 1>(t[1][1]);
      t[1][2] = Rot<T>::template by<SIGN, 8, 2>(t[1][2]);
      t[1][3] = Rot<T>::template by<SIGN, 8, 3>(t[1][3]);
    } else if constexpr (P == 9) {
      t[1][1] = Rot<T>::template by<SIGN, 9, 1>(t[1][1]);
      t[1][2] = Rot<T>::template by<SIGN, 9, 2>(t[1][2]);
      t[2][1] = Rot<T>::template by<SIGN, 9, 2>(t[2][1]);
      t[2][2] = Rot<T>::template by<SIGN, 9, 4>(t[2][2]);
    } else {
      t[1][1] = Rot<T>::template by<SIGN, 16, 1>(t[1][1]);
      t[1][2] = Rot<T>::template by<SIGN, 16, 2>(t[1][2]);
      t[1][3] = Rot<T>::template by<SIGN, 16, 3>(t[1][3]);
      t[2][1] = Rot<T>::template by<SIGN, 16, 2>(t[2][1]);
      t[2][2] = Rot<T>::template by<SIGN, 16, 4>(t[2][2]);
      t[2][3] = Rot<T>::template by<SIGN, 16, 6>(t[2][3]);
      t[3][1] = Rot<T>::template by<SIGN, 16, 3>(t[3][1]);
      t[3][2] = Rot<T>::template by<SIGN, 16, 6>(t[3][2]);
      t[3][3] = Rot<T>::template by<SIGN, 16, 9>(t[3][3]);
    }
#pragma unroll
    for (int a = 0; a < A; a++) {
      cpx<T> x[B];
#pragma unroll
      for (int b = 0; b < B; b++) x[b] = t[b][a];
      dft<T, SIGN, B>(x);
#pragma unroll
      for (int b = 0; b < B; b++) v[a + A * b] = x[b];
    }
  }
}

// Radices of the compiled lengths: few passes over shared memory, with few enough complex
// values in registers for the kernels' blocks per SM (nsp_fx.cuh: at 192 points 8 x 4 x 6 takes
// 665, 16 x 12 733 ns per member and mode); 0: the length has no compiled transform.  768, one plan
// for both forms: 16 x 8 x 6 takes 88 us in the mixed z stage of a pipe of 48 x 64 x 256 modes and
// 450 in the FP64 form's, 8 x 8 x 12 96 and 435 with an error some 4% lower; the rounding of the
// first leaves the unstable NR=96 run of tests/test_gpu_c1_diag.py in single corrector passes as long
// as the reference's.
// Columns (the theta transforms) have no padding and more lines: two passes where three would do.
__host__ __device__ constexpr int pass_radix(int n, int s, bool cols) {
  if (cols && n == 192) return s == 0 ? 16 : s == 1 ? 12 : 0;
  if (cols && n == 144) return s < 2 ? 12 : 0;
  if (cols && n == 72) return s == 0 ? 9 : s == 1 ? 8 : 0;
  constexpr int R[][4] = {{12, 12, 0, 0}, {18, 2, 9, 0}, {24, 4, 6, 0}, {36, 6, 6, 0}, {48, 8, 6, 0},
                          {54, 6, 9, 0}, {72, 8, 9, 0}, {96, 8, 4, 3}, {108, 9, 12, 0}, {144, 16, 9, 0},
                          {162, 9, 6, 3}, {192, 8, 4, 6}, {216, 6, 6, 6}, {288, 8, 6, 6}, {384, 8, 6, 8},
                          {432, 16, 9, 3}, {576, 8, 9, 8}, {768, 16, 8, 6}};
  for (const auto& r : R)
    if (r[0] == n) return s < 3 ? r[1 + s] : 0;
  return 0;
}

// The compiled lengths, of both forms' kernels and of the cross sections: theta and z.  Any other
// 2^a 3^b length takes the run-time plan (fft_batch), whose kernels all hold at least RT_TASKS
// butterflies of 16 theta columns or of 6 z lines in registers (transform_supported refuses more).
#define NSP_NTP_LIST(X) X(12) X(18) X(24) X(36) X(48) X(54) X(72) X(96) X(108) X(144) X(192)
#define NSP_NZR_LIST(X) X(24) X(36) X(48) X(54) X(72) X(96) X(108) X(144) X(162) X(192) X(216) X(288) X(384) X(432) \
  X(576) X(768)
constexpr int RT_TASKS = 1024;
constexpr bool ntp_compiled(int n) {
#define NSP_IS(m) if (n == m) return true;
  NSP_NTP_LIST(NSP_IS)
  return false;
}
constexpr bool nzr_compiled(int n) {
  NSP_NZR_LIST(NSP_IS)
#undef NSP_IS
  return false;
}
constexpr int pass_length(int n, bool cols) {
  int m = 1;
  for (int s = 0; s < 3 && pass_radix(n, s, cols) > 0; s++) m *= pass_radix(n, s, cols);
  return m;
}
#define NSP_HAS_PLAN_T(n) static_assert(pass_length(n, true) == n, "radices of a compiled theta length");
#define NSP_HAS_PLAN_Z(n) static_assert(pass_length(n, false) == n, "radices of a compiled z length");
NSP_NTP_LIST(NSP_HAS_PLAN_T)
NSP_NZR_LIST(NSP_HAS_PLAN_Z)
#undef NSP_HAS_PLAN_T
#undef NSP_HAS_PLAN_Z

// Place of element e in a line of contiguous elements between passes: one gap per 16 so that
// the strided stores of a first pass spread over the banks.  A transform's input and output
// are without gaps.
__host__ __device__ constexpr int line_pad(int e) { return e + (e >> 4); }
// Place of element b + q D (b of stride-1 origin with b % 16 < R known, q a constant): the gap
// count splits into b's and a constant's wherever no carry can join them.
template <int D, int R> __device__ __forceinline__ int line_at(int b, int q) {
  const int o = q * D;
  if (D % 16 == 0) return line_pad(b) + o + (o >> 4);
  if (R + (o & 15) <= 16) return line_pad(b) + o + (o >> 4);
  return line_pad(b + o);
}
// The number of residues mod 16 that the origin of a pass's reads (j < NBF) or stores
// (multiples of NS P plus k < NS) takes.
__host__ __device__ constexpr int line_res_read(int nbf) { return nbf <= 16 ? nbf : 16; }
__host__ __device__ constexpr int line_res_store(int ns, int p) {
  return ns * p % 16 == 0 ? (ns < 16 ? ns : 16) : ns * p == 8 ? 8 + ns : 16;
}

// One Stockham pass of radix P over NB transforms (contiguous lines: the first nb) of length N,
// in place, length, batch, strides and block size compiled in (so every index division is by a
// constant and the register staging holds exactly the rounds the pass needs):
// element e of transform t at t BS + e ES (COLS: neighbouring threads on neighbouring
// transforms) or at t BS + e
// (line_pad(e) between passes).  Elements [Z0, Z1] are known to be zero on the way in
// (first pass), elements [D0, D1] not needed on the way out (last pass); empty if Z1 < Z0.
template <typename T, int SIGN, int N, int NB, int ES, int BS, bool COLS, int NTH, int P, int NS, int Z0, int Z1, int D0, int D1>
__device__ __forceinline__ void fft_pass(cpx<T>* buf, const typename vec2<T>::type* __restrict__ tw, int nb) {
  constexpr int NBF = N / P, TOTAL = NB * NBF, R = (TOTAL + NTH - 1) / NTH, TSTR = N / (NS * P);
  const int total = COLS ? TOTAL : nb * NBF;
  const bool full = (COLS || nb == NB) && TOTAL % NTH == 0;  // (constant where nb is)
  cpx<T> v[R][P];
#pragma unroll
  for (int rr = 0; rr < R; rr++) {
    const int b = threadIdx.x + rr * NTH;
    if (full || b < total) {
      const int t = COLS ? b % NB : b / NBF, j = COLS ? b / NB : b - t * NBF;
#pragma unroll
      for (int q = 0; q < P; q++) {
        const int e = j + q * NBF;
        if (NS == 1 && q * NBF >= Z0 && (q + 1) * NBF - 1 <= Z1) v[rr][q] = mk<T>(0, 0);
        else if (COLS) v[rr][q] = buf[t * BS + e * ES];
        else if (NS == 1) v[rr][q] = buf[t * BS + e];
        else v[rr][q] = buf[t * BS + line_at<NBF, line_res_read(NBF)>(j, q)];
      }
    }
  }
  __syncthreads();
#pragma unroll
  for (int rr = 0; rr < R; rr++) {
    const int b = threadIdx.x + rr * NTH;
    if (full || b < total) {
      const int t = COLS ? b % NB : b / NBF, j = COLS ? b / NB : b - t * NBF;
      const int k = (NS == 1) ? 0 : j % NS;
      if (NS > 1) {
#pragma unroll
        for (int q = 1; q < P; q++) v[rr][q] = twmul<T, SIGN>(v[rr][q], __ldg(tw + q * k * TSTR));
      }
      reg_dft<T, SIGN, P>(v[rr]);
      const int base = (NS == 1) ? j * P : (j / NS) * NS * P + k;
#pragma unroll
      for (int q = 0; q < P; q++) {
        if (NS * P == N && q * NS >= D0 && (q + 1) * NS - 1 <= D1) continue;
        if (COLS) buf[t * BS + (base + q * NS) * ES] = v[rr][q];
        else if (NS * P == N) buf[t * BS + base + q * NS] = v[rr][q];
        else buf[t * BS + line_at<NS, line_res_store(NS, P)>(base, q)] = v[rr][q];
      }
    }
  }
  __syncthreads();
}

template <typename T, int SIGN, int N, int NB, int ES, int BS, bool COLS, int NTH, int Z0, int Z1, int D0, int D1, int S = 0, int NS = 1>
__device__ __forceinline__ void pass_fft(cpx<T>* buf, const typename vec2<T>::type* __restrict__ tw, int nb = NB) {
  constexpr int P = pass_radix(N, S, COLS);
  if constexpr (P > 0) {
    fft_pass<T, SIGN, N, NB, ES, BS, COLS, NTH, P, NS, Z0, Z1, D0, D1>(buf, tw, nb);
    pass_fft<T, SIGN, N, NB, ES, BS, COLS, NTH, Z0, Z1, D0, D1, S + 1, NS * P>(buf, tw, nb);
  }
}

// Largest butterfly count of any stage (for the MAXR bound check on the host).
inline int max_butterflies(const FftPlan& pl, int nb) {
  int mx = 0;
  for (int s = 0; s < pl.nst; s++) {
    int b = nb * (pl.n / pl.rad[s]);
    if (b > mx) mx = b;
  }
  return mx;
}

inline bool make_plan(int n, FftPlan& pl) {
  pl.n = n;
  pl.nst = 0;
  int m = n;
  while (m % 4 == 0 && pl.nst < MAXPLAN) { pl.rad[pl.nst++] = 4; m /= 4; }
  while (m % 2 == 0 && pl.nst < MAXPLAN) { pl.rad[pl.nst++] = 2; m /= 2; }
  while (m % 3 == 0 && pl.nst < MAXPLAN) { pl.rad[pl.nst++] = 3; m /= 3; }
  return m == 1;
}

}  // namespace nsp
