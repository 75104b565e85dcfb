// nsp_transform.cu -- the 3/2-dealiased nonlinear term, one radial level at a time.
//
// Replaces nonlinear() (mod_io_nonlinear.cu:380-409): derivr x3, padForward x12,
// derivt/derivz x6, 12 batched 2-D Z2D and 3 D2Z cuFFT transforms
// (mod_fft.cu:37-48), calcNonlinear_k (:142-170), normalize (mod_utils.cu:10-17),
// padBackward x3 (:195-214) and pressGrad (mod_radialFD.cu:100-111).  Three
// kernels per evaluation:
//
//   nl_theta_inv  per (member, level, 16 (field, l) columns): builds the padded
//                 theta columns of u, d_r u (7-point stencil over levels, parity
//                 tables) and i m u / r straight from the spectral state and runs
//                 the length-NTP inverse FFTs -> G[f][level][theta_j][l] (9 fields);
//   nl_z          per (member, level, theta rows): forms the 12 Hermitian z
//                 spectra (d_z u = i k_z times the u columns of G), packs them
//                 two real fields per complex length-NZR inverse FFT, evaluates
//                 -(u.grad)u pointwise, packs the 3 products into complex forward
//                 FFTs and unpacks the half spectra l < NZ-1 -> H;
//   nl_theta_fwd  per (member, level, 16 (component, l) columns): length-NTP
//                 forward FFTs of H, scale by 1/(NTP*NZR), keep the retained modes
//                 (theta Nyquist and l = NZ-1 zeroed) and apply the wall-shear
//                 forcing to N_z(0,0).
//
// These are the mixed form's kernels (T = float: the transforms read the FP32 mirror of
// the state, the stencils and products run in FP32); the FP64 form's, over the same
// arrays, are in nsp_transform_fx.cu.  Transform lengths used by the supported configurations are
// compile-time template arguments (all index arithmetic by constants); other
// 2^a 3^b lengths use the run-time FFT.
#include <cmath>
#include <cstdio>
#include <cstdlib>

#include "nsp_bounds.cuh"
#include "nsp_cvt.cuh"
#include "nsp_fft.cuh"
#include "nsp_internal.h"
#include "nsp_state.cuh"

namespace nsp {

constexpr int MAXR = 4;   // register rounds of the run-time FFT
// Theta columns per block: 32 while that gives a pass about as many butterflies as threads.
constexpr int theta_cols(int ntp) { return ntp == 0 || ntp > 108 ? 16 : 32; }
constexpr int TTH = 256;  // threads of the theta kernels
constexpr int ZTH = 256;  // threads of the run-time z kernel
static_assert(MAXR * TTH >= RT_TASKS && MAXR * ZTH >= RT_TASKS, "register rounds of the run-time FFT");
constexpr int Z2TH = 192; // threads of the two-pass z kernel (its passes run 192, 144, 384, 48, 36, 384 tasks)

template <typename T> __device__ __forceinline__ const typename vec2<T>::type* tw_t(const Tables& tb);
template <> __device__ __forceinline__ const float2* tw_t<float>(const Tables& tb) { return tb.tw_t32; }
template <typename T> __device__ __forceinline__ const typename vec2<T>::type* tw_z(const Tables& tb);
template <> __device__ __forceinline__ const float2* tw_z<float>(const Tables& tb) { return tb.tw_z32; }

template <typename T, int NTPC, int SIGN>
__device__ __forceinline__ void theta_fft(cpx<T>* buf, const Tables& tb) {
  constexpr int LC = theta_cols(NTPC);
  if constexpr (NTPC > 0) {
    // zero (inverse) or dropped (forward) middle third
    constexpr int A = NTPC / 3, B = 2 * NTPC / 3 - 1;
    if constexpr (SIGN > 0) pass_fft<T, SIGN, NTPC, LC, LC, 1, true, TTH, A, B, 0, -1>(buf, tw_t<T>(tb));
    else pass_fft<T, SIGN, NTPC, LC, LC, 1, true, TTH, 0, -1, A, B>(buf, tw_t<T>(tb));
  } else {
    fft_batch<T, SIGN, MAXR, true>(buf, tb.pt, LC, LC, 1, tw_t<T>(tb));
  }
}

// ---------------------------------------------------------------- theta inverse
// A thread keeps one column (TTH is a multiple of LC): its field, its place in the state and
// its twiddle-free index arithmetic are computed once.
template <typename T, int NTPC>
__global__ void __launch_bounds__(TTH) nl_theta_inv(Tables tb, Bufs bf, const Ctl* ctl, const double2* src_override,
                                                    const float2* src32_override) {
  constexpr int LC = theta_cols(NTPC), PS = TTH / LC;
  static_assert(TTH % LC == 0, "a thread stays on one column");
  const int mloc = blockIdx.z, i = blockIdx.y, c0 = blockIdx.x * LC;
  bool skip;
  member_source(tb, bf, ctl, mloc, src_override, skip);
  if (skip) return;
  const StateIn<T> U = member_input<T>(tb, bf, ctl, mloc, src_override, src32_override);
  const float2* DR = member_dr32(tb, bf, ctl, mloc, src_override);
  extern __shared__ __align__(16) unsigned char smraw[];
  cpx<T>* buf = reinterpret_cast<cpx<T>*>(smraw);
  const int NR = tb.NR, NT = NTPC > 0 ? 2 * NTPC / 3 : tb.NT, NZ = tb.NZ, NTNZ = tb.NTNZ;
  const int NTP = NTPC > 0 ? NTPC : tb.NTP;
  const long long S = tb.S;
  const int lc = threadIdx.x % LC, c = c0 + lc, f = c < 9 * NZ ? c / NZ : -1, l = c - max(f, 0) * NZ, comp = max(f, 0) % 3;
  const int left = max(0, i - IW), right = min(i + IW, NR - 1);
  const int len = right + 1 - left, i0 = i + IW - right;
  const T rinv = tb_rinv<T>(tb, i);
  const T ktsT = tb_kts<T>(tb);
  // the padded middle third is zero
  for (int p = NT / 2 + threadIdx.x / LC; p < NT; p += PS) buf[p * LC + lc] = mk<T>(0, 0);
  const size_t col0 = (size_t)comp * S + l, row0 = (size_t)i * NTNZ + col0;
  const bool live = f >= 0 && NSP_IN_BOUNDS(tb, (size_t)right * NTNZ + col0 + (size_t)(NT - 1) * NZ, 3 * S, BC_THETA_IN);
  const bool mirror = f >= 3 && f < 6 && DR;  // d_r: the mirror the linear pass wrote (the same stencil's bits)
  for (int it = threadIdx.x / LC; it < NT; it += PS) {
    const int m = it < NT / 2 ? it : it - NT;
    const unsigned off = (unsigned)it * (unsigned)NZ;
    cpx<T> v = mk<T>(0, 0);
    if (live) {
      if (f >= 3 && f < 6 && !mirror) {  // derivr_k, mod_radialFD.cu:10-30 (flag 1 for u_r, u_theta; 0 for u_z)
        const int tab = abs((abs(m) % 2) - (comp < 2 ? 1 : 0));
        const T* Dr = dtab<T>(tb) + tab * STEN * NR + STEN * i + i0;
        T sx = 0, sy = 0;
        for (int j = 0; j < len; j++) {
          T de = __ldg(Dr + j);
          cpx<T> a = U.ld((size_t)(left + j) * NTNZ + col0 + off);
          sx += de * a.x;
          sy += de * a.y;
        }
        v = mk<T>(sx, sy);
      } else {
        const float2 a = __ldg((mirror ? DR : U.p) + row0 + off);
        v = mk<T>(a.x, a.y);
        if (f >= 6) {  // derivt_k, mod_deriv.cu:10-21
          const T kt = (T)m * ktsT;
          v = mk<T>(-kt * a.y * rinv, kt * a.x * rinv);
        }
      }
      // mixed form: the mean flow is recorded for the linear pass (member steps) and kept
      // out of the transforms; its terms are added by the linear pass, or for an explicit
      // field by nl_theta_fwd
      if (it == 0 && l == 0) {
        const int slot = f == 0 ? MEAN_V : f == 1 ? MEAN_W : f == 2 ? MEAN_U : f == 4 ? MEAN_WP : f == 5 ? MEAN_UP : -1;
        if (!src_override && slot >= 0) bf.MEAN[((size_t)mloc * NR + i) * MEAN_N + slot] = (float)v.x;
        if (mean_field(f)) v = mk<T>(0, 0);
      }
    }
    buf[(it < NT / 2 ? it : it + NT / 2) * LC + lc] = v;
  }
  __syncthreads();
  theta_fft<T, NTPC, +1>(buf, tb);
  if (f < 0) return;
  const size_t g0 = (((size_t)f * NR + i) * NTP) * NZ + l;
  if (!NSP_IN_BOUNDS(tb, g0 + (size_t)(NTP - 1) * NZ, (size_t)9 * NR * NTP * NZ, BC_THETA_OUT)) return;
  cpx<T>* G = reinterpret_cast<cpx<T>*>(bf.G) + (size_t)mloc * 9 * NR * NTP * NZ + g0;
  for (int p = threadIdx.x / LC; p < NTP; p += PS) G[(size_t)p * NZ] = buf[p * LC + lc];
}

// ---------------------------------------------------------------- z stage
// Field order of the 12 physical arrays: u_r,u_t,u_z, dr u_r,dr u_t,dr u_z,
// dt u_r,dt u_t,dt u_z, dz u_r,dz u_t,dz u_z.  Pair t holds fields (2t, 2t+1).
//
// In place: a warp writes a pair's packed Hermitian spectrum into its line, the passes
// (nsp_fft.cuh) keep a thread's butterflies in registers between their loads and stores, so a
// block holds 6 RPB lines and no second buffer.  That is what large lengths need: at 768 points
// the two-pass kernel's two buffers leave one block of 192 threads on an SM (225 ns per member
// and mode at NR=48 x 32, this kernel 162).  Below, the two-pass kernel's fewer trips through
// shared memory win (192 points: 115 against 140; 576: 176 and 185); the autotuner chooses.
// Threads about the butterflies of a pass; blocks per SM that the registers are limited for
// (768 points: 192 x 5 162, 288 x 4 226, 384 x 2 with two rows 162).
constexpr int zp_threads(int n) { return n == 0 ? 256 : n == 432 ? 288 : n >= 96 ? 192 : 96; }
constexpr int zp_blocks(int n) { return n == 0 ? 1 : n == 432 ? 4 : n >= 96 ? 5 : 8; }
template <typename T, int NZRC, int RPB>
__global__ void __launch_bounds__(zp_threads(NZRC), zp_blocks(NZRC)) nl_z(Tables tb, Bufs bf, const Ctl* ctl, int standalone) {
  constexpr int NTH = zp_threads(NZRC);
  const int mloc = blockIdx.z, i = blockIdx.y, j0 = blockIdx.x * RPB;
  if (!standalone && ctl->phase[tb.mem0 + mloc] < 0) return;
  extern __shared__ __align__(16) unsigned char smraw[];
  cpx<T>* Z = reinterpret_cast<cpx<T>*>(smraw);  // [RPB*6] lines of ZP
  const int NR = tb.NR, NTP = tb.NTP;
  const int NZR = NZRC > 0 ? NZRC : tb.NZR, NZ = NZRC > 0 ? NZRC / 3 + 1 : tb.NZ;
  const int ZP = NZRC > 0 ? line_pad(NZRC - 1) + 1 : NZR;
  const cpx<T>* G = reinterpret_cast<const cpx<T>*>(bf.G) + (size_t)mloc * 9 * NR * NTP * NZ;
  cpx<T>* H = reinterpret_cast<cpx<T>*>(bf.H) + (size_t)mloc * 3 * NR * NTP * NZ;
  const T kzs = tb_kzs<T>(tb);
  const int lane = threadIdx.x & 31;
  // Hermitian-extended spectra, two real fields per complex transform.
  for (int task = threadIdx.x >> 5; task < RPB * 6; task += NTH / 32) {
    const int t = task % 6, rr = task / 6, j = j0 + rr;
    cpx<T>* Zt = Z + (size_t)task * ZP;
    if (j >= NTP || !NSP_IN_BOUNDS(tb, ((size_t)i * NTP + j) * NZ + NZ - 1, (size_t)NR * NTP * NZ, BC_Z_IN)) {
      for (int q = lane; q < NZR; q += 32) Zt[q] = mk<T>(0, 0);
      continue;
    }
    const int fa = 2 * t, fb = 2 * t + 1;  // dz u_c comes from the u_c columns
    const cpx<T>* Ga = G + (((size_t)(fa < 9 ? fa : fa - 9) * NR + i) * NTP + j) * NZ;
    const cpx<T>* Gb = G + (((size_t)(fb < 9 ? fb : fb - 9) * NR + i) * NTP + j) * NZ;
    auto put = [&](int q, cpx<T> a, cpx<T> b) {
      const T kz = kzs * (T)q;
      if (fa >= 9) a = mk<T>(-kz * a.y, kz * a.x);
      if (fb >= 9) b = mk<T>(-kz * b.y, kz * b.x);
      if (q == 0) a.y = b.y = (T)0;  // C2R ignores Im of the k_z = 0 coefficient
      Zt[q] = mk<T>(a.x - b.y, a.y + b.x);
      if (q) Zt[NZR - q] = mk<T>(a.x + b.y, b.x - a.y);
    };
    constexpr int U = 4;  // loads in flight per lane and field
    for (int q0 = 0; q0 < NZ; q0 += 32 * U) {
      cpx<T> a[U], b[U];
#pragma unroll
      for (int k = 0; k < U; k++) {
        const int q = q0 + 32 * k + lane;
        if (q < NZ) a[k] = Ga[q], b[k] = Gb[q];
      }
#pragma unroll
      for (int k = 0; k < U; k++) {
        const int q = q0 + 32 * k + lane;
        if (q < NZ) put(q, a[k], b[k]);
      }
    }
    for (int q = NZ + lane; q <= NZR - NZ; q += 32) Zt[q] = mk<T>(0, 0);
  }
  __syncthreads();
  constexpr int NFWD = (RPB == 2) ? 3 : 2;
  if constexpr (NZRC > 0)
    pass_fft<T, +1, NZRC, RPB * 6, 1, line_pad(NZRC - 1) + 1, false, NTH, NZRC / 3 + 1, 2 * NZRC / 3 - 1, 0, -1>(Z, tw_z<T>(tb));
  else
    fft_batch<T, +1, MAXR, false>(Z, tb.pz, RPB * 6, 1, NZR, tw_z<T>(tb));
  // -(u.grad)u (calcNonlinear_k), packed for the forward transforms:
  // RPB 2: slot0 = (Nr0, Nt0), slot1 = (Nr1, Nt1), slot2 = (Nz0, Nz1); RPB 1: slot0 = (Nr, Nt), slot1 = (Nz, 0).
  const T rinv = tb_rinv<T>(tb, i);
  for (int n = threadIdx.x; n < NZR; n += NTH) {
    T nr[RPB], nt[RPB], nz[RPB];
#pragma unroll
    for (int rr = 0; rr < RPB; rr++) {
      const cpx<T>* Zr = Z + (size_t)rr * 6 * ZP + n;
      cpx<T> a0 = Zr[0], a1 = Zr[ZP], a2 = Zr[2 * ZP], a3 = Zr[3 * ZP], a4 = Zr[4 * ZP], a5 = Zr[5 * ZP];
      T ur = a0.x, ut = a0.y, uz = a1.x;
      T drr = a1.y, drt = a2.x, drz = a2.y, dtr = a3.x, dtt = a3.y, dtz = a4.x, dzr = a4.y, dzt = a5.x, dzz = a5.y;
      T utr = ut * rinv;
      nr[rr] = -(ur * drr + ut * dtr + uz * dzr - ut * utr);
      nt[rr] = -(ur * drt + ut * dtt + uz * dzt + ur * utr);
      nz[rr] = -(ur * drz + ut * dtz + uz * dzz);
    }
    if (RPB == 2) {
      Z[n] = mk<T>(nr[0], nt[0]);
      Z[ZP + n] = mk<T>(nr[RPB - 1], nt[RPB - 1]);
      Z[2 * ZP + n] = mk<T>(nz[0], nz[RPB - 1]);
    } else {
      Z[n] = mk<T>(nr[0], nt[0]);
      Z[ZP + n] = mk<T>(nz[0], (T)0);
    }
  }
  __syncthreads();
  if constexpr (NZRC > 0)
    pass_fft<T, -1, NZRC, NFWD, 1, line_pad(NZRC - 1) + 1, false, NTH, 0, -1, NZRC / 3, 2 * NZRC / 3>(Z, tw_z<T>(tb));
  else
    fft_batch<T, -1, MAXR, false>(Z, tb.pz, NFWD, 1, NZR, tw_z<T>(tb));
  // Unpack: x = a + i b  ->  A_q = (X_q + conj X_{-q})/2,  B_q = (X_q - conj X_{-q})/(2i).
  const int NQ = NZ - 1;
  for (int idx = threadIdx.x; idx < RPB * 3 * NQ; idx += NTH) {
    const int q = idx % NQ, c = (idx / NQ) % 3, rr = idx / (3 * NQ), j = j0 + rr;
    if (j >= NTP) continue;
    int slot;
    bool takeB;
    if (c < 2) { slot = rr; takeB = (c == 1); }
    else { slot = (RPB == 2) ? 2 : 1; takeB = (RPB == 2) && rr == 1; }
    const cpx<T>* X = Z + (size_t)slot * ZP;
    const cpx<T> xq = X[q], xm = X[q ? NZR - q : 0];
    const cpx<T> v = takeB ? mk<T>((T)0.5 * (xq.y + xm.y), (T)-0.5 * (xq.x - xm.x))
                           : mk<T>((T)0.5 * (xq.x + xm.x), (T)0.5 * (xq.y - xm.y));
    if (NSP_IN_BOUNDS(tb, (((size_t)c * NR + i) * NTP + j) * NZ + q, (size_t)3 * NR * NTP * NZ, BC_Z_OUT))
      H[(((size_t)c * NR + i) * NTP + j) * NZ + q] = v;
  }
}

// ---------------------------------------------------------------- z stage, two-pass
// The same z stage with each length-NZR transform split as NZR = N1 x N2 ("four-step"):
//   X[N2 k1 + k2] = sum_n1 w_N1^(n1 k1) [ w_NZR^(n1 k2) sum_n2 x[n1 + N1 n2] w_N2^(n2 k2) ],
// pass A: one thread per (transform, n1) runs the N2-point DFT in registers and
// applies the twiddle; pass B: one thread per (transform, k2) runs the N1-point DFT.
// Between the passes a padded [k2][n1] transpose buffer keeps shared memory free of
// bank conflicts; pass A of the inverse gathers the Hermitian spectra straight from
// G.  Two shared-memory round trips per transform instead of one per radix stage.

// exp(-2 pi i e / 288): every register sub-transform length used (4 .. 32) divides 288.
constexpr int WN = 288;
__constant__ float2 c_wf[WN];
template <typename T> __device__ __forceinline__ cpx<T> wreg(int e);
template <> __device__ __forceinline__ cpx<float> wreg<float>(int e) { float2 w = c_wf[e]; return mk<float>(w.x, w.y); }

// In-register Stockham FFT of length N | WN (every index a compile-time constant
// once unrolled, so the array stays in registers); natural order in and out.
template <typename T, int SIGN, int N, int S = 0, int NS = 1>
__device__ __forceinline__ void reg_fft(cpx<T>* v) {
  if constexpr (S < ct_nstages(N)) {
    constexpr int P = ct_radix(N, S), NB = N / P;
    static_assert(WN % (NS * P) == 0, "sub-transform length must divide WN");
    cpx<T> o[N];
#pragma unroll
    for (int j = 0; j < NB; j++) {
      const int k = j % NS;
      cpx<T> x[P];
#pragma unroll
      for (int q = 0; q < P; q++) x[q] = v[j + q * NB];
      if (NS > 1 && k > 0) {
#pragma unroll
        for (int q = 1; q < P; q++) {
          const cpx<T> w = wreg<T>((q * k * (WN / (NS * P))) % WN);
          x[q] = cmulv(x[q], mk<T>(w.x, SIGN > 0 ? -w.y : w.y));
        }
      }
      dft<T, SIGN, P>(x);
#pragma unroll
      for (int q = 0; q < P; q++) o[(j / NS) * NS * P + k + q * NS] = x[q];
    }
#pragma unroll
    for (int n = 0; n < N; n++) v[n] = o[n];
    reg_fft<T, SIGN, N, S + 1, NS * P>(v);
  }
}

// Spectrum value n (0 <= n < NZR) of a packed pair of fields, Hermitian-extended:
// Ga / Gb are the fields' columns (d_z fields read the u columns and multiply by i k_z).
// Branch-free: the load index is clamped and the value selected.
template <typename T, int NZ, int NZR>
__device__ __forceinline__ cpx<T> z_pair_spec(const cpx<T>* Ga, const cpx<T>* Gb, bool dza, bool dzb, int n, T kzs) {
  const bool direct = n < NZ, mirror = n > NZR - NZ;
  const int qq = direct ? n : (mirror ? NZR - n : 0);
  cpx<T> a = Ga[qq], b = Gb[qq];
  const T kz = kzs * (T)qq;
  if (dza) a = mk<T>(-kz * a.y, kz * a.x);
  if (dzb) b = mk<T>(-kz * b.y, kz * b.x);
  // C2R ignores Im of the k_z = 0 coefficient; the mirrored half is the conjugate.
  const T sy = (qq == 0) ? (T)0 : (mirror ? (T)-1 : (T)1);
  a.y *= sy;
  b.y *= sy;
  const cpx<T> z = mk<T>(a.x - b.y, a.y + b.x);
  return (direct || mirror) ? z : mk<T>(0, 0);
}

// The same for an index range known to be all direct (MIRROR false: q = n) or all
// mirrored (MIRROR true: q = NZR - n, conjugated); q = 0 only where ZERO_OK.
template <typename T, bool MIRROR, bool ZERO_OK>
__device__ __forceinline__ cpx<T> z_pair_spec_in(const cpx<T>* Ga, const cpx<T>* Gb, bool dza, bool dzb, int qq, T kzs) {
  cpx<T> a = Ga[qq], b = Gb[qq];
  const T kz = kzs * (T)qq;
  if (dza) a = mk<T>(-kz * a.y, kz * a.x);
  if (dzb) b = mk<T>(-kz * b.y, kz * b.x);
  if (MIRROR) { a.y = -a.y; b.y = -b.y; }
  if (ZERO_OK && qq == 0) { a.y = (T)0; b.y = (T)0; }
  return mk<T>(a.x - b.y, a.y + b.x);
}

// Pitch (complex values) of a physical row of the two-pass z stage: the smallest
// value >= NZR that is 12 mod 16, so that the rows written by one warp in pass B
// (12 lanes per transform, 8-byte values) fall on disjoint bank ranges.
constexpr int z2_pitch(int nzr) { return nzr + (28 - nzr % 16) % 16; }

template <typename T, int NZRC, int N1, int N2, int R>
__global__ void __launch_bounds__(Z2TH) nl_z2(Tables tb, Bufs bf, const Ctl* ctl, int standalone) {
  static_assert(N1 * N2 == NZRC && R % 2 == 0 && NZRC % 3 == 0, "z split");
  constexpr int NZ = NZRC / 3 + 1;    // NZR = 3 (NZ - 1) (3/2 rule)
  constexpr int NQ = NZ - 1;          // retained z modes of the output
  constexpr int YP = N1 + 1;          // padded transpose row
  constexpr int YT = N2 * YP;         // one transform in the transpose buffer
  constexpr int PS = z2_pitch(NZRC);  // padded physical row (complex pairs)
  constexpr int NF = R + R / 2;       // forward transforms: (N_r, N_t) per row, (N_z, N_z) per row pair
  const int mloc = blockIdx.z, i = blockIdx.y, j0 = blockIdx.x * R;  // NTP % R == 0 (host check)
  if (!standalone && ctl->phase[tb.mem0 + mloc] < 0) return;
  extern __shared__ __align__(16) unsigned char smraw[];
  cpx<T>* Y = reinterpret_cast<cpx<T>*>(smraw);  // [R*6][N2][N1+1]
  cpx<T>* Ph = Y + R * 6 * YT;                   // [R][6][PS]: physical field pairs (2t, 2t+1), then products
  const int NR = tb.NR, NTP = tb.NTP;
  const cpx<T>* G = reinterpret_cast<const cpx<T>*>(bf.G) + (size_t)mloc * 9 * NR * NTP * NZ;
  cpx<T>* H = reinterpret_cast<cpx<T>*>(bf.H) + (size_t)mloc * 3 * NR * NTP * NZ;
  const T kzs = tb_kzs<T>(tb);
  const auto* twz = tw_z<T>(tb);  // exp(-2 pi i e / NZR)
  const size_t fstride = (size_t)NR * NTP * NZ;

  // 1. inverse, pass A (spectra gathered from G)
  for (int task = threadIdx.x; task < R * 6 * N1; task += Z2TH) {
    const int n1 = task % N1, t = (task / N1) % 6, r = task / (6 * N1);
    const cpx<T>* Gi = G + ((size_t)i * NTP + j0 + r) * NZ;
    const int fa = 2 * t, fb = 2 * t + 1;  // d_z u_c (fields 9-11) comes from the u_c columns
    const cpx<T>* Ga = Gi + (size_t)(fa < 9 ? fa : fa - 9) * fstride;
    const cpx<T>* Gb = Gi + (size_t)(fb < 9 ? fb : fb - 9) * fstride;
    if (!NSP_IN_BOUNDS(tb, ((size_t)i * NTP + j0 + r) * NZ + NZ - 1, fstride, BC_Z_IN)) continue;
    cpx<T> x[N2];
#pragma unroll
    for (int n2 = 0; n2 < N2; n2++) {
      // The 16-wide range of n = n1 + N1 n2 is classified at compile time; only a
      // range that straddles a boundary of the Hermitian extension takes the general path.
      const int lo = N1 * n2, hi = lo + N1 - 1;
      if (hi < NZ) x[n2] = z_pair_spec_in<T, false, true>(Ga, Gb, fa >= 9, fb >= 9, n1 + lo, kzs);
      else if (lo > NZRC - NZ) x[n2] = z_pair_spec_in<T, true, false>(Ga, Gb, fa >= 9, fb >= 9, NZRC - n1 - lo, kzs);
      else if (lo >= NZ && hi <= NZRC - NZ) x[n2] = mk<T>(0, 0);  // dealiasing band: no load
      else x[n2] = z_pair_spec<T, NZ, NZRC>(Ga, Gb, fa >= 9, fb >= 9, n1 + lo, kzs);
    }
    reg_fft<T, +1, N2>(x);
    cpx<T>* Yt = Y + (r * 6 + t) * YT + n1;
#pragma unroll
    for (int k2 = 0; k2 < N2; k2++) {
      cpx<T> v = x[k2];
      if (k2 > 0) {
        const auto w = __ldg(twz + n1 * k2);
        v = cmulv(v, mk<T>(w.x, -w.y));
      }
      Yt[k2 * YP] = v;
    }
  }
  __syncthreads();
  // 2. inverse, pass B -> physical point z = N2 k1 + k2 of the pair (2t, 2t+1)
  for (int task = threadIdx.x; task < R * 6 * N2; task += Z2TH) {
    const int k2 = task % N2, t = (task / N2) % 6, r = task / (6 * N2);
    cpx<T> y[N1];
    const cpx<T>* Yt = Y + (r * 6 + t) * YT + k2 * YP;
#pragma unroll
    for (int n1 = 0; n1 < N1; n1++) y[n1] = Yt[n1];
    reg_fft<T, +1, N1>(y);
    cpx<T>* pz = Ph + (r * 6 + t) * PS + k2;
#pragma unroll
    for (int k1 = 0; k1 < N1; k1++) pz[N2 * k1] = y[k1];
  }
  __syncthreads();
  // 3. -(u.grad)u (calcNonlinear_k, mod_io_nonlinear.cu:142-170).  Pairs: (u_r,u_t) (u_z,dr u_r)
  // (dr u_t,dr u_z) (dt u_r,dt u_t) (dt u_z,dz u_r) (dz u_t,dz u_z).  Written back as
  // pair 0 = (N_r, N_t), pair 1 .x = N_z.
  const T rinv = tb_rinv<T>(tb, i);
  for (int task = threadIdx.x; task < R * NZRC; task += Z2TH) {
    const int z = task % NZRC, r = task / NZRC;
    cpx<T>* p = Ph + r * 6 * PS + z;
    const cpx<T> a0 = p[0], a1 = p[PS], a2 = p[2 * PS], a3 = p[3 * PS], a4 = p[4 * PS], a5 = p[5 * PS];
    const T ur = a0.x, ut = a0.y, uz = a1.x;
    const T drr = a1.y, drt = a2.x, drz = a2.y, dtr = a3.x, dtt = a3.y, dtz = a4.x, dzr = a4.y, dzt = a5.x, dzz = a5.y;
    const T utr = ut * rinv;
    p[0] = mk<T>(-(ur * drr + ut * dtr + uz * dzr - ut * utr), -(ur * drt + ut * dtt + uz * dzt + ur * utr));
    p[PS].x = -(ur * drz + ut * dtz + uz * dzz);
  }
  __syncthreads();
  // 4. forward, pass A: transform t < R is (N_r, N_t) of row t; t >= R packs N_z of rows 2(t-R), 2(t-R)+1.
  for (int task = threadIdx.x; task < NF * N1; task += Z2TH) {
    const int n1 = task % N1, t = task / N1;
    cpx<T> x[N2];
    if (t < R) {
      const cpx<T>* pa = Ph + t * 6 * PS + n1;
#pragma unroll
      for (int n2 = 0; n2 < N2; n2++) x[n2] = pa[N1 * n2];
    } else {
      const cpx<T>* pa = Ph + (2 * (t - R) * 6 + 1) * PS + n1;
      const cpx<T>* pb = pa + 6 * PS;
#pragma unroll
      for (int n2 = 0; n2 < N2; n2++) x[n2] = mk<T>(pa[N1 * n2].x, pb[N1 * n2].x);
    }
    reg_fft<T, -1, N2>(x);
    cpx<T>* Yt = Y + t * YT + n1;
#pragma unroll
    for (int k2 = 0; k2 < N2; k2++) {
      cpx<T> v = x[k2];
      if (k2 > 0) {
        const auto w = __ldg(twz + n1 * k2);
        v = cmulv(v, mk<T>(w.x, w.y));
      }
      Yt[k2 * YP] = v;
    }
  }
  __syncthreads();
  // 5. forward, pass B -> spectrum X[N2 k1 + k2] (natural order, over the physical buffer)
  cpx<T>* Xs = Ph;
  for (int task = threadIdx.x; task < NF * N2; task += Z2TH) {
    const int k2 = task % N2, t = task / N2;
    cpx<T> y[N1];
    const cpx<T>* Yt = Y + t * YT + k2 * YP;
#pragma unroll
    for (int n1 = 0; n1 < N1; n1++) y[n1] = Yt[n1];
    reg_fft<T, -1, N1>(y);
#pragma unroll
    for (int k1 = 0; k1 < N1; k1++) Xs[t * PS + N2 * k1 + k2] = y[k1];
  }
  __syncthreads();
  // 6. unpack x = a + i b: A_q = (X_q + conj X_-q)/2, B_q = (X_q - conj X_-q)/(2i); keep q < NZ-1.
  for (int task = threadIdx.x; task < R * 3 * NQ; task += Z2TH) {
    const int q = task % NQ, c = (task / NQ) % 3, r = task / (3 * NQ), j = j0 + r;
    const int slot = c < 2 ? r : R + r / 2;
    const bool takeB = c < 2 ? (c == 1) : (r & 1);
    const cpx<T>* X = Xs + slot * PS;
    const cpx<T> xq = X[q], xm = X[(NZRC - q) % NZRC];
    const cpx<T> v = takeB ? mk<T>((T)0.5 * (xq.y + xm.y), (T)-0.5 * (xq.x - xm.x))
                           : mk<T>((T)0.5 * (xq.x + xm.x), (T)0.5 * (xq.y - xm.y));
    if (NSP_IN_BOUNDS(tb, (((size_t)c * NR + i) * NTP + j) * NZ + q, 3 * fstride, BC_Z_OUT))
      H[(((size_t)c * NR + i) * NTP + j) * NZ + q] = v;
  }
}

// ---------------------------------------------------------------- theta forward
template <typename T, int NTPC>
__global__ void __launch_bounds__(TTH) nl_theta_fwd(Tables tb, Bufs bf, const Ctl* ctl, const double2* src_override,
                                                    const float2* src32_override, double2* dst_override) {
  constexpr int LC = theta_cols(NTPC), PS = TTH / LC;
  const int mloc = blockIdx.z, i = blockIdx.y, c0 = blockIdx.x * LC;
  bool skip;
  const double2* U = member_source(tb, bf, ctl, mloc, src_override, skip);
  if (skip) return;
  extern __shared__ __align__(16) unsigned char smraw[];
  cpx<T>* buf = reinterpret_cast<cpx<T>*>(smraw);
  const int NR = tb.NR, NT = NTPC > 0 ? 2 * NTPC / 3 : tb.NT, NZ = tb.NZ, NTNZ = tb.NTNZ;
  const int NTP = NTPC > 0 ? NTPC : tb.NTP;
  const long long S = tb.S;
  const int lc = threadIdx.x % LC, q = c0 + lc, c = q < 3 * NZ ? q / NZ : -1, l = q - max(c, 0) * NZ;
  const size_t h0 = (((size_t)max(c, 0) * NR + i) * NTP) * NZ + l;
  const cpx<T>* H = reinterpret_cast<const cpx<T>*>(bf.H) + (size_t)mloc * 3 * NR * NTP * NZ + h0;
  const bool live = c >= 0 && l < NZ - 1 &&
                    NSP_IN_BOUNDS(tb, h0 + (size_t)(NTP - 1) * NZ, (size_t)3 * NR * NTP * NZ, BC_THETA_IN);
  for (int p = threadIdx.x / LC; p < NTP; p += PS) buf[p * LC + lc] = live ? H[(size_t)p * NZ] : mk<T>(0, 0);
  __syncthreads();
  theta_fft<T, NTPC, -1>(buf, tb);
  if (c < 0) return;
  // Wall derivative of u_z(0,0) for the mean forcing (pressGrad_k).
  double dwall = 0.0;
  if (c == 2 && l == 0) {
    const double* Dw = tb.D + STEN * (NR - 1) + IW;
    for (int j = 0; j <= IW; j++) dwall += Dw[j] * U[2 * S + (size_t)(NR - 1 - IW + j) * NTNZ].x;
  }
  const T scale = tb_inv_norm<T>(tb);
  const size_t e0 = (size_t)c * S + (size_t)i * NTNZ + l;
  if (!NSP_IN_BOUNDS(tb, e0 + (size_t)(NT - 1) * NZ, 3 * S, BC_THETA_OUT)) return;
  if (!dst_override) {
    // a member's N in the mixed form: FP32 (its values are FP32 numbers), the wall forcing
    // of Re N_z(0,0) kept apart in FP64 -- the same at every level, written by level 0
    if (c == 2 && l == 0 && i == 0 && threadIdx.x < LC) bf.NF[mloc] = -(tb.sscal[4 * member_set(tb, mloc) + 1] * dwall);
    float2* N32 = bf.N32 + (size_t)mloc * 3 * S + e0;
    for (int it = threadIdx.x / LC; it < NT; it += PS) {
      const cpx<T> b = buf[(it < NT / 2 ? it : NTP + it - NT) * LC + lc];
      N32[(size_t)it * NZ] = it == NT / 2 || l == NZ - 1 ? make_float2(0.f, 0.f) : make_float2(b.x * scale, b.y * scale);
    }
    return;
  }
  // explicit field: the mean-flow terms (nsp_state.cuh), from its FP32 copy (a member state's
  // terms are added by the linear pass)
  const float2* U32 = src_override ? src32_override : nullptr;
  Mean32 mf{};
  if (U32) mf = mean_flow32(tb, U32, nullptr, i);
  double2* Nout = dst_override + e0;
  for (int it = threadIdx.x / LC; it < NT; it += PS) {
    const cpx<T> b = buf[(it < NT / 2 ? it : NTP + it - NT) * LC + lc];
    float2 w = make_float2(b.x * scale, b.y * scale);
    if (U32 && it != NT / 2 && l != NZ - 1) {
      const bool zm = it == 0 && l == 0;
      const size_t hq = (size_t)i * NTNZ + (size_t)it * NZ + l;
      const float2 ur = U32[hq], uq = zm ? make_float2(0.f, 0.f) : U32[(c == 2 ? 2 : 1) * S + hq];
      const float kt = (float)(it < NT / 2 ? it : it - NT) * tb.kts32;
      const float2 ml = mean_terms32(mf, c, zm, kt, tb.kzs32 * (float)l, ur, c < 2 ? uq : make_float2(0.f, 0.f),
                                     c == 2 ? uq : make_float2(0.f, 0.f));
      w.x += ml.x;
      w.y += ml.y;
    }
    double2 v = make_double2(f32_to_f64(w.x), f32_to_f64(w.y));  // exact, integer pipe
    if (it == NT / 2 || l == NZ - 1) v = make_double2(0.0, 0.0);
    if (c == 2 && it == 0 && l == 0) v.x -= tb.sscal[4 * member_set(tb, mloc) + 1] * dwall;  // 2/Re
    Nout[(size_t)it * NZ] = v;
  }
}

// ---------------------------------------------------------------- launcher
template <typename T, int NTPC>
static void launch_theta(const Tables& tb, const Bufs& bf, Ctl* dctl, const double2* src, const float2* src32,
                         double2* dst, cudaStream_t st, int mask, int nm) {
  constexpr int LC = theta_cols(NTPC);
  size_t sm = sizeof(cpx<T>) * tb.NTP * LC;
  if (mask & 1) {
    dim3 g((9 * tb.NZ + LC - 1) / LC, tb.NR, nm);
    nl_theta_inv<T, NTPC><<<g, TTH, sm, st>>>(tb, bf, dctl, src, src32);
  }
  if (mask & 4) {
    dim3 g((3 * tb.NZ + LC - 1) / LC, tb.NR, nm);
    nl_theta_fwd<T, NTPC><<<g, TTH, sm, st>>>(tb, bf, dctl, src, src32, dst);
  }
}

template <typename T, int NZRC, int RPB>
static void launch_z(const Tables& tb, const Bufs& bf, Ctl* dctl, bool standalone, cudaStream_t st, int nm) {
  size_t sm = sizeof(cpx<T>) * 6 * RPB * (NZRC > 0 ? line_pad(NZRC - 1) + 1 : tb.NZR);
  dim3 g((tb.NTP + RPB - 1) / RPB, tb.NR, nm);
  nl_z<T, NZRC, RPB><<<g, zp_threads(NZRC), sm, st>>>(tb, bf, dctl, standalone ? 1 : 0);
}

template <typename T, int NZRC, int N1, int N2, int R>
static constexpr size_t z2_smem() {
  return sizeof(cpx<T>) * ((size_t)R * 6 * N2 * (N1 + 1) + (size_t)R * 6 * z2_pitch(NZRC));
}

template <typename T, int NZRC, int N1, int N2, int R>
static void launch_z2(const Tables& tb, const Bufs& bf, Ctl* dctl, bool standalone, cudaStream_t st, int nm) {
  dim3 g((tb.NTP + R - 1) / R, tb.NR, nm);
  nl_z2<T, NZRC, N1, N2, R><<<g, Z2TH, z2_smem<T, NZRC, N1, N2, R>(), st>>>(tb, bf, dctl, standalone ? 1 : 0);
}

// Theta rows per block of the in-place z kernel.
constexpr int zp_rows(int n) { return n == 0 || n == 384 || n >= 576 ? 1 : 2; }
// Two-pass z stage: (NZR, N1, N2, rows per block); the setup-time autotuner picks among
// the splits and the in-place passes per shape (which win at 432 and 768 points, so those have no
// split).  The run-time kernel, bound by its index arithmetic, takes 1066 us where the 18 x 9 split
// takes 89 (7 members of NR=61, 36 x 54 modes); its theta transforms (NTP = 54) 274 and 85 us where
// the compiled ones take 80 and 27.  Of the accepted lengths 6, 12, 18 and 324 points stay with it.
#define NSP_Z2_LIST(X) X(24, 4, 6, 2) X(36, 6, 6, 2) X(48, 8, 6, 2) X(54, 9, 6, 2) X(72, 12, 6, 2) \
  X(108, 9, 12, 2) X(108, 12, 9, 2) X(144, 12, 12, 2) X(162, 9, 18, 2) X(162, 18, 9, 2) X(216, 18, 12, 2) \
  X(288, 16, 18, 2) X(288, 12, 24, 2) X(96, 8, 12, 2) X(96, 12, 8, 2) X(192, 16, 12, 2) \
  X(192, 12, 16, 2) X(384, 16, 24, 2) X(384, 24, 16, 2) X(576, 24, 24, 2)

int z_variants(int NZR, int NTP, bool fp32) {
  int n = 0;
#define NSP_Z2_COUNT(len, a, b, r) n += (NZR == len && NTP % r == 0);
  if (fp32) { NSP_Z2_LIST(NSP_Z2_COUNT) }
#undef NSP_Z2_COUNT
  return n;
}

// The two-pass kernel where one is compiled for the length (the FP32 default, measured
// faster than the in-place kernel on the bench shape), else the in-place one.
int z_default_variant(int NZR, int NTP, bool fp32) {
  const char* e = getenv("NSP_Z2");
  if (e && e[0] == '0') return 0;
  return fp32 && z_variants(NZR, NTP, true) > 0 ? 1 : 0;
}

std::string z_variant_name(int NZR, int NTP, bool fp32, int v) {
  // variant 0: the compiled passes in place, or the run-time plan's radix stages
  if (!fp32) return nzr_compiled(NZR) ? "passes, 64-bit fixed point" : "radix, 64-bit fixed point";
  std::string s = nzr_compiled(NZR) ? "in-place passes" : "radix";
  if (v <= 0) return s;
  int k = 0;
#define NSP_Z2_NAME(len, a, b, r) \
  if (NZR == len && NTP % r == 0 && ++k == v) s = "two-pass " #a "x" #b;
  NSP_Z2_LIST(NSP_Z2_NAME)
#undef NSP_Z2_NAME
  return s;
}

template <typename T>
static void launch_nl_t(const Tables& tb, const Bufs& bf, Ctl* dctl, const double2* src, const float2* src32,
                        double2* dst, cudaStream_t st, int mask) {
  int nm = src ? 1 : tb.nmem;
  const bool tc = tb.tc_theta;  // mixed form: theta transforms on the tensor cores
  if ((mask & 1) && tc) {
    launch_theta_tc(tb, bf, dctl, 0, src, src32, dst, st);
  } else if (mask & 1) {
    switch (tb.NTP) {
#define NSP_CASE_T(n) \
  case n: launch_theta<T, n>(tb, bf, dctl, src, src32, dst, st, 1, nm); break;
      NSP_NTP_LIST(NSP_CASE_T)
#undef NSP_CASE_T
      default: launch_theta<T, 0>(tb, bf, dctl, src, src32, dst, st, 1, nm);
    }
  }
  if (mask & 2) {
    bool done = false;
    // the group's z-stage variant: the k-th two-pass split of the length, or (0) in place
    if (tb.z_variant > 0) {
      int k = 0;
#define NSP_CASE_Z2(n, a, b, r)                                                      \
  if (!done && tb.NZR == n && tb.NTP % r == 0 && ++k == tb.z_variant) {             \
    launch_z2<T, n, a, b, r>(tb, bf, dctl, src != nullptr, st, nm);                  \
    done = true;                                                                     \
  }
      NSP_Z2_LIST(NSP_CASE_Z2)
#undef NSP_CASE_Z2
    }
    if (!done) {
      switch (tb.NZR) {
#define NSP_CASE_Z(n) \
  case n: launch_z<T, n, zp_rows(n)>(tb, bf, dctl, src != nullptr, st, nm); break;
        NSP_NZR_LIST(NSP_CASE_Z)
#undef NSP_CASE_Z
        default: launch_z<T, 0, zp_rows(0)>(tb, bf, dctl, src != nullptr, st, nm);
      }
    }
  }
  if ((mask & 4) && tc) {
    launch_theta_tc(tb, bf, dctl, 1, src, src32, dst, st);
  } else if (mask & 4) {
    switch (tb.NTP) {
#define NSP_CASE_T(n) \
  case n: launch_theta<T, n>(tb, bf, dctl, src, src32, dst, st, 4, nm); break;
      NSP_NTP_LIST(NSP_CASE_T)
#undef NSP_CASE_T
      default: launch_theta<T, 0>(tb, bf, dctl, src, src32, dst, st, 4, nm);
    }
  }
}

int kernels_per_nonlinear() { return 3; }

template <typename T>
static void configure_t() {
  const int big = 200 * 1024;
#define NSP_CFG_T(n)                                                                            \
  cudaFuncSetAttribute(nl_theta_inv<T, n>, cudaFuncAttributeMaxDynamicSharedMemorySize, big); \
  cudaFuncSetAttribute(nl_theta_fwd<T, n>, cudaFuncAttributeMaxDynamicSharedMemorySize, big);
  NSP_NTP_LIST(NSP_CFG_T)
  NSP_CFG_T(0)
#undef NSP_CFG_T
#define NSP_CFG_Z(n) cudaFuncSetAttribute(nl_z<T, n, zp_rows(n)>, cudaFuncAttributeMaxDynamicSharedMemorySize, big);
  NSP_NZR_LIST(NSP_CFG_Z)
  NSP_CFG_Z(0)
#undef NSP_CFG_Z
}

void configure_transform_kernels() {
  configure_t<float>();
#define NSP_CFG_Z2F(n, a, b, r)                                                          \
  cudaFuncSetAttribute(nl_z2<float, n, a, b, r>, cudaFuncAttributeMaxDynamicSharedMemorySize, \
                       (int)z2_smem<float, n, a, b, r>());
  NSP_Z2_LIST(NSP_CFG_Z2F)
#undef NSP_CFG_Z2F
  // Twiddles of the register sub-transforms, exp(-2 pi i e / WN), from long double.
  float2 wf[WN];
  for (int e = 0; e < WN; e++) {
    const long double a = -6.283185307179586476925286766559L * (long double)e / (long double)WN;
    wf[e] = make_float2((float)cosl(a), (float)sinl(a));
  }
  cudaMemcpyToSymbol(c_wf, wf, sizeof(wf));
}

bool transform_supported(int NTP, int NZR) {
  FftPlan pt, pz;
  make_plan(NTP, pt);
  make_plan(NZR, pz);
  return (ntp_compiled(NTP) || max_butterflies(pt, 16) <= RT_TASKS) && (nzr_compiled(NZR) || max_butterflies(pz, 6) <= RT_TASKS);
}

void launch_nonlinear(const Tables& tb, const Bufs& bf, Ctl* dctl, bool mixed, const double2* src, double2* dst,
                      cudaStream_t st, int mask, const float2* src32) {
  if (mixed) launch_nl_t<float>(tb, bf, dctl, src, src32, dst, st, mask);
  else launch_nonlinear_fx(tb, bf, dctl, src, dst, st, mask);
}

__global__ void to_f32_k(const double2* __restrict__ src, float2* __restrict__ dst, long long n) {
  for (long long h = blockIdx.x * (long long)blockDim.x + threadIdx.x; h < n; h += (long long)gridDim.x * blockDim.x) {
    double2 a = src[h];
    dst[h] = make_float2(f64_to_f32(a.x), f64_to_f32(a.y));
  }
}

// FP32 mirror U32 and its radial derivative DR32 of a group's state (step start):
// the same conversion and stencil as the linear pass's stages I and J.  A block holds
// a tile of MR levels x MK modes of one member component (line), plus IW levels on
// either side, converted once into shared memory; the stencil reads the tile.  Lanes
// run along the modes (coalesced); lines are S = NR*NT*NZ < 2^31 values.
constexpr int MIR_K = 32, MIR_R = 24, MIR_T = 256;
__global__ void __launch_bounds__(MIR_T) mirror_k(Tables tb, const double2* __restrict__ U, float2* __restrict__ U32,
                                                  float2* __restrict__ DR32) {
  __shared__ float2 tile[(MIR_R + 2 * IW) * MIR_K];
  const int NR = tb.NR, NT = tb.NT, NZ = tb.NZ, NTNZ = tb.NTNZ;
  const int kx = threadIdx.x % MIR_K, ry = threadIdx.x / MIR_K;
  constexpr int RY = MIR_T / MIR_K;
  const int k = blockIdx.x * MIR_K + kx, r0 = blockIdx.y * MIR_R;
  const int lo = max(0, r0 - IW), hi = min(NR, r0 + MIR_R + IW), r1 = min(NR, r0 + MIR_R);
  const int it = k / NZ, m = it < NT / 2 ? it : it - NT, par_m = abs(m) % 2;
  for (int line = blockIdx.z; line < 3 * tb.nmem; line += gridDim.z) {
    const size_t base = (size_t)line * tb.S;
    __syncthreads();  // the previous line's tile has been read
    if (k < NTNZ)
      for (int r = lo + ry; r < hi; r += RY) {
        if (!NSP_IN_BOUNDS(tb, base + (size_t)r * NTNZ + k, (size_t)3 * tb.nmem * tb.S, BC_MIRROR)) break;
        const double2 a = U[base + (size_t)r * NTNZ + k];
        tile[(r - lo) * MIR_K + kx] = make_float2(f64_to_f32(a.x), f64_to_f32(a.y));
      }
    __syncthreads();
    if (k >= NTNZ) continue;
    const int tab = abs(par_m - (line % 3 < 2 ? 1 : 0));
    for (int i = r0 + ry; i < r1; i += RY) {
      const size_t h = base + (size_t)i * NTNZ + k;
      if (!NSP_IN_BOUNDS(tb, h, (size_t)3 * tb.nmem * tb.S, BC_MIRROR)) break;
      U32[h] = tile[(i - lo) * MIR_K + kx];
      const int left = max(0, i - IW), right = min(i + IW, NR - 1), len = right + 1 - left, i0 = i + IW - right;
      const float* Dr = tb.D32 + tab * STEN * NR + STEN * i + i0;
      DR32[h] = dr32_line(Dr, left, len, [&](int row) { return tile[(row - lo) * MIR_K + kx]; });
    }
  }
}

void launch_mirror(const Tables& tb, const double2* U, float2* U32, float2* DR32, cudaStream_t st) {
  const dim3 grid((unsigned)((tb.NTNZ + MIR_K - 1) / MIR_K), (unsigned)((tb.NR + MIR_R - 1) / MIR_R),
                  (unsigned)std::min(3 * tb.nmem, 65535));
  mirror_k<<<grid, MIR_T, 0, st>>>(tb, U, U32, DR32);
}

void launch_to_f32(const double2* src, float2* dst, long long n, cudaStream_t st) {
  int blocks = (int)std::min<long long>((n + 255) / 256, 152LL * 16);
  to_f32_k<<<blocks, 256, 0, st>>>(src, dst, n);
}

// x = hi + lo with hi = fl32(x), lo = fl32(x - hi) (x - hi is exact in FP64): the
// double-float form of set-up tables, about 48 bits of x.
__global__ void split_df_k(const double* __restrict__ src, float2* __restrict__ dst, long long n) {
  for (long long h = blockIdx.x * (long long)blockDim.x + threadIdx.x; h < n; h += (long long)gridDim.x * blockDim.x) {
    const double x = src[h];
    const float hi = f64_to_f32(x);
    dst[h] = make_float2(hi, f64_to_f32(x - f32_to_f64(hi)));
  }
}

void launch_split_df(const double* src, float2* dst, long long n, cudaStream_t st) {
  int blocks = (int)std::min<long long>((n + 255) / 256, 152LL * 16);
  split_df_k<<<blocks, 256, 0, st>>>(src, dst, n);
}

// The banded-LU factor tables [kk][NR][NFAC][NTNZ] in double-float and FP32 for the mixed
// form's solves, [kk][NR][NTNZ][NPACK]: a row's factors of a mode together, in the order the
// solves use them (L(i-3), L(i-2), L(i-1), 0, U(i+3), U(i+2), U(i+1), 1/U_ii).  The backward
// entries U(i, i+j) are pre-divided by U_ii: a backward row is then x_i = y_i / U_ii -
// sum U'_ij x_j, the division applied to y_i off the row-to-row dependency chain.  n: rows
// times modes.
__global__ void split_fac_k(const double* __restrict__ fac, float2* __restrict__ dfo, float* __restrict__ f32o,
                            long long n, int NTNZ) {
  for (long long h = blockIdx.x * (long long)blockDim.x + threadIdx.x; h < n; h += (long long)gridDim.x * blockDim.x) {
    const double* f = fac + h / NTNZ * NFAC * NTNZ + h % NTNZ;
    const double d = f[3 * (long long)NTNZ];
#pragma unroll
    for (int e = 0; e < NPACK; e++) {
      const double x = e < 3 ? f[(long long)e * NTNZ] : e == 3 ? 0.0 : e < 7 ? f[(long long)(10 - e) * NTNZ] * d : d;
      const float hi = f64_to_f32(x);
      dfo[h * NPACK + e] = make_float2(hi, f64_to_f32(x - f32_to_f64(hi)));
      f32o[h * NPACK + e] = hi;
    }
  }
}

void launch_split_fac(const double* fac, float2* dfo, float* f32o, long long n, int NTNZ, cudaStream_t st) {
  int blocks = (int)std::min<long long>((n + 255) / 256, 152LL * 16);
  split_fac_k<<<blocks, 256, 0, st>>>(fac, dfo, f32o, n, NTNZ);
}

}  // namespace nsp
