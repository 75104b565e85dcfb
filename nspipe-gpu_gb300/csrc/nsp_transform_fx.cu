// nsp_transform_fx.cu -- the FP64 form's transforms: FP64 fields in and out, the FFTs
// themselves in 64-bit fixed point on the integer pipe (nsp_fx.cuh).
//
// The same three kernels per evaluation of the nonlinear term as the mixed form's
// (nsp_transform.cu), over the same arrays G and H (complex FP64 here):
//
//   fx_theta_inv  per (member, level, 16 (field, l) columns): u, d_r u (FP64 stencil) and
//                 i m u / r, inverse transforms along theta -> G;
//   fx_z          per (member, level, theta rows): 12 Hermitian z spectra, packed two real
//                 fields per complex inverse transform, -(u.grad)u in FP64, packed forward
//                 transforms, unpack -> H;
//   fx_theta_fwd  per (member, level, 16 (component, l) columns): forward transforms, scale,
//                 retained modes, wall-shear forcing -> N (FP64).
//
// Each transform line gets its own scale: the values are loaded in FP64, the largest
// exponent and then the sum of magnitudes are reduced over the line as integers (so the
// scale, and with it every bit, is independent of the order), and the line is converted
// in place.
// Bound: integer issue, the barriers between the passes and instruction fetch (z stage, 16
// members of NR=48 x 32 x 64 modes: issue 70%, ALU pipe 64%, FMA pipe 31%, FP64 pipe 26%).  FP64 transforms
// were bound by the FP64 pipe alone.  Per launch there, before and after: theta-inverse 903 ->
// 285 us, z stage 3457 -> 699 us, theta-forward 283 -> 84 us; one member of 48 x 64 x 256
// modes: 530 -> 160, 2154 -> 450, 168 -> 47 us.
#include <cmath>
#include <cstdio>
#include <cstdlib>

#include "nsp_bounds.cuh"
#include "nsp_fx.cuh"
#include "nsp_internal.h"
#include "nsp_state.cuh"

namespace nsp {

namespace {

constexpr int MAXR = 4;   // register rounds of the run-time FFT along theta
constexpr int TTH = 256;  // threads of the theta kernels
static_assert(MAXR * TTH >= RT_TASKS, "register rounds of the run-time FFT");

// Columns per block of the theta kernels: 32 (512-byte rows of G) while that leaves several
// blocks' columns in shared memory, so that a pass has about as many butterflies as threads.
constexpr int theta_lc(int ntp) { return ntp == 0 || ntp >= 96 ? 16 : 32; }
template <int NTPC, int SIGN>
__device__ __forceinline__ void theta_fft(cpx<fx>* buf, const Tables& tb) {
  constexpr int LC = theta_lc(NTPC);
  if constexpr (NTPC > 0) {
    // zero (inverse) or dropped (forward) middle third
    constexpr int A = NTPC / 3, B = 2 * NTPC / 3 - 1;
    if constexpr (SIGN > 0) pass_fft<fx, SIGN, NTPC, LC, LC, 1, true, TTH, A, B, 0, -1>(buf, tb.tw_tx);
    else pass_fft<fx, SIGN, NTPC, LC, LC, 1, true, TTH, 0, -1, A, B>(buf, tb.tw_tx);
  } else {
    fft_batch<fx, SIGN, MAXR, true>(buf, tb.pt, LC, LC, 1, tb.tw_tx);
  }
}

// Scale of a column whose V values per thread (threads t and t + LC, t + 2 LC ... hold one
// column) are in registers: its exponent, from its largest key and its sum of magnitudes.
// skey / ssum: zeroed shared arrays of LC.
template <int LC, int V>
__device__ __forceinline__ int column_exponent(const double2 (&g)[V], unsigned* skey, unsigned* ssum) {
  const int lc = threadIdx.x % LC;
  unsigned kmax = 0u, sum = 0u;
#pragma unroll
  for (int k = 0; k < V; k++) kmax = max(kmax, max(fx_key(g[k].x), fx_key(g[k].y)));
  if (LC < 32) kmax = max(kmax, __shfl_xor_sync(0xFFFFFFFFu, kmax, LC));
  if ((threadIdx.x & 31) < LC) atomicMax(skey + lc, kmax);
  __syncthreads();
  kmax = skey[lc];
#pragma unroll
  for (int k = 0; k < V; k++) sum += fx_mag(fx_key(g[k].x), kmax >> 20) + fx_mag(fx_key(g[k].y), kmax >> 20);
  if (LC < 32) sum += __shfl_xor_sync(0xFFFFFFFFu, sum, LC);
  if ((threadIdx.x & 31) < LC) atomicAdd(ssum + lc, sum);
  __syncthreads();
  return fx_exponent((int)(kmax >> 20), ssum[lc]);
}

// The same for a run-time length: the block's columns, in FP64 at buf (element p of column
// lc at p LC + lc), to fixed point in place; kmax: the thread's largest key.
template <int LC>
__device__ __forceinline__ int columns_to_fx(double2* buf, int total, unsigned kmax, unsigned* skey, unsigned* ssum) {
  const int lc = threadIdx.x % LC;
  if (LC < 32) kmax = max(kmax, __shfl_xor_sync(0xFFFFFFFFu, kmax, LC));
  if ((threadIdx.x & 31) < LC) atomicMax(skey + lc, kmax);
  __syncthreads();
  kmax = skey[lc];
  const unsigned emax = kmax >> 20;
  unsigned sum = 0;
  for (int idx = threadIdx.x; idx < total; idx += TTH) {
    const double2 v = buf[idx];
    sum += fx_mag(fx_key(v.x), emax) + fx_mag(fx_key(v.y), emax);
  }
  if (LC < 32) sum += __shfl_xor_sync(0xFFFFFFFFu, sum, LC);
  if ((threadIdx.x & 31) < LC) atomicAdd(ssum + lc, sum);
  __syncthreads();
  const int E = fx_exponent((int)emax, ssum[lc]);
  cpx<fx>* o = reinterpret_cast<cpx<fx>*>(buf);
  for (int idx = threadIdx.x; idx < total; idx += TTH) {
    const double2 v = buf[idx];
    o[idx] = mk<fx>(fx_from(v.x, E), fx_from(v.y, E));
  }
  __syncthreads();
  return E;
}

}  // namespace

// ---------------------------------------------------------------- theta inverse
template <int NTPC>
__global__ void __launch_bounds__(TTH) fx_theta_inv(Tables tb, Bufs bf, const Ctl* ctl, const double2* src_override) {
  const int mloc = blockIdx.z, i = blockIdx.y, c0 = blockIdx.x * theta_lc(NTPC);
  bool skip;
  const double2* U = member_source(tb, bf, ctl, mloc, src_override, skip);
  if (skip) return;
  extern __shared__ __align__(16) unsigned char smraw[];
  double2* buf = reinterpret_cast<double2*>(smraw);
  constexpr int LC = theta_lc(NTPC);
  __shared__ unsigned skey[LC], ssum[LC];
  const int NR = tb.NR, NT = NTPC > 0 ? 2 * NTPC / 3 : tb.NT, NZ = tb.NZ, NTNZ = tb.NTNZ;
  const int NTP = NTPC > 0 ? NTPC : tb.NTP;
  const long long S = tb.S;
  const int lc = threadIdx.x % LC, c = c0 + lc;
  const int f = c < 9 * NZ ? c / NZ : -1, l = c % NZ;
  if (threadIdx.x < LC) skey[threadIdx.x] = ssum[threadIdx.x] = 0u;
  __syncthreads();
  const int left = max(0, i - IW), right = min(i + IW, NR - 1);
  const int len = right + 1 - left, i0 = i + IW - right;
  const double rinv = tb.rinv[i];
  const size_t col0 = (size_t)max(f, 0) % 3 * S + l;
  const bool live = f >= 0 && NSP_IN_BOUNDS(tb, (size_t)right * NTNZ + col0 + (size_t)(NT - 1) * NZ, 3 * S, BC_THETA_IN);
  auto value = [&](int it) {
    double2 v = make_double2(0.0, 0.0);
    if (!live) return v;
    const int m = it < NT / 2 ? it : it - NT;
    const double2* col = U + col0 + (unsigned)it * (unsigned)NZ;
    if (f >= 3 && f < 6) {  // derivr_k, mod_radialFD.cu:10-30 (flag 1 for u_r, u_theta; 0 for u_z)
      const int tab = abs((abs(m) % 2) - (f < 5 ? 1 : 0));
      const double* Dr = tb.D + tab * STEN * NR + STEN * i + i0;
      for (int j = 0; j < len; j++) {
        const double de = __ldg(Dr + j);
        const double2 a = col[(size_t)(left + j) * NTNZ];
        v.x += de * a.x;
        v.y += de * a.y;
      }
    } else {
      v = col[(size_t)i * NTNZ];
      if (f >= 6) {  // derivt_k, mod_deriv.cu:10-21
        const double kt = tb.kts * (double)m;
        v = make_double2(-kt * v.y * rinv, kt * v.x * rinv);
      }
    }
    return v;
  };
  // the padded middle third is zero
  cpx<fx>* X = reinterpret_cast<cpx<fx>*>(buf);
  constexpr int PS = TTH / LC;
  const int t0 = threadIdx.x / LC;
  for (int p = NT / 2 + t0; p < NT; p += PS) X[p * LC + lc] = mk<fx>(0, 0);
  int E;
  if constexpr (NTPC > 0) {
    constexpr int V = (2 * NTPC / 3 + PS - 1) / PS;
    double2 g[V];
#pragma unroll
    for (int k = 0; k < V; k++) {
      const int it = t0 + k * PS;
      g[k] = it < NT ? value(it) : make_double2(0.0, 0.0);
    }
    E = column_exponent<LC, V>(g, skey, ssum);
#pragma unroll
    for (int k = 0; k < V; k++) {
      const int it = t0 + k * PS;
      if (it < NT) X[(it < NT / 2 ? it : it + NT / 2) * LC + lc] = mk<fx>(fx_from(g[k].x, E), fx_from(g[k].y, E));
    }
    __syncthreads();
  } else {
    unsigned kmax = 0u;
    for (int it = t0; it < NT; it += PS) {
      const double2 v = value(it);
      kmax = max(kmax, max(fx_key(v.x), fx_key(v.y)));
      buf[(it < NT / 2 ? it : it + NT / 2) * LC + lc] = v;
    }
    E = columns_to_fx<LC>(buf, NTP * LC, kmax, skey, ssum);
  }
  theta_fft<NTPC, +1>(X, tb);
  if (f < 0) return;
  const size_t g0 = (((size_t)f * NR + i) * NTP) * NZ + l;
  if (!NSP_IN_BOUNDS(tb, g0 + (size_t)(NTP - 1) * NZ, (size_t)9 * NR * NTP * NZ, BC_THETA_OUT)) return;
  double2* G = reinterpret_cast<double2*>(bf.G) + (size_t)mloc * 9 * NR * NTP * NZ + g0;
  for (int p = t0; p < NTP; p += PS) G[(unsigned)p * (unsigned)NZ] = fx_value(X[p * LC + lc], E);
}

// ---------------------------------------------------------------- z stage
// Field order of the 12 physical arrays: u_r,u_t,u_z, dr u_r,dr u_t,dr u_z,
// dt u_r,dt u_t,dt u_z, dz u_r,dz u_t,dz u_z (the last three from the u columns times the
// whole number l, their physical values times 2 pi / LZ).  Pair t holds fields (2t, 2t+1); a
// warp takes a pair of a row: both half spectra's scales, then their packed Hermitian extension.
template <int NZRC, int RPB>
__global__ void __launch_bounds__(z_threads(NZRC), z_blocks(NZRC)) fx_z(Tables tb, Bufs bf, const Ctl* ctl, int standalone) {
  const int NTH = NZRC > 0 ? z_threads(NZRC) : blockDim.x;
  const int mloc = blockIdx.z, i = blockIdx.y, j0 = blockIdx.x * RPB;
  if (!standalone && ctl->phase[tb.mem0 + mloc] < 0) return;
  extern __shared__ __align__(16) unsigned char smraw[];
  cpx<fx>* Z = reinterpret_cast<cpx<fx>*>(smraw);  // [RPB*6] lines of ZP
  __shared__ int sE[RPB * 12];                     // exponents of the physical fields
  __shared__ unsigned skey[RPB * 3], ssum[RPB * 3];
  const int NR = tb.NR, NTP = tb.NTP;
  const int NZR = NZRC > 0 ? NZRC : tb.NZR, NZ = NZRC > 0 ? NZRC / 3 + 1 : tb.NZ;
  const int ZP = NZRC > 0 ? line_pitch(NZRC) : NZR;
  const double2* G = reinterpret_cast<const double2*>(bf.G) + (size_t)mloc * 9 * NR * NTP * NZ;
  double2* H = reinterpret_cast<double2*>(bf.H) + (size_t)mloc * 3 * NR * NTP * NZ;
  const int lane = threadIdx.x & 31;
  if (threadIdx.x < RPB * 3) skey[threadIdx.x] = ssum[threadIdx.x] = 0u;
  // A pair's two columns are copied asynchronously into its own line -- field 2t at slot q,
  // field 2t+1 at NZ + q, its last two values behind the line -- where the Hermitian extension
  // then replaces them: slot q is written by the lane that has read it, the mirrored half
  // starts behind the second field's slots (2 NZ - 2 = NZR - NZ + 1).  (Run-time lengths read
  // G in place.)
  auto live_row = [&](int rr) {
    return j0 + rr < NTP && NSP_IN_BOUNDS(tb, ((size_t)i * NTP + j0 + rr) * NZ + NZ - 1, (size_t)NR * NTP * NZ, BC_Z_IN);
  };
  auto column = [&](int fld, int rr) {  // dz u_c comes from the u_c columns
    return G + (((size_t)(fld >= 9 ? fld - 9 : fld) * NR + i) * NTP + j0 + rr) * NZ;
  };
  auto raw2 = [&](int q) { return q < NZ - 2 ? NZ + q : NZR - NZ + 2 + q; };
  if constexpr (NZRC > 0) {
    for (int task = threadIdx.x >> 5; task < RPB * 6; task += NTH / 32) {
      const int t = task % 6, rr = task / 6;
      if (!live_row(rr)) continue;
      cpx<fx>* Zt = Z + (size_t)task * ZP;
      const double2 *a = column(2 * t, rr), *b = column(2 * t + 1, rr);
      for (int q = lane; q < NZ; q += 32) {
        cp_async16(Zt + q, a + q);
        cp_async16(Zt + raw2(q), b + q);
      }
    }
    cp_async_commit();
    cp_async_wait<0>();
    __syncwarp();
  }
  for (int task = threadIdx.x >> 5; task < RPB * 6; task += NTH / 32) {
    const int t = task % 6, rr = task / 6;
    cpx<fx>* Zt = Z + (size_t)task * ZP;
    if (!live_row(rr)) {
      for (int q = lane; q < NZR; q += 32) Zt[q] = mk<fx>(0, 0);
      if (lane < 2) sE[rr * 12 + 2 * t + lane] = 0;
      continue;
    }
    const double2* Gr[2] = {column(2 * t, rr), column(2 * t + 1, rr)};
    const double2* raw = reinterpret_cast<const double2*>(Zt);
    const bool dz[2] = {2 * t >= 9, 2 * t + 1 >= 9};
    auto load = [&](int h, int q) { return NZRC > 0 ? raw[h ? raw2(q) : q] : Gr[h][q]; };
    // A dz field's coefficient is the u column's times the whole number l, formed exactly in
    // its conversion; its share of the key is rounded up.  Loops kept short: this kernel
    // is bound by instruction fetch as much as by issue.
    auto value = [&](int h, int q) {
      const double2 v = load(h, q);
      return q ? v : make_double2(v.x, 0.0);  // C2R ignores Im of the k_z = 0 coefficient
    };
    int E[2];
#pragma unroll
    for (int h = 0; h < 2; h++) {
      FxSum sum;
      if (dz[h]) {
#pragma unroll 1
        for (int q = lane ? lane : 32; q < NZ; q += 32) {
          const double2 v = load(h, q);
          const unsigned w = q > 1 ? (unsigned)(32 - __clz(q - 1)) << 20 : 0u;
          const unsigned kx = fx_key(v.x), ky = fx_key(v.y);
          sum.add(min(max(kx, 0x100000u) + w, 0x7FF00000u), min(max(ky, 0x100000u) + w, 0x7FF00000u));
        }
      } else {
#pragma unroll 1
        for (int q = lane; q < NZ; q += 32) {
          const double2 v = value(h, q);
          sum.add(fx_key(v.x), fx_key(v.y));
        }
      }
      E[h] = sum.warp_exponent();
      if (E[h] != FX_BAD) E[h] += 1;  // two-sided
      if (lane == 0) sE[rr * 12 + 2 * t + h] = E[h];
    }
#pragma unroll 1
    for (int q = lane; q < NZ; q += 32) {
      const double2 v = value(0, q), w = value(1, q);
      cpx<fx> x, y;
      if (dz[1]) {  // pairs (dt u_z, dz u_r) and (dz u_theta, dz u_z)
        x = dz[0] ? muli<fx, +1>(mk<fx>(fx_from_times(v.x, q, E[0]), fx_from_times(v.y, q, E[0])))
                  : mk<fx>(fx_from(v.x, E[0]), fx_from(v.y, E[0]));
        y = muli<fx, +1>(mk<fx>(fx_from_times(w.x, q, E[1]), fx_from_times(w.y, q, E[1])));
      } else {
        x = mk<fx>(fx_from(v.x, E[0]), fx_from(v.y, E[0]));
        y = mk<fx>(fx_from(w.x, E[1]), fx_from(w.y, E[1]));
      }
      Zt[q] = mk<fx>(x.x - y.y, x.y + y.x);
      if (q) Zt[NZR - q] = mk<fx>(x.x + y.y, y.x - x.y);
    }
    __syncwarp();  // the second field's slots have been read
    for (int q = NZ + lane; q <= NZR - NZ; q += 32) Zt[q] = mk<fx>(0, 0);
  }
  __syncthreads();
  constexpr int BS = NZRC > 0 ? line_pitch(NZRC) : 0;
  if constexpr (NZRC > 0)
    pass_fft<fx, +1, NZRC, RPB * 6, 1, BS, false, z_threads(NZRC), NZRC / 3 + 1, 2 * NZRC / 3 - 1, 0, -1>(Z, tb.tw_zx);
  else
    fft_batch<fx, +1, MAXRZ, false>(Z, tb.pz, RPB * 6, 1, NZR, tb.tw_zx);
  // -(u.grad)u (calcNonlinear_k) in FP64, packed for the forward transforms:
  // RPB 2: slot0 = (Nr0, Nt0), slot1 = (Nr1, Nt1), slot2 = (Nz0, Nz1); RPB 1: slot0 = (Nr, Nt), slot1 = (Nz, 0).
  const double rinv = tb.rinv[i], kzs = tb.kzs;
  double2* P = reinterpret_cast<double2*>(Z);
  unsigned kn[RPB * 3];
#pragma unroll
  for (int e = 0; e < RPB * 3; e++) kn[e] = 0u;
  for (int n = threadIdx.x; n < NZR; n += NTH) {
    double nr[RPB], nt[RPB], nz[RPB];
#pragma unroll
    for (int rr = 0; rr < RPB; rr++) {
      const cpx<fx>* Zr = Z + (size_t)rr * 6 * ZP + n;
      const int* e = sE + rr * 12;
      double u[12];
      int top = 0;
#pragma unroll
      for (int t = 0; t < 6; t++) {
        const cpx<fx> a = Zr[t * ZP];
        top = max(top, max(e[2 * t], e[2 * t + 1]));
        u[2 * t] = fx_to(a.x, e[2 * t] - FX_BITS);
        u[2 * t + 1] = fx_to(a.y, e[2 * t + 1] - FX_BITS);
      }
      const double ur = u[0], ut = u[1], uz = u[2] * kzs, utr = ut * rinv;
      nr[rr] = -(ur * u[3] + ut * u[6] + uz * u[9] - ut * utr);
      nt[rr] = -(ur * u[4] + ut * u[7] + uz * u[10] + ur * utr);
      nz[rr] = -(ur * u[5] + ut * u[8] + uz * u[11]);
      if (top == FX_BAD) nr[rr] = nt[rr] = nz[rr] = fx_nan();
      kn[rr * 3] = max(kn[rr * 3], fx_key(nr[rr]));
      kn[rr * 3 + 1] = max(kn[rr * 3 + 1], fx_key(nt[rr]));
      kn[rr * 3 + 2] = max(kn[rr * 3 + 2], fx_key(nz[rr]));
    }
    if (RPB == 2) {
      P[n] = make_double2(nr[0], nt[0]);
      P[ZP + n] = make_double2(nr[RPB - 1], nt[RPB - 1]);
      P[2 * ZP + n] = make_double2(nz[0], nz[RPB - 1]);
    } else {
      P[n] = make_double2(nr[0], nt[0]);
      P[ZP + n] = make_double2(nz[0], 0.0);
    }
  }
#pragma unroll
  for (int e = 0; e < RPB * 3; e++) {
    const unsigned k = __reduce_max_sync(0xFFFFFFFFu, kn[e]);
    if (lane == 0) atomicMax(skey + e, k);
  }
  __syncthreads();
  // value e = 3 rr + c of the products sits in slot s_of(e), part p_of(e)
  constexpr int NFWD = (RPB == 2) ? 3 : 2;
  auto s_of = [](int e) { return e % 3 < 2 ? e / 3 : (RPB == 2 ? 2 : 1); };
  auto p_of = [](int e) { return e % 3 < 2 ? e % 3 : (RPB == 2 ? e / 3 : 0); };
  unsigned sn[RPB * 3];
#pragma unroll
  for (int e = 0; e < RPB * 3; e++) sn[e] = 0u;
  for (int n = threadIdx.x; n < NZR; n += NTH) {
#pragma unroll
    for (int s = 0; s < NFWD; s++) {
      const double2 v = P[s * ZP + n];
#pragma unroll
      for (int e = 0; e < RPB * 3; e++)
        if (s_of(e) == s) sn[e] += fx_mag(fx_key(p_of(e) ? v.y : v.x), skey[e] >> 20);
    }
  }
#pragma unroll
  for (int e = 0; e < RPB * 3; e++) {
    sn[e] = __reduce_add_sync(0xFFFFFFFFu, sn[e]);
    if (lane == 0) atomicAdd(ssum + e, sn[e]);
  }
  __syncthreads();
  int EN[RPB * 3];
#pragma unroll
  for (int e = 0; e < RPB * 3; e++) EN[e] = fx_exponent((int)(skey[e] >> 20), ssum[e]);
  for (int n = threadIdx.x; n < NZR; n += NTH) {
#pragma unroll
    for (int s = 0; s < NFWD; s++) {
      const double2 v = P[s * ZP + n];
      cpx<fx> x = mk<fx>(0, 0);
#pragma unroll
      for (int e = 0; e < RPB * 3; e++)
        if (s_of(e) == s) (p_of(e) ? x.y : x.x) = fx_from(p_of(e) ? v.y : v.x, EN[e]);
      Z[s * ZP + n] = x;
    }
  }
  __syncthreads();
  if constexpr (NZRC > 0)
    pass_fft<fx, -1, NZRC, NFWD, 1, BS, false, z_threads(NZRC), 0, -1, NZRC / 3, 2 * NZRC / 3>(Z, tb.tw_zx);
  else
    fft_batch<fx, -1, MAXRZ, false>(Z, tb.pz, NFWD, 1, NZR, tb.tw_zx);
  // Unpack: x = a + i b  ->  A_q = (X_q + conj X_{-q})/2,  B_q = (X_q - conj X_{-q})/(2i).
  const int NQ = NZ - 1;
  for (int idx = threadIdx.x; idx < RPB * 3 * NQ; idx += NTH) {
    const int q = idx % NQ, e = idx / NQ, c = e % 3, rr = e / 3, j = j0 + rr;
    if (j >= NTP) continue;
    const cpx<fx>* X = Z + (size_t)s_of(e) * ZP;
    const cpx<fx> xq = X[q], xm = X[q ? NZR - q : 0];
    const cpx<fx> v = p_of(e) ? mk<fx>(xq.y + xm.y, xm.x - xq.x) : mk<fx>(xq.x + xm.x, xq.y - xm.y);
    const int E = fx_exponent((int)(skey[e] >> 20), ssum[e]);
    const size_t h = (((size_t)c * NR + i) * NTP + j) * NZ + q;
    if (NSP_IN_BOUNDS(tb, h, (size_t)3 * NR * NTP * NZ, BC_Z_OUT)) H[h] = fx_value(v, E == FX_BAD ? E : E - 1);
  }
}

// ---------------------------------------------------------------- theta forward
template <int NTPC>
__global__ void __launch_bounds__(TTH) fx_theta_fwd(Tables tb, Bufs bf, const Ctl* ctl, const double2* src_override,
                                                    double2* dst_override) {
  const int mloc = blockIdx.z, i = blockIdx.y, c0 = blockIdx.x * theta_lc(NTPC);
  bool skip;
  const double2* U = member_source(tb, bf, ctl, mloc, src_override, skip);
  if (skip) return;
  extern __shared__ __align__(16) unsigned char smraw[];
  double2* buf = reinterpret_cast<double2*>(smraw);
  constexpr int LC = theta_lc(NTPC);
  __shared__ unsigned skey[LC], ssum[LC];
  const int NR = tb.NR, NT = NTPC > 0 ? 2 * NTPC / 3 : tb.NT, NZ = tb.NZ, NTNZ = tb.NTNZ;
  const int NTP = NTPC > 0 ? NTPC : tb.NTP;
  const long long S = tb.S;
  const int lc = threadIdx.x % LC, q = c0 + lc;
  const int c = q < 3 * NZ ? q / NZ : -1, l = q % NZ;
  if (threadIdx.x < LC) skey[threadIdx.x] = ssum[threadIdx.x] = 0u;
  __syncthreads();
  const size_t h0 = (((size_t)max(c, 0) * NR + i) * NTP) * NZ + l;
  const double2* H = reinterpret_cast<const double2*>(bf.H) + (size_t)mloc * 3 * NR * NTP * NZ + h0;
  const bool live = c >= 0 && l < NZ - 1 &&
                    NSP_IN_BOUNDS(tb, h0 + (size_t)(NTP - 1) * NZ, (size_t)3 * NR * NTP * NZ, BC_THETA_IN);
  double2* Nout = dst_override ? dst_override : bf.N + (size_t)mloc * 3 * S;
  cpx<fx>* X = reinterpret_cast<cpx<fx>*>(buf);
  constexpr int PS = TTH / LC;
  const int t0 = threadIdx.x / LC;
  int E;
  if constexpr (NTPC > 0) {
    constexpr int V = (NTPC + PS - 1) / PS;
    double2 g[V];
#pragma unroll
    for (int k = 0; k < V; k++) {
      const int p = t0 + k * PS;
      g[k] = live && p < NTP ? H[(unsigned)p * (unsigned)NZ] : make_double2(0.0, 0.0);
    }
    E = column_exponent<LC, V>(g, skey, ssum);
#pragma unroll
    for (int k = 0; k < V; k++)
      if (t0 + k * PS < NTP) X[(t0 + k * PS) * LC + lc] = mk<fx>(fx_from(g[k].x, E), fx_from(g[k].y, E));
    __syncthreads();
  } else {
    unsigned kmax = 0u;
    for (int p = t0; p < NTP; p += PS) {
      const double2 v = live ? H[(unsigned)p * (unsigned)NZ] : make_double2(0.0, 0.0);
      kmax = max(kmax, max(fx_key(v.x), fx_key(v.y)));
      buf[p * LC + lc] = v;
    }
    E = columns_to_fx<LC>(buf, NTP * LC, kmax, skey, ssum);
  }
  theta_fft<NTPC, -1>(X, tb);
  if (c < 0) return;
  // Wall derivative of u_z(0,0) for the mean forcing (pressGrad_k).
  double dwall = 0.0;
  if (c == 2 && l == 0) {
    const double* Dw = tb.D + STEN * (NR - 1) + IW;
    for (int j = 0; j <= IW; j++) dwall += Dw[j] * U[2 * S + (size_t)(NR - 1 - IW + j) * NTNZ].x;
  }
  for (int idx = threadIdx.x; idx < NT * LC; idx += TTH) {
    const int it = idx / LC, p = it < NT / 2 ? it : NTP + it - NT;
    double2 v = fx_value(X[p * LC + lc], E);
    v.x *= tb.inv_norm;
    v.y *= tb.inv_norm;
    if (it == NT / 2 || l == NZ - 1) v = make_double2(0.0, 0.0);
    if (c == 2 && it == 0 && l == 0) v.x -= tb.sscal[4 * member_set(tb, mloc) + 1] * dwall;  // 2/Re
    const size_t o = c * S + (size_t)i * NTNZ + (size_t)it * NZ + l;
    if (NSP_IN_BOUNDS(tb, o, 3 * S, BC_THETA_OUT)) Nout[o] = v;
  }
}

// ---------------------------------------------------------------- launcher
template <int NTPC>
static void launch_theta_fx(const Tables& tb, const Bufs& bf, Ctl* dctl, const double2* src, double2* dst,
                            cudaStream_t st, int mask, int nm) {
  constexpr int LC = theta_lc(NTPC);
  const size_t sm = sizeof(double2) * tb.NTP * LC;
  if (mask & 1)
    fx_theta_inv<NTPC><<<dim3((9 * tb.NZ + LC - 1) / LC, tb.NR, nm), TTH, sm, st>>>(tb, bf, dctl, src);
  if (mask & 4)
    fx_theta_fwd<NTPC><<<dim3((3 * tb.NZ + LC - 1) / LC, tb.NR, nm), TTH, sm, st>>>(tb, bf, dctl, src, dst);
}

template <int NZRC, int RPB>
static void launch_z_fx(const Tables& tb, const Bufs& bf, Ctl* dctl, bool standalone, cudaStream_t st, int nm) {
  const size_t sm = sizeof(cpx<fx>) * 6 * RPB * (NZRC > 0 ? line_pitch(NZRC) : tb.NZR);
  fx_z<NZRC, RPB><<<dim3((tb.NTP + RPB - 1) / RPB, tb.NR, nm), NZRC > 0 ? z_threads(NZRC) : rt_z_threads(tb.NZR), sm, st>>>(
      tb, bf, dctl, standalone ? 1 : 0);
}

void launch_nonlinear_fx(const Tables& tb, const Bufs& bf, Ctl* dctl, const double2* src, double2* dst,
                         cudaStream_t st, int mask) {
  const int nm = src ? 1 : tb.nmem;
  auto theta = [&](int which) {
    switch (tb.NTP) {
#define NSP_CASE_T(n) \
  case n: launch_theta_fx<n>(tb, bf, dctl, src, dst, st, which, nm); break;
      NSP_NTP_LIST(NSP_CASE_T)
#undef NSP_CASE_T
      default: launch_theta_fx<0>(tb, bf, dctl, src, dst, st, which, nm);
    }
  };
  if (mask & 1) theta(1);
  if (mask & 2) {
    switch (tb.NZR) {
#define NSP_CASE_Z(n) \
  case n: launch_z_fx<n, z_rows(n)>(tb, bf, dctl, src != nullptr, st, nm); break;
      NSP_NZR_LIST(NSP_CASE_Z)
#undef NSP_CASE_Z
      default: launch_z_fx<0, z_rows(0)>(tb, bf, dctl, src != nullptr, st, nm);
    }
  }
  if (mask & 4) theta(4);
}

void configure_transform_fx_kernels() {
  const int big = 200 * 1024;
#define NSP_CFG_T(n)                                                                              \
  cudaFuncSetAttribute(fx_theta_inv<n>, cudaFuncAttributeMaxDynamicSharedMemorySize, big); \
  cudaFuncSetAttribute(fx_theta_fwd<n>, cudaFuncAttributeMaxDynamicSharedMemorySize, big);
  NSP_NTP_LIST(NSP_CFG_T)
  NSP_CFG_T(0)
#undef NSP_CFG_T
#define NSP_CFG_Z(n) cudaFuncSetAttribute(fx_z<n, z_rows(n)>, cudaFuncAttributeMaxDynamicSharedMemorySize, big);
  NSP_NZR_LIST(NSP_CFG_Z)
  NSP_CFG_Z(0)
#undef NSP_CFG_Z
}

// exp(-2 pi i e / n) as fractions of 2^62 in signed 32-bit halves: (Re h, Re l, Im h, Im l).
std::vector<int4> fx_twiddles(int n) {
  // Octant reduction with long-double sine and cosine of angles up to pi/4, exact at the
  // quarter turns; on hosts whose long double has 64 bits the last one or two bits of the
  // fractions are rounding, 2^-62 of 1.
  const long double PI_L = 3.141592653589793238462643383279502884L, one = 4611686018427387904.0L;  // 2^62
  auto halves = [&](long double v, int& h, int& l) {
    long long x = llrintl(v * one);
    if ((int)x == (int)0x80000000) x += 1;  // keeps the low half's negation in range
    l = (int)x;
    h = (int)(x >> 32) - (l >> 31);
  };
  std::vector<int4> w(n);
  struct Angle {  // cosine and sine of (pi/2) rest / n, each rest evaluated once (128-bit long doubles are slow)
    bool set = false;
    long double c, s;
  };
  std::vector<Angle> first(n / 2 + 1);
  for (int e = 0; e < n; e++) {
    const int q = (int)(4LL * e / n);                      // quarter turn
    const int rest = (int)(4LL * e - (long long)q * n);    // angle within it: (pi/2) rest / n
    Angle& a = first[2 * rest <= n ? rest : n - rest];
    if (!a.set) {
      const long double x = PI_L * 0.5L * (long double)(2 * rest <= n ? rest : n - rest) / (long double)n;
      a = Angle{true, cosl(x), sinl(x)};
    }
    const long double c = 2 * rest <= n ? a.c : a.s, s = 2 * rest <= n ? a.s : a.c;
    const long double re[4] = {c, -s, -c, s}, im[4] = {-s, -c, s, c};
    int4& o = w[e];
    halves(re[q], o.x, o.y);
    halves(im[q], o.z, o.w);
  }
  return w;
}

}  // namespace nsp
