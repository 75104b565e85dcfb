// nsp_cross.cu -- the cross-section diagnostics, transforms in 64-bit fixed point (nsp_fx.cuh).
#include <algorithm>

#include "nsp_bounds.cuh"
#include "nsp_fx.cuh"
#include "nsp_internal.h"

namespace nsp {

// Cross-section diagnostics of a state (wrt_qcr / wrt_ucr with q0kernel_k, u0kernel_k,
// q1kernel_k and intq, mod_io_nonlinear.cu:54-117, 572-660 and mod_cublasflux.cu:119-130):
// at every physical axial point z_n,
//   q(z_n) = sum_i rdr_i (1/NTP) sum_theta (u_r^2 + u_theta^2),   u(z_n) = the same with u_z^2.
// (The reference's periodic Simpson rule in theta with unit weights sums to the plain mean.)
// The theta mean is taken by Parseval: with q_mu(z) the theta spectrum of the real field at
// (r_i, z), it is q_0^2 + 2 sum_{0<mu<NT/2} |q_mu|^2 + |P|^2 / 2, P the mode -NT/2 that has no
// partner.  q_mu is one complex transform along z of c_{mu,l} at +l and conj c_{-mu,l} at -l
// (their mean at l = 0), P / 2 one of c_{-NT/2,l}, c_{.,0} halved.
//
// A block takes one component at one level of a member and runs its NT/2 + 1 transforms
// NB at a time in fixed point, a warp filling each line, a thread adding the squares of its
// points in the order of mu; cross_sum_k then adds the levels in order.  64 members of 48 x 32
// x 64 modes, with the other diagnostics of a sample: 41.7 ms as direct sums in FP64 (NT NZ NZR
// complex products per level and component), 1.35 ms with transforms.
template <int NZRC, int RPB>
__global__ void __launch_bounds__(z_threads(NZRC), z_blocks(NZRC)) fx_cross(Tables tb, const double2* __restrict__ U,
                                                                            double* __restrict__ part) {
  constexpr int ZTH = z_threads(NZRC), NB = RPB * 6, KZ = NZRC > 0 ? (NZRC + ZTH - 1) / ZTH : 4;
  static_assert(NZRC > 0 || 6 * (KZ * ZTH / 4) >= RT_TASKS, "points of a run-time length (radices up to 4)");
  const int NTH = NZRC > 0 ? ZTH : blockDim.x;
  const int i = blockIdx.x, c = blockIdx.y, lane = threadIdx.x & 31;
  extern __shared__ __align__(16) unsigned char smraw[];
  cpx<fx>* Z = reinterpret_cast<cpx<fx>*>(smraw);  // [NB] lines of ZP
  __shared__ int sE[NB];
  const int NT = tb.NT, NZR = NZRC > 0 ? NZRC : tb.NZR, NZ = NZRC > 0 ? NZRC / 3 + 1 : tb.NZ;
  const int ZP = NZRC > 0 ? line_pitch(NZRC) : NZR;
  const double2* row = U + ((size_t)blockIdx.z * 3 + c) * tb.S + (size_t)i * tb.NTNZ;
  double ms[KZ];
#pragma unroll
  for (int k = 0; k < KZ; k++) ms[k] = 0.0;
  for (int mu0 = 0; mu0 <= NT / 2; mu0 += NB) {
    const int nb = min(NB, NT / 2 + 1 - mu0);
    // both lines of a pair copied asynchronously into the line they become (fx_z)
    auto plus = [&](int mu) { return row + (size_t)mu * NZ; };
    auto minus = [&](int mu) { return row + (size_t)(mu ? NT - mu : 0) * NZ; };  // (mu = NT/2: the same line, unused)
    auto live = [&](int mu) {  // both lines inside the member's component
      const int last = mu && mu < NT / 2 ? NT - mu : mu;
      return NSP_IN_BOUNDS(tb, (size_t)i * tb.NTNZ + (size_t)last * NZ + NZ - 1, tb.S, BC_DIAG);
    };
    auto raw2 = [&](int q) { return q < NZ - 2 ? NZ + q : NZR - NZ + 2 + q; };
    if constexpr (NZRC > 0) {
      for (int b = threadIdx.x >> 5; b < nb; b += NTH / 32) {
        if (!live(mu0 + b)) continue;
        cpx<fx>* Zt = Z + (size_t)b * ZP;
        const double2 *P = plus(mu0 + b), *M = minus(mu0 + b);
        for (int q = lane; q < NZ; q += 32) {
          cp_async16(Zt + q, P + q);
          cp_async16(Zt + raw2(q), M + q);
        }
      }
      cp_async_commit();
      cp_async_wait<0>();
      __syncwarp();
    }
    for (int b = threadIdx.x >> 5; b < nb; b += NTH / 32) {
      const int mu = mu0 + b;
      cpx<fx>* Zt = Z + (size_t)b * ZP;
      if (!live(mu)) {
        for (int q = lane; q < NZR; q += 32) Zt[q] = mk<fx>(0, 0);
        if (lane == 0) sE[b] = 0;
        continue;
      }
      const double2* raw = reinterpret_cast<const double2*>(Zt);
      const double2 *P = plus(mu), *M = minus(mu);
      auto at_p = [&](int q) { return NZRC > 0 ? raw[q] : P[q]; };
      auto at_m = [&](int q) { return NZRC > 0 ? raw[raw2(q)] : M[q]; };
      const bool pair = mu < NT / 2;
      FxSum sum;
#pragma unroll 1
      for (int q = lane; q < NZ; q += 32) {
        const double2 a = at_p(q), m = at_m(q);
        sum.add(fx_key(a.x), fx_key(a.y));
        if (pair) sum.add(fx_key(m.x), fx_key(m.y));
      }
      const int E = sum.warp_exponent();
      if (lane == 0) sE[b] = E;
#pragma unroll 1
      for (int q = lane; q < NZ; q += 32) {
        const double2 a = at_p(q), m = at_m(q);
        const cpx<fx> x = mk<fx>(fx_from(a.x, E), fx_from(a.y, E));
        const cpx<fx> y = pair ? mk<fx>(fx_from(m.x, E), -fx_from(m.y, E)) : mk<fx>(0, 0);
        if (q) {
          Zt[q] = x;
          Zt[NZR - q] = y;
        } else {
          Zt[0] = mk<fx>(fx_half(x.x + y.x), fx_half(x.y + y.y));
        }
      }
      __syncwarp();  // the second line's slots have been read
      for (int q = NZ + lane; q <= NZR - NZ; q += 32) Zt[q] = mk<fx>(0, 0);
    }
    __syncthreads();
    if constexpr (NZRC > 0)
      pass_fft<fx, +1, NZRC, NB, 1, line_pitch(NZRC), false, ZTH, NZRC / 3 + 1, 2 * NZRC / 3 - 1, 0, -1>(Z, tb.tw_zx, nb);
    else
      fft_batch<fx, +1, MAXRZ, false>(Z, tb.pz, nb, 1, NZR, tb.tw_zx);
#pragma unroll
    for (int k = 0; k < KZ; k++) {
      const int n = threadIdx.x + k * NTH;
      if (n < NZR)
        for (int b = 0; b < nb; b++) {
          const double2 v = fx_value(Z[(size_t)b * ZP + n], sE[b]);
          if (mu0 + b == 0) ms[k] = 0.5 * (v.x * v.x);
          else ms[k] = fma(v.x, v.x, fma(v.y, v.y, ms[k]));
        }
    }
    __syncthreads();
  }
  const size_t o0 = (((size_t)blockIdx.z * 3 + c) * tb.NR + i) * NZR;
  if (!NSP_IN_BOUNDS(tb, o0 + NZR - 1, (size_t)gridDim.z * 3 * tb.NR * NZR, BC_CROSS)) return;
  double* o = part + o0;
#pragma unroll
  for (int k = 0; k < KZ; k++) {
    const int n = threadIdx.x + k * NTH;
    if (n < NZR) o[n] = 2.0 * ms[k];
  }
}

// The radial quadrature of one member's mean squares [3][NR][NZR], in level order:
// out[member][0] = sum_i rdr_i (ms_r + ms_theta), out[member][1] = sum_i rdr_i ms_z.
__global__ void cross_sum_k(Tables tb, const double* __restrict__ part, double* __restrict__ out) {
  const int n = blockIdx.x * blockDim.x + threadIdx.x, NR = tb.NR, NZR = tb.NZR;
  if (n >= NZR) return;
  const double* p = part + (size_t)blockIdx.y * 3 * NR * NZR + n;
  double q = 0.0, u = 0.0;
  constexpr int B = 8;  // rows whose loads are in flight together (one by one: a chain of NR latencies)
  for (int i0 = 0; i0 < NR; i0 += B) {
    double w[B], r[B], t[B], z[B];
#pragma unroll
    for (int k = 0; k < B; k++) {
      const size_t i = min(i0 + k, NR - 1);
      w[k] = tb.rdr[i];
      r[k] = p[i * NZR];
      t[k] = p[(NR + i) * NZR];
      z[k] = p[(2 * NR + i) * NZR];
    }
#pragma unroll
    for (int k = 0; k < B; k++) {
      if (i0 + k < NR) {
        q += w[k] * (r[k] + t[k]);
        u += w[k] * z[k];
      }
    }
  }
  if (!NSP_IN_BOUNDS(tb, ((size_t)blockIdx.y * 2 + 1) * NZR + n, (size_t)gridDim.y * 2 * NZR, BC_CROSS)) return;
  out[((size_t)blockIdx.y * 2) * NZR + n] = q;
  out[((size_t)blockIdx.y * 2 + 1) * NZR + n] = u;
}

template <int NZRC, int RPB>
static void launch_cross_t(const Tables& tb, const double2* U, double* part, cudaStream_t st, int nmem) {
  const size_t sm = sizeof(cpx<fx>) * 6 * RPB * (NZRC > 0 ? line_pitch(NZRC) : tb.NZR);
  fx_cross<NZRC, RPB><<<dim3(tb.NR, 3, nmem), NZRC > 0 ? z_threads(NZRC) : rt_z_threads(tb.NZR), sm, st>>>(tb, U, part);
}

void launch_diag_cross(const Tables& tb, const double2* U, double* part, double* out, cudaStream_t st, int nmem) {
  for (int m0 = 0; m0 < nmem; m0 += 65535) {  // (grid limits)
    const int nm = std::min(nmem - m0, 65535);
    const double2* Um = U + (size_t)m0 * 3 * tb.S;
    switch (tb.NZR) {
#define NSP_CASE_C(n) \
  case n: launch_cross_t<n, z_rows(n)>(tb, Um, part, st, nm); break;
      NSP_NZR_LIST(NSP_CASE_C)
#undef NSP_CASE_C
      default: launch_cross_t<0, z_rows(0)>(tb, Um, part, st, nm);
    }
    cross_sum_k<<<dim3((tb.NZR + 127) / 128, nm), 128, 0, st>>>(tb, part, out);
    part += (size_t)nm * 3 * tb.NR * tb.NZR;
    out += (size_t)nm * 2 * tb.NZR;
  }
}

void configure_cross_kernels() {
#define NSP_CFG_C(n) cudaFuncSetAttribute(fx_cross<n, z_rows(n)>, cudaFuncAttributeMaxDynamicSharedMemorySize, 200 * 1024);
  NSP_NZR_LIST(NSP_CFG_C)
  NSP_CFG_C(0)
#undef NSP_CFG_C
}

}  // namespace nsp
