// fluid_plain.cuh - per-mode arithmetic of the reference-structured FP64 form,
// shared by its z kernels (compile-time and run-time sizes) and axis passes.
// sym[2 t] = cos(2 pi t / n) - 1.
#pragma once
#include "common.cuh"
#include "selm_kernels.h"

namespace selm {

// p_hat / (sum_d 2(cos(2 pi i_d/N_d) - 1)/dx^2), zero mode -> 0 (cuda/SELM_Kernel.cu:3-34)
__device__ __forceinline__ double2 poisson_mode(double2 v, const double* __restrict__ sym, int i, int j, int k,
                                                double dxsq) {
  if (i == 0 && j == 0 && k == 0) return make_double2(0.0, 0.0);
  const double coef = 2.0 * (sym[2 * i] + sym[2 * j] + sym[2 * k]) / dxsq;
  return make_double2(v.x / coef, v.y / coef);
}

// Half-spectrum draw of cuda/SELM_Kernel.cu:37-85 with Philox instead of a
// per-mode XORWOW state: amplitude sqrt(lambda_h)/sqrt(2) on re and im, or
// (sqrt(lambda_h), 0) on self-conjugate modes.  noise_mode 1 (exact) scales
// the non-self-conjugate modes of the x=0 / x=Nx/2 planes by sqrt(2) so the
// Hermitian average the c2r takes keeps the full variance.  The forcing's
// prefactor (cuda/SELM_Eulerian_Period.cu:141) is in na.scale.
__device__ __forceinline__ void noise_mode_draw(const NoiseArgs& na, uint64_t step, const double* __restrict__ sym,
                                                int n, int nh, int i, int j, int k, double2* out, int ostep) {
  const double coef = na.scale * sqrt(-2.0 * (sym[2 * i] + sym[2 * j] + sym[2 * k]) / na.dxsq);
  const bool selfc = (k == 0 || 2 * k == n) && (j == 0 || 2 * j == n) && (i == 0 || 2 * i == n);
  const bool edge = i == 0 || 2 * i == n;
  const double re = (selfc || (na.noise_mode == 1 && edge)) ? coef : coef * 0.7071067811865476;
  const double im = selfc ? 0.0 : re;
  const uint32_t q = (uint32_t)(((long)k * n + j) * nh + i);
#pragma unroll
  for (int d = 0; d < 3; d++) {
    double z0, z1;
    philox_normal2(na.rk, q, (uint32_t)d, step, z0, z1);
    out[d * ostep] = make_double2(z0 * re, z1 * im);
  }
}

}  // namespace selm
