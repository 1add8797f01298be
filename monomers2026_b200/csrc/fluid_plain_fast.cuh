// fluid_plain_fast.cuh - the z passes of the reference-structured FP64 form for
// compile-time sizes N = N1 N2 (four-step FFT, as fluid_fused_fast.cuh).
#pragma once
#include "fft_fast.cuh"
#include "fluid_fused_fast.cuh"
#include "fluid_plain.cuh"
#include "fluid_plane.cuh"

namespace selm {

// inverse z FFT of NL lines whose modes lie at dpos(k) (element t of line l at
// A[t NL + l]): the second factor's pass here, the first factor's to global
// memory through store(l, plane, value)
template <int N, int N1, int NL, int TPB> __device__ __forceinline__ void z_inverse_b(double2* A, const double2* tw) {
  constexpr int N2 = N / N1;
  for (int u = threadIdx.x; u < NL * N1; u += TPB) {
    const int l = u % NL, k1 = u / NL;
    double2 v[N2];
#pragma unroll
    for (int j = 0; j < N2; j++) v[j] = A[(N2 * k1 + j) * NL + l];
    fftk::dft<N2, +1>(v);
#pragma unroll
    for (int n2 = 1; n2 < N2; n2++) {
      double2 w = tw[n2 * k1];
      w.y = -w.y;
      v[n2] = cmul(v[n2], w);
    }
#pragma unroll
    for (int n2 = 0; n2 < N2; n2++) A[(N2 * k1 + n2) * NL + l] = v[n2];
  }
}
template <int N, int N1, int NL, int WB, int TPB>
__device__ __forceinline__ void z_inverse_a(const double2* A, double2* __restrict__ work, long plane, long col0, int wn) {
  constexpr int N2 = N / N1;
  for (int u = threadIdx.x; u < NL * N2; u += TPB) {
    const int l = u % NL, n2 = u / NL, c = l / WB, w = l % WB;
    if (w >= wn) continue;
    double2 v[N1];
#pragma unroll
    for (int k1 = 0; k1 < N1; k1++) v[k1] = A[(N2 * k1 + n2) * NL + l];
    fftk::dft<N1, +1>(v);
    double2* d = work + ((long)c * N + n2) * plane + col0 + w;
#pragma unroll
    for (int n1 = 0; n1 < N1; n1++) d[n1 * (N2 * plane)] = v[n1];
  }
}

// Columns per block of the Poisson pass: 16 (256-byte runs) while two blocks
// per SM remain, then fewer.
template <int N> constexpr int poisson_columns() {
  constexpr long ncol = (long)N * (N / 2 + 1);
  return ncol / 16 >= 296 ? 16 : (ncol / 8 >= 148 ? 8 : 4);
}

// z FFT, Poisson solve, inverse z FFT of one component: the second factor's
// DFT, the division and the second factor's inverse DFT in registers, so a
// column goes through shared memory twice
template <int N, int N1, int WB, int TPB>
__global__ void __launch_bounds__(TPB) k_z_poisson_fast(double2* work, const double2* __restrict__ twz,
                                                        const double* __restrict__ sym, double dxsq) {
  constexpr int N2 = N / N1, NH = N / 2 + 1;
  constexpr long plane = (long)N * NH;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  double2* A = reinterpret_cast<double2*>(smem_raw);
  double2* tw = A + N * WB;
  const long col0 = (long)blockIdx.x * WB;
  const int wn = (int)min((long)WB, plane - col0);
  for (int t = threadIdx.x; t < N; t += TPB) tw[t] = twz[t];
  previous_done();
  __syncthreads();
  for (int u = threadIdx.x; u < WB * N2; u += TPB) {
    const int l = u % WB, n2 = u / WB;
    double2 v[N1];
#pragma unroll
    for (int n1 = 0; n1 < N1; n1++)
      v[n1] = l < wn ? work[(N2 * n1 + n2) * plane + col0 + l] : make_double2(0.0, 0.0);
    fftk::dft<N1, -1>(v);
#pragma unroll
    for (int k1 = 0; k1 < N1; k1++) A[(N2 * k1 + n2) * WB + l] = (k1 == 0) ? v[0] : cmul(v[k1], tw[n2 * k1]);
  }
  __syncthreads();
  for (int u = threadIdx.x; u < WB * N1; u += TPB) {
    const int l = u % WB, k1 = u / WB;
    const int col = (int)col0 + min(l, wn - 1), j = col / NH, i = col - j * NH;
    double2 v[N2];
#pragma unroll
    for (int n2 = 0; n2 < N2; n2++) v[n2] = A[(N2 * k1 + n2) * WB + l];
    fftk::dft<N2, -1>(v);
#pragma unroll
    for (int k2 = 0; k2 < N2; k2++) v[k2] = poisson_mode(v[k2], sym, i, j, k1 + N1 * k2, dxsq);
    fftk::dft<N2, +1>(v);
#pragma unroll
    for (int n2 = 1; n2 < N2; n2++) {
      double2 w = tw[n2 * k1];
      w.y = -w.y;
      v[n2] = cmul(v[n2], w);
    }
#pragma unroll
    for (int n2 = 0; n2 < N2; n2++) A[(N2 * k1 + n2) * WB + l] = v[n2];
  }
  __syncthreads();
  z_inverse_a<N, N1, WB, WB, TPB>(A, work, plane, col0, wn);
}

// the thermal forcing's spectrum (three components), drawn and inverse transformed along z
template <int N, int N1, int WB, int TPB>
__global__ void __launch_bounds__(TPB, 2) k_z_noise_fast(double2* __restrict__ work, const double2* __restrict__ twz,
                                                         const double* __restrict__ sym, NoiseArgs na) {
  constexpr int N2 = N / N1, NH = N / 2 + 1, NL = 3 * WB;
  constexpr long plane = (long)N * NH;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  double2* A = reinterpret_cast<double2*>(smem_raw);
  double2* tw = A + N * NL;
  const long col0 = (long)blockIdx.x * WB;
  const int wn = (int)min((long)WB, plane - col0);
  for (int t = threadIdx.x; t < N; t += TPB) tw[t] = twz[t];
  const uint64_t step = *na.step + 1;
#pragma unroll 1
  for (int u = threadIdx.x; u < WB * N; u += TPB) {
    const int w = u % WB, k = u / WB;
    if (w >= wn) continue;
    const int col = (int)col0 + w, j = col / NH, i = col - j * NH;
    noise_mode_draw(na, step, sym, N, NH, i, j, k, A + dpos<N1, N2>(k) * NL + w, WB);
  }
  __syncthreads();
  z_inverse_b<N, N1, NL, TPB>(A, tw);
  __syncthreads();
  z_inverse_a<N, N1, NL, WB, TPB>(A, work, plane, col0, wn);
}

template <int N> struct PlainKernels {
  static constexpr int N1 = fftk::SplitBalanced<N>::N1, NP = plane_balanced<N>();
  using P = PlaneShape<double, N, NP>;
  static constexpr int PB = poisson_columns<N>(), PT = 128;
  static constexpr int WB = ZShape<double, N>::WB, ZT = 256;
  static constexpr size_t smem_p = sizeof(double2) * (size_t)(N * PB + N), smem_n = sizeof(double2) * (size_t)(3 * N * WB + N);

  static cudaError_t attrs() {
    cudaError_t e = cudaSuccess;
    auto set = [&](const void* k, size_t b) {
      if (e == cudaSuccess) e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)b);
    };
    set((const void*)k_xy_forward_fast<double, N, NP, DivergencePlanes>, P::smem);
    set((const void*)k_xy_inverse_fast<double, N, NP>, P::smem);
    set((const void*)k_z_poisson_fast<N, N1, PB, PT>, smem_p);
    set((const void*)k_z_noise_fast<N, N1, WB, ZT>, smem_n);
    return e;
  }
  static cudaError_t run(int stage, const PlainBufs& b, const FftTables<double>& tb, cudaStream_t st) {
    constexpr long ncol = (long)N * (N / 2 + 1);
    switch (stage) {
      case kPlainForward:
        launch_next(k_xy_forward_fast<double, N, NP, DivergencePlanes>, N, P::TPB, P::smem, st,
                    DivergencePlanes{b.u, 1.0 / b.dx}, b.work, tb.wx_f);
        break;
      case kPlainPoisson:
        launch_next(k_z_poisson_fast<N, N1, PB, PT>, (unsigned)((ncol + PB - 1) / PB), PT, smem_p, st, b.work,
                    tb.wz_f, b.sym, b.dx * b.dx);
        break;
      case kPlainInverse:
        launch_next(k_xy_inverse_fast<double, N, NP>, N, P::TPB, P::smem, st, b.work, b.p, tb.wx_f, nullptr);
        break;
      case kPlainNoise:
        k_z_noise_fast<N, N1, WB, ZT>
            <<<(unsigned)((ncol + WB - 1) / WB), ZT, smem_n, st>>>(b.nwork, tb.wz_f, b.sym, b.noise);
        break;
      default:
        launch_next(k_xy_inverse_fast<double, N, NP>, 3 * N, P::TPB, P::smem, st, b.nwork, b.f, tb.wx_f,
                    (uint64_t*)b.noise.step);
    }
    count_launches(1);
    return cudaGetLastError();
  }
};

}  // namespace selm
