// fluid_plain.cu - the reference-structured FP64 fluid step (drop-in form).
//
// The steps of the reference's kernels (cuda/SELM_Kernel.cu) in its order, in
// real space: u*, divergence, Poisson solve, gradient correction, mean removal
// and the next thermal forcing.  The library FFTs (cuFFT D2Z/Z2D,
// cuda/SELM_Eulerian_Period.cu:26-30,113,117,146) are this project's: plane
// and pencil kernels (fluid_plain_fast.cuh, fluid_any.cu) that take the
// divergence as they load and divide or draw in the z pass; sizes with prime
// factors above 13, or whose planes do not fit in shared memory, keep
// Stockham passes per axis.  The CUB sums
// (cuda/SELM_Eulerian_Period.cu:121-123) are a fixed-tree reduction.
// Layout: planar [3][Nz][Ny][Nx] doubles; half spectrum [Nz][Ny][Nx/2+1].
#include <algorithm>

#include "common.cuh"
#include "fluid_any.h"
#include "fluid_fast.h"
#include "fluid_plain.cuh"
#include "selm_kernels.h"

namespace selm {

// ---------------------------------------------------------------- viscous step
// u* = u + (mu*dt*lap7(u) + f)/rho   (cuda/SELM_Kernel.cu:155-195), f the
// forcing with the spread impulses.  A thread per cell of a
// row (block: threadIdx.x along x, blockIdx = (row, plane)), by the reciprocals
// of dx^2 and rho: with two FP64 divisions per component and three integer ones
// per cell the kernel was bound by them (51 us at 128^3; its 150 MB take 23).
__global__ void __launch_bounds__(256) k_u2uAsterisk(const double* u, const double* f, double* us, double c, double irho,
                                                     int Nx, int Ny, int Nz) {
  const int j = blockIdx.x * blockDim.y + threadIdx.y, k = blockIdx.y;
  previous_done();
  if (j >= Ny) return;
  const long Nyx = (long)Ny * Nx, N = Nyx * Nz;
  const double* up = u + k * Nyx + (long)j * Nx;
  const long j1 = (j != Ny - 1) ? Nx : -(long)j * Nx, j0 = (j != 0) ? -(long)Nx : (long)(Ny - 1) * Nx;
  const long k1 = (k != Nz - 1) ? Nyx : -(long)k * Nyx, k0 = (k != 0) ? -Nyx : (long)(Nz - 1) * Nyx;
  for (int i = threadIdx.x; i < Nx; i += blockDim.x) {
    const int i1 = (i != Nx - 1) ? i + 1 : 0, i0 = (i != 0) ? i - 1 : Nx - 1;
#pragma unroll
    for (int d = 0; d < 3; d++) {
      const double* ud = up + d * N;
      const long n = d * N + k * Nyx + (long)j * Nx + i;
      const double r = ud[i];
      const double lap = ud[i1] + ud[i0] + ud[i + j1] + ud[i + j0] + ud[i + k1] + ud[i + k0] - 6 * r;
      us[n] = r + (c * lap + f[n]) * irho;
    }
  }
}

// p = div(u*) with forward differences (cuda/SELM_Kernel.cu:100-116)
__global__ void k_div(const double* __restrict__ in, double* __restrict__ out, int Nx, int Ny, int Nz, double idx) {
  const long N = (long)Nx * Ny * Nz;
  const long n = (long)blockIdx.x * blockDim.x + threadIdx.x;
  if (n >= N) return;
  const long Nyx = (long)Ny * Nx;
  const int k = (int)(n / Nyx), j = (int)((n - k * Nyx) / Nx), i = (int)(n - k * Nyx - (long)j * Nx);
  const long i1 = (i != Nx - 1) ? 1 : -i;
  const long j1 = (j != Ny - 1) ? Nx : -(long)j * Nx;
  const long k1 = (k != Nz - 1) ? Nyx : -(long)k * Nyx;
  const double* a = in;
  const double* b = in + N;
  const double* c = in + 2 * N;
  out[n] = (a[n + i1] - a[n] + b[n + j1] - b[n] + c[n + k1] - c[n]) * idx;
}

// the Poisson solve in the half spectrum (sizes of the axis passes)
__global__ void k_poisson(double2* in, int Nx, int Ny, int Nz, const double* __restrict__ sym, double dxsq) {
  const long n = (long)blockIdx.x * blockDim.x + threadIdx.x;
  const int Nxh = Nx / 2 + 1;
  const long N2 = (long)Nxh * Ny * Nz;
  if (n >= N2) return;
  const long Nyx = (long)Ny * Nxh;
  const int k = (int)(n / Nyx), j = (int)(n % Nyx / Nxh), i = (int)(n % Nxh);
  in[n] = poisson_mode(in[n], sym, i, j, k, dxsq);
}

// ---------------------------------------------------------------- gradient and mean removal
// u = u* - (p[n] - p[n - e_d])/(dx*N) (cuda/SELM_Kernel.cu:119-152), with the
// sums of the new components: one partial per block and component, in a fixed
// order.  At 128^3 the separate passes read the velocity three times and wrote
// it twice; the sums' own pass is gone, and the division by dx N, three a cell,
// is a product (34 us with it; 117 MB take 18).
constexpr int kGradThreads = 512;
__device__ __forceinline__ double block_total(double v, double* sh) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  const int t = threadIdx.y * blockDim.x + threadIdx.x, w = t >> 5, nw = (blockDim.x * blockDim.y) >> 5;
  __syncthreads();
  if ((t & 31) == 0) sh[w] = v;
  __syncthreads();
  double s = 0.0;
  for (int i = 0; i < nw; i++) s += sh[i];
  return s;
}
__global__ void __launch_bounds__(kGradThreads) k_grad_sum(const double* p, double* u, int Nx,
                                                           int Ny, int Nz, double c, double* partial) {
  __shared__ double sh[kGradThreads / 32];
  const long N = (long)Nx * Ny * Nz, Nyx = (long)Ny * Nx;
  const int rows = Ny * Nz;
  previous_done();
  double s0 = 0.0, s1 = 0.0, s2 = 0.0;
  // a row of blockDim.x lanes (threadIdx.y rows at a time)
  for (int row = blockIdx.x * blockDim.y + threadIdx.y; row < rows; row += gridDim.x * blockDim.y) {
    const int k = row / Ny, j = row - k * Ny;
    const long o1 = (j != 0) ? -(long)Nx : (long)(Ny - 1) * Nx;
    const long o2 = (k != 0) ? -Nyx : (long)(Nz - 1) * Nyx;
    for (int i = threadIdx.x; i < Nx; i += blockDim.x) {
      const long n = (long)row * Nx + i;
      const double pn = p[n];
      const double a = u[n] - (pn - p[n + ((i != 0) ? -1 : Nx - 1)]) * c;
      const double b = u[N + n] - (pn - p[n + o1]) * c;
      const double e = u[2 * N + n] - (pn - p[n + o2]) * c;
      u[n] = a;
      u[N + n] = b;
      u[2 * N + n] = e;
      s0 += a;
      s1 += b;
      s2 += e;
    }
  }
  s0 = block_total(s0, sh);
  s1 = block_total(s1, sh);
  s2 = block_total(s2, sh);
  if (threadIdx.x == 0 && threadIdx.y == 0) {
    partial[blockIdx.x] = s0;
    partial[gridDim.x + blockIdx.x] = s1;
    partial[2 * gridDim.x + blockIdx.x] = s2;
  }
}

// u -= sum/N (cuda/SELM_Kernel.cu:197-207); every block adds the partials of
// its component itself, in the same order
__global__ void __launch_bounds__(kGradThreads) k_subtract_mean(double* u, const double* partial, int nparts, long N) {
  __shared__ double sh[kGradThreads / 32];
  const int d = blockIdx.y;
  previous_done();
  double s = 0.0;
  for (int i = threadIdx.x; i < nparts; i += kGradThreads) s += partial[d * nparts + i];
  const double mean = block_total(s, sh) / N;
  double* ud = u + d * N;
  for (long n = (long)blockIdx.x * kGradThreads + threadIdx.x; n < N; n += (long)gridDim.x * kGradThreads) ud[n] -= mean;
}

// ---------------------------------------------------------------- thermal noise
// the forcing's half spectrum (sizes of the axis passes)
__global__ void k_noise_generate(double2* __restrict__ out, int Nx, int Ny, int Nz, const double* __restrict__ sym,
                                 NoiseArgs na) {
  const long n = (long)blockIdx.x * blockDim.x + threadIdx.x;
  const int Nxh = Nx / 2 + 1;
  const long N2 = (long)Nxh * Ny * Nz;
  if (n >= N2) return;
  const long Nyx = (long)Ny * Nxh;
  const int k = (int)(n / Nyx), j = (int)(n % Nyx / Nxh), i = (int)(n % Nxh);
  double2 z[3];
  noise_mode_draw(na, *na.step + 1, sym, Nx, Nxh, i, j, k, z, 1);
#pragma unroll
  for (int d = 0; d < 3; d++) out[d * N2 + n] = z[d];
}
__global__ void k_step_advance(uint64_t* step) { *step += 1; }

// ---------------------------------------------------------------- FFT passes
// Complex FFT along a strided axis.  Line (o, i), i < ni: element t at
// data[o*os + i + t*es].  A block takes B consecutive i of one o, so every
// row t is one contiguous run of B complex values.
template <typename T>
__global__ void k_fft_axis(cpx<T>* __restrict__ data, int ni, long os, long es, FftRadix R,
                           const cpx<T>* __restrict__ tw, int sign, int B) {
  using C = cpx<T>;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  C* w = reinterpret_cast<C*>(smem_raw);
  const int n = R.n;
  C* A = w + n;
  C* Bb = A + n * B;
  const int i0 = blockIdx.x * B;
  const int nl = min(B, ni - i0);
  C* base = data + (long)blockIdx.y * os + i0;
  for (int t = threadIdx.x; t < n; t += blockDim.x) w[t] = tw[t];
  for (int idx = threadIdx.x; idx < n * B; idx += blockDim.x) {
    const int t = idx / B, b = idx % B;
    A[idx] = (b < nl) ? base[b + t * es] : cmk<C>(T(0), T(0));
  }
  __syncthreads();
  C* res = line_fft(A, Bb, w, R, B, 1, B, true, sign);
  for (int idx = threadIdx.x; idx < n * B; idx += blockDim.x) {
    const int t = idx / B, b = idx % B;
    if (b < nl) base[b + t * es] = res[idx];
  }
}

// x-direction real -> half complex for B rows of length nx (rows contiguous)
template <typename T>
__global__ void k_fft_x_r2c(const T* __restrict__ in, cpx<T>* __restrict__ out, long nrows, FftRadix R,
                            const cpx<T>* __restrict__ tw, int B) {
  using C = cpx<T>;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  C* w = reinterpret_cast<C*>(smem_raw);
  const int n = R.n, nxh = n / 2 + 1;
  C* A = w + n;
  C* Bb = A + n * B;
  const long r0 = (long)blockIdx.x * B;
  const int nl = (int)min((long)B, nrows - r0);
  for (int t = threadIdx.x; t < n; t += blockDim.x) w[t] = tw[t];
  for (int idx = threadIdx.x; idx < n * B; idx += blockDim.x) {
    const int b = idx / n;
    A[idx] = cmk<C>(b < nl ? in[r0 * n + idx] : T(0), T(0));
  }
  __syncthreads();
  C* res = line_fft(A, Bb, w, R, B, n, 1, false, -1);
  for (int idx = threadIdx.x; idx < nxh * B; idx += blockDim.x) {
    const int b = idx / nxh, m = idx % nxh;
    if (b < nl) out[(r0 + b) * nxh + m] = res[b * n + m];
  }
}

// x-direction half complex -> real (imaginary parts of the m=0 and m=n/2
// entries drop out, as in FFTW's c2r), times `scale`
template <typename T>
__global__ void k_fft_x_c2r(const cpx<T>* __restrict__ in, T* __restrict__ out, long nrows, FftRadix R,
                            const cpx<T>* __restrict__ tw, int B, T scale) {
  using C = cpx<T>;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  C* w = reinterpret_cast<C*>(smem_raw);
  const int n = R.n, nxh = n / 2 + 1;
  C* A = w + n;
  C* Bb = A + n * B;
  const long r0 = (long)blockIdx.x * B;
  const int nl = (int)min((long)B, nrows - r0);
  for (int t = threadIdx.x; t < n; t += blockDim.x) w[t] = tw[t];
  for (int idx = threadIdx.x; idx < n * B; idx += blockDim.x) {
    const int b = idx / n, m = idx % n;
    C v = cmk<C>(T(0), T(0));
    if (b < nl) {
      if (m < nxh) v = in[(r0 + b) * nxh + m];
      else {
        const C h = in[(r0 + b) * nxh + (n - m)];
        v = cmk<C>(h.x, -h.y);
      }
    }
    A[idx] = v;
  }
  __syncthreads();
  C* res = line_fft(A, Bb, w, R, B, n, 1, false, +1);
  for (int idx = threadIdx.x; idx < n * B; idx += blockDim.x) {
    const int b = idx / n;
    if (b < nl) out[r0 * n + idx] = res[idx].x * scale;
  }
}

// ---------------------------------------------------------------- host launchers
static int fft_lines_per_block(int n, size_t elem, size_t smem_cap) {
  int B = (elem == 16) ? 16 : 32;
  while (B > 1 && (size_t)(n + 2 * n * B) * elem > smem_cap) B /= 2;
  return B;
}

template <typename T> static cudaError_t set_smem(const void* fn, size_t bytes) {
  return cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
}

template <typename T>
cudaError_t fft3_r2c(const T* in, cpx<T>* out, int nx, int ny, int nz, int ncomp, const FftTables<T>& tb,
                     cudaStream_t st) {
  using C = cpx<T>;
  const int nxh = nx / 2 + 1;
  const size_t cap = 160 * 1024;
  cudaError_t e;
  {  // x pass
    const int B = fft_lines_per_block(nx, sizeof(C), cap);
    const size_t sm = (size_t)(nx + 2 * nx * B) * sizeof(C);
    if ((e = set_smem<T>((const void*)k_fft_x_r2c<T>, sm)) != cudaSuccess) return e;
    const long rows = (long)ny * nz * ncomp;
    k_fft_x_r2c<T><<<(unsigned)((rows + B - 1) / B), 256, sm, st>>>(in, out, rows, tb.rx, tb.wx_f, B);
    count_launches(1);
  }
  {  // y pass: lines (o=(c,k), i), element stride nxh
    const int B = fft_lines_per_block(ny, sizeof(C), cap);
    const size_t sm = (size_t)(ny + 2 * ny * B) * sizeof(C);
    if ((e = set_smem<T>((const void*)k_fft_axis<T>, sm)) != cudaSuccess) return e;
    dim3 g((nxh + B - 1) / B, nz * ncomp);
    k_fft_axis<T><<<g, 256, sm, st>>>(out, nxh, (long)ny * nxh, nxh, tb.ry, tb.wy_f, -1, B);
    count_launches(1);
  }
  {  // z pass: lines (o=c, i=(j,i)), element stride ny*nxh
    const int B = fft_lines_per_block(nz, sizeof(C), cap);
    const size_t sm = (size_t)(nz + 2 * nz * B) * sizeof(C);
    if ((e = set_smem<T>((const void*)k_fft_axis<T>, sm)) != cudaSuccess) return e;
    const int ni = ny * nxh;
    dim3 g((ni + B - 1) / B, ncomp);
    k_fft_axis<T><<<g, 256, sm, st>>>(out, ni, (long)nz * ny * nxh, (long)ny * nxh, tb.rz, tb.wz_f, -1, B);
    count_launches(1);
  }
  return cudaGetLastError();
}

template <typename T>
cudaError_t fft3_c2r(cpx<T>* in, T* out, int nx, int ny, int nz, int ncomp, T scale, const FftTables<T>& tb,
                     cudaStream_t st) {
  using C = cpx<T>;
  const int nxh = nx / 2 + 1;
  const size_t cap = 160 * 1024;
  cudaError_t e;
  {  // z pass (inverse)
    const int B = fft_lines_per_block(nz, sizeof(C), cap);
    const size_t sm = (size_t)(nz + 2 * nz * B) * sizeof(C);
    if ((e = set_smem<T>((const void*)k_fft_axis<T>, sm)) != cudaSuccess) return e;
    const int ni = ny * nxh;
    dim3 g((ni + B - 1) / B, ncomp);
    k_fft_axis<T><<<g, 256, sm, st>>>(in, ni, (long)nz * ny * nxh, (long)ny * nxh, tb.rz, tb.wz_b, +1, B);
    count_launches(1);
  }
  {  // y pass (inverse)
    const int B = fft_lines_per_block(ny, sizeof(C), cap);
    const size_t sm = (size_t)(ny + 2 * ny * B) * sizeof(C);
    if ((e = set_smem<T>((const void*)k_fft_axis<T>, sm)) != cudaSuccess) return e;
    dim3 g((nxh + B - 1) / B, nz * ncomp);
    k_fft_axis<T><<<g, 256, sm, st>>>(in, nxh, (long)ny * nxh, nxh, tb.ry, tb.wy_b, +1, B);
    count_launches(1);
  }
  {  // x pass c2r
    const int B = fft_lines_per_block(nx, sizeof(C), cap);
    const size_t sm = (size_t)(nx + 2 * nx * B) * sizeof(C);
    if ((e = set_smem<T>((const void*)k_fft_x_c2r<T>, sm)) != cudaSuccess) return e;
    const long rows = (long)ny * nz * ncomp;
    k_fft_x_c2r<T><<<(unsigned)((rows + B - 1) / B), 256, sm, st>>>(in, out, rows, tb.rx, tb.wx_b, B, scale);
    count_launches(1);
  }
  return cudaGetLastError();
}

template cudaError_t fft3_r2c<double>(const double*, double2*, int, int, int, int, const FftTables<double>&,
                                      cudaStream_t);
template cudaError_t fft3_c2r<double>(double2*, double*, int, int, int, int, double, const FftTables<double>&,
                                      cudaStream_t);
template cudaError_t fft3_r2c<float>(const float*, float2*, int, int, int, int, const FftTables<float>&,
                                     cudaStream_t);
template cudaError_t fft3_c2r<float>(float2*, float*, int, int, int, int, float, const FftTables<float>&,
                                     cudaStream_t);

static cudaError_t plain_stage(int stage, const PlainPlan& pp, const PlainBufs& b, int n, const FftTables<double>& tb,
                               cudaStream_t st) {
  return pp.fast ? plain_fast_stage(stage, n, b, tb, st) : any_plain_stage(stage, *pp.any, b, tb, st);
}

// One fluid step of the reference structure (cuda/SELM_Eulerian_Period.cu:96-126):
// u_new = P(u_old + (mu dt lap u_old + f)/rho) - mean.
cudaError_t plain_ustar(const double* u_old, double* u_new, const PlainBufs& b, int nx, int ny, int nz, double dt,
                        double mu, double rho, cudaStream_t st) {
  const int tx = nx <= 32 ? 32 : nx <= 64 ? 64 : 128, ty = 256 / tx;
  launch_next(k_u2uAsterisk, dim3((unsigned)((ny + ty - 1) / ty), (unsigned)nz), dim3(tx, ty), 0, st, u_old, b.f, u_new,
              mu * dt / (b.dx * b.dx), 1.0 / rho, nx, ny, nz);
  count_launches(1);
  return cudaGetLastError();
}

cudaError_t plain_project(double* u_new, const PlainPlan& pp, const PlainBufs& b, double* partial, int nx, int ny,
                          int nz, const FftTables<double>& tb, cudaStream_t st) {
  const long N = (long)nx * ny * nz;
  const long N2 = (long)(nx / 2 + 1) * ny * nz;
  cudaError_t e = cudaSuccess;
  if (pp.fast || pp.any) {
    for (int stage : {kPlainForward, kPlainPoisson, kPlainInverse})
      if (e == cudaSuccess) e = plain_stage(stage, pp, b, nx, tb, st);
    if (e != cudaSuccess) return e;
  } else {
    k_div<<<(unsigned)((N + 127) / 128), 128, 0, st>>>(u_new, b.p, nx, ny, nz, 1.0 / b.dx);
    count_launches(1);
    if ((e = fft3_r2c<double>(b.p, b.work, nx, ny, nz, 1, tb, st)) != cudaSuccess) return e;
    k_poisson<<<(unsigned)((N2 + 127) / 128), 128, 0, st>>>(b.work, nx, ny, nz, b.sym, b.dx * b.dx);
    count_launches(1);
    if ((e = fft3_c2r<double>(b.work, b.p, nx, ny, nz, 1, 1.0, tb, st)) != cudaSuccess) return e;
  }
  const unsigned parts = (unsigned)std::min<long>(kSumParts, (N + kGradThreads - 1) / kGradThreads);
  const int tx = nx <= 32 ? 32 : nx <= 64 ? 64 : 128;
  launch_next(k_grad_sum, parts, dim3(tx, kGradThreads / tx), 0, st, b.p, u_new, nx, ny, nz, 1.0 / (b.dx * N), partial);
  launch_next(k_subtract_mean, dim3(parts, 3), kGradThreads, 0, st, u_new, partial, (int)parts, N);
  count_launches(2);
  return cudaGetLastError();
}

// Thermal forcing of cuda/SELM_Eulerian_Period.cu:128-153 for the step after
// the device counter's, which the second part advances:
// f = sqrt(2 kB T dt mu / N) * c2r(noise half spectrum), or f = 0.
cudaError_t plain_forcing_draw(const PlainPlan& pp, const PlainBufs& b, int nx, int ny, int nz, bool stochastic,
                               const FftTables<double>& tb, cudaStream_t st) {
  if (!stochastic) return cudaSuccess;
  if (pp.fast || pp.any) return plain_stage(kPlainNoise, pp, b, nx, tb, st);
  const long N2 = (long)(nx / 2 + 1) * ny * nz;
  k_noise_generate<<<(unsigned)((N2 + 127) / 128), 128, 0, st>>>(b.nwork, nx, ny, nz, b.sym, b.noise);
  count_launches(1);
  return cudaGetLastError();
}

cudaError_t plain_forcing_finish(const PlainPlan& pp, const PlainBufs& b, int nx, int ny, int nz, bool stochastic,
                                 const FftTables<double>& tb, cudaStream_t st) {
  if (!stochastic) return cudaMemsetAsync(b.f, 0, sizeof(double) * 3L * nx * ny * nz, st);
  if (pp.fast || pp.any) return plain_stage(kPlainNoiseInverse, pp, b, nx, tb, st);
  const cudaError_t e = fft3_c2r<double>(b.nwork, b.f, nx, ny, nz, 3, 1.0, tb, st);
  if (e != cudaSuccess) return e;
  k_step_advance<<<1, 1, 0, st>>>((uint64_t*)b.noise.step);
  count_launches(1);
  return cudaGetLastError();
}

}  // namespace selm
