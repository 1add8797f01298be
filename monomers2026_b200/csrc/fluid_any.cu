// fluid_any.cu - the fused spectral kernels for run-time grid sizes (every
// prime factor at most 13), on the line FFTs of fft_any.cuh.  The same three
// kernels and arithmetic as fluid_fused_fast.cuh, whose compile-time sizes
// keep their own: per (component, z) plane the x and y FFTs, per block of WB
// columns the z FFT, the spectral update and the inverse z FFT.
#include <algorithm>

#include "fft_any.cuh"
#include "fluid_fused_fast.cuh"
#include "fluid_plane.cuh"
#include "fluid_plain.cuh"

namespace selm {

template <typename T> struct PlaneSmem {
  cpx<T>*P, *A, *twx, *twy;
  int *posx, *posy;  // position of mode k after the forward order
};
template <typename T> __device__ __forceinline__ PlaneSmem<T> plane_smem(const PlaneGeom& g, unsigned char* raw) {
  PlaneSmem<T> s;
  s.P = reinterpret_cast<cpx<T>*>(raw);
  s.A = s.P + g.y.n * g.pitch;
  s.twx = s.A + g.x.n * (g.rp + 1) + g.x.n / g.x.r[g.x.np - 1];
  s.twy = s.twx + g.x.n;
  s.posx = reinterpret_cast<int*>(s.twy + g.y.n);
  s.posy = s.posx + g.x.n;
  return s;
}
// load(row, x): the plane's real values
template <typename T, typename LD>
__device__ __forceinline__ void xy_forward_any(const PlaneGeom& g, const cpx<T>* __restrict__ twx,
                                               const cpx<T>* __restrict__ twy, cpx<T>* dst,
                                               unsigned char* raw, LD&& load) {
  using C = cpx<T>;
  const PlaneSmem<T> s = plane_smem<T>(g, raw);
  const int nx = g.x.n, ny = g.y.n, nh = g.nh, rp = g.rp, rpp = rp + 1;
  for (int t = threadIdx.x; t < nx; t += blockDim.x) {
    s.twx[t] = twx[t];
    s.posx[t] = mode_pos(g.x, t);
  }
  for (int t = threadIdx.x; t < ny; t += blockDim.x) s.twy[t] = twy[t];
  previous_done();
  for (int y0 = 0; y0 < g.hp; y0 += rp) {
    __syncthreads();
    for (int idx = threadIdx.x; idx < rp * nx; idx += blockDim.x) {
      const int lr = div_by(g.dnx, idx), x = idx - lr * nx;
      const int ya = y0 + lr, yb = ya + g.hp;
      s.A[x * rpp + lr] = fftk::mk<C>(ya < g.hp ? load(ya, x) : T(0), ya < g.hp && yb < ny ? load(yb, x) : T(0));
    }
    __syncthreads();
    for (int q = 0; q < g.x.np; q++) {
      smem_pass<-1, false>(g.x, q, rp, g.drp, s.twx, s.A, rpp, 0);
      __syncthreads();
    }
    // two real rows from one complex line: A = (Z[m] + conj Z[-m])/2, B = (Z[m] - conj Z[-m])/(2i)
    for (int u = threadIdx.x; u < rp * nh; u += blockDim.x) {
      const int m = div_by(g.drp, u), lr = u - m * rp;
      const int ya = y0 + lr, yb = ya + g.hp;
      if (ya >= g.hp) continue;
      const C z = s.A[s.posx[m] * rpp + lr];
      const C zr = s.A[s.posx[m == 0 ? 0 : nx - m] * rpp + lr];
      s.P[ya * g.pitch + m] = fftk::mk<C>((z.x + zr.x) * T(0.5), (z.y - zr.y) * T(0.5));
      if (yb < ny) s.P[yb * g.pitch + m] = fftk::mk<C>((z.y + zr.y) * T(0.5), -(z.x - zr.x) * T(0.5));
    }
  }
  __syncthreads();
  for (int q = 0; q + 1 < g.y.np; q++) {
    smem_pass<-1, false>(g.y, q, nh, g.dnh, s.twy, s.P, g.pitch, 0);
    __syncthreads();
  }
  // the last y pass, straight to global memory: thread (m, block), m fastest
  with_radix(g.y.r[g.y.np - 1], [&](auto rc) {
    constexpr int R = decltype(rc)::value;
    const int nb = ny / R;
    for (int u = threadIdx.x; u < nh * nb; u += blockDim.x) {
      const int blk = div_by(g.dnh, u), m = u - blk * nh;
      const C* e = s.P + blk * R * g.pitch + m;
      C v[R];
#pragma unroll
      for (int j = 0; j < R; j++) v[j] = e[j * g.pitch];
      fftk::dft<R, -1>(v);
      C* d = dst + block_mode(g.y, blk) * nh + m;
#pragma unroll
      for (int j = 0; j < R; j++) d[j * nb * nh] = v[j];
    }
  });
}

// y inverse FFT and x c2r of one plane
template <typename T>
__device__ __forceinline__ void xy_inverse_any(const PlaneGeom& g, const cpx<T>* __restrict__ twx,
                                               const cpx<T>* __restrict__ twy, const cpx<T>* src,
                                               T* dst, unsigned char* raw) {
  using C = cpx<T>;
  const PlaneSmem<T> s = plane_smem<T>(g, raw);
  const int nx = g.x.n, ny = g.y.n, nh = g.nh, rp = g.rp, rpp = rp + 1;
  for (int t = threadIdx.x; t < nx; t += blockDim.x) s.twx[t] = twx[t];
  for (int t = threadIdx.x; t < ny; t += blockDim.x) {
    s.twy[t] = twy[t];
    s.posy[t] = mode_pos(g.y, t);
  }
  previous_done();
  __syncthreads();
  // the first y pass, straight from global memory: thread (m, n2), m fastest
  with_radix(g.y.r[0], [&](auto rc) {
    constexpr int R = decltype(rc)::value;
    const int M = ny / R;
    for (int u = threadIdx.x; u < nh * M; u += blockDim.x) {
      const int n2 = div_by(g.dnh, u), m = u - n2 * nh;
      const C* e = src + n2 * nh + m;
      C v[R];
#pragma unroll
      for (int j = 0; j < R; j++) v[j] = e[j * M * nh];
      fftk::dft<R, +1>(v);
      if (M > 1) twiddle_points<R, +1>(v, s.twy, n2);
      C* d = s.P + n2 * g.pitch + m;
#pragma unroll
      for (int j = 0; j < R; j++) d[j * M * g.pitch] = v[j];
    }
  });
  for (int q = 1; q < g.y.np; q++) {
    __syncthreads();
    smem_pass<+1, false>(g.y, q, nh, g.dnh, s.twy, s.P, g.pitch, 0);
  }
  const int rl = g.x.r[g.x.np - 1];
  for (int y0 = 0; y0 < g.hp; y0 += rp) {
    __syncthreads();
    // two rows per complex line; the imaginary parts of m = 0 and m = nx/2 drop out
    for (int idx = threadIdx.x; idx < rp * nx; idx += blockDim.x) {
      const int lr = div_by(g.dnx, idx), m = idx - lr * nx;
      const int ya = y0 + lr, yb = ya + g.hp;
      C a = fftk::mk<C>(T(0), T(0)), b = a;
      const int mm = m < nh ? m : nx - m;
      if (ya < g.hp) a = s.P[s.posy[ya] * g.pitch + mm];
      if (ya < g.hp && yb < ny) b = s.P[s.posy[yb] * g.pitch + mm];
      if (m >= nh) {
        a.y = -a.y;
        b.y = -b.y;
      }
      if (m == 0 || 2 * m == nx) {
        a.y = T(0);
        b.y = T(0);
      }
      s.A[m * rpp + div_by(g.x.dl, m) + lr] = fftk::mk<C>(a.x - b.y, a.y + b.x);
    }
    __syncthreads();
    for (int q = 0; q + 1 < g.x.np; q++) {
      smem_pass<+1, false>(g.x, q, rp, g.drp, s.twx, s.A, rpp, 1);
      __syncthreads();
    }
    // the last x pass, straight to global memory: thread (q, row pair), q fastest (consecutive x)
    with_radix(rl, [&](auto rc) {
      constexpr int R = decltype(rc)::value;
      const int nb = nx / R;
      for (int u = threadIdx.x; u < rp * nb; u += blockDim.x) {
        int lr, q;
        if (g.x.np == 2) {
          lr = div_by(g.x.d0, u);
          q = u - lr * nb;
        } else {
          lr = u / nb;
          q = u - lr * nb;
        }
        const int ya = y0 + lr, yb = ya + g.hp;
        if (ya >= g.hp) continue;
        const int blk = mode_block(g.x, q);
        const C* e = s.A + blk * (R * rpp + 1) + lr;
        C v[R];
#pragma unroll
        for (int j = 0; j < R; j++) v[j] = e[j * rpp];
        fftk::dft<R, +1>(v);
        T* d = dst + ya * nx + q;
#pragma unroll
        for (int j = 0; j < R; j++) d[j * nb] = v[j].x;
        if (yb < ny) {
          d = dst + yb * nx + q;
#pragma unroll
          for (int j = 0; j < R; j++) d[j * nb] = v[j].y;
        }
      }
    });
  }
}

template <typename T, typename In>
__global__ void __launch_bounds__(plane_threads_max<T>()) k_xy_forward_any(In in, cpx<T>* out, PlaneGeom g,
                                                                         const cpx<T>* __restrict__ twx,
                                                                         const cpx<T>* __restrict__ twy) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const auto src = in.plane(blockIdx.x, g.x.n);
  xy_forward_any<T>(g, twx, twy, out + (long)blockIdx.x * g.y.n * g.nh, smem_raw,
                    [&](int y, int x) { return src.at(y, x, g.x.n); });
}

template <typename T>
__global__ void __launch_bounds__(plane_threads_max<T>()) k_xy_inverse_any(const cpx<T>* in, T* out,
                                                                         PlaneGeom g, const cpx<T>* __restrict__ twx,
                                                                         const cpx<T>* __restrict__ twy,
                                                                         uint64_t* step) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const long plane = blockIdx.x;
  xy_inverse_any<T>(g, twx, twy, in + plane * g.y.n * g.nh, out + plane * g.x.n * g.y.n, smem_raw);
  if (step && blockIdx.x == 0 && threadIdx.x == 0) *step += 1;  // as k_xy_inverse_fast
}

// ---------------------------------------------------------------- z pencils
// forward z FFT of the block's columns, global memory to shared
template <typename T>
__device__ __forceinline__ void z_load_forward(const PencilGeom& p, const cpx<T>* __restrict__ work, long plane,
                                               long col0, int wn, const cpx<T>* tw, cpx<T>* A) {
  using C = cpx<T>;
  const int nl = p.nl, nz = p.z.n;
  with_radix(p.z.r[0], [&](auto rc) {
    constexpr int R = decltype(rc)::value;
    const int M = nz / R;
    for (int u = threadIdx.x; u < nl * M; u += blockDim.x) {
      const int n2 = div_by(p.dnl, u), l = u - n2 * nl;
      const int c = div_by(p.dwb, l), w = l - c * p.wb;
      C v[R];
      if (w < wn) {
        const C* e = work + ((long)c * nz + n2) * plane + col0 + w;
#pragma unroll
        for (int j = 0; j < R; j++) v[j] = e[j * M * plane];
      } else {
#pragma unroll
        for (int j = 0; j < R; j++) v[j] = fftk::mk<C>(T(0), T(0));
      }
      fftk::dft<R, -1>(v);
      if (M > 1) twiddle_points<R, -1>(v, tw, n2);
      C* d = A + n2 * nl + l;
#pragma unroll
      for (int j = 0; j < R; j++) d[j * M * nl] = v[j];
    }
  });
  for (int q = 1; q < p.z.np; q++) {
    __syncthreads();
    smem_pass<-1, false>(p.z, q, nl, p.dnl, tw, A, nl, 0);
  }
}

// inverse z FFT of the block's columns (modes at their forward positions), shared memory to global
template <typename T>
__device__ __forceinline__ void z_inverse_store(const PencilGeom& p, cpx<T>* __restrict__ work, long plane, long col0,
                                                int wn, const cpx<T>* tw, cpx<T>* A) {
  using C = cpx<T>;
  const int nl = p.nl, nz = p.z.n;
  for (int q = p.z.np - 1; q > 0; q--) {
    smem_pass<+1, true>(p.z, q, nl, p.dnl, tw, A, nl, 0);
    __syncthreads();
  }
  with_radix(p.z.r[0], [&](auto rc) {
    constexpr int R = decltype(rc)::value;
    const int M = nz / R;
    for (int u = threadIdx.x; u < nl * M; u += blockDim.x) {
      const int n2 = div_by(p.dnl, u), l = u - n2 * nl;
      const int c = div_by(p.dwb, l), w = l - c * p.wb;
      if (w >= wn) continue;
      const C* e = A + n2 * nl + l;
      C v[R];
#pragma unroll
      for (int j = 0; j < R; j++) v[j] = e[j * M * nl];
      if (M > 1) twiddle_points<R, +1>(v, tw, n2);
      fftk::dft<R, +1>(v);
      C* d = work + ((long)c * nz + n2) * plane + col0 + w;
#pragma unroll
      for (int j = 0; j < R; j++) d[j * M * plane] = v[j];
    }
  });
}

template <typename T>
__global__ void __launch_bounds__(256, sizeof(T) == 4 ? 3 : 2) k_z_update_any(cpx<T>* __restrict__ work,
                                                                              cpx<T>* __restrict__ uhat, ZGeom g,
                                                                              PencilGeom p,
                                                                              const cpx<T>* __restrict__ twz,
                                                                              const double* __restrict__ symx,
                                                                              const double* __restrict__ symy,
                                                                              const double* __restrict__ symz) {
  using C = cpx<T>;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int nz = p.z.n, nl = p.nl, wb = p.wb;
  C* A = reinterpret_cast<C*>(smem_raw);
  C* tw = A + nz * nl;
  PlaneSym<T>* pz = reinterpret_cast<PlaneSym<T>*>(tw + nz);
  ColArrays<T> col;
  col.dx = reinterpret_cast<C*>(pz + nz);
  col.dy = col.dx + wb;
  col.c = reinterpret_cast<double*>(col.dy + wb);
  col.ij = reinterpret_cast<int*>(col.c + wb);
  int* pos = col.ij + wb;  // nz positions
  const long plane = (long)g.ny * g.nxh, col0 = (long)blockIdx.x * wb;
  const int wn = (int)min((long)wb, plane - col0);
  for (int t = threadIdx.x; t < nz; t += blockDim.x) {
    tw[t] = twz[t];
    pos[t] = mode_pos(p.z, t);
    pz[t] = plane_sym<T>(g, t, symz);
  }
  if (threadIdx.x < wn) put_col(col, threadIdx.x, col_sym<T>(g, col0 + threadIdx.x, symx, symy));
  __syncthreads();
  z_load_forward<T>(p, work, plane, col0, wn, tw, A);
  __syncthreads();
  const ModeConsts<T> mc = mode_consts<T>(g, nz);
  const ModeOrder order = mode_order((int)col0, wn, g.nx, g.nxh);
#pragma unroll 1
  for (int u = threadIdx.x; u < wn * nz; u += blockDim.x) {
    int w, k;
    mode_unit(order, nz, u, w, k);
    C* a = A + pos[k] * nl + w;
    mode_update<T, true>(g, mc, nz, get_col(col, w), pz[k], k, uhat + (long)k * plane + col0 + w, (long)nz * plane, a, wb);
  }
  __syncthreads();
  z_inverse_store<T>(p, work, plane, col0, wn, tw, A);
}

// ---------------------------------------------------------------- the reference-structured form's z passes (FP64)
// z FFT, Poisson solve and inverse z FFT of one component
__global__ void __launch_bounds__(256, 2) k_z_poisson_any(double2* work, int nh, PencilGeom p,
                                                          const double2* __restrict__ twz,
                                                          const double* __restrict__ sym, double dxsq) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int nz = p.z.n, wb = p.wb;
  double2* A = reinterpret_cast<double2*>(smem_raw);
  double2* tw = A + nz * p.nl;
  int* pos = reinterpret_cast<int*>(tw + nz);
  const long plane = (long)nz * nh, col0 = (long)blockIdx.x * wb;
  const int wn = (int)min((long)wb, plane - col0);
  for (int t = threadIdx.x; t < nz; t += blockDim.x) {
    tw[t] = twz[t];
    pos[t] = mode_pos(p.z, t);
  }
  previous_done();
  __syncthreads();
  z_load_forward<double>(p, work, plane, col0, wn, tw, A);
  __syncthreads();
  for (int u = threadIdx.x; u < wb * nz; u += blockDim.x) {
    const int k = div_by(p.dwb, u), w = u - k * wb;
    if (w >= wn) continue;
    const int col = (int)col0 + w, j = col / nh, i = col - j * nh;
    A[pos[k] * p.nl + w] = poisson_mode(A[pos[k] * p.nl + w], sym, i, j, k, dxsq);
  }
  __syncthreads();
  z_inverse_store<double>(p, work, plane, col0, wn, tw, A);
}

// the thermal forcing's spectrum (three components), drawn and inverse transformed along z
__global__ void __launch_bounds__(256, 2) k_z_noise_any(double2* __restrict__ work, int nh, PencilGeom p,
                                                        const double2* __restrict__ twz, const double* __restrict__ sym,
                                                        NoiseArgs na) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int nz = p.z.n, wb = p.wb;
  double2* A = reinterpret_cast<double2*>(smem_raw);
  double2* tw = A + nz * p.nl;
  int* pos = reinterpret_cast<int*>(tw + nz);
  const long plane = (long)nz * nh, col0 = (long)blockIdx.x * wb;
  const int wn = (int)min((long)wb, plane - col0);
  for (int t = threadIdx.x; t < nz; t += blockDim.x) {
    tw[t] = twz[t];
    pos[t] = mode_pos(p.z, t);
  }
  __syncthreads();
  const uint64_t step = *na.step + 1;
#pragma unroll 1
  for (int u = threadIdx.x; u < wb * nz; u += blockDim.x) {
    const int k = div_by(p.dwb, u), w = u - k * wb;
    if (w >= wn) continue;
    const int col = (int)col0 + w, j = col / nh, i = col - j * nh;
    noise_mode_draw(na, step, sym, nz, nh, i, j, k, A + pos[k] * p.nl + w, wb);
  }
  __syncthreads();
  z_inverse_store<double>(p, work, plane, col0, wn, tw, A);
}

// ---------------------------------------------------------------- launchers
cudaError_t any_plain_stage(int stage, const AnyPlan& p, const PlainBufs& b, const FftTables<double>& tb,
                            cudaStream_t st) {
  const int n = p.xy.x.n, nh = p.xy.nh;
  // one component: its lines only, in blocks of three times the columns
  PencilGeom one = p.z;
  one.wb = one.nl;
  one.dwb = one.dnl;
  const unsigned nz1 = (unsigned)(((long)n * nh + one.wb - 1) / one.wb);
  const unsigned nz3 = (unsigned)(((long)n * nh + p.z.wb - 1) / p.z.wb);
  switch (stage) {
    case kPlainForward:
      launch_next(k_xy_forward_any<double, DivergencePlanes>, (unsigned)n, p.threads_xy, p.smem_xy, st,
                  DivergencePlanes{b.u, 1.0 / b.dx}, b.work, p.xy, tb.wx_f, tb.wy_f);
      break;
    case kPlainPoisson:
      launch_next(k_z_poisson_any, nz1, 256, p.smem_z, st, b.work, nh, one, tb.wz_f, b.sym, b.dx * b.dx);
      break;
    case kPlainInverse:
      launch_next(k_xy_inverse_any<double>, (unsigned)n, p.threads_xy, p.smem_xy, st, b.work, b.p, p.xy,
                  tb.wx_f, tb.wy_f, nullptr);
      break;
    case kPlainNoise:
      k_z_noise_any<<<nz3, 256, p.smem_z, st>>>(b.nwork, nh, p.z, tb.wz_f, b.sym, b.noise);
      break;
    default:
      launch_next(k_xy_inverse_any<double>, (unsigned)(3 * n), p.threads_xy, p.smem_xy, st, b.nwork, b.f,
                  p.xy, tb.wx_f, tb.wy_f, (uint64_t*)b.noise.step);
  }
  count_launches(1);
  return cudaGetLastError();
}

cudaError_t any_attrs() {
  cudaError_t e = cudaSuccess;
  for (const void* k : {(const void*)k_xy_forward_any<float, ArrayPlanes<float>>,
                        (const void*)k_xy_forward_any<double, ArrayPlanes<double>>,
                        (const void*)k_xy_forward_any<double, DivergencePlanes>, (const void*)k_z_poisson_any,
                        (const void*)k_z_noise_any,
                        (const void*)k_xy_inverse_any<float>, (const void*)k_xy_inverse_any<double>,
                        (const void*)k_z_update_any<float>, (const void*)k_z_update_any<double>})
    if (e == cudaSuccess) e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSmBytes);
  return e;
}

template <typename T>
cudaError_t any_xy_forward(const AnyPlan& p, const T* in, cpx<T>* out, const FftTables<T>& tb, int planes,
                           cudaStream_t st) {
  k_xy_forward_any<T><<<(unsigned)planes, p.threads_xy, p.smem_xy, st>>>(ArrayPlanes<T>{in}, out, p.xy, tb.wx_f,
                                                                         tb.wy_f);
  count_launches(1);
  return cudaGetLastError();
}

template <typename T>
cudaError_t any_xy_inverse(const AnyPlan& p, const cpx<T>* in, T* out, const FftTables<T>& tb, int planes,
                           uint64_t* step, cudaStream_t st) {
  k_xy_inverse_any<T><<<(unsigned)planes, p.threads_xy, p.smem_xy, st>>>(in, out, p.xy, tb.wx_f, tb.wy_f, step);
  count_launches(1);
  return cudaGetLastError();
}

template <typename T>
cudaError_t any_z_update(const AnyPlan& p, cpx<T>* work, cpx<T>* uhat, const ZGeom& g, const FftTables<T>& tb,
                         const double* symx, const double* symy, const double* symz, cudaStream_t st) {
  const long ncol = (long)g.ny * g.nxh;
  k_z_update_any<T><<<(unsigned)((ncol + p.z.wb - 1) / p.z.wb), 256, p.smem_z, st>>>(work, uhat, g, p.z, tb.wz_f, symx,
                                                                                   symy, symz);
  count_launches(1);
  return cudaGetLastError();
}

#define SELM_ANY(T)                                                                                                   \
  template cudaError_t any_xy_forward<T>(const AnyPlan&, const T*, cpx<T>*, const FftTables<T>&, int, cudaStream_t);    \
  template cudaError_t any_xy_inverse<T>(const AnyPlan&, const cpx<T>*, T*, const FftTables<T>&, int, uint64_t*,         \
                                         cudaStream_t);                                                                 \
  template cudaError_t any_z_update<T>(const AnyPlan&, cpx<T>*, cpx<T>*, const ZGeom&, const FftTables<T>&,              \
                                       const double*, const double*, const double*, cudaStream_t);
SELM_ANY(float)
SELM_ANY(double)
#undef SELM_ANY

}  // namespace selm
