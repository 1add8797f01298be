// fluid_fused_fast.cuh - the fused z kernel for compile-time grid sizes
// N = N1*N2 (N1, N2 <= 16), built on the four-step FFT of fft_fast.cuh, and the
// spectral update that the run-time sizes share.  Same arithmetic contract as
// the generic kernels of fluid_fused.cu:
//   k_z_update_fast   : per block of Wb consecutive (x, y) columns of the
//                       half spectrum, three components each: z FFT, the spectral update
//                       (viscous factor, projection, Philox noise, zero mode)
//                       with u_hat read and written in place, inverse z FFT
//                       with the 1/N normalisation.
// The plane kernels before and after it are in fluid_plane.cuh.
// Shared-memory lines are stored line-fastest (element t of line l at
// t*stride + l), so threads of consecutive lines touch consecutive words.
#pragma once
#include <cuda.h>

#include <type_traits>

#include "common.cuh"
#include "fft_fast.cuh"
#include "selm_kernels.h"

namespace selm {

// ---------------------------------------------------------------- helpers
// position of natural index k after pass A + pass B (in place): N2 (k mod N1) + k / N1
template <int N1, int N2> __device__ __forceinline__ int dpos(int k) { return N2 * (k % N1) + k / N1; }

// ---------------------------------------------------------------- z pencils + update
template <typename T>
__device__ __forceinline__ ColSym<T> col_sym(const ZGeom& g, long col, const double* __restrict__ symx,
                                             const double* __restrict__ symy) {
  ColSym<T> s;
  s.j = (int)(col / g.nxh);
  s.i = (int)(col - (long)s.j * g.nxh);
  const T idx1 = (T)(1.0 / g.dx);
  s.c = symx[2 * s.i] + symy[2 * s.j];
  s.dx = fftk::mk<cpx<T>>((T)symx[2 * s.i] * idx1, (T)symx[2 * s.i + 1] * idx1);
  s.dy = fftk::mk<cpx<T>>((T)symy[2 * s.j] * idx1, (T)symy[2 * s.j + 1] * idx1);
  return s;
}
template <typename T> __device__ __forceinline__ void put_col(const ColArrays<T>& A, int w, const ColSym<T>& s) {
  A.c[w] = s.c;
  A.dx[w] = s.dx;
  A.dy[w] = s.dy;
  A.ij[w] = s.i | (s.j << 16);
}
template <typename T> __device__ __forceinline__ ColSym<T> get_col(const ColArrays<T>& A, int w) {
  const int ij = A.ij[w];
  return ColSym<T>{A.c[w], A.dx[w], A.dy[w], ij & 0xffff, ij >> 16};
}
template <typename T>
__device__ __forceinline__ PlaneSym<T> plane_sym(const ZGeom& g, int k, const double* __restrict__ symz) {
  const T idx1 = (T)(1.0 / g.dx);
  return PlaneSym<T>{symz[2 * k], fftk::mk<cpx<T>>((T)symz[2 * k] * idx1, (T)symz[2 * k + 1] * idx1)};
}

// The order in which a block updates the modes of its wn columns (from column
// c0 of the flattened half spectrum): last those of the first column on the
// planes i = 0 and i = nx/2 and of its neighbour if that is on them too (i = nx/2
// and the next row's i = 0).  These modes draw twice (the Hermitian average); in
// the columns' own order every warp of a block that holds them, a third of the
// blocks at 128^3, went through the second draw for a few lanes: 128^3 z
// kernel 57.8 -> 47.6 us FP32, 87.8 -> 82.9 FP64; 100^3 FP32 45.4 -> 35.3 (48.0
// and 37.8 since, with the draws' full precision).
struct ModeOrder {
  int n, first, edges;  // columns before the edge ones, the first of those, how many
  unsigned mn, me;      // ceil(2^32 / d) of the two groups' sizes d (0: d <= 1)
};
__device__ __forceinline__ ModeOrder mode_order(int c0, int wn, int nx, int nh) {
  const int i0 = c0 % nh;
  int first = i0 == 0 ? 0 : nx % 2 == 0 ? nh - 1 - i0 : nh - i0;
  int edges = 0;
  if (first < wn) edges = nx % 2 == 0 && i0 + first == nh - 1 && first + 1 < wn ? 2 : 1;
  ModeOrder o{wn - edges, first, edges, 0u, 0u};
  if (o.n > 1) o.mn = 0xffffffffu / (unsigned)o.n + 1u;
  if (o.edges > 1) o.me = 0x80000000u;
  return o;
}
// unit u < wn nz: column w of the block and mode k (exact while u d < 2^32)
__device__ __forceinline__ void mode_unit(const ModeOrder& o, int nz, int u, int& w, int& k) {
  const bool edge = u >= o.n * nz;
  const int v = edge ? u - o.n * nz : u;
  const unsigned m = edge ? o.me : o.mn;
  k = m ? (int)__umulhi((unsigned)v, m) : v;
  const int r = v - k * (edge ? o.edges : o.n);
  w = edge ? o.first + r : r + (r >= o.first ? o.edges : 0);
}

// reference noise draw of a half-spectrum mode (cuda/SELM_Kernel.cu:56-79).
// The FP64 forms draw FP64 normals (same stream as the plain form) and scale
// them in FP64 by coef = sqrt(lambda_h); the caller multiplies by the prefactor
// noise_amp.  The FP32 form draws FP32 normals from the same Philox counters
// (philox_normal2_f32, the FP64 normals to FP32 precision) and scales them by
// the whole per-mode amplitude coef = noise_amp sqrt(lambda_h) (times 1/sqrt 2
// for a complex draw), which is formed in FP64 and rounded to FP32 once: the
// noise-variance prefactor stays FP64 (cuda/SELM_Eulerian_Period.cu:141-148).
// W: the type of the draw; FP64 in the FP32 form takes the FP64 normals, scaled
// (and averaged, mode_update) in FP64 and rounded once.
template <typename W>
__device__ __forceinline__ void noise_draw_fast(const ZGeom& g, uint64_t step, int nz, int i, int j, int k, double coef,
                                                cpx<W> out[3]) {
  const bool selfc = (k == 0 || 2 * k == nz) && (j == 0 || 2 * j == g.ny) && (i == 0 || 2 * i == g.nx);
  const uint32_t q = (uint32_t)(((long)k * g.ny + j) * g.nxh + i);
  const double re = selfc ? coef : coef * 0.7071067811865476, im = selfc ? 0.0 : re;
  const W rew = (W)re, imw = (W)im;
#pragma unroll
  for (int d = 0; d < 3; d++) {
    W z0, z1;
    if constexpr (sizeof(W) == 8) philox_normal2(g.rk, q, (uint32_t)d, step, z0, z1);
    else philox_normal2_f32(g.rk, q, (uint32_t)d, step, z0, z1);
    out[d] = fftk::mk<cpx<W>>(z0 * rew, z1 * imw);
  }
}

// constants of the spectral update
template <typename T> struct ModeConsts {
  uint64_t step;
  double idx2, visc;  // 1/dx^2, mu dt / rho
  T invN, irho;
};
template <typename T> __device__ __forceinline__ ModeConsts<T> mode_consts(const ZGeom& g, int nz) {
  return ModeConsts<T>{*g.step, 1.0 / (g.dx * g.dx), g.mu * g.dt / g.rho, (T)(1.0 / ((double)g.nx * g.ny * nz)),
                       (T)(1.0 / g.rho)};
}

// The spectral update of mode (i, j, k), all three components: the
// transformed forcing at a[c astep] is replaced by the new velocity over N,
// u_hat (component c at uh[c cplane]) by the new velocity.  W64: the
// FP32 form draws FP64 normals (noise_draw_fast).
template <typename T, bool W64>
__device__ __forceinline__ void mode_update(const ZGeom& g, const ModeConsts<T>& mc, int nz, const ColSym<T>& col,
                                            const PlaneSym<T>& pz, int k, cpx<T>* __restrict__ uh, long cplane,
                                            cpx<T>* a, int astep) {
  using C = cpx<T>;
  const int i = col.i, j = col.j, ny = g.ny;
  const double Lk = 2.0 * (col.c + pz.c) * mc.idx2;  // sum_d 2(cos - 1)/dx^2 (<= 0)
  C X[3];
#pragma unroll
  for (int c = 0; c < 3; c++) X[c] = a[c * astep];
  const bool zero = i == 0 && j == 0 && k == 0;
  if (g.stochastic && !zero) {  // (the zero mode's draw has amplitude 0)
    double coef = sqrt(-Lk);
    if (sizeof(T) == 4) coef *= g.noise_amp;
    using W = typename std::conditional<W64, double, T>::type;
    using CW = cpx<W>;
    CW Xn[3];
    noise_draw_fast<W>(g, mc.step, nz, i, j, k, coef, Xn);
    if (i == 0 || 2 * i == g.nx) {
      const int jc = (j == 0) ? 0 : ny - j, kc = (k == 0) ? 0 : nz - k;
      if (jc != j || kc != k) {
        CW Xc[3];
        noise_draw_fast<W>(g, mc.step, nz, i, jc, kc, coef, Xc);
        const W s = (g.noise_mode == 1 || g.qs) ? W(0.7071067811865476) : W(0.5);
#pragma unroll
        for (int c = 0; c < 3; c++) Xn[c] = fftk::mk<CW>((Xn[c].x + Xc[c].x) * s, (Xn[c].y - Xc[c].y) * s);
      } else {
#pragma unroll
        for (int c = 0; c < 3; c++) Xn[c].y = W(0);
      }
    }
    // FP32: the FP64 prefactor is already in the draw
    const T amp = sizeof(T) == 8 ? (T)g.noise_amp : T(1);
#pragma unroll
    for (int c = 0; c < 3; c++) {
      X[c].x += amp * (T)Xn[c].x;
      X[c].y += amp * (T)Xn[c].y;
    }
  }
  C un[3];
  const C D[3] = {col.dx, col.dy, pz.d};
  if (zero) {
#pragma unroll
    for (int c = 0; c < 3; c++) un[c] = fftk::mk<C>(T(0), T(0));
  } else if (g.qs) {
    // steady Stokes: u_hat = P f_hat / (mu lambda_h), lambda_h = -L_h > 0
    C s = cmul(D[0], X[0]);
    s = cadd(s, cmul(D[1], X[1]));
    s = cadd(s, cmul(D[2], X[2]));
    const T iL = (T)(1.0 / Lk), imuL = (T)(-1.0 / (g.mu * Lk));
    s = fftk::mk<C>(s.x * iL, s.y * iL);
#pragma unroll
    for (int c = 0; c < 3; c++) {
      const C pf = csub(X[c], cmul(fftk::mk<C>(-D[c].x, D[c].y), s));
      un[c] = fftk::mk<C>(pf.x * imuL, pf.y * imuL);
    }
  } else {
    const T visc = (T)fma(mc.visc, Lk, 1.0);
    C us[3];
#pragma unroll
    for (int c = 0; c < 3; c++) {
      const C q = uh[c * cplane];
      us[c] = fftk::mk<C>(q.x * visc + X[c].x * mc.irho, q.y * visc + X[c].y * mc.irho);
    }
    C s = cmul(D[0], us[0]);
    s = cadd(s, cmul(D[1], us[1]));
    s = cadd(s, cmul(D[2], us[2]));
    const T iL = (T)(1.0 / Lk);
    s = fftk::mk<C>(s.x * iL, s.y * iL);
#pragma unroll
    for (int c = 0; c < 3; c++) un[c] = csub(us[c], cmul(fftk::mk<C>(-D[c].x, D[c].y), s));
  }
#pragma unroll
  for (int c = 0; c < 3; c++) {
    if (!g.qs) uh[c * cplane] = un[c];
    a[c * astep] = fftk::mk<C>(un[c].x * mc.invN, un[c].y * mc.invN);
  }
}

// ---- TMA staging of the z kernel's columns (single-CTA tensor copies, no
// multicast): one thread loads a block's WB columns x 3 components x N
// planes into shared memory on an mbarrier, and stores them back after the
// inverse pass.  Every wait is bounded: a copy that does not complete sets
// the status bit ERR_COPY_TIMEOUT and the block returns.
__device__ __forceinline__ unsigned smem_u32(const void* p) { return (unsigned)__cvta_generic_to_shared(p); }
__device__ __forceinline__ void zbar_init(unsigned long long* bar) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(smem_u32(bar)) : "memory");
  asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
}
__device__ __forceinline__ void zbar_load(void* dst, const CUtensorMap* map, unsigned long long* bar, unsigned bytes,
                                          int x, int y, int z) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)), "r"(bytes) : "memory");
  asm volatile(
      "cp.async.bulk.tensor.3d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4}], "
      "[%5];" ::"r"(smem_u32(dst)),
      "l"(map), "r"(x), "r"(y), "r"(z), "r"(smem_u32(bar))
      : "memory");
}
// true once phase 0 of the barrier has completed, false after `limit` polls
__device__ __forceinline__ bool zbar_wait(unsigned long long* bar, long limit) {
  for (long i = 0; i < limit; i++) {
    unsigned done;
    asm volatile(
        "{ .reg .pred p; mbarrier.try_wait.parity.shared::cta.b64 p, [%1], 0; selp.u32 %0, 1, 0, p; }"
        : "=r"(done)
        : "r"(smem_u32(bar))
        : "memory");
    if (done) return true;
  }
  return false;
}
__device__ __forceinline__ void zbar_store(const CUtensorMap* map, const void* src, int x, int y, int z) {
  asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  asm volatile("cp.async.bulk.tensor.3d.global.shared::cta.tile.bulk_group [%0, {%2, %3, %4}], [%1];" ::"l"(map),
               "r"(smem_u32(src)), "r"(x), "r"(y), "r"(z)
               : "memory");
  asm volatile("cp.async.bulk.commit_group;" ::: "memory");
  asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory");  // shared memory read out: the block may end
}
constexpr long kZbarPolls = 1L << 22;

// Block b of the z kernel takes the WB consecutive columns b*WB .. b*WB+WB-1 of
// the flattened (y, x) half-spectrum plane (column index j*nxh + i, also its
// offset within a z plane), the last block fewer.
// TMA: the block's columns of work come into shared memory and go back by
// tensor copies (tmap: work as [plane][component][column], 3-D, box WB x 3
// x N), instead of the passes' own global loads and stores.
template <typename T, int N, int N1_, int WB, int TPB, int MINB, bool TMA, bool W64>
__global__ void __launch_bounds__(TPB, MINB) k_z_update_fast(cpx<T>* __restrict__ work, cpx<T>* __restrict__ uhat, ZGeom g,
                                                       const cpx<T>* __restrict__ twz,
                                                       const double* __restrict__ symx,
                                                       const double* __restrict__ symy,
                                                       const double* __restrict__ symz,
                                                       const __grid_constant__ CUtensorMap tmap) {
  using C = cpx<T>;
  constexpr int N1 = N1_, N2 = N / N1_;
  static_assert(N1 * N2 == N && N1 <= 16 && N2 <= 16, "four-step split");
  constexpr int NL = 3 * WB;
  extern __shared__ __align__(128) unsigned char zsmem_raw[];
  // element t of line (c, w) at t*NL + c*WB + w; with TMA at a 128-byte
  // boundary, the tensor copies' rule (the launch adds 128 bytes for it)
  C* A = reinterpret_cast<C*>(TMA ? ((reinterpret_cast<uintptr_t>(zsmem_raw) + 127) & ~(uintptr_t)127)
                                  : reinterpret_cast<uintptr_t>(zsmem_raw));
  C* tw = A + N * NL;
  const long col0 = (long)blockIdx.x * WB;
  const long plane = g.ncol ? g.ncol : (long)g.ny * g.nxh;
  const int wn = (int)min((long)WB, plane - col0);
  __shared__ double col_c[WB];
  __shared__ C col_dx[WB], col_dy[WB];
  __shared__ int col_ij[WB];
  const ColArrays<T> col{col_c, col_dx, col_dy, col_ij};
  __shared__ PlaneSym<T> pz[N];
  __shared__ __align__(8) unsigned long long zbar;
  if constexpr (TMA) {
    if (threadIdx.x == 0) {
      zbar_init(&zbar);
      zbar_load(A, &tmap, &zbar, (unsigned)(sizeof(C) * N * NL), (int)col0, 0, 0);
    }
  }
  for (int t = threadIdx.x; t < N; t += blockDim.x) {
    tw[t] = twz[t];
    pz[t] = plane_sym<T>(g, t, symz);
  }
  if (threadIdx.x < wn) put_col(col, threadIdx.x, col_sym<T>(g, g.c0 + col0 + threadIdx.x, symx, symy));
  __syncthreads();
  if constexpr (TMA) {
    // one thread polls (bounded) and tells the block, so that all of it goes on or stops
    __shared__ int zok;
    if (threadIdx.x == 0) {
      zok = zbar_wait(&zbar, kZbarPolls);
      if (!zok && g.err) atomicOr(g.err, (uint32_t)ERR_COPY_TIMEOUT);
    }
    __syncthreads();
    if (!zok) return;  // the copy may still be in flight: its memory is left alone
  }
  // pass A forward, loading straight from global (or from the staged columns): thread (line, n2)
  for (int u = threadIdx.x; u < NL * N2; u += blockDim.x) {
    const int l = u % NL, n2 = u / NL;
    const int c = l / WB, w = l % WB;
    const bool ok = w < wn;
    const long cb = (long)c * N * plane + col0 + w;
    C v[N1];
#pragma unroll
    for (int n1 = 0; n1 < N1; n1++) {
      if constexpr (TMA) v[n1] = A[(N2 * n1 + n2) * NL + l];  // columns past the end arrive as zeros
      else v[n1] = ok ? work[cb + (N2 * n1 + n2) * plane] : fftk::mk<C>(T(0), T(0));
    }
    fftk::dft<N1, -1>(v);
#pragma unroll
    for (int k1 = 0; k1 < N1; k1++) A[(N2 * k1 + n2) * NL + l] = (k1 == 0) ? v[0] : cmul(v[k1], tw[n2 * k1]);
  }
  __syncthreads();
  // pass B forward in place: thread (line, k1); position N2 k1 + k2 then holds mode k1 + N1 k2
  for (int u = threadIdx.x; u < NL * N1; u += blockDim.x) {
    const int l = u % NL, k1 = u / NL;
    C v[N2];
#pragma unroll
    for (int n2 = 0; n2 < N2; n2++) v[n2] = A[(N2 * k1 + n2) * NL + l];
    fftk::dft<N2, -1>(v);
#pragma unroll
    for (int k2 = 0; k2 < N2; k2++) A[(N2 * k1 + k2) * NL + l] = v[k2];
  }
  __syncthreads();
  // spectral update: thread (w, k) for all three components, u_hat read and written in place
  const ModeConsts<T> mc = mode_consts<T>(g, N);
  const ModeOrder order = mode_order((int)(g.c0 + col0), wn, N, N / 2 + 1);
#pragma unroll 1
  for (int u = threadIdx.x; u < wn * N; u += blockDim.x) {
    int w, k;
    mode_unit(order, N, u, w, k);
    mode_update<T, W64>(g, mc, N, get_col(col, w), pz[k], k, uhat + (long)k * plane + col0 + w, (long)N * plane,
                        A + dpos<N1, N2>(k) * NL + w, WB);
  }
  __syncthreads();
  // pass B inverse in place: thread (line, k1)
  for (int u = threadIdx.x; u < NL * N1; u += blockDim.x) {
    const int l = u % NL, k1 = u / NL;
    C v[N2];
#pragma unroll
    for (int k2 = 0; k2 < N2; k2++) v[k2] = A[(N2 * k1 + k2) * NL + l];
    fftk::dft<N2, +1>(v);
#pragma unroll
    for (int n2 = 0; n2 < N2; n2++) {
      C w2 = tw[n2 * k1];
      w2.y = -w2.y;
      A[(N2 * k1 + n2) * NL + l] = (n2 == 0 || k1 == 0) ? v[n2] : cmul(v[n2], w2);
    }
  }
  __syncthreads();
  // pass A inverse, storing straight to global: thread (line, n2)
  for (int u = threadIdx.x; u < NL * N2; u += blockDim.x) {
    const int l = u % NL, n2 = u / NL;
    const int c = l / WB, w = l % WB;
    C v[N1];
#pragma unroll
    for (int k1 = 0; k1 < N1; k1++) v[k1] = A[(N2 * k1 + n2) * NL + l];
    fftk::dft<N1, +1>(v);
    if constexpr (TMA) {
#pragma unroll
      for (int n1 = 0; n1 < N1; n1++) A[(N2 * n1 + n2) * NL + l] = v[n1];  // the thread's own positions
    } else if (w < wn) {
      const long cb = (long)c * N * plane + col0 + w;
#pragma unroll
      for (int n1 = 0; n1 < N1; n1++) work[cb + (N2 * n1 + n2) * plane] = v[n1];
    }
  }
  if constexpr (TMA) {
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");  // this thread's writes, seen by the copy
    __syncthreads();
    if (threadIdx.x == 0) zbar_store(&tmap, A, (int)col0, 0, 0);  // columns past the end are not written
  }
}

}  // namespace selm
