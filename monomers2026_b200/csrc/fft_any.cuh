// fft_any.cuh - line FFTs of run-time length in shared memory, built on the
// in-register DFTs of fft_fast.cuh.
//
// A length n whose prime factors are at most 13 splits into one to three
// factors of at most 16 (LinePlan), and the FFT takes one pass over shared
// memory per factor: a thread holds one factor's points of one line in
// registers, does the DFT with compile-time twiddles and multiplies by the
// table's twiddles of the split.  With L the length of a pass' blocks, R its
// factor and M = L / R:
//   forward order (lines_dif): element M n1 + n2 of a block -> R-point DFT over
//     n1, times W_L^{n2 k1}, stored at M k1 + n2; the next pass transforms the
//     blocks of M.  Natural input; mode k ends at position pos(k).
//   backward order (lines_dit): the same passes in the opposite order, twiddles
//     before the DFT.  Input at pos(k), natural output.
// Everything is in place, one buffer, with the passes' indices worked out by
// multiplication (FastDiv).  Against the Stockham stages of common.cuh
// (radix 2-7 by run-time loops over local arrays, two buffers, an integer
// division or two per point): the FP32 step at 100^3 637 -> 200 us, at 192^3
// 2976 -> 763.  The same size at compile time is 1.3 to 2 times faster (128^3
// plane kernels 49 us here against 25, twice the instructions): what has such
// kernels takes them.
#pragma once
#include "common.cuh"
#include "fft_fast.cuh"
#include "fluid_any.h"

namespace selm {

__device__ __forceinline__ int div_by(const FastDiv& f, int u) {
  return f.m ? (int)__umulhi((uint32_t)u, f.m) : u;
}

// block of the last pass that holds the modes q + (n / r_last) k, q < n / r_last
__device__ __forceinline__ int mode_block(const LinePlan& p, int q) {
  if (p.np < 3) return q;
  const int k2 = div_by(p.d0, q);  // q = k1 + r0 k2
  return (q - k2 * p.r[0]) * p.r[1] + k2;
}
// position of mode k after lines_dif
__device__ __forceinline__ int mode_pos(const LinePlan& p, int k) {
  if (p.np == 1) return k;
  const int nq = p.np == 2 ? p.r[0] : p.r[0] * p.r[1];
  int kl = 0;  // k / nq (at most 16 steps: tables are filled once per block)
  while (k >= nq) {
    k -= nq;
    kl++;
  }
  return mode_block(p, k) * p.r[p.np - 1] + kl;
}

// first mode of block blk of the last pass (the inverse of mode_block)
__device__ __forceinline__ int block_mode(const LinePlan& p, int blk) {
  if (p.np < 3) return blk;
  const int k1 = div_by(p.d1, blk);  // blk = k1 r1 + k2
  return k1 + (blk - k1 * p.r[1]) * p.r[0];
}

template <int R> struct RadixC {
  static constexpr int value = R;
};
// f(RadixC<r>{}) for the run-time factor r (the same for every thread)
template <typename F> __device__ __forceinline__ void with_radix(int r, F&& f) {
  switch (r) {
#define SELM_RADIX(R)    \
  case R:                \
    f(RadixC<R>{});      \
    break;
    SELM_RADIX(2) SELM_RADIX(3) SELM_RADIX(4) SELM_RADIX(5) SELM_RADIX(6) SELM_RADIX(7) SELM_RADIX(8) SELM_RADIX(9)
    SELM_RADIX(10) SELM_RADIX(11) SELM_RADIX(12) SELM_RADIX(13) SELM_RADIX(14) SELM_RADIX(15) SELM_RADIX(16)
#undef SELM_RADIX
    default:
      break;
  }
}

// v[j] *= W_n^{S t j} from the table tw of W_n^{-t} (sign -1)
template <int R, int S, typename C> __device__ __forceinline__ void twiddle_points(C (&v)[R], const C* tw, int t) {
#pragma unroll
  for (int j = 1; j < R; j++) {
    C w = tw[t * j];
    if (S > 0) w.y = -w.y;
    v[j] = cmul(v[j], w);
  }
}

// One pass over nl lines in shared memory, in place: element e of line l at
// s[e stride + (e / r_last) pad + l].  DIT: the backward order.
template <int S, bool DIT, typename C>
__device__ __forceinline__ void smem_pass(const LinePlan& p, int q, int nl, const FastDiv& dnl, const C* tw, C* s,
                                          int stride, int pad) {
  const int L = p.L[q], M = p.M[q], rl = p.r[p.np - 1];
  const int step = M * stride + (M > 1 ? (M == rl ? 1 : div_by(p.dl, M)) * pad : 0);
  with_radix(p.r[q], [&](auto rc) {
    constexpr int R = decltype(rc)::value;
    const int units = nl * (p.n / R), ts = p.n / L;
    for (int u = threadIdx.x; u < units; u += blockDim.x) {
      const int rest = div_by(dnl, u), l = u - rest * nl;
      const int blk = div_by(p.dM[q], rest), n2 = rest - blk * M, x0 = blk * L + n2;
      C* e = s + x0 * stride + (pad ? div_by(p.dl, x0) * pad : 0) + l;
      C v[R];
#pragma unroll
      for (int j = 0; j < R; j++) v[j] = e[j * step];
      if (DIT && M > 1) twiddle_points<R, S>(v, tw, ts * n2);
      fftk::dft<R, S>(v);
      if (!DIT && M > 1) twiddle_points<R, S>(v, tw, ts * n2);
#pragma unroll
      for (int j = 0; j < R; j++) e[j * step] = v[j];
    }
  });
}

}  // namespace selm
