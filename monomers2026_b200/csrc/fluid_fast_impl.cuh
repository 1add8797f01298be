// fluid_fast_impl.cuh - instantiation of the compile-time spectral kernels for
// one precision (included by fluid_fast32.cu and fluid_fast64.cu).
#pragma once
#include "fluid_fast.h"
#include "fluid_fused_fast.cuh"
#include "fluid_plane.cuh"

namespace selm {

template <typename T, int N> constexpr bool tuned_size() {
  switch (N) {
#define SELM_CASE(M) case M:
    SELM_TUNED_SIZES(SELM_CASE)
#undef SELM_CASE
    return true;
    default:
      return false;
  }
}

// First factor of the plane kernels: N1 if even, else the largest even one.
template <int N, int N1> constexpr int plane_n1() {
  int a = 16;
  while (N % a != 0 || N / a > 16) a -= 2;
  return N1 % 2 == 0 ? N1 : a;
}
// The most balanced split with an even first factor (14 at most for the second).
template <int N> constexpr int plane_balanced() {
  int best = 0, worst = 1 << 20;
  for (int a = 2; a <= 16; a += 2)
    if (N % a == 0 && N / a <= 14) {
      const int m = a > N / a ? a : N / a;
      if (m <= worst) {
        worst = m;
        best = a;
      }
    }
  return best;
}

// Shape of a z-kernel block: WB columns, TPB threads, at least MINB blocks
// per SM (register bound).  FP32: three, 80 registers a thread; left alone
// 96^3 and 48^3 took 84, which is two blocks: nothing alone (25.0 us at 96^3), but
// 48 members at 32^3 to 96^3, which share the SMs, 1.11 -> 1.17 ms a step.
// The 128^3 FP32 kernel takes 20 columns in blocks held to three per SM's
// registers: its 416 blocks then all fit at once, where 16 columns left a
// second wave of 76 blocks (measured, when the kernel took 64 us, against 78
// with 19 columns; 48.0 us now, bound by issue and dependent arithmetic, its 102
// MB take 16; 20 makes the block's columns a whole number of 16-byte units,
// which its tensor copies need: kTma).  FP64 at 128^3, 83 us for 204 MB that
// take 31, has the same bound with two blocks of 128 registers a thread: 10
// columns (three waves instead of four) measured 82.5.  The sizes that are not tuned take the multiple
// of 4 (32-byte runs) up to 24 (FP32) or 12 (FP64) with the least of: columns
// on the fullest SM, as iterations of the update over the SM's threads, plus
// half an iteration of latency for each of a block's, in every wave; from 8
// columns on where those fill the chip once (192^3 FP32, with shorter normals: 201 us with the model's 4, 183).
template <typename T, int N> struct ZShape {
  static constexpr bool kTuned = tuned_size<T, N>();
  static constexpr bool kWide = sizeof(T) == 4 && N == kZTmaSize;
  static constexpr bool kTma = kWide;
  static constexpr int TPB = 256;
  static constexpr int MINB = sizeof(T) == 8 ? 2 : 3;
  static constexpr int columns() {
    if (kTuned) return sizeof(T) == 8 ? 8 : (kWide ? kZTmaColumns : 16);
    constexpr long ncol = (long)N * (N / 2 + 1);
    constexpr int least = ncol >= 8L * 148 * MINB ? 8 : 4;
    int best = least;
    long cost = -1;
    for (int wb = least; wb <= (sizeof(T) == 4 ? 24 : 12); wb += 4) {
      const long smem = (long)sizeof(cpx<T>) * (3L * N * wb + N) + 1024;
      if (MINB * smem > 228 * 1024) break;
      const long blocks = (ncol + wb - 1) / wb, waves = (blocks + 148 * MINB - 1) / (148 * MINB);
      const long iters = (wb * N + TPB - 1) / TPB;
      const long c = 2 * ((blocks + 147) / 148) * wb * N / (MINB * TPB) + iters * waves;
      if (cost < 0 || c <= cost) {
        cost = c;
        best = wb;
      }
    }
    return best;
  }
  static constexpr int WB = columns();
};
static_assert(ZShape<float, kZTmaSize>::WB == kZTmaColumns, "the tensor map's box");

// Shared memory of the z kernel: what its lines need, or more when the
// blocks per SM are capped (the request then leaves room for no more).  By
// default at most three blocks share an SM: with the 128^3 FP32 kernel, four
// resident blocks per SM measured slower than three.
template <typename T, int N> constexpr size_t smem_z_need() {
  // the TMA form places its columns at a 128-byte boundary: up to 128 bytes more
  return sizeof(cpx<T>) * ((size_t)N * 3 * ZShape<T, N>::WB + N) + (ZShape<T, N>::kTma ? 128 : 0);
}
inline size_t smem_z_request(size_t need, int blocks_per_sm) {
  if (blocks_per_sm <= 0) return need;
  const size_t cap = 228 * 1024 / (size_t)(blocks_per_sm + 1) + 1024;  // blocks_per_sm + 1 do not fit
  return need < cap ? cap : need;
}
constexpr size_t kZSmemMax = 228 * 1024 / 3 + 1024;  // the largest capped request (two blocks per SM)

template <typename T, int N, int N1, int NP> struct FastKernels {
  using Z = ZShape<T, N>;
  using P = PlaneShape<T, N, NP>;
  static constexpr bool kWide64 = sizeof(T) == 4 && !Z::kTuned;

  static cudaError_t attrs() {
    cudaError_t e;
    for (const void* k : {(const void*)k_xy_forward_fast<T, N, NP, ArrayPlanes<T>>, (const void*)k_xy_inverse_fast<T, N, NP>})
      if ((e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)P::smem))) return e;
    const size_t zmax = smem_z_need<T, N>() > kZSmemMax ? smem_z_need<T, N>() : kZSmemMax;
    if constexpr (Z::kTma) {
      if ((e = cudaFuncSetAttribute((const void*)k_z_update_fast<T, N, N1, Z::WB, Z::TPB, Z::MINB, true, kWide64>,
                                    cudaFuncAttributeMaxDynamicSharedMemorySize, (int)zmax)))
        return e;
    }
    return cudaFuncSetAttribute((const void*)k_z_update_fast<T, N, N1, Z::WB, Z::TPB, Z::MINB, false, kWide64>,
                                cudaFuncAttributeMaxDynamicSharedMemorySize, (int)zmax);
  }

  static cudaError_t run(int stage, int z_blocks_per_sm, const FastBufs<T>& b, const ZGeom& zg, const FftTables<T>& tb,
                         const double* symx, const double* symy, const double* symz, int planes, long ncol,
                         const CUtensorMap* zmap, cudaStream_t st) {
    count_launches(1);
    if (stage == kStageXyForward) {
      k_xy_forward_fast<T, N, NP><<<(unsigned)planes, P::TPB, P::smem, st>>>(ArrayPlanes<T>{b.fp}, b.work, tb.wx_f);
    } else if (stage == kStageXyInverse) {
      k_xy_inverse_fast<T, N, NP><<<(unsigned)planes, P::TPB, P::smem, st>>>(b.work, b.u, tb.wx_f, (uint64_t*)zg.step);
    } else {
      const unsigned nb = (unsigned)((ncol + Z::WB - 1) / Z::WB);
      const size_t zs = smem_z_request(smem_z_need<T, N>(), z_blocks_per_sm);
      if constexpr (Z::kTma) {
        if (zmap) {  // the block's columns by tensor copies (the map covers work)
          k_z_update_fast<T, N, N1, Z::WB, Z::TPB, Z::MINB, true, kWide64><<<nb, Z::TPB, zs, st>>>(
              b.work, b.uhat, zg, tb.wz_f, symx, symy, symz, *zmap);
          return cudaGetLastError();
        }
      }
      k_z_update_fast<T, N, N1, Z::WB, Z::TPB, Z::MINB, false, kWide64><<<nb, Z::TPB, zs, st>>>(
          b.work, b.uhat, zg, tb.wz_f, symx, symy, symz, CUtensorMap{});
    }
    return cudaGetLastError();
  }
};

template <typename T, int N> using FastLargest = FastKernels<T, N, fftk::Split<N>::N1, plane_n1<N, fftk::Split<N>::N1>()>;
template <typename T, int N> using FastBalanced = FastKernels<T, N, fftk::SplitBalanced<N>::N1, plane_balanced<N>()>;


template <typename T> cudaError_t fast_attrs_for(int n) {
  switch (n) {
#define SELM_CASE(N)                                \
  case N: {                                         \
    const cudaError_t e = FastLargest<T, N>::attrs(); \
    return e ? e : FastBalanced<T, N>::attrs();     \
  }
    SELM_TUNED_SIZES(SELM_CASE)
#undef SELM_CASE
#define SELM_CASE(N) \
  case N:            \
    return FastBalanced<T, N>::attrs();
    SELM_EVEN_SIZES(SELM_CASE)
#undef SELM_CASE
    default:
      return cudaErrorInvalidValue;
  }
}

template <typename T>
cudaError_t fast_stage(int stage, int n, int split, int z_blocks_per_sm, const FastBufs<T>& b, const ZGeom& zg,
                       const FftTables<T>& tb, const double* symx, const double* symy, const double* symz, int planes,
                       long ncol, const CUtensorMap* zmap, cudaStream_t st) {
  switch (n) {
#define SELM_CASE(N)                                                                                              \
  case N:                                                                                                         \
    if (split == 1)                                                                                               \
      return FastBalanced<T, N>::run(stage, z_blocks_per_sm, b, zg, tb, symx, symy, symz, planes, ncol, zmap, st); \
    return FastLargest<T, N>::run(stage, z_blocks_per_sm, b, zg, tb, symx, symy, symz, planes, ncol, zmap, st);
    SELM_TUNED_SIZES(SELM_CASE)
#undef SELM_CASE
#define SELM_CASE(N) \
  case N:            \
    return FastBalanced<T, N>::run(stage, z_blocks_per_sm, b, zg, tb, symx, symy, symz, planes, ncol, zmap, st);
    SELM_EVEN_SIZES(SELM_CASE)
#undef SELM_CASE
    default:
      return cudaErrorInvalidValue;
  }
}

}  // namespace selm
