// fluid_fast.h - launchers of the compile-time spectral kernels
// (fluid_plane.cuh, fluid_fused_fast.cuh), instantiated by fluid_fast32.cu and
// fluid_fast64.cu.
#pragma once
#include <cuda.h>

#include "selm_kernels.h"

namespace selm {

// Sizes with two four-step splits to choose from (the tuning knob) and, in
// FP32, the fast FP32 normals.
#define SELM_TUNED_SIZES(X) X(16) X(24) X(30) X(32) X(48) X(64) X(96) X(128)
// The other sizes: even with prime factors up to 7, two factors of at most 16
// of which the plane kernels' first is even and the second at most 14 (two
// groups of the second are held in registers), up to the largest plane that
// fits in shared memory (224 in FP32, 160 in FP64).  Their FP32 form draws FP64
// normals: the velocity's error against 64 bits is 2.1e-7 over these sizes,
// with the fast FP32 ones 2.5e-7 to 3.2e-7.
#define SELM_EVEN_SIZES_64(X)                                                                                       \
  X(36) X(40) X(42) X(50) X(54) X(56) X(60) X(70) X(72) X(80) X(84) X(90) X(98) X(100) X(108) X(112) X(120) X(126) \
      X(140) X(144) X(160)
#define SELM_EVEN_SIZES_ABOVE_64(X) X(168) X(192) X(196) X(224)
#define SELM_EVEN_SIZES_32(X) SELM_EVEN_SIZES_64(X) SELM_EVEN_SIZES_ABOVE_64(X)

// the z kernel's TMA staging: FP32 grids of kZTmaSize^3, kZTmaColumns columns a block
constexpr int kZTmaSize = 128, kZTmaColumns = 20;
constexpr int kZDefaultBlocksPerSm = 3;

enum FluidStage { kStageXyForward = 0, kStageZ = 1, kStageXyInverse = 2 };
template <typename T> struct FastBufs {
  const T* fp;     // spread impulse, planes of the forward stage
  cpx<T>* work;    // half spectrum (the z stage: the columns)
  cpx<T>* uhat;
  T* u;
};

bool fast_tuned_size(int n);
bool fast_size(int n, int precision);
template <typename T> cudaError_t fast_attrs_for(int n);
// One stage of the fluid solve: planes (xy stages) or ncol columns (z).
// split 0: the four-step split with the largest factor, 1: the most balanced
// one (the tuned sizes; the others have the balanced one only).
template <typename T>
cudaError_t fast_stage(int stage, int n, int split, int z_blocks_per_sm, const FastBufs<T>& b, const ZGeom& zg,
                       const FftTables<T>& tb, const double* symx, const double* symy, const double* symz, int planes,
                       long ncol, const CUtensorMap* zmap, cudaStream_t st);

// the reference-structured FP64 form's stages (PlainStage), fast_size(n, 64)
cudaError_t plain_fast_attrs(int n);
cudaError_t plain_fast_stage(int stage, int n, const PlainBufs& b, const FftTables<double>& tb, cudaStream_t st);

}  // namespace selm
