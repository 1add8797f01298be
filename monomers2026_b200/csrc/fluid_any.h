// fluid_any.h - plans and launchers of the spectral kernels for run-time grid
// sizes (fluid_any.cu).
#pragma once
#include <algorithm>

#include "selm_kernels.h"

namespace selm {

// u / d and u % d for u < 2^20, 1 <= d < 2^12: with m = ceil(2^32 / d) the
// product u m exceeds u 2^32 / d by less than u d / d < 2^32 / d
struct FastDiv {
  uint32_t d = 1, m = 0;  // m = 0: d = 1
};
inline FastDiv fast_div(int d) {
  FastDiv f;
  f.d = (uint32_t)d;
  f.m = d > 1 ? (uint32_t)((0x100000000ull + (uint64_t)d - 1) / (uint64_t)d) : 0u;
  return f;
}
constexpr int kMaxFactors = 3;
constexpr int kMaxRadix = 16;

struct LinePlan {
  int n = 0, np = 0;           // length, passes
  int r[kMaxFactors] = {};     // factors, in forward order
  int L[kMaxFactors] = {};     // block length of each pass
  int M[kMaxFactors] = {};     // L / r
  FastDiv dM[kMaxFactors];
  FastDiv d0, d1, dl;          // r[0], r[1] and the last factor
};

// the fewest factors, then the smallest largest factor; false: n has a prime factor above 13
inline bool make_line_plan(int n, LinePlan* out) {
  LinePlan p;
  p.n = n;
  int best = kMaxRadix + 1;
  for (int a = 1; a <= kMaxRadix && p.np == 0; a++)
    if (a == n) {
      p.np = 1;
      p.r[0] = a;
    }
  if (p.np == 0)
    for (int a = 2; a <= kMaxRadix; a++)
      if (n % a == 0 && n / a <= a && a < best) {
        best = a;
        p.np = 2;
        p.r[0] = a;
        p.r[1] = n / a;
      }
  if (p.np == 0)
    for (int a = 2; a <= kMaxRadix; a++)
      for (int b = 2; b <= a; b++)
        if (n % (a * b) == 0 && n / (a * b) <= b && a < best) {
          best = a;
          p.np = 3;
          p.r[0] = a;
          p.r[1] = b;
          p.r[2] = n / (a * b);
        }
  if (p.np == 0) return false;
  int L = n;
  for (int q = 0; q < p.np; q++) {
    p.L[q] = L;
    p.M[q] = L / p.r[q];
    p.dM[q] = fast_div(p.M[q]);
    L = p.M[q];
  }
  p.d0 = fast_div(p.r[0]);
  p.d1 = fast_div(p.np > 1 ? p.r[1] : 1);
  p.dl = fast_div(p.r[p.np - 1]);
  *out = p;
  return true;
}

// Geometry of the plane kernels: a plane of ny rows of nx values; the rows go
// in pairs (y, y + hp) as one complex line, rp pairs at a time.
struct PlaneGeom {
  LinePlan x, y;
  int nh, pitch;  // nx/2+1; row pitch of the plane in shared memory (odd: consecutive rows on distinct banks)
  int hp, rp;
  FastDiv dnx, dnh, drp;
};

// shared memory in complex values: the plane, a chunk of row pairs (stride
// rp + 1, one slot more every r_last elements), x twiddles, y twiddles, positions
inline size_t plane_smem_elems(const PlaneGeom& g) {
  const int rl = g.x.r[g.x.np - 1];
  return (size_t)g.y.n * g.pitch + (size_t)g.x.n * (g.rp + 1) + g.x.n / rl + g.x.n + g.y.n;
}

template <typename T> inline size_t plane_smem_bytes(const PlaneGeom& g) {
  return sizeof(cpx<T>) * plane_smem_elems(g) + sizeof(int) * (size_t)(g.x.n + g.y.n);
}

// Geometry of a z block: wb columns (of the flattened (y, x) half spectrum)
// by nc components, all nz planes, element (plane, component, column) of the
// block at plane nl + component wb + column (nl = nc wb).
struct PencilGeom {
  LinePlan z;
  int wb, nl;
  FastDiv dnl, dwb;
};

constexpr size_t kSmBytes = 227 * 1024;

// FP32: 64 registers a thread, blocks of up to 1024; FP64: 128 and 512
template <typename T> constexpr int plane_threads_max() { return sizeof(T) == 4 ? 1024 : 512; }

struct AnyPlan {
  PlaneGeom xy{};
  PencilGeom z{};
  size_t smem_xy = 0, smem_z = 0;
  int threads_xy = 0;
};

// The plan of an n^3 grid: false where a prime factor of n is above 13 or a
// plane does not fit in shared memory.
// Plane kernels: candidates are 1 to 4 blocks per SM, each with the fewest
// chunks that fit (at most 4) and as many threads as the registers give; taken
// is the one whose 3 n planes need the fewest block rounds (waves times blocks
// per SM), then the most blocks per SM, which fill each other's barriers.
template <typename T> bool any_plan(int n, AnyPlan* out) {
  AnyPlan p;
  if (!make_line_plan(n, &p.xy.x)) return false;
  p.xy.y = p.z.z = p.xy.x;
  p.xy.nh = n / 2 + 1;
  p.xy.pitch = p.xy.nh | 1;
  p.xy.hp = (n + 1) / 2;
  p.xy.dnx = fast_div(n);
  p.xy.dnh = fast_div(p.xy.nh);
  const int tmax = plane_threads_max<T>();
  long best = -1;
  for (int nb = 1; nb <= 4; nb++)
    for (int chunks = 1; chunks <= 4; chunks++) {
      PlaneGeom g = p.xy;
      g.rp = (g.hp + chunks - 1) / chunks;
      const size_t bytes = plane_smem_bytes<T>(g);
      if (nb * (bytes + 1024) > kSmBytes + 1024) continue;
      const long rounds = (3L * n + 148 * nb - 1) / (148 * nb) * nb;
      if (best < 0 || rounds <= best) {
        best = rounds;
        p.xy.rp = g.rp;
        p.smem_xy = bytes;
        p.threads_xy = tmax / nb / 32 * 32;
      }
      break;
    }
  if (best < 0) return false;
  p.xy.drp = fast_div(p.xy.rp);
  // z: columns of 128 bytes (16 FP32, 8 FP64), fewer where three (FP32) or two blocks would not fit on an SM
  p.z.wb = sizeof(T) == 4 ? 16 : 8;
  // (columns, twiddles, symbols of columns and planes, positions)
  auto bytes = [&](int wb) {
    return sizeof(cpx<T>) * ((size_t)n * 3 * wb + n) + col_bytes<T>() * (size_t)wb +
           (sizeof(PlaneSym<T>) + sizeof(int)) * (size_t)n;
  };
  while (p.z.wb > 4 && bytes(p.z.wb) > kSmBytes / (sizeof(T) == 4 ? 3 : 2) - 1024) p.z.wb /= 2;
  p.smem_z = bytes(p.z.wb);
  if (p.smem_z > kSmBytes) return false;
  p.z.nl = 3 * p.z.wb;
  p.z.dnl = fast_div(p.z.nl);
  p.z.dwb = fast_div(p.z.wb);
  *out = p;
  return true;
}

cudaError_t any_attrs();
template <typename T>
cudaError_t any_xy_forward(const AnyPlan& p, const T* in, cpx<T>* out, const FftTables<T>& tb, int planes,
                           cudaStream_t st);
template <typename T>
cudaError_t any_xy_inverse(const AnyPlan& p, const cpx<T>* in, T* out, const FftTables<T>& tb, int planes,
                           uint64_t* step, cudaStream_t st);
template <typename T>
cudaError_t any_z_update(const AnyPlan& p, cpx<T>* work, cpx<T>* uhat, const ZGeom& g, const FftTables<T>& tb,
                         const double* symx, const double* symy, const double* symz, cudaStream_t st);

// a stage (PlainStage) of the reference-structured form
cudaError_t any_plain_stage(int stage, const AnyPlan& p, const PlainBufs& b, const FftTables<double>& tb,
                            cudaStream_t st);

}  // namespace selm
