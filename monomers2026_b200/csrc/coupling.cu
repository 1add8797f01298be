// coupling.cu - monomer <-> grid coupling on sm_100a.
//
//  * bin_particles  : counting sort of monomers into buckets (grid tiles for
//                     the coupling, force cells for the pair list).  Bucket
//                     contents are ordered by monomer index, so every later
//                     traversal has a fixed order.
//  * interp_update  : Peskin 4-point interpolation of the staggered velocity
//                     (gamma(), cuda/SELM_Kernel.cu:375-422) fused with the
//                     drag/noise impulse and the explicit monomer update of
//                     lagrangian_update() (cuda/SELM_Kernel.cu:302-373).
//  * spread         : the spreading lambda() (cuda/SELM_Kernel.cu:424-470) by
//                     tiles of 16 x 8 x 16 cells accumulated in shared memory
//                     in fixed point, so results do not depend on candidate
//                     order or scheduling; FP32 with many monomers by boxes
//                     with a halo and a fold of the boxes.
#include <algorithm>
#include <mutex>
#include <type_traits>

#include "common.cuh"
#include "selm_kernels.h"

namespace selm {

// ================================================================ binning
__device__ __forceinline__ int axis_bucket(double x, int a, const BinSpec& bs) {
  int c;
  if (bs.mode == 0) {
    c = (int)floor((x - bs.lo) / bs.dx);
    c = wrapi(c, bs.n[a]);
    return c / bs.tile[a];
  }
  c = (int)floor((x - bs.lo) / bs.L * bs.n[a]);
  return wrapi(c, bs.n[a]);
}

__global__ void k_bin_count(const double* __restrict__ x, int M, BinSpec bs, int* __restrict__ bucket_of,
                            int* __restrict__ counts) {
  const int p = blockIdx.x * blockDim.x + threadIdx.x;
  if (p >= M) return;
  int b3[3];
#pragma unroll
  for (int a = 0; a < 3; a++) {
    const double xa = x[3 * p + a];
    b3[a] = isfinite(xa) ? axis_bucket(xa, a, bs) : 0;
  }
  const int b = (b3[2] * bs.nb[1] + b3[1]) * bs.nb[0] + b3[0];
  bucket_of[p] = b;
  atomicAdd(&counts[b], 1);
}

// Mode 2: file a monomer under every spread tile its union stencil reaches.
__device__ __forceinline__ int axis_tiles(double x, int a, const BinSpec& bs, int out[5]) {
  double g = (x - bs.lo) / bs.dx;
  if (!isfinite(g)) g = 0.0;
  const int c0 = (int)floor(g - 0.5) - 1;
  int cnt = 0;
  for (int i = 0; i < 5; i++) {
    const int t = wrapi(c0 + i, bs.n[a]) / bs.tile[a];
    bool dup = false;
    for (int j = 0; j < cnt; j++) dup |= (out[j] == t);
    if (!dup) out[cnt++] = t;
  }
  return cnt;
}

// the same from a stored stencil: c0 = wrapped shifted base of the axis
__device__ __forceinline__ int axis_tiles_from_base(int c0, int a, const BinSpec& bs, int out[5]) {
  int cnt = 0;
  for (int i = 0; i < 5; i++) {
    int c = c0 + i;
    if (c >= bs.n[a]) c -= bs.n[a];
    const int t = c / bs.tile[a];
    bool dup = false;
    for (int j = 0; j < cnt; j++) dup |= (out[j] == t);
    if (!dup) out[cnt++] = t;
  }
  return cnt;
}

__device__ __forceinline__ void monomer_tiles(const double* __restrict__ x, const int* __restrict__ rec_b,
                                              int rec_stride, int p, const BinSpec& bs, int (&tx)[5], int (&ty)[5],
                                              int (&tz)[5], int& nxt, int& nyt, int& nzt) {
  if (rec_b) {
    const int* b = rec_b + (long)p * rec_stride;  // b[axis][shift]
    nxt = axis_tiles_from_base(b[1], 0, bs, tx);
    nyt = axis_tiles_from_base(b[3], 1, bs, ty);
    nzt = axis_tiles_from_base(b[5], 2, bs, tz);
  } else {
    nxt = axis_tiles(x[3 * p], 0, bs, tx);
    nyt = axis_tiles(x[3 * p + 1], 1, bs, ty);
    nzt = axis_tiles(x[3 * p + 2], 2, bs, tz);
  }
}

__global__ void k_bin_count_multi(const double* __restrict__ x, const int* __restrict__ rec_b, int rec_stride, int M,
                                  BinSpec bs, int* __restrict__ counts) {
  const int p = blockIdx.x * blockDim.x + threadIdx.x;
  if (p >= M) return;
  int tx[5], ty[5], tz[5], nxt, nyt, nzt;
  monomer_tiles(x, rec_b, rec_stride, p, bs, tx, ty, tz, nxt, nyt, nzt);
  for (int k = 0; k < nzt; k++)
    for (int j = 0; j < nyt; j++)
      for (int i = 0; i < nxt; i++) atomicAdd(&counts[(tz[k] * bs.nb[1] + ty[j]) * bs.nb[0] + tx[i]], 1);
}

__global__ void k_bin_scatter_multi(const double* __restrict__ x, const int* __restrict__ rec_b, int rec_stride,
                                    int M, BinSpec bs, int* __restrict__ cursor, int* __restrict__ unsorted) {
  const int p = blockIdx.x * blockDim.x + threadIdx.x;
  if (p >= M) return;
  int tx[5], ty[5], tz[5], nxt, nyt, nzt;
  monomer_tiles(x, rec_b, rec_stride, p, bs, tx, ty, tz, nxt, nyt, nzt);
  for (int k = 0; k < nzt; k++)
    for (int j = 0; j < nyt; j++)
      for (int i = 0; i < nxt; i++) {
        const int pos = atomicAdd(&cursor[(tz[k] * bs.nb[1] + ty[j]) * bs.nb[0] + tx[i]], 1);
        unsorted[pos] = p;
      }
}

__global__ void k_bin_scatter(const int* __restrict__ bucket_of, int M, int* __restrict__ cursor,
                              int* __restrict__ unsorted) {
  const int p = blockIdx.x * blockDim.x + threadIdx.x;
  if (p >= M) return;
  const int pos = atomicAdd(&cursor[bucket_of[p]], 1);
  unsorted[pos] = p;
}

// One thread per bucket: rank of every member by monomer index.  Buckets with
// more than kThreadSortMax members (dense clusters, or every monomer of a job
// whose state went non-finite) are queued for k_bucket_sort_big instead.
constexpr int kThreadSortMax = 32;
__global__ void k_bucket_sort(const int* __restrict__ offsets, int nbuckets, const int* __restrict__ unsorted,
                              int* __restrict__ sorted, int* __restrict__ big_list, int* __restrict__ big_count) {
  const int b = blockIdx.x * blockDim.x + threadIdx.x;
  if (b >= nbuckets) return;
  const int s = offsets[b], n = offsets[b + 1] - s;
  if (n > kThreadSortMax) {
    big_list[atomicAdd(big_count, 1)] = b;
    return;
  }
  for (int i = 0; i < n; i++) {
    const int id = unsorted[s + i];
    int rank = 0;
    for (int j = 0; j < n; j++) rank += (unsorted[s + j] < id);
    sorted[s + rank] = id;
  }
}

// Large buckets: one block per bucket (grid-stride over the queued list),
// members staged in shared memory when they fit.
constexpr int kBigSortThreads = 1024, kBigSortSmem = 8192;
__global__ void __launch_bounds__(kBigSortThreads) k_bucket_sort_big(const int* __restrict__ offsets,
                                                                     const int* __restrict__ unsorted,
                                                                     int* __restrict__ sorted,
                                                                     const int* __restrict__ big_list,
                                                                     const int* __restrict__ big_count) {
  __shared__ int ids[kBigSortSmem];
  const int nbig = *big_count;
  for (int q = blockIdx.x; q < nbig; q += gridDim.x) {
    const int b = big_list[q];
    const int s = offsets[b], n = offsets[b + 1] - s;
    const bool staged = n <= kBigSortSmem;
    __syncthreads();
    if (staged)
      for (int i = threadIdx.x; i < n; i += blockDim.x) ids[i] = unsorted[s + i];
    __syncthreads();
    const int* src = staged ? ids : unsorted + s;
    for (int i = threadIdx.x; i < n; i += blockDim.x) {
      const int id = src[i];
      int rank = 0;
      for (int j = 0; j < n; j++) rank += (src[j] < id);
      sorted[s + rank] = id;
    }
  }
}

// ---- exclusive scan over n ints (two levels of 4096-element blocks)
constexpr int kScanThreads = 1024, kScanIpt = 4, kScanBlock = kScanThreads * kScanIpt;

__device__ __forceinline__ int block_exclusive_scan(int v, int* sh_warp, int& total) {
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  int incl = v;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int t = __shfl_up_sync(0xffffffffu, incl, o);
    if (lane >= o) incl += t;
  }
  if (lane == 31) sh_warp[wid] = incl;
  __syncthreads();
  if (wid == 0) {
    int w = (lane < (int)(blockDim.x >> 5)) ? sh_warp[lane] : 0;
    int wi = w;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int t = __shfl_up_sync(0xffffffffu, wi, o);
      if (lane >= o) wi += t;
    }
    sh_warp[lane] = wi - w;  // exclusive warp offsets
    if (lane == 31) sh_warp[32] = wi;
  }
  __syncthreads();
  total = sh_warp[32];
  const int r = sh_warp[wid] + incl - v;
  __syncthreads();
  return r;
}

__global__ void k_scan_block(const int* __restrict__ in, int* __restrict__ out, long n, int* __restrict__ bsum,
                             const int* __restrict__ flag) {
  if (flag && *flag == 0) return;
  __shared__ int sh[33];
  const long base = (long)blockIdx.x * kScanBlock + (long)threadIdx.x * kScanIpt;
  int v[kScanIpt];
  int s = 0;
#pragma unroll
  for (int q = 0; q < kScanIpt; q++) {
    v[q] = (base + q < n) ? in[base + q] : 0;
    s += v[q];
  }
  int total;
  int run = block_exclusive_scan(s, sh, total);
#pragma unroll
  for (int q = 0; q < kScanIpt; q++) {
    if (base + q < n) out[base + q] = run;
    run += v[q];
  }
  if (threadIdx.x == 0 && bsum) bsum[blockIdx.x] = total;
}

// one element per thread: every block-level offset is added by an independent load and store
__global__ void k_scan_add(int* __restrict__ out, long n, const int* __restrict__ boff, const int* __restrict__ flag) {
  if (flag && *flag == 0) return;
  const long i = (long)blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n && i >= kScanBlock) out[i] += boff[i / kScanBlock];
}

long scan_tmp_size(long n) {
  const long nb = (n + kScanBlock - 1) / kScanBlock;
  return 2 * nb + 2;
}

cudaError_t exclusive_scan(const int* in, int* out, long n, int* tmp, cudaStream_t st, const int* flag) {
  const long nb = (n + kScanBlock - 1) / kScanBlock;
  if (nb > kScanBlock) return cudaErrorInvalidValue;
  if (nb == 1) {
    k_scan_block<<<1, kScanThreads, 0, st>>>(in, out, n, nullptr, flag);
    count_launches(1);
    return cudaGetLastError();
  }
  int* bsum = tmp;
  int* boff = tmp + nb;
  k_scan_block<<<(unsigned)nb, kScanThreads, 0, st>>>(in, out, n, bsum, flag);
  count_launches(1);
  k_scan_block<<<1, kScanThreads, 0, st>>>(bsum, boff, nb, nullptr, flag);
  count_launches(1);
  k_scan_add<<<(unsigned)((n + 255) / 256), 256, 0, st>>>(out, n, boff, flag);
  count_launches(1);
  return cudaGetLastError();
}

cudaError_t bin_particles(const double* x, int M, const BinSpec& bs, const BinBuffers& bb, cudaStream_t st,
                          const int* rec_b, int rec_stride) {
  const long nbk = (long)bs.nb[0] * bs.nb[1] * bs.nb[2];
  cudaError_t e = cudaMemsetAsync(bb.counts, 0, sizeof(int) * (nbk + 1), st);
  if (e != cudaSuccess) return e;
  if (M > 0) {
    if (bs.mode == 2)
      k_bin_count_multi<<<(M + 255) / 256, 256, 0, st>>>(x, rec_b, rec_stride, M, bs, bb.counts);
    else k_bin_count<<<(M + 255) / 256, 256, 0, st>>>(x, M, bs, bb.bucket_of, bb.counts);
    count_launches(1);
  }
  if ((e = exclusive_scan(bb.counts, bb.offsets, nbk + 1, bb.scan_tmp, st)) != cudaSuccess) return e;
  if ((e = cudaMemcpyAsync(bb.cursor, bb.offsets, sizeof(int) * nbk, cudaMemcpyDeviceToDevice, st)) != cudaSuccess)
    return e;
  if (M > 0) {
    if (bs.mode == 2) {
      // spread tiles: the fixed-point spread does not depend on the order inside a bucket
      k_bin_scatter_multi<<<(M + 255) / 256, 256, 0, st>>>(x, rec_b, rec_stride, M, bs, bb.cursor, bb.sorted);
      count_launches(1);
      return cudaGetLastError();
    }
    k_bin_scatter<<<(M + 255) / 256, 256, 0, st>>>(bb.bucket_of, M, bb.cursor, bb.unsorted);
    count_launches(1);
    if ((e = cudaMemsetAsync(bb.big_count, 0, sizeof(int), st)) != cudaSuccess) return e;
    k_bucket_sort<<<(unsigned)((nbk + 255) / 256), 256, 0, st>>>(bb.offsets, (int)nbk, bb.unsorted, bb.sorted,
                                                                 bb.big_list, bb.big_count);
    count_launches(1);
    k_bucket_sort_big<<<148, kBigSortThreads, 0, st>>>(bb.offsets, bb.unsorted, bb.sorted, bb.big_list, bb.big_count);
    count_launches(1);
  }
  return cudaGetLastError();
}

// ================================================================ Peskin weights
// Weight factor of the reference's loop nest for a distance r (grid units):
// the branches of cuda/SELM_Kernel.cu:391-395; a distance of exactly 2 (a
// coordinate on a grid node) leaves the factor at 1.0 there, which is kept.
// The branch is taken on the FP64 distance so that the FP32 form never rounds
// a distance just below 2 onto the edge case.
template <typename T> __device__ __forceinline__ T ref_weight(double rd) {
  const T r = (T)rd;
  if (rd < 1.0) return (T(3) - T(2) * r + sqrt(T(1) + T(4) * r * (T(1) - r))) / T(8);
  if (rd < 2.0) return (T(5) - T(2) * r - sqrt(T(-7) + T(4) * r * (T(3) - r))) / T(8);
  return T(1);
}

// gamma() of cuda/SELM_Kernel.cu:375-422 (same loop and product order)
template <typename T>
__device__ __forceinline__ T interp_one(double rx, double ry, double rz, int Nx, int Ny, int Nz,
                                        const T* __restrict__ u) {
  const int p0 = (int)floor(rx) - 1, p1 = (int)floor(ry) - 1, p2 = (int)floor(rz) - 1;
  T wx[4], wy[4];
#pragma unroll
  for (int i = 0; i < 4; i++) {
    wx[i] = ref_weight<T>(fabs(rx - (double)(p0 + i)));
    wy[i] = ref_weight<T>(fabs(ry - (double)(p1 + i)));
  }
  int ix[4];
#pragma unroll
  for (int i = 0; i < 4; i++) ix[i] = wrapi(p0 + i, Nx);
  T rv = T(0);
#pragma unroll
  for (int k = 0; k < 4; k++) {
    const T dk = T(1) * ref_weight<T>(fabs(rz - (double)(p2 + k)));
    const long zoff = (long)wrapi(p2 + k, Nz) * Ny;
#pragma unroll
    for (int j = 0; j < 4; j++) {
      const T dj = dk * wy[j];
      const T* row = u + (zoff + wrapi(p1 + j, Ny)) * Nx;
#pragma unroll
      for (int i = 0; i < 4; i++) rv += __ldg(row + ix[i]) * (dj * wx[i]);
    }
  }
  return rv;
}

// Spread tiles: kTX x kTY x kTZ cells (see the spread below).
constexpr int kTX = 16, kTY = 8, kTZ = 16;  // 16 cells in z: fewer candidates straddle two tiles
static_assert(kTX == kTZ, "tile indices of x and z");

// Home cell of a grid coordinate along one axis: floor(g) wrapped into
// [0, n), and whether frac(g) < 1/2 (the half-shifted stencil then starts two
// cells below it, else one).  Non-finite or absurd coordinates count as 0, so
// that tile and box indices stay in range (their impulses are non-finite
// anyway, or the step has already flagged the displacement).
__device__ __forceinline__ int home_cell(double g, int n, bool& low_half) {
  if (!(fabs(g) < 1.0e9)) g = 0.0;
  const double fl = floor(g);
  low_half = (g - fl) < 0.5;
  return wrapi((int)fl, n);
}

// File monomer p under every spread tile its union stencil reaches: tiles
// t[axis][0 .. n[axis]).  A slot of the tile while it has room, else the
// overflow list.  Home mode files it under one tile.
__device__ __forceinline__ void tile_place(const TileSlots& ts, int p, int t, int slot, uint32_t* err) {
  if (slot < ts.cap) {
    ts.slots[(long)t * ts.cap + slot] = p;
  } else {
    const int q = atomicAdd(ts.ovf_count, 1);
    if (q < ts.ovf_cap) ts.ovf[q] = make_int2(t, p);
    else atomicOr(err, ERR_BUCKET_OVERFLOW);
  }
}
__device__ __forceinline__ void tile_append(const TileSlots& ts, int p, const int (*t)[3], uint32_t* err) {
  const int nbx = ts.bs.nb[0], nby = ts.bs.nb[1];
  // a slab of a decomposed instance files only under its own tile layers
  auto zin = [&](int tz) { return ts.tz1 == 0 || (tz >= ts.tz0 && tz < ts.tz1); };
  if (t[0][2] < 0 && t[1][2] < 0 && t[2][2] < 0) {
    // at most 2 x 2 x 2 tiles: all counters bumped before any slot is written, so the atomics overlap
    int tt[8], sl[8];
#pragma unroll
    for (int c = 0; c < 8; c++) {
      const int tx = t[0][c & 1], ty = t[1][(c >> 1) & 1], tz = t[2][c >> 2];
      const bool ok = tx >= 0 && ty >= 0 && tz >= 0 && zin(tz);
      tt[c] = ok ? (tz * nby + ty) * nbx + tx : -1;
      sl[c] = ok ? atomicAdd(&ts.count[tt[c]], 1) : 0;
    }
#pragma unroll
    for (int c = 0; c < 8; c++)
      if (tt[c] >= 0) tile_place(ts, p, tt[c], sl[c], err);
    return;
  }
#pragma unroll 1
  for (int c = 0; c < 27; c++) {
    const int tx = t[0][c % 3], ty = t[1][(c / 3) % 3], tz = t[2][c / 9];
    if (tx < 0 || ty < 0 || tz < 0 || !zin(tz)) continue;
    const int q = (tz * nby + ty) * nbx + tx;
    tile_place(ts, p, q, atomicAdd(&ts.count[q], 1), err);
  }
}

// ================================================================ interpolation and monomer update
// A block takes mb consecutive monomers (runs of a chain, whose stencils
// overlap) in three phases:
//   A  thread (monomer, axis): grid coordinate, stencil bases and weights of the
//      axis, unshifted and shifted, into the monomer's record in shared memory,
//      and the tiles it is filed under;
//   B  16 lanes per monomer component, lane (i, j) with the four z points of
//      stencil column (i, j): a row's four points are one access, so a component
//      costs its 16 rows of L1 lookups and four loads a lane, all independent;
//      the 16 partial sums are added by shuffles in a fixed order;
//   C  thread (monomer, component): drag, noise and the explicit update of
//      lagrangian_update() (cuda/SELM_Kernel.cu:302-373); the records go to
//      memory as 16-byte vectors.
// A thread per component that gathered its own 16 rows took two 16-byte loads
// a row on 32 distinct lines each (8.4 M L1 lookups at 1e5 monomers against
// 4.8 M), recomputed the axes' weights and tiles in every component (2300
// instructions a thread), and for few monomers was one long chain of dependent
// latencies and instruction misses on few SMs (19 us for 20 monomers, 11 now).
// At 128^3 with 1e5 monomers 54 -> 46 us FP32 and 85 -> 59 FP64, bound by L1
// lookups and the latency of the gathers.
constexpr int kMonThreads = 192, kMonMax = kMonThreads / 3, kMonGroups = kMonThreads / 16;
// Monomers per block: four blocks on each of the 148 SMs while there are
// enough, 64 at most (a thread per component in phases A and C) and 4 at least
// (a group of lanes per component in phase B).
static int monomers_per_block(int M) { return std::max(4, std::min(kMonMax, (M + 591) / 592)); }

template <typename T> struct alignas(4 * sizeof(T) < 16 ? 4 * sizeof(T) : 16) Vec4 { T v[4]; };

// a record in shared memory: 16 bytes more than in memory, so that the threads
// of ten monomers, which write the same field, spread over the banks
template <typename T> struct MonRec : WRec<T> {
  uint4 pad;
};
template <typename T> struct MonBlock {
  MonRec<T> rec[kMonMax];
  T val[3 * kMonMax];
  int tiles[kMonMax][3][3];  // per axis: the tiles of the union stencil, -1: none (home mode: [axis][0] the home tile)
  int home[kMonMax][3];      // home mode: per axis 2 (cell in tile) + (frac < 1/2)
};

// tiles of one axis that the cells c0 .. c0 + 4 (wrapped) reach: up to three
// distinct ones (a partial last tile can add a third)
template <int TILE> __device__ __forceinline__ void axis_tile_set(double g, int n, int (&t)[3]) {
  if (!isfinite(g)) g = 0.0;
  const int c0 = wrapi((int)floor(g - 0.5) - 1, n);
  t[0] = c0 / TILE;
  t[1] = t[2] = -1;
#pragma unroll
  for (int i = 1; i < 5; i++) {
    int c = c0 + i;
    if (c >= n) c -= n;
    const int q = c / TILE;
    if (q != t[0] && q != t[1] && q != t[2]) {
      if (t[1] < 0) t[1] = q;
      else t[2] = q;
    }
  }
}

// phase A: the records of monomers p0 .. p0 + mc - 1 (and their tiles)
template <typename T>
__device__ __forceinline__ void stage_axis(MonBlock<T>& S, const double* __restrict__ x, int p0, int mc,
                                           const CouplingArgs& a, const TileSlots& ts) {
  const int q = threadIdx.x;
  if (q >= 3 * mc) return;
  const int m = q / 3, ax = q - 3 * m;
  const int n = ax == 0 ? a.nx : ax == 1 ? a.ny : a.nz;
  const double g = (x[3L * p0 + q] - a.lo) / a.dx;
  WRec<T>& R = S.rec[m];
#pragma unroll 1
  for (int sh = 0; sh < 2; sh++) {
    const double r = sh ? g - 0.5 : g;
    const int base = (int)floor(r) - 1;
    Vec4<T> w;
#pragma unroll
    for (int i = 0; i < 4; i++) w.v[i] = ref_weight<T>(fabs(r - (double)(base + i)));
    *reinterpret_cast<Vec4<T>*>(R.w[ax][sh]) = w;
    R.b[ax][sh] = wrapi(base, n);
  }
  if (!ts.count) return;
  if (ts.home) {
    bool low;
    const int c = home_cell(g, n, low);
    const int t = ax == 1 ? c / kTY : c / kTX;  // (kTZ = kTX)
    S.tiles[m][ax][0] = t;
    S.home[m][ax] = 2 * (c - t * (ax == 1 ? kTY : kTX)) + (low ? 1 : 0);
  } else {
    int t[3];
    if (ax == 1) axis_tile_set<kTY>(g, n, t);
    else axis_tile_set<kTX>(g, n, t);
#pragma unroll
    for (int i = 0; i < 3; i++) S.tiles[m][ax][i] = t[i];
  }
}

// The home tile of monomer m of the block
template <typename T> __device__ __forceinline__ int staged_home_tile(const MonBlock<T>& S, int m, const BinSpec& bs) {
  return (S.tiles[m][2][0] * bs.nb[1] + S.tiles[m][1][0]) * bs.nb[0] + S.tiles[m][0][0];
}

// after phase A, thread (monomer, component): the box slot of the component
// (home mode), and the filing by the thread of component 0
template <typename T>
__device__ __forceinline__ void file_staged(MonBlock<T>& S, int p0, int mc, const TileSlots& ts, uint32_t* err) {
  const int q = threadIdx.x;
  if (!ts.count || q >= 3 * mc) return;
  const int m = q / 3, d = q - 3 * m;
  if (ts.home) {
    // With home cell c (tile origin t0) the unshifted base floor(g) - 1 sits at
    // box coordinate c - t0 + 1, the shifted base floor(g - 1/2) - 1 at c - t0
    // or c - t0 + 1: always in [0, tile], and the 4 stencil points stay inside
    // the box of the tile plus 2 cells on each side (x fastest).
    int c[3];
#pragma unroll
    for (int ax = 0; ax < 3; ax++) {
      const int l = S.home[m][ax] >> 1, low = S.home[m][ax] & 1;
      c[ax] = (ax != d && low) ? l : l + 1;
    }
    S.rec[m].hs[d] = (unsigned short)((c[2] * (kTY + 4) + c[1]) * (kTX + 4) + c[0]);
    if (d == 0) {
      const int t = staged_home_tile(S, m, ts.bs);
      tile_place(ts, p0 + m, t, atomicAdd(&ts.count[t], 1), err);
    }
  } else if (d == 0) {
    tile_append(ts, p0 + m, S.tiles[m], err);
  }
}

// phase B: S.val[3 m + d] = Gamma_d u at monomer m.  SLAB: u holds only the
// planes [z0, z0 + nzl) of the grid (a decomposed instance's slab); points on
// other planes are left out (the slabs' sums add up to the whole gather).
template <typename T, bool SLAB>
__device__ __forceinline__ void gather_staged(MonBlock<T>& S, int mc, const T* __restrict__ u, const CouplingArgs& a,
                                              int z0, int nzl) {
  const int lane = threadIdx.x & 15, i = lane & 3, j = lane >> 2;
  const unsigned half = 0xffffu << (threadIdx.x & 16);
  const long cstride = (long)a.nx * a.ny * (SLAB ? nzl : a.nz);
  const int plane = a.nx * a.ny;
  constexpr int U = 4;  // components in flight per group of lanes
  for (int q0 = threadIdx.x >> 4; q0 < 3 * mc; q0 += U * kMonGroups) {
    T v[U][4], sum[U];
#pragma unroll
    for (int s = 0; s < U; s++) {
      const int q = q0 + s * kMonGroups;
#pragma unroll
      for (int k = 0; k < 4; k++) v[s][k] = T(0);
      if (q < 3 * mc) {
        const int m = q / 3, d = q - 3 * m;
        const WRec<T>& R = S.rec[m];
        int xi = R.b[0][d != 0] + i, yj = R.b[1][d != 1] + j, zk = R.b[2][d != 2];
        if (xi >= a.nx) xi -= a.nx;
        if (yj >= a.ny) yj -= a.ny;
        const T* col = u + d * cstride + yj * a.nx + xi;
#pragma unroll
        for (int k = 0; k < 4; k++) {
          const int zr = SLAB ? zk - z0 : zk;
          if (!SLAB || (unsigned)zr < (unsigned)nzl) v[s][k] = __ldg(col + (long)zr * plane);
          if (++zk == a.nz) zk = 0;
        }
      }
    }
#pragma unroll
    for (int s = 0; s < U; s++) {
      const int q = min(q0 + s * kMonGroups, 3 * mc - 1);
      const int m = q / 3, d = q - 3 * m;
      const WRec<T>& R = S.rec[m];
      const Vec4<T> wz = *reinterpret_cast<const Vec4<T>*>(R.w[2][d != 2]);
      T t = v[s][0] * wz.v[0];
#pragma unroll
      for (int k = 1; k < 4; k++) t += v[s][k] * wz.v[k];
      sum[s] = t * (R.w[0][d != 0][i] * R.w[1][d != 1][j]);
    }
    // the sums over the 16 lanes, four at once: after two exchanges a lane
    // holds a quarter of component (lane >> 2)'s sum, two more add the quarters
    const bool up8 = lane & 8, up4 = lane & 4;
    T a0 = up8 ? sum[2] : sum[0], a1 = up8 ? sum[3] : sum[1];
    a0 += __shfl_xor_sync(half, up8 ? sum[0] : sum[2], 8);
    a1 += __shfl_xor_sync(half, up8 ? sum[1] : sum[3], 8);
    T t = up4 ? a1 : a0;
    t += __shfl_xor_sync(half, up4 ? a0 : a1, 4);
    t += __shfl_xor_sync(half, t, 2);
    t += __shfl_xor_sync(half, t, 1);
    const int q = q0 + (lane >> 2) * kMonGroups;
    if ((lane & 3) == 0 && q < 3 * mc) S.val[q] = t;
  }
}

// the block's records to memory
template <typename T>
__device__ __forceinline__ void store_records(const MonBlock<T>& S, int p0, int mc, WRec<T>* __restrict__ rec) {
  constexpr int V = sizeof(WRec<T>) / 16, VS = sizeof(MonRec<T>) / 16;
  const uint4* s = reinterpret_cast<const uint4*>(S.rec);
  uint4* d = reinterpret_cast<uint4*>(rec + p0);
  for (int i = threadIdx.x; i < V * mc; i += kMonThreads) d[i] = s[(i / V) * VS + i % V];
}

// Home mode: the scale data of the home tile's fixed-point box, from the
// thread of one component: its impulse |tf| and its weight factors.
template <typename T>
__device__ __forceinline__ void home_scale_note(const TileSlots& ts, const MonBlock<T>& S, int m, int d, double tf) {
  const int t = staged_home_tile(S, m, ts.bs);
  atomicMax(&ts.tmax[t], (unsigned long long)__double_as_longlong(fabs(tf)));
  bool big = false;
#pragma unroll
  for (int ax = 0; ax < 3; ax++)
#pragma unroll
    for (int i = 0; i < 4; i++) big |= (S.rec[m].w[ax][ax != d][i] > T(0.5));
  if (big) atomicOr(&ts.quirk[t], 1);
}

// GATHERED: u is the interpolated velocity itself, [3M] by monomer component
// (a decomposed instance sums it over its slabs), and only the update and the
// filing run.
template <typename T, bool GATHERED = false>
__global__ void __launch_bounds__(kMonThreads, sizeof(T) == 4 ? 6 : 5)
    k_interp_update(const T* __restrict__ u, const double* __restrict__ x_old, double* __restrict__ x_new,
                    double* __restrict__ v, double* __restrict__ f, const double* __restrict__ m,
                    double* __restrict__ tf_out, WRec<T>* __restrict__ rec, CouplingArgs a,
                    uint32_t* __restrict__ err, TileSlots ts, int mb) {
  __shared__ __align__(16) MonBlock<T> S;
  const int p0 = blockIdx.x * mb, mc = min(mb, a.M - p0), q = threadIdx.x;
  stage_axis<T>(S, x_old, p0, mc, a, ts);
  __syncthreads();
  const bool mine = q < 3 * mc;
  const long g = 3L * p0 + q;
  const int mq = q / 3, d = q - 3 * mq;
  double kick = 0.0, vg = 0.0, fg = 0.0, xg = 0.0;
  if (mine) {
    vg = v[g];
    fg = f[g];
    xg = x_old[g];
    if (a.stochastic) {
      double z1;
      const uint64_t step = a.step_ptr ? *a.step_ptr : a.step;
      philox_normal2(a.seed, (uint32_t)(p0 + mq), 4u + (uint32_t)d, step, kick, z1);
      kick *= a.coef;
    }
  }
  file_staged<T>(S, p0, mc, ts, err);  // the spread of this step reads x_old
  if (!GATHERED) gather_staged<T, false>(S, mc, u, a, 0, 0);
  __syncthreads();
  store_records<T>(S, p0, mc, rec);
  if (!mine) return;
  const T val = GATHERED ? u[g] : S.val[q];
  double t_f = -a.upsilon * (vg - (double)val) * a.dt;
  if (a.stochastic) t_f += kick;
  tf_out[g] = t_f;
  if (ts.home) home_scale_note<T>(ts, S, mq, d, t_f);
  t_f += a.dt * fg;
  f[g] = t_f / a.dt;
  const double tmp = vg * a.dt;
  const double L = a.hi - a.lo;
  if (fabs(tmp) > L / 2) atomicOr(err, ERR_DISPLACEMENT);
  double tx = xg + tmp;
  if (tx > a.hi) tx -= L;
  else if (tx < a.lo) tx += L;
  x_new[g] = tx;
  const double vn = vg + t_f / m[p0 + mq];
  v[g] = vn;
  if (!isfinite(vn) || !isfinite(tx)) atomicOr(err, ERR_NONFINITE);
}

// ---- quasi-steady (overdamped) form, no reference counterpart
// Before the fluid solve: the stencil records at x^n for binning, spreading and
// the move, and the impulse array the spread subtracts, tf = -F / dV, so that
// the grid receives the force density +F / dV of the conservative forces.
template <typename T>
__global__ void __launch_bounds__(kMonThreads) k_qs_prepare(const double* __restrict__ x, const double* __restrict__ f,
                                                            double* __restrict__ tf_out, WRec<T>* __restrict__ rec,
                                                            CouplingArgs a, double inv_dv, TileSlots ts,
                                                            uint32_t* __restrict__ err, int mb) {
  __shared__ __align__(16) MonBlock<T> S;
  const int p0 = blockIdx.x * mb, mc = min(mb, a.M - p0), q = threadIdx.x;
  stage_axis<T>(S, x, p0, mc, a, ts);
  __syncthreads();
  file_staged<T>(S, p0, mc, ts, err);
  if (q < 3 * mc) {
    const long g = 3L * p0 + q;
    const double t = -f[g] * inv_dv;
    tf_out[g] = t;
    if (ts.home) home_scale_note<T>(ts, S, q / 3, q % 3, t);
  }
  __syncthreads();
  store_records<T>(S, p0, mc, rec);
}

// After the fluid solve: v = Gamma u (x^n) with the records of x^n, x^{n+1} =
// x^n + dt v with the inertial form's single periodic wrap; f keeps the
// conservative force.
template <typename T>
__global__ void __launch_bounds__(kMonThreads, sizeof(T) == 4 ? 8 : 6)
    k_qs_move(const T* __restrict__ u, const double* __restrict__ x_old, double* __restrict__ x_new,
              double* __restrict__ v, const WRec<T>* __restrict__ rec, CouplingArgs a, uint32_t* __restrict__ err,
              int mb) {
  __shared__ __align__(16) MonBlock<T> S;
  const int p0 = blockIdx.x * mb, mc = min(mb, a.M - p0), q = threadIdx.x;
  {
    constexpr int V = sizeof(WRec<T>) / 16, VS = sizeof(MonRec<T>) / 16;
    uint4* s = reinterpret_cast<uint4*>(S.rec);
    const uint4* src = reinterpret_cast<const uint4*>(rec + p0);
    for (int i = q; i < V * mc; i += kMonThreads) s[(i / V) * VS + i % V] = src[i];
  }
  __syncthreads();
  gather_staged<T, false>(S, mc, u, a, 0, 0);
  __syncthreads();
  if (q >= 3 * mc) return;
  const long g = 3L * p0 + q;
  const double vel = (double)S.val[q];
  const double tmp = vel * a.dt;
  const double L = a.hi - a.lo;
  if (fabs(tmp) > L / 2) atomicOr(err, ERR_DISPLACEMENT);
  double tx = x_old[g] + tmp;
  if (tx > a.hi) tx -= L;
  else if (tx < a.lo) tx += L;
  x_new[g] = tx;
  v[g] = vel;
  if (!isfinite(vel) || !isfinite(tx)) atomicOr(err, ERR_NONFINITE);
}

template <typename T>
cudaError_t qs_prepare(const double* x, const double* f, double* tf, WRec<T>* rec, const CouplingArgs& a,
                       double inv_dv, cudaStream_t st, const TileSlots* ts, uint32_t* err) {
  if (a.M <= 0) return cudaSuccess;
  const int mb = monomers_per_block(a.M);
  k_qs_prepare<T><<<(unsigned)((a.M + mb - 1) / mb), kMonThreads, 0, st>>>(x, f, tf, rec, a, inv_dv,
                                                                           ts ? *ts : TileSlots{}, err, mb);
  count_launches(1);
  return cudaGetLastError();
}

template <typename T>
cudaError_t qs_move(const T* u, const double* x_old, double* x_new, double* v, const WRec<T>* rec, const CouplingArgs& a,
                    uint32_t* err, cudaStream_t st) {
  if (a.M <= 0) return cudaSuccess;
  const int mb = monomers_per_block(a.M);
  k_qs_move<T><<<(unsigned)((a.M + mb - 1) / mb), kMonThreads, 0, st>>>(u, x_old, x_new, v, rec, a, err, mb);
  count_launches(1);
  return cudaGetLastError();
}
template cudaError_t qs_prepare<double>(const double*, const double*, double*, WRec<double>*, const CouplingArgs&,
                                        double, cudaStream_t, const TileSlots*, uint32_t*);
template cudaError_t qs_prepare<float>(const double*, const double*, double*, WRec<float>*, const CouplingArgs&,
                                       double, cudaStream_t, const TileSlots*, uint32_t*);
template cudaError_t qs_move<double>(const double*, const double*, double*, double*, const WRec<double>*,
                                     const CouplingArgs&, uint32_t*, cudaStream_t);
template cudaError_t qs_move<float>(const float*, const double*, double*, double*, const WRec<float>*,
                                    const CouplingArgs&, uint32_t*, cudaStream_t);

// Pure interpolation (operator entry point): out[p][d] = Gamma_d u (x_p)
template <typename T>
__global__ void k_interp_only(const T* __restrict__ u, const double* __restrict__ x, int M, int nx, int ny, int nz,
                              double lo, double dx, double* __restrict__ out) {
  const long gid = (long)blockIdx.x * blockDim.x + threadIdx.x;
  if (gid >= 3L * M) return;
  const int p = (int)(gid / 3), d = (int)(gid % 3);
  const long N = (long)nx * ny * nz;
  const double gx = (x[3L * p] - lo) / dx, gy = (x[3L * p + 1] - lo) / dx, gz = (x[3L * p + 2] - lo) / dx;
  T val;
  if (d == 0) val = interp_one<T>(gx, gy - 0.5, gz - 0.5, nx, ny, nz, u);
  else if (d == 1) val = interp_one<T>(gx - 0.5, gy, gz - 0.5, nx, ny, nz, u + N);
  else val = interp_one<T>(gx - 0.5, gy - 0.5, gz, nx, ny, nz, u + 2 * N);
  out[gid] = (double)val;
}

template <typename T>
cudaError_t interp_only(const T* u, const double* x, int M, int nx, int ny, int nz, double lo, double dx, double* out,
                        cudaStream_t st) {
  if (M <= 0) return cudaSuccess;
  k_interp_only<T><<<(unsigned)((3L * M + 255) / 256), 256, 0, st>>>(u, x, M, nx, ny, nz, lo, dx, out);
  count_launches(1);
  return cudaGetLastError();
}
template cudaError_t interp_only<double>(const double*, const double*, int, int, int, int, double, double, double*,
                                         cudaStream_t);
template cudaError_t interp_only<float>(const float*, const double*, int, int, int, int, double, double, double*,
                                        cudaStream_t);

template <typename T>
cudaError_t interp_update(const T* u, const double* x_old, double* x_new, double* v, double* f, const double* m,
                          double* tf, WRec<T>* rec, const CouplingArgs& a, uint32_t* err, cudaStream_t st,
                          const TileSlots* ts) {
  if (a.M <= 0) return cudaSuccess;
  const int mb = monomers_per_block(a.M);
  k_interp_update<T><<<(unsigned)((a.M + mb - 1) / mb), kMonThreads, 0, st>>>(u, x_old, x_new, v, f, m, tf, rec, a, err,
                                                                              ts ? *ts : TileSlots{}, mb);
  count_launches(1);
  return cudaGetLastError();
}

// a decomposed instance's slab: the part of every monomer component's
// interpolation that comes from the slab's planes [z0, z0 + nzl) (u: the
// slab's velocity [3][nzl][ny][nx]), into out [3M]
template <typename T>
__global__ void __launch_bounds__(kMonThreads) k_interp_partial(const T* __restrict__ u, const double* __restrict__ x,
                                                                CouplingArgs a, int z0, int nzl, T* __restrict__ out,
                                                                int mb) {
  __shared__ __align__(16) MonBlock<T> S;
  const int p0 = blockIdx.x * mb, mc = min(mb, a.M - p0);
  stage_axis<T>(S, x, p0, mc, a, TileSlots{});
  __syncthreads();
  gather_staged<T, true>(S, mc, u, a, z0, nzl);
  __syncthreads();
  if (threadIdx.x < 3 * mc) out[3L * p0 + threadIdx.x] = S.val[threadIdx.x];
}

template <typename T>
cudaError_t interp_partial(const T* u_slab, const double* x, const CouplingArgs& a, int z0, int nzl, T* out,
                           cudaStream_t st) {
  if (a.M <= 0) return cudaSuccess;
  const int mb = monomers_per_block(a.M);
  k_interp_partial<T><<<(unsigned)((a.M + mb - 1) / mb), kMonThreads, 0, st>>>(u_slab, x, a, z0, nzl, out, mb);
  count_launches(1);
  return cudaGetLastError();
}
template cudaError_t interp_partial<float>(const float*, const double*, const CouplingArgs&, int, int, float*,
                                           cudaStream_t);
template cudaError_t interp_partial<double>(const double*, const double*, const CouplingArgs&, int, int, double*,
                                            cudaStream_t);

// the update of a decomposed instance from the summed interpolation `gathered` [3M]
template <typename T>
cudaError_t interp_update_gathered(const T* gathered, const double* x_old, double* x_new, double* v, double* f,
                                   const double* m, double* tf, WRec<T>* rec, const CouplingArgs& a, uint32_t* err,
                                   cudaStream_t st, const TileSlots& ts) {
  if (a.M <= 0) return cudaSuccess;
  const int mb = monomers_per_block(a.M);
  k_interp_update<T, true><<<(unsigned)((a.M + mb - 1) / mb), kMonThreads, 0, st>>>(gathered, x_old, x_new, v, f, m, tf,
                                                                                    rec, a, err, ts, mb);
  count_launches(1);
  return cudaGetLastError();
}
template cudaError_t interp_update_gathered<float>(const float*, const double*, double*, double*, double*,
                                                   const double*, double*, WRec<float>*, const CouplingArgs&,
                                                   uint32_t*, cudaStream_t, const TileSlots&);
template cudaError_t interp_update_gathered<double>(const double*, const double*, double*, double*, double*,
                                                    const double*, double*, WRec<double>*, const CouplingArgs&,
                                                    uint32_t*, cudaStream_t, const TileSlots&);

// ================================================================ spread (gather)
// Tiles of kTX x kTY x kTZ cells.  bin_particles (mode 2) files every monomer
// under each tile its union stencil reaches (5 cells per axis,
// floor(g - 1/2) - 1 .. floor(g) + 2), so a tile's bucket is exactly its list
// of candidates, in no particular order.  A block per tile accumulates the
// tile in shared memory; a thread takes one z-plane kz of one candidate's
// component d (12 per candidate), reads the candidate's stencil record, and
// adds the plane's in-tile points -tf_d wz[kz] wy[jy] wx[ix].
//
// Accumulation is in fixed point with shared-memory integer atomics, so the
// result does not depend on candidate order or thread scheduling (integer
// addition is exact and associative; no sort, no floating-point atomics).
// Each contribution carries the impulse pre-scaled by 2^S, chosen per tile
// from its largest impulse m and its candidate count n, and is rounded to an
// integer v:
//   split3 (FP64 grids, n <= 2048): three 32-bit accumulators per cell,
//          v = hi 2^42 + mid 2^21 + lo with 0 <= lo, mid < 2^21, |v| < 2^(61-k):
//          the step of the wide form, with native 32-bit atomics (64-bit
//          shared-memory atomics measured 2.6x slower for the whole spread);
//   wide   (FP64 grids beyond 2048 candidates, or FP32 beyond 2^16): one
//          64-bit accumulator per cell, n m 2^S < 2^61, a step of about n m 2^-61;
//   split  (FP32 grids): two 32-bit accumulators per cell, v = hi 2^L + lo
//          with 0 <= lo < 2^L, L = 32 - k and k = ceil(log2 n), so that
//          neither the sum of the lo parts nor that of the hi parts can
//          overflow for |v| < 2^(62 - 2k); a step of m 2^-(62-2k), 2^-44 of
//          the tile's largest impulse for n <= 512.  Shared-memory 32-bit
//          integer atomics are native; 64-bit ones are not.
constexpr int kSpreadThreads = 3 * kTY * kTZ;  // also the number of tile rows (component, y, z)
constexpr int kSpreadCells = 3 * kTZ * kTY * kTX;
constexpr int kSpreadPad = 32;  // per-lane dummy slots: points outside the tile add there (never read)
constexpr int kAccWords = kSpreadCells + kSpreadPad;
// accumulator words per cell: two 32-bit words (FP32 grids) or three (FP64)
template <typename T> constexpr size_t spread_smem() { return sizeof(unsigned) * (sizeof(T) == 4 ? 2 : 3) * kAccWords; }
constexpr int kMaxSpreadDevices = 64;
static_assert(kTX == 16, "spread_rot assumes 16-cell rows");

// Accumulator slot of cell (cx, cy, cz) of component d.  The x position is
// rotated by 4 cz + 3 d within its 16-cell row, so that the twelve
// (component, z-plane) lanes of one candidate, which add at the same time,
// fall on twelve distinct banks whatever the half-cell shifts between the
// three staggered frames (x and y bases differing by 0 or 1; a rotation of
// 4 cz + d collides for a quarter of the shift patterns).
__device__ __forceinline__ int spread_row(int d, int cy, int cz) { return ((d * kTZ + cz) * kTY + cy) * kTX; }
__device__ __forceinline__ int spread_rot(int cx, int cz, int d) { return (cx + 4 * cz + 3 * d) & (kTX - 1); }

__device__ __forceinline__ long long to_fixed(float v) { return __float2ll_rn(v); }
__device__ __forceinline__ long long to_fixed(double v) { return __double2ll_rn(v); }

__device__ __forceinline__ int round_small(float v) {  // rint(v) for |v| < 2^22
  return __float_as_int(v + 12582912.0f) - 0x4B400000;
}

// Tile geometry and fixed-point state shared by the plane additions of a block.
struct SpreadTile {
  int t0x, t0y, t0z, ex, ey, ez;
  double scale;
  int mode;  // kSplit20, kSplitK or kWide
  int k, L;
};
// Fixed-point modes (v = rounded contribution, n candidates, k = ceil(log2 n)):
//   kSplit20 (FP32, n <= 4096): lo = v mod 2^20, hi = v >> 20, |v| < 2^(50-k);
//   kSplitK  (FP32, n <= 65536): lo = v mod 2^(32-k), hi = v >> (32-k), |v| < 2^(62-2k);
//   kSplit3  (FP64, n <= 2048): lo = v mod 2^21, mid = (v >> 21) mod 2^21, hi = v >> 42,
//            |v| < 2^(61-k), so that n 2^21 <= 2^32 and n |hi| <= 2^19;
//   kWide    (more candidates): one 64-bit word, n |v| < 2^61.
// In the split modes neither the lo sums (< n 2^L <= 2^32) nor the hi sums
// (< 2^30 in magnitude) can overflow their 32-bit words.
enum { kSplit20 = 0, kSplitK = 1, kWide = 2, kSplit3 = 3 };

// Add the 16 points of z-plane kz of candidate p's component d (points
// outside the tile go to the lane's dummy slot, so every lane does the same work).
template <int MODE, typename T>
__device__ __forceinline__ void spread_plane(int p, int d, int kz, const SpreadTile& tl, unsigned long long* acc,
                                             const double* __restrict__ x_old, const double* __restrict__ tf,
                                             const WRec<T>* __restrict__ rec, const CouplingArgs& a) {
  unsigned* acc_lo = reinterpret_cast<unsigned*>(acc);
  unsigned* acc_hi = acc_lo + kAccWords;
  unsigned* acc_top = acc_lo + 2 * kAccWords;
  const int nx = a.nx, ny = a.ny, nz = a.nz;
  const int sx = (d != 0), sy = (d != 1), sz = (d != 2);
  int bx, by, bz;
  Vec4<T> wx, wy;
  T wzk;
  if (rec) {
    const WRec<T>& R = rec[p];
    bx = R.b[0][sx];
    by = R.b[1][sy];
    bz = R.b[2][sz];
    wx = *reinterpret_cast<const Vec4<T>*>(R.w[0][sx]);
    wy = *reinterpret_cast<const Vec4<T>*>(R.w[1][sy]);
    wzk = R.w[2][sz][kz];
  } else {
    const double gx = (x_old[3L * p] - a.lo) / a.dx - (sx ? 0.5 : 0.0);
    const double gy = (x_old[3L * p + 1] - a.lo) / a.dx - (sy ? 0.5 : 0.0);
    const double gz = (x_old[3L * p + 2] - a.lo) / a.dx - (sz ? 0.5 : 0.0);
    const int fx = (int)floor(gx) - 1, fy = (int)floor(gy) - 1, fz = (int)floor(gz) - 1;
    bx = wrapi(fx, nx);
    by = wrapi(fy, ny);
    bz = wrapi(fz, nz);
#pragma unroll
    for (int i = 0; i < 4; i++) {
      wx.v[i] = ref_weight<T>(fabs(gx - (double)(fx + i)));
      wy.v[i] = ref_weight<T>(fabs(gy - (double)(fy + i)));
    }
    wzk = ref_weight<T>(fabs(gz - (double)(fz + kz)));
  }
  // tile-relative plane and rows
  int cz = bz + kz - tl.t0z;
  if (cz < 0) cz += nz;
  if (cz >= nz) cz -= nz;
  if (cz >= tl.ez) return;
  int cx0 = bx - tl.t0x;
  if (cx0 < 0) cx0 += nx;
  int cy0 = by - tl.t0y;
  if (cy0 < 0) cy0 += ny;
  const T fz = (T)(-tf[3L * p + d] * tl.scale) * wzk;
  const int dummy = kSpreadCells + (threadIdx.x & (kSpreadPad - 1));
  // x-points of the plane: slot within a row, or -1 outside the tile
  int xo[4];
#pragma unroll
  for (int ix = 0; ix < 4; ix++) {
    int cx = cx0 + ix;
    if (cx >= nx) cx -= nx;
    xo[ix] = (cx < tl.ex) ? spread_rot(cx, cz, d) : -1;
  }
  const int plane = spread_row(d, 0, cz);
#pragma unroll
  for (int jy = 0; jy < 4; jy++) {
    int cy = cy0 + jy;
    if (cy >= ny) cy -= ny;
    const bool yin = cy < tl.ey;
    const T rowf = fz * wy.v[jy];
    const int row = plane + cy * kTX;
#pragma unroll
    for (int ix = 0; ix < 4; ix++) {
      const int slot = (yin && xo[ix] >= 0) ? row + xo[ix] : dummy;
      const long long v = to_fixed(rowf * wx.v[ix]);
      if (MODE == kSplit20) {
        atomicAdd(acc_lo + slot, (unsigned)v & 0xfffffu);
        atomicAdd(acc_hi + slot, (unsigned)(v >> 20));
      } else if (MODE == kSplitK) {
        atomicAdd(acc_lo + slot, (unsigned)v & (0xffffffffu >> tl.k));
        atomicAdd(acc_hi + slot, (unsigned)(v >> tl.L));
      } else if (MODE == kSplit3) {
        atomicAdd(acc_lo + slot, (unsigned)v & 0x1fffffu);
        atomicAdd(acc_hi + slot, (unsigned)(v >> 21) & 0x1fffffu);
        atomicAdd(acc_top + slot, (unsigned)(v >> 42));
      } else {
        atomicAdd(acc + slot, (unsigned long long)v);
      }
    }
  }
}

template <int MODE, typename T>
__device__ __forceinline__ void spread_candidates(const int* __restrict__ ids, int n_prim, int n_ovf, const TileSlots& ts,
                                                  int tb, const SpreadTile& tl, unsigned long long* acc,
                                                  const double* __restrict__ x_old, const double* __restrict__ tf,
                                                  const WRec<T>* __restrict__ rec, const CouplingArgs& a) {
  for (int u = threadIdx.x; u < 12 * n_prim; u += kSpreadThreads) {
    const int c = u / 12, r = u - 12 * c;
    spread_plane<MODE, T>(ids[c], r >> 2, r & 3, tl, acc, x_old, tf, rec, a);
  }
  // beyond the tile's capacity (rare): a thread takes all planes of an entry
  for (int q = threadIdx.x; q < n_ovf; q += kSpreadThreads) {
    const int2 e = ts.ovf[q];
    if (e.x == tb)
      for (int r = 0; r < 12; r++) spread_plane<MODE, T>(e.y, r >> 2, r & 3, tl, acc, x_old, tf, rec, a);
  }
}

// one block of a spread has read its candidates: the last one clears the overflow
// counter (no block reads it any more; the next kernel files new entries)
__device__ __forceinline__ void spread_tile_done(const TileSlots& ts) {
  if (atomicAdd(ts.done, 1u) == gridDim.x - 1) {
    *ts.ovf_count = 0;
    *ts.done = 0u;
  }
}

// With few monomers a block is a chain of loads (count, candidates, impulses,
// records): the candidates are read beside the count, the records beside the
// impulses, and the block is counted as done before its cells go out (64^3
// step, 1000 monomers, 44.1 -> 43.4 us FP32 and 64.3 -> 63.5 plain; 30^3 spread
// alone 14.4 -> 12.8).
// Candidates of tile tb: the CSR bucket offsets[tb] .. offsets[tb+1] of
// `entries` (counting-sort binning), or, when ts.count is set, the tile's
// slots plus its entries in the overflow list (slots filled during the
// interpolation).
template <typename T>
__global__ void __launch_bounds__(kSpreadThreads, sizeof(T) == 4 ? 3 : 2) k_spread_tiles(T* __restrict__ fgrid, int accumulate,
                                                                 const double* __restrict__ x_old,
                                                                 const double* __restrict__ tf, BinSpec bs,
                                                                 const int* __restrict__ offsets,
                                                                 const int* __restrict__ entries, TileSlots ts,
                                                                 const WRec<T>* __restrict__ rec, CouplingArgs a) {
  extern __shared__ __align__(16) unsigned long long acc[];  // u64[kAccWords] (wide), or u32 lo[kAccWords], hi[kAccWords] (, top[kAccWords])
  __shared__ double wmax[kSpreadThreads / 32];
  __shared__ int wbad[kSpreadThreads / 32];
  const unsigned* acc_lo = reinterpret_cast<const unsigned*>(acc);
  const unsigned* acc_hi = acc_lo + kAccWords;
  const unsigned* acc_top = acc_lo + 2 * kAccWords;
  const int nx = a.nx, ny = a.ny, nz = a.nz;
  const int tb = blockIdx.x + ts.tile0;
  const int tbx = tb % bs.nb[0], tby = (tb / bs.nb[0]) % bs.nb[1], tbz = tb / (bs.nb[0] * bs.nb[1]);
  SpreadTile tl;
  tl.t0x = tbx * kTX;
  tl.t0y = tby * kTY;
  tl.t0z = tbz * kTZ;
  tl.ex = min(kTX, nx - tl.t0x);
  tl.ey = min(kTY, ny - tl.t0y);
  tl.ez = min(kTZ, nz - tl.t0z);
  const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
  const long N = (long)nx * ny * nz;
  const bool slots = ts.count != nullptr;
  int n, n_prim;
  const int* ids;
  int first = 0;  // ids[tid], read beside the count
  if (slots) {
    ids = ts.slots + (long)tb * ts.cap;
    if (tid < ts.cap) first = ids[tid];
    n = ts.count[tb];
    n_prim = min(n, ts.cap);
  } else {
    const int s0 = offsets[tb];
    n = n_prim = offsets[tb + 1] - s0;
    ids = entries + s0;
  }
  const int n_ovf = (n > n_prim) ? min(*ts.ovf_count, ts.ovf_cap) : 0;  // only a tile beyond its capacity scans it
  if (n > 0) {
    uint4* w = reinterpret_cast<uint4*>(acc);
    static_assert(kAccWords % 4 == 0, "16-byte clears");
    for (int i = tid; i < (sizeof(T) == 4 ? 2 : 3) * kAccWords / 4; i += kSpreadThreads) w[i] = make_uint4(0u, 0u, 0u, 0u);
  }
  if (n == 0) {
    if (slots && tid == 0) spread_tile_done(ts);
    // no monomer reaches the tile: zeros, or the grid as it is
    if (!accumulate) {
      const long cs = ts.cstride ? ts.cstride : N;
      for (int idx = tid; idx < kSpreadCells; idx += kSpreadThreads) {
        const int row = idx / kTX, cx = idx % kTX, cy = row % kTY, cz = (row / kTY) % kTZ, d = row / (kTY * kTZ);
        if (cx < tl.ex && cy < tl.ey && cz < tl.ez)
          fgrid[d * cs + ((long)(tl.t0z + cz - ts.z0) * ny + (tl.t0y + cy)) * nx + tl.t0x + cx] = T(0);
      }
    }
    return;
  }
  // fixed-point scale of this tile from its largest impulse component
  double m = 0.0;
  int bad = 0;
  auto see = [&](int p) {
#pragma unroll
    for (int c = 0; c < 3; c++) {
      const double v = fabs(tf[3L * p + c]);
      bad |= !(v <= 1.0e300);
      m = fmax(m, v);
    }
  };
  for (int q = tid; q < n_prim; q += kSpreadThreads) {
    const int p = (slots && q == tid) ? first : ids[q];
    if (rec) {
      // the records come in beside the impulses
      const char* r = reinterpret_cast<const char*>(rec + p);
      asm volatile("prefetch.global.L1 [%0];" ::"l"(r));
      asm volatile("prefetch.global.L1 [%0];" ::"l"(r + sizeof(WRec<T>) - 1));
    }
    see(p);
  }
  for (int q = tid; q < n_ovf; q += kSpreadThreads) {
    const int2 e = ts.ovf[q];
    if (e.x == tb) see(e.y);
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) m = fmax(m, __shfl_xor_sync(0xffffffffu, m, o));
  bad = __any_sync(0xffffffffu, bad);
  if (lane == 0) {
    wmax[wid] = m;
    wbad[wid] = bad;
  }
  __syncthreads();
#pragma unroll
  for (int w = 0; w < kSpreadThreads / 32; w++) {
    m = fmax(m, wmax[w]);
    bad |= wbad[w];
  }
  tl.k = (n > 1) ? 32 - __clz(n - 1) : 1;  // ceil(log2 n)
  if (sizeof(T) == 4) tl.mode = (tl.k > 16) ? kWide : (tl.k <= 12) ? kSplit20 : kSplitK;
  else tl.mode = (tl.k <= 11) ? kSplit3 : kWide;
  tl.L = (tl.mode == kSplit20) ? 20 : 32 - tl.k;
  int em = 0;
  if (m > 0.0 && !bad) frexp(tl.mode == kWide ? m * (double)n : m, &em);  // m (or n m) < 2^em
  const int bits = (tl.mode == kSplit20) ? 50 - tl.k
                   : (tl.mode == kSplitK) ? 62 - 2 * tl.k
                   : (tl.mode == kSplit3) ? 61 - tl.k
                                          : 61;
  const int S = max(-1000, min(1000, bits - em));
  tl.scale = ldexp(1.0, S);
  const double inv_scale = ldexp(1.0, -S);
  if (!bad) {
    if (tl.mode == kSplit20) spread_candidates<kSplit20, T>(ids, n_prim, n_ovf, ts, tb, tl, acc, x_old, tf, rec, a);
    else if (tl.mode == kSplitK) spread_candidates<kSplitK, T>(ids, n_prim, n_ovf, ts, tb, tl, acc, x_old, tf, rec, a);
    else if (tl.mode == kSplit3) spread_candidates<kSplit3, T>(ids, n_prim, n_ovf, ts, tb, tl, acc, x_old, tf, rec, a);
    else spread_candidates<kWide, T>(ids, n_prim, n_ovf, ts, tb, tl, acc, x_old, tf, rec, a);
  }
  __syncthreads();
  if (slots && tid == 0) {
    // every thread has read count[tb], its candidates and the overflow list
    ts.count[tb] = 0;
    spread_tile_done(ts);
  }
  // cells out, a half-warp per 16-cell row
  // a non-finite impulse makes the whole tile non-finite, as a floating-point sum would
  const double nan_or_zero = bad ? __longlong_as_double(0x7ff8000000000000LL) : 0.0;
  const long cstride = ts.cstride ? ts.cstride : N;
  auto cell = [&](int idx, int& slot) -> T* {  // the grid's cell of tile cell idx, or null outside the grid
    const int row = idx / kTX, cx = idx % kTX;
    const int cy = row % kTY, cz = (row / kTY) % kTZ, d = row / (kTY * kTZ);
    slot = row * kTX + spread_rot(cx, cz, d);
    if (cx >= tl.ex || cy >= tl.ey || cz >= tl.ez) return nullptr;
    return fgrid + d * cstride + ((long)(tl.t0z + cz - ts.z0) * ny + (tl.t0y + cy)) * nx + tl.t0x + cx;
  };
  auto value = [&](int slot) {
    const long long sum =
        (tl.mode == kSplit3) ? (long long)(int)acc_top[slot] * (1ll << 42) + (long long)acc_hi[slot] * (1ll << 21) +
                                   (long long)acc_lo[slot]
        : (tl.mode != kWide) ? (long long)(int)acc_hi[slot] * (1ll << tl.L) + (long long)acc_lo[slot]
                             : (long long)acc[slot];
    return (double)sum * inv_scale + nan_or_zero;
  };
  if (!accumulate) {
    for (int idx = tid; idx < kSpreadCells; idx += kSpreadThreads) {
      int slot;
      T* dst = cell(idx, slot);
      if (dst) *dst = (T)value(slot);
    }
  } else {
    // four cells of a thread at a time, what the grid holds read before the
    // sums (one after another they took 25 of 114 us at 128^3 FP64)
    constexpr int kPerThread = kSpreadCells / kSpreadThreads, kBatch = 4;
    static_assert(kSpreadCells % kSpreadThreads == 0 && kPerThread % kBatch == 0, "whole batches of cells");
#pragma unroll 1
    for (int q0 = 0; q0 < kPerThread; q0 += kBatch) {
      T* dst[kBatch];
      T old[kBatch];
      int slot[kBatch];
#pragma unroll
      for (int q = 0; q < kBatch; q++) {
        dst[q] = cell(tid + (q0 + q) * kSpreadThreads, slot[q]);
        old[q] = dst[q] ? *dst[q] : T(0);
      }
#pragma unroll
      for (int q = 0; q < kBatch; q++)
        if (dst[q]) *dst[q] = (T)((double)old[q] + value(slot[q]));
    }
  }
}


// ================================================================ FP32 spread by home tiles
// Every monomer is filed once, under the tile of its cell; the block of a
// tile adds its monomers' 3 x 64 stencil points into a shared-memory box of
// the tile plus two cells on each side (20 x 12 x 20 cells per component:
// the union of the staggered stencils of a monomer is 5 cells wide, from 2
// below its cell to 2 above), writes the box to global memory, and
// k_spread_fold sums the boxes that cover each cell in a fixed order.
//
// Accumulation: one warp per monomer and component, lane l adding the points
// (ix, jy, kz) = (l & 3, (l >> 2) & 3, l >> 4) and (ix, jy, kz + 2) of the
// 4^3 stencil.  Rows of the box are 20 words and planes 240 (= 16 mod 32), so
// the 32 lanes of one atomic instruction hit 32 distinct banks wherever the
// stencil sits.  Values are fixed point in one 32-bit word per cell, at a
// per-tile scale 2^S: integer sums do not depend on the order of addition,
// so the box, and the fold's fixed-order float sum of at most 8 boxes, repeat
// bit for bit.
//
// Scale: with n monomers in the tile (k = ceil(log2 n)), the largest impulse
// component m < 2^em and every weight factor <= 2^(ew/3) (ew = -3 when all
// factors are <= 1/2, as the Peskin function is; 0 when the reference's
// distance-2 factor of 1 occurs; m and the flag come from the interpolation,
// TileSlots::tmax and ::quirk), a contribution is < 2^(em + ew + S) and a
// cell's sum < n 2^(em + ew + S).  S = min(30 - k, 22) - em - ew keeps a
// cell's sum below 2^30 (plus n/2 of rounding) and a contribution below 2^22,
// the range of the float-to-integer rounding by adding 1.5 2^23.  That is a
// step of 2^-25 of the tile's largest impulse for n <= 256.  Tiles of more
// than 2048 monomers take the split path: one component at a time, two words
// per cell (low word L = 32 - k bits, unsigned; high word signed), a step of
// 2^-(62 - 2k - ew) of the largest impulse, below the FP32 rounding of the
// products for k <= 16.
constexpr int kHX = kTX + 4, kHY = kTY + 4, kHZ = kTZ + 4;
constexpr int kHBox = kHX * kHY * kHZ;  // cells per component
constexpr int kHomeThreads = 512;
constexpr int kHomeWarps = kHomeThreads / 32;
constexpr int kHomeSplitK = 11;  // single-word path for n <= 2^11
static_assert(kHX % 32 == 20 && (kHX * kHY) % 32 == 16, "bank pattern of the box atomics");
static_assert(kHBox <= 65536, "box slots of the stencil records are 16-bit");
constexpr int kHomeStage = 128;  // candidates staged in shared memory at a time (three blocks per SM)
constexpr size_t kHomeBoxBytes = sizeof(unsigned) * 3 * kHBox;  // 57,600 B
constexpr size_t kHomeSmem = kHomeBoxBytes + kHomeStage * sizeof(WRec<float>);  // 73,984 B
static_assert(sizeof(WRec<float>) % 16 == 0 && kHomeBoxBytes % 16 == 0, "16-byte staging copies");

// 16- and 8-byte asynchronous copies global -> shared (LDGSTS), and the wait for all of this thread's
__device__ __forceinline__ void cp_async16(void* dst, const void* src) {
  const unsigned d = (unsigned)__cvta_generic_to_shared(dst);
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(d), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async8(void* dst, const void* src) {
  const unsigned d = (unsigned)__cvta_generic_to_shared(dst);
  asm volatile("cp.async.ca.shared.global [%0], [%1], 8;\n" ::"r"(d), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async_wait_all() { asm volatile("cp.async.wait_all;\n" ::: "memory"); }

// One staged candidate: the first 96 bytes of its record (the weights), and in
// place of the bases its impulses at the tile's scale (FP32) and box slots.
struct HomeCand {
  float w[3][2][4];
  float t[3];
  unsigned pad;
  uint2 hs;
  uint2 pad2;
};
static_assert(sizeof(HomeCand) == sizeof(WRec<float>) && offsetof(WRec<float>, hs) == 120, "staged records");

// The staged candidates 0 .. nc-1: a warp each, lane l adding the points
// (l & 3, (l >> 2) & 3, l >> 4) and two z-planes apart of all three components.
__device__ __forceinline__ void home_add_staged(const HomeCand* __restrict__ cand, int nc, unsigned* acc) {
  const int lane = threadIdx.x & 31;
  const int ix = lane & 3, jy = (lane >> 2) & 3, kz = lane >> 4;
  unsigned* base = acc + (kz * kHY + jy) * kHX + ix;
#pragma unroll 2
  for (int c = threadIdx.x >> 5; c < nc; c += kHomeWarps) {
    const HomeCand& R = cand[c];
    const float4 t = *reinterpret_cast<const float4*>(R.t);
    const uint2 h = R.hs;
    const float wx[2] = {R.w[0][0][ix], R.w[0][1][ix]}, wy[2] = {R.w[1][0][jy], R.w[1][1][jy]};
    const float wz[2][2] = {{R.w[2][0][kz], R.w[2][0][kz + 2]}, {R.w[2][1][kz], R.w[2][1][kz + 2]}};
#pragma unroll
    for (int d = 0; d < 3; d++) {
      const int sx = (d != 0), sy = (d != 1), sz = (d != 2);
      const float A = (d == 0 ? t.x : d == 1 ? t.y : t.z) * wy[sy] * wx[sx];
      const unsigned slot = d * kHBox + (d == 0 ? (h.x & 0xffffu) : d == 1 ? (h.x >> 16) : (h.y & 0xffffu));
      atomicAdd(base + slot, (unsigned)round_small(A * wz[sz][0]));
      atomicAdd(base + slot + 2 * kHY * kHX, (unsigned)round_small(A * wz[sz][1]));
    }
  }
}

// Candidates taken from memory: the entries of the overflow list (SPLIT 0), or
// every candidate of a tile on the split path, one component at a time.
template <int SPLIT>
__device__ __forceinline__ void home_add(const int* __restrict__ ids, int n_prim, int n_ovf, const TileSlots& ts, int tb,
                                         int dsel, double scale, int L, unsigned* acc,
                                         const double* __restrict__ tf, const WRec<float>* __restrict__ rec) {
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  const int ix = lane & 3, jy = (lane >> 2) & 3, kz = lane >> 4;
  const int loff = (kz * kHY + jy) * kHX + ix;
  auto one = [&](int p) {
    const WRec<float>& R = rec[p];
    const uint2 hsw = *reinterpret_cast<const uint2*>(&R.hs[0]);  // hs[0..2] and two bytes of padding
    const unsigned short* hs = reinterpret_cast<const unsigned short*>(&hsw);
#pragma unroll
    for (int d = 0; d < 3; d++) {
      if (SPLIT && d != dsel) continue;
      const int sx = (d != 0), sy = (d != 1), sz = (d != 2);
      const float wx = R.w[0][sx][ix], wy = R.w[1][sy][jy];
      const float wz0 = R.w[2][sz][kz], wz1 = R.w[2][sz][kz + 2];
      const float A = (float)(-tf[3L * p + d] * scale) * wy * wx;
      const int slot = (SPLIT ? 0 : d * kHBox) + hs[d] + loff;
      if (!SPLIT) {
        atomicAdd(acc + slot, (unsigned)round_small(A * wz0));
        atomicAdd(acc + slot + 2 * kHY * kHX, (unsigned)round_small(A * wz1));
      } else {
        // v = hi 2^L + lo, 0 <= lo < 2^L, split exactly in FP32, lo rounded
        const float tL = ldexpf(1.0f, L), itL = ldexpf(1.0f, -L);
        const float p0 = A * wz0, p1 = A * wz1;
        const float h0 = floorf(p0 * itL), h1 = floorf(p1 * itL);
        const float r0 = fmaf(-h0, tL, p0), r1 = fmaf(-h1, tL, p1);
        int l0 = (int)rintf(r0), l1 = (int)rintf(r1);
        int g0 = (int)h0, g1 = (int)h1;
        if (l0 >= (1 << L)) { l0 -= (1 << L); g0 += 1; }  // r rounded up onto 2^L
        if (l1 >= (1 << L)) { l1 -= (1 << L); g1 += 1; }
        atomicAdd(acc + slot, (unsigned)l0);
        atomicAdd(acc + kHBox + slot, (unsigned)g0);
        atomicAdd(acc + slot + 2 * kHY * kHX, (unsigned)l1);
        atomicAdd(acc + kHBox + slot + 2 * kHY * kHX, (unsigned)g1);
      }
    }
  };
  for (int c = wid; c < n_prim; c += kHomeWarps) one(ids[c]);
  for (int q = wid; q < n_ovf; q += kHomeWarps) {
    const int2 e = ts.ovf[q];
    if (e.x == tb) one(e.y);
  }
}

__global__ void __launch_bounds__(kHomeThreads, 3) k_spread_home(const double* __restrict__ tf, TileSlots ts,
                                                                 const WRec<float>* __restrict__ rec) {
  extern __shared__ __align__(16) unsigned hacc[];  // [3][kHZ][kHY][kHX], or [2][kHZ][kHY][kHX] (split path)
  HomeCand* cand = reinterpret_cast<HomeCand*>(reinterpret_cast<unsigned char*>(hacc) + kHomeBoxBytes);
  const int tb = blockIdx.x, tid = threadIdx.x;
  const int n = ts.count[tb];
  const int n_prim = min(n, ts.cap);
  const int* ids = ts.slots + (long)tb * ts.cap;
  const int n_ovf = (n > n_prim) ? min(*ts.ovf_count, ts.ovf_cap) : 0;
  float* out = ts.box + (long)tb * 3 * kHBox;
  if (tid == 0) ts.live[tb] = (n > 0);
  {
    const double m = __longlong_as_double((long long)ts.tmax[tb]);  // largest |impulse| of the tile (0 if none)
    const bool bad = !(m <= 1.0e300);
    const int ew = ts.quirk[tb] ? 0 : -3;
    uint4* z4 = reinterpret_cast<uint4*>(hacc);
    if (bad) {
      // a non-finite impulse makes the tile non-finite, as a floating-point sum would
      for (int i = tid; i < 3 * kHBox; i += kHomeThreads) out[i] = __int_as_float(0x7fc00000);
    } else {
      const int k = (n > 1) ? 32 - __clz(n - 1) : 1;  // ceil(log2 n)
      int em = 0;
      if (m > 0.0) frexp(m, &em);  // m < 2^em
      if (k <= kHomeSplitK) {
        const int S = max(-1000, min(1000, min(30 - k, 22) - em - ew));
        const double scale = ldexp(1.0, S);
        // The candidates' records go to shared memory in chunks, the weights and
        // slots by asynchronous copies that every thread issues at once (the
        // first chunk's while the box is zeroed), so that their load latency is
        // paid once per chunk; the impulses are scaled and rounded to FP32 by
        // the staging thread, once per candidate (every lane of the adding warp
        // multiplied and converted three FP64 values: 90 instructions a
        // candidate against 55)
        auto stage = [&](int c0, int nc) {
          for (int i = tid; i < nc * 8; i += kHomeThreads) {
            const int c = i >> 3, q = i & 7;
            const int p = ids[c0 + c];
            unsigned char* dst = reinterpret_cast<unsigned char*>(cand + c);
            if (q < 6) {
              cp_async16(dst + 16 * q, reinterpret_cast<const unsigned char*>(rec + p) + 16 * q);
            } else if (q == 6) {
              const float t0 = (float)(-tf[3L * p] * scale), t1 = (float)(-tf[3L * p + 1] * scale),
                          t2 = (float)(-tf[3L * p + 2] * scale);
              *reinterpret_cast<float4*>(cand[c].t) = make_float4(t0, t1, t2, 0.0f);
            } else {
              cp_async8(&cand[c].hs, &rec[p].hs[0]);
            }
          }
        };
        int c0 = 0, nc = min(kHomeStage, n_prim);
        stage(0, nc);
        for (int i = tid; i < 3 * kHBox / 4; i += kHomeThreads) z4[i] = make_uint4(0u, 0u, 0u, 0u);
        for (;;) {
          cp_async_wait_all();
          __syncthreads();  // the chunk and the zeroed box are visible to every thread
          home_add_staged(cand, nc, hacc);
          c0 += nc;
          if (c0 >= n_prim) break;
          nc = min(kHomeStage, n_prim - c0);
          __syncthreads();  // every warp is done with the chunk
          stage(c0, nc);
        }
        if (n_ovf > 0) home_add<0>(ids, 0, n_ovf, ts, tb, 0, scale, 0, hacc, tf, rec);
        __syncthreads();
        if (S >= -100 && S <= 100) {
          // the integer rounded to FP32 once, then scaled by a power of two (exact)
          const float inv = ldexpf(1.0f, -S);
          const uint4* h4 = reinterpret_cast<const uint4*>(hacc);
          float4* o4 = reinterpret_cast<float4*>(out);
          for (int i = tid; i < 3 * kHBox / 4; i += kHomeThreads) {
            const uint4 h = h4[i];
            o4[i] = make_float4(__int2float_rn((int)h.x) * inv, __int2float_rn((int)h.y) * inv,
                                __int2float_rn((int)h.z) * inv, __int2float_rn((int)h.w) * inv);
          }
        } else {
          const double inv = ldexp(1.0, -S);
          for (int i = tid; i < 3 * kHBox; i += kHomeThreads) out[i] = (float)((double)(int)hacc[i] * inv);
        }
      } else {
        const int L = 32 - k;
        const int S = max(-1000, min(1000, 62 - 2 * k - em - ew));
        const double inv = ldexp(1.0, -S);
        for (int i = tid; i < 2 * kHBox / 4; i += kHomeThreads) z4[i] = make_uint4(0u, 0u, 0u, 0u);
        __syncthreads();
        for (int d = 0; d < 3; d++) {
          if (d > 0) {
            __syncthreads();
            for (int i = tid; i < 2 * kHBox / 4; i += kHomeThreads) z4[i] = make_uint4(0u, 0u, 0u, 0u);
            __syncthreads();
          }
          home_add<1>(ids, n_prim, n_ovf, ts, tb, d, ldexp(1.0, S), L, hacc, tf, rec);
          __syncthreads();
          for (int i = tid; i < kHBox; i += kHomeThreads) {
            const long long v = (long long)(int)hacc[kHBox + i] * (1ll << L) + (long long)hacc[i];
            out[d * kHBox + i] = (float)((double)v * inv);
          }
        }
      }
    }
  }
  __syncthreads();  // every thread has read count[tb], tmax[tb], quirk[tb] and the overflow counter
  if (tid == 0) {
    ts.count[tb] = 0;
    ts.tmax[tb] = 0ull;
    ts.quirk[tb] = 0;
    __threadfence();
    if (atomicAdd(ts.done, 1u) == gridDim.x - 1) {  // the last block to finish: no block reads it any more
      *ts.ovf_count = 0;
      *ts.done = 0u;
    }
  }
}

// The fold on grids of 4 m cells along x whose tiles are at least 4 cells wide
// (a partial last tile included): block per (tile, component), a thread per
// four x cells of a (y, z) row.  Cell l of a tile of e cells lies in the boxes
// of its own tile at coordinate l + 2; of the tile below (cells 0, 1) at
// l + 2 + that tile's e; of the tile above (cells e - 2, e - 1) at l - e + 2:
// along x two float2 of the tile's own box and, for the first and the last four
// cells, one of the neighbour's.  Per cell the order of addition is fixed: z,
// then y, then x, each ascending.  Tiles one or two per axis wrap onto
// themselves by the same rule.  Every box is written, zeros for a tile without
// monomers.
// All loads of a row's boxes are issued before the first is added.  A thread
// per (x, y) column that walked z with scalar loads, and a thread per cell where
// the tiles do not divide the grid, took, with the home kernel, 55.5 us at 128^3
// (49.4 now), 60 at 100^3 (32), 146 at 192^3 (130).  Box rows in memory split
// into 64-byte tile rows and halo columns were slower (52.6 and 150: the home
// kernel's writes), so were rows of the z boxes one after another (52.7).
constexpr int kFoldThreads = 128;
struct FoldAxis {
  int t[2], b[2], n;  // tiles, box coordinates of the row, how many
};
__device__ __forceinline__ FoldAxis fold_axis(int l, int t, int nb, int T, int n) {
  FoldAxis f;
  const int e = min(T, n - t * T);
  f.t[0] = f.t[1] = t;
  f.b[0] = f.b[1] = l + 2;
  f.n = 1;
  if (l < 2) {
    const int q = (t == 0 ? nb : t) - 1;
    f.t[0] = q;
    f.b[0] = l + 2 + min(T, n - q * T);
    f.n = 2;
  } else if (l >= e - 2) {
    f.t[1] = (t + 1 == nb) ? 0 : t + 1;
    f.b[1] = l - e + 2;
    f.n = 2;
  }
  return f;
}
template <typename T>
__global__ void __launch_bounds__(kFoldThreads, 8) k_spread_fold4(T* __restrict__ f, int accumulate,
                                                               const float* __restrict__ box, BinSpec bs) {
  const int tb = blockIdx.x, d = blockIdx.y;
  const int nbx = bs.nb[0], nby = bs.nb[1], nbz = bs.nb[2], nx = bs.n[0], ny = bs.n[1], nz = bs.n[2];
  const int tx = tb % nbx, ty = (tb / nbx) % nby, tz = tb / (nbx * nby);
  const int ex = min(kTX, nx - tx * kTX), ey = min(kTY, ny - ty * kTY), ez = min(kTZ, nz - tz * kTZ);
  const int x4 = (threadIdx.x & 3) * 4, y = (threadIdx.x >> 2) & (kTY - 1);
  if (x4 >= ex || y >= ey) return;
  const int txl = (tx == 0 ? nbx : tx) - 1, txr = (tx + 1 == nbx) ? 0 : tx + 1;
  const int xl = min(kTX, nx - txl * kTX) + 2;  // the left tile's box column of cell 0
  const bool first = x4 == 0, last = x4 + 4 == ex;
  const FoldAxis fy = fold_axis(y, ty, nby, kTY, ny);
  for (int z = threadIdx.x >> 5; z < ez; z += kFoldThreads / 32) {
    const FoldAxis fz = fold_axis(z, tz, nbz, kTZ, nz);
    float2 a[4], b[4], l[4], r[4];
#pragma unroll
    for (int q = 0; q < 4; q++) {
      const int iz = q >> 1, iy = q & 1;
      a[q] = b[q] = l[q] = r[q] = make_float2(0.0f, 0.0f);
      if (iz < fz.n && iy < fy.n) {
        const float* row = box + (long)d * kHBox + (fz.b[iz] * kHY + fy.b[iy]) * kHX;
        const int t = (fz.t[iz] * nby + fy.t[iy]) * nbx;
        const float* own = row + (long)(t + tx) * (3 * kHBox) + x4 + 2;
        a[q] = __ldg(reinterpret_cast<const float2*>(own));
        b[q] = __ldg(reinterpret_cast<const float2*>(own + 2));
        if (first) l[q] = __ldg(reinterpret_cast<const float2*>(row + (long)(t + txl) * (3 * kHBox) + xl));
        if (last) r[q] = __ldg(reinterpret_cast<const float2*>(row + (long)(t + txr) * (3 * kHBox)));
      }
    }
    // (adding the zeros of the boxes that do not hold the cell changes nothing)
    float s0 = 0.0f, s1 = 0.0f, s2 = 0.0f, s3 = 0.0f;
#pragma unroll
    for (int q = 0; q < 4; q++) {
      s0 = (s0 + l[q].x) + a[q].x;
      s1 = (s1 + l[q].y) + a[q].y;
      s2 = (s2 + b[q].x) + r[q].x;
      s3 = (s3 + b[q].y) + r[q].y;
    }
    T* o = f + ((long)(d * nz + tz * kTZ + z) * ny + ty * kTY + y) * nx + tx * kTX + x4;
    if (!accumulate && sizeof(T) == 4 && ((uintptr_t)f & 15) == 0) {
      *reinterpret_cast<float4*>(o) = make_float4(s0, s1, s2, s3);
    } else {
      const float s[4] = {s0, s1, s2, s3};
#pragma unroll
      for (int i = 0; i < 4; i++) o[i] = accumulate ? (T)((double)o[i] + (double)s[i]) : (T)s[i];
    }
  }
}

// Boxes of the tiles along one axis that hold cell c: (tile, box coordinate)
// pairs in a fixed order.  Tile t covers cells [t T, t T + e) (e = T but for
// a partial last tile); its box holds coordinates 0 .. e + 3 for the cells
// t T - 2 .. t T + e + 1, taken periodically.  Tiles up to two away are
// looked at (a last tile of one cell lets the box two tiles away reach past
// it); small grids can hold a cell twice in one box.
struct BoxAxis {
  int t[8], b[8];
  int n;
};
__device__ __forceinline__ void box_axis(int c, int n, int T, int nb, BoxAxis& L) {
  const int th = c / T;
  L.n = 0;
  int seen[5];
#pragma unroll
  for (int dt = -2; dt <= 2; dt++) {
    int t = (th + dt) % nb;
    if (t < 0) t += nb;
    bool dup = false;
#pragma unroll
    for (int q = 0; q < dt + 2; q++) dup |= (seen[q] == t);
    seen[dt + 2] = t;
    if (dup) continue;
    const int t0 = t * T, e = min(T, n - t0);
#pragma unroll
    for (int kk = -1; kk <= 1; kk++) {
      const int bc = c - t0 + 2 + kk * n;
      if (bc >= 0 && bc < e + 4 && L.n < 8) {
        L.t[L.n] = t;
        L.b[L.n] = bc;
        L.n++;
      }
    }
  }
}

// f[d][z][y][x] (=, or +=) the sum over the boxes holding the cell, in a
// fixed order (z, y, x entries nested); boxes of empty tiles are skipped.  Any
// grid.
template <typename T>
__global__ void __launch_bounds__(256) k_spread_fold(T* __restrict__ f, int accumulate, const float* __restrict__ box,
                                                     const int* __restrict__ live, BinSpec bs) {
  const int x = blockIdx.x * 32 + threadIdx.x, y = blockIdx.y * 8 + threadIdx.y;
  const int nx = bs.n[0], ny = bs.n[1], nz = bs.n[2];
  const int z = blockIdx.z % nz, d = blockIdx.z / nz;
  if (x >= nx || y >= ny) return;
  float s = 0.0f;
  BoxAxis Lx, Ly, Lz;
  box_axis(x, nx, bs.tile[0], bs.nb[0], Lx);
  box_axis(y, ny, bs.tile[1], bs.nb[1], Ly);
  box_axis(z, nz, bs.tile[2], bs.nb[2], Lz);
  for (int iz = 0; iz < Lz.n; iz++)
    for (int iy = 0; iy < Ly.n; iy++)
      for (int ix = 0; ix < Lx.n; ix++) {
        const int t = (Lz.t[iz] * bs.nb[1] + Ly.t[iy]) * bs.nb[0] + Lx.t[ix];
        if (!live[t]) continue;
        s += __ldg(box + ((long)t * 3 + d) * kHBox + (Lz.b[iz] * kHY + Ly.b[iy]) * kHX + Lx.b[ix]);
      }
  T* dst = f + ((long)(d * nz + z) * ny + y) * nx + x;
  *dst = accumulate ? (T)((double)*dst + (double)s) : (T)s;
}

BinSpec spread_bin_spec(const int dims[3], double lo, double dx) {
  BinSpec bs{};
  bs.mode = 2;
  bs.lo = lo;
  bs.dx = dx;
  bs.L = dx * dims[0];
  const int t[3] = {kTX, kTY, kTZ};
  for (int a = 0; a < 3; a++) {
    bs.n[a] = dims[a];
    bs.tile[a] = t[a];
    bs.nb[a] = (dims[a] + t[a] - 1) / t[a];
  }
  return bs;
}

// most tiles one monomer can be filed under (product over axes of the most
// distinct tiles 5 consecutive cells can touch)
long spread_entries_per_monomer(const BinSpec& bs) {
  long prod = 1;
  for (int a = 0; a < 3; a++) {
    int best = 1;
    for (int c0 = 0; c0 < bs.n[a]; c0++) {
      int tl[5], cnt = 0;
      for (int i = 0; i < 5; i++) {
        const int t = ((c0 + i) % bs.n[a]) / bs.tile[a];
        bool dup = false;
        for (int j = 0; j < cnt; j++) dup |= (tl[j] == t);
        if (!dup) tl[cnt++] = t;
      }
      best = std::max(best, cnt);
    }
    prod *= best;
  }
  return prod;
}

template <typename T>
cudaError_t spread_gather(T* fgrid, bool accumulate, const double* x_old, const double* tf, const BinSpec& bs,
                          const int* offsets, const int* sorted, const CouplingArgs& a, cudaStream_t st,
                          const WRec<T>* rec) {
  const int ntiles = bs.nb[0] * bs.nb[1] * bs.nb[2];
  if (!accumulate && a.M == 0) {
    return cudaMemsetAsync(fgrid, 0, sizeof(T) * 3L * a.nx * a.ny * a.nz, st);
  }
  if (bs.mode != 2 || bs.tile[0] != kTX || bs.tile[1] != kTY || bs.tile[2] != kTZ) return cudaErrorInvalidValue;
  cudaError_t e = spread_prepare_attributes();
  if (e != cudaSuccess) return e;
  k_spread_tiles<T><<<ntiles, kSpreadThreads, spread_smem<T>(), st>>>(fgrid, accumulate ? 1 : 0, x_old, tf, bs, offsets,
                                                                  sorted, TileSlots{}, rec, a);
  count_launches(1);
  return cudaGetLastError();
}

template <typename T>
cudaError_t spread_slots(T* fgrid, bool accumulate, const double* x_old, const double* tf, const TileSlots& ts,
                         const CouplingArgs& a, cudaStream_t st, const WRec<T>* rec) {
  const BinSpec& bs = ts.bs;
  const int ntiles = bs.nb[0] * bs.nb[1] * bs.nb[2];
  if (!accumulate && a.M == 0) {
    return cudaMemsetAsync(fgrid, 0, sizeof(T) * 3L * (ts.cstride ? ts.cstride : (long)a.nx * a.ny * a.nz), st);
  }
  if (bs.mode != 2 || bs.tile[0] != kTX || bs.tile[1] != kTY || bs.tile[2] != kTZ || !ts.count)
    return cudaErrorInvalidValue;
  cudaError_t e = spread_prepare_attributes();
  if (e != cudaSuccess) return e;
  if constexpr (sizeof(T) == 4) {
    if (ts.home) {
      if (!ts.box || !ts.live || !rec) return cudaErrorInvalidValue;
      if (!ts.tmax || !ts.quirk) return cudaErrorInvalidValue;
      k_spread_home<<<ntiles, kHomeThreads, kHomeSmem, st>>>(tf, ts, rec);
      bool four = bs.n[0] % 4 == 0;  // no tile narrower than 4 cells, whole groups of 4 along x
      for (int ax = 0; ax < 3; ax++) four &= bs.n[ax] >= 4 && (bs.n[ax] % bs.tile[ax] == 0 || bs.n[ax] % bs.tile[ax] >= 4);
      if (four) {
        k_spread_fold4<T><<<dim3((unsigned)ntiles, 3), kFoldThreads, 0, st>>>(fgrid, accumulate ? 1 : 0, ts.box, bs);
      } else {
        const dim3 fb(32, 8), fg((unsigned)((a.nx + 31) / 32), (unsigned)((a.ny + 7) / 8), (unsigned)(3 * a.nz));
        k_spread_fold<T><<<fg, fb, 0, st>>>(fgrid, accumulate ? 1 : 0, ts.box, ts.live, bs);
      }
      count_launches(2);
      return cudaGetLastError();
    }
  }
  if (ts.home) return cudaErrorInvalidValue;
  // a slab of a decomposed instance: its tile layers only
  const int nlaunch = ts.tz1 ? (ts.tz1 - ts.tz0) * bs.nb[0] * bs.nb[1] : ntiles;
  k_spread_tiles<T><<<nlaunch, kSpreadThreads, spread_smem<T>(), st>>>(fgrid, accumulate ? 1 : 0, x_old, tf, bs, nullptr,
                                                                  nullptr, ts, rec, a);
  count_launches(1);
  return cudaGetLastError();
}
template cudaError_t spread_slots<double>(double*, bool, const double*, const double*, const TileSlots&,
                                          const CouplingArgs&, cudaStream_t, const WRec<double>*);
template cudaError_t spread_slots<float>(float*, bool, const double*, const double*, const TileSlots&,
                                         const CouplingArgs&, cudaStream_t, const WRec<float>*);

template cudaError_t interp_update<double>(const double*, const double*, double*, double*, double*, const double*,
                                           double*, WRec<double>*, const CouplingArgs&, uint32_t*, cudaStream_t,
                                           const TileSlots*);
template cudaError_t interp_update<float>(const float*, const double*, double*, double*, double*, const double*,
                                          double*, WRec<float>*, const CouplingArgs&, uint32_t*, cudaStream_t,
                                          const TileSlots*);
// The tile accumulators (49 KB in FP32, 74 KB in FP64) exceed the default 48 KB of dynamic
// shared memory: raise the limit once per device (the first call on a device
// does it; make that call before any stream capture).
cudaError_t spread_prepare_attributes() {
  static std::mutex mu;
  static bool done[kMaxSpreadDevices] = {false};
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return e;
  std::lock_guard<std::mutex> lk(mu);
  if (dev >= 0 && dev < kMaxSpreadDevices && done[dev]) return cudaSuccess;
  if ((e = cudaFuncSetAttribute((const void*)k_spread_tiles<float>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                (int)spread_smem<float>())) != cudaSuccess)
    return e;
  if ((e = cudaFuncSetAttribute((const void*)k_spread_tiles<double>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                (int)spread_smem<double>())) != cudaSuccess)
    return e;
  if ((e = cudaFuncSetAttribute((const void*)k_spread_home, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                (int)kHomeSmem)) != cudaSuccess)
    return e;
  if (dev >= 0 && dev < kMaxSpreadDevices) done[dev] = true;
  return cudaSuccess;
}

// ---------------------------------------------------------------- staged monomer upload
// Positions staged in device memory are checked there: cnt[0] counts the
// entries that are non-finite or more than `lim` from lo, cnt[1] those
// outside [lo, hi).  The commit copies the staged positions (and velocities;
// zeros without them) into the simulation only when both counts are zero, so
// a refused upload leaves the state as it was.
constexpr int kStageThreads = 256;
constexpr long kStageBlocks = 4 * 148;  // four blocks on each of the B200's 148 SMs

__global__ void __launch_bounds__(kStageThreads) k_stage_check(const double* __restrict__ x, long n, double lo,
                                                               double hi, double lim,
                                                               unsigned long long* __restrict__ cnt) {
  unsigned b = 0, o = 0;
  for (long i = blockIdx.x * (long)kStageThreads + threadIdx.x; i < n; i += (long)gridDim.x * kStageThreads) {
    const double q = x[i];
    b += !(fabs(q - lo) <= lim);  // NaN and infinities fail too
    o += (q < lo) | (q >= hi);
  }
#pragma unroll
  for (int w = 16; w > 0; w >>= 1) {
    b += __shfl_xor_sync(0xffffffffu, b, w);
    o += __shfl_xor_sync(0xffffffffu, o, w);
  }
  if ((threadIdx.x & 31) == 0) {
    if (b) atomicAdd(cnt, (unsigned long long)b);
    if (o) atomicAdd(cnt + 1, (unsigned long long)o);
  }
}

__global__ void __launch_bounds__(kStageThreads) k_stage_commit(const double* __restrict__ xin,
                                                                const double* __restrict__ vin, double* __restrict__ x,
                                                                double* __restrict__ v, long n,
                                                                const unsigned long long* __restrict__ cnt) {
  if (cnt[0] != 0ull || cnt[1] != 0ull) return;
  for (long i = blockIdx.x * (long)kStageThreads + threadIdx.x; i < n; i += (long)gridDim.x * kStageThreads) {
    x[i] = xin[i];
    v[i] = vin ? vin[i] : 0.0;
  }
}

static unsigned stage_blocks(long n) {
  return (unsigned)std::max(1L, std::min(kStageBlocks, (n + kStageThreads - 1) / kStageThreads));
}

cudaError_t stage_check(const double* xin, long n, double lo, double hi, double lim, unsigned long long* cnt,
                        cudaStream_t st) {
  cudaError_t e = cudaMemsetAsync(cnt, 0, 2 * sizeof(unsigned long long), st);
  if (e != cudaSuccess) return e;
  if (n == 0) return cudaSuccess;
  k_stage_check<<<stage_blocks(n), kStageThreads, 0, st>>>(xin, n, lo, hi, lim, cnt);
  count_launches(1);
  return cudaGetLastError();
}

cudaError_t stage_commit(const double* xin, const double* vin, double* x, double* v, long n,
                         const unsigned long long* cnt, cudaStream_t st) {
  if (n == 0) return cudaSuccess;
  k_stage_commit<<<stage_blocks(n), kStageThreads, 0, st>>>(xin, vin, x, v, n, cnt);
  count_launches(1);
  return cudaGetLastError();
}

template cudaError_t spread_gather<double>(double*, bool, const double*, const double*, const BinSpec&, const int*,
                                           const int*, const CouplingArgs&, cudaStream_t, const WRec<double>*);
template cudaError_t spread_gather<float>(float*, bool, const double*, const double*, const BinSpec&, const int*,
                                          const int*, const CouplingArgs&, cudaStream_t, const WRec<float>*);

}  // namespace selm
