// fluid_plane.cuh - the x/y plane kernels of every form for compile-time
// grid sizes N = N1 N2 (N and N1 even, both factors <= 16), one block per
// (component, z) plane.
//
// Every phase holds one factor's points in registers and the plane lies in
// shared memory once; there is no buffer beside it and three barriers:
//   forward  1 global -> N1-point DFTs of x        2 N2-point DFTs of x, split
//            into the two rows of each pair         3 N1-point DFTs of y
//            4 N2-point DFTs of y -> global
//   inverse  1 global -> N1-point DFTs of y        2 N2-point DFTs of y
//            3 rows joined in pairs, N2-point DFTs of x
//            4 N1-point DFTs of x -> global
// Two real rows make one complex line: N complex values, then 2 (N/2 + 1)
// half-spectrum values, which take the line's own slots: mode m of the first
// row where Z[m] was, mode m of the second where Z[N-m] was (the modes 0 and
// N/2 of the second row in two slots at the end), so a thread that holds Z[m]
// and Z[N-m] splits or joins in registers.  A line's slots are groups of odd
// pitch, lines an odd pitch apart, so that lanes one group or one line apart
// hit distinct banks.
//
// 128^3 FP32 (384 planes of 75 KB: three blocks per SM, one wave; the chunked
// form with its row-pair buffer had two per SM, 1.3 waves, seven barriers per
// chunk and twice the shared-memory traffic) is bound by shared-memory and
// barrier latency: forward 24.9 -> 22.9 us and inverse 28.0 -> 22.3, for 51 MB
// each that take 8; FP64 (150 KB a plane, one block per SM) 47.5 and 53.4 ->
// 38.3 both, for 101 MB that take 16.
#pragma once
#include "common.cuh"
#include "fft_fast.cuh"

namespace selm {

template <typename T, int N, int N1> struct PlaneShape {
  static constexpr int N2 = N / N1, NH = N / 2 + 1, HP = N / 2;
  static_assert(N1 * N2 == N && N1 <= 16 && N2 <= 16 && N1 % 2 == 0, "N = N1 N2, N1 even");
  // forward: slot of mode m = (m % N1) GF + m / N1; inverse: (m / N1) GI + m % N1
  static constexpr int GF = N2 | 1, PWF = (N1 * GF + 2) | 1;
  static constexpr int GI = N1 | 1, PWI = (N2 * GI + 2) | 1;
  static constexpr int PW = PWF > PWI ? PWF : PWI;
  static constexpr size_t smem = sizeof(cpx<T>) * (size_t)(HP * PW + N);
  // 64 registers a thread in FP32, 128 in FP64
  static constexpr int kThreadsPerSm = sizeof(T) == 4 ? 1024 : 512;
  // blocks per SM: the fewest block rounds (waves of the 3 N planes times
  // blocks per SM), then the most
  static constexpr int blocks() {
    int best = 1;
    long rounds = -1;
    for (int nb = 1; nb <= 4; nb++) {
      if (nb * (smem + 1024) > 228 * 1024) break;
      const long r = (3L * N + 148 * nb - 1) / (148 * nb) * nb;
      if (rounds < 0 || r <= rounds) {
        rounds = r;
        best = nb;
      }
    }
    return best;
  }
  static constexpr int NB = blocks();
  // points that a thread of t goes through, one after another, in the four phases
  static constexpr int chain(int t) {
    const int units[4] = {HP * N2, HP * (N1 / 2 + 1), NH * N2, NH * N1}, points[4] = {N1, 2 * N2, N1, N2};
    int c = 0;
    for (int i = 0; i < 4; i++) c += (units[i] + t - 1) / t * points[i];
    return c;
  }
  // threads: the largest phase's units in equal rounds of at most what the
  // registers give; more where that shortens the chain by a quarter or more
  // below that limit (a phase then needs a round less: FP64 112^3 39.4 -> 35.3
  // us, 60^3 12.8 -> 11.2).  For less, and at the limit itself, more threads
  // lost: FP64 128^3 37.6 -> 38.3, FP32 168^3 inverse 59.8 -> 66, 120^3 25.4 -> 28.1.
  static constexpr int threads() {
    const int cap = kThreadsPerSm / NB / 32 * 32, units = NH * (N1 > N2 ? N1 : N2);
    const int rounds = (units + cap - 1) / cap;
    const int even = ((units + rounds - 1) / rounds + 31) / 32 * 32;
    int best = even < 64 ? 64 : even;
    for (int t = best + 32; t < cap; t += 32)
      if (4 * chain(t) <= 3 * chain(even) && chain(t) < chain(best)) best = t;
    return best;
  }
  static constexpr int TPB = threads();
};

template <int R, int S, typename C> __device__ __forceinline__ void twiddle_row(C (&v)[R], const C* tw, int t) {
#pragma unroll
  for (int j = 1; j < R; j++) {
    C w = tw[t * j];
    if (S > 0) w.y = -w.y;
    v[j] = cmul(v[j], w);
  }
}

// What the forward kernel transforms: the planes of an array, or the
// divergence of a velocity (forward differences, cuda/SELM_Kernel.cu:100-116).
template <typename T> struct ArrayPlanes {
  const T* in;
  struct Plane {
    const T* src;
    __device__ __forceinline__ T at(int y, int x, int n) const { return src[y * n + x]; }
  };
  __device__ __forceinline__ Plane plane(int p, int n) const { return Plane{in + (long)p * (n * n)}; }
};
struct DivergencePlanes {
  const double* u;
  double idx;  // 1/dx
  struct Plane {
    const double *a, *b, *c, *cn;  // the three components, the third's next plane
    double idx;
    __device__ __forceinline__ double at(int y, int x, int n) const {
      const int q = y * n + x;
      const int i1 = (x != n - 1) ? 1 : -x, j1 = (y != n - 1) ? n : -y * n;
      return (a[q + i1] - a[q] + b[q + j1] - b[q] + cn[q] - c[q]) * idx;
    }
  };
  __device__ __forceinline__ Plane plane(int z, int n) const {
    const long pl = (long)n * n, N = pl * n;
    const double* c = u + 2 * N + z * pl;
    return Plane{u + z * pl, u + N + z * pl, c, (z != n - 1) ? c + pl : u + 2 * N, idx};
  }
};

template <typename T, int N, int N1, typename In>
__global__ void __launch_bounds__(PlaneShape<T, N, N1>::TPB, PlaneShape<T, N, N1>::NB)
    k_xy_forward_fast(In in, cpx<T>* out, const cpx<T>* __restrict__ twx) {
  using C = cpx<T>;
  using S = PlaneShape<T, N, N1>;
  constexpr int N2 = S::N2, NH = S::NH, HP = S::HP, G = S::GF, PW = S::PW;
  constexpr int X0 = N1 * G;  // slots of the second row's modes 0 and N/2
  extern __shared__ __align__(16) unsigned char smem_raw[];
  C* P = reinterpret_cast<C*>(smem_raw);  // [HP][PW]
  C* tw = P + HP * PW;
  const auto src = in.plane(blockIdx.x, N);
  C* dst = out + (long)blockIdx.x * (N * NH);
  for (int t = threadIdx.x; t < N; t += S::TPB) tw[t] = twx[t];
  previous_done();
  __syncthreads();
  // x, first factor: thread (row pair, n2), n2 fastest (runs of N2 values of a row)
  for (int u = threadIdx.x; u < HP * N2; u += S::TPB) {
    const int lr = u / N2, n2 = u % N2;
    C v[N1];
#pragma unroll
    for (int n1 = 0; n1 < N1; n1++)
      v[n1] = fftk::mk<C>(src.at(lr, N2 * n1 + n2, N), src.at(lr + HP, N2 * n1 + n2, N));
    fftk::dft<N1, -1>(v);
    if (N2 > 1) twiddle_row<N1, -1>(v, tw, n2);
    C* p = P + lr * PW + n2;
#pragma unroll
    for (int k1 = 0; k1 < N1; k1++) p[k1 * G] = v[k1];
  }
  __syncthreads();
  // x, second factor and the split: thread (row pair, k1), with the modes of k1
  // and N1 - k1.  A = (Z[m] + conj Z[N-m])/2, B = (Z[m] - conj Z[N-m])/(2i)
  for (int u = threadIdx.x; u < HP * (N1 / 2 + 1); u += S::TPB) {
    const int kp = u / HP, lr = u % HP;
    C* line = P + lr * PW;
    const T h = T(0.5);
    auto first = [&](C z, C zr) { return fftk::mk<C>((z.x + zr.x) * h, (z.y - zr.y) * h); };
    auto second = [&](C z, C zr) { return fftk::mk<C>((z.y + zr.y) * h, (zr.x - z.x) * h); };
    if (kp == 0) {
      // modes N1 k2: N1 (N2 - k2) is the partner
      C c[N2];
#pragma unroll
      for (int j = 0; j < N2; j++) c[j] = line[j];
      fftk::dft<N2, -1>(c);
      line[0] = fftk::mk<C>(c[0].x, T(0));
      line[X0] = fftk::mk<C>(c[0].y, T(0));
#pragma unroll
      for (int k2 = 1; k2 <= N2 / 2; k2++) {
        if (2 * k2 == N2) {
          line[k2] = fftk::mk<C>(c[k2].x, T(0));
          line[X0 + 1] = fftk::mk<C>(c[k2].y, T(0));
        } else {
          line[k2] = first(c[k2], c[N2 - k2]);
          line[N2 - k2] = second(c[k2], c[N2 - k2]);
        }
      }
    } else {
      // modes kp + N1 k2: N1 - kp + N1 (N2 - 1 - k2) is the partner (kp = N1/2: its own group)
      C a[N2], b[N2];
      C *pa = line + kp * G, *pb = line + (N1 - kp) * G;
#pragma unroll
      for (int j = 0; j < N2; j++) {
        a[j] = pa[j];
        b[j] = pb[j];
      }
      fftk::dft<N2, -1>(a);
      fftk::dft<N2, -1>(b);
#pragma unroll
      for (int k2 = 0; k2 < N2; k2++) {
        const int q = N2 - 1 - k2;
        if (k2 <= (N2 - 1) / 2) {  // kp + N1 k2 <= N/2
          const C fa = first(a[k2], b[q]), fb = second(a[k2], b[q]);
          if (k2 == q && 2 * kp == N1) {  // mode N/2
            pa[k2] = fa;
            line[X0 + 1] = fb;
          } else {
            pa[k2] = fa;
            pb[q] = fb;
          }
        } else {
          pb[q] = first(b[q], a[k2]);
          pa[k2] = second(b[q], a[k2]);
        }
      }
    }
  }
  __syncthreads();
  auto slot_a = [](int m) { return (m % N1) * G + m / N1; };
  auto slot_b = [&](int m) { return m == 0 ? X0 : (2 * m == N ? X0 + 1 : slot_a(N - m)); };
  // y, first factor: thread (m, n2); rows N2 n1 + n2, the first N/2 in the pairs' first rows
  for (int u = threadIdx.x; u < NH * N2; u += S::TPB) {
    const int n2 = u / NH, m = u % NH;
    C *a = P + n2 * PW + slot_a(m), *b = P + n2 * PW + slot_b(m);
    C v[N1];
#pragma unroll
    for (int n1 = 0; n1 < N1; n1++) v[n1] = (n1 < N1 / 2 ? a : b)[(n1 % (N1 / 2)) * (N2 * PW)];
    fftk::dft<N1, -1>(v);
    if (N2 > 1) twiddle_row<N1, -1>(v, tw, n2);
#pragma unroll
    for (int k1 = 0; k1 < N1; k1++) (k1 < N1 / 2 ? a : b)[(k1 % (N1 / 2)) * (N2 * PW)] = v[k1];
  }
  __syncthreads();
  // y, second factor: thread (m, k1), to rows k1 + N1 k2 of the half spectrum
  for (int u = threadIdx.x; u < NH * N1; u += S::TPB) {
    const int k1 = u / NH, m = u % NH;
    const bool lo = k1 < N1 / 2;
    const C* p = P + (lo ? k1 : k1 - N1 / 2) * (N2 * PW) + (lo ? slot_a(m) : slot_b(m));
    C v[N2];
#pragma unroll
    for (int j = 0; j < N2; j++) v[j] = p[j * PW];
    fftk::dft<N2, -1>(v);
    C* d = dst + k1 * NH + m;
#pragma unroll
    for (int k2 = 0; k2 < N2; k2++) d[k2 * (N1 * NH)] = v[k2];
  }
}

template <typename T, int N, int N1>
__global__ void __launch_bounds__(PlaneShape<T, N, N1>::TPB, PlaneShape<T, N, N1>::NB)
    k_xy_inverse_fast(const cpx<T>* in, T* out, const cpx<T>* __restrict__ twx,
                      uint64_t* step) {
  using C = cpx<T>;
  using S = PlaneShape<T, N, N1>;
  constexpr int N2 = S::N2, NH = S::NH, HP = S::HP, G = S::GI, PW = S::PW;
  constexpr int X0 = N2 * G;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  C* P = reinterpret_cast<C*>(smem_raw);
  C* tw = P + HP * PW;
  const C* src = in + (long)blockIdx.x * (N * NH);
  T* dst = out + (long)blockIdx.x * (N * N);
  for (int t = threadIdx.x; t < N; t += S::TPB) tw[t] = twx[t];
  previous_done();
  // the last kernel of the step's fluid solve advances the device step counter
  // (the step's noise has been drawn; nothing later in the step reads it)
  if (step && blockIdx.x == 0 && threadIdx.x == 0) *step += 1;
  __syncthreads();
  auto slot_a = [](int m) { return (m / N1) * G + m % N1; };
  auto slot_b = [&](int m) { return m == 0 ? X0 : (2 * m == N ? X0 + 1 : slot_a(N - m)); };
  // y, first factor: thread (m, n2), modes N2 n1 + n2
  for (int u = threadIdx.x; u < NH * N2; u += S::TPB) {
    const int n2 = u / NH, m = u % NH;
    const C* s = src + n2 * NH + m;
    C v[N1];
#pragma unroll
    for (int n1 = 0; n1 < N1; n1++) v[n1] = s[n1 * (N2 * NH)];
    fftk::dft<N1, +1>(v);
    if (N2 > 1) twiddle_row<N1, +1>(v, tw, n2);
    C *a = P + n2 * PW + slot_a(m), *b = P + n2 * PW + slot_b(m);
#pragma unroll
    for (int k1 = 0; k1 < N1; k1++) (k1 < N1 / 2 ? a : b)[(k1 % (N1 / 2)) * (N2 * PW)] = v[k1];
  }
  __syncthreads();
  // y, second factor: thread (m, k1); row k1 + N1 k2 ends at N2 k1 + k2, so that
  // pair lr holds rows y = lr / N2 + N1 (lr % N2) and y + N1/2
  for (int u = threadIdx.x; u < NH * N1; u += S::TPB) {
    const int k1 = u / NH, m = u % NH;
    const bool lo = k1 < N1 / 2;
    C* p = P + (lo ? k1 : k1 - N1 / 2) * (N2 * PW) + (lo ? slot_a(m) : slot_b(m));
    C v[N2];
#pragma unroll
    for (int j = 0; j < N2; j++) v[j] = p[j * PW];
    fftk::dft<N2, +1>(v);
#pragma unroll
    for (int j = 0; j < N2; j++) p[j * PW] = v[j];
  }
  __syncthreads();
  // rows joined, x first factor (N2 points, modes N1 n1 + n2): thread (row pair,
  // n2) with the modes of n2 and N1 - n2.  Z[m] = A + i B, Z[N-m] = conj A + i conj B;
  // the imaginary parts of the modes 0 and N/2 drop out
  for (int u = threadIdx.x; u < HP * (N1 / 2 + 1); u += S::TPB) {
    const int np = u / HP, lr = u % HP;
    C* line = P + lr * PW;
    auto joined = [](C a, C b) { return fftk::mk<C>(a.x - b.y, a.y + b.x); };
    auto mirror = [](C a, C b) { return fftk::mk<C>(a.x + b.y, b.x - a.y); };
    if (np == 0) {
      C c[N2];
      c[0] = fftk::mk<C>(line[0].x, line[X0].x);
#pragma unroll
      for (int n1 = 1; n1 <= N2 / 2; n1++) {
        if (2 * n1 == N2) {
          c[n1] = fftk::mk<C>(line[n1 * G].x, line[X0 + 1].x);
        } else {
          const C a = line[n1 * G], b = line[(N2 - n1) * G];
          c[n1] = joined(a, b);
          c[N2 - n1] = mirror(a, b);
        }
      }
      fftk::dft<N2, +1>(c);
#pragma unroll
      for (int k1 = 0; k1 < N2; k1++) line[k1 * G] = c[k1];
    } else {
      C a[N2], b[N2];
      C *pa = line + np, *pb = line + (N1 - np);
#pragma unroll
      for (int n1 = 0; n1 <= (N2 - 1) / 2; n1++) {
        const int q = N2 - 1 - n1;
        // mode np + N1 n1 <= N/2 of the pair, and, where that differs, N1 - np + N1 n1
        C fa = pa[n1 * G], fb = pb[q * G];
        if (n1 == q && 2 * np == N1) {  // mode N/2
          fa.y = T(0);
          fb = fftk::mk<C>(line[X0 + 1].x, T(0));
        }
        a[n1] = joined(fa, fb);
        b[q] = mirror(fa, fb);
        if (n1 != q) {
          const C ga = pb[n1 * G], gb = pa[q * G];
          b[n1] = joined(ga, gb);
          a[q] = mirror(ga, gb);
        }
      }
      fftk::dft<N2, +1>(a);
      fftk::dft<N2, +1>(b);
      twiddle_row<N2, +1>(a, tw, np);
      twiddle_row<N2, +1>(b, tw, N1 - np);
#pragma unroll
      for (int k1 = 0; k1 < N2; k1++) {
        pa[k1 * G] = a[k1];
        pb[k1 * G] = b[k1];
      }
    }
  }
  __syncthreads();
  // x, second factor: thread (row pair, k1), k1 fastest, to x = k1 + N2 k2
  for (int u = threadIdx.x; u < HP * N2; u += S::TPB) {
    const int lr = u / N2, k1 = u % N2;
    const C* p = P + lr * PW + k1 * G;
    C v[N1];
#pragma unroll
    for (int j = 0; j < N1; j++) v[j] = p[j];
    fftk::dft<N1, +1>(v);
    T* d = dst + (lr / N2 + N1 * (lr % N2)) * N + k1;
#pragma unroll
    for (int k2 = 0; k2 < N1; k2++) {
      d[N2 * k2] = v[k2].x;
      d[(N1 / 2) * N + N2 * k2] = v[k2].y;
    }
  }
}

}  // namespace selm
