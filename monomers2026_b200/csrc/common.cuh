// common.cuh - device helpers shared by every SELM kernel (sm_100a).
//
// Philox4x32-10 is the published counter-based generator of Salmon, Moraes,
// Dror and Shaw (SC'11).  Counter layout (one call per use):
//   fluid noise   : {mode q, component d (0..2), step lo, step hi}
//   monomer noise : {monomer p, 4 + component d, step lo, step hi}
//   key           : {seed lo, seed hi}
// Normals are Box-Muller pairs of two 52-bit open-interval uniforms, so the
// draws are a pure function of (seed, step, index) and do not depend on the
// launch shape, the batch a job runs in, or the number of jobs.
#pragma once
#include <cstdint>
#include <cuda_runtime.h>

namespace selm {

constexpr double kPi = 3.14159265358979323846;

// error word bits (per job, device resident, read back by the host)
enum : uint32_t {
  ERR_NONFINITE = 1u << 0,        // NaN/Inf in a monomer state
  ERR_DISPLACEMENT = 1u << 1,     // |v dt| > L/2 (reference warns, cuda/SELM_Kernel.cu:363)
  ERR_FENE_STRETCH = 1u << 2,     // FENE bond past 0.9 R0^2, clamped
  ERR_FENE_BROKEN = 1u << 3,      // FENE bond past the LAMMPS error limit
  ERR_BUCKET_OVERFLOW = 1u << 4,  // candidate list longer than the kernel bound
  ERR_NLIST_OVERFLOW = 1u << 5,   // more pair partners within the list radius than the list holds
  ERR_COPY_TIMEOUT = 1u << 6,     // an asynchronous (TMA) copy did not complete within its wait bound
};

template <typename T> struct cpx_t;
template <> struct cpx_t<float> { using type = float2; };
template <> struct cpx_t<double> { using type = double2; };
template <typename T> using cpx = typename cpx_t<T>::type;

template <typename C> __device__ __forceinline__ C cmk(decltype(C::x) a, decltype(C::x) b) {
  C c; c.x = a; c.y = b; return c;
}
template <typename C> __device__ __forceinline__ C cadd(C a, C b) { return cmk<C>(a.x + b.x, a.y + b.y); }
template <typename C> __device__ __forceinline__ C csub(C a, C b) { return cmk<C>(a.x - b.x, a.y - b.y); }
template <typename C> __device__ __forceinline__ C cmul(C a, C b) {
  return cmk<C>(a.x * b.x - a.y * b.y, a.x * b.y + a.y * b.x);
}
template <typename C> __device__ __forceinline__ C cscale(C a, decltype(C::x) s) { return cmk<C>(a.x * s, a.y * s); }

// ---------------------------------------------------------------- dependent launches
// Kernels launched by launch_next (selm_kernels.h) may start while the kernel
// before them on the stream still runs: what they do before previous_done()
// may not touch memory that an earlier kernel reads or writes.  The call waits
// until that kernel has finished (so everything before it has), then lets the
// next one start.  Every block makes it before it returns, and pointers to what
// earlier kernels write are not __restrict__: the compiler may not move or
// cache those reads across it.
__device__ __forceinline__ void previous_done() {
  cudaGridDependencySynchronize();
  cudaTriggerProgrammaticLaunchCompletion();
}

// ---------------------------------------------------------------- Philox
__host__ __device__ __forceinline__ void philox4x32_10(uint32_t c0, uint32_t c1, uint32_t c2, uint32_t c3,
                                                       uint32_t k0, uint32_t k1, uint32_t out[4]) {
#ifdef __CUDA_ARCH__
#pragma unroll
#endif
  for (int r = 0; r < 10; r++) {
    const uint64_t p0 = (uint64_t)0xD2511F53u * c0;
    const uint64_t p1 = (uint64_t)0xCD9E8D57u * c2;
    const uint32_t hi0 = (uint32_t)(p0 >> 32), lo0 = (uint32_t)p0;
    const uint32_t hi1 = (uint32_t)(p1 >> 32), lo1 = (uint32_t)p1;
    c0 = hi1 ^ c1 ^ k0;
    c1 = lo1;
    c2 = hi0 ^ c3 ^ k1;
    c3 = lo0;
    k0 += 0x9E3779B9u;
    k1 += 0xBB67AE85u;
  }
  out[0] = c0; out[1] = c1; out[2] = c2; out[3] = c3;
}

// The ten round keys of a Philox4x32-10 key (k0 + r W0, k1 + r W1, r = 0..9):
// the same for every counter of a simulation, so kernels take them as
// parameters instead of stepping the key in every draw.
struct PhiloxKeys {
  uint32_t k[20];
};
inline PhiloxKeys philox_keys(uint64_t seed) {
  PhiloxKeys K{};
  uint32_t k0 = (uint32_t)seed, k1 = (uint32_t)(seed >> 32);
  for (int r = 0; r < 10; r++) {
    K.k[2 * r] = k0;
    K.k[2 * r + 1] = k1;
    k0 += 0x9E3779B9u;
    k1 += 0xBB67AE85u;
  }
  return K;
}
// philox4x32_10 with the round keys given (the same output)
__device__ __forceinline__ void philox4x32_10(uint32_t c0, uint32_t c1, uint32_t c2, uint32_t c3, const PhiloxKeys& K,
                                              uint32_t out[4]) {
#pragma unroll
  for (int r = 0; r < 10; r++) {
    const uint64_t p0 = (uint64_t)0xD2511F53u * c0;
    const uint64_t p1 = (uint64_t)0xCD9E8D57u * c2;
    const uint32_t hi0 = (uint32_t)(p0 >> 32), lo0 = (uint32_t)p0;
    const uint32_t hi1 = (uint32_t)(p1 >> 32), lo1 = (uint32_t)p1;
    c0 = hi1 ^ c1 ^ K.k[2 * r];
    c1 = lo1;
    c2 = hi0 ^ c3 ^ K.k[2 * r + 1];
    c3 = lo0;
  }
  out[0] = c0; out[1] = c1; out[2] = c2; out[3] = c3;
}

// Box-Muller pair of two 52-bit uniforms in FP64, from their Philox words.
//   u in (0, 1) is built from its 52 bits plus 1/2 (exact in 53 bits);
//   u1 = m 2^e with m in [1/sqrt 2, sqrt 2): -ln u1 = -(e ln 2 + 2 atanh s),
//   s = (m - 1)/(m + 1), |s| < 0.1716, by the odd series of atanh; the quotient
//   and the square root by Newton steps from FP32 approximations; the angle's
//   quarter turns come off exactly (4 u2 minus its nearest integer), and sine
//   and cosine of the rest, within pi/4, are Taylor sums.
// Series to s^21 (left out: below 1e-18 of it), to a^17 and a^16 (below 1e-19 and
// 3e-18), quotient and root corrected to FP64, ln 2 in two parts: log, sqrt and
// sincos to about an ulp each at two thirds of their operations (128^3 FP64 z
// kernel 96 us with the library's functions).
__device__ __forceinline__ void box_muller(const uint32_t (&o)[4], double& z0, double& z1) {
  const double u1 = __hiloint2double((int)(0x3ff00000u | (o[0] >> 12)), (int)((o[0] << 20) | (o[1] >> 12))) -
                    (1.0 - 0x1p-53);
  const double u2 = __hiloint2double((int)(0x3ff00000u | (o[2] >> 12)), (int)((o[2] << 20) | (o[3] >> 12))) -
                    (1.0 - 0x1p-53);
  const int hi = __double2hiint(u1);
  int e = (hi >> 20) - 1023;
  double m = __hiloint2double((hi & 0xfffff) | 0x3ff00000, __double2loint(u1));
  if (m > 1.4142135623730951) {
    m *= 0.5;
    e += 1;
  }
  const double mm = m - 1.0, mp = m + 1.0;
  double q = (double)__frcp_rn((float)mp);
  q = fma(q, fma(-mp, q, 1.0), q);
  double s = mm * q;
  s = fma(fma(-(m - (mp - 1.0)), s, fma(-mp, s, mm)), q, s);  // with the rounding of m + 1
  const double s2 = s * s;
  double p = 1.0 / 21.0;
  p = fma(p, s2, 1.0 / 19.0);
  p = fma(p, s2, 1.0 / 17.0);
  p = fma(p, s2, 1.0 / 15.0);
  p = fma(p, s2, 1.0 / 13.0);
  p = fma(p, s2, 1.0 / 11.0);
  p = fma(p, s2, 1.0 / 9.0);
  p = fma(p, s2, 1.0 / 7.0);
  p = fma(p, s2, 1.0 / 5.0);
  p = fma(p, s2, 1.0 / 3.0);
  // -2 ln u1 > 0; ln 2 = hi + lo, hi with 20 trailing zero bits: e hi is exact
  constexpr double ln2hi = 0x1.62e42fefap-1, ln2lo = 0x1.cf79abc9e3b3ap-40;
  const double y = -2.0 * fma((double)e, ln2hi, fma((double)e, ln2lo, 2.0 * fma(s * s2, p, s)));
  double g = (double)rsqrtf((float)y);
  g = fma(g, fma(-0.5 * y * g, g, 0.5), g);
  const double h = y * g;
  const double r = fma(fma(-h, h, y), 0.5 * g, h);
  const double w = 4.0 * u2, big = w + 6755399441055744.0;  // 1.5 2^52: rounds w to an integer
  const int n = __double2loint(big);
  const double a = (w - (big - 6755399441055744.0)) * 1.5707963267948966, a2 = a * a;
  double sn = 1.0 / 355687428096000.0;
  sn = fma(sn, a2, -1.0 / 1307674368000.0);
  sn = fma(sn, a2, 1.0 / 6227020800.0);
  double cs = 1.0 / 20922789888000.0;
  cs = fma(cs, a2, -1.0 / 87178291200.0);
  cs = fma(cs, a2, 1.0 / 479001600.0);
  sn = fma(sn, a2, -1.0 / 39916800.0);
  sn = fma(sn, a2, 1.0 / 362880.0);
  cs = fma(cs, a2, -1.0 / 3628800.0);
  sn = fma(sn, a2, -1.0 / 5040.0);
  cs = fma(cs, a2, 1.0 / 40320.0);
  sn = fma(sn, a2, 1.0 / 120.0);
  cs = fma(cs, a2, -1.0 / 720.0);
  sn = fma(sn, a2, -1.0 / 6.0);
  cs = fma(cs, a2, 1.0 / 24.0);
  cs = fma(cs, a2, -0.5);
  sn = fma(sn * a2, a, a);
  cs = fma(cs, a2, 1.0);
  const double c = (n & 1) ? sn : cs, d = (n & 1) ? cs : sn;
  z0 = r * (((n + 1) & 2) ? -c : c);  // cos of n quarter turns plus a
  z1 = r * ((n & 2) ? -d : d);        // sin
}

// Box-Muller pair from one Philox block
template <typename Key>
__device__ __forceinline__ void philox_normal2(const Key& key, uint32_t c0, uint32_t c1, uint64_t step, double& z0,
                                               double& z1) {
  uint32_t o[4];
  if constexpr (sizeof(Key) == sizeof(PhiloxKeys))
    philox4x32_10(c0, c1, (uint32_t)step, (uint32_t)(step >> 32), key, o);
  else
    philox4x32_10(c0, c1, (uint32_t)step, (uint32_t)(step >> 32), (uint32_t)key, (uint32_t)(key >> 32), o);
  box_muller(o, z0, z1);
}

// FP32 Box-Muller pair from the same Philox block, the same normals as
// philox_normal2 to FP32 precision.  The FP64 uniforms are u = (x + 1/2) 2^-52
// with x = o0 2^20 + (o1 >> 12).  Rounding u to FP32 costs 2^-24 absolute,
// which near u = 1 (radius sqrt(-2 ln u) ~ sqrt(2 (1 - u))) is a large
// relative error of the radius; so for u >= 3/4 the complement 1 - u is built
// from the complemented integer bits (exact to FP32 rounding, relative) and
// taken as m - 1 = -(1 - u), e = 0; for smaller u = m 2^e, m in [3/4, 3/2),
// m - 1 is exact in FP32.  Then -ln u = -(e ln 2 + 2 atanh s), s = (m - 1)/(m + 1),
// |s| <= 1/5, by its odd series to s^9 (the first term left out is below 1e-8 of
// the sum): one path for both, where a branch on u took the series and the fast
// logarithm in every warp.  The angle 2 pi u2 is taken as pi t with the signed
// t = 2 u2 (mod 2) in [-1, 1), so the fast sine and cosine see |pi t| <= pi,
// where their absolute error is below 2^-21.4.
__device__ __forceinline__ void box_muller(const uint32_t (&o)[4], float& z0, float& z1) {
  const uint32_t flip = o[0] >= 0xc0000000u ? 0xffffffffu : 0u;
  // u, or 1 - u where u >= 3/4
  const float q = fmaf((float)(o[0] ^ flip), 0x1p-32f, ((float)((o[1] ^ flip) >> 12) + 0.5f) * 0x1p-52f);
  const int bits = __float_as_int(q);
  const int e = (bits - 0x3f400000) >> 23;                  // q = m 2^e, m in [3/4, 3/2)
  const float mm = __int_as_float(bits - (e << 23)) - 1.0f;
  const float t1 = flip ? -q : mm, fe = flip ? 0.0f : (float)e;
  const float s = __fdividef(t1, 2.0f + t1), s2 = s * s;
  float p = 2.0f / 9.0f;
  p = fmaf(p, s2, 2.0f / 7.0f);
  p = fmaf(p, s2, 2.0f / 5.0f);
  p = fmaf(p, s2, 2.0f / 3.0f);
  p = fmaf(p, s2, 2.0f);
  // -2 ln u
  const float r = sqrtf(-2.0f * fmaf(fe, 0.693147180559945f, s * p));
  const float t = fmaf((float)(int32_t)o[2], 0x1p-31f, ((float)(o[3] >> 12) + 0.5f) * 0x1p-51f);
  float sn, cs;
  __sincosf(3.14159265358979f * t, &sn, &cs);
  z0 = r * cs;
  z1 = r * sn;
}
template <typename Key>
__device__ __forceinline__ void philox_normal2_f32(const Key& key, uint32_t c0, uint32_t c1, uint64_t step, float& z0,
                                                   float& z1) {
  uint32_t o[4];
  if constexpr (sizeof(Key) == sizeof(PhiloxKeys))
    philox4x32_10(c0, c1, (uint32_t)step, (uint32_t)(step >> 32), key, o);
  else
    philox4x32_10(c0, c1, (uint32_t)step, (uint32_t)(step >> 32), (uint32_t)key, (uint32_t)(key >> 32), o);
  box_muller(o, z0, z1);
}

// ---------------------------------------------------------------- Peskin
// phi(r) of cuda/SELM_Kernel.cu:391-395 for r = |distance| (grid units)
template <typename T> __device__ __forceinline__ T peskin4(T r) {
  if (r < T(1)) return (T(3) - T(2) * r + sqrt(T(1) + T(4) * r * (T(1) - r))) / T(8);
  if (r < T(2)) return (T(5) - T(2) * r - sqrt(T(-7) + T(4) * r * (T(3) - r))) / T(8);
  return T(0);
}

// p mod n in [0, n).  Arguments within one period of [0, n) (stencil and
// neighbour-cell offsets of in-box positions) take two compares; the integer
// division only runs for the rest.
__device__ __forceinline__ int wrapi(int p, int n) {
  int q = p < 0 ? p + n : (p >= n ? p - n : p);
  if ((unsigned)q >= (unsigned)n) {
    q = p % n;
    if (q < 0) q += n;
  }
  return q;
}

// ---------------------------------------------------------------- FFT plans
// Radix schedule of a line FFT (same factorisation order as the oracle:
// 4 first, then 2, 3, 5, 7, larger odd primes).
struct FftRadix {
  int n;
  int nstage;
  int radix[12];
};

inline FftRadix make_radix(int n) {
  FftRadix r{};
  r.n = n;
  int m = n, ns = 0;
  while (m > 1 && ns < 12) {
    int p;
    if (m % 4 == 0) p = 4;
    else if (m % 2 == 0) p = 2;
    else if (m % 3 == 0) p = 3;
    else if (m % 5 == 0) p = 5;
    else { p = 7; while (m % p) p += 2; }
    r.radix[ns++] = p;
    m /= p;
  }
  r.nstage = ns;
  return r;
}

// One Stockham decimation-in-time stage for many lines held in shared memory.
// Element t of line b lives at  b*sb + t*st  (sb, st in elements).
//   Y[k][q + Ls v] = sum_s w_p^{s v} ( w_L^{s q} Y*[k + s r][q] )
// Y* (input) at  q*rs + k  ,  Y (output) at  q*r + k ,  L = p*Ls, r = n/L.
// w[t] = exp(sign*2*pi*i*t/n) for t < n.
template <typename C>
__device__ __forceinline__ void stockham_stage(const C* __restrict__ a, C* __restrict__ b, const C* __restrict__ w,
                                               int n, int p, int Ls, int nlines, int sb, int st, bool line_fast,
                                               int sign, int tid, int nthr) {
  using T = decltype(C::x);
  const int L = Ls * p, r = n / L, rs = n / Ls;
  const int nbf = nlines * r * Ls;  // butterflies
  if (p > 8) {
    // primes 11..61, a p-point DFT: an item per output, its two twiddles one
    // power w^(s (q r + v n/p)); bound by the shared-memory reads of the terms.
    // A thread per butterfly, with two products and a remainder a term, was one
    // chain of p^2 terms on few threads: the step at 34^3 282 -> 104 us FP32,
    // 61^3 2636 -> 207 FP32, 6809 -> 233 FP64 and 2920 -> 282 plain, 122^3
    // 11510 -> 1095 FP32 and 46070 -> 1510 FP64.
    const int np = n / p;
    for (int it = tid; it < nbf * p; it += nthr) {
      const int v = it / nbf, bf = it - v * nbf;
      int line, k, q;
      if (line_fast) {
        line = bf % nlines;
        const int rest = bf / nlines;
        k = rest % r;
        q = rest / r;
      } else {
        k = bf % r;
        const int rest = bf / r;
        q = rest % Ls;
        line = rest / Ls;
      }
      const C* y = a + line * sb + (q * rs + k) * st;
      const int step = q * r + v * np, ys = r * st;
      C acc = y[0];
      int e = 0;
#pragma unroll 4
      for (int s = 1; s < p; s++) {
        e += step;
        if (e >= n) e -= n;
        const C t = y[s * ys], z = w[e];
        acc.x += t.x * z.x - t.y * z.y;
        acc.y += t.x * z.y + t.y * z.x;
      }
      b[line * sb + ((q + v * Ls) * r + k) * st] = acc;
    }
    return;
  }
  for (int it = tid; it < nbf; it += nthr) {
    int line, k, q;
    if (line_fast) {
      line = it % nlines;
      const int rest = it / nlines;
      k = rest % r;
      q = rest / r;
    } else {
      k = it % r;
      const int rest = it / r;
      q = rest % Ls;
      line = rest / Ls;
    }
    const C* ai = a + line * sb;
    C* bo = b + line * sb;
    C c[8];
#pragma unroll 1
    for (int s = 0; s < p; s++) {
      C y = ai[(q * rs + k + s * r) * st];
      c[s] = (s == 0 || q == 0) ? y : cmul(y, w[s * q * r]);
    }
    if (p == 4) {
      const C s02p = cadd(c[0], c[2]), s02m = csub(c[0], c[2]);
      const C s13p = cadd(c[1], c[3]), s13m = csub(c[1], c[3]);
      const C js = cmk<C>(-T(sign) * s13m.y, T(sign) * s13m.x);
      bo[(q * r + k) * st] = cadd(s02p, s13p);
      bo[((q + Ls) * r + k) * st] = cadd(s02m, js);
      bo[((q + 2 * Ls) * r + k) * st] = csub(s02p, s13p);
      bo[((q + 3 * Ls) * r + k) * st] = csub(s02m, js);
    } else if (p == 2) {
      bo[(q * r + k) * st] = cadd(c[0], c[1]);
      bo[((q + Ls) * r + k) * st] = csub(c[0], c[1]);
    } else {
      const int np = n / p;
      for (int v = 0; v < p; v++) {
        C acc = c[0];
        for (int s = 1; s < p; s++) acc = cadd(acc, cmul(c[s], w[((s * v) % p) * np]));
        bo[((q + v * Ls) * r + k) * st] = acc;
      }
    }
  }
}

// Full line FFT over all stages; ping-pongs between bufA and bufB and returns
// the buffer that holds the result.  Caller synchronises before the call.
template <typename C>
__device__ C* line_fft(C* bufA, C* bufB, const C* w, const FftRadix& R, int nlines, int sb, int st,
                       bool line_fast, int sign) {
  C* a = bufA;
  C* b = bufB;
  int Ls = 1;
  for (int s = 0; s < R.nstage; s++) {
    stockham_stage(a, b, w, R.n, R.radix[s], Ls, nlines, sb, st, line_fast, sign, threadIdx.x, blockDim.x);
    __syncthreads();
    C* t = a; a = b; b = t;
    Ls *= R.radix[s];
  }
  return a;
}

}  // namespace selm
