// Test kernels over the spectral update's draws (built by test_draws_gpu.py).
#include "../monomers2026_b200/csrc/fluid_fused_fast.cuh"

using namespace selm;

namespace {
__global__ void k_words(PhiloxKeys rk, uint32_t q, uint64_t step0, int steps, uint32_t* out) {
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= 3 * steps) return;
  uint32_t o[4];
  const uint64_t step = step0 + t / 3;
  philox4x32_10(q, (uint32_t)(t % 3), (uint32_t)step, (uint32_t)(step >> 32), rk, o);
  for (int i = 0; i < 4; i++) out[4 * t + i] = o[i];
}

// The update of mode (0, 0, k) of an n^3 grid of unit cells at rest, rho = 1,
// without forcing: its first two components are the draw itself.
__global__ void k_mode(ZGeom g, int n, int k, uint64_t step0, int steps, float2* out) {
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= steps) return;
  const ColSym<float> col{0.0, make_float2(0.0f, 0.0f), make_float2(0.0f, 0.0f), 0, 0};
  const double h = sin(kPi * k / n);
  const PlaneSym<float> pz{-2.0 * h * h, make_float2((float)(-2.0 * h * h), (float)sin(2.0 * kPi * k / n))};
  const ModeConsts<float> mc{step0 + (uint64_t)t, 1.0, 0.0, 1.0f, 1.0f};
  float2 uh[3] = {}, a[3] = {};
  mode_update<float, true>(g, mc, n, col, pz, k, uh, 1, a, 1);
  for (int c = 0; c < 3; c++) out[3 * t + c] = uh[c];
}

__global__ void k_normals(int fp32, int n, const uint32_t* words, double* z) {
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= n) return;
  const uint32_t o[4] = {words[4 * t], words[4 * t + 1], words[4 * t + 2], words[4 * t + 3]};
  if (fp32) {
    float a, b;
    box_muller(o, a, b);
    z[2 * t] = a;
    z[2 * t + 1] = b;
  } else {
    box_muller(o, z[2 * t], z[2 * t + 1]);
  }
}

// f(device copy of out) and the result back
template <typename F> int with_output(void* out, size_t bytes, F&& f) {
  void* d = nullptr;
  cudaError_t e = cudaMalloc(&d, bytes);
  if (e != cudaSuccess) return (int)e;
  f(d);
  e = cudaGetLastError();
  if (e == cudaSuccess) e = cudaMemcpy(out, d, bytes, cudaMemcpyDeviceToHost);
  cudaFree(d);
  return (int)e;
}
}  // namespace

// the Philox words of a mode's three components, [steps][3][4]
extern "C" int probe_words(unsigned long long seed, unsigned q, unsigned long long step0, int steps, uint32_t* out) {
  return with_output(out, sizeof(uint32_t) * 12 * (size_t)steps, [&](void* d) {
    k_words<<<(3 * steps + 255) / 256, 256>>>(philox_keys(seed), q, step0, steps, (uint32_t*)d);
  });
}

// u_hat of mode (0, 0, k), [steps][3] complex
extern "C" int probe_mode(int n, int k, unsigned long long seed, unsigned long long step0, int steps, double amp,
                          int exact, float* out) {
  ZGeom g{};
  g.nx = g.ny = n;
  g.nxh = n / 2 + 1;
  g.dx = g.rho = 1.0;
  g.noise_amp = amp;
  g.stochastic = 1;
  g.noise_mode = exact;
  g.rk = philox_keys(seed);
  return with_output(out, sizeof(float) * 6 * (size_t)steps, [&](void* d) {
    k_mode<<<(steps + 255) / 256, 256>>>(g, n, k, step0, steps, (float2*)d);
  });
}

// the pairs of normals of given Philox words [n][4], z [n][2]
extern "C" int probe_normals(int fp32, int n, const uint32_t* words, double* z) {
  uint32_t* w = nullptr;
  cudaError_t e = cudaMalloc(&w, sizeof(uint32_t) * 4 * (size_t)n);
  if (e != cudaSuccess) return (int)e;
  e = cudaMemcpy(w, words, sizeof(uint32_t) * 4 * (size_t)n, cudaMemcpyHostToDevice);
  int rc = (int)e;
  if (e == cudaSuccess)
    rc = with_output(z, sizeof(double) * 2 * (size_t)n,
                     [&](void* d) { k_normals<<<(n + 255) / 256, 256>>>(fp32, n, w, (double*)d); });
  cudaFree(w);
  return rc;
}
