// Test program: hf::wb_face_moderate (and hf::wb_face_wet where it accepts)
// against hf::wb_face on faces with one side or both dry, below a step of the
// bed, at or around the velocity and wetness thresholds, or deep; bit for bit,
// zeros of both signs among the velocities. Exits 1 on any mismatch.
#include <cstdio>
#include <cstdlib>

#include <cuda_runtime.h>

#include "../../hydroflux_b200/csrc/hf_device.cuh"

using namespace hf;

__device__ __forceinline__ unsigned long long mix(unsigned long long x) {
  x += 0x9E3779B97F4A7C15ull;
  x = (x ^ (x >> 30)) * 0xBF58476D1CE4E5B9ull;
  x = (x ^ (x >> 27)) * 0x94D049BB133111EBull;
  return x ^ (x >> 31);
}
__device__ __forceinline__ double unit(unsigned long long k) {
  return (mix(k) >> 11) * (1.0 / 9007199254740992.0);
}
__device__ double depth(unsigned long long k) {
  const double u = unit(k + 9);
  switch (mix(k) % 8) {
    case 0: return 0.0;
    case 1: return -u;
    case 2: return H_VEL * u;
    case 3: return 3.0 * DRY_TOL * u;
    case 4: return H_VEL * (1.0 + 1.0e-6 * (u - 0.5));
    case 5: return exp2(-60.0 + 60.0 * u);
    default: return exp2(-18.0 + 22.0 * u);
  }
}
__device__ __forceinline__ bool same(double x, double y) {
  return __double_as_longlong(x) == __double_as_longlong(y);
}
__device__ __forceinline__ bool same(const FaceFlux& a, const FaceFlux& b) {
  return same(a.mass, b.mass) && same(a.n_minus, b.n_minus) && same(a.n_plus, b.n_plus) &&
         same(a.tang, b.tang);
}

__global__ void k_faces(long long n, unsigned long long* bad) {
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n;
       i += (long long)gridDim.x * blockDim.x) {
    const unsigned long long k = 64ull * i;
    double hL = depth(k), hR = depth(k + 20);
    const double z = (i & 4) ? 0.0 : 300.0 * unit(k + 2);
    const double scale = exp2(-30.0 + 34.0 * unit(k + 7));
    double a = scale * (2.0 * unit(k + 3) - 1.0), b = 2.0 * unit(k + 4) - 1.0;
    double c = scale * (2.0 * unit(k + 5) - 1.0), d = 2.0 * unit(k + 6) - 1.0;
    if (i % 16 == 1) hR = hL;
    if (i & 2) { c = a; d = 0.0; b = -0.0; }
    if (i % 64 == 8) { a = 0.0; c = 0.0; }
    if (i % 64 == 9) { a = -0.0; b = -0.0; c = -0.0; d = -0.0; }
    const double l = fmax(hL, 0.0), r = fmax(hR, 0.0);
    FaceFlux g, w;
    wb_face<double>(l, l * a, l * b, r, r * c, r * d, z, g.mass, g.n_minus, g.n_plus, g.tang);
    if (!same(wb_face_moderate(hL, a, b, hR, c, d, z), g)) atomicAdd(&bad[0], 1ull);
    if (wb_face_wet(hL, a, b, hR, c, d, z, w) && !same(w, g)) atomicAdd(&bad[1], 1ull);
  }
}

int main(int argc, char** argv) {
  const long long n = argc > 1 ? atoll(argv[1]) : (1ll << 26);
  unsigned long long *bad = nullptr, h[2];
  if (cudaMalloc(&bad, sizeof h) != cudaSuccess) return 2;
  cudaMemset(bad, 0, sizeof h);
  k_faces<<<148 * 8, 256>>>(n, bad);
  if (cudaMemcpy(h, bad, sizeof h, cudaMemcpyDeviceToHost) != cudaSuccess) return 2;
  printf("faces: %lld; mismatches moderate %llu, wet %llu\n", n, h[0], h[1]);
  return h[0] || h[1];
}
