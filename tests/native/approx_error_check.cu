// Test program: the hardware approximations under hfa::recip_rn and
// hfa::sqrt_rn_moderate are as good as their error arguments take them to be.
// Over every high word of [1, 2) (reciprocal) and [1, 4) (root), with the low
// word zero, all ones and random: |1 - b y| below 2^-19.67, so that its cube is
// below 2^-59, and |1 - x y^2| at most 2^-19. Prints both maxima as powers of
// two; exits 1 beyond a bound.
#include <cmath>
#include <cstdio>

#include <cuda_runtime.h>

__device__ unsigned long long mix(unsigned long long x) {  // splitmix64
  x += 0x9E3779B97F4A7C15ull;
  x = (x ^ (x >> 30)) * 0xBF58476D1CE4E5B9ull;
  x = (x ^ (x >> 27)) * 0x94D049BB133111EBull;
  return x ^ (x >> 31);
}

// worst[0], worst[1]: bits of the largest errors (non-negative doubles order
// as their bits).
__global__ void k_errors(unsigned long long* worst) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;  // high word 0x3ff00000 + i
  double e0 = 0.0, e1 = 0.0;
  for (int k = 0; k < 18; ++k) {
    const unsigned lo = k == 0 ? 0u : k == 1 ? 0xffffffffu : (unsigned)mix(18ull * i + k);
    const double b = __hiloint2double(0x3ff00000 + i, (int)lo);
    double y;
    if (i < 1 << 20) {
      asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(b));
      e0 = fmax(e0, fabs(fma(-b, y, 1.0)));
    }
    asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(b));
    e1 = fmax(e1, fabs(fma(-b * y, y, 1.0)));
  }
  atomicMax(&worst[0], (unsigned long long)__double_as_longlong(e0));
  atomicMax(&worst[1], (unsigned long long)__double_as_longlong(e1));
}

int main() {
  unsigned long long* d = nullptr;
  double h[2];
  if (cudaMalloc(&d, sizeof h) != cudaSuccess) return 2;
  cudaMemset(d, 0, sizeof h);
  k_errors<<<(1 << 21) / 256, 256>>>(d);
  if (cudaMemcpy(h, d, sizeof h, cudaMemcpyDeviceToHost) != cudaSuccess) return 2;
  printf("reciprocal 2^%.2f, root 2^%.2f\n", std::log2(h[0]), std::log2(h[1]));
  return !(h[0] < std::exp2(-19.67) && h[1] <= std::exp2(-19.0));
}
