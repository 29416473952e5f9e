// Test program: the unguarded arithmetic of moderate tiles against the IEEE
// operations, bit for bit, on the GPU. Prints one line per batch and exits 1
// on any mismatch.
//   hfa::recip_rn, quo_keep, quo_plus, sqrt_rn_moderate on random operands, on
//   significands within 64 ulp of a power of two, on zeros of both signs, and
//   the square root on every significand whose root lies next to the middle
//   of two numbers (x = n (n + 1) - c for an even |c| <= 4);
//   hf::wb_face_wet against hf::wb_face on random faces, both directions of
//   flow, deep to nearly dry, level and with jumps.
#include <cstdio>
#include <vector>

#include <cuda_runtime.h>

#include "../../hydroflux_b200/csrc/hf_device.cuh"

using namespace hf;

__device__ __forceinline__ unsigned long long mix(unsigned long long x) {
  x += 0x9E3779B97F4A7C15ull;
  x = (x ^ (x >> 30)) * 0xBF58476D1CE4E5B9ull;
  x = (x ^ (x >> 27)) * 0x94D049BB133111EBull;
  return x ^ (x >> 31);
}
__device__ __forceinline__ bool same(double x, double y) {
  return __double_as_longlong(x) == __double_as_longlong(y);
}
__device__ __forceinline__ double unit(unsigned long long k) {
  return (mix(k) >> 11) * (1.0 / 9007199254740992.0);
}
// A number with an exponent in [lo, hi]; `near`: a significand within 64 ulp
// of a power of two.
__device__ double number(unsigned long long k, int lo, int hi, bool near) {
  const unsigned long long r = mix(k), e = 1023 + lo + mix(k ^ 0x5bd1e995u) % (hi - lo + 1);
  unsigned long long m = r >> 12;
  if (near) m = (r & 1) ? 0xfffffffffffffull - (m & 63) : (m & 63);
  return __longlong_as_double((long long)((e << 52) | m));
}

__global__ void k_ops(unsigned long long seed, long long n, bool near, unsigned long long* bad) {
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n;
       i += (long long)gridDim.x * blockDim.x) {
    const unsigned long long k = seed * 0x1000003ull + 4ull * i;
    const double b = number(k, -60, 60, near);
    double a = number(k + 1, -200, 99, near && (mix(k + 3) & 2));
    const unsigned long long s = mix(k + 2);
    if (s & 1) a = -a;
    if ((s >> 8) % 16 == 0) a = (s & 1) ? -0.0 : 0.0;
    if (!hfa::low_word_ones(b)) {
      const double y = hfa::recip_rn(b), yn = hfa::recip_rn(-b);
      if (!same(y, 1.0 / b)) atomicAdd(&bad[0], 1ull);
      if (!same(hfa::quo_keep(a, b, y), a / b)) atomicAdd(&bad[1], 1ull);
      if (!same(hfa::quo_plus(a, -b, yn), a / -b)) atomicAdd(&bad[2], 1ull);
      const double q = a / b;
      if (!same(hfa::quo_plus(a, b, y), q == 0.0 ? 0.0 : q)) atomicAdd(&bad[2], 1ull);
    }
    if (!same(hfa::sqrt_rn_moderate(b), sqrt(b))) atomicAdd(&bad[3], 1ull);
  }
}

__global__ void k_roots(const double* x, int n, unsigned long long* bad) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  for (int e = -100; e <= 100; e += 2) {
    const double v = ldexp(x[i], e);
    if (!same(hfa::sqrt_rn_moderate(v), sqrt(v))) atomicAdd(bad, 1ull);
  }
}

__global__ void k_faces(long long n, unsigned long long* bad) {
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n;
       i += (long long)gridDim.x * blockDim.x) {
    const unsigned long long k = 16ull * i;
    double hL = exp2(-18.0 + 22.0 * unit(k)), hR = exp2(-18.0 + 22.0 * unit(k + 1));
    const double z = (i & 4) ? 0.0 : 300.0 * unit(k + 2);
    const double scale = exp2(-30.0 + 34.0 * unit(k + 7));
    double a = scale * (2.0 * unit(k + 3) - 1.0), b = 2.0 * unit(k + 4) - 1.0;
    double c = scale * (2.0 * unit(k + 5) - 1.0), d = 2.0 * unit(k + 6) - 1.0;
    if (i & 1) hR = hL;
    if (i & 2) { c = a; d = 0.0; b = -0.0; }
    if (i % 64 == 8) { a = 0.0; c = 0.0; }
    FaceFlux f, g;
    if (!wb_face_wet(hL, a, b, hR, c, d, z, f)) {
      atomicAdd(&bad[1], 1ull);
      continue;
    }
    wb_face<double>(hL, hL * a, hL * b, hR, hR * c, hR * d, z, g.mass, g.n_minus, g.n_plus, g.tang);
    if (!same(f.mass, g.mass) || !same(f.n_minus, g.n_minus) || !same(f.n_plus, g.n_plus) ||
        !same(f.tang, g.tang))
      atomicAdd(&bad[0], 1ull);
  }
}

// x = n (n + 1) - c with 53 significant bits, by lifting the roots of
// n^2 + n - c modulo 2^bits (its derivative is odd: one lift per root).
static std::vector<double> hard_roots() {
  std::vector<double> out;
  for (int bits = 52; bits <= 53; ++bits)
    for (int c = -4; c <= 4; c += 2)
      for (int r = 0; r < 2; ++r) {
        unsigned __int128 n = r;
        for (int j = 1; j < bits; ++j) {
          const unsigned __int128 m = (n * n + n - (unsigned __int128)(__int128)c);
          if ((m >> j) & 1) n += (unsigned __int128)1 << j;
        }
        for (; n < ((unsigned __int128)1 << 53); n += (unsigned __int128)1 << bits) {
          if (n < ((unsigned __int128)1 << 52)) continue;
          const unsigned __int128 X = (n * n + n - (unsigned __int128)(__int128)c) >> bits;
          if (X < ((unsigned __int128)1 << 52) || X >= ((unsigned __int128)1 << 53)) continue;
          out.push_back((double)(unsigned long long)X * (bits == 52 ? 1.0 : 2.0));
        }
      }
  return out;
}

int main(int argc, char** argv) {
  const long long n = argc > 1 ? atoll(argv[1]) : (1ll << 28);
  unsigned long long* bad = nullptr;
  if (cudaMalloc(&bad, 8 * sizeof(unsigned long long)) != cudaSuccess) return 2;
  unsigned long long h[4];
  int fails = 0;
  for (int near = 0; near < 2; ++near) {
    cudaMemset(bad, 0, 8 * sizeof(unsigned long long));
    k_ops<<<148 * 8, 256>>>(1 + near, n, near != 0, bad);
    if (cudaMemcpy(h, bad, sizeof h, cudaMemcpyDeviceToHost) != cudaSuccess) return 2;
    printf("%s: %lld operands; mismatches recip %llu, quo_keep %llu, quo_plus %llu, sqrt %llu\n",
           near ? "near powers of two" : "random", n, h[0], h[1], h[2], h[3]);
    fails += (h[0] || h[1] || h[2] || h[3]);
  }
  const std::vector<double> x = hard_roots();
  double* dx = nullptr;
  if (cudaMalloc(&dx, (x.size() + 1) * sizeof(double)) != cudaSuccess) return 2;
  cudaMemcpy(dx, x.data(), x.size() * sizeof(double), cudaMemcpyHostToDevice);
  cudaMemset(bad, 0, 8 * sizeof(unsigned long long));
  k_roots<<<1, 64>>>(dx, (int)x.size(), bad);
  if (cudaMemcpy(h, bad, sizeof h, cudaMemcpyDeviceToHost) != cudaSuccess) return 2;
  printf("hard roots: %zu significands; mismatches %llu\n", x.size(), h[0]);
  fails += h[0] != 0 || x.empty() || x.size() > 20;
  cudaMemset(bad, 0, 8 * sizeof(unsigned long long));
  k_faces<<<148 * 8, 256>>>(n / 16, bad);
  if (cudaMemcpy(h, bad, sizeof h, cudaMemcpyDeviceToHost) != cudaSuccess) return 2;
  printf("faces: %lld; mismatches %llu, left to the general face %llu\n", n / 16, h[0], h[1]);
  fails += h[0] != 0 || h[1] > (unsigned long long)(n / 16 / 4);
  return fails ? 1 : 0;
}
