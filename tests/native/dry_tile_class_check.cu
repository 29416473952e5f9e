// Test program: a dry tile that holds a value outside the moderate range does
// not make the next tile of its CTA a general one. One CTA runs the stage of
// two interior tiles of one grid in turn: all dry with an infinite bed, then wet
// and moderate; it prints the class of each. Exits 1 unless they are dry and
// moderate (the other order, and a wet tile with the infinity: general).
#include <cstdio>
#include <cstring>
#include <vector>

#include <cuda_runtime.h>

#include "../../hydroflux_b200/csrc/hf_stage.cuh"

using namespace hf;

// Runs `tiles` of the grid in turn as k_stage_pf does; cls[k]: class of the k-th.
__global__ void __launch_bounds__(NTHREADS, HF_MIN_BLOCKS)
    k_tiles(const StageArgs A, int a, int b, int* cls) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  StagePfSmem& P = *reinterpret_cast<StagePfSmem*>(smem_raw);
  double sxm = 0.0, sym = 0.0;
  unsigned long long nonfin = 0;
  if (threadIdx.x == 0) {
    P.s.extreme = 0;
    stage_step_dt(A, P.s.dt);
  }
  for (int k = 0; k < 2; ++k) {
    const int tile = k == 0 ? a : b;
    stage_prefetch(A, P.s, P.hst, tile);
    cp_async_wait_all();
    __syncthreads();
    const TileClass c = stage_tile<double, true, true, true>(A, P.s, tile, sxm, sym, nonfin, P.hst);
    if (threadIdx.x == 0) cls[k] = c;
    __syncthreads();
  }
}

int main() {
  // Tiles (1, 1) and (1, 3) of 3 x 5 tiles are interior with apart halos.
  const int nr = 3 * TY, nc = 5 * TX, t0 = 5 + 1, t1 = 5 + 3;
  const size_t cells = (size_t)nr * nc;
  std::vector<double> h(cells, 0.0), z(cells, 0.5), zero(cells, 0.0);
  for (int i = 0; i < nr; ++i)
    for (int j = 3 * TX - 4; j < nc; ++j) h[(size_t)i * nc + j] = 1.0;
  double *d[9];
  for (double*& p : d)
    if (cudaMalloc(&p, cells * sizeof(double)) != cudaSuccess) return 2;
  Ctrl c;
  std::memset(&c, 0, sizeof c);
  c.dt = 0.01;
  c.active = 1;
  Ctrl* dc = nullptr;
  int *dcls = nullptr, cls[2];
  if (cudaMalloc(&dc, sizeof c) != cudaSuccess || cudaMalloc(&dcls, sizeof cls) != cudaSuccess)
    return 2;
  cudaMemcpy(dc, &c, sizeof c, cudaMemcpyHostToDevice);
  cudaFuncSetAttribute(k_tiles, cudaFuncAttributeMaxDynamicSharedMemorySize,
                       (int)sizeof(StagePfSmem));
  StageArgs a;
  std::memset(&a, 0, sizeof a);
  a.nr = nr;
  a.nc = nc;
  a.tiles_x = 5;
  a.tiles_y = 3;
  a.dx = a.dy = 1.0;
  a.rx = hfa::make_recip(a.dx);
  a.ry = hfa::make_recip(a.dy);
  a.ctrl = dc;
  a.z = d[0];
  a.in_h = d[1];
  a.in_hu = d[2];
  a.in_hv = d[3];
  a.un_h = d[1];
  a.un_hu = d[2];
  a.un_hv = d[3];
  a.out_h = d[4];
  a.out_hu = d[5];
  a.out_hv = d[6];
  a.n = d[7];
  cudaMemcpy(d[1], h.data(), cells * sizeof(double), cudaMemcpyHostToDevice);
  for (int k : {2, 3, 7}) cudaMemcpy(d[k], zero.data(), cells * sizeof(double), cudaMemcpyHostToDevice);
  int bad = 0;
  auto run = [&](int first, int second, int inf_tile, int want0, int want1) {
    std::vector<double> bed = z;
    if (inf_tile >= 0) bed[(size_t)(TY + 2) * nc + (inf_tile % 5) * TX + 7] = 1.0 / 0.0;
    cudaMemcpy(d[0], bed.data(), cells * sizeof(double), cudaMemcpyHostToDevice);
    k_tiles<<<1, NTHREADS, sizeof(StagePfSmem)>>>(a, first, second, dcls);
    if (cudaMemcpy(cls, dcls, sizeof cls, cudaMemcpyDeviceToHost) != cudaSuccess) return 2;
    printf("classes %d %d, expected %d %d\n", cls[0], cls[1], want0, want1);
    bad += cls[0] != want0 || cls[1] != want1;
    return 0;
  };
  if (run(t0, t1, -1, TILE_DRY, TILE_MODERATE) || run(t0, t1, t0, TILE_DRY, TILE_MODERATE) ||
      run(t1, t0, t0, TILE_MODERATE, TILE_DRY) || run(t1, t0, t1, TILE_GENERAL, TILE_DRY) ||
      run(t0, t1, t1, TILE_DRY, TILE_GENERAL))
    return 2;
  return bad != 0;
}
