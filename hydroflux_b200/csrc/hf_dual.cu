// hf_dual.cu -- the forward-mode tangent stage (T = DualD), compiled for two
// CTAs of the 32 x 8 tiles (112 KB of shared memory each):
// - 256 threads, two CTAs per SM (g8);
// - 512 threads, one CTA per SM (g8d): fewer passes per phase where tiles times
//   lanes leave SMs idle and a stage is the latency of one tile (64 x 64, 8
//   lanes, 128 CTAs: 84 -> 66 us a step). With more tiles than SMs two smaller
//   CTAs per SM overlap each other's barriers.
#include <cuda_runtime.h>

#include "hf_device.cuh"
#include "hf_internal.h"
#include "hf_stage.cuh"

namespace hf {
inline namespace HF_GEOM {

// One stage of one grid over a persistent tile loop. blockIdx.y is the tangent
// lane (vector mode); the CFL reduction and the clock belong to lane 0.
__global__ void __launch_bounds__(NTHREADS, HF_MIN_BLOCKS == 1 ? 1 : 2)
    k_stage_dual(const StageArgs A) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  StageSmemT<DualD>& S = *reinterpret_cast<StageSmemT<DualD>*>(smem_raw);
  if (!A.ctrl->active) return;
  const int ntiles = A.tiles_x * A.tiles_y;
  double sxm = 0.0, sym = 0.0;
  unsigned long long nonfin = 0;
  __shared__ __align__(16) unsigned char lane_raw[sizeof(StageArgs)];
  StageArgs& L = *reinterpret_cast<StageArgs*>(lane_raw);
  if (threadIdx.x == 0) {
    lane_args(A, blockIdx.y, L);
    stage_step_dt(A, S.dt);
  }
  __syncthreads();
  for (int tile = blockIdx.x; tile < ntiles; tile += gridDim.x) {
    if (interior_tile(L, tile))
      stage_tile<DualD, false, true>(L, S, tile, sxm, sym, nonfin);
    else
      stage_tile<DualD>(L, S, tile, sxm, sym, nonfin);
  }
  if (A.finalize && blockIdx.y == 0) {
    block_reduce_speeds(sxm, sym, nonfin, A.ctrl);
    if (blockIdx.x == 0 && threadIdx.x == 0) commit_clock(A.ctrl);
  }
}

namespace {
// CTAs resident per SM; raises the kernel's shared-memory limit on the current
// device.
int dual_prepare() {
  int per_sm = 0;
  cudaFuncSetAttribute(k_stage_dual, cudaFuncAttributeMaxDynamicSharedMemorySize,
                       (int)sizeof(StageSmemT<DualD>));
  // two 112 KB tiles per SM need the largest shared-memory carveout
  cudaFuncSetAttribute(k_stage_dual, cudaFuncAttributePreferredSharedMemoryCarveout,
                       (int)cudaSharedmemCarveoutMaxShared);
  cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_stage_dual, NTHREADS,
                                                sizeof(StageSmemT<DualD>));
  return per_sm < 1 ? 1 : per_sm;
}
}  // namespace
}  // namespace HF_GEOM

#if HF_GEOM_INDEX == 5
void dual_wide_prepare() { dual_prepare(); }
void launch_stage_dual_wide(const StageArgs& a, int grid, void* stream, int lanes) {
  k_stage_dual<<<dim3(grid, lanes), NTHREADS, sizeof(StageSmemT<DualD>), (cudaStream_t)stream>>>(a);
}
#else
inline namespace HF_GEOM {
int stage_dual_grid_size(int tiles, int device) {
  static int cached[64] = {0};
  int per_sm = 0, sms = 0;
  if (device >= 0 && device < 64 && cached[device] > 0) {
    per_sm = cached[device];
  } else {
    int prev = -1;
    cudaGetDevice(&prev);
    if (device >= 0 && prev != device) cudaSetDevice(device);
    per_sm = dual_prepare();
    dual_wide_prepare();
    if (prev >= 0 && prev != device) cudaSetDevice(prev);
    if (device >= 0 && device < 64) cached[device] = per_sm;
  }
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device);
  int g = per_sm * (sms > 0 ? sms : 148);
  return tiles < g ? (tiles < 1 ? 1 : tiles) : g;
}

// DualD (tangent) stage: value arrays in a.in_* / a.out_* / a.un_* / a.n,
// tangent arrays in a.tan. Grid from stage_dual_grid_size().
int launch_stage_dual(const StageArgs& a, int grid, void* stream, int lanes) {
  if ((int64_t)grid * lanes <= sm_count())
    launch_stage_dual_wide(a, grid, stream, lanes);
  else
    k_stage_dual<<<dim3(grid, lanes), NTHREADS, sizeof(StageSmemT<DualD>),
                   (cudaStream_t)stream>>>(a);
  return launched(stream);
}
}  // namespace HF_GEOM
#endif

}  // namespace hf
