// The trajectory kernel for programs with segments (trajectory.cuh says why it is a
// translation unit of its own).
#include "trajectory.cuh"

namespace {

__global__ void __launch_bounds__(kTMinThreads, 1)
    k_trajectories_seg(const TOp *__restrict__ ops, uint32_t n_ops, const float2 *__restrict__ pool,
                       float2 *__restrict__ ws, uint32_t n, const TRun *__restrict__ run,
                       double *__restrict__ out_z, uint32_t *__restrict__ out_sample,
                       const __grid_constant__ TSegs segs) {
  extern __shared__ __align__(16) unsigned char seg_smem[];
  trajectories<kTMinThreads, true>(ops, n_ops, pool, ws, n, run, out_z, out_sample, segs, seg_smem);
}

// Shared memory of the largest launch: a full pass of 4-qubit gates and two tiles of
// the largest size.  The limit is the kernel's, shared by every program of the
// process: set to what one program needs, it would fall under the launch of another
// that a second thread is making.
constexpr size_t kSegSmemMost =
    cb2::kMaxPassGates * cb2::kPass32MatBytes + kSegArgBytes + (sizeof(float2) << (1 + kSegMaxTile));
static_assert(kSegSmemMost + sizeof(Shared) + (sizeof(float2) << (2 * kTrajMaxGate)) +
                      sizeof(double) * kTMinThreads <= 227 * 1024,
              "fits a CTA beside the static arrays");

}  // namespace

namespace cb2 {

cudaError_t launch_trajectory_segments(unsigned grid, cudaStream_t s, const void *ops, uint32_t n_ops,
                                       const float2 *pool, float2 *ws, uint32_t n, const void *run,
                                       double *z, uint32_t *sample, const void *segs) {
  const TSegs &g = *static_cast<const TSegs *>(segs);
  const size_t smem = g.mat_cap + kSegArgBytes + (sizeof(float2) << (1 + std::min(n, kSegMaxTile)));
  const cudaError_t rc =
      cudaFuncSetAttribute(k_trajectories_seg, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSegSmemMost);
  if (rc != cudaSuccess) return rc;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(grid);
  cfg.blockDim = dim3(kTMinThreads);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = s;
  return cudaLaunchKernelEx(&cfg, k_trajectories_seg, static_cast<const TOp *>(ops), n_ops, pool, ws, n,
                            static_cast<const TRun *>(run), z, sample, g);
}

}  // namespace cb2
