// Instantiations and launch of resident_kernel (svs_resident.cuh) for every storage mode and shape.
#include "svs_resident.cuh"

namespace svs {
namespace {

template <typename SU, typename SP, typename C>
bool run(int op, unsigned grid, unsigned threads, const ResLaunch* L, const Desc* descs, const ResidentArgs* a,
         int* status, cudaStream_t s, int* occ) {
  const auto k = resident_kernel<SU, SP, C>;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(grid);
  cfg.blockDim = dim3(threads);
  cfg.dynamicSmemBytes = C::SMEM;
  cfg.stream = s;
  cudaLaunchAttribute attr;
  cfg.attrs = &attr;
  cfg.numAttrs = 1;
  if constexpr (C::CLUSTER) {
    attr.id = cudaLaunchAttributeClusterDimension;
    attr.val.clusterDim.x = op ? L->cluster : kResClusterBlocks;
    attr.val.clusterDim.y = attr.val.clusterDim.z = 1;
  } else {
    // its CTAs wait for one another: a cooperative launch starts only a grid that fits the GPU at once
    attr.id = cudaLaunchAttributeCooperative;
    attr.val.cooperative = 1;
  }
  if (op == 0) {
    bool ok = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, C::SMEM) == cudaSuccess;
    if constexpr (C::CLUSTER) {
      cfg.gridDim = dim3(kResClusterBlocks);
      cfg.blockDim = dim3(C::NT);
      ok = ok && cudaFuncSetAttribute(k, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) == cudaSuccess &&
           cudaOccupancyMaxActiveClusters(occ, k, &cfg) == cudaSuccess;
    } else {
      ok = ok && cudaOccupancyMaxActiveBlocksPerMultiprocessor(occ, k, C::NT, C::SMEM) == cudaSuccess;
    }
    if (!ok) cudaGetLastError();
    return ok && *occ > 0;
  }
  return cudaLaunchKernelEx(&cfg, k, *L, descs, *a, status) == cudaSuccess;
}

template <typename SU, typename SP>
bool dispatch(int shape, int op, unsigned grid, unsigned threads, const ResLaunch* L, const Desc* descs,
              const ResidentArgs* a, int* status, cudaStream_t s, int* occ) {
  switch (shape) {
    case 0: return run<SU, SP, ResSmall>(op, grid, threads, L, descs, a, status, s, occ);
    case 1: return run<SU, SP, ResMid>(op, grid, threads, L, descs, a, status, s, occ);
    case 2: return run<SU, SP, ResLarge<SP>>(op, grid, threads, L, descs, a, status, s, occ);
    case 3: return run<SU, SP, ResCluster>(op, grid, threads, L, descs, a, status, s, occ);
    default: return false;
  }
}

}  // namespace

bool resident_variant(int storage, int shape, int op, unsigned grid, unsigned threads, const ResLaunch* L,
                      const Desc* descs, const ResidentArgs* a, int* status, cudaStream_t s, int* occ) {
  switch (storage) {
    case SVS_STORAGE_BF16:
      return dispatch<__nv_bfloat16, __nv_bfloat16>(shape, op, grid, threads, L, descs, a, status, s, occ);
    case SVS_STORAGE_F16: return dispatch<__half, __half>(shape, op, grid, threads, L, descs, a, status, s, occ);
    case SVS_STORAGE_BF16_FLOW32:
      return dispatch<float, __nv_bfloat16>(shape, op, grid, threads, L, descs, a, status, s, occ);
    case SVS_STORAGE_F16_FLOW32: return dispatch<float, __half>(shape, op, grid, threads, L, descs, a, status, s, occ);
    default: return dispatch<float, float>(shape, op, grid, threads, L, descs, a, status, s, occ);
  }
}

}  // namespace svs
