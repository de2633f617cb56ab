// Instantiations and launch of resident_kernel (svs_resident.cuh) for every storage mode and shape.
#include "svs_resident.cuh"

namespace svs {
namespace {

template <typename SU, typename SP>
bool dispatch(int shape, int op, unsigned grid, unsigned threads, const ResLaunch* L, const Desc* descs,
              const ResidentArgs* a, int* status, cudaStream_t s, int* occ) {
  switch (shape) {
    case 0: return resident_run<SU, SP, ResSmall>(op, grid, threads, L, descs, a, status, s, occ);
    case 1: return resident_run<SU, SP, ResMid>(op, grid, threads, L, descs, a, status, s, occ);
    case 2: return resident_run<SU, SP, ResLarge<SP>>(op, grid, threads, L, descs, a, status, s, occ);
    case 3: return resident_run<SU, SP, ResCluster>(op, grid, threads, L, descs, a, status, s, occ);
    default: return false;
  }
}

}  // namespace

bool resident_variant(int storage, int shape, int op, unsigned grid, unsigned threads, const ResLaunch* L,
                      const Desc* descs, const ResidentArgs* a, int* status, cudaStream_t s, int* occ) {
  if (a && a->mute >= 0) return resident_mute(storage, shape, op, grid, threads, L, descs, a, status, s, occ);
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
