// The on-chip iterations with the test hook of their waits (ResShape::MUTE), for the two storage modes that
// the test runs. Its launches are not part of any solve without svs_tvl1_plan_set_mute_test.
#include "svs_resident.cuh"

namespace svs {
namespace {

template <typename SU, typename SP>
bool dispatch(int shape, unsigned grid, unsigned threads, const ResLaunch* L, const Desc* descs, const ResidentArgs* a,
              int* status, cudaStream_t s) {
  auto go = [&](auto run) {
    int occ = 0;
    return run(0, 0u, 0u, nullptr, nullptr, nullptr, nullptr, nullptr, &occ) &&
           run(1, grid, threads, L, descs, a, status, s, nullptr);
  };
  switch (shape) {
    case 0: return go(resident_run<SU, SP, ResSmall::WithMute>);
    case 1: return go(resident_run<SU, SP, ResMid::WithMute>);
    case 2: return go(resident_run<SU, SP, typename ResLarge<SP>::WithMute>);
    case 3: return go(resident_run<SU, SP, ResCluster::WithMute>);
    default: return false;
  }
}

}  // namespace

bool resident_mute(int storage, int shape, int op, unsigned grid, unsigned threads, const ResLaunch* L, const Desc* descs,
                   const ResidentArgs* a, int* status, cudaStream_t s, int* occ) {
  if (op != 1) return false;
  if (storage == SVS_STORAGE_F32) return dispatch<float, float>(shape, grid, threads, L, descs, a, status, s);
  if (storage == SVS_STORAGE_F16_FLOW32) return dispatch<float, __half>(shape, grid, threads, L, descs, a, status, s);
  return false;
}

}  // namespace svs
