// ci_resident10.cu -- resident step kernels of tet10 meshes (ci_resident.cuh).
#include "ci_resident.cuh"

namespace ci {

namespace {
template <int MODE, bool BATCH>
const void* pick(int threads) {
  if constexpr (BATCH)
    if (threads == 64) return resident_fn<10, MODE, 64, BATCH>();
  return threads == 128 ? resident_fn<10, MODE, 128, BATCH>() : nullptr;
}
}  // namespace

const void* resident_kernel_tet10(bool refcompat, bool batch, int threads) {
  if (batch) return refcompat ? nullptr : pick<EM_J2, true>(threads);
  return refcompat ? pick<EM_REFCOMPAT, false>(threads) : pick<EM_J2, false>(threads);
}

}  // namespace ci
