// ci_resident10.cu -- resident step kernels of tet10 meshes (ci_resident.cuh).
#include "ci_resident.cuh"

namespace ci {

namespace {
template <int MODE, bool BATCH>
const void* pick(int threads, bool chip) {
  if constexpr (BATCH)
    if (threads == 64 && chip) return resident_fn<10, MODE, 64, true, BATCH>();
  if (threads == 128 && chip) return resident_fn<10, MODE, 128, true, BATCH>();
  if constexpr (BATCH)
    if (threads == 128) return resident_fn<10, MODE, 128, false, BATCH>();
  return nullptr;
}
}  // namespace

const void* resident_kernel_tet10(bool refcompat, bool batch, int threads, bool chip) {
  if (batch) return refcompat ? nullptr : pick<EM_J2, true>(threads, chip);
  return refcompat ? pick<EM_REFCOMPAT, false>(threads, chip) : pick<EM_J2, false>(threads, chip);
}

}  // namespace ci
