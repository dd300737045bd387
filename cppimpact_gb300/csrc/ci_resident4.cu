// ci_resident4.cu -- resident step kernels of tet4 meshes (ci_resident.cuh).
#include <algorithm>

#include "ci_resident.cuh"

namespace ci {

namespace {
template <int MODE, bool BATCH>
const void* pick(int threads) {
  if constexpr (BATCH)
    if (threads == 32) return resident_fn<4, MODE, 32, BATCH>();
  if (threads == 64) return resident_fn<4, MODE, 64, BATCH>();
  return threads == 128 ? resident_fn<4, MODE, 128, BATCH>() : nullptr;
}
}  // namespace

const void* resident_kernel_tet4(bool refcompat, bool batch, int threads) {
  if (batch) return refcompat ? nullptr : pick<EM_J2, true>(threads);
  return refcompat ? pick<EM_REFCOMPAT, false>(threads) : pick<EM_J2, false>(threads);
}

}  // namespace ci

namespace ci {

const void* resident_kernel_tet10(bool refcompat, bool batch, int threads);

int resident_threads(int npe, bool batch, int elements) {
  if (npe == 10) return batch && elements <= 24 ? 64 : 128;
  if (!batch) return elements <= 32 ? 64 : 128;
  return elements <= 24 ? 32 : elements <= 64 ? 64 : 128;
}

cudaError_t pick_resident(int npe, bool refcompat, bool batch, const std::vector<ChunkInfo>& chunks,
                          const std::vector<ResidentChunk>& rchunks, int energy_threads,
                          int need_ctas, int device, ResidentPick* out) {
  *out = ResidentPick();
  int smem_max = 0, sms = 0, coop = 0;
  cudaError_t e;
  if ((e = cudaDeviceGetAttribute(&smem_max, cudaDevAttrMaxSharedMemoryPerBlockOptin, device)))
    return e;
  if ((e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device))) return e;
  if ((e = cudaDeviceGetAttribute(&coop, cudaDevAttrCooperativeLaunch, device))) return e;
  if (!coop) return cudaSuccess;
  int most = 0;
  for (const ChunkInfo& c : chunks) most = std::max(most, c.elem_end - c.elem_begin);
  const int threads = resident_threads(npe, batch, most);
  // the same work sums as the fused kernel's: its CTA size, or no thread of either with more
  // than one element or point (further warps only add zeros)
  if (energy_threads && threads != energy_threads &&
      (npe == 10 ? 4 : 1) * most > std::min(threads, energy_threads))
    return cudaSuccess;
  const void* fn = npe == 4 ? resident_kernel_tet4(refcompat, batch, threads)
                            : resident_kernel_tet10(refcompat, batch, threads);
  if (!fn) return cudaSuccess;
  size_t smem = 0;
  for (size_t i = 0; i < chunks.size(); i++) {
    const ChunkInfo& c = chunks[i];
    const int ne = c.elem_end - c.elem_begin, ns = rchunks[i].n_slots;
    if (npe * ne > 65535 || ns > 65535) return cudaSuccess;  // 16-bit positions
    smem = std::max(smem, resident_smem(npe, c.n_local, ne, ns));
  }
  if ((long long)smem + 2048 > smem_max) return cudaSuccess;
  // one limit for every solver (a smaller one set later would refuse this one's launch)
  if ((e = cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, smem_max - 2048)))
    return e;
  int per_sm = 0;
  if ((e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, fn, threads, smem))) return e;
  if ((long long)per_sm * sms < need_ctas) return cudaSuccess;
  out->kernel = fn;
  out->threads = threads;
  out->smem = smem;
  out->ctas = per_sm * sms;
  return cudaSuccess;
}

}  // namespace ci
