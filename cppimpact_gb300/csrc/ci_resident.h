// ci_resident.h -- the resident form of the fused step: see ci_resident.cuh.
#pragma once
#include <cuda_runtime.h>

#include <cstdint>
#include <vector>

#include "ci_kernels.cuh"
#include "ci_plan.h"

namespace ci {

struct ResidentArgs {
  DevPlan P;
  double* u[3];  // the complete state, read at the start and written at the end
  double* v[3];
  float4* halo[2];  // [S] partial force and step tag per slot, one buffer per step parity
  const float* mass;
  const double* d0;
  const float* d0f;
  unsigned char* contact;
  float* acc[3];
  float4* sig_a;
  float2* sig_b;
  float* epbar;
  double* chunk_work;
  unsigned int* status;
  const ResidentChunk* rchunk;  // [chunks] parts of the tables below
  const uint32_t* node_ent;     // [Lt] begin | count << 16 of a local node's entries in ent
  const uint16_t* ent;          // [npe E] corner * elements + element, by chunk and node
  const int* slots;             // every slot of a chunk's boundary nodes, by node
  const uint32_t* node_slots;   // [Lt] begin | count << 16 of a boundary node's part of them
  int* abort_flag;
  unsigned long long wait_ns;  // a wait gives up after this long
  int stall_chunk;             // test hook, single solves: this chunk leaves at once (-1: none)
  unsigned tag0;               // step k of the launch carries the tag tag0 + k
  int nsteps;                  // steps of this launch (batches: at most)
  ElemParams ep;
  NodeParams np;
  // batches: per-instance parameters and step counts, the steps done before this launch,
  // the order in which CTAs take chunks and its counter, and the snapshots
  const ElemParams* inst_ep;
  const NodeParams* inst_np;
  const int* inst_nsteps;
  const int* order;
  int* claim;
  int n_chunks;
  int step0;
  // snapshot s is the state after (s + 1) every steps; this launch writes those below
  // snap_end that earlier ones have not (0: no snapshots)
  int every, snap_end, snap_nodes;
  float* snap;  // [][snap_nodes][3], or null
  float* peak;  // [instances] largest snapshot displacement, or null
};

// The kernel that runs a plan resident: threads per chunk, shared bytes and CTAs held.
struct ResidentPick {
  const void* kernel = nullptr;
  int threads = 0;
  size_t smem = 0;
  int ctas = 0;  // co-resident on the whole GPU
};

// Bytes of the buffer that holds the element forces, then the received slots.
__host__ __device__ constexpr size_t resident_exchange(int npe, int ne, int ns) {
  const size_t f = 16 * (size_t)(npe * ne), r = 12 * (size_t)ns;
  return ((f > r ? f : r) + 15) & ~(size_t)15;
}

// Shared bytes of a chunk of `nl` local nodes, `ne` elements and `ns` boundary slots.
__host__ __device__ constexpr size_t resident_smem(int npe, int nl, int ne, int ns) {
  const int nq = npe == 4 ? 1 : 4;
  return 121 * (size_t)nl + 28 * (size_t)(nq * ne) + 4 * (size_t)(npe * ne) + 4 * (size_t)ns +
         resident_exchange(npe, ne, ns) + 64;
}

// Threads of the kernel for chunks of at most `elements` elements.  A single solve has SMs to
// spare and wants a warp for the elements beside one for the nodes; a batch wants as many
// chunks on an SM as it can get.  us per instance and step, 16 equal cubes: tet4 of 16 elements
// per chunk 0.86 with 32 threads, 1.19 with 64; 28 and 41 elements 1.73 and 2.02 with 64, 1.92
// and 2.10 with 32; tet10 of 16 and 18 elements 2.2 and 4.4 with 64 threads, 5.5 and 5.7 with
// 128; 28 and 41 elements 6.4 and 6.8 with 128, 9.6 and 11.6 with 64 (a launch per step of all
// 16: tet4 2.81, 4.73, 5.30, tet10 3.24, 5.52, 6.84, 8.34).
int resident_threads(int npe, bool batch, int elements);

// Picks the kernel for `chunks`; `energy_threads`: the fused kernel's CTA size whose work sums
// have to come out the same (0: the sums are not read).  No kernel if the chunks do not fit or
// `need_ctas` of them cannot be on the GPU together.
cudaError_t pick_resident(int npe, bool refcompat, bool batch, const std::vector<ChunkInfo>& chunks,
                          const std::vector<ResidentChunk>& rchunks, int energy_threads,
                          int need_ctas, int device, ResidentPick* out);

}  // namespace ci
