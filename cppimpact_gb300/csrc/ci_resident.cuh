// ci_resident.cuh -- the fused step with its chunks held on the SMs for all steps of a call.
//
// What bounds a mesh of up to a few chunks per SM is not memory or arithmetic but the chain
// launch -> chunk table -> node state -> elements -> halo -> launch boundary of every step.
// Here every chunk's CTA stays for all the steps of the call (a cooperative launch, so that
// all of them run at the same time): displacements and velocities of its local nodes stay
// in shared memory, and per step the only global traffic is the partial force of each
// boundary node to its slot and the slots of the boundary nodes back.
//
// Steps are not separated by a barrier over the grid.  A slot is written with the tag of
// its step as one 16-byte store (st.relaxed b128, single-copy atomic), and a reader polls
// the slot itself until the tag is there: one L2 round trip for the data and its signal.
// Two slot buffers by step parity suffice: a chunk writes step k + 2 of a slot only after
// it has read, at step k + 1, the slots of every chunk sharing that node, which those
// chunks wrote after they had read step k.  Every wait is bounded in time.
//
// Arithmetic, order of sums and rounding are the fused kernels' on the same plan (the same
// functions; a node's element contributions are added in colour order, which is the
// elements' order in the chunk), so the results are the same bits.  Per step and chunk:
//   0  positions of the next state and the wall's push (they need no forces), written to
//      the other of two record buffers, so other warps may do the elements meanwhile
//   1  element forces to a (corner, element) buffer in shared memory, from which each node
//      then adds its entries in element order (no barrier per colour, and an element may
//      name a node twice)
//   2  boundary nodes' partial forces to their slots; work sums
//   3  every slot of the boundary nodes polled into shared memory, sums in slot order,
//      velocities and increments
// Ghost nodes are updated by every chunk that holds them, to the same bits.
//
// us per step in 300-step calls, one launch per step before: 6,000 tet4 6.6 -> 3.5, 20,250
// tet4 7.6 -> 4.1, 162,000 tet4 14.5 -> 8.2, 6,000 tet10 7.0 -> 4.9, 34,992 tet10 12.6 -> 8.7.
// What is left at 6,000 tet4 (7,000 cycles): elements 1,500-2,500 (one warp's chain), slots
// there and back 1,500-3,000 (an L2 round trip is 800), partial and total sums 2,000,
// velocities 600 (an FP64 instruction takes a warp 64 cycles).  At 34,992 tet10 the node
// updates, which every holder of a boundary node repeats, weigh as much as the elements.
//
// Stored stress, connectivity, entry and slot lists are in shared memory too (121 B per local
// node, 112 B per tet4 and 312 B per tet10 element, 4 to 16 B per slot: up to about 58 tet10
// or 270 tet4 elements per chunk at four CTAs per SM).  Read through the caches instead,
// for larger chunks, they made it slower than a launch per step (48,000 tet10: 15.2 and 14.5).
#pragma once
#include "ci_resident.h"

namespace ci {

__device__ __forceinline__ unsigned long long res_pack(float a, float b) {
  return (unsigned long long)__float_as_uint(a) | ((unsigned long long)__float_as_uint(b) << 32);
}

__device__ __forceinline__ float4 ld_slot(const float4* p) {
  unsigned long long a, b;
  asm volatile(
      "{\n .reg .b128 t;\n ld.relaxed.gpu.global.b128 t, [%2];\n mov.b128 {%0, %1}, t;\n}"
      : "=l"(a), "=l"(b)
      : "l"(p)
      : "memory");
  return make_float4(__uint_as_float((unsigned)a), __uint_as_float((unsigned)(a >> 32)),
                     __uint_as_float((unsigned)b), __uint_as_float((unsigned)(b >> 32)));
}

__device__ __forceinline__ void st_slot(float4* p, float x, float y, float z, unsigned tag) {
  asm volatile(
      "{\n .reg .b128 t;\n mov.b128 t, {%1, %2};\n st.relaxed.gpu.global.b128 [%0], t;\n}" ::"l"(p),
      "l"(res_pack(x, y)), "l"(res_pack(z, __uint_as_float(tag)))
      : "memory");
}

template <int P>
__device__ __forceinline__ void res_sync() {
  if (P == 32)
    __syncwarp();
  else
    __syncthreads();
}

template <int P>
__device__ __forceinline__ bool res_sync_and(bool ok) {
  if (P == 32) return __all_sync(0xffffffffu, ok);
  return __syncthreads_and(ok) != 0;
}

// One failed poll: every 64th looks at the abort flag and the clock; false = give up, which
// the status word always tells: a chunk that leaves has stored nothing.
static __device__ __noinline__ bool res_patience(const ResidentArgs& A, unsigned spins,
                                          unsigned long long& t0) {
  if (spins >= 2) __nanosleep(32);
  if ((spins & 63u) != 63u) return true;
  if (!*(volatile int*)A.abort_flag) {
    const unsigned long long t = global_ns();
    if (t0 == 0) t0 = t;
    if (t - t0 <= A.wait_ns) return true;
  }
  report(A.status, ST_FLOW_TIMEOUT);
  atomicExch(A.abort_flag, 1);
  return false;
}

// The slots of step `tag` at halo[slot[k]], k < n, into recv [3][n]: U polled at once by
// each of the P threads, those that are not there yet again after a pause (the polls of
// the waiting chunks would otherwise take the load pipe from the working ones).
template <int P>
__device__ __forceinline__ bool res_receive(const ResidentArgs& A, const float4* halo,
                                            const int* slot, int n, unsigned tag, float* recv) {
  constexpr int U = 4;
  for (int k0 = threadIdx.x; k0 < n; k0 += U * P) {
    float4 h[U];
    const float4* p[U];
#pragma unroll
    for (int i = 0; i < U; i++) {
      p[i] = k0 + i * P < n ? halo + slot[k0 + i * P] : nullptr;
      h[i].w = __uint_as_float(tag);
    }
#pragma unroll
    for (int i = 0; i < U; i++)
      if (p[i]) h[i] = ld_slot(p[i]);
    unsigned spins = 0;
    unsigned long long t0 = 0;
    for (;;) {
      bool all = true;
#pragma unroll
      for (int i = 0; i < U; i++) all = all && __float_as_uint(h[i].w) == tag;
      if (all) break;
      if (!res_patience(A, spins++, t0)) return false;
#pragma unroll
      for (int i = 0; i < U; i++)
        if (__float_as_uint(h[i].w) != tag) h[i] = ld_slot(p[i]);
    }
#pragma unroll
    for (int i = 0; i < U; i++) {
      const int k = k0 + i * P;
      if (k < n) {
        recv[k] = h[i].x;
        recv[n + k] = h[i].y;
        recv[2 * n + k] = h[i].z;
      }
    }
  }
  return true;
}

struct ResidentParams {
  ElemParams ep;
  NodeParams np;
};

// A status bit: to the status word at once, or kept by the thread until it is done with its
// chunk.  Which of the two leaves the better code differs.  us per step with the elements' bit
// kept, the nodes', both, neither: 34,992 tet10 8.71, 8.95, 8.90, 8.74; 6,000 tet4 (CTAs of 64
// threads) 3.60, 3.52, 3.55, 3.56; 48,000 tet4 (128) 5.02, 4.96, 4.99, 4.89; mixed batch of 24 cubes
// both 81.1 ms, neither 83.2.
template <bool KEEP>
__device__ __forceinline__ void res_flag(unsigned* status, unsigned& bits, unsigned bit) {
  if (KEEP)
    bits |= bit;
  else
    report(status, bit);
}

// The chunk's stress and plastic strain in shared memory.
template <bool KEEP>
struct ResidentState {
  float4* sig_a;
  float2* sig_b;
  float* epbar;
  unsigned* status;
  unsigned* bits;
  __device__ __forceinline__ void flag(unsigned bit) const { res_flag<KEEP>(status, *bits, bit); }
  __device__ __forceinline__ void load(size_t q, float4& a, float2& b, float& e) const {
    a = sig_a[q];
    b = sig_b[q];
    e = epbar[q];
  }
  __device__ __forceinline__ void store(size_t q, float4 a, float2 b, float e) const {
    sig_a[q] = a;
    sig_b[q] = b;
    epbar[q] = e;
  }
};

template <int NPE, int MODE, int P, bool BATCH>
__device__ __forceinline__ bool res_chunk(const ResidentArgs& A, unsigned char* sm, int ci,
                                          float (*red)[2][P / 32], ResidentParams* par) {
  constexpr int NQ = Rule<NPE>::NQ;
  constexpr int LN = NPE == 10 ? 4 : 1;  // lanes per element
  constexpr int EPW = P / LN;            // elements per window
  constexpr int EU = NPE == 4 ? 8 : 4;   // a node's entries and slots loaded at once
  const int tid = threadIdx.x;
  if (!BATCH && ci == A.stall_chunk) return false;
  const ChunkInfo ch = A.P.chunks[ci];
  // an instance's parameters are read where they are used (a copy per thread would take some
  // thirty registers), a single solve's come as constants
  if (BATCH) {
    if (tid == 0) {
      par->ep = A.inst_ep[ch.inst];
      par->np = A.inst_np[ch.inst];
    }
    res_sync<P>();
  }
  const ElemParams& ep = BATCH ? par->ep : A.ep;
  const NodeParams& np = BATCH ? par->np : A.np;
  int n = A.nsteps;
  if (BATCH) n = max(0, min(n, A.inst_nsteps[ch.inst] - A.step0));
  const bool snaps = BATCH && A.snap_end > 0;
  if (BATCH && n == 0 && !snaps) return true;
  const int L = ch.n_local, ne = ch.elem_end - ch.elem_begin, E = A.P.E;
  const ResidentChunk rc = A.rchunk[ci];
  const int ns = rc.n_slots;

  // shared memory (see resident_smem)
  double* su = reinterpret_cast<double*>(sm);
  double* sv = su + 3 * L;
  // records, double-buffered by step parity: node_step's positions of S^{k+1} do not wait
  // for the elements of step k
  float4* const p0 = reinterpret_cast<float4*>(sv + 3 * L);  // [2][L]
  int4* const m1 = reinterpret_cast<int4*>(p0 + 2 * L);  // own slot, received slots, element entries, 1/m
  float4* const fbuf = reinterpret_cast<float4*>(m1 + L);  // [NPE][ne] element forces
  float* const recv = reinterpret_cast<float*>(fbuf);  // [3][ns] the boundary nodes' slots, in its place
  constexpr bool KEEP_E = BATCH || NPE == 10, KEEP_N = BATCH || (NPE == 4 && P == 64);  // res_flag
  unsigned bits = 0;
  ResidentState<KEEP_E> S;
  S.status = A.status;
  S.bits = &bits;
  S.sig_a = fbuf + resident_exchange(NPE, ne, ns) / 16;
  float2* const p1 = reinterpret_cast<float2*>(S.sig_a + NQ * ne);
  double* const sw = reinterpret_cast<double*>(p1 + 2 * L);  // the wall's push on a node in contact
  S.sig_b = reinterpret_cast<float2*>(sw + L);
  S.epbar = reinterpret_cast<float*>(S.sig_b + NQ * ne);
  int* const sslot = reinterpret_cast<int*>(S.epbar + NQ * ne);  // the boundary nodes' slots' ids
  uint16_t* const sconn = reinterpret_cast<uint16_t*>(sslot + ns);
  uint16_t* const sent = sconn + NPE * ne;
  unsigned char* const flags = reinterpret_cast<unsigned char*>(sent + NPE * ne);
  auto tile = [&](int parity) {
    Tile T;
    T.p0 = p0 + parity * L;
    T.p1 = p1 + parity * L;
    T.acc = nullptr;
    return T;
  };

  auto gid = [&](int l) { return l < ch.n_own ? ch.own_begin + l : A.P.local_gid[ch.local_begin + l]; };

  // ---- load the state S^0 and its records
  for (int l = tid; l < L; l += P) {
    const int lb = ch.local_begin + l, g = gid(l);
    float x0[3], uf[3], vf[3];
#pragma unroll
    for (int k = 0; k < 3; k++) {
      x0[k] = A.P.local_x0[k * (size_t)A.P.Lt + lb];
      const double u = A.u[k][g], v = A.v[k][g];
      su[k * L + l] = u;
      sv[k * L + l] = v;
      uf[k] = f64_to_f32(u);
      vf[k] = f64_to_f32(v);
    }
    store_record(tile(0), l, x0[0] + uf[0], x0[1] + uf[1], x0[2] + uf[2], ep.dt * vf[0],
                 ep.dt * vf[1], ep.dt * vf[2]);
    flags[l] = A.contact[g];
    m1[l] = make_int4(A.P.local_slot[lb], (int)A.node_slots[lb], (int)A.node_ent[lb],
                      __float_as_int(__frcp_rn(A.mass[g])));
  }
  for (int i = tid; i < ne; i += P)
#pragma unroll
    for (int a = 0; a < NPE; a++)
      sconn[a * ne + i] = A.P.conn_local[(size_t)a * E + ch.elem_begin + i];
  for (int i = tid; i < ns; i += P) sslot[i] = A.slots[rc.slot_begin + i];
  for (int i = tid; i < NPE * ne; i += P) sent[i] = A.ent[(size_t)NPE * ch.elem_begin + i];
  if (MODE == EM_J2)
    for (int i = tid; i < NQ * ne; i += P) {
      const size_t qi = (size_t)NQ * ch.elem_begin + i;
      S.sig_a[i] = A.sig_a[qi];
      S.sig_b[i] = A.sig_b[qi];
      S.epbar[i] = A.epbar[qi];
    }
  double w0 = 0.0, w1 = 0.0;  // thread 0: the chunk's running work sums
  if (tid == 0) {
    w0 = A.chunk_work[4 * (size_t)ci];
    w1 = A.chunk_work[4 * (size_t)ci + 1];
  }
  const int q = tid & (LN - 1);
  const Tet10QP t10 = tet10_qp(q);
  // the owned nodes' displacement as snapshot si (FP32) and its largest norm
  auto snapshot = [&](int si) {
    if (si >= A.snap_end) return;
    float m = 0.f;
    for (int l = tid; l < ch.n_own; l += P) {
      const float x = (float)su[l], y = (float)su[L + l], z = (float)su[2 * L + l];
      if (A.snap) {
        float* o = A.snap + ((size_t)si * A.snap_nodes + ch.own_begin + l) * 3;
        o[0] = x;
        o[1] = y;
        o[2] = z;
      }
      m = fmaxf(m, sqrtf(x * x + y * y + z * z));
    }
    // non-negative floats order like their bits
    if (A.peak) atomicMax(reinterpret_cast<int*>(A.peak) + ch.inst, __float_as_int(m));
  };
  // this chunk's partial force of local node l
  auto own_force = [&](int l) {
    const unsigned en = (unsigned)m1[l].z;
    const uint16_t* e = sent + (en & 0xffffu);
    const int c = (int)(en >> 16);
    float4 f = make_float4(0.f, 0.f, 0.f, 0.f);
    for (int j0 = 0; j0 < c; j0 += EU) {  // EU entries' loads at once, added in order
      float4 b[EU];
#pragma unroll
      for (int j = 0; j < EU; j++) b[j] = fbuf[e[min(j0 + j, c - 1)]];
#pragma unroll
      for (int j = 0; j < EU; j++)
        if (j0 + j < c) {
          f.x += b[j].x;
          f.y += b[j].y;
          f.z += b[j].z;
        }
    }
    return f;
  };
  // node_step's operations in two parts: the positions of S^{k+1} and the wall's push do
  // not depend on the forces of step k and come before (or, by other warps, beside) its
  // elements: about 600 cycles of FP64 latency, 1,600 more for a node in contact.
  // flags bit 0: in contact, with the push in sw.
  auto move = [&](const Tile& T, int l) {
    const int g = gid(l);
    const float d0f = A.d0f[g];
    float x0[3], uf[3];
#pragma unroll
    for (int c = 0; c < 3; c++) x0[c] = A.P.local_x0[c * (size_t)A.P.Lt + ch.local_begin + l];
    double un[3];
#pragma unroll
    for (int c = 0; c < 3; c++) {
      un[c] = __fma_rn(np.dt, sv[c * L + l], su[c * L + l]);
      uf[c] = f64_to_f32(un[c]);
      su[c * L + l] = un[c];
    }
    float* r = reinterpret_cast<float*>(T.p0 + l);
    r[0] = x0[0] + uf[0];
    r[2] = x0[1] + uf[1];
    T.p1[l].x = x0[2] + uf[2];
    unsigned char fl = flags[l] & 2;
    if (wall_near(np, d0f, uf)) {
      const double d = wall_distance(np, A.d0[g], un);
      if (d < 0.0) {
        fl = 3;
        sw[l] = wall_push(np, d, A.mass[g]);
      }
    }
    flags[l] = fl;
  };
  auto push = [&](const Tile& T, int l, bool last, float fx, float fy, float fz) {
    const float rm = __int_as_float(m1[l].w);
    float a[3] = {__fadd_rn(__fmul_rn(-fx, rm), np.gf[0]), __fadd_rn(__fmul_rn(-fy, rm), np.gf[1]),
                  __fadd_rn(__fmul_rn(-fz, rm), np.gf[2])};
    double ad[3] = {f32_to_f64(a[0]), f32_to_f64(a[1]), f32_to_f64(a[2])};
    if (flags[l] & 1) {
      const double w = sw[l];
#pragma unroll
      for (int c = 0; c < 3; c++) {
        ad[c] = __fma_rn(w, np.wall_n[c], ad[c]);
        a[c] = f64_to_f32(ad[c]);
      }
    }
    bool finite = true;
    float vf[3];
#pragma unroll
    for (int c = 0; c < 3; c++) {
      const double v = __fma_rn(np.dt, ad[c], sv[c * L + l]);
      sv[c * L + l] = v;
      vf[c] = f64_to_f32(v);
      finite = finite && isfinite(vf[c]);
    }
    float* r = reinterpret_cast<float*>(T.p0 + l);
    r[1] = ep.dt * vf[0];
    r[3] = ep.dt * vf[1];
    T.p1[l].y = ep.dt * vf[2];
    if (!finite) res_flag<KEEP_N>(A.status, bits, ST_NONFINITE);
    if (last && l < ch.n_own)
#pragma unroll
      for (int c = 0; c < 3; c++) A.acc[c][ch.own_begin + l] = a[c];
  };
  res_sync<P>();

  for (int k = 0; k < n; k++) {
    float wint = 0.f, wp = 0.f, vol = 0.f;
    const Tile T = tile(k & 1), Tn = tile((k & 1) ^ 1);  // records of S^k and S^{k+1}
    // nodes go to the threads from the last one down, elements from the first one up: in a
    // chunk that does not fill the CTA different warps have them
    const int nd = P - 1 - tid;
    for (int l = nd; l < L; l += P) move(Tn, l);
    // ---- 1: element forces
    for (int w = 0; w < ne; w += EPW) {
      const int i = w + tid / LN;
      const bool act = i < ne;
      const int ii = act ? i : 0;
      if (NPE == 10) {
        // a warp past the last element skips the window (its lanes have no part in the sums)
        if (w + (tid & ~31) / LN >= ne) break;
        int ln[10];
#pragma unroll
        for (int a = 0; a < 10; a++) ln[a] = sconn[a * ne + ii];
        const size_t qi = (size_t)ii * 4 + q;
        float4 s4 = make_float4(0.f, 0.f, 0.f, 0.f);
        float2 s2 = make_float2(0.f, 0.f);
        float ep0 = 0.f;
        if (MODE == EM_J2) {
          s4 = S.sig_a[qi];
          s2 = S.sig_b[qi];
          ep0 = S.epbar[qi];
        }
        float keep[3][3];
        auto work = [&](float h, float wd, float hp, float wdp) {
          wint = fmaf(h, wd, wint);
          if (MODE == EM_J2) wp = fmaf(hp, wdp, wp);
        };
        auto flag = [&](unsigned bit) { S.flag(bit); };
        qp10_point<MODE>(ep, t10, q, T, ln, act, s4, s2, ep0, flag, work, keep,
                         [&](float4 a4, float2 a2, float epn) {
                           S.sig_a[qi] = a4;
                           S.sig_b[qi] = a2;
                           S.epbar[qi] = epn;
                         });
        if (act) {
          fbuf[q * ne + i] = make_float4(keep[0][0], keep[0][1], keep[0][2], 0.f);
          fbuf[(q + 4) * ne + i] = make_float4(keep[1][0], keep[1][1], keep[1][2], 0.f);
          if (q < 2) fbuf[(q + 8) * ne + i] = make_float4(keep[2][0], keep[2][1], keep[2][2], 0.f);
        }
      } else {
        int ln[NPE];
        float f[NPE][3];
        if (act) {
          float x[NPE][3], du[NPE][3];
#pragma unroll
          for (int a = 0; a < NPE; a++) {
            ln[a] = sconn[a * ne + i];
            float2 pr[3];
            load_pairs(T, ln[a], pr);
#pragma unroll
            for (int c = 0; c < 3; c++) {
              x[a][c] = pr[c].x;
              du[a][c] = pr[c].y;
            }
          }
          element_force<NPE, MODE>(ep, S, i, x, du, f, wint, wp, vol);
#pragma unroll
          for (int a = 0; a < NPE; a++) fbuf[a * ne + i] = make_float4(f[a][0], f[a][1], f[a][2], 0.f);
        }
      }
    }
    res_sync<P>();

    // ---- 2: partial forces to their slots, everything that needs no other chunk
    float4* const halo = A.halo[k & 1];
    const unsigned tag = A.tag0 + (unsigned)k;
    const bool last = k + 1 == n;
    for (int l = nd; l < L; l += P) {
      const float4 f = own_force(l);
      if (l >= ch.n_int) {
        st_slot(halo + m1[l].x, f.x, f.y, f.z, tag);
      } else {  // kept in the next record's increments until the node's push
        float* r = reinterpret_cast<float*>(Tn.p0 + l);
        r[1] = f.x;
        r[3] = f.y;
        Tn.p1[l].y = f.z;
      }
    }
    // the work of the step: the fused kernel's block sums, finished by thread 0 below
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      wint += __shfl_xor_sync(0xffffffffu, wint, o);
      wp += __shfl_xor_sync(0xffffffffu, wp, o);
    }
    if ((tid & 31) == 0) {
      red[k & 1][0][tid >> 5] = wint;
      red[k & 1][1][tid >> 5] = wp;
    }
    // interior nodes: now where the CTA takes several rounds anyway, else with the others
    const int early = L > P ? ch.n_int : 0;
    auto total = [&](int l, float (&f)[3]) {
      if (l < ch.n_int) {
        const float* r = reinterpret_cast<const float*>(Tn.p0 + l);
        f[0] = __fadd_rn(0.f, r[1]);
        f[1] = __fadd_rn(0.f, r[3]);
        f[2] = __fadd_rn(0.f, Tn.p1[l].y);
        return;
      }
      const unsigned sl = (unsigned)m1[l].y;
      const float* r = recv + (sl & 0xffffu);
      const int cnt = (int)(sl >> 16);
      f[0] = f[1] = f[2] = 0.f;
      for (int j0 = 0; j0 < cnt; j0 += EU) {
        float h[EU][3];
#pragma unroll
        for (int j = 0; j < EU; j++)
#pragma unroll
          for (int c = 0; c < 3; c++) h[j][c] = r[c * ns + min(j0 + j, cnt - 1)];
#pragma unroll
        for (int j = 0; j < EU; j++)
          if (j0 + j < cnt)
#pragma unroll
            for (int c = 0; c < 3; c++) f[c] = __fadd_rn(f[c], h[j][c]);
      }
    };
    for (int l = nd; l < early; l += P) {
      float f[3];
      total(l, f);
      push(Tn, l, last, f[0], f[1], f[2]);
    }
    // ---- 3: boundary nodes
    res_sync<P>();  // the element forces make room for the received slots
    // (four FP64 operations of latency, here beside the wait for the slots)
    if (tid == 0 && ep.accum_energy) {
      float a = 0.f, b = 0.f;
#pragma unroll
      for (int w = 0; w < P / 32; w++) {
        a += red[k & 1][0][w];
        b += red[k & 1][1][w];
      }
      w0 += (double)a;
      w1 += (double)b;
    }
    const bool ok = res_receive<P>(A, halo, sslot, ns, tag, recv);
    if (!res_sync_and<P>(ok)) {
      if (bits) report(A.status, bits);
      return false;
    }
    for (int l = early + nd; l < L; l += P) {
      float f[3];
      total(l, f);
      push(Tn, l, last, f[0], f[1], f[2]);
    }
    res_sync<P>();
    if (snaps && (A.step0 + k + 1) % A.every == 0) {
      snapshot((A.step0 + k + 1) / A.every - 1);
      res_sync<P>();
    }
  }
  // an instance that has ended keeps its last state in the snapshots that follow
  if (snaps)
    for (int si = (A.step0 + n) / A.every; si < A.snap_end; si++) snapshot(si);

  if (bits) report(A.status, bits);
  // ---- store the owned nodes' state, the stress and the work sums
  for (int l = tid; l < ch.n_own; l += P) {
    const int g = ch.own_begin + l;
#pragma unroll
    for (int c = 0; c < 3; c++) {
      A.u[c][g] = su[c * L + l];
      A.v[c][g] = sv[c * L + l];
    }
    A.contact[g] = flags[l];
  }
  if (MODE == EM_J2)
    for (int i = tid; i < NQ * ne; i += P) {
      const size_t qi = (size_t)NQ * ch.elem_begin + i;
      A.sig_a[qi] = S.sig_a[i];
      A.sig_b[qi] = S.sig_b[i];
      A.epbar[qi] = S.epbar[i];
    }
  if (tid == 0) {
    A.chunk_work[4 * (size_t)ci] = w0;
    A.chunk_work[4 * (size_t)ci + 1] = w1;
  }
  return true;
}

// Resident CTAs per SM: at most 128 registers for four CTAs of 128 threads; batches of small
// chunks up to the register count at which they spill little (tet4: 64 threads at 64
// registers 1.77 us per instance and step of 28-element chunks, at 96 2.65).
constexpr int resident_min_ctas(int npe, int p, bool batch) {
  if (p == 128) return 4;
  if (!batch || npe == 10) return 10;
  return p == 64 ? 16 : 20;
}

template <int NPE, int MODE, int P, bool BATCH>
__global__ void __launch_bounds__(P, resident_min_ctas(NPE, P, BATCH))
    k_resident(const __grid_constant__ ResidentArgs A) {
  extern __shared__ __align__(16) unsigned char res_sm[];
  __shared__ float red[2][2][P / 32];
  if constexpr (!BATCH) {
    res_chunk<NPE, MODE, P, BATCH>(A, res_sm, blockIdx.x, red, nullptr);
  } else {
    // batches: chunks taken in order, an instance's chunks next to each other.  A CTA waits
    // only for chunks of its own instance; those before it in the order are running or
    // done, and the earliest instance with a chunk still to be taken gets every CTA that
    // comes free until all its chunks (no more than there are CTAs) are running.
    __shared__ int taken;
    __shared__ ResidentParams par;
    for (;;) {
      if (threadIdx.x == 0) taken = atomicAdd(A.claim, 1);
      res_sync<P>();
      const int c = taken;
      res_sync<P>();
      if (c >= A.n_chunks) return;
      if (!res_chunk<NPE, MODE, P, BATCH>(A, res_sm, A.order[c], red, &par)) return;
      res_sync<P>();
    }
  }
}

template <int NPE, int MODE, int P, bool BATCH>
const void* resident_fn() {
  return reinterpret_cast<const void*>(&k_resident<NPE, MODE, P, BATCH>);
}

}  // namespace ci
