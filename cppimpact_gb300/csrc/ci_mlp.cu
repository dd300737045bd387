// ci_mlp.cu -- the surrogate's MLP (n_in -> H -> H -> n_out, tanh hidden layers):
// forward, backward and Adam on the GPU, every matrix product through ci_gemm_bf16
// (BF16 operands, FP32 accumulation), FP32 master weights, fixed-order reductions.
// The products of layers 2 and 3 are arranged as A B^T with both operands K-major (the
// form of the TMA-pipelined tcgen05 kernel): BF16 copies of W2 and W3 are kept
// transposed, and the weight gradients read transposed activations and output
// gradients.  A training batch is bound by its chain of small kernels, so what lies between
// the products is fused into one kernel per product: layer 1 from the rows of X with its
// transposed copy, the loss gradient with its transpose and bias gradient, the tanh
// derivative with the same, Adam with the BF16 copies in both orders (23 launches a batch
// before, 14 now, each set up while the one before runs, ci_pdl.h; 4 -> 256 -> 256 -> 5120, batches
// of 256: 238 us a batch before, 95 now).
//
// Parameters, in the order ci_mlp_get_params / set_params use:
//   W1 [n_in x H], b1 [H], W2 [H x H], b2 [H], W3 [H x n_out], b3 [n_out]
// (row-major; a layer computes Z = X W + b).
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstdint>
#include <random>
#include <string>
#include <vector>

#include "../../include/cppimpact_gb300.h"
#include "ci_pdl.h"

namespace ci {
int set_last_error(int code, const char* msg);
}

namespace {

using bf16 = __nv_bfloat16;

#define CM_CUDA(call)                                                                    \
  do {                                                                                   \
    cudaError_t e_ = (call);                                                             \
    if (e_ != cudaSuccess)                                                               \
      return ci::set_last_error(CI_ERR_CUDA, (std::string(#call) + ": " + cudaGetErrorString(e_)).c_str()); \
  } while (0)

#define CM_OK(call)              \
  do {                           \
    const int rc_ = (call);      \
    if (rc_ != CI_OK) return rc_; \
  } while (0)

__global__ void k_to_bf16(const float* in, bf16* out, long long n) {
  ci::pdl_next();
  ci::pdl_wait();
  const long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  if (i < n) out[i] = __float2bfloat16(in[i]);
}

// Partial sums of (Y - T)^2 over 256 columns of row r, whose targets are row idx[r] of T (row r
// when idx is null): part[r][block of columns], the 256 squares added as a tree of halves.  A warp
// per partial sum with 16 values in flight a lane (256 x 5,120, cold under a profiler: 27.3 us
// with a CTA and eight barriers per partial sum, 13.3 so; FP64 bounds it).
__global__ void __launch_bounds__(256) k_mse_loss(const float* Y, const float* T, const int* idx,
                                                  int rows, int cols, double* part) {
  ci::pdl_next();
  ci::pdl_wait();
  const int lane = threadIdx.x & 31, blocks = (cols + 255) / 256;
  const long long w = blockIdx.x * 8LL + (threadIdx.x >> 5);
  if (w >= (long long)rows * blocks) return;
  const int r = (int)(w / blocks), c0 = (int)(w % blocks) * 256 + lane;
  const float* y = Y + (size_t)r * cols;
  const float* t = T + (size_t)(idx ? idx[r] : r) * cols;
  float d[8];
#pragma unroll
  for (int j = 0; j < 8; j++) {
    const int c = min(c0 + 32 * j, cols - 1);
    d[j] = y[c] - t[c];
  }
  double s[8];
#pragma unroll
  for (int j = 0; j < 8; j++) s[j] = c0 + 32 * j < cols ? (double)d[j] * d[j] : 0.0;
#pragma unroll
  for (int o = 4; o > 0; o >>= 1)
#pragma unroll
    for (int j = 0; j < o; j++) s[j] += s[j + o];
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) s[0] += __shfl_down_sync(0xffffffffu, s[0], o);
  if (lane == 0) part[w] = s[0];
}

// The passes over a [rows x cols] gradient between two products, CB columns and kPassRows rows
// per CTA of 8 CB threads (thread: column tx, row group g): the value of entry (r, c) from
// `value`, its BF16 copy in row order (vb, may be null) and transposed (vT, may be null), and the
// column sums (group g of 8 sums rows r = g, g + 8, ... in order, then the 8 partial sums in group
// order), those of the blocks of rows one after the other in colsum.  Products and sums are
// rounded one by one.  What bounds it is latency: 32 rows of a thread are in flight at once (256 x
// 5,120, cold under a profiler: 8 behind branches about 25 us, 14.4 so), narrow gradients take 8
// columns per CTA, and tall ones several CTAs a column (gradients of 60,000 rows, 40 -> 64 -> 64 ->
// 64: 2.50 ms with one CTA over all rows, 1.01 so).
constexpr int kPassRows = 16384;

template <int CB, bool BLOCKS, class Value>
__device__ __forceinline__ void column_pass(int rows, int cols, bf16* vb, bf16* vT, float* colsum,
                                            Value value) {
  ci::pdl_next();
  ci::pdl_wait();
  constexpr int U = 32, TR = 8 * U;  // rows per turn
  __shared__ bf16 tile[CB][TR + 2];
  __shared__ float part[8][CB];
  const int tx = threadIdx.x % CB, g = threadIdx.x / CB;
  const int c0 = blockIdx.x * CB, c = c0 + tx;
  // (BLOCKS false, one block: the arithmetic of the bounds alone cost 4 % of a training epoch)
  const int begin = BLOCKS ? blockIdx.y * kPassRows : 0;
  const int end = BLOCKS ? min(rows, begin + kPassRows) : rows;
  float s = 0.f;
  for (int r0 = begin; r0 < end; r0 += TR) {
    // (indices past the end load the last entry, so that no branch holds a load back)
    float v[U];
#pragma unroll
    for (int i = 0; i < U; i++) v[i] = value(min(r0 + g + 8 * i, end - 1), min(c, cols - 1));
#pragma unroll
    for (int i = 0; i < U; i++) {
      const int r = r0 + g + 8 * i;
      if (r < end && c < cols) {
        s = __fadd_rn(s, v[i]);
        const bf16 h = __float2bfloat16(v[i]);
        if (vb) vb[(size_t)r * cols + c] = h;
        tile[tx][g + 8 * i] = h;
      }
    }
    if (vT) {
      __syncthreads();
      for (int i = threadIdx.x; i < CB * TR; i += 8 * CB) {
        const int k = i / TR, r = i % TR;
        if (c0 + k < cols && r0 + r < end) vT[(size_t)(c0 + k) * rows + r0 + r] = tile[k][r];
      }
      __syncthreads();
    }
  }
  part[g][tx] = s;
  __syncthreads();
  if (g == 0 && c < cols) {
    float t = part[0][tx];
    for (int k = 1; k < 8; k++) t += part[k][tx];
    colsum[(BLOCKS ? (size_t)blockIdx.y * cols : 0) + c] = t;
  }
}

// gb = the sums of the blocks of rows, in order
__global__ void k_add_colsums(const float* colsum, int blocks, int cols, float* gb) {
  ci::pdl_next();
  ci::pdl_wait();
  const int c = blockIdx.x * blockDim.x + threadIdx.x;
  if (c >= cols) return;
  float s = colsum[c];
  for (int b = 1; b < blocks; b++) s = __fadd_rn(s, colsum[(size_t)b * cols + c]);
  gb[c] = s;
}

// dY = scale (Y - T) (scale = 2 / (rows * cols)) for row r, whose targets are row idx[r] of T
// (row r when idx is null): BF16 in both orders, and gb = its column sums
template <int CB, bool BLOCKS>
__global__ void __launch_bounds__(8 * CB) k_mse_grad(const float* __restrict__ Y,
                                                     const float* __restrict__ T,
                                                     const int* __restrict__ idx, int rows, int cols,
                                                     float scale, bf16* dYb, bf16* dYbT, float* gb) {
  column_pass<CB, BLOCKS>(rows, cols, dYb, dYbT, gb, [&](int r, int c) {
    return __fmul_rn(scale, Y[(size_t)r * cols + c] - T[(size_t)(idx ? idx[r] : r) * cols + c]);
  });
}

// dZ = dH (1 - H^2): BF16 in row order and transposed (either may be null), and gb
template <int CB, bool BLOCKS>
__global__ void __launch_bounds__(8 * CB) k_tanh_back(const float* __restrict__ dH,
                                                      const float* __restrict__ H, int rows,
                                                      int cols, bf16* dZb, bf16* dZbT, float* gb) {
  column_pass<CB, BLOCKS>(rows, cols, dZb, dZbT, gb, [&](int r, int c) {
    const size_t i = (size_t)r * cols + c;
    const float h = H[i];
    return __fmul_rn(dH[i], __fmaf_rn(-h, h, 1.f));
  });
}

// Layer 1 when n_in is small (the surrogate's 4 impact parameters): Z = tanh(X W1 + b1)
// with the BF16 operands of the GEMM path, FP32 products summed in input order, from row
// idx[r] of X (row r when idx is null); the FP32 activation and its BF16 copies in row order
// and (HbT, may be null) transposed.  32 x 32 entries per CTA.
__global__ void __launch_bounds__(256) k_layer1_fwd(const float* X, const int* idx, const bf16* W1,
                                                    const float* b1, int rows, int n_in, int H,
                                                    float* Z, bf16* Hb, bf16* HbT) {
  ci::pdl_next();
  ci::pdl_wait();
  __shared__ bf16 tile[32][34];
  const int tx = threadIdx.x & 31, ty = threadIdx.x >> 5;
  const int h0 = blockIdx.x * 32, r0 = blockIdx.y * 32, h = h0 + tx;
  for (int j = ty; j < 32; j += 8) {
    const int r = r0 + j;
    if (r < rows && h < H) {
      const float* x = X + (size_t)(idx ? idx[r] : r) * n_in;
      float acc = 0.f;
      for (int k = 0; k < n_in; k++)
        acc = fmaf(__bfloat162float(__float2bfloat16(x[k])), __bfloat162float(W1[(size_t)k * H + h]), acc);
      const float z = tanhf(acc + b1[h]);
      Z[(size_t)r * H + h] = z;
      const bf16 zb = __float2bfloat16(z);
      Hb[(size_t)r * H + h] = zb;
      tile[j][tx] = zb;
    }
  }
  if (!HbT) return;
  __syncthreads();
  for (int j = ty; j < 32; j += 8)
    if (h0 + j < H && r0 + tx < rows) HbT[(size_t)(h0 + j) * rows + r0 + tx] = tile[tx][j];
}

// gW1 = X^T dZ1 [n_in x H] for small n_in from the transposed dZ1 [H x rows]: one warp per
// entry; lane j sums rows j, j+32, ... in order, then the 32 lane sums in a fixed butterfly order
__global__ void k_layer1_wgrad(const float* X, const int* idx, const bf16* dZbT, int rows, int n_in,
                               int H, float* gW) {
  ci::pdl_next();
  ci::pdl_wait();
  const int w = (int)((blockIdx.x * (long long)blockDim.x + threadIdx.x) >> 5);
  const int lane = threadIdx.x & 31;
  if (w >= n_in * H) return;
  const int k = w / H, h = w % H;
  float acc = 0.f;
#pragma unroll 4
  for (int r = lane; r < rows; r += 32)
    acc = fmaf(__bfloat162float(__float2bfloat16(X[(size_t)(idx ? idx[r] : r) * n_in + k])),
               __bfloat162float(dZbT[(size_t)h * rows + r]), acc);
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
  if (lane == 0) gW[w] = acc;
}

// out [cols x rows] (leading dimension ld_out) = in^T, in [rows x cols] (ld_in); 32 x 32
// tiles through shared memory
__global__ void __launch_bounds__(256) k_transpose_bf16(const bf16* in, int rows, int cols,
                                                        int ld_in, bf16* out, int ld_out) {
  ci::pdl_next();
  ci::pdl_wait();
  __shared__ bf16 tile[32][34];
  const int c0 = blockIdx.x * 32, r0 = blockIdx.y * 32;
  const int tx = threadIdx.x & 31, ty = threadIdx.x >> 5;
  for (int k = ty; k < 32; k += 8) {
    const int r = r0 + k, c = c0 + tx;
    if (r < rows && c < cols) tile[k][tx] = in[(size_t)r * ld_in + c];
  }
  __syncthreads();
  for (int k = ty; k < 32; k += 8) {
    const int c = c0 + k, r = r0 + tx;
    if (r < rows && c < cols) out[(size_t)c * ld_out + r] = tile[tx][k];
  }
}

inline cudaError_t transpose_bf16(const bf16* in, int rows, int cols, bf16* out, cudaStream_t st) {
  const dim3 grid((cols + 31) / 32, (rows + 31) / 32);
  return ci::launch_pdl(k_transpose_bf16, grid, 256, 0, st, in, rows, cols, cols, out, rows);
}

// Adam (Kingma & Ba 2015) on FP32 master weights, rounded one operation at a time; refreshes
// the BF16 copy, which it returns
struct AdamArgs {
  float *p, *m, *v;
  const float* g;
  bf16* pb;
  float lr, b1, b2, eps, c1, c2;
};

// N entries at once, entry i[k] used where on[k] (its loads are made in any case)
template <int N>
__device__ __forceinline__ void adam_step(const AdamArgs& A, const long long (&i)[N],
                                          const bool (&on)[N], bf16 (&h)[N]) {
  float g[N], m[N], v[N], p[N];
#pragma unroll
  for (int k = 0; k < N; k++) {
    g[k] = A.g[i[k]];
    m[k] = A.m[i[k]];
    v[k] = A.v[i[k]];
    p[k] = A.p[i[k]];
  }
#pragma unroll
  for (int k = 0; k < N; k++) {
    m[k] = __fmaf_rn(1.f - A.b1, g[k], __fmul_rn(A.b1, m[k]));
    v[k] = __fmaf_rn(__fmul_rn(1.f - A.b2, g[k]), g[k], __fmul_rn(A.b2, v[k]));
    const float mh = m[k] / A.c1, vh = v[k] / A.c2;
    p[k] = p[k] - __fmul_rn(A.lr, mh) / (sqrtf(vh) + A.eps);
    h[k] = __float2bfloat16(p[k]);
    if (on[k]) {
      A.m[i[k]] = m[k];
      A.v[i[k]] = v[k];
      A.p[i[k]] = p[k];
      A.pb[i[k]] = h[k];
    }
  }
}

// All parameters: W2 [H x H] and W3 [H x n_out] in 32 x 32 tiles, whose BF16 copies also go
// transposed to wT (W2^T then W3^T), then the rest (W1 b1, b2, b3) by entries
__global__ void __launch_bounds__(256) k_adam(const AdamArgs A, int n_in, int H, int n_out, bf16* wT) {
  ci::pdl_next();
  ci::pdl_wait();
  __shared__ bf16 tile[32][34];
  const int tr = (H + 31) / 32, t2 = tr * tr, tc3 = (n_out + 31) / 32, t3 = tr * tc3;
  const long long o2 = (long long)n_in * H + H, o3 = o2 + (long long)H * H + H;
  const int b = blockIdx.x;
  if (b < t2 + t3) {
    const bool third = b >= t2;
    const int t = third ? b - t2 : b, ncol = third ? n_out : H, tc = third ? tc3 : tr;
    const int r0 = t / tc * 32, c0 = t % tc * 32;
    const long long off = third ? o3 : o2;
    bf16* out = wT + (third ? (size_t)H * H : 0);
    const int tx = threadIdx.x & 31, ty = threadIdx.x >> 5;
    long long i[4];
    bool on[4];
    bf16 h[4];
#pragma unroll
    for (int k = 0; k < 4; k++) {
      const int r = r0 + ty + 8 * k, c = c0 + tx;
      on[k] = r < H && c < ncol;
      i[k] = off + (long long)min(r, H - 1) * ncol + min(c, ncol - 1);
    }
    adam_step<4>(A, i, on, h);
#pragma unroll
    for (int k = 0; k < 4; k++) tile[ty + 8 * k][tx] = h[k];
    __syncthreads();
    for (int j = ty; j < 32; j += 8)
      if (c0 + j < ncol && r0 + tx < H) out[(size_t)(c0 + j) * H + r0 + tx] = tile[tx][j];
    return;
  }
  // the entries before W2, then b2, then b3
  const long long e = (long long)(b - t2 - t3) * 256 + threadIdx.x;
  if (e >= o2 + H + n_out) return;
  const long long i[1] = {e < o2       ? e
                          : e < o2 + H ? e + (long long)H * H
                                       : e + (long long)H * H + (long long)H * n_out};
  const bool on[1] = {true};
  bf16 h[1];
  adam_step<1>(A, i, on, h);
}

// rows of X picked by idx -> Xb (BF16)
__global__ void k_gather_rows(const float* X, const int* idx, int rows, int nx, bf16* Xb) {
  ci::pdl_next();
  ci::pdl_wait();
  const int r = blockIdx.x;
  if (r >= rows) return;
  const int s = idx[r];
  for (int j = threadIdx.x; j < nx; j += blockDim.x)
    Xb[(size_t)r * nx + j] = __float2bfloat16(X[(size_t)s * nx + j]);
}

template <typename T>
struct DBuf {
  T* p = nullptr;
  size_t n = 0;
  ~DBuf() {
    if (p) cudaFree(p);
  }
  cudaError_t alloc(size_t count) {
    if (p) cudaFree(p);
    p = nullptr;
    n = count;
    return count ? cudaMalloc(&p, sizeof(T) * count) : cudaSuccess;
  }
};

inline unsigned nb(long long n) { return (unsigned)((n + 255) / 256); }

}  // namespace

struct ci_mlp {
  int n_in = 0, H = 0, n_out = 0;
  long long np = 0;           // parameter count
  long long off[6] = {0};     // W1 b1 W2 b2 W3 b3 offsets in the flat arrays
  DBuf<float> p, g, m, v;     // FP32 master params, grads, Adam moments
  DBuf<bf16> pb;              // BF16 copy of the parameters
  DBuf<bf16> wT;              // BF16 W2^T [H x H] then W3^T [n_out x H]
  DBuf<int> err;
  long long step = 0;
  int cap = 0;                // rows the activation buffers hold
  DBuf<float> Z1, Z2, Y, dH2, dH1;
  DBuf<bf16> Xb, H1b, H2b, dYb, dZ2b, dZ1b;
  DBuf<bf16> H1bT, H2bT, dYbT, dZ2bT, dZ1bT;  // transposes [cols x rows] for the weight gradients
  DBuf<double> part;
  DBuf<float> colpart;  // column sums by blocks of kPassRows rows, where there are several
  DBuf<int> idx;
};

namespace {

int ensure_cap(ci_mlp* M, int rows) {
  if (rows <= M->cap) return CI_OK;
  const size_t r = rows;
  CM_CUDA(M->Z1.alloc(r * M->H));
  CM_CUDA(M->Z2.alloc(r * M->H));
  CM_CUDA(M->Y.alloc(r * M->n_out));
  CM_CUDA(M->dH2.alloc(r * M->H));
  CM_CUDA(M->dH1.alloc(r * M->H));
  CM_CUDA(M->Xb.alloc(r * M->n_in));
  CM_CUDA(M->H1b.alloc(r * M->H));
  CM_CUDA(M->H2b.alloc(r * M->H));
  CM_CUDA(M->dYb.alloc(r * M->n_out));
  CM_CUDA(M->dZ2b.alloc(r * M->H));
  CM_CUDA(M->dZ1b.alloc(r * M->H));
  CM_CUDA(M->H1bT.alloc(r * M->H));
  CM_CUDA(M->H2bT.alloc(r * M->H));
  CM_CUDA(M->dYbT.alloc(r * M->n_out));
  CM_CUDA(M->dZ2bT.alloc(r * M->H));
  CM_CUDA(M->dZ1bT.alloc(r * M->H));
  CM_CUDA(M->part.alloc(r * nb(M->n_out)));
  CM_CUDA(M->colpart.alloc(rows > kPassRows ? (r + kPassRows - 1) / kPassRows * std::max(M->H, M->n_out) : 0));
  CM_CUDA(M->idx.alloc(r));
  M->cap = rows;
  return CI_OK;
}

int gemm(ci_mlp* M, const void* A, int lda, int tA, const void* B, int ldb, int tB, float* C, int ldc,
         void* Cb, int m, int n, int k, float beta, const float* bias, int act, cudaStream_t st) {
  return ci_gemm_bf16(A, lda, tA, B, ldb, tB, C, ldc, Cb, m, n, k, 1.0f, beta, bias, act,
                      M->err.p, st);
}

// BF16 W2^T and W3^T from the BF16 parameter copy (after every parameter update)
int refresh_wT(ci_mlp* M, cudaStream_t st) {
  CM_CUDA(transpose_bf16(M->pb.p + M->off[2], M->H, M->H, M->wT.p, st));
  CM_CUDA(transpose_bf16(M->pb.p + M->off[4], M->H, M->n_out, M->wT.p + (size_t)M->H * M->H, st));
  return CI_OK;
}

// forward of `rows` rows of X (idx[r], or r when idx is null); writes Y and the hidden
// activations, with keep also what the weight gradients read of them
int forward(ci_mlp* M, const float* X, const int* idx, int rows, bool keep, cudaStream_t st) {
  const bf16* W1 = M->pb.p + M->off[0];
  const bf16* W2T = M->wT.p;
  const bf16* W3T = M->wT.p + (size_t)M->H * M->H;
  const float* b1 = M->p.p + M->off[1];
  const float* b2 = M->p.p + M->off[3];
  const float* b3 = M->p.p + M->off[5];
  if (M->n_in < 16) {
    CM_CUDA(ci::launch_pdl(k_layer1_fwd, dim3((M->H + 31) / 32, (rows + 31) / 32), 256, 0, st, 
        X, idx, W1, b1, rows, M->n_in, M->H, M->Z1.p, M->H1b.p, keep ? M->H1bT.p : nullptr));
  } else {
    if (idx)
      CM_CUDA(ci::launch_pdl(k_gather_rows, rows, 32, 0, st, X, idx, rows, M->n_in, M->Xb.p));
    else
      CM_CUDA(ci::launch_pdl(k_to_bf16, nb((long long)rows * M->n_in), 256, 0, st, X, M->Xb.p,
                             (long long)rows * M->n_in));
    CM_OK(gemm(M, M->Xb.p, M->n_in, 0, W1, M->H, 0, M->Z1.p, M->H, M->H1b.p, rows, M->H, M->n_in,
               0.f, b1, 1, st));
    if (keep) CM_CUDA(transpose_bf16(M->H1b.p, rows, M->H, M->H1bT.p, st));
  }
  CM_OK(gemm(M, M->H1b.p, M->H, 0, W2T, M->H, 1, M->Z2.p, M->H, M->H2b.p, rows, M->H, M->H, 0.f, b2,
             1, st));
  if (keep) CM_CUDA(transpose_bf16(M->H2b.p, rows, M->H, M->H2bT.p, st));
  CM_OK(gemm(M, M->H2b.p, M->H, 0, W3T, M->H, 1, M->Y.p, M->n_out, nullptr, rows, M->n_out, M->H,
             0.f, b3, 0, st));
  return CI_OK;
}

// loss and gradients into M->g after forward(keep) of the same rows, whose targets are rows
// idx[r] of T (rows r when idx is null); *loss (may be NULL) gets the mean squared error (host,
// synchronises)
int backward(ci_mlp* M, const float* X, const float* T, const int* idx, int rows, cudaStream_t st,
             double* loss) {
  const long long ny = (long long)rows * M->n_out;
  float* gW1 = M->g.p + M->off[0];
  float* gb1 = M->g.p + M->off[1];
  float* gW2 = M->g.p + M->off[2];
  float* gb2 = M->g.p + M->off[3];
  float* gW3 = M->g.p + M->off[4];
  float* gb3 = M->g.p + M->off[5];
  const bf16* W2 = M->pb.p + M->off[2];
  const bf16* W3 = M->pb.p + M->off[4];
  if (loss) {
    CM_CUDA(ci::launch_pdl(k_mse_loss, (unsigned)(((long long)rows * nb(M->n_out) + 7) / 8), 256, 0, st, M->Y.p, T,
                           idx, rows, M->n_out, M->part.p));
  }
  // layer 3: gW3 = H2^T dY as (H2^T) (dY^T)^T
  const float scale = 2.0f / (float)ny;
  // (an epoch of 4,096 rows, 8 and 32 columns per CTA: 1,536 outputs 1,114 and 1,132 us, 2,048 1,124 and
  // 1,123, 2,560 1,172 and 1,154, 5,120 1,429 and 1,315)
  const bool wide = M->n_out > 2048;
  const unsigned blocks = (rows + kPassRows - 1) / kPassRows;
  auto sums = [&](float* gb) { return blocks > 1 ? M->colpart.p : gb; };
  auto add_sums = [&](int cols, float* gb) {
    return blocks > 1 ? ci::launch_pdl(k_add_colsums, nb(cols), 256, 0, st, M->colpart.p, (int)blocks, cols, gb)
                      : cudaSuccess;
  };
  CM_CUDA(ci::launch_pdl(blocks > 1 ? (wide ? k_mse_grad<32, true> : k_mse_grad<8, true>)
                                    : (wide ? k_mse_grad<32, false> : k_mse_grad<8, false>),
                         dim3(wide ? (M->n_out + 31) / 32 : (M->n_out + 7) / 8, blocks), wide ? 256 : 64,
                         0, st, M->Y.p, T, idx, rows, M->n_out, scale, M->dYb.p, M->dYbT.p, sums(gb3)));
  CM_CUDA(add_sums(M->n_out, gb3));
  CM_OK(gemm(M, M->H2bT.p, rows, 0, M->dYbT.p, rows, 1, gW3, M->n_out, nullptr, M->H, M->n_out,
             rows, 0.f, nullptr, 0, st));
  CM_OK(gemm(M, M->dYb.p, M->n_out, 0, W3, M->n_out, 1, M->dH2.p, M->H, nullptr, rows, M->H,
             M->n_out, 0.f, nullptr, 0, st));
  // layer 2: gW2 = H1^T dZ2 as (H1^T) (dZ2^T)^T; Z2 holds tanh(Z2) = H2 (the GEMM wrote the
  // activated values)
  CM_CUDA(ci::launch_pdl(blocks > 1 ? k_tanh_back<8, true> : k_tanh_back<8, false>, dim3((M->H + 7) / 8, blocks), 64, 0, st, M->dH2.p, M->Z2.p,
                         rows, M->H, M->dZ2b.p, M->dZ2bT.p, sums(gb2)));
  CM_CUDA(add_sums(M->H, gb2));
  CM_OK(gemm(M, M->H1bT.p, rows, 0, M->dZ2bT.p, rows, 1, gW2, M->H, nullptr, M->H, M->H, rows, 0.f,
             nullptr, 0, st));
  CM_OK(gemm(M, M->dZ2b.p, M->H, 0, W2, M->H, 1, M->dH1.p, M->H, nullptr, rows, M->H, M->H, 0.f,
             nullptr, 0, st));
  // layer 1
  const bool small = M->n_in < 16;
  CM_CUDA(ci::launch_pdl(blocks > 1 ? k_tanh_back<8, true> : k_tanh_back<8, false>, dim3((M->H + 7) / 8, blocks), 64, 0, st, M->dH1.p, M->Z1.p,
                         rows, M->H, small ? nullptr : M->dZ1b.p, small ? M->dZ1bT.p : nullptr,
                         sums(gb1)));
  CM_CUDA(add_sums(M->H, gb1));
  if (small) {
    CM_CUDA(ci::launch_pdl(k_layer1_wgrad, nb(32LL * M->n_in * M->H), 256, 0, st, X, idx, M->dZ1bT.p, rows, M->n_in,
                                                               M->H, gW1));
  } else {
    CM_OK(gemm(M, M->Xb.p, M->n_in, 1, M->dZ1b.p, M->H, 0, gW1, M->H, nullptr, M->n_in, M->H, rows,
               0.f, nullptr, 0, st));
  }
  if (loss) {
    std::vector<double> part((size_t)rows * nb(M->n_out));
    CM_CUDA(cudaMemcpyAsync(part.data(), M->part.p, sizeof(double) * part.size(),
                            cudaMemcpyDeviceToHost, st));
    CM_CUDA(cudaStreamSynchronize(st));
    double s = 0.0;
    for (double x : part) s += x;
    *loss = s / (double)ny;
  }
  return CI_OK;
}

int check_err(ci_mlp* M, cudaStream_t st) {
  int e = 0;
  CM_CUDA(cudaMemcpyAsync(&e, M->err.p, sizeof(int), cudaMemcpyDeviceToHost, st));
  CM_CUDA(cudaStreamSynchronize(st));
  if (e) return ci::set_last_error(CI_ERR_CUDA, "tensor-core GEMM wait timed out");
  return CI_OK;
}

}  // namespace

extern "C" {

int ci_mlp_create(int n_in, int n_hidden, int n_out, unsigned long long seed, ci_mlp** out) {
  if (!out || n_in <= 0 || n_hidden <= 0 || n_out <= 0)
    return ci::set_last_error(CI_ERR_INVALID, "ci_mlp_create: bad sizes");
  ci_mlp* M = new ci_mlp();
  M->n_in = n_in;
  M->H = n_hidden;
  M->n_out = n_out;
  const long long sz[6] = {(long long)n_in * n_hidden, n_hidden, (long long)n_hidden * n_hidden,
                           n_hidden, (long long)n_hidden * n_out, n_out};
  long long o = 0;
  for (int i = 0; i < 6; i++) {
    M->off[i] = o;
    o += sz[i];
  }
  M->np = o;
  // Glorot-uniform weights, zero biases, from the seed
  std::vector<float> h(o, 0.f);
  std::mt19937_64 rng(seed);
  const int fan[3][2] = {{n_in, n_hidden}, {n_hidden, n_hidden}, {n_hidden, n_out}};
  for (int l = 0; l < 3; l++) {
    const double a = std::sqrt(6.0 / (fan[l][0] + fan[l][1]));
    std::uniform_real_distribution<double> U(-a, a);
    for (long long i = 0; i < sz[2 * l]; i++) h[M->off[2 * l] + i] = (float)U(rng);
  }
  int rc = CI_OK;
  if (M->p.alloc(o) || M->g.alloc(o) || M->m.alloc(o) || M->v.alloc(o) || M->pb.alloc(o) ||
      M->wT.alloc((size_t)n_hidden * n_hidden + (size_t)n_hidden * n_out) || M->err.alloc(1))
    rc = ci::set_last_error(CI_ERR_NOMEM, "ci_mlp_create: device allocation failed");
  if (!rc) rc = ci_mlp_set_params(M, h.data());
  if (!rc && (cudaMemset(M->m.p, 0, sizeof(float) * o) || cudaMemset(M->v.p, 0, sizeof(float) * o) ||
              cudaMemset(M->err.p, 0, sizeof(int))))
    rc = ci::set_last_error(CI_ERR_CUDA, "ci_mlp_create: memset failed");
  if (rc) {
    delete M;
    return rc;
  }
  *out = M;
  return CI_OK;
}

int ci_mlp_destroy(ci_mlp* M) {
  delete M;
  return CI_OK;
}

long long ci_mlp_num_params(const ci_mlp* M) { return M ? M->np : 0; }

int ci_mlp_set_params(ci_mlp* M, const float* h) {
  if (!M || !h) return ci::set_last_error(CI_ERR_INVALID, "null argument");
  CM_CUDA(cudaMemcpy(M->p.p, h, sizeof(float) * M->np, cudaMemcpyHostToDevice));
  k_to_bf16<<<nb(M->np), 256>>>(M->p.p, M->pb.p, M->np);
  CM_CUDA(cudaGetLastError());
  CM_OK(refresh_wT(M, 0));
  CM_CUDA(cudaDeviceSynchronize());
  M->step = 0;
  return CI_OK;
}

int ci_mlp_get_params(ci_mlp* M, float* h) {
  if (!M || !h) return ci::set_last_error(CI_ERR_INVALID, "null argument");
  CM_CUDA(cudaMemcpy(h, M->p.p, sizeof(float) * M->np, cudaMemcpyDeviceToHost));
  return CI_OK;
}

int ci_mlp_predict(ci_mlp* M, const float* d_X, int n, float* d_Y, void* stream) {
  if (!M || !d_X || !d_Y || n <= 0) return ci::set_last_error(CI_ERR_INVALID, "bad argument");
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  for (int r0 = 0; r0 < n; r0 += 4096) {
    const int rows = std::min(4096, n - r0);
    CM_OK(ensure_cap(M, rows));
    CM_OK(forward(M, d_X + (size_t)r0 * M->n_in, nullptr, rows, false, st));
    CM_CUDA(cudaMemcpyAsync(d_Y + (size_t)r0 * M->n_out, M->Y.p, sizeof(float) * rows * M->n_out,
                            cudaMemcpyDeviceToDevice, st));
  }
  return check_err(M, st);
}

int ci_mlp_gradients(ci_mlp* M, const float* d_X, const float* d_T, int n, float* h_grad,
                     double* loss) {
  if (!M || !d_X || !d_T || n <= 0) return ci::set_last_error(CI_ERR_INVALID, "bad argument");
  CM_OK(ensure_cap(M, n));
  CM_OK(forward(M, d_X, nullptr, n, true, 0));
  CM_OK(backward(M, d_X, d_T, nullptr, n, 0, loss));
  if (h_grad) CM_CUDA(cudaMemcpy(h_grad, M->g.p, sizeof(float) * M->np, cudaMemcpyDeviceToHost));
  return check_err(M, 0);
}

int ci_mlp_train(ci_mlp* M, const float* d_X, const float* d_T, int n, int batch, int epochs,
                 float lr, unsigned long long seed, double* h_loss, void* stream) {
  if (!M || !d_X || !d_T || n <= 0 || batch <= 0 || epochs <= 0)
    return ci::set_last_error(CI_ERR_INVALID, "bad argument");
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  batch = std::min(batch, n);
  CM_OK(ensure_cap(M, n));
  std::mt19937_64 rng(seed);
  std::vector<int> perm(n);
  for (int i = 0; i < n; i++) perm[i] = i;
  const float b1 = 0.9f, b2 = 0.999f, eps = 1e-8f;
  for (int ep = 0; ep < epochs; ep++) {
    std::shuffle(perm.begin(), perm.end(), rng);
    CM_CUDA(cudaMemcpyAsync(M->idx.p, perm.data(), sizeof(int) * n, cudaMemcpyHostToDevice, st));
    double ep_loss = 0.0;
    int nbatches = 0;
    for (int b0 = 0; b0 + batch <= n; b0 += batch) {
      const int* idx = M->idx.p + b0;
      CM_OK(forward(M, d_X, idx, batch, true, st));
      const bool last = b0 + 2 * batch > n;
      double l = 0.0;
      CM_OK(backward(M, d_X, d_T, idx, batch, st, (h_loss && last) ? &l : nullptr));
      ep_loss += l;
      nbatches += last ? 1 : 0;
      M->step++;
      const float c1 = 1.f - std::pow(b1, (float)M->step), c2 = 1.f - std::pow(b2, (float)M->step);
      const AdamArgs A{M->p.p, M->m.p, M->v.p, M->g.p, M->pb.p, lr, b1, b2, eps, c1, c2};
      const int tr = (M->H + 31) / 32;
      const long long rest = (long long)M->n_in * M->H + 2LL * M->H + M->n_out;
      CM_CUDA(ci::launch_pdl(k_adam, (unsigned)(tr * tr + tr * ((M->n_out + 31) / 32)) + nb(rest), 256, 0, st, 
          A, M->n_in, M->H, M->n_out, M->wT.p));
    }
    if (h_loss) h_loss[ep] = nbatches ? ep_loss / nbatches : 0.0;
  }
  return check_err(M, st);
}

}  // extern "C"
