// Training kernels of the candidate pruner's MLP (x -> 256 -> 256 -> 1; BF16 weights, FP32 accumulation).
//
// One tiled GEMM serves the forward pass and both backward products of every layer:
//   forward      Y[n x o]  = X[n x i] * W[o x i]^T + b    (optionally ReLU, optionally rounded to BF16 values)
//   input grad   dX[n x i] = dY[n x o] * W[o x i]
//   weight grad  dW[o x i] = dY^T[o x n] * X[n x i]
// Operands are addressed through strides, so transposes cost nothing; W is read as BF16 (the weights the
// inference kernel uses), activations and gradients are FP32.  Every output element is summed over k in a fixed
// order by one thread: results are deterministic, run to run.  Then BCE-with-logits loss/gradient, the ReLU mask of
// a backward gradient, the bias gradient (column sums) and an Adam step on the FP32 master weights that also writes
// their BF16 copy.
#include <cuda_bf16.h>

#include "common.cuh"

namespace {

constexpr int GT = 64;    // output tile (GT x GT) per CTA
constexpr int GK = 16;    // k tile
constexpr int GTHR = 256; // threads: each computes a 4 x 4 sub-tile

template <typename TB>
__device__ __forceinline__ float ld(const TB* p, int64_t i);
template <>
__device__ __forceinline__ float ld<float>(const float* p, int64_t i) { return p[i]; }
template <>
__device__ __forceinline__ float ld<__nv_bfloat16>(const __nv_bfloat16* p, int64_t i) { return __bfloat162float(p[i]); }

// C[m, n] = sum_k A[m*sam + k*sak] * B[k*sbk + n*sbn]  (+ bias[n]) (ReLU) (BF16 rounding)
template <typename TB>
__global__ void __launch_bounds__(GTHR)
gemm_k(int M, int N, int K, const float* __restrict__ A, int64_t sam, int64_t sak, const TB* __restrict__ B,
       int64_t sbk, int64_t sbn, const float* __restrict__ bias, int relu, int round_bf16, float* __restrict__ C,
       int64_t scm, int64_t scn) {
  __shared__ float As[GK][GT + 1];
  __shared__ float Bs[GK][GT + 1];
  const int tx = threadIdx.x % 16, ty = threadIdx.x / 16;
  const int m0 = blockIdx.y * GT, n0 = blockIdx.x * GT;
  float acc[4][4];
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j) acc[i][j] = 0.f;
  for (int k0 = 0; k0 < K; k0 += GK) {
    for (int e = threadIdx.x; e < GK * GT; e += GTHR) {
      const int kk = e / GT, mm = e % GT;
      const int m = m0 + mm, k = k0 + kk;
      As[kk][mm] = (m < M && k < K) ? A[m * sam + k * sak] : 0.f;
      const int nn = mm, n = n0 + nn;
      Bs[kk][nn] = (n < N && k < K) ? ld<TB>(B, k * sbk + n * sbn) : 0.f;
    }
    __syncthreads();
#pragma unroll
    for (int kk = 0; kk < GK; ++kk) {
      float a[4], b[4];
#pragma unroll
      for (int i = 0; i < 4; ++i) a[i] = As[kk][ty * 4 + i];
#pragma unroll
      for (int j = 0; j < 4; ++j) b[j] = Bs[kk][tx * 4 + j];
#pragma unroll
      for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) acc[i][j] = __fadd_rn(acc[i][j], __fmul_rn(a[i], b[j]));
    }
    __syncthreads();
  }
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const int m = m0 + ty * 4 + i;
    if (m >= M) continue;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const int n = n0 + tx * 4 + j;
      if (n >= N) continue;
      float v = acc[i][j];
      if (bias) v = __fadd_rn(v, bias[n]);
      if (relu) v = fmaxf(v, 0.f);
      if (round_bf16) v = __bfloat162float(__float2bfloat16_rn(v));
      C[m * scm + n * scn] = v;
    }
  }
}

// The products of the 1-wide layer 3, which a 64 x 64 tile would compute mostly for padding, in gemm_k's order (k
// ascending from zero, each product rounded, then added): bit-identical to it.
//
// N = 1 (logits): GV_ROWS rows of A are staged with coalesced loads, then a thread sums one row.  Its 256 dependent
// additions bound it.  8,192 x 256: 20.3 -> 8.1 us.
constexpr int GV_ROWS = 64;
constexpr int GV_K = 128;      // k per stage

template <typename TB>
__global__ void __launch_bounds__(GTHR)
gemv_k(int M, int K, const float* __restrict__ A, int64_t sam, const TB* __restrict__ B, int64_t sbk,
       const float* __restrict__ bias, int relu, int round_bf16, float* __restrict__ C, int64_t scm) {
  __shared__ float As[GV_ROWS][GV_K + 1];
  __shared__ float Bs[GV_K];
  const int m0 = blockIdx.x * GV_ROWS, row = threadIdx.x;
  float acc = 0.f;
  for (int k0 = 0; k0 < K; k0 += GV_K) {
    const int kc = min(GV_K, K - k0);
#pragma unroll 8
    for (int e = threadIdx.x; e < GV_ROWS * GV_K; e += GTHR) {
      const int r = e / GV_K, k = e % GV_K;
      As[r][k] = m0 + r < M && k < kc ? A[(int64_t)(m0 + r) * sam + k0 + k] : 0.f;
    }
    if (threadIdx.x < kc) Bs[threadIdx.x] = ld<TB>(B, (int64_t)(k0 + threadIdx.x) * sbk);
    __syncthreads();
    if (row < GV_ROWS)
#pragma unroll 16
      for (int k = 0; k < kc; ++k) acc = __fadd_rn(acc, __fmul_rn(As[row][k], Bs[k]));
    __syncthreads();
  }
  if (row < GV_ROWS && m0 + row < M) {
    if (bias) acc = __fadd_rn(acc, bias[0]);
    if (relu) acc = fmaxf(acc, 0.f);
    if (round_bf16) acc = __bfloat162float(__float2bfloat16_rn(acc));
    C[(int64_t)(m0 + row) * scm] = acc;
  }
}

// K = 1 (the layer-3 input gradient): one product per element, four columns per thread, bound by the writes.
// 8,192 x 256: 20.3 -> 3.7 us.
template <typename TB>
__global__ void __launch_bounds__(GTHR)
outer_k(int M, int N, const float* __restrict__ A, int64_t sam, const TB* __restrict__ B, int64_t sbn,
        const float* __restrict__ bias, int relu, int round_bf16, float* __restrict__ C, int64_t scm) {
  const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  const int quads = N >> 2;
  if (i >= (int64_t)M * quads) return;
  const int m = (int)(i / quads), n = (int)(i % quads) * 4;
  const float a = A[m * sam];
  float v[4];
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    v[j] = __fadd_rn(0.f, __fmul_rn(a, ld<TB>(B, (n + j) * sbn)));
    if (bias) v[j] = __fadd_rn(v[j], bias[n + j]);
    if (relu) v[j] = fmaxf(v[j], 0.f);
    if (round_bf16) v[j] = __bfloat162float(__float2bfloat16_rn(v[j]));
  }
  *reinterpret_cast<float4*>(C + m * scm + n) = make_float4(v[0], v[1], v[2], v[3]);
}

template <typename TB>
void gemm_launch(int M, int N, int K, const float* A, int64_t sam, int64_t sak, const TB* B, int64_t sbk, int64_t sbn,
                 const float* bias, int relu, int round_bf16, float* C, int64_t scm, int64_t scn, cudaStream_t st) {
  if (N == 1 && sak == 1) {
    gemv_k<TB><<<(unsigned)((M + GV_ROWS - 1) / GV_ROWS), GTHR, 0, st>>>(M, K, A, sam, B, sbk, bias, relu, round_bf16,
                                                                         C, scm);
  } else if (K == 1 && scn == 1 && ((N | scm) & 3) == 0 && ((uintptr_t)C & 15) == 0) {
    const int64_t quads = (int64_t)M * (N / 4);
    outer_k<TB><<<(unsigned)((quads + GTHR - 1) / GTHR), GTHR, 0, st>>>(M, N, A, sam, B, sbn, bias, relu, round_bf16,
                                                                        C, scm);
  } else {
    dim3 grid((unsigned)((N + GT - 1) / GT), (unsigned)((M + GT - 1) / GT));
    gemm_k<TB><<<grid, GTHR, 0, st>>>(M, N, K, A, sam, sak, B, sbk, sbn, bias, relu, round_bf16, C, scm, scn);
  }
}

// Column sums db[j] = sum_i dY[i, j] (v[i] dY[i, j] when v is given: the weighted sum of layer 3's weight
// gradient), in a fixed order: rows in chunks of CS_ROWS, each chunk summed sequentially (colsum_chunk_k, one thread
// per (chunk, column)), the chunk sums added in chunk order (colsum_total_k).
constexpr int CS_ROWS = 64;

__global__ void colsum_chunk_k(int n, int o, const float* dY, const float* v, float* part) {
  const int j = blockIdx.x * blockDim.x + threadIdx.x;
  const int c = blockIdx.y;
  if (j >= o) return;
  const int i1 = min(n, (c + 1) * CS_ROWS);
  float s = 0.f;
#pragma unroll 16   // the loads ahead of the dependent additions
  for (int i = c * CS_ROWS; i < i1; ++i) {
    const float x = dY[(int64_t)i * o + j];
    s = __fadd_rn(s, v ? __fmul_rn(x, v[i]) : x);
  }
  part[(int64_t)c * o + j] = s;
}

__global__ void colsum_total_k(int chunks, int o, const float* part, float* db) {
  const int j = blockIdx.x * blockDim.x + threadIdx.x;
  if (j >= o) return;
  float s = 0.f;
#pragma unroll 32
  for (int c = 0; c < chunks; ++c) s = __fadd_rn(s, part[(int64_t)c * o + j]);
  db[j] = s;
}

// dY *= (Y > 0)
__global__ void relu_mask_k(int64_t n, const float* Y, float* dY) {
  const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (i < n && !(Y[i] > 0.f)) dY[i] = 0.f;
}

// ... four values per thread where both arrays are 16-byte aligned
__global__ void relu_mask4_k(int64_t quads, const float4* __restrict__ Y, float4* __restrict__ dY) {
  const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (i >= quads) return;
  const float4 y = Y[i];
  float4 d = dY[i];
  if (!(y.x > 0.f)) d.x = 0.f;
  if (!(y.y > 0.f)) d.y = 0.f;
  if (!(y.z > 0.f)) d.z = 0.f;
  if (!(y.w > 0.f)) d.w = 0.f;
  dY[i] = d;
}

// Weighted BCE with logits: dz = w (sigmoid(z) - y) / sum_w; per-block loss partial sums (fixed order).
__global__ void bce_k(int n, const float* z, const float* y, const float* w, float inv_wsum, float* dz,
                      float* loss_part) {
  __shared__ float red[256];
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  float l = 0.f;
  if (i < n) {
    const float zi = z[i], yi = y[i], wi = w[i];
    const float p = 1.f / (1.f + expf(-zi));
    dz[i] = wi * (p - yi) * inv_wsum;
    // log(1 + exp(-|z|)) + max(z, 0) - z*y
    l = wi * (log1pf(expf(-fabsf(zi))) + fmaxf(zi, 0.f) - zi * yi) * inv_wsum;
  }
  red[threadIdx.x] = l;
  __syncthreads();
  for (int s = blockDim.x / 2; s > 0; s >>= 1) {
    if (threadIdx.x < s) red[threadIdx.x] += red[threadIdx.x + s];
    __syncthreads();
  }
  if (threadIdx.x == 0) loss_part[blockIdx.x] = red[0];
}

__global__ void adam_k(int64_t n, float* p, const float* g, float* m, float* v, float lr, float b1, float b2,
                       float eps, float c1, float c2, float wd, __nv_bfloat16* p_bf16) {
  const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (i >= n) return;
  const float gi = g[i] + wd * p[i];
  const float mi = b1 * m[i] + (1.f - b1) * gi;
  const float vi = b2 * v[i] + (1.f - b2) * gi * gi;
  m[i] = mi;
  v[i] = vi;
  const float pi = p[i] - lr * (mi / c1) / (sqrtf(vi / c2) + eps);
  p[i] = pi;
  if (p_bf16) p_bf16[i] = __float2bfloat16_rn(pi);
}

// adam_k over several tensors (blockIdx.y): the six of the network take one launch of 2.5 us instead of six of 2 us
// with 10 us of host between them.
struct AdamGroup {
  vk_adam_tensor t[VK_ADAM_MAX];
};

__global__ void adam_group_k(AdamGroup group, float lr, float b1, float b2, float eps, float c1, float c2, float wd) {
  const vk_adam_tensor t = group.t[blockIdx.y];
  const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (i >= t.n) return;
  const float gi = t.g[i] + wd * t.p[i];
  const float mi = b1 * t.m[i] + (1.f - b1) * gi;
  const float vi = b2 * t.v[i] + (1.f - b2) * gi * gi;
  t.m[i] = mi;
  t.v[i] = vi;
  const float pi = t.p[i] - lr * (mi / c1) / (sqrtf(vi / c2) + eps);
  t.p[i] = pi;
  if (t.p_bf16) reinterpret_cast<__nv_bfloat16*>(t.p_bf16)[i] = __float2bfloat16_rn(pi);
}

// A mini-batch's rows, targets and weights: a group of 4 lanes copies 16 bytes each of a 16-float row; the writes and
// the scattered 64-byte reads bound it (8,192 rows: 4 us; three indexing kernels before took 18 and 45 us of host).
__global__ void gather_batch_k(const int64_t* __restrict__ idx, int n, const float* __restrict__ X, int width,
                               const float* __restrict__ y, const float* __restrict__ w, float* Xb, float* yb,
                               float* wb, int wide) {
  const int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  const int per = wide ? width >> 2 : width;    // elements (16 bytes or 4) a row
  const int64_t i = t / per;
  if (i >= n) return;
  const int j = (int)(t % per);
  const int64_t s = idx[i];
  if (wide)
    reinterpret_cast<float4*>(Xb)[t] = __ldg(reinterpret_cast<const float4*>(X) + s * per + j);
  else
    Xb[t] = X[s * per + j];
  if (j == 0) {
    yb[i] = y[s];
    wb[i] = w[s];
  }
}

__global__ void to_bf16_k(int64_t n, const float* x, __nv_bfloat16* y) {
  const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (i < n) y[i] = __float2bfloat16_rn(x[i]);
}

__global__ void bf16_to_f32_k(int64_t n, const __nv_bfloat16* x, float* y) {
  const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (i < n) y[i] = __bfloat162float(x[i]);
}

}  // namespace

extern "C" {

// b_bf16 != 0: B holds BF16 values, else FP32.
int vk_gemm(int M, int N, int K, const float* A, int64_t sam, int64_t sak, const void* B, int b_bf16, int64_t sbk,
            int64_t sbn, const float* bias, int relu, int round_bf16, float* C, int64_t scm, int64_t scn,
            void* stream) {
  if (M <= 0 || N <= 0) return 0;
  cudaStream_t st = (cudaStream_t)stream;
  if (b_bf16)
    gemm_launch(M, N, K, A, sam, sak, reinterpret_cast<const __nv_bfloat16*>(B), sbk, sbn, bias, relu, round_bf16, C,
                scm, scn, st);
  else
    gemm_launch(M, N, K, A, sam, sak, reinterpret_cast<const float*>(B), sbk, sbn, bias, relu, round_bf16, C, scm, scn,
                st);
  return vk_launch_status();
}

int64_t vk_colsum_ws_floats(int n, int o) {
  return n > 0 && o > 0 ? (int64_t)((n + CS_ROWS - 1) / CS_ROWS) * o : 0;
}

int vk_colsum(int n, int o, const float* dY, const float* v, float* ws, int64_t ws_floats, float* db, void* stream) {
  if (o <= 0) return 0;
  cudaStream_t st = (cudaStream_t)stream;
  const int chunks = n > 0 ? (n + CS_ROWS - 1) / CS_ROWS : 0;
  if (chunks > 0 && (!ws || ws_floats < vk_colsum_ws_floats(n, o))) return VK_E_ARG;
  if (chunks > 0) {
    dim3 grid((unsigned)((o + 127) / 128), (unsigned)chunks);
    colsum_chunk_k<<<grid, 128, 0, st>>>(n, o, dY, v, ws);
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return vk_err(e);
  }
  colsum_total_k<<<(unsigned)((o + 255) / 256), 256, 0, st>>>(chunks, o, ws, db);
  return vk_launch_status();
}

int vk_relu_mask(int64_t n, const float* Y, float* dY, void* stream) {
  if (n <= 0) return 0;
  if (n % 4 == 0 && (((uintptr_t)Y | (uintptr_t)dY) & 15) == 0)
    relu_mask4_k<<<(unsigned)((n / 4 + 255) / 256), 256, 0, (cudaStream_t)stream>>>(
        n / 4, reinterpret_cast<const float4*>(Y), reinterpret_cast<float4*>(dY));
  else
    relu_mask_k<<<(unsigned)((n + 255) / 256), 256, 0, (cudaStream_t)stream>>>(n, Y, dY);
  return vk_launch_status();
}

int vk_bce(int n, const float* z, const float* y, const float* w, float inv_wsum, float* dz, float* loss_part,
           void* stream) {
  if (n <= 0) return 0;
  bce_k<<<(unsigned)((n + 255) / 256), 256, 0, (cudaStream_t)stream>>>(n, z, y, w, inv_wsum, dz, loss_part);
  return vk_launch_status();
}

int vk_adam(int64_t n, float* p, const float* g, float* m, float* v, float lr, float b1, float b2, float eps,
            int step, float wd, void* p_bf16, void* stream) {
  if (n <= 0) return 0;
  float c1 = 1.f - powf(b1, (float)step), c2 = 1.f - powf(b2, (float)step);
  adam_k<<<(unsigned)((n + 255) / 256), 256, 0, (cudaStream_t)stream>>>(
      n, p, g, m, v, lr, b1, b2, eps, c1, c2, wd, reinterpret_cast<__nv_bfloat16*>(p_bf16));
  return vk_launch_status();
}

int vk_adam_group(const vk_adam_tensor* t, int n_tensors, float lr, float b1, float b2, float eps, int step, float wd,
                  void* stream) {
  if (n_tensors < 0 || n_tensors > VK_ADAM_MAX || (n_tensors > 0 && !t)) return VK_E_ARG;
  AdamGroup group{};
  int64_t most = 0;
  for (int k = 0; k < n_tensors; ++k) {
    group.t[k] = t[k];
    if (t[k].n > most) most = t[k].n;
  }
  if (most <= 0) return 0;
  const float c1 = 1.f - powf(b1, (float)step), c2 = 1.f - powf(b2, (float)step);
  dim3 grid((unsigned)((most + 255) / 256), (unsigned)n_tensors);
  adam_group_k<<<grid, 256, 0, (cudaStream_t)stream>>>(group, lr, b1, b2, eps, c1, c2, wd);
  return vk_launch_status();
}

int vk_gather_batch(const int64_t* idx, int n, const float* X, int width, const float* y, const float* w, float* Xb,
                    float* yb, float* wb, void* stream) {
  if (n <= 0) return 0;
  if (!idx || !X || !y || !w || !Xb || !yb || !wb || width < 1) return VK_E_ARG;
  const int wide = width % 4 == 0 && (((uintptr_t)X | (uintptr_t)Xb) & 15) == 0;
  const int64_t threads = (int64_t)n * (wide ? width / 4 : width);
  gather_batch_k<<<(unsigned)((threads + 255) / 256), 256, 0, (cudaStream_t)stream>>>(idx, n, X, width, y, w, Xb, yb,
                                                                                      wb, wide);
  return vk_launch_status();
}

int vk_to_bf16(int64_t n, const float* x, void* y, void* stream) {
  if (n <= 0) return 0;
  to_bf16_k<<<(unsigned)((n + 255) / 256), 256, 0, (cudaStream_t)stream>>>(n, x, reinterpret_cast<__nv_bfloat16*>(y));
  return vk_launch_status();
}

int vk_bf16_to_f32(int64_t n, const void* x, float* y, void* stream) {
  if (n <= 0) return 0;
  bf16_to_f32_k<<<(unsigned)((n + 255) / 256), 256, 0, (cudaStream_t)stream>>>(
      n, reinterpret_cast<const __nv_bfloat16*>(x), y);
  return vk_launch_status();
}

}  // extern "C"
