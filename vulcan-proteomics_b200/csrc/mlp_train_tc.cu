// Training GEMMs of the candidate pruner on the 5th-generation tensor cores (tcgen05, FP32 accumulation in TMEM).
//
// C[m, n] = sum_k A(m, k) B(k, n) (+ bias[n]) (ReLU) (rounded to BF16 values), with A(m, k) = A[m*sam + k*sak]
// (FP32) and B(k, n) = B[k*sbk + n*sbn] (BF16, or FP32); strides make every transpose of the backward pass free.
// Both operands are rounded to BF16 (round to nearest) as they are staged into shared memory -- the weights, the
// features and the BF16-rounded layer-1 activations are BF16 values already, so only the backward gradients lose
// bits -- and the products are summed in FP32 by the tensor core (an order of its own: not the fixed order of the
// SIMT kernel in mlp_train.cu, which stays the bit-exact reference of the oracle test).
//
// CTA: 256 threads, tile 128 (M) x Nt (N <= 128, a multiple of 16), K in chunks of 128 staged into the canonical
// K-major layout (tc_common.cuh): a thread stages eight k of a row at a time -- two 16-byte loads (one of BF16
// values) where k is contiguous, eight loads that share 32-byte sectors with the neighbouring rows where the row is
// -- and stores them as one 16-byte row of a core matrix, eight lanes filling the 128 bytes of one (no bank
// conflicts).  One thread issues the UMMAs (K 16 each) and commits them to the buffer's mbarrier; two buffers, so a
// chunk is staged while the previous one is multiplied, and a buffer is overwritten only after its MMAs completed.
// Weight gradients reduce over the batch (K = batch rows): the K range is split over blockIdx.z, each split writes
// its partial tile to a workspace, and tc_gemm_reduce_k sums the splits in split order (deterministic) and applies
// bias / ReLU / rounding.  Waits are bounded: on a timeout the CTA records VK_STATUS_WAIT_TIMEOUT, stops issuing,
// waits (bounded) for its last commit and frees its TMEM.
//
// What bounds it at the training's sizes (8,192 x 256 x 256 and 256 x 256 x 8,192): the latency of staging a tile and
// of the launch, on 128-256 CTAs.  With one 2-byte store per element into 16-way bank conflicts, 128 threads and 256
// columns a CTA (64 CTAs) the forward and input-gradient GEMMs took 96 us on average and the weight gradients 45; now
// 11 (K = 16), 21 and 23, and 17 and 8 us.  Eight items loaded ahead per thread instead of four change nothing.
#include <cuda_bf16.h>

#include "common.cuh"
#include "tc_common.cuh"

namespace {

constexpr int TG_M = 128;
constexpr int TG_N = 128;
constexpr int TG_KC = 128;
constexpr int TG_THREADS = 256;
constexpr uint32_t TG_WAIT = 1u << 24;
constexpr int TG_SMEM_A = TG_M * TG_KC * 2;        // 32 KB
constexpr int TG_SMEM_B = TG_N * TG_KC * 2;        // 32 KB
constexpr int TG_BUF = TG_SMEM_A + TG_SMEM_B;
constexpr int TG_SLACK = 128;                      // alignment of the dynamic shared memory
constexpr size_t TG_MOST = 2 * TG_BUF + TG_SLACK;
constexpr int TG_BATCH = 4;                        // items loaded ahead per thread

__device__ __forceinline__ uint32_t bf16_pair(float a, float b) {
  const __nv_bfloat162 v = __floats2bfloat162_rn(a, b);
  return *reinterpret_cast<const uint32_t*>(&v);
}

// Eight k of one row as BF16: from eight contiguous values, 16-byte aligned ...
__device__ __forceinline__ uint4 load8(const float* p) {
  const float4 a = __ldg(reinterpret_cast<const float4*>(p)), b = __ldg(reinterpret_cast<const float4*>(p) + 1);
  return make_uint4(bf16_pair(a.x, a.y), bf16_pair(a.z, a.w), bf16_pair(b.x, b.y), bf16_pair(b.z, b.w));
}
__device__ __forceinline__ uint4 load8(const __nv_bfloat16* p) { return __ldg(reinterpret_cast<const uint4*>(p)); }
__device__ __forceinline__ float ld_f(const float* p) { return __ldg(p); }
__device__ __forceinline__ float ld_f(const __nv_bfloat16* p) { return __bfloat162float(*p); }
// ... or one by one, zero from the n-th on
template <typename T>
__device__ __forceinline__ uint4 gather8(const T* p, int64_t sk, int n) {
  float v[8];
#pragma unroll
  for (int j = 0; j < 8; ++j) v[j] = j < n ? ld_f(p + j * sk) : 0.f;
  return make_uint4(bf16_pair(v[0], v[1]), bf16_pair(v[2], v[3]), bf16_pair(v[4], v[5]), bf16_pair(v[6], v[7]));
}

// Rows r0.. (R of them, a multiple of 16) x 8 << nk_log k from k0 of X(r, k) = X[r*sr + k*sk] into the canonical
// layout at dst; zeros past nr rows and past ke.
template <typename T>
__device__ __forceinline__ void stage(uint8_t* dst, const T* __restrict__ X, int64_t sr, int64_t sk, int r0, int R,
                                      int nr, int k0, int nk_log, int ke) {
  const int items = R << nk_log, nk1 = (1 << nk_log) - 1;
  const bool wide = sk == 1 && (sr * (int64_t)sizeof(T)) % 16 == 0 && (reinterpret_cast<uintptr_t>(X) & 15) == 0;
  for (int i0 = threadIdx.x; i0 < items; i0 += TG_THREADS * TG_BATCH) {
    uint4 v[TG_BATCH];
#pragma unroll
    for (int b = 0; b < TG_BATCH; ++b) {
      const int i = i0 + b * TG_THREADS, u = i >> 3;
      const int r = (i & 7) | (u >> nk_log) << 3, k = (u & nk1) << 3;   // eight neighbouring lanes: one core matrix
      const int left = ke - (k0 + k);
      v[b] = make_uint4(0u, 0u, 0u, 0u);
      if (i < items && r0 + r < nr && left > 0) {
        const T* p = X + (int64_t)(r0 + r) * sr + (int64_t)(k0 + k) * sk;
        v[b] = wide && left >= 8 ? load8(p) : gather8(p, sk, left);
      }
    }
#pragma unroll
    for (int b = 0; b < TG_BATCH; ++b) {
      const int i = i0 + b * TG_THREADS, u = i >> 3;
      if (i < items)
        *reinterpret_cast<uint4*>(dst + canon_off((i & 7) | (u >> nk_log) << 3, (u & nk1) << 3, TG_KC)) = v[b];
    }
  }
}

__device__ __forceinline__ float tg_out(float v, const float* bias, int n, int relu, int round_bf16) {
  if (bias) v = __fadd_rn(v, bias[n]);
  if (relu) v = fmaxf(v, 0.f);
  if (round_bf16) v = __bfloat162float(__float2bfloat16_rn(v));
  return v;
}

template <typename TB>
__global__ void __launch_bounds__(TG_THREADS)
tc_gemm_k(int M, int N, int K, int k_split, int buffers, const float* __restrict__ A, int64_t sam, int64_t sak,
          const TB* __restrict__ B, int64_t sbk, int64_t sbn, const float* __restrict__ bias, int relu,
          int round_bf16, float* __restrict__ C, int64_t scm, int64_t scn, float* __restrict__ ws,
          int32_t* status) {
  extern __shared__ uint8_t tg_raw[];
  __shared__ __align__(8) uint64_t bar[2];
  __shared__ uint32_t tmem_slot;
  __shared__ int abort_flag;
  uint8_t* sm = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(tg_raw) + 127) & ~uintptr_t(127));
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int m0 = blockIdx.x * TG_M;
  const int n0 = blockIdx.y * TG_N;
  const int Nt = min(TG_N, N - n0);               // a multiple of 16
  const int kb = blockIdx.z * k_split, ke = min(K, kb + k_split);
  if (tid == 0) {
    abort_flag = 0;
    vk::mbar_init(&bar[0], 1);
    vk::mbar_init(&bar[1], 1);
    vk::fence_mbar_init();
  }
  if (warp == 0) tmem_alloc_warp(&tmem_slot, TG_N);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = tmem_slot;
  const uint32_t idesc = instr_desc(TG_M, Nt);
  int chunk = 0;      // chunks staged and issued; chunk c uses buffer c % buffers for the (c / buffers)-th time
  bool fail = false;
  for (int k0 = kb; k0 < ke; k0 += TG_KC, ++chunk) {
    const int b = chunk % buffers;
    uint8_t* sA = sm + b * TG_BUF;
    uint8_t* sB = sA + TG_SMEM_A;
    if (chunk >= buffers) {   // the buffer's former MMAs have read it
      if (!vk::mbar_wait(&bar[b], (uint32_t)(chunk / buffers - 1) & 1u, TG_WAIT)) atomicOr(&abort_flag, 1);
      __syncthreads();
      if (abort_flag) {
        fail = true;
        break;
      }
    }
    const int kc = min(TG_KC, (ke - k0 + 15) & ~15);
    int nk_log = 1;
    while ((8 << nk_log) < kc) ++nk_log;
    stage<float>(sA, A, sam, sak, m0, TG_M, M, k0, nk_log, ke);
    stage<TB>(sB, B, sbn, sbk, n0, Nt, N, k0, nk_log, ke);
    async_proxy_fence();
    tc_fence_before();
    __syncthreads();
    if (tid == 0) {
      tc_fence_after();
      const uint32_t sA_addr = (uint32_t)__cvta_generic_to_shared(sA);
      const uint32_t sB_addr = (uint32_t)__cvta_generic_to_shared(sB);
      for (int ks = 0; ks < kc / 16; ++ks) {
        const uint64_t dA = smem_desc(sA_addr + ks * 256, 128, (TG_KC / 8) * 128);
        const uint64_t dB = smem_desc(sB_addr + ks * 256, 128, (TG_KC / 8) * 128);
        umma_bf16(tmem, dA, dB, idesc, (chunk > 0 || ks > 0) ? 1u : 0u);
      }
      umma_commit(&bar[b]);
    }
  }
  // the last commit covers every MMA of the tile
  const int last = max(chunk - 1, 0);
  const bool done = chunk == 0 || vk::mbar_wait(&bar[last % buffers], (uint32_t)(last / buffers) & 1u, TG_WAIT);
  if (!done) atomicOr(&abort_flag, 1);
  __syncthreads();
  if (abort_flag || fail) {
    if (tid == 0) {
      atomicOr(status, VK_STATUS_WAIT_TIMEOUT);
      // the MMAs in flight, once more (bounded), before TMEM is freed
      vk::mbar_wait(&bar[last % buffers], (uint32_t)(last / buffers) & 1u, TG_WAIT);
    }
  } else if (chunk > 0) {
    tc_fence_after();
    // epilogue: warps w and w + 4 hold rows 32 (w % 4).. of the tile (their TMEM lane quarter), every other 16 columns
    const int row = m0 + (warp & 3) * 32 + lane;
    const uint32_t lane_off = (uint32_t)((warp & 3) * 32) << 16;
    const bool split = gridDim.z > 1;
    float* out = split ? ws + ((int64_t)blockIdx.z * M + row) * N + n0 : C + (int64_t)row * scm + (int64_t)n0 * scn;
    const int64_t step = split ? 1 : scn;
    const bool wide = step == 1 && (reinterpret_cast<uintptr_t>(out) & 15) == 0;
    for (int c0 = (warp >> 2) * 16; c0 < Nt; c0 += 32) {
      uint32_t v[16];
      tmem_ld16(tmem + lane_off + (uint32_t)c0, v);
      tmem_wait_ld();
      if (row < M) {
        float x[16];
#pragma unroll
        for (int j = 0; j < 16; ++j) {
          x[j] = __uint_as_float(v[j]);
          if (!split) x[j] = tg_out(x[j], bias, n0 + c0 + j, relu, round_bf16);
        }
        if (wide) {
#pragma unroll
          for (int j = 0; j < 16; j += 4)
            *reinterpret_cast<float4*>(out + c0 + j) = make_float4(x[j], x[j + 1], x[j + 2], x[j + 3]);
        } else {
#pragma unroll
          for (int j = 0; j < 16; ++j) out[(int64_t)(c0 + j) * step] = x[j];
        }
      }
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 0) {
    tc_fence_after();
    tmem_dealloc_warp(tmem, TG_N);
  }
}

// C[m, n] = out(sum over the splits z, in order, of ws[z][m][n])
__global__ void tc_gemm_reduce_k(int M, int N, int splits, const float* __restrict__ ws, const float* bias, int relu,
                                 int round_bf16, float* __restrict__ C, int64_t scm, int64_t scn) {
  const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (i >= (int64_t)M * N) return;
  const int m = (int)(i / N), n = (int)(i % N);
  float s = 0.f;
#pragma unroll 16
  for (int z = 0; z < splits; ++z) s = __fadd_rn(s, ws[(int64_t)z * M * N + i]);
  C[(int64_t)m * scm + (int64_t)n * scn] = tg_out(s, bias, n, relu, round_bf16);
}

// K per split: splits only when the output (in tiles of 128 x 256) would leave most SMs idle.  The split decides the
// order of the FP32 sums, so it does not follow the CTA's tile.
int tc_gemm_k_split(int M, int N, int K) {
  const int tiles = ((M + 127) / 128) * ((N + 255) / 256);
  if (tiles >= 64 || K <= 256) return K;
  int splits = (128 + tiles - 1) / tiles;
  int ks = (K + splits - 1) / splits;
  ks = (ks + 63) / 64 * 64;
  return ks < 64 ? 64 : ks;
}

}  // namespace

extern "C" {

int64_t vk_tc_gemm_ws_floats(int M, int N, int K) {
  if (M <= 0 || N <= 0 || K <= 0) return 0;
  const int ks = tc_gemm_k_split(M, N, K);
  const int splits = (K + ks - 1) / ks;
  return splits > 1 ? (int64_t)splits * M * N : 0;
}

int vk_tc_gemm(int M, int N, int K, const float* A, int64_t sam, int64_t sak, const void* B, int b_bf16, int64_t sbk,
               int64_t sbn, const float* bias, int relu, int round_bf16, float* C, int64_t scm, int64_t scn,
               float* ws, int64_t ws_floats, int32_t* status, void* stream) {
  if (M <= 0 || N <= 0) return 0;
  if (K <= 0 || (N % 16) != 0 || !A || !B || !C || !status) return VK_E_ARG;
  const int ks = tc_gemm_k_split(M, N, K);
  const int splits = (K + ks - 1) / ks;
  if (splits > 1 && (!ws || ws_floats < (int64_t)splits * M * N)) return VK_E_ARG;
  cudaStream_t st = (cudaStream_t)stream;
  dim3 grid((unsigned)((M + TG_M - 1) / TG_M), (unsigned)((N + TG_N - 1) / TG_N), (unsigned)splits);
  const int buffers = ks > TG_KC ? 2 : 1;
  const int smem = buffers * TG_BUF + TG_SLACK;
  if (b_bf16) {
    const int rc = vk_max_smem(tc_gemm_k<__nv_bfloat16>, TG_MOST);
    if (rc != 0) return rc;
    tc_gemm_k<__nv_bfloat16><<<grid, TG_THREADS, smem, st>>>(
        M, N, K, ks, buffers, A, sam, sak, reinterpret_cast<const __nv_bfloat16*>(B), sbk, sbn, bias, relu, round_bf16,
        C, scm, scn, ws, status);
  } else {
    const int rc = vk_max_smem(tc_gemm_k<float>, TG_MOST);
    if (rc != 0) return rc;
    tc_gemm_k<float><<<grid, TG_THREADS, smem, st>>>(M, N, K, ks, buffers, A, sam, sak,
                                                     reinterpret_cast<const float*>(B), sbk, sbn, bias, relu,
                                                     round_bf16, C, scm, scn, ws, status);
  }
  const int rc = vk_launch_status();
  if (rc != 0) return rc;
  if (splits > 1) {
    const int64_t n = (int64_t)M * N;
    tc_gemm_reduce_k<<<(unsigned)((n + 255) / 256), 256, 0, st>>>(M, N, splits, ws, bias, relu, round_bf16, C, scm,
                                                                  scn);
  }
  return vk_launch_status();
}

}  // extern "C"
