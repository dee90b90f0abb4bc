// FP8 (e4m3) expert path: per-tensor dynamic scaling ("tensorwise": one amax per tensor, scale = 448 / amax,
// q = saturate(x * scale), the recipe named by optimization/fp8_native.py:103-110 of the reference), and the
// grouped expert GEMMs on tcgen05 kind::f8f6f4.  The reference applies this recipe to nn.Linear modules only;
// using it for the routed experts is this path's extension.  A tensor is quantised once and serves every GEMM
// that reads it (forward, dgrad as K-major operand, wgrad as MN-major operand) because the scale is per tensor.
#include <cuda_bf16.h>
#include <cuda_fp8.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include "../../include/lmoe.h"
#include "counters.h"
#include "fp8_device.cuh"
#include "gemm.cuh"
#include "gemm_host.h"
#include "rowops.h"

namespace lmoe {

// Both passes take four 16-byte vectors per thread and iteration (one per iteration kept too few bytes in flight: 600 MB
// of the cast took 190 us = 3.2 TB/s) and up to LMOE_FP8_MAX_TENSORS tensors per launch, one grid row each.
constexpr int kQuantUnroll = 4;
struct Fp8Tensors {
  const uint4* x[LMOE_FP8_MAX_TENSORS];
  uint2* q[LMOE_FP8_MAX_TENSORS];
  long long n_vec[LMOE_FP8_MAX_TENSORS];
  long long vec_per_tile[LMOE_FP8_MAX_TENSORS];
  const int* n_tiles[LMOE_FP8_MAX_TENSORS];
  float* amax[LMOE_FP8_MAX_TENSORS];
  float* deq[LMOE_FP8_MAX_TENSORS];
};
__device__ __forceinline__ long long fp8_vecs(const Fp8Tensors& t, int k) {
  return t.n_tiles[k] ? min(t.n_vec[k], static_cast<long long>(t.n_tiles[k][0]) * t.vec_per_tile[k]) : t.n_vec[k];
}

// block-wide maximum of non-negative values -> atomicMax on the bit pattern (non-negative floats order like integers)
__device__ __forceinline__ void block_amax(float m, float* amax) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, o));
  __shared__ float s[8];
  if ((threadIdx.x & 31) == 0) s[threadIdx.x >> 5] = m;
  __syncthreads();
  if (threadIdx.x == 0) {
    for (int i = 1; i < 8; ++i) m = fmaxf(m, s[i]);
    atomicMax(reinterpret_cast<int*>(amax), __float_as_int(m));
  }
}

// amax[0] = max(amax[0], max |x|); with n_tiles over the first 128 * n_tiles[0] rows.
__global__ void __launch_bounds__(256) amax_kernel(const Fp8Tensors t) {
  const int k = blockIdx.y;
  const long long n = fp8_vecs(t, k);
  const uint4* __restrict__ x = t.x[k];
  float m = 0.f;
  for (long long i0 = static_cast<long long>(blockIdx.x) * 256 * kQuantUnroll + threadIdx.x; i0 < n;
       i0 += static_cast<long long>(gridDim.x) * 256 * kQuantUnroll) {
    uint4 v[kQuantUnroll];
#pragma unroll
    for (int u = 0; u < kQuantUnroll; ++u) v[u] = (i0 + 256 * u < n) ? x[i0 + 256 * u] : make_uint4(0, 0, 0, 0);
#pragma unroll
    for (int u = 0; u < kQuantUnroll; ++u) m = absmax8(v[u], m);
  }
  block_amax(m, t.amax[k]);
}

// q = saturate_e4m3(x * 448 / amax); deq[0] = amax / 448 (1 when the tensor is all zero).
__global__ void __launch_bounds__(256) quantize_kernel(const Fp8Tensors t) {
  const int k = blockIdx.y;
  const long long n = fp8_vecs(t, k);
  const uint4* __restrict__ x = t.x[k];
  uint2* __restrict__ q = t.q[k];
  const float a = t.amax[k][0];
  const float scale = (a > 0.f) ? kE4M3Max / a : 1.0f;
  if (blockIdx.x == 0 && threadIdx.x == 0) t.deq[k][0] = (a > 0.f) ? a / kE4M3Max : 1.0f;
  for (long long i0 = static_cast<long long>(blockIdx.x) * 256 * kQuantUnroll + threadIdx.x; i0 < n;
       i0 += static_cast<long long>(gridDim.x) * 256 * kQuantUnroll) {
    uint4 v[kQuantUnroll];
#pragma unroll
    for (int u = 0; u < kQuantUnroll; ++u) v[u] = (i0 + 256 * u < n) ? x[i0 + 256 * u] : make_uint4(0, 0, 0, 0);
#pragma unroll
    for (int u = 0; u < kQuantUnroll; ++u)
      if (i0 + 256 * u < n) q[i0 + 256 * u] = quantize8(v[u], scale);
  }
}

// amax[0] = max over (token, slot) of |bf16(w[t,k] * d_routed[t,:])|: rounding is monotone and w >= 0, so it is the rounded
// product of the token's largest weight and largest |element| -- no pass over the K rows per token.  One warp per token.
__global__ void __launch_bounds__(256)
amax_weighted_kernel(const uint4* __restrict__ rows, const float* __restrict__ w, int T, int K, int vec_per_row,
                     float* __restrict__ amax) {
  const int lane = threadIdx.x & 31;
  float m = 0.f;
  for (long long t = static_cast<long long>(blockIdx.x) * 8 + (threadIdx.x >> 5); t < T; t += static_cast<long long>(gridDim.x) * 8) {
    float wm = lane < K ? fabsf(w[t * K + lane]) : 0.f;
    float g = 0.f;
    for (int v = lane; v < vec_per_row; v += 32) g = absmax8(rows[t * vec_per_row + v], g);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      wm = fmaxf(wm, __shfl_xor_sync(0xffffffffu, wm, o));
      g = fmaxf(g, __shfl_xor_sync(0xffffffffu, g, o));
    }
    m = fmaxf(m, __bfloat162float(__float2bfloat16_rn(wm * g)));
  }
  block_amax(m, amax);
}

static int fp8_tensors(int count, const lmoe_fp8_tensor* t, bool cast, Fp8Tensors& o, int& blocks) {
  if (count <= 0 || count > LMOE_FP8_MAX_TENSORS || !t) return LMOE_ERR_ARG;
  long long most = 0;
  for (int k = 0; k < count; ++k) {
    if (!t[k].x || !t[k].amax || (cast && (!t[k].q || !t[k].deq)) || t[k].rows <= 0 || t[k].row_len <= 0) return LMOE_ERR_ARG;
    if ((t[k].row_len & 7) != 0) return LMOE_ERR_SHAPE;
    if ((reinterpret_cast<uintptr_t>(t[k].x) & 15) != 0 || (cast && (reinterpret_cast<uintptr_t>(t[k].q) & 7) != 0))
      return LMOE_ERR_ALIGN;
    o.x[k] = static_cast<const uint4*>(t[k].x);
    o.q[k] = static_cast<uint2*>(t[k].q);
    o.n_vec[k] = t[k].rows * (t[k].row_len / 8);
    o.vec_per_tile[k] = static_cast<long long>(LMOE_ROW_PAD) * (t[k].row_len / 8);
    o.n_tiles[k] = t[k].n_tiles;
    o.amax[k] = t[k].amax;
    o.deq[k] = t[k].deq;
    most = o.n_vec[k] > most ? o.n_vec[k] : most;
  }
  const long long b = (most + 256 * kQuantUnroll - 1) / (256 * kQuantUnroll);
  blocks = static_cast<int>(b < 148ll * 8 ? b : 148ll * 8);
  return 0;
}

static inline int fp8_last_error() {
  count_launch();
  cudaError_t e = cudaGetLastError();
  return e == cudaSuccess ? 0 : static_cast<int>(e);
}

}  // namespace lmoe

using namespace lmoe;

extern "C" int lmoe_fp8_amax(int count, const lmoe_fp8_tensor* t, void* stream) {
  Fp8Tensors o = {};
  int blocks = 0;
  if (int rc = fp8_tensors(count, t, false, o, blocks)) return rc;
  amax_kernel<<<dim3(blocks, count), 256, 0, static_cast<cudaStream_t>(stream)>>>(o);
  return fp8_last_error();
}

extern "C" int lmoe_fp8_cast(int count, const lmoe_fp8_tensor* t, void* stream) {
  Fp8Tensors o = {};
  int blocks = 0;
  if (int rc = fp8_tensors(count, t, true, o, blocks)) return rc;
  quantize_kernel<<<dim3(blocks, count), 256, 0, static_cast<cudaStream_t>(stream)>>>(o);
  return fp8_last_error();
}

extern "C" int lmoe_fp8_quantize(const void* x_bf16, int64_t rows, int row_len, const int32_t* n_tiles_dev, void* q_e4m3,
                                 float* amax, float* deq, void* stream) {
  if (!x_bf16 || !q_e4m3 || !amax || !deq || rows <= 0 || row_len <= 0) return LMOE_ERR_ARG;
  cudaError_t e = cudaMemsetAsync(amax, 0, sizeof(float), static_cast<cudaStream_t>(stream));
  if (e != cudaSuccess) return static_cast<int>(e);
  const lmoe_fp8_tensor t = {x_bf16, q_e4m3, rows, row_len, n_tiles_dev, amax, deq};
  if (int rc = lmoe_fp8_amax(1, &t, stream)) return rc;
  return lmoe_fp8_cast(1, &t, stream);
}

extern "C" int lmoe_fp8_combine_bwd(const lmoe_shape* s, const void* d_routed, const void* y_sorted, const float* weights,
                                    const lmoe_route* r, float* amax, float* deq, void* d_y_q, float* d_weights, void* stream) {
  if (!s || !d_routed || !y_sorted || !weights || !r || !amax || !deq || !d_y_q || !d_weights) return LMOE_ERR_ARG;
  if (s->T <= 0 || s->K <= 0 || s->K > 32 || (s->L & 7) != 0) return LMOE_ERR_SHAPE;
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  const long long b = (static_cast<long long>(s->T) + 7) / 8;
  amax_weighted_kernel<<<static_cast<int>(b < 148 * 8 ? b : 148 * 8), 256, 0, st>>>(static_cast<const uint4*>(d_routed), weights, s->T,
                                                                                    s->K, s->L / 8, amax);
  if (int rc = fp8_last_error()) return rc;
  return combine_bwd_tokens(s, d_routed, y_sorted, weights, r, d_y_q, d_weights, amax, deq, st);
}

// Generic e4m3 GEMM (test hook): C[M,N] bf16 = deq_a * deq_b * A_q[M,K] * B_q[N,K]^T.
extern "C" int lmoe_gemm_fp8(int M, int N, int K, const void* A, int64_t lda, int a_mn, const void* B, int64_t ldb,
                             int b_mn, const float* deq_a, const float* deq_b, void* C, int64_t ldc, int32_t* status,
                             void* stream) {
  if (!A || !B || !C || M <= 0 || N <= 0 || K <= 0) return LMOE_ERR_ARG;
  GemmCall c;
  c.esz = 1;
  c.a_mn = a_mn ? 1 : 0;
  c.b_mn = b_mn ? 1 : 0;
  c.epi = EPI_BF16;
  c.grp = GRP_NONE;
  c.A[0] = A;
  c.lda[0] = lda;
  c.B[0] = B;
  c.ldb[0] = ldb;
  c.Kseg[0] = K;
  c.M = M;
  c.N = N;
  c.C = C;
  c.ldc = ldc;
  c.deq_a = deq_a;
  c.deq_b = deq_b;
  c.status = status;
  c.stream = static_cast<cudaStream_t>(stream);
  return launch_gemm(c);
}

// Routed gate_up in e4m3 with the SwiGLU epilogue: h1 = deq * xq * Wq[e], hidden = silu(gate) * up (both bf16).
extern "C" int lmoe_grouped_gateup_fp8(int64_t P, int E, int L, int F, const void* xq, const void* wq, const float* deq_x,
                                       const float* deq_w, const int32_t* tile_expert, const int32_t* n_tiles, void* h1,
                                       void* hidden, int32_t* status, void* stream) {
  return lmoe_grouped_gateup_fp8_amax(P, E, L, F, xq, wq, deq_x, deq_w, tile_expert, n_tiles, h1, hidden, nullptr, status, stream);
}

// ... and the maximum of |hidden| on the way (amax_hidden[0] = max(amax_hidden[0], .)), for its quantisation.
extern "C" int lmoe_grouped_gateup_fp8_amax(int64_t P, int E, int L, int F, const void* xq, const void* wq, const float* deq_x,
                                            const float* deq_w, const int32_t* tile_expert, const int32_t* n_tiles, void* h1,
                                            void* hidden, float* amax_hidden, int32_t* status, void* stream) {
  if (!xq || !wq || !deq_x || !deq_w || !tile_expert || !n_tiles || !hidden) return LMOE_ERR_ARG;
  if (P <= 0 || (P % LMOE_ROW_PAD) != 0 || E <= 0 || (L % 128) != 0 || (F % 128) != 0) return LMOE_ERR_SHAPE;
  GemmCall a;
  a.esz = 1;
  a.a_mn = 0;
  a.b_mn = 1;
  a.epi = EPI_SWIGLU;
  a.grp = GRP_M;
  a.A[0] = xq;
  a.lda[0] = L;
  a.B[0] = wq;
  a.ldb[0] = 2ll * F;
  a.Kseg[0] = L;
  a.M = static_cast<int>(P);
  a.N = F;
  a.C = h1;
  a.ldc = 2ll * F;
  a.C2 = hidden;
  a.ldc2 = F;
  a.padded_rows = P;
  a.groups = E;
  a.b_group_rows = L;
  a.tile_expert = tile_expert;
  a.n_m_tiles = n_tiles;
  a.deq_a = deq_x;
  a.deq_b = deq_w;
  a.status = status;
  a.stream = static_cast<cudaStream_t>(stream);
  a.amax = amax_hidden;
  return launch_gemm(a);
}

// Grouped-by-rows e4m3 GEMM: out[P,N] bf16 = deq * aq[P,K] * Bq[e], Bq stacked per expert either [E*K, N]
// (b_mn = 1, the forward layout of the expert weights) or [E*N, K] (b_mn = 0, the same weights read as dgrad operand).
extern "C" int lmoe_grouped_rows_fp8(int64_t P, int E, int K, int N, const void* aq, const void* bq, int b_mn,
                                     const float* deq_a, const float* deq_b, const int32_t* tile_expert,
                                     const int32_t* n_tiles, void* out, int32_t* status, void* stream) {
  if (!aq || !bq || !deq_a || !deq_b || !tile_expert || !n_tiles || !out) return LMOE_ERR_ARG;
  if (P <= 0 || (P % LMOE_ROW_PAD) != 0 || E <= 0 || (K % 128) != 0 || (N % 16) != 0) return LMOE_ERR_SHAPE;
  GemmCall a;
  a.esz = 1;
  a.a_mn = 0;
  a.b_mn = b_mn ? 1 : 0;
  a.epi = EPI_BF16;
  a.grp = GRP_M;
  a.A[0] = aq;
  a.lda[0] = K;
  a.B[0] = bq;
  a.ldb[0] = b_mn ? N : K;
  a.Kseg[0] = K;
  a.M = static_cast<int>(P);
  a.N = N;
  a.C = out;
  a.ldc = N;
  a.padded_rows = P;
  a.groups = E;
  a.b_group_rows = b_mn ? K : N;
  a.tile_expert = tile_expert;
  a.n_m_tiles = n_tiles;
  a.deq_a = deq_a;
  a.deq_b = deq_b;
  a.status = status;
  a.stream = static_cast<cudaStream_t>(stream);
  return launch_gemm(a);
}

// d_h1 = swiglu'(h1, deq * dyq * Wdq[e]^T) with the adjoint in the epilogue (d_hidden never reaches memory), and the maximum
// of |d_h1| on the way.  The separate form (GEMM, streaming adjoint, amax pass) took 221 + 742 + 250 us at 1.57 M rows.
extern "C" int lmoe_grouped_swiglu_bwd_fp8(int64_t P, int E, int L, int F, const void* dyq, const void* wdq, const float* deq_dy,
                                           const float* deq_wd, const int32_t* tile_expert, const int32_t* n_tiles, const void* h1,
                                           void* d_h1, float* amax_d_h1, int32_t* status, void* stream) {
  if (!dyq || !wdq || !deq_dy || !deq_wd || !tile_expert || !n_tiles || !h1 || !d_h1) return LMOE_ERR_ARG;
  if (P <= 0 || (P % LMOE_ROW_PAD) != 0 || E <= 0 || (L % 128) != 0 || (F % 128) != 0) return LMOE_ERR_SHAPE;
  GemmCall a;
  a.esz = 1;
  a.a_mn = 0;
  a.b_mn = 0;
  a.epi = EPI_SWIGLU_BWD;
  a.grp = GRP_M;
  a.A[0] = dyq;
  a.lda[0] = L;
  a.B[0] = wdq;
  a.ldb[0] = L;
  a.Kseg[0] = L;
  a.M = static_cast<int>(P);
  a.N = F;
  a.C = d_h1;
  a.ldc = 2ll * F;
  a.aux = h1;
  a.ld_aux = 2ll * F;
  a.padded_rows = P;
  a.groups = E;
  a.b_group_rows = F;
  a.tile_expert = tile_expert;
  a.n_m_tiles = n_tiles;
  a.deq_a = deq_dy;
  a.deq_b = deq_wd;
  a.exact_sigmoid = true;
  a.amax = amax_d_h1;
  a.status = status;
  a.stream = static_cast<cudaStream_t>(stream);
  return launch_gemm(a);
}

// Grouped-by-contraction e4m3 GEMM (expert weight gradients): out[e][M,N] bf16 = deq * aq[rows_e, M]^T * bq[rows_e, N].
extern "C" int lmoe_grouped_wgrad_fp8(int64_t P, int E, int M, int N, const void* aq, const void* bq, const float* deq_a,
                                      const float* deq_b, const int32_t* pad_offsets, void* out, int32_t* status,
                                      void* stream) {
  if (!aq || !bq || !deq_a || !deq_b || !pad_offsets || !out) return LMOE_ERR_ARG;
  if (P <= 0 || (P % LMOE_ROW_PAD) != 0 || E <= 0 || (M % 16) != 0 || (N % 16) != 0) return LMOE_ERR_SHAPE;
  GemmCall a;
  a.esz = 1;
  a.a_mn = 1;
  a.b_mn = 1;
  a.epi = EPI_BF16;
  a.grp = GRP_K;
  a.A[0] = aq;
  a.lda[0] = M;
  a.B[0] = bq;
  a.ldb[0] = N;
  a.M = M;
  a.N = N;
  a.C = out;
  a.ldc = N;
  a.c_group_stride = static_cast<long long>(M) * N;
  a.padded_rows = P;
  a.groups = E;
  a.pad_offsets = pad_offsets;
  a.deq_a = deq_a;
  a.deq_b = deq_b;
  a.status = status;
  a.stream = static_cast<cudaStream_t>(stream);
  return launch_gemm(a);
}
