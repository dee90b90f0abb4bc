// The two steps either side of the MoE layer inside the reference's block: x_out = x + ffn(ffn_norm(x))
// (models/mla_block.py:83-85, 159) with ffn_norm = RMSNorm (models/normalization.py:25-39).
//
//   rmsnorm_fwd   xn[t] = w * x[t] * rstd[t],  rstd[t] = rsqrt(mean(x[t]^2) + eps)      one read of x, one write of xn
//   add           out = a + b                                                            the residual add
//   rmsnorm_bwd   dx[t] = rstd * (g - x * rstd^2 * mean(g * x)) + d_res[t],  g = d_xn * w     one kernel for the adjoint of the
//                 d_w[d] = sum_t d_xn[t,d] * x[t,d] * rstd[t]                                  norm AND the residual branch
//
// Rows in bf16 or fp32 (the residual stream of mixed-precision training), fp32 arithmetic, one warp per row with the row held
// in registers (D <= 2048).  HBM-bound by design, latency-bound in practice below some 10,000 rows: what counts is that
// every load of a row is in flight at once and that no pass over the activations is spent on a conversion (with fp32 rows
// converted before and after, the norm, its adjoint and the add of a 4,095-row block took 120 us in 11 launches; now four).
// The weight gradient is a two-stage sum in a fixed order (per-warp registers -> the block's warps in order -> per-block
// partials -> final kernel), so it is deterministic; no atomics.
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include "../../include/lmoe.h"
#include "counters.h"

namespace lmoe {

constexpr int kNormWarps = 8;
constexpr int kNormMaxChunks = 8;  // 8-element chunks per lane: D <= 8 * 32 * 8 = 2048
constexpr int kNormMaxBlocks = 296;

__device__ __forceinline__ void nrm_unpack(const uint4& v, float (&f)[8]) {
  const __nv_bfloat162* h = reinterpret_cast<const __nv_bfloat162*>(&v);
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const float2 x = __bfloat1622float2(h[i]);
    f[2 * i] = x.x;
    f[2 * i + 1] = x.y;
  }
}
__device__ __forceinline__ uint4 nrm_pack(const float (&f)[8]) {
  uint4 v;
  __nv_bfloat162* h = reinterpret_cast<__nv_bfloat162*>(&v);
#pragma unroll
  for (int i = 0; i < 4; ++i) h[i] = __floats2bfloat162_rn(f[2 * i], f[2 * i + 1]);
  return v;
}
// Eight consecutive elements of a row in either type, kept as loaded until they are used.
template <bool F32>
struct Chunk {
  uint4 v[F32 ? 2 : 1];
  __device__ __forceinline__ void load(const void* base, long long chunk) {
    const uint4* p = static_cast<const uint4*>(base) + chunk * (F32 ? 2 : 1);
    v[0] = p[0];
    if (F32) v[F32 ? 1 : 0] = p[1];
  }
  __device__ __forceinline__ void get(float (&f)[8]) const {
    if (F32) {
      const float* q = reinterpret_cast<const float*>(v);
#pragma unroll
      for (int j = 0; j < 8; ++j) f[j] = q[F32 ? j : 0];
    } else {
      nrm_unpack(v[0], f);
    }
  }
  // The row as the norm sees it: in bf16, whatever the stream's type.  The router behind the norm decides by score order, so
  // an fp32 stream that was not rounded here would select other experts than the same stream handed over in bf16.
  __device__ __forceinline__ void get_rounded(float (&f)[8]) const {
    get(f);
    if (F32) {
#pragma unroll
      for (int j = 0; j < 8; ++j) f[j] = __bfloat162float(__float2bfloat16_rn(f[j]));
    }
  }
};
template <bool F32>
__device__ __forceinline__ void store_chunk(void* base, long long chunk, const float (&f)[8]) {
  if (F32) {
    float4* p = static_cast<float4*>(base) + chunk * 2;
    p[0] = make_float4(f[0], f[1], f[2], f[3]);
    p[1] = make_float4(f[4], f[5], f[6], f[7]);
  } else {
    static_cast<uint4*>(base)[chunk] = nrm_pack(f);
  }
}
// Eight weights from chunk v of a bf16 or fp32 vector (L1-resident; the type is uniform over the launch).
__device__ __forceinline__ void load_weight(const void* w, bool f32, int v, float (&f)[8]) {
  if (f32) {
    const float4 a = static_cast<const float4*>(w)[2 * v], b = static_cast<const float4*>(w)[2 * v + 1];
    f[0] = a.x, f[1] = a.y, f[2] = a.z, f[3] = a.w, f[4] = b.x, f[5] = b.y, f[6] = b.z, f[7] = b.w;
  } else {
    nrm_unpack(static_cast<const uint4*>(w)[v], f);
  }
}
__device__ __forceinline__ float warp_sum(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

// X32: type of x; Y32: type of xn.  CH chunks per lane cover the row.
// x_keep, w_keep (may be NULL): what the adjoint needs, in buffers of the call's own, so that the stream and a bf16 weight may
// be changed in place before it runs: the rounded row (an fp32 x; the adjoint then reads half the bytes that this writes more)
// and the weight in fp32.
template <bool X32, bool Y32, int CH>
__global__ void __launch_bounds__(kNormWarps * 32)
rmsnorm_fwd_kernel(const void* __restrict__ x, const void* __restrict__ w, bool w32, float eps, long long T, int vec_per_row,
                   void* __restrict__ xn, float* __restrict__ rstd, void* __restrict__ x_keep, float* __restrict__ w_keep) {
  const int lane = threadIdx.x & 31;
  if (w_keep && blockIdx.x == 0)
    for (int v = threadIdx.x; v < vec_per_row; v += blockDim.x) {
      float ww[8];
      load_weight(w, w32, v, ww);
      store_chunk<true>(w_keep, v, ww);
    }
  const float inv_d = 1.0f / static_cast<float>(vec_per_row * 8);
  for (long long t = static_cast<long long>(blockIdx.x) * kNormWarps + (threadIdx.x >> 5); t < T;
       t += static_cast<long long>(gridDim.x) * kNormWarps) {
    Chunk<X32> row[CH];
#pragma unroll
    for (int i = 0; i < CH; ++i)
      if (lane + 32 * i < vec_per_row) row[i].load(x, t * vec_per_row + lane + 32 * i);
    float ss = 0.f;
#pragma unroll
    for (int i = 0; i < CH; ++i)
      if (lane + 32 * i < vec_per_row) {
        float f[8];
        row[i].get_rounded(f);
#pragma unroll
        for (int j = 0; j < 8; ++j) ss = fmaf(f[j], f[j], ss);
      }
    ss = warp_sum(ss);
    const float r = rsqrtf(ss * inv_d + eps);
    if (lane == 0) rstd[t] = r;
#pragma unroll
    for (int i = 0; i < CH; ++i) {
      const int v = lane + 32 * i;
      if (v < vec_per_row) {
        float f[8], ww[8], o[8];
        row[i].get_rounded(f);
        load_weight(w, w32, v, ww);
#pragma unroll
        for (int j = 0; j < 8; ++j) o[j] = ww[j] * (f[j] * r);
        store_chunk<Y32>(xn, t * vec_per_row + v, o);
        if (X32 && x_keep) store_chunk<false>(x_keep, t * vec_per_row + v, f);
      }
    }
  }
}

__global__ void __launch_bounds__(256)
add_bf16_kernel(const uint4* __restrict__ a, const uint4* __restrict__ b, uint4* __restrict__ out, long long n_vec) {
  for (long long i = static_cast<long long>(blockIdx.x) * blockDim.x + threadIdx.x; i < n_vec;
       i += static_cast<long long>(gridDim.x) * blockDim.x) {
    float fa[8], fb[8];
    nrm_unpack(a[i], fa);
    nrm_unpack(b[i], fb);
#pragma unroll
    for (int j = 0; j < 8; ++j) fa[j] += fb[j];
    out[i] = nrm_pack(fa);
  }
}
// out = a + b with a wide stream and bf16 addends: no widened copy of b
__global__ void __launch_bounds__(256)
add_f32_bf16_kernel(const void* __restrict__ a, const void* __restrict__ b, void* __restrict__ out, long long n_vec) {
  for (long long i = static_cast<long long>(blockIdx.x) * blockDim.x + threadIdx.x; i < n_vec;
       i += static_cast<long long>(gridDim.x) * blockDim.x) {
    Chunk<true> ca;
    Chunk<false> cb;
    ca.load(a, i);
    cb.load(b, i);
    float fa[8], fb[8];
    ca.get(fa);
    cb.get(fb);
#pragma unroll
    for (int j = 0; j < 8; ++j) fa[j] += fb[j];
    store_chunk<true>(out, i, fa);
  }
}

// partial[blockIdx.x][D]: this block's share of d_w.  Shared memory: one row of D floats per warp (dynamic).
// X32: type of x; S32: type of the stream's gradients, d_res and dx; G32: type of d_xn.
template <bool X32, bool S32, bool G32, int CH>
__global__ void __launch_bounds__(kNormWarps * 32)
rmsnorm_bwd_kernel(const void* __restrict__ x, const void* __restrict__ w, bool w32, const float* __restrict__ rstd,
                   const void* __restrict__ d_xn, const void* __restrict__ d_res, long long T, int vec_per_row,
                   void* __restrict__ dx, float* __restrict__ partial) {
  extern __shared__ float s_dw[];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int D = vec_per_row * 8;
  const float inv_d = 1.0f / static_cast<float>(D);
  float dw[CH][8];
#pragma unroll
  for (int i = 0; i < CH; ++i)
#pragma unroll
    for (int j = 0; j < 8; ++j) dw[i][j] = 0.f;

  for (long long t = static_cast<long long>(blockIdx.x) * kNormWarps + warp; t < T;
       t += static_cast<long long>(gridDim.x) * kNormWarps) {
    const float r = rstd[t];
    Chunk<X32> xr[CH];
    Chunk<S32> rr[CH];
    Chunk<G32> gr[CH];
#pragma unroll
    for (int i = 0; i < CH; ++i) {
      const int v = lane + 32 * i;
      if (v < vec_per_row) {
        xr[i].load(x, t * vec_per_row + v);
        gr[i].load(d_xn, t * vec_per_row + v);
        if (d_res) rr[i].load(d_res, t * vec_per_row + v);
      }
    }
    float dot = 0.f;
#pragma unroll
    for (int i = 0; i < CH; ++i) {
      const int v = lane + 32 * i;
      if (v < vec_per_row) {
        float fx[8], fg[8], ww[8];
        xr[i].get_rounded(fx);
        gr[i].get(fg);
        load_weight(w, w32, v, ww);
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          dot = fmaf(fg[j] * ww[j], fx[j], dot);
          dw[i][j] = fmaf(fg[j], fx[j] * r, dw[i][j]);
        }
      }
    }
    dot = warp_sum(dot);
    const float c = r * r * r * dot * inv_d;  // rstd^3 * mean(g * x)
#pragma unroll
    for (int i = 0; i < CH; ++i) {
      const int v = lane + 32 * i;
      if (v < vec_per_row) {
        float fx[8], fg[8], ww[8], o[8];
        xr[i].get_rounded(fx);
        gr[i].get(fg);
        load_weight(w, w32, v, ww);
#pragma unroll
        for (int j = 0; j < 8; ++j) o[j] = fg[j] * ww[j] * r - fx[j] * c;
        if (d_res) {
          float fr[8];
          rr[i].get(fr);
#pragma unroll
          for (int j = 0; j < 8; ++j) o[j] += fr[j];
        }
        store_chunk<S32>(dx, t * vec_per_row + v, o);
      }
    }
  }
#pragma unroll
  for (int i = 0; i < CH; ++i) {
    const int v = lane + 32 * i;
    if (v < vec_per_row) {
      float4* q = reinterpret_cast<float4*>(s_dw + warp * D + v * 8);
      q[0] = make_float4(dw[i][0], dw[i][1], dw[i][2], dw[i][3]);
      q[1] = make_float4(dw[i][4], dw[i][5], dw[i][6], dw[i][7]);
    }
  }
  __syncthreads();
  for (int d = threadIdx.x; d < D; d += blockDim.x) {
    float s = s_dw[d];
#pragma unroll
    for (int wi = 1; wi < kNormWarps; ++wi) s += s_dw[wi * D + d];
    partial[static_cast<long long>(blockIdx.x) * D + d] = s;
  }
}

// d_w[d] = sum over the blocks' partials: 32 columns per block, each warp sums a contiguous share of the blocks, then the
// warps' sums are added in order.  (One thread per column over all 296 blocks took 11 us, a chain of dependent loads.)
__global__ void __launch_bounds__(kNormWarps * 32)
rmsnorm_dw_finalize_kernel(const float* __restrict__ partial, int blocks, int D, void* __restrict__ d_w, bool f32) {
  __shared__ float s_sum[kNormWarps][32];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int d = blockIdx.x * 32 + lane;
  const int per = (blocks + kNormWarps - 1) / kNormWarps, b0 = warp * per, b1 = min(b0 + per, blocks);
  float s = 0.f;
  if (d < D) {
#pragma unroll 8
    for (int b = b0; b < b1; ++b) s += partial[static_cast<long long>(b) * D + d];
  }
  s_sum[warp][lane] = s;
  __syncthreads();
  if (warp == 0 && d < D) {
    float v = s_sum[0][lane];
#pragma unroll
    for (int wi = 1; wi < kNormWarps; ++wi) v += s_sum[wi][lane];
    if (f32)
      static_cast<float*>(d_w)[d] = v;
    else
      static_cast<__nv_bfloat16*>(d_w)[d] = __float2bfloat16_rn(v);
  }
}

static inline int norm_blocks(long long T) {
  long long b = (T + kNormWarps - 1) / kNormWarps;
  if (b > kNormMaxBlocks) b = kNormMaxBlocks;
  if (b < 1) b = 1;
  return static_cast<int>(b);
}
static inline int norm_last_error() {
  count_launch();
  cudaError_t e = cudaGetLastError();
  return e == cudaSuccess ? 0 : static_cast<int>(e);
}
static inline bool norm_dims_ok(long long T, int D) {
  return T > 0 && D > 0 && (D & 7) == 0 && D <= kNormMaxChunks * 256;
}
static inline bool aligned16(const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15) == 0; }
static inline bool is_type(int t) { return t == LMOE_BF16 || t == LMOE_F32; }

}  // namespace lmoe

using namespace lmoe;

extern "C" size_t lmoe_rmsnorm_workspace_bytes(int D) {
  return D > 0 ? static_cast<size_t>(kNormMaxBlocks) * D * sizeof(float) : 0;
}

extern "C" int lmoe_rmsnorm_fwd_keep(const void* x, int x_type, const void* weight, int w_type, float eps, int64_t T, int D,
                                     void* xn, int xn_type, float* rstd, void* x_keep, float* w_keep, void* stream) {
  if (!x || !weight || !xn || !rstd || !is_type(x_type) || !is_type(w_type) || !is_type(xn_type)) return LMOE_ERR_ARG;
  if (!norm_dims_ok(T, D)) return LMOE_ERR_SHAPE;
  if (!aligned16(x) || !aligned16(xn) || !aligned16(weight) || !aligned16(x_keep) || !aligned16(w_keep)) return LMOE_ERR_ALIGN;
  auto pick = [&](auto narrow, auto wide) { return D <= 1024 ? narrow : wide; };
  auto k = x_type == LMOE_BF16 ? (xn_type == LMOE_BF16 ? pick(rmsnorm_fwd_kernel<false, false, 4>, rmsnorm_fwd_kernel<false, false, 8>)
                                                       : pick(rmsnorm_fwd_kernel<false, true, 4>, rmsnorm_fwd_kernel<false, true, 8>))
                               : (xn_type == LMOE_BF16 ? pick(rmsnorm_fwd_kernel<true, false, 4>, rmsnorm_fwd_kernel<true, false, 8>)
                                                       : pick(rmsnorm_fwd_kernel<true, true, 4>, rmsnorm_fwd_kernel<true, true, 8>));
  long long blocks = (T + kNormWarps - 1) / kNormWarps;   // no per-block result here: a warp per row up to 16 blocks per SM
  if (blocks > 148 * 16) blocks = 148 * 16;
  k<<<static_cast<int>(blocks), kNormWarps * 32, 0, static_cast<cudaStream_t>(stream)>>>(x, weight, w_type == LMOE_F32, eps, T, D / 8, xn,
                                                                                        rstd, x_keep, w_keep);
  return norm_last_error();
}

extern "C" int lmoe_rmsnorm_fwd_typed(const void* x, int x_type, const void* weight, int w_type, float eps, int64_t T, int D,
                                      void* xn, int xn_type, float* rstd, void* stream) {
  return lmoe_rmsnorm_fwd_keep(x, x_type, weight, w_type, eps, T, D, xn, xn_type, rstd, nullptr, nullptr, stream);
}

extern "C" int lmoe_rmsnorm_fwd(const void* x, const float* weight, float eps, int64_t T, int D, void* xn, float* rstd,
                                void* stream) {
  return lmoe_rmsnorm_fwd_typed(x, LMOE_BF16, weight, LMOE_F32, eps, T, D, xn, LMOE_BF16, rstd, stream);
}

static int add_blocks(long long n_vec) {
  const long long blocks = (n_vec + 255) / 256;
  return static_cast<int>(blocks > 148ll * 16 ? 148ll * 16 : blocks);
}
extern "C" int lmoe_add_bf16(const void* a, const void* b, void* out, int64_t n, void* stream) {
  if (!a || !b || !out) return LMOE_ERR_ARG;
  if (n <= 0 || (n & 7) != 0) return LMOE_ERR_SHAPE;
  if (!aligned16(a) || !aligned16(b) || !aligned16(out)) return LMOE_ERR_ALIGN;
  add_bf16_kernel<<<add_blocks(n / 8), 256, 0, static_cast<cudaStream_t>(stream)>>>(
      static_cast<const uint4*>(a), static_cast<const uint4*>(b), static_cast<uint4*>(out), n / 8);
  return norm_last_error();
}
extern "C" int lmoe_add_f32_bf16(const float* a, const void* b, float* out, int64_t n, void* stream) {
  if (!a || !b || !out) return LMOE_ERR_ARG;
  if (n <= 0 || (n & 7) != 0) return LMOE_ERR_SHAPE;
  if (!aligned16(a) || !aligned16(b) || !aligned16(out)) return LMOE_ERR_ALIGN;
  add_f32_bf16_kernel<<<add_blocks(n / 8), 256, 0, static_cast<cudaStream_t>(stream)>>>(a, b, out, n / 8);
  return norm_last_error();
}

static int rmsnorm_bwd(const void* x, int x_type, const void* weight, int w_type, const float* rstd, const void* d_xn, int g_type,
                       const void* d_residual, int s_type, int64_t T, int D, void* dx, void* d_weight, int dw_type,
                       void* workspace, size_t workspace_bytes, void* stream) {
  if (!x || !weight || !rstd || !d_xn || !dx || !d_weight || !workspace) return LMOE_ERR_ARG;
  if (!is_type(x_type) || !is_type(w_type) || !is_type(g_type) || !is_type(s_type) || !is_type(dw_type)) return LMOE_ERR_ARG;
  if (x_type == LMOE_F32 && s_type != LMOE_F32) return LMOE_ERR_ARG;
  if (!norm_dims_ok(T, D)) return LMOE_ERR_SHAPE;
  if (workspace_bytes < lmoe_rmsnorm_workspace_bytes(D)) return LMOE_ERR_WORKSPACE;
  if (!aligned16(x) || !aligned16(d_xn) || !aligned16(dx) || !aligned16(weight) || (d_residual && !aligned16(d_residual)))
    return LMOE_ERR_ALIGN;
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  auto pick = [&](auto narrow, auto wide) { return D <= 1024 ? narrow : wide; };
  const bool g32 = g_type == LMOE_F32;
  auto k = s_type == LMOE_BF16
               ? (g32 ? pick(rmsnorm_bwd_kernel<false, false, true, 4>, rmsnorm_bwd_kernel<false, false, true, 8>)
                      : pick(rmsnorm_bwd_kernel<false, false, false, 4>, rmsnorm_bwd_kernel<false, false, false, 8>))
               : x_type == LMOE_BF16
                     ? (g32 ? pick(rmsnorm_bwd_kernel<false, true, true, 4>, rmsnorm_bwd_kernel<false, true, true, 8>)
                            : pick(rmsnorm_bwd_kernel<false, true, false, 4>, rmsnorm_bwd_kernel<false, true, false, 8>))
                     : (g32 ? pick(rmsnorm_bwd_kernel<true, true, true, 4>, rmsnorm_bwd_kernel<true, true, true, 8>)
                            : pick(rmsnorm_bwd_kernel<true, true, false, 4>, rmsnorm_bwd_kernel<true, true, false, 8>));
  const size_t smem = static_cast<size_t>(kNormWarps) * D * sizeof(float);   // up to 64 KB
  if (smem > 48 * 1024) {
    const cudaError_t e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(smem));
    if (e != cudaSuccess) return static_cast<int>(e);
  }
  const int blocks = norm_blocks(T);
  k<<<blocks, kNormWarps * 32, smem, st>>>(x, weight, w_type == LMOE_F32, rstd, d_xn, d_residual, T, D / 8, dx,
                                          static_cast<float*>(workspace));
  if (int rc = norm_last_error()) return rc;
  rmsnorm_dw_finalize_kernel<<<(D + 31) / 32, kNormWarps * 32, 0, st>>>(static_cast<const float*>(workspace), blocks, D, d_weight,
                                                                       dw_type == LMOE_F32);
  return norm_last_error();
}

extern "C" int lmoe_rmsnorm_bwd_typed(const void* x, int x_type, const void* weight, int w_type, const float* rstd,
                                      const void* d_xn, int g_type, const void* d_residual, int64_t T, int D, void* dx,
                                      void* d_weight, int dw_type, void* workspace, size_t workspace_bytes, void* stream) {
  return rmsnorm_bwd(x, x_type, weight, w_type, rstd, d_xn, g_type, d_residual, x_type, T, D, dx, d_weight, dw_type, workspace,
                     workspace_bytes, stream);
}

extern "C" int lmoe_rmsnorm_bwd_kept(const void* x_bf16, const void* weight, int w_type, const float* rstd, const void* d_xn,
                                     int g_type, const void* d_residual, int s_type, int64_t T, int D, void* dx, void* d_weight,
                                     int dw_type, void* workspace, size_t workspace_bytes, void* stream) {
  return rmsnorm_bwd(x_bf16, LMOE_BF16, weight, w_type, rstd, d_xn, g_type, d_residual, s_type, T, D, dx, d_weight, dw_type,
                     workspace, workspace_bytes, stream);
}

extern "C" int lmoe_rmsnorm_bwd(const void* x, const float* weight, const float* rstd, const void* d_xn,
                                const void* d_residual, int64_t T, int D, void* dx, float* d_weight, void* workspace,
                                size_t workspace_bytes, void* stream) {
  return lmoe_rmsnorm_bwd_typed(x, LMOE_BF16, weight, LMOE_F32, rstd, d_xn, LMOE_BF16, d_residual, T, D, dx, d_weight, LMOE_F32,
                                workspace, workspace_bytes, stream);
}
