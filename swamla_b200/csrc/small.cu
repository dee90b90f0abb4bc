// Forward of a few tokens (generation): at most kFewTokens rows, no backward.
//
// What bounds it: the weights (12 MB for one token of the 1,024-wide layer with 12 of 128 experts: 2 us of HBM, less from L2)
// and, far above that, latency: the padded tensor-core path needs nine dependent launches of 4-10 us each (56 us), most of
// it pipeline set-up for tiles of 128 rows that hold one.  Here the call is four kernels whose CTAs are cut along the WEIGHT
// rows, so that every SM pulls a share of the weights with plain 16-byte loads that are all in flight at once:
//   in      router logits and selection (one cluster of eight CTAs, then a warp per token), latent projection, shared expert's
//           gate/up with SwiGLU: 16 weight rows per CTA against all tokens on mma.sync (m16n8k16: the weight rows are M, the
//           tokens N; tensor memory tiles start at 128 rows)
//   rows x2 routed experts: a CTA owns one expert's slice of columns, finds the expert's tokens itself, keeps the slice in
//           registers and multiplies it with every one of them; no permutation, no padding
//   out     weighted combine, up-projection, shared down-projection, z-loss
// The last three are launched with programmatic stream serialisation: they are resident when their predecessor ends, and the
// output kernel has its weights in registers by then (the weights are older than the first kernel, which is not).
// Rounding points are those of the padded path (bf16 latents, gate/up, hidden, expert outputs, routed); sums are fp32 in
// another order.
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include "../../include/lmoe.h"
#include "common/ptx.cuh"
#include "counters.h"
#include "device_once.h"
#include "gemm.cuh"
#include "topk.cuh"

namespace lmoe {

constexpr int kFewTokens = LMOE_FEW_TOKENS;
constexpr int kFewThreads = 256;
constexpr int kFewWarps = kFewThreads / 32;
constexpr int kFewCluster = 8;

__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void pdl_launch() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }

__device__ __forceinline__ float bf_lo(uint32_t v) { return __uint_as_float(v << 16); }
__device__ __forceinline__ float bf_hi(uint32_t v) { return __uint_as_float(v & 0xffff0000u); }

__device__ __forceinline__ void mma_16816(float (&d)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0,
                                          uint32_t b1) {
  asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"
               : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
               : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}
// One 32-wide step of the contraction for 16 weight rows and 8 tokens.  A lane holds eight CONSECUTIVE k of rows g and g + 8
// and of token g (one 16-byte load each); the contraction index is the same permutation of the 32 k on both sides.
__device__ __forceinline__ void mma_step(float (&d)[4], const uint4& ra, const uint4& rb, const uint4& x) {
  mma_16816(d, ra.x, rb.x, ra.y, rb.y, x.x, x.y);
  mma_16816(d, ra.z, rb.z, ra.w, rb.w, x.z, x.w);
}

// Sum over the CTA's warps of 16 x (8 NT) partial products, fixed order: red[warp][row][token].
template <int NT>
__device__ __forceinline__ void store_partial(float* red, int warp, int lane, const float (&acc)[NT][4]) {
  const int g = lane >> 2, t = lane & 3;
  float* p = red + warp * (16 * 8 * NT);
#pragma unroll
  for (int n = 0; n < NT; ++n) {
    *reinterpret_cast<float2*>(p + g * (8 * NT) + n * 8 + 2 * t) = make_float2(acc[n][0], acc[n][1]);
    *reinterpret_cast<float2*>(p + (g + 8) * (8 * NT) + n * 8 + 2 * t) = make_float2(acc[n][2], acc[n][3]);
  }
}
template <int NT>
__device__ __forceinline__ float sum_partial(const float* red, int row, int tok) {
  float s = 0.f;
#pragma unroll
  for (int w = 0; w < kFewWarps; ++w) s += red[w * (16 * 8 * NT) + row * (8 * NT) + tok];
  return s;
}

struct FewParams {
  const __nv_bfloat16 *x, *wg, *wdn, *wup, *wgus, *wds, *wgu, *wde;
  const float* bias;
  int T, D, L, E, K, F, Fs;   // L: width the experts work at (D without a latent projection: wdn, wup NULL)
  float* logits;              // [T, E]
  __nv_bfloat16* x_latent;    // [T, L]
  __nv_bfloat16* hidden_s;    // [T, Fs]
  __nv_bfloat16* hidden;      // [T*K, F]
  __nv_bfloat16* y_slot;      // [T*K, L]
  int* sel;                   // [T, K]
  float *weights, *lse;       // [T, K], [T]
  float z_scale;              // z_loss = z_scale * sum lse^2
  float* z_loss;
  __nv_bfloat16* y;           // [T, D]
};

// 16 weight rows (lane's two row pointers) against all tokens over D.
template <int NT>
__device__ __forceinline__ void rows_times_x(const __nv_bfloat16* row_a, const __nv_bfloat16* row_b, const __nv_bfloat16* x, int T,
                                             int D, int warp, int lane, float (&acc)[NT][4]) {
  const int g = lane >> 2, t = lane & 3, chunks = D / 32;
#pragma unroll
  for (int n = 0; n < NT; ++n)
#pragma unroll
    for (int i = 0; i < 4; ++i) acc[n][i] = 0.f;
  constexpr int U = 4;
  for (int c0 = warp; c0 < chunks; c0 += U * kFewWarps) {
    uint4 a[U], b[U];
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const int c = c0 + u * kFewWarps;
      a[u] = b[u] = make_uint4(0, 0, 0, 0);
      if (c < chunks) {
        a[u] = __ldg(reinterpret_cast<const uint4*>(row_a + c * 32 + t * 8));
        b[u] = __ldg(reinterpret_cast<const uint4*>(row_b + c * 32 + t * 8));
      }
    }
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const int c = c0 + u * kFewWarps;
      if (c >= chunks) break;
#pragma unroll
      for (int n = 0; n < NT; ++n) {
        const int tok = n * 8 + g;
        const uint4 xv = tok < T ? __ldg(reinterpret_cast<const uint4*>(x + static_cast<long long>(tok) * D + c * 32 + t * 8))
                                 : make_uint4(0, 0, 0, 0);
        mma_step(acc[n], a[u], b[u], xv);
      }
    }
  }
}

template <int NT, int PER>
__global__ void __cluster_dims__(kFewCluster, 1, 1) __launch_bounds__(kFewThreads) few_in_kernel(const FewParams p) {
  __shared__ float red[kFewWarps * 16 * 8 * NT];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2;
  pdl_launch();
  float acc[NT][4];
  if (blockIdx.x < kFewCluster) {
    // ---- router: the cluster's CTAs take the expert groups in turn, then a warp per token
    for (int grp = blockIdx.x; grp * 16 < p.E; grp += kFewCluster) {
      const int ra = min(grp * 16 + g, p.E - 1), rb = min(grp * 16 + g + 8, p.E - 1);
      rows_times_x<NT>(p.wg + static_cast<long long>(ra) * p.D, p.wg + static_cast<long long>(rb) * p.D, p.x, p.T, p.D, warp, lane, acc);
      store_partial<NT>(red, warp, lane, acc);
      __syncthreads();
      for (int i = threadIdx.x; i < 16 * p.T; i += kFewThreads) {
        const int e = grp * 16 + (i & 15), tok = i >> 4;
        if (e < p.E) p.logits[tok * p.E + e] = sum_partial<NT>(red, i & 15, tok);
      }
      __syncthreads();
    }
    cluster_sync_all();  // every CTA's logits are visible to the cluster
    for (int t = blockIdx.x * kFewWarps + warp; t < p.T; t += kFewCluster * kFewWarps) {
      int idx;
      float aff, aff_sum, lse;
      topk_row<PER>(p.logits + t * p.E, p.bias, p.E, p.K, lane, idx, aff, aff_sum, lse);
      if (lane == 0) p.lse[t] = lse;
      if (lane < p.K) {
        p.sel[t * p.K + lane] = idx;
        p.weights[t * p.K + lane] = aff / (aff_sum + 1e-9f);
      }
    }
    return;
  }
  const int lat_units = p.wdn ? p.L / 16 : 0, units = lat_units + p.Fs / 8;
  for (int u = blockIdx.x - kFewCluster; u < units; u += gridDim.x - kFewCluster) {
    const bool latent = u < lat_units;
    const int su = u - lat_units;
    // latent: 16 rows of the down-projection; shared: 8 gate rows and the 8 up rows of the same hidden columns
    const __nv_bfloat16* ra = latent ? p.wdn + static_cast<long long>(u * 16 + g) * p.D : p.wgus + static_cast<long long>(su * 8 + g) * p.D;
    const __nv_bfloat16* rb = latent ? ra + 8ll * p.D : p.wgus + static_cast<long long>(p.Fs + su * 8 + g) * p.D;
    rows_times_x<NT>(ra, rb, p.x, p.T, p.D, warp, lane, acc);
    store_partial<NT>(red, warp, lane, acc);
    __syncthreads();
    if (latent) {
      for (int i = threadIdx.x; i < 16 * p.T; i += kFewThreads)
        p.x_latent[static_cast<long long>(i >> 4) * p.L + u * 16 + (i & 15)] = __float2bfloat16_rn(sum_partial<NT>(red, i & 15, i >> 4));
    } else {
      for (int i = threadIdx.x; i < 8 * p.T; i += kFewThreads) {
        const int r = i & 7, tok = i >> 3;
        const float gate = bf16_round(sum_partial<NT>(red, r, tok)), up = bf16_round(sum_partial<NT>(red, r + 8, tok));
        p.hidden_s[static_cast<long long>(tok) * p.Fs + su * 8 + r] = __float2bfloat16_rn(silu_f(gate) * up);
      }
    }
    __syncthreads();
  }
}

// Routed experts.  GATE_UP: hidden[slot, f] = silu(gate) * up with W = Wgu[e] [L, 2F]: 32 hidden columns per CTA (four 16-byte
// vectors of gate columns, four of up columns).  Otherwise y_slot[slot, c] = hidden[slot, :] * Wd[e] [F, L]: 64 columns per CTA.
// A thread owns one vector of 8 columns and kRowsPerThread rows of the contraction; its slice of W stays in registers for
// all tokens of the expert.  CUDA-core FMAs: an expert has one or two tokens (T*K / E), a matrix instruction would idle on
// the other rows.
constexpr int kRowsPerThread = 8;
constexpr int kRowGroups = kFewThreads / 8;             // groups of rows walked side by side
constexpr int kTokBatch = 4;

template <bool GATE_UP>
__global__ void __launch_bounds__(kFewThreads) few_expert_kernel(const FewParams p) {
  __shared__ int s_slot[kFewTokens];
  __shared__ int s_n;
  __shared__ float red[kFewWarps][kTokBatch][64];
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  pdl_launch();
  pdl_wait();
  const int slots = p.T * p.K;
  // ---- which expert: block x owns an expert, or, with fewer slots than experts, the slot that names it first
  int e = blockIdx.x;
  if (tid == 0) s_n = 0;
  if (slots < p.E) {
    e = p.sel[blockIdx.x];
    int earlier = 0;
    for (int i = tid; i < static_cast<int>(blockIdx.x); i += kFewThreads) earlier |= p.sel[i] == e;
    if (__syncthreads_or(earlier)) return;
  } else {
    __syncthreads();
  }
  if (warp == 0) {  // its slots, in order
    int n = 0;
    for (int i0 = 0; i0 < slots; i0 += 32) {
      const bool mine = i0 + lane < slots && p.sel[i0 + lane] == e;
      const unsigned m = __ballot_sync(0xffffffffu, mine);
      if (mine) s_slot[n + __popc(m & ((1u << lane) - 1u))] = i0 + lane;  // at most one per token: n <= kFewTokens
      n += __popc(m);
    }
    if (lane == 0) s_n = n;
  }
  __syncthreads();
  const int n = s_n;
  if (n == 0) return;

  const int kdim = GATE_UP ? p.L : p.F, ncols = GATE_UP ? 2 * p.F : p.L;
  const __nv_bfloat16* W = (GATE_UP ? p.wgu : p.wde) + static_cast<long long>(e) * kdim * ncols;
  const __nv_bfloat16* in = GATE_UP ? (p.wdn ? p.x_latent : p.x) : p.hidden;
  const int vec = tid & 7, rg = tid >> 3;
  const int col = GATE_UP ? ((vec < 4 ? 0 : p.F) + blockIdx.y * 32 + (vec & 3) * 8) : (blockIdx.y * 64 + vec * 8);
  constexpr int kSpan = kRowGroups * kRowsPerThread;   // rows of the contraction per pass: 256
  for (int b0 = 0; b0 < n; b0 += kTokBatch) {
    float acc[kTokBatch][8];
#pragma unroll
    for (int b = 0; b < kTokBatch; ++b)
#pragma unroll
      for (int j = 0; j < 8; ++j) acc[b][j] = 0.f;
    for (int k0 = rg * kRowsPerThread; k0 < kdim; k0 += kSpan) {
      uint4 w[kRowsPerThread];   // (one pass and further batches: the loads hit L1)
#pragma unroll
      for (int r = 0; r < kRowsPerThread; ++r) w[r] = __ldg(reinterpret_cast<const uint4*>(W + static_cast<long long>(k0 + r) * ncols + col));
#pragma unroll
      for (int b = 0; b < kTokBatch; ++b) {
        if (b0 + b >= n) break;
        const int slot = s_slot[b0 + b];
        const long long row = GATE_UP ? slot / p.K : slot;
        const uint4 xv = *reinterpret_cast<const uint4*>(in + row * kdim + k0);
        const uint32_t xw[4] = {xv.x, xv.y, xv.z, xv.w};
#pragma unroll
        for (int r = 0; r < kRowsPerThread; ++r) {
          const float xr = (r & 1) ? bf_hi(xw[r >> 1]) : bf_lo(xw[r >> 1]);
          const uint32_t ww[4] = {w[r].x, w[r].y, w[r].z, w[r].w};
#pragma unroll
          for (int j = 0; j < 4; ++j) {
            acc[b][2 * j] = fmaf(xr, bf_lo(ww[j]), acc[b][2 * j]);
            acc[b][2 * j + 1] = fmaf(xr, bf_hi(ww[j]), acc[b][2 * j + 1]);
          }
        }
      }
    }
    // over the four row groups of a warp, then over the warps (fixed order)
#pragma unroll
    for (int b = 0; b < kTokBatch; ++b) {
      if (b0 + b >= n) break;
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        float v = acc[b][j];
        v += __shfl_xor_sync(0xffffffffu, v, 8);
        v += __shfl_xor_sync(0xffffffffu, v, 16);
        if (lane < 8) red[warp][b][vec * 8 + j] = v;
      }
    }
    __syncthreads();
    constexpr int kOut = GATE_UP ? 32 : 64;
    for (int i = tid; i < kOut * min(kTokBatch, n - b0); i += kFewThreads) {
      const int b = i / kOut, c = i - b * kOut, slot = s_slot[b0 + b];
      float s0 = 0.f, s1 = 0.f;
#pragma unroll
      for (int w = 0; w < kFewWarps; ++w) {
        s0 += red[w][b][c];
        if (GATE_UP) s1 += red[w][b][c + 32];
      }
      if (GATE_UP) {
        const float gate = bf16_round(s0), up = bf16_round(s1);
        p.hidden[static_cast<long long>(slot) * p.F + blockIdx.y * 32 + c] = __float2bfloat16_rn(silu_f(gate) * up);
      } else {
        p.y_slot[static_cast<long long>(slot) * p.L + blockIdx.y * 64 + c] = __float2bfloat16_rn(s0);
      }
    }
    __syncthreads();
  }
}

// y = hidden_s * Wd_s^T + routed * Wup^T (16 output columns per CTA), routed = sum_k w_k y_slot.  Without an up-projection the
// weighted sum is added to the shared expert's output instead, which is rounded first as the separate GEMM's result is.
template <int NT>
__global__ void __launch_bounds__(kFewThreads) few_out_kernel(const FewParams p) {
  extern __shared__ uint4 s_routed[];                   // [T][L] bf16 (latent form only)
  __shared__ float red[kFewWarps * 16 * 8 * NT];
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, g = lane >> 2, t = lane & 3;
  const int c_s = p.Fs / 32, chunks = c_s + (p.wup ? p.L / 32 : 0);
  const int row = blockIdx.x * 16;
  constexpr int U = 5;
  uint4 a[U], b[U];
  auto load = [&](int c, uint4& va, uint4& vb) {
    const __nv_bfloat16* base = c < c_s ? p.wds + static_cast<long long>(row + g) * p.Fs + c * 32 + t * 8
                                        : p.wup + static_cast<long long>(row + g) * p.L + (c - c_s) * 32 + t * 8;
    va = __ldg(reinterpret_cast<const uint4*>(base));
    vb = row + g + 8 < p.D ? __ldg(reinterpret_cast<const uint4*>(base + 8ll * (c < c_s ? p.Fs : p.L))) : make_uint4(0, 0, 0, 0);
  };
#pragma unroll
  for (int u = 0; u < U; ++u)
    if (warp + u * kFewWarps < chunks) load(warp + u * kFewWarps, a[u], b[u]);
  pdl_wait();
  if (p.wup) {
    const int vecs = p.L / 8;
    for (int i = tid; i < p.T * vecs; i += kFewThreads) {
      const int tok = i / vecs, v = i - tok * vecs;
      float acc[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
      for (int k0 = 0; k0 < p.K; k0 += 4) {
        uint4 yv[4];
        float wk[4];
#pragma unroll
        for (int u = 0; u < 4; ++u) {
          const int s = tok * p.K + min(k0 + u, p.K - 1);
          yv[u] = *reinterpret_cast<const uint4*>(p.y_slot + static_cast<long long>(s) * p.L + v * 8);
          wk[u] = k0 + u < p.K ? p.weights[s] : 0.f;
        }
#pragma unroll
        for (int u = 0; u < 4; ++u) {
          const uint32_t yw[4] = {yv[u].x, yv[u].y, yv[u].z, yv[u].w};
#pragma unroll
          for (int j = 0; j < 4; ++j) {
            acc[2 * j] = fmaf(wk[u], bf_lo(yw[j]), acc[2 * j]);
            acc[2 * j + 1] = fmaf(wk[u], bf_hi(yw[j]), acc[2 * j + 1]);
          }
        }
      }
      s_routed[i] = make_uint4(pack_bf16x2(acc[0], acc[1]), pack_bf16x2(acc[2], acc[3]), pack_bf16x2(acc[4], acc[5]),
                               pack_bf16x2(acc[6], acc[7]));
    }
    __syncthreads();
  }
  float acc[NT][4];
#pragma unroll
  for (int n = 0; n < NT; ++n)
#pragma unroll
    for (int i = 0; i < 4; ++i) acc[n][i] = 0.f;
  const __nv_bfloat16* routed = reinterpret_cast<const __nv_bfloat16*>(s_routed);
  for (int u0 = 0; warp + u0 * kFewWarps < chunks; u0 += U) {
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const int c = warp + (u0 + u) * kFewWarps;
      if (c >= chunks) break;
      if (u0 > 0) load(c, a[u], b[u]);
#pragma unroll
      for (int n = 0; n < NT; ++n) {
        const int tok = n * 8 + g;
        uint4 xv = make_uint4(0, 0, 0, 0);
        if (tok < p.T)
          xv = c < c_s ? *reinterpret_cast<const uint4*>(p.hidden_s + static_cast<long long>(tok) * p.Fs + c * 32 + t * 8)
                       : *reinterpret_cast<const uint4*>(routed + tok * p.L + (c - c_s) * 32 + t * 8);
        mma_step(acc[n], a[u], b[u], xv);
      }
    }
  }
  store_partial<NT>(red, warp, lane, acc);
  __syncthreads();
  for (int i = tid; i < 16 * p.T; i += kFewThreads) {
    const int c = i & 15, tok = i >> 4;
    if (row + c >= p.D) continue;
    float v = sum_partial<NT>(red, c, tok);
    if (!p.wup) {
      v = bf16_round(v);
      for (int k = 0; k < p.K; ++k)
        v = fmaf(p.weights[tok * p.K + k], __bfloat162float(p.y_slot[static_cast<long long>(tok * p.K + k) * p.L + row + c]), v);
    }
    p.y[static_cast<long long>(tok) * p.D + row + c] = __float2bfloat16_rn(v);
  }
  if (blockIdx.x == 0 && warp == 0) {
    double z = 0.0;
    for (int i = lane; i < p.T; i += 32) z += static_cast<double>(p.lse[i]) * static_cast<double>(p.lse[i]);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) z += __shfl_xor_sync(0xffffffffu, z, o);
    if (lane == 0) p.z_loss[0] = static_cast<float>(z * static_cast<double>(p.z_scale));
  }
}

template <typename Kernel>
static int few_launch(Kernel kernel, dim3 grid, size_t smem, bool after, const FewParams& p, cudaStream_t st) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = dim3(kFewThreads);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cudaLaunchAttribute attr;
  attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr.val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = &attr;
  cfg.numAttrs = after ? 1 : 0;
  count_launch();
  const cudaError_t e = cudaLaunchKernelEx(&cfg, kernel, p);
  return e == cudaSuccess ? 0 : static_cast<int>(e);
}

template <int NT>
static int few_forward(const FewParams& p, cudaStream_t st) {
  const int units = (p.wdn ? p.L / 16 : 0) + p.Fs / 8;
  const int cap = 512;  // two rounds of 256-thread CTAs over the SMs' slots at most; the rest loops
  const int rest = ((units < cap ? units : cap) + kFewCluster - 1) / kFewCluster * kFewCluster;
  auto in = p.E <= 32 ? few_in_kernel<NT, 1> : p.E <= 64 ? few_in_kernel<NT, 2> : p.E <= 128 ? few_in_kernel<NT, 4> : few_in_kernel<NT, 8>;
  if (int rc = few_launch(in, dim3(kFewCluster + rest), 0, false, p, st)) return rc;
  const int owners = p.T * p.K < p.E ? p.T * p.K : p.E;
  if (int rc = few_launch(few_expert_kernel<true>, dim3(owners, p.F / 32), 0, true, p, st)) return rc;
  if (int rc = few_launch(few_expert_kernel<false>, dim3(owners, p.L / 64), 0, true, p, st)) return rc;
  const size_t smem = p.wup ? static_cast<size_t>(p.T) * p.L * 2 : 0;
  if (smem > 0) {  // with the static partial sums beyond the default limit of 48 KB
    static PerDeviceOnce once;  // one per instantiation
    if (int rc = once.run([] {
          return static_cast<int>(cudaFuncSetAttribute(few_out_kernel<NT>, cudaFuncAttributeMaxDynamicSharedMemorySize, 160 * 1024));
        }))
      return rc;
  }
  return few_launch(few_out_kernel<NT>, dim3((p.D + 15) / 16), smem, true, p, st);
}

}  // namespace lmoe

using namespace lmoe;

static bool few_dims(const lmoe_shape* s, int L) {
  return s && s->T > 0 && s->T <= kFewTokens && s->D > 0 && (s->D % 32) == 0 && L > 0 && (L % 64) == 0 && s->E > 0 &&
         s->E <= LMOE_MAX_EXPERTS && s->K > 0 && s->K <= LMOE_MAX_TOPK && s->K <= s->E && s->F > 0 && (s->F % 64) == 0 &&
         s->Fs > 0 && (s->Fs % 32) == 0 && static_cast<long long>(s->T) * L * 2 <= 128 * 1024;
}

extern "C" int lmoe_few_applies(const lmoe_shape* s) { return few_dims(s, s ? s->L : 0) ? 1 : 0; }

extern "C" size_t lmoe_few_workspace_bytes(const lmoe_shape* s) {
  if (!few_dims(s, s ? s->L : 0)) return 0;
  const size_t T = s->T, slots = T * s->K;
  const size_t n[8] = {T * s->E * 4, slots * 4, slots * 4, T * 4, T * s->L * 2, T * s->Fs * 2, slots * s->F * 2, slots * s->L * 2};
  size_t sum = 0;
  for (size_t v : n) sum += (v + 255) / 256 * 256;
  return sum;
}

extern "C" int lmoe_few_forward(const lmoe_shape* s, const void* x, const void* w_gate, const void* w_down, const void* w_up,
                                const void* w_gate_up_s, const void* w_down_s, const void* w_gate_up, const void* w_down_e,
                                const float* expert_bias, float z_coef, void* y, float* z_loss, void* workspace,
                                size_t workspace_bytes, void* stream) {
  if (!few_dims(s, s ? s->L : 0)) return LMOE_ERR_SHAPE;
  if (!x || !w_gate || !w_gate_up_s || !w_down_s || !w_gate_up || !w_down_e || !expert_bias || !y || !z_loss || !workspace ||
      (w_down == nullptr) != (w_up == nullptr))
    return LMOE_ERR_ARG;
  if (!w_down && s->L != s->D) return LMOE_ERR_SHAPE;
  if (workspace_bytes < lmoe_few_workspace_bytes(s)) return LMOE_ERR_WORKSPACE;
  const void* const ptrs[10] = {x, w_gate, w_down, w_up, w_gate_up_s, w_down_s, w_gate_up, w_down_e, y, workspace};
  for (const void* q : ptrs)
    if ((reinterpret_cast<uintptr_t>(q) & 15) != 0) return LMOE_ERR_ALIGN;
  typedef const __nv_bfloat16* W;
  char* ws = static_cast<char*>(workspace);
  auto take = [&ws](size_t bytes) {
    char* at = ws;
    ws += (bytes + 255) / 256 * 256;
    return at;
  };
  const size_t T = s->T, slots = T * s->K;
  FewParams p = {};
  p.x = static_cast<W>(x);
  p.wg = static_cast<W>(w_gate);
  p.wdn = static_cast<W>(w_down);
  p.wup = static_cast<W>(w_up);
  p.wgus = static_cast<W>(w_gate_up_s);
  p.wds = static_cast<W>(w_down_s);
  p.wgu = static_cast<W>(w_gate_up);
  p.wde = static_cast<W>(w_down_e);
  p.bias = expert_bias;
  p.T = s->T;
  p.D = s->D;
  p.L = s->L;
  p.E = s->E;
  p.K = s->K;
  p.F = s->F;
  p.Fs = s->Fs;
  p.logits = reinterpret_cast<float*>(take(T * s->E * 4));
  p.sel = reinterpret_cast<int*>(take(slots * 4));
  p.weights = reinterpret_cast<float*>(take(slots * 4));
  p.lse = reinterpret_cast<float*>(take(T * 4));
  p.x_latent = reinterpret_cast<__nv_bfloat16*>(take(T * s->L * 2));
  p.hidden_s = reinterpret_cast<__nv_bfloat16*>(take(T * s->Fs * 2));
  p.hidden = reinterpret_cast<__nv_bfloat16*>(take(slots * s->F * 2));
  p.y_slot = reinterpret_cast<__nv_bfloat16*>(take(slots * s->L * 2));
  p.z_scale = z_coef / static_cast<float>(s->T);
  p.z_loss = z_loss;
  p.y = static_cast<__nv_bfloat16*>(y);
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  if (s->T <= 8) return few_forward<1>(p, st);
  if (s->T <= 16) return few_forward<2>(p, st);
  if (s->T <= 32) return few_forward<4>(p, st);
  return few_forward<8>(p, st);
}
