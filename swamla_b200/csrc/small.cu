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
#include "gemm_host.h"
#include "topk.cuh"

namespace lmoe {

constexpr int kFewTokens = LMOE_FEW_TOKENS;
constexpr int kFewThreads = 256;
constexpr int kFewWarps = kFewThreads / 32;
constexpr int kFewCluster = 8;
constexpr int kFewMaxLatent = 8192;  // 8 tokens' combined expert output of this width fit the output kernel's shared memory

__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void pdl_launch() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }

// Weight load that stays where it is written: a plain __ldg may be moved past griddepcontrol.wait, down to its first use, and
// then every step of the contraction waits for memory by itself (the output kernel took 8 us instead of 4).
__device__ __forceinline__ uint4 ld_weight(const void* p) {
  uint4 v;
  asm volatile("ld.global.nc.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "l"(p));
  return v;
}

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
  int* status;
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
        a[u] = ld_weight(row_a + c * 32 + t * 8);
        b[u] = ld_weight(row_b + c * 32 + t * 8);
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

__device__ __forceinline__ void load_slice(uint4 (&w)[kRowsPerThread], const __nv_bfloat16* W, int k0, int ncols, int col) {
#pragma unroll
  for (int r = 0; r < kRowsPerThread; ++r) w[r] = ld_weight(W + static_cast<long long>(k0 + r) * ncols + col);
}
// the first pass's slice into L2, one request per 64-byte piece of a row
__device__ __forceinline__ void prefetch_slice(const __nv_bfloat16* W, int kdim, int ncols, int col, int rg) {
  if ((threadIdx.x & 3) == 0)
#pragma unroll
    for (int r = 0; r < kRowsPerThread; ++r)
      if (rg * kRowsPerThread < kdim)
        asm volatile("prefetch.global.L2 [%0];" ::"l"(W + static_cast<long long>(rg * kRowsPerThread + r) * ncols + col));
}

template <bool GATE_UP>
__global__ void __launch_bounds__(kFewThreads, 2) few_expert_kernel(const FewParams p) {
  __shared__ int s_slot[kFewTokens];
  __shared__ unsigned s_mask[kFewTokens / 32];
  __shared__ float red[kFewWarps][kTokBatch][64];
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int slots = p.T * p.K;
  const int kdim = GATE_UP ? p.L : p.F, ncols = GATE_UP ? 2 * p.F : p.L;
  const int vec = tid & 7, rg = tid >> 3;
  const int col = GATE_UP ? ((vec < 4 ? 0 : p.F) + blockIdx.y * 32 + (vec & 3) * 8) : (blockIdx.y * 64 + vec * 8);
  const __nv_bfloat16* in = GATE_UP ? (p.wdn ? p.x_latent : p.x) : p.hidden;
  if (tid < kFewTokens / 32) s_mask[tid] = 0u;

  // The selection comes from the first kernel.  The gate/up launch waits for it here and lets its successor start only
  // then, so for the down launch it is complete from the start: that one waits for `hidden` after its weights are on the way.
  if (GATE_UP) {
    if (slots >= p.E) prefetch_slice(p.wgu + static_cast<long long>(blockIdx.x) * kdim * ncols, kdim, ncols, col, rg);
    pdl_wait();
  }
  pdl_launch();
  // ---- which expert: block x owns an expert, or, with fewer slots than experts, the slot that names it first
  int e = blockIdx.x;
  if (slots < p.E) {
    e = p.sel[blockIdx.x];
    int earlier = 0;
    for (int i = tid; i < static_cast<int>(blockIdx.x); i += kFewThreads) earlier |= p.sel[i] == e;
    if (__syncthreads_or(earlier)) return;
  } else {
    __syncthreads();
  }
  const __nv_bfloat16* W = (GATE_UP ? p.wgu : p.wde) + static_cast<long long>(e) * kdim * ncols;
  uint4 w[kRowsPerThread];
  if (rg * kRowsPerThread < kdim) load_slice(w, W, rg * kRowsPerThread, ncols, col);
  // ---- its slots, by token (a token names an expert at most once)
  for (int i = tid; i < slots; i += kFewThreads)
    if (p.sel[i] == e) atomicOr(&s_mask[(i / p.K) >> 5], 1u << ((i / p.K) & 31));
  __syncthreads();
  const unsigned m0 = s_mask[0], m1 = s_mask[1];
  const int n = __popc(m0) + __popc(m1);
  if (n == 0) return;
  for (int i = tid; i < slots; i += kFewThreads) {
    if (p.sel[i] != e) continue;
    const int tok = i / p.K;
    s_slot[tok < 32 ? __popc(m0 & ((1u << tok) - 1u)) : __popc(m0) + __popc(m1 & ((1u << (tok - 32)) - 1u))] = i;
  }
  __syncthreads();
  if (!GATE_UP) pdl_wait();

  constexpr int kSpan = kRowGroups * kRowsPerThread;   // rows of the contraction per pass: 256
  for (int b0 = 0; b0 < n; b0 += kTokBatch) {
    float acc[kTokBatch][8];
#pragma unroll
    for (int b = 0; b < kTokBatch; ++b)
#pragma unroll
      for (int j = 0; j < 8; ++j) acc[b][j] = 0.f;
    for (int k0 = rg * kRowsPerThread; k0 < kdim; k0 += kSpan) {
      if (b0 + k0 != rg * kRowsPerThread && kdim > kSpan) load_slice(w, W, k0, ncols, col);  // more than one pass over kdim
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

// Routed experts with at least as many (token, slot) pairs as experts: one CTA per expert streams that expert's two weight
// matrices, each contiguous in memory, through a ring of stages, gate_up -> SwiGLU -> down in one go.  The first stages are on
// their way before the selection is known; the ring takes most of an SM's shared memory (bytes in flight are the rate) unless
// there are more experts than SMs, when two CTAs share one.  The weights are [k, n] with n contiguous, so the columns become
// the rows of an m16n8k16 product through ldmatrix.trans and the tokens its eight columns; a stage row is padded by 16 bytes
// so that the eight rows of a matrix lie in different banks.  Every thread copies with cp.async: one bulk copy per padded row
// costs the TMA unit some 50 ns each (34 us for this launch alone).
// At 23 tokens of the 128-expert layer the two launches of the register kernel above take 16 + 9 us (several rounds of CTAs per
// SM), products on CUDA cores instead 44 us (an expert with six tokens is then bound by them); the whole call of three
// launches takes 31.8 us on the device.
template <int N>
__device__ __forceinline__ void cp_async_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }

__device__ __forceinline__ void ldmatrix_x4_trans(uint32_t addr, uint32_t (&r)[4]) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0, %1, %2, %3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
               : "r"(addr)
               : "memory");
}

struct StreamPlan {
  int rows_up, rows_dn;   // weight rows per stage: a multiple of 16 that divides the matrix
  int stage_bytes, part_cols;
  size_t smem;
};
// tokens: tokens per pass over the weights
static StreamPlan stream_plan(int L, int F, int tokens, int stages) {
  StreamPlan s;
  auto rows_of = [](int row_bytes) { return 32 * row_bytes <= 20480 ? (64 * row_bytes <= 20480 ? 64 : 32) : 16; };
  s.rows_up = rows_of(4 * F);
  s.rows_dn = rows_of(2 * L);
  const int up = s.rows_up * (4 * F + 16), dn = s.rows_dn * (2 * L + 16);
  s.stage_bytes = ((up > dn ? up : dn) + 127) / 128 * 128;
  s.part_cols = 2 * F > L ? 2 * F : L;
  s.smem = stages * static_cast<size_t>(s.stage_bytes) + static_cast<size_t>(tokens) * (2 * (L + F + 16) + 4 * s.part_cols);
  return s;
}

// TILES: tiles of 16 columns per warp, NT: tiles of 8 tokens per pass, STAGES: stages of the ring.
template <int TILES, int NT, int STAGES>
__global__ void __launch_bounds__(kFewThreads) few_stream_kernel(const FewParams p, const StreamPlan sp) {
  constexpr int kTok = 8 * NT;
  extern __shared__ __align__(128) uint8_t sm[];
  __shared__ int s_slot[kFewTokens];
  __shared__ unsigned s_mask[kFewTokens / 32];
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, e = blockIdx.x;
  const int xld = p.L + 8, hld = p.F + 8;                                                 // padded: eight tokens, eight banks
  float* const part = reinterpret_cast<float*>(sm + STAGES * sp.stage_bytes);             // [token][columns]
  __nv_bfloat16* const xs = reinterpret_cast<__nv_bfloat16*>(part + kTok * sp.part_cols);  // [token][L]
  __nv_bfloat16* const hs = xs + kTok * xld;                                              // [token][F]
  const int st_up = p.L / sp.rows_up, st_all = st_up + p.F / sp.rows_dn;                  // stages per pass over the weights
  const __nv_bfloat16* const w_up = p.wgu + static_cast<long long>(e) * p.L * 2 * p.F;
  const __nv_bfloat16* const w_dn = p.wde + static_cast<long long>(e) * p.F * p.L;
  // this thread's 16-byte column and first row of a stage, and the rows between its copies (rows of at most 256 vectors)
  const int vec_up = p.F / 4, vec_dn = p.L / 8, step_up = kFewThreads / vec_up, step_dn = kFewThreads / vec_dn;
  const int r0_up = tid / vec_up, v_up = tid - r0_up * vec_up, r0_dn = tid / vec_dn, v_dn = tid - r0_dn * vec_dn;
  int fill = 0, fill_j = 0, filled = 0;  // next ring slot to fill, its place in the walk, stages asked for so far
  auto issue = [&](bool there) {         // all threads; one group per call, empty when the walk is over
    if (there) {
      const bool up = fill_j < st_up;
      const int cols = up ? 2 * p.F : p.L, rows = up ? sp.rows_up : sp.rows_dn, r0 = up ? r0_up : r0_dn;
      const int step = up ? step_up : step_dn, pitch = 2 * cols + 16;
      const __nv_bfloat16* src = (up ? w_up + static_cast<long long>(fill_j) * rows * cols
                                     : w_dn + static_cast<long long>(fill_j - st_up) * rows * cols) + r0 * cols + (up ? v_up : v_dn) * 8;
      uint32_t dst = smem_u32(sm + fill * sp.stage_bytes) + r0 * pitch + (up ? v_up : v_dn) * 16;
      if (r0 < step)
#pragma unroll 4
        for (int r = r0; r < rows; r += step) {
          asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(src) : "memory");
          dst += step * pitch;
          src += step * cols;
        }
      fill = fill + 1 == STAGES ? 0 : fill + 1;
      fill_j = fill_j + 1 == st_all ? 0 : fill_j + 1;
      ++filled;
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
#pragma unroll 1
  for (int i = 0; i < STAGES - 1; ++i) issue(true);  // (a walk shorter than the ring begins again: group i is stage i)
  if (tid < kFewTokens / 32) s_mask[tid] = 0u;
  pdl_launch();
  pdl_wait();
  __syncthreads();
  const int slots = p.T * p.K;
  for (int i = tid; i < slots; i += kFewThreads)
    if (p.sel[i] == e) atomicOr(&s_mask[(i / p.K) >> 5], 1u << ((i / p.K) & 31));
  __syncthreads();
  const unsigned m0 = s_mask[0], m1 = s_mask[1];
  const int n = __popc(m0) + __popc(m1);
  for (int i = tid; i < slots && n > 0; i += kFewThreads) {
    if (p.sel[i] != e) continue;
    const int tok = i / p.K;
    s_slot[tok < 32 ? __popc(m0 & ((1u << tok) - 1u)) : __popc(m0) + __popc(m1 & ((1u << (tok - 32)) - 1u))] = i;
  }
  __syncthreads();

  // stages of this CTA: every group of kTok tokens walks the weights once
  const int total = n > 0 ? ((n + kTok - 1) / kTok) * st_all : 0;
  if (n == 0) {
    cp_async_wait<0>();
    return;
  }
  const __nv_bfloat16* in = p.wdn ? p.x_latent : p.x;
  float acc[TILES][NT][4];
  int slot_i = 0, j = 0, b0 = 0;
  for (int i = 0; i < total; ++i) {
    const int nb = min(kTok, n - b0);
    const bool up = j < st_up;
    const int cols = up ? 2 * p.F : p.L, rows = up ? sp.rows_up : sp.rows_dn, tiles = cols / 16;
    if (j == 0) {  // a new group of tokens: their input rows (absent tokens: zeros)
      const int vecs = p.L / 8;
      for (int k = tid; k < kTok * vecs; k += kFewThreads) {
        const int b = k / vecs, v = k - b * vecs;
        uint4 x = make_uint4(0, 0, 0, 0);
        // (the absent tokens' rows of hs stay what they are: a product's column depends on its own token only)
        if (b < nb) x = *reinterpret_cast<const uint4*>(in + static_cast<long long>(s_slot[b0 + b] / p.K) * p.L + v * 8);
        *reinterpret_cast<uint4*>(xs + b * xld + v * 8) = x;
      }
    }
    if (j == 0 || j == st_up) {
#pragma unroll
      for (int q = 0; q < TILES; ++q)
#pragma unroll
        for (int t = 0; t < NT; ++t)
#pragma unroll
          for (int c = 0; c < 4; ++c) acc[q][t][c] = 0.f;
    }
    cp_async_wait<STAGES - 2>();
    __syncthreads();  // everybody's part of stage i has landed, and everybody is done with stage i - 1: refill that one's slot
    issue(filled < total);
    {
      const int ld = up ? xld : hld, pitch = 2 * cols + 16;
      const __nv_bfloat16* src = up ? xs + j * rows : hs + (j - st_up) * rows;
      const uint32_t base = smem_u32(sm + slot_i * sp.stage_bytes);
      // matrices of the x4: (k 0-7, n 0-7), (k 0-7, n 8-15), (k 8-15, n 0-7), (k 8-15, n 8-15) = the A fragment's order
      const uint32_t lane_off = ((lane & 7) + ((lane >> 4) << 3)) * pitch + ((lane >> 3) & 1) * 16;
      for (int k = 0; k < rows; k += 16) {
        uint32_t xb[NT][2];
#pragma unroll
        for (int t = 0; t < NT; ++t) {
          const __nv_bfloat16* q = src + (t * 8 + (lane >> 2)) * ld + k + 2 * (lane & 3);
          xb[t][0] = *reinterpret_cast<const uint32_t*>(q);
          xb[t][1] = *reinterpret_cast<const uint32_t*>(q + 8);
        }
#pragma unroll
        for (int q = 0; q < TILES; ++q) {
          const int tile = warp + q * kFewWarps;
          if (tile < tiles) {
            uint32_t a[4];
            ldmatrix_x4_trans(base + k * pitch + tile * 32 + lane_off, a);
#pragma unroll
            for (int t = 0; t < NT; ++t) mma_16816(acc[q][t], a[0], a[1], a[2], a[3], xb[t][0], xb[t][1]);
          }
        }
      }
    }
    if (j == st_up - 1 || j == st_all - 1) {  // a matrix is done
#pragma unroll
      for (int q = 0; q < TILES; ++q) {
        const int c = (warp + q * kFewWarps) * 16 + (lane >> 2);
        if (c < cols)
#pragma unroll
          for (int t = 0; t < NT; ++t) {
            float* o = part + (t * 8 + 2 * (lane & 3)) * cols + c;
            o[0] = acc[q][t][0];
            o[cols] = acc[q][t][1];
            o[8] = acc[q][t][2];
            o[cols + 8] = acc[q][t][3];
          }
      }
      __syncthreads();
      const int width = up ? p.F : p.L;
      if (up) {
        for (int k = tid; k < nb * width; k += kFewThreads) {
          const int b = k / width, c = k - b * width;
          const float gate = bf16_round(part[b * cols + c]), upv = bf16_round(part[b * cols + p.F + c]);
          hs[b * hld + c] = __float2bfloat16_rn(silu_f(gate) * upv);
        }
      } else {
        for (int k = tid; k < nb * width; k += kFewThreads) {
          const int b = k / width, c = k - b * width;
          p.y_slot[static_cast<long long>(s_slot[b0 + b]) * p.L + c] = __float2bfloat16_rn(part[b * cols + c]);
        }
      }
      __syncthreads();
    }
    slot_i = slot_i + 1 == STAGES ? 0 : slot_i + 1;
    if (++j == st_all) {
      j = 0;
      b0 += kTok;
    }
  }
  cp_async_wait<0>();
}

// y = hidden_s * Wd_s^T + routed * Wup^T: 16 output columns and 8 tokens per CTA (the weighted sum over a token's K expert rows
// is each column block's own, so more tokens go to more CTAs, whose weights then come from L2).  routed = sum_k w_k y_slot.  Without an up-projection the
// weighted sum is added to the shared expert's output instead, which is rounded first as the separate GEMM's result is.
__global__ void __launch_bounds__(kFewThreads) few_out_kernel(const FewParams p) {
  extern __shared__ uint4 s_routed[];                   // [T][L] bf16 (latent form only)
  __shared__ float red[kFewWarps * 16 * 8];
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, g = lane >> 2, t = lane & 3;
  const int c_s = p.Fs / 32, chunks = c_s + (p.wup ? p.L / 32 : 0);
  const int row = blockIdx.x * 16, tok0 = blockIdx.y * 8, n_tok = min(8, p.T - tok0);
  constexpr int U = 5;  // steps in flight: (Fs + L) / 256 of a 1,024-wide layer; other sizes loop (3: up to 1.7 us slower)
  uint4 a[U], b[U];
  auto load = [&](int c, uint4& va, uint4& vb) {
    const __nv_bfloat16* base = c < c_s ? p.wds + static_cast<long long>(row + g) * p.Fs + c * 32 + t * 8
                                        : p.wup + static_cast<long long>(row + g) * p.L + (c - c_s) * 32 + t * 8;
    va = ld_weight(base);
    vb = ld_weight(base + 8ll * (c < c_s ? p.Fs : p.L));
  };
#pragma unroll
  for (int u = 0; u < U; ++u)
    if (warp + u * kFewWarps < chunks) load(warp + u * kFewWarps, a[u], b[u]);
  pdl_wait();
  if (p.wup) {
    const int vecs = p.L / 8;
    for (int i = tid; i < n_tok * vecs; i += kFewThreads) {
      const int tok = i / vecs, v = i - tok * vecs;
      float acc[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
      for (int k0 = 0; k0 < p.K; k0 += 6) {  // slots in flight (4 measures the same, within 0.3 us)
        uint4 yv[6];
        float wk[6];
#pragma unroll
        for (int u = 0; u < 6; ++u) {
          const int s = (tok0 + tok) * p.K + min(k0 + u, p.K - 1);
          yv[u] = *reinterpret_cast<const uint4*>(p.y_slot + static_cast<long long>(s) * p.L + v * 8);
          wk[u] = p.weights[s];
        }
#pragma unroll
        for (int u = 0; u < 6; ++u) {
          const uint32_t yw[4] = {yv[u].x, yv[u].y, yv[u].z, yv[u].w};
          if (k0 + u < p.K)  // (a weight of zero instead would turn an infinite row into NaN)
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
  float acc[1][4] = {{0.f, 0.f, 0.f, 0.f}};
  const __nv_bfloat16* routed = reinterpret_cast<const __nv_bfloat16*>(s_routed);
  for (int u0 = 0; warp + u0 * kFewWarps < chunks; u0 += U) {
    uint4 xv[U];
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const int c = warp + (u0 + u) * kFewWarps;
      xv[u] = make_uint4(0, 0, 0, 0);
      if (c < chunks) {
        if (u0 > 0) load(c, a[u], b[u]);
        if (g < n_tok)
          xv[u] = c < c_s ? *reinterpret_cast<const uint4*>(p.hidden_s + static_cast<long long>(tok0 + g) * p.Fs + c * 32 + t * 8)
                          : *reinterpret_cast<const uint4*>(routed + g * p.L + (c - c_s) * 32 + t * 8);
      }
    }
#pragma unroll
    for (int u = 0; u < U; ++u)
      if (warp + (u0 + u) * kFewWarps < chunks) mma_step(acc[0], a[u], b[u], xv[u]);
  }
  store_partial<1>(red, warp, lane, acc);
  __syncthreads();
  for (int i = tid; i < 16 * n_tok; i += kFewThreads) {
    const int c = i & 15, tok = tok0 + (i >> 4);
    float v = sum_partial<1>(red, c, i >> 4);
    if (!p.wup) {
      v = bf16_round(v);
      for (int k = 0; k < p.K; ++k)
        v = fmaf(p.weights[tok * p.K + k], __bfloat162float(p.y_slot[static_cast<long long>(tok * p.K + k) * p.L + row + c]), v);
    }
    p.y[static_cast<long long>(tok) * p.D + row + c] = __float2bfloat16_rn(v);
  }
  if (blockIdx.x == 0 && blockIdx.y == 0 && warp == 0) {
    double z = 0.0;
    for (int i = lane; i < p.T; i += 32) z += static_cast<double>(p.lse[i]) * static_cast<double>(p.lse[i]);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) z += __shfl_xor_sync(0xffffffffu, z, o);
    if (lane == 0) p.z_loss[0] = static_cast<float>(z * static_cast<double>(p.z_scale));
  }
}

template <typename Kernel, typename... Args>
static int few_launch(Kernel kernel, dim3 grid, size_t smem, bool after, cudaStream_t st, const Args&... args) {
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
  const cudaError_t e = cudaLaunchKernelEx(&cfg, kernel, args...);
  return e == cudaSuccess ? 0 : static_cast<int>(e);
}

// Whether an expert's rows fit four tiles of 16 columns per warp: the streamed kernel then takes 16 tokens per pass over the
// weights, else eight.
static int few_widest(int L, int F) { return 2 * F > L ? 2 * F : L; }
static bool few_narrow(int L, int F) { return few_widest(L, F) <= 4 * kFewWarps * 16; }
// Up to how many tokens these kernels beat the padded path (device time of a captured call, us, these kernels / padded):
//   rows of at most 512: L 256, F 256, 128 experts: 1 token 16 / 44, 23 32 / 57, 64 42 / 59; 256 experts: 64 70 / 74.  The masks of
//     an expert's tokens hold kFewTokens.
//   wider ones, where a second pass over the weights of the experts with more than eight tokens costs as much as the first:
//     L 256, F 768, 128 experts: 24 71 / 90, 28 72 / 90, 32 96 / 91, 64 138 / 92;
//     L 1,024, F 1,024, 32 experts (each streamed by one SM): 24 80 / 83, 28 88 / 87, 32 92 / 87, 64 158 / 89.
static int few_tokens(int L, int F) { return few_narrow(L, F) ? kFewTokens : 24; }

template <int NT>
static int few_forward(const FewParams& p, cudaStream_t st) {
  const int units = (p.wdn ? p.L / 16 : 0) + p.Fs / 8;
  const int cap = 512;  // CTAs of 256 threads, the rest loops (256 and 1,024 measure the same, within 0.3 us)
  const int rest = ((units < cap ? units : cap) + kFewCluster - 1) / kFewCluster * kFewCluster;
  auto in = p.E <= 32 ? few_in_kernel<NT, 1> : p.E <= 64 ? few_in_kernel<NT, 2> : p.E <= 128 ? few_in_kernel<NT, 4> : few_in_kernel<NT, 8>;
  if (int rc = few_launch(in, dim3(kFewCluster + rest), 0, false, st, p)) return rc;
  // the stream kernel wherever every expert is likely to have a token and its rows fit the tiles of a warp
  const int widest = few_widest(p.L, p.F);
  const bool narrow = few_narrow(p.L, p.F);
  // Stages of the ring: many, as bytes in flight are the rate (128 experts, 23 tokens: 10 stages 31.8 us, 8 32.3, 6 32.7; wide rows:
  // 3 71.6, 4 91.3, which leaves one CTA per SM).  More experts than SMs: two CTAs per SM share its memory.
  const int stages = !narrow ? 3 : p.E <= num_sms() ? 10 : 5;
  const StreamPlan sp = stream_plan(p.L, p.F, narrow ? 16 : 8, stages);
  constexpr size_t kMost = 220 * 1024;
  if (p.T * p.K >= p.E && widest <= 16 * kFewWarps * 16 && sp.smem <= kMost) {
    static PerDeviceOnce once;
    if (int rc = once.run([] {
          auto most = [](auto kernel) { return cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(kMost)); };
          cudaError_t e = most(few_stream_kernel<4, 2, 10>);
          if (e == cudaSuccess) e = most(few_stream_kernel<4, 2, 5>);
          if (e == cudaSuccess) e = most(few_stream_kernel<16, 1, 3>);
          return static_cast<int>(e);
        }))
      return rc;
    auto kernel = !narrow ? few_stream_kernel<16, 1, 3> : stages == 10 ? few_stream_kernel<4, 2, 10> : few_stream_kernel<4, 2, 5>;
    if (int rc = few_launch(kernel, dim3(p.E), sp.smem, true, st, p, sp)) return rc;
  } else {
    const int owners = p.T * p.K < p.E ? p.T * p.K : p.E;
    if (int rc = few_launch(few_expert_kernel<true>, dim3(owners, p.F / 32), 0, true, st, p)) return rc;
    if (int rc = few_launch(few_expert_kernel<false>, dim3(owners, p.L / 64), 0, true, st, p)) return rc;
  }
  const size_t smem = p.wup ? static_cast<size_t>(8) * p.L * 2 : 0;
  static PerDeviceOnce once;
  if (int rc = once.run([] {
        return static_cast<int>(cudaFuncSetAttribute(few_out_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kFewMaxLatent * 16));
      }))
    return rc;
  return few_launch(few_out_kernel, dim3(p.D / 16, (p.T + 7) / 8), smem, true, st, p);
}

}  // namespace lmoe

using namespace lmoe;

static bool few_dims(const lmoe_shape* s, int L) {
  return s && s->T > 0 && s->T <= few_tokens(L, s->F) && s->D > 0 && (s->D % 32) == 0 && L > 0 && (L % 64) == 0 && s->E > 0 &&
         s->E <= LMOE_MAX_EXPERTS && s->K > 0 && s->K <= LMOE_MAX_TOPK && s->K <= s->E && s->F > 0 && (s->F % 64) == 0 &&
         s->Fs > 0 && (s->Fs % 32) == 0 && L <= kFewMaxLatent;
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
                                size_t workspace_bytes, int32_t* status, void* stream) {
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
  p.status = status;
  p.y = static_cast<__nv_bfloat16*>(y);
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  if (s->T <= 8) return few_forward<1>(p, st);
  if (s->T <= 16) return few_forward<2>(p, st);
  if (s->T <= 32) return few_forward<4>(p, st);
  return few_forward<8>(p, st);
}
