// Router kernels: warp-level top-k with z-loss, and the deterministic histogram / scan / stable
// permutation that lays the (token, slot) pairs out expert by expert.  All HBM-bound integer work.
#include <cuda_runtime.h>
#include <math_constants.h>
#include <stdint.h>

#include <mutex>

#include "../../include/lmoe.h"
#include "counters.h"
#include "device_once.h"
#include "topk.cuh"

namespace lmoe {

constexpr int kTopkWarps = 8;       // warps of a top-k block, and the fewest of one that also counts
constexpr int kMaxTopkWarps = 32;
constexpr int kMaxChunkTokens = 128;  // tokens of a block
// z_partial: the fp32 sum of lse^2 over eight consecutive tokens each, whatever the block's size; the rest of the sum is fp64.
constexpr int kZGroup = 8;

// One warp per token, `per_warp` consecutive tokens each.  With chunk_hist the block also counts its selections:
// chunk_hist[blockIdx.x][E] is the first pass of the routing tables (whole numbers: the order of the shared-memory
// additions does not matter).
template <int PER>
__global__ void __launch_bounds__(kMaxTopkWarps * 32)
gate_topk_kernel(const float* __restrict__ logits, const float* __restrict__ bias, int T, int E, int K, int* __restrict__ sel,
                 float* __restrict__ weights, float* __restrict__ lse_out, float* __restrict__ z_partial, int per_warp,
                 int* __restrict__ chunk_hist) {
  __shared__ float s_lse2[kMaxChunkTokens];
  __shared__ int s_hist[32 * PER];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, warps = blockDim.x >> 5;
  if (chunk_hist) {
    for (int e = threadIdx.x; e < E; e += blockDim.x) s_hist[e] = 0;
    __syncthreads();
  }
  for (int r = 0; r < per_warp; ++r) {
    const int slot = warp * per_warp + r, t = blockIdx.x * warps * per_warp + slot;
    if (t >= T) {
      if (lane == 0) s_lse2[slot] = 0.f;
      continue;
    }
    int idx;
    float aff, aff_sum, lse;
    topk_row<PER>(logits + static_cast<long long>(t) * E, bias, E, K, lane, idx, aff, aff_sum, lse);
    if (lane == 0) {
      s_lse2[slot] = lse * lse;
      lse_out[t] = lse;
    }
    if (lane < K) {
      sel[static_cast<long long>(t) * K + lane] = idx;
      weights[static_cast<long long>(t) * K + lane] = aff / (aff_sum + 1e-9f);
      if (chunk_hist) atomicAdd(&s_hist[idx], 1);
    }
  }
  __syncthreads();
  const int groups = warps * per_warp / kZGroup;
  if (static_cast<int>(threadIdx.x) < groups) {
    const int g = blockIdx.x * groups + threadIdx.x;
    float s = 0.f;
    for (int i = 0; i < kZGroup; ++i) s += s_lse2[threadIdx.x * kZGroup + i];
    if (g * kZGroup < T) z_partial[g] = s;
  }
  if (chunk_hist)
    for (int e = threadIdx.x; e < E; e += blockDim.x) chunk_hist[static_cast<long long>(blockIdx.x) * E + e] = s_hist[e];
}

// Deterministic final reduction of the z-loss partials (fixed order, one block).
__global__ void __launch_bounds__(256) zloss_finalize_kernel(const float* __restrict__ partial, int n, float scale,
                                                             float* __restrict__ z_loss) {
  __shared__ double s[256];
  double acc = 0.0;
  for (int i = threadIdx.x; i < n; i += 256) acc += static_cast<double>(partial[i]);
  s[threadIdx.x] = acc;
  __syncthreads();
  for (int o = 128; o > 0; o >>= 1) {
    if (threadIdx.x < o) s[threadIdx.x] += s[threadIdx.x + o];
    __syncthreads();
  }
  if (threadIdx.x == 0) z_loss[0] = static_cast<float>(s[0] * static_cast<double>(scale));
}

// ----------------------------------------------------------------------------- routing tables
// The flat (token, slot) list is cut into chunks of kChunk entries, one warp per chunk.
constexpr int kChunk = 256;
constexpr int kRouteWarps = 8;

// Pass 1: per-chunk histogram -> chunk_hist[chunk][E].
__global__ void __launch_bounds__(kRouteWarps * 32)
route_hist_kernel(const int* __restrict__ sel, int n, int E, int* __restrict__ chunk_hist) {
  __shared__ int hist[kRouteWarps][LMOE_MAX_EXPERTS];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int chunk = blockIdx.x * kRouteWarps + warp;
  for (int e = lane; e < E; e += 32) hist[warp][e] = 0;
  __syncwarp();
  const long long base = static_cast<long long>(chunk) * kChunk;
  if (base < n) {
    for (int s = 0; s < kChunk; s += 32) {
      const long long i = base + s + lane;
      const bool valid = i < n;
      const int e = valid ? sel[i] : -1;
      const unsigned peers = __match_any_sync(0xffffffffu, e);
      if (valid && (__ffs(peers) - 1) == lane) hist[warp][e] += __popc(peers);  // one writer per distinct expert
      __syncwarp();
    }
    for (int e = lane; e < E; e += 32) chunk_hist[static_cast<long long>(chunk) * E + e] = hist[warp][e];
  }
}

// Pass 2: one block per expert: exclusive scan of that expert's counts over the chunks (in place),
// total -> counts[e].
__global__ void __launch_bounds__(256) route_scan_chunks_kernel(int* __restrict__ chunk_hist, int n_chunks, int E,
                                                                int* __restrict__ counts) {
  __shared__ int warp_sums[8];
  __shared__ int carry_s;
  const int e = blockIdx.x;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  if (threadIdx.x == 0) carry_s = 0;
  __syncthreads();
  for (int c0 = 0; c0 < n_chunks; c0 += 256) {
    const int c = c0 + threadIdx.x;
    const int v = (c < n_chunks) ? chunk_hist[static_cast<long long>(c) * E + e] : 0;
    int incl = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int y = __shfl_up_sync(0xffffffffu, incl, o);
      if (lane >= o) incl += y;
    }
    if (lane == 31) warp_sums[warp] = incl;
    __syncthreads();
    int warp_off = 0;
    for (int w = 0; w < warp; ++w) warp_off += warp_sums[w];
    const int carry = carry_s;
    if (c < n_chunks) chunk_hist[static_cast<long long>(c) * E + e] = carry + warp_off + incl - v;
    __syncthreads();
    if (threadIdx.x == 255) carry_s = carry + warp_off + incl;
    __syncthreads();
  }
  if (threadIdx.x == 0) counts[e] = carry_s;
}

// Pass 3: stable scatter.  Every block first scans the per-expert counts in shared memory (canonical
// and padded offsets); block b also publishes the tables of experts b, b + gridDim.x, ... (offsets,
// tile -> expert entries, -1 markers of the pad rows).  Then each warp walks its chunk in index order
// again: rank inside the warp step by match_any + popc, running per-expert cursors in shared memory.
__global__ void __launch_bounds__(kRouteWarps * 32)
route_scatter_kernel(const int* __restrict__ sel, int n, int E, const int* __restrict__ chunk_base,
                     const int* __restrict__ counts, int* __restrict__ offsets, int* __restrict__ pad_offsets,
                     int* __restrict__ tile_expert, int* __restrict__ n_tiles, int* __restrict__ perm,
                     int* __restrict__ pos, int* __restrict__ row_src) {
  __shared__ int cursor[kRouteWarps][LMOE_MAX_EXPERTS];
  __shared__ int s_off[LMOE_MAX_EXPERTS + 1], s_poff[LMOE_MAX_EXPERTS + 1], s_cnt[LMOE_MAX_EXPERTS];
  __shared__ int s_wsum[2][kRouteWarps];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int tid = threadIdx.x;  // blockDim.x == LMOE_MAX_EXPERTS == 256
  {
    const int c = (tid < E) ? counts[tid] : 0;
    const int pc = (c + LMOE_ROW_PAD - 1) / LMOE_ROW_PAD * LMOE_ROW_PAD;
    int ic = c, ip = pc;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int a = __shfl_up_sync(0xffffffffu, ic, o), b = __shfl_up_sync(0xffffffffu, ip, o);
      if (lane >= o) {
        ic += a;
        ip += b;
      }
    }
    if (lane == 31) {
      s_wsum[0][warp] = ic;
      s_wsum[1][warp] = ip;
    }
    __syncthreads();
    int wc = 0, wp = 0;
    for (int w = 0; w < warp; ++w) {
      wc += s_wsum[0][w];
      wp += s_wsum[1][w];
    }
    if (tid < E) {
      s_cnt[tid] = c;
      s_off[tid] = wc + ic - c;
      s_poff[tid] = wp + ip - pc;
      if (tid == E - 1) {
        s_off[E] = wc + ic;
        s_poff[E] = wp + ip;
      }
    }
    __syncthreads();
  }
  // publish the tables of the experts this block is responsible for
  for (int e = blockIdx.x; e < E; e += gridDim.x) {
    if (tid == 0) {
      offsets[e] = s_off[e];
      pad_offsets[e] = s_poff[e];
    }
    for (int t = s_poff[e] / LMOE_ROW_PAD + tid; t < s_poff[e + 1] / LMOE_ROW_PAD; t += blockDim.x) tile_expert[t] = e;
    for (int r = s_poff[e] + s_cnt[e] + tid; r < s_poff[e + 1]; r += blockDim.x) row_src[r] = -1;
  }
  if (blockIdx.x == 0 && tid == 0) {
    offsets[E] = s_off[E];
    pad_offsets[E] = s_poff[E];
    n_tiles[0] = s_poff[E] / LMOE_ROW_PAD;
  }

  const int chunk = blockIdx.x * kRouteWarps + warp;
  const long long base = static_cast<long long>(chunk) * kChunk;
  if (base >= n) return;
  for (int e = lane; e < E; e += 32) cursor[warp][e] = chunk_base[static_cast<long long>(chunk) * E + e];
  __syncwarp();
  for (int s = 0; s < kChunk; s += 32) {
    const long long i = base + s + lane;
    const bool valid = i < n;
    const int e = valid ? sel[i] : -1;
    const unsigned peers = __match_any_sync(0xffffffffu, e);
    if (valid) {
      const int rank = cursor[warp][e] + __popc(peers & ((1u << lane) - 1u));
      perm[s_off[e] + rank] = static_cast<int>(i);
      const int prow = s_poff[e] + rank;
      pos[i] = prow;
      row_src[prow] = static_cast<int>(i);
    }
    __syncwarp();
    if (valid && (__ffs(peers) - 1) == lane) cursor[warp][e] += __popc(peers);
    __syncwarp();
  }
}

// The same tables from the chunk histograms of the top-k kernel, and the gather in the same launch.  A chunk is the
// `tokens` (at most 128) consecutive tokens of one top-k block, a token selects an expert at most once; so the rank of an
// entry among its expert's entries of the chunk is a population count over a bit mask of the tokens before it, and no warp
// walks its entries in order.  Every latent row is read ONCE and written to its K places (a gather by destination row reads
// it K times).  Blocks beyond the last chunk, and every block besides its chunk, publish the tables and zero the pad rows of
// experts b, b + gridDim.x, ...; block 0 also adds up the z-loss.
constexpr int kDirectChunks = 128;
constexpr int kMaskWords = kMaxChunkTokens / 32;

__global__ void __launch_bounds__(256)
route_gather_kernel(const int* __restrict__ sel, int T, int E, int K, int tokens, int chunks, int direct,
                    const int* __restrict__ hist, const float* __restrict__ z_partial, float z_scale, float* __restrict__ z_loss,
                    const lmoe_route r, const uint4* __restrict__ src, int vec_per_row, uint4* __restrict__ dst) {
  __shared__ int s_cnt[LMOE_MAX_EXPERTS], s_base[LMOE_MAX_EXPERTS];
  __shared__ int s_off[LMOE_MAX_EXPERTS + 1], s_poff[LMOE_MAX_EXPERTS + 1];
  __shared__ unsigned s_mask[LMOE_MAX_EXPERTS][kMaskWords];
  __shared__ int s_wsum[2][8];
  __shared__ double s_z[256];
  extern __shared__ int s_row[];  // [tokens * K] padded row of every entry of the chunk
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int chunk = blockIdx.x;
  const int mask_words = (tokens + 31) / 32;

  for (int i = tid; i < E * mask_words; i += 256) s_mask[i / mask_words][i % mask_words] = 0u;
  if (direct) {
    // thread t sums a share of the chunks for expert t % E': per = threads per expert (E <= 128 leaves room for more)
    const int per = E <= 64 ? 4 : (E <= 128 ? 2 : 1);
    if (tid < E) s_cnt[tid] = s_base[tid] = 0;
    __syncthreads();
    const int e = tid / per, part = tid - e * per;
    if (e < E) {
      int before = 0, all = 0;
#pragma unroll 8
      for (int c = part; c < chunks; c += per) {
        const int v = hist[static_cast<long long>(c) * E + e];
        all += v;
        if (c < chunk) before += v;
      }
      atomicAdd(&s_cnt[e], all);
      atomicAdd(&s_base[e], before);
    }
  } else if (tid < E) {
    s_cnt[tid] = r.counts[tid];
    if (chunk < chunks) s_base[tid] = hist[static_cast<long long>(chunk) * E + tid];
  }
  __syncthreads();
  {  // canonical and padded offsets of every expert (blockDim.x == LMOE_MAX_EXPERTS == 256)
    const int c = (tid < E) ? s_cnt[tid] : 0;
    const int pc = (c + LMOE_ROW_PAD - 1) / LMOE_ROW_PAD * LMOE_ROW_PAD;
    int ic = c, ip = pc;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int a = __shfl_up_sync(0xffffffffu, ic, o), b = __shfl_up_sync(0xffffffffu, ip, o);
      if (lane >= o) {
        ic += a;
        ip += b;
      }
    }
    if (lane == 31) {
      s_wsum[0][warp] = ic;
      s_wsum[1][warp] = ip;
    }
    __syncthreads();
    int wc = 0, wp = 0;
    for (int w = 0; w < warp; ++w) {
      wc += s_wsum[0][w];
      wp += s_wsum[1][w];
    }
    if (tid < E) {
      s_off[tid] = wc + ic - c;
      s_poff[tid] = wp + ip - pc;
      if (tid == E - 1) {
        s_off[E] = wc + ic;
        s_poff[E] = wp + ip;
      }
    }
    __syncthreads();
  }
  // ---- tables and pad rows of this block's experts
  for (int e = blockIdx.x; e < E; e += gridDim.x) {
    if (tid == 0) {
      if (direct) r.counts[e] = s_cnt[e];
      r.offsets[e] = s_off[e];
      r.pad_offsets[e] = s_poff[e];
    }
    for (int t = s_poff[e] / LMOE_ROW_PAD + tid; t < s_poff[e + 1] / LMOE_ROW_PAD; t += 256) r.tile_expert[t] = e;
    const int first = s_poff[e] + s_cnt[e];
    for (int q = first + tid; q < s_poff[e + 1]; q += 256) r.row_src[q] = -1;
    if (dst)
      for (long long i = static_cast<long long>(first) * vec_per_row + tid; i < static_cast<long long>(s_poff[e + 1]) * vec_per_row;
           i += 256)
        dst[i] = make_uint4(0, 0, 0, 0);
  }
  if (blockIdx.x == 0) {
    if (tid == 0) {
      r.offsets[E] = s_off[E];
      r.pad_offsets[E] = s_poff[E];
      r.n_tiles[0] = s_poff[E] / LMOE_ROW_PAD;
    }
    double acc = 0.0;
    const int n_z = (T + kZGroup - 1) / kZGroup;
#pragma unroll 8
    for (int i = tid; i < n_z; i += 256) acc += static_cast<double>(z_partial[i]);
    s_z[tid] = acc;
    __syncthreads();
    for (int o = 128; o > 0; o >>= 1) {
      if (tid < o) s_z[tid] += s_z[tid + o];
      __syncthreads();
    }
    if (tid == 0) z_loss[0] = static_cast<float>(s_z[0] * static_cast<double>(z_scale));
  }
  if (chunk >= chunks) return;

  // ---- this chunk's entries
  const int t0 = chunk * tokens;
  const int n_tok = min(tokens, T - t0), n = n_tok * K;
  const int* my = sel + static_cast<long long>(t0) * K;
  for (int i = tid; i < n; i += 256) {
    const int tok = i / K;
    atomicOr(&s_mask[my[i]][tok >> 5], 1u << (tok & 31));
  }
  __syncthreads();
  for (int i = tid; i < n; i += 256) {
    const int tok = i / K, e = my[i];
    int rank = s_base[e];
    for (int w = 0; w < (tok >> 5); ++w) rank += __popc(s_mask[e][w]);
    rank += __popc(s_mask[e][tok >> 5] & ((1u << (tok & 31)) - 1u));
    const int row = s_poff[e] + rank, flat = t0 * K + i;
    r.perm[s_off[e] + rank] = flat;
    r.pos[flat] = row;
    r.row_src[row] = flat;
    s_row[i] = row;
  }
  if (!dst) return;
  __syncthreads();
  for (int tok = warp; tok < n_tok; tok += 8) {
    const uint4* from = src + static_cast<long long>(t0 + tok) * vec_per_row;
    for (int v = lane; v < vec_per_row; v += 32) {
      const uint4 x = from[v];
      for (int k = 0; k < K; ++k) dst[static_cast<long long>(s_row[tok * K + k]) * vec_per_row + v] = x;
    }
  }
}

// Router bias update from the routing histogram.  The expected load per expert is taken from the histogram itself
// (sum of the counts / E = tokens * K / E): a histogram summed over several ranks then gives the global figure
// whatever the ranks' own token counts were.  One block; E <= LMOE_MAX_EXPERTS threads carry one expert each.
__global__ void __launch_bounds__(LMOE_MAX_EXPERTS)
bias_update_kernel(const int* __restrict__ counts, int E, float gamma, float* __restrict__ bias,
                   float* __restrict__ history, long long* __restrict__ update_count) {
  __shared__ long long total_s;
  const int e = threadIdx.x;
  const int c = (e < E) ? counts[e] : 0;
  if (e == 0) {
    total_s = 0;
    if (update_count) update_count[0] += 1;
  }
  __syncthreads();
  long long part = c;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) part += __shfl_xor_sync(0xffffffffu, part, o);
  if ((e & 31) == 0) atomicAdd(reinterpret_cast<unsigned long long*>(&total_s), static_cast<unsigned long long>(part));
  __syncthreads();
  if (e >= E) return;
  const float expected = static_cast<float>(static_cast<double>(total_s) / static_cast<double>(E));
  const float load = static_cast<float>(c);
  const float d = load - expected;
  const float sg = (d > 0.f) ? 1.f : ((d < 0.f) ? -1.f : 0.f);
  bias[e] -= gamma * sg;
  history[e] = 0.99f * history[e] + 0.01f * load;
}

// Kernels of this file that use static shared memory ask for the same (maximum) shared-memory carveout as the GEMM
// kernel: an SM runs kernels with different carveouts only one after the other, and these kernels are meant to run
// beside a GEMM of another stream.
template <typename F>
static inline void prefer_max_carveout(F* fn) {
  cudaFuncSetAttribute(fn, cudaFuncAttributePreferredSharedMemoryCarveout, cudaSharedmemCarveoutMaxShared);
}
static void configure_route_kernels() {
  static PerDeviceOnce once;
  once.run([] {
  prefer_max_carveout(gate_topk_kernel<1>);
  prefer_max_carveout(gate_topk_kernel<2>);
  prefer_max_carveout(gate_topk_kernel<4>);
  prefer_max_carveout(gate_topk_kernel<8>);
  prefer_max_carveout(zloss_finalize_kernel);
  prefer_max_carveout(route_hist_kernel);
  prefer_max_carveout(route_scan_chunks_kernel);
  prefer_max_carveout(route_scatter_kernel);
  prefer_max_carveout(route_gather_kernel);
  return 0;
  });
}

static inline int check_shape(const lmoe_shape* s) {
  if (!s) return LMOE_ERR_ARG;
  if (s->T <= 0 || s->E <= 0 || s->E > LMOE_MAX_EXPERTS || s->K <= 0 || s->K > LMOE_MAX_TOPK || s->K > s->E)
    return LMOE_ERR_SHAPE;
  if (static_cast<long long>(s->T) * s->K >= (1ll << 31)) return LMOE_ERR_SHAPE;
  return 0;
}

}  // namespace lmoe

using namespace lmoe;

static void launch_topk(const lmoe_shape* s, const float* logits, const float* bias, int32_t* sel, float* weights, float* lse,
                        float* z_partial, int warps, int per_warp, int* chunk_hist, cudaStream_t st) {
  configure_route_kernels();
  const int per_block = warps * per_warp;
  const int blocks = (s->T + per_block - 1) / per_block;
  auto kernel = s->E <= 32 ? gate_topk_kernel<1> : s->E <= 64 ? gate_topk_kernel<2> : s->E <= 128 ? gate_topk_kernel<4> : gate_topk_kernel<8>;
  kernel<<<blocks, warps * 32, 0, st>>>(logits, bias, s->T, s->E, s->K, sel, weights, lse, z_partial, per_warp, chunk_hist);
  count_launch();
}

extern "C" int lmoe_gate_topk_fwd(const lmoe_shape* s, const float* logits, const float* expert_bias, float z_coef,
                                  int32_t* sel, float* weights, float* lse, float* z_partial, float* z_loss,
                                  void* stream) {
  if (int rc = check_shape(s)) return rc;
  if (!logits || !expert_bias || !sel || !weights || !lse || !z_partial || !z_loss) return LMOE_ERR_ARG;
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  launch_topk(s, logits, expert_bias, sel, weights, lse, z_partial, kTopkWarps, 1, nullptr, st);
  const int blocks = (s->T + kZGroup - 1) / kZGroup;
  count_launch();
  zloss_finalize_kernel<<<1, 256, 0, st>>>(z_partial, blocks, z_coef / static_cast<float>(s->T), z_loss);
  cudaError_t e = cudaGetLastError();
  return e == cudaSuccess ? 0 : static_cast<int>(e);
}

// ----------------------------------------------------------------------------- routing in two or three launches
// lmoe_topk_hist_fwd + lmoe_route_gather_fwd do what lmoe_gate_topk_fwd, lmoe_route_permute and lmoe_gather_rows do in six
// launches.  Tokens are cut into chunks of one top-k block each.  Up to kDirectChunks of them, every block of the scatter
// adds up the chunk histograms itself (they are a few KB per block, from L2); beyond, a scan kernel does it once.
// A token takes a warp about 2 us, so a batch is spread over as many warps as it has tokens; the blocks get larger (8 to 32
// warps) to keep at most kDirectChunks of them up to 4,096 tokens, and then each warp takes more tokens, for about 1,024 chunks.
struct RouteChunks {
  int warps, per_warp, tokens, n;
};
static RouteChunks route_chunks(int T) {
  RouteChunks c;
  c.warps = T <= kTopkWarps * kDirectChunks ? kTopkWarps : T <= 2 * kTopkWarps * kDirectChunks ? 2 * kTopkWarps : kMaxTopkWarps;
  c.per_warp = (T + kMaxTopkWarps * 1024 - 1) / (kMaxTopkWarps * 1024);
  if (c.per_warp > kMaxChunkTokens / kMaxTopkWarps) c.per_warp = kMaxChunkTokens / kMaxTopkWarps;
  c.tokens = c.warps * c.per_warp;
  c.n = (T + c.tokens - 1) / c.tokens;
  return c;
}

extern "C" size_t lmoe_route_fwd_workspace_bytes(const lmoe_shape* s) {
  if (check_shape(s)) return 0;
  const size_t chunks = static_cast<size_t>(route_chunks(s->T).n), z = (static_cast<size_t>(s->T) + kZGroup - 1) / kZGroup;
  return (chunks * s->E + (z + 3) / 4 * 4) * sizeof(int);
}

extern "C" int lmoe_topk_hist_fwd(const lmoe_shape* s, const float* logits, const float* expert_bias, int32_t* sel,
                                  float* weights, float* lse, void* workspace, size_t workspace_bytes, void* stream) {
  if (int rc = check_shape(s)) return rc;
  if (!logits || !expert_bias || !sel || !weights || !lse || !workspace) return LMOE_ERR_ARG;
  if (workspace_bytes < lmoe_route_fwd_workspace_bytes(s)) return LMOE_ERR_WORKSPACE;
  int* hist = static_cast<int*>(workspace);
  const RouteChunks c = route_chunks(s->T);
  float* z_partial = reinterpret_cast<float*>(hist + static_cast<size_t>(c.n) * s->E);
  launch_topk(s, logits, expert_bias, sel, weights, lse, z_partial, c.warps, c.per_warp, hist, static_cast<cudaStream_t>(stream));
  cudaError_t e = cudaGetLastError();
  return e == cudaSuccess ? 0 : static_cast<int>(e);
}

extern "C" int lmoe_route_gather_fwd(const lmoe_shape* s, const int32_t* sel, void* workspace, size_t workspace_bytes,
                                     float z_coef, float* z_loss, const lmoe_route* r, const void* src, int row_bytes, void* dst,
                                     void* stream) {
  if (int rc = check_shape(s)) return rc;
  if (!sel || !workspace || !z_loss || !r || !r->counts || !r->offsets || !r->perm || !r->pad_offsets || !r->pos ||
      !r->row_src || !r->tile_expert || !r->n_tiles || (src == nullptr) != (dst == nullptr))
    return LMOE_ERR_ARG;
  if (src && (row_bytes <= 0 || (row_bytes & 15) != 0)) return LMOE_ERR_SHAPE;
  if (workspace_bytes < lmoe_route_fwd_workspace_bytes(s)) return LMOE_ERR_WORKSPACE;
  configure_route_kernels();
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  const RouteChunks rc = route_chunks(s->T);
  const int chunks = rc.n, tokens = rc.tokens;
  int* hist = static_cast<int*>(workspace);
  const float* z_partial = reinterpret_cast<float*>(hist + static_cast<size_t>(chunks) * s->E);
  const bool direct = chunks <= kDirectChunks;
  if (!direct) {
    count_launch();
    route_scan_chunks_kernel<<<s->E, 256, 0, st>>>(hist, chunks, s->E, r->counts);
  }
  // at least one block per expert: the pad rows of an expert (up to 127 rows to zero) are a block's extra duty
  const int blocks = chunks > s->E ? chunks : s->E;
  const size_t smem = static_cast<size_t>(tokens) * s->K * sizeof(int);
  count_launch();
  route_gather_kernel<<<blocks, 256, smem, st>>>(sel, s->T, s->E, s->K, tokens, chunks, direct ? 1 : 0, hist, z_partial,
                                                 z_coef / static_cast<float>(s->T), z_loss, *r, static_cast<const uint4*>(src),
                                                 row_bytes / 16, static_cast<uint4*>(dst));
  cudaError_t e = cudaGetLastError();
  return e == cudaSuccess ? 0 : static_cast<int>(e);
}

extern "C" size_t lmoe_route_workspace_bytes(const lmoe_shape* s) {
  if (check_shape(s)) return 0;
  const long long n = static_cast<long long>(s->T) * s->K;
  const long long chunks = (n + kChunk - 1) / kChunk;
  return static_cast<size_t>(chunks) * s->E * sizeof(int);
}

extern "C" int64_t lmoe_padded_rows(const lmoe_shape* s) {
  if (check_shape(s)) return 0;
  const long long n = static_cast<long long>(s->T) * s->K;
  return (n + LMOE_ROW_PAD - 1) / LMOE_ROW_PAD * LMOE_ROW_PAD + static_cast<long long>(s->E) * LMOE_ROW_PAD;
}

extern "C" int lmoe_route_permute(const lmoe_shape* s, const int32_t* sel, const lmoe_route* r, void* workspace,
                                  size_t workspace_bytes, void* stream) {
  if (int rc = check_shape(s)) return rc;
  if (!sel || !r || !workspace || !r->counts || !r->offsets || !r->perm || !r->pad_offsets || !r->pos || !r->row_src ||
      !r->tile_expert || !r->n_tiles)
    return LMOE_ERR_ARG;
  if (workspace_bytes < lmoe_route_workspace_bytes(s)) return LMOE_ERR_WORKSPACE;
  configure_route_kernels();
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  const int n = s->T * s->K;
  const int chunks = (n + kChunk - 1) / kChunk;
  const int blocks = (chunks + kRouteWarps - 1) / kRouteWarps;
  int* chunk_hist = static_cast<int*>(workspace);
  count_launch(3);
  route_hist_kernel<<<blocks, kRouteWarps * 32, 0, st>>>(sel, n, s->E, chunk_hist);
  route_scan_chunks_kernel<<<s->E, 256, 0, st>>>(chunk_hist, chunks, s->E, r->counts);
  route_scatter_kernel<<<blocks, kRouteWarps * 32, 0, st>>>(sel, n, s->E, chunk_hist, r->counts, r->offsets,
                                                           r->pad_offsets, r->tile_expert, r->n_tiles, r->perm, r->pos,
                                                           r->row_src);
  cudaError_t e = cudaGetLastError();
  return e == cudaSuccess ? 0 : static_cast<int>(e);
}

// ----------------------------------------------------------------------------- no-allocation variant
// Scratch of lmoe_route_permute_static: the per-chunk histograms live in this file-scope device array
// instead of a caller-provided workspace.  Every GPU that loads the library holds these 4 MiB until
// the process exits.  Host code must not hand `g_route_scratch` itself to a kernel (in host code the
// name is only a handle): the device address is looked up once per device with cudaGetSymbolAddress.
constexpr size_t kStaticRouteScratchInts = LMOE_STATIC_ROUTE_SCRATCH_BYTES / sizeof(int);
static __device__ __align__(256) int g_route_scratch[kStaticRouteScratchInts];

namespace {
std::mutex g_static_scratch_mutex;
int* g_static_scratch_ptr[kMaxDevices] = {nullptr};

// Device address of the scratch array on the CURRENT device; resolved on the first call per device.
int static_route_scratch(int** out) {
  int dev = -1;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return static_cast<int>(e);
  if (dev < 0 || dev >= kMaxDevices) return LMOE_ERR_ARG;
  std::lock_guard<std::mutex> lock(g_static_scratch_mutex);
  if (!g_static_scratch_ptr[dev]) {
    void* p = nullptr;
    e = cudaGetSymbolAddress(&p, g_route_scratch);
    if (e != cudaSuccess) return static_cast<int>(e);
    if (!p) return LMOE_ERR_DRIVER;
    g_static_scratch_ptr[dev] = static_cast<int*>(p);
  }
  *out = g_static_scratch_ptr[dev];
  return 0;
}
}  // namespace

extern "C" int lmoe_route_permute_static(const lmoe_shape* s, const int32_t* sel, const lmoe_route* r, void* stream) {
  if (int rc = check_shape(s)) return rc;
  if (!sel || !r || !r->counts || !r->offsets || !r->perm || !r->pad_offsets || !r->pos || !r->row_src ||
      !r->tile_expert || !r->n_tiles)
    return LMOE_ERR_ARG;
  if (lmoe_route_workspace_bytes(s) > LMOE_STATIC_ROUTE_SCRATCH_BYTES) return LMOE_ERR_TOO_LARGE;
  int* chunk_hist = nullptr;
  if (int rc = static_route_scratch(&chunk_hist)) return rc;
  configure_route_kernels();
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  const int n = s->T * s->K;
  const int chunks = (n + kChunk - 1) / kChunk;
  const int blocks = (chunks + kRouteWarps - 1) / kRouteWarps;
  // Nothing in the scratch has to start at zero: pass 1 writes every word that passes 2 and 3 read,
  // so what an earlier call left behind is never observed.
  count_launch(3);
  route_hist_kernel<<<blocks, kRouteWarps * 32, 0, st>>>(sel, n, s->E, chunk_hist);
  route_scan_chunks_kernel<<<s->E, 256, 0, st>>>(chunk_hist, chunks, s->E, r->counts);
  route_scatter_kernel<<<blocks, kRouteWarps * 32, 0, st>>>(sel, n, s->E, chunk_hist, r->counts, r->offsets,
                                                           r->pad_offsets, r->tile_expert, r->n_tiles, r->perm, r->pos,
                                                           r->row_src);
  cudaError_t e = cudaGetLastError();
  return e == cudaSuccess ? 0 : static_cast<int>(e);
}

static int launch_bias_update(int E, const int32_t* counts, float gamma, float* expert_bias, float* load_history,
                              int64_t* update_count, void* stream) {
  if (!counts || !expert_bias || !load_history) return LMOE_ERR_ARG;
  if (E <= 0 || E > LMOE_MAX_EXPERTS) return LMOE_ERR_SHAPE;
  count_launch();
  bias_update_kernel<<<1, LMOE_MAX_EXPERTS, 0, static_cast<cudaStream_t>(stream)>>>(
      counts, E, gamma, expert_bias, load_history, reinterpret_cast<long long*>(update_count));
  cudaError_t e = cudaGetLastError();
  return e == cudaSuccess ? 0 : static_cast<int>(e);
}

extern "C" int lmoe_router_bias_update(const lmoe_shape* s, const int32_t* counts, float gamma, float* expert_bias,
                                       float* load_history, void* stream) {
  if (int rc = check_shape(s)) return rc;
  return launch_bias_update(s->E, counts, gamma, expert_bias, load_history, nullptr, stream);
}

extern "C" int lmoe_router_bias_update_counted(int E, const int32_t* counts, float gamma, float* expert_bias,
                                               float* load_history, int64_t* update_count, void* stream) {
  if (!update_count) return LMOE_ERR_ARG;
  return launch_bias_update(E, counts, gamma, expert_bias, load_history, update_count, stream);
}
