// Warp-level router selection of one token: sigmoid affinities, canonical top-K of affinity + bias (higher score first, lower
// expert index on ties), logsumexp.  Shared by the router kernel and the few-token kernel.
#pragma once
#include <cuda_runtime.h>
#include <math_constants.h>
#include <stdint.h>

namespace lmoe {

__device__ __forceinline__ float sigmoid_f(float x) { return 1.0f / (1.0f + expf(-x)); }

// Compare-exchange of two (key, slot) pairs: the larger key first, the lower slot on equal keys.
__device__ __forceinline__ void topk_order(unsigned& ka, unsigned& ja, unsigned& kb, unsigned& jb) {
  const bool swap = kb > ka || (kb == ka && jb < ja);
  const unsigned k = ka, j = ja;
  ka = swap ? kb : ka;
  ja = swap ? jb : ja;
  kb = swap ? k : kb;
  jb = swap ? j : jb;
}

// Lane l holds the PER consecutive experts l*PER .. l*PER+PER-1 (PER * 32 >= E), so "lower expert index" is "lower lane, then
// lower slot".  Every lane sorts its keys once; a round is then one redux over the lanes' heads, one ballot and a
// find-first-set, and only the winning lane drops its head.  (Searching all PER keys in every round took three times the
// instructions: 135 us for 131,072 tokens, top-12 of 128.)  Keys order like the scores (-0 folded onto +0); a used or
// absent key is 0, below every real one.
// On return lane k < K holds the k-th expert and its affinity, all lanes aff_sum (slot order) and lse.
template <int PER>
__device__ __forceinline__ void topk_row(const float* row, const float* bias, int E, int K, int lane,
                                         int& my_idx, float& my_aff, float& aff_sum, float& lse) {
  float x[PER];
  unsigned key[PER], slot[PER];
  float mx = -CUDART_INF_F;
#pragma unroll
  for (int j = 0; j < PER; ++j) {
    const int e = lane * PER + j;
    slot[j] = j;
    key[j] = 0u;
    x[j] = -CUDART_INF_F;
    if (e < E) {
      x[j] = row[e];
      mx = fmaxf(mx, x[j]);
      const unsigned u = __float_as_uint((sigmoid_f(x[j]) + bias[e]) + 0.0f);
      key[j] = (u & 0x80000000u) ? ~u : (u | 0x80000000u);
    }
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
  float se = 0.f;
#pragma unroll
  for (int j = 0; j < PER; ++j)
    if (lane * PER + j < E) se += expf(x[j] - mx);
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) se += __shfl_xor_sync(0xffffffffu, se, o);
  lse = mx + logf(se);

  // odd-even merge sort, descending (1, 5 and 19 compare-exchanges for 2, 4 and 8 keys)
#pragma unroll
  for (int p = 1; p < PER; p <<= 1)
#pragma unroll
    for (int k = p; k >= 1; k >>= 1)
#pragma unroll
      for (int j = k % p; j + k < PER; j += 2 * k)
#pragma unroll
        for (int i = 0; i < k; ++i)
          if ((i + j) / (2 * p) == (i + j + k) / (2 * p) && i + j + k < PER)
            topk_order(key[i + j], slot[i + j], key[i + j + k], slot[i + j + k]);
  unsigned packed = 0u;  // four bits per sorted position
#pragma unroll
  for (int j = 0; j < PER; ++j) packed |= slot[j] << (4 * j);

  my_idx = 0;
  for (int k = 0; k < K; ++k) {
    const unsigned wmax = __reduce_max_sync(0xffffffffu, key[0]);
    const int wl = __ffs(__ballot_sync(0xffffffffu, key[0] == wmax)) - 1;  // lowest lane = lowest expert among the maxima
    const int bi = __shfl_sync(0xffffffffu, lane * PER + static_cast<int>(packed & 15u), wl);
    if (lane == k) my_idx = bi;
    if (lane == wl) {
#pragma unroll
      for (int j = 0; j + 1 < PER; ++j) key[j] = key[j + 1];
      key[PER - 1] = 0u;
      packed >>= 4;
    }
  }
  my_aff = lane < K ? sigmoid_f(row[my_idx]) : 0.f;
  aff_sum = 0.f;
  for (int k = 0; k < K; ++k) aff_sum += __shfl_sync(0xffffffffu, my_aff, k);  // slot 0, 1, ...: the same on every lane
}

}  // namespace lmoe
