// knj_topk.cuh -- softmax + exact top-k + renormalise over one token's router
// logits by one warp; shared by the router kernels and the fused decode stack.
#pragma once
#include "knj_common.cuh"

namespace knj {

// ---------------------------------------------------------------------------
// Softmax + exact top-k + renormalise: one warp per token. Selection is by
// (value descending, expert id ascending), the tie rule of the CPU path's
// strict '>' scan (src/model/model.cpp:442-451). An expert with logit -inf
// (masked by its bias) is a candidate like any other, below every finite one:
// with fewer than k finite logits the rest are the masked experts of lowest id,
// weight 0, as in the CPU path, so that a selection is always an expert of the
// layer (it indexes tables). A row of -inf alone has weights 0.
// ---------------------------------------------------------------------------
constexpr int kMaxEPerLane = 8;  // E <= 256

// A lane's EPL logits of a token: experts 32 i + lane (-inf past the last).
template <int EPL>
__device__ __forceinline__ void topk_load(const float *lg, int E, int lane, float (&v)[EPL]) {
#pragma unroll
  for (int i = 0; i < EPL; ++i) v[i] = i * 32 + lane < E ? __ldcg(lg + i * 32 + lane) : -INFINITY;
}

// One warp: softmax over the E logits of a token (topk_load), exact top-k, renormalised weights. Lane s < k ends up with
// the s-th selection. k <= E <= 32 * EPL; fewer experts per lane than the maximum only shortens the loops.
// A token's selection is one dependent chain, so it is kept short: every lane sorts its own few keys first (stable, so
// equal keys stay in id order), and a round is then one warp maximum over the lanes' heads, one ballot, and the
// winner's queue moving up; the values are fetched from the winner off the chain, and only the k selected are divided by
// the softmax sum. (Two warp reductions, a scan and a shuffle in each round, and EPL divisions, took 2.2 us a token.)
// NT tokens at a time share the chain's latency: their steps are independent of each other.
template <int EPL, int NT>
__device__ __forceinline__ void warp_topk(const float (&v)[NT][EPL], int E, int k, int lane, int (&sel_e)[NT], float (&sel_w)[NT]) {
  float mx[NT], sum[NT], ex[NT][EPL];
  unsigned key[NT][EPL];
  int id[NT][EPL];
#pragma unroll
  for (int n = 0; n < NT; ++n) {
    mx[n] = v[n][0];
#pragma unroll
    for (int i = 1; i < EPL; ++i) mx[n] = fmaxf(mx[n], v[n][i]);
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1)
#pragma unroll
    for (int n = 0; n < NT; ++n) mx[n] = fmaxf(mx[n], __shfl_xor_sync(0xffffffffu, mx[n], o));
#pragma unroll
  for (int n = 0; n < NT; ++n) {
    sum[n] = 0.f;
    sel_e[n] = 0;
    sel_w[n] = 0.f;
#pragma unroll
    for (int i = 0; i < EPL; ++i) {
      // order-preserving integer keys: larger float <=> larger unsigned key; 0 only past the last expert
      const unsigned u = __float_as_uint(v[n][i]);
      key[n][i] = i * 32 + lane < E ? max(1u, (u & 0x80000000u) ? ~u : (u | 0x80000000u)) : 0u;
      ex[n][i] = (v[n][i] == -INFINITY) ? 0.f : expf(v[n][i] - mx[n]);
      sum[n] += ex[n][i];
      id[n][i] = i * 32 + lane;
    }
#pragma unroll
    for (int r = 0; r < EPL - 1; ++r)
#pragma unroll
      for (int i = EPL - 1; i > r; --i)
        if (key[n][i] > key[n][i - 1]) {
          const unsigned tk = key[n][i]; key[n][i] = key[n][i - 1]; key[n][i - 1] = tk;
          const float te = ex[n][i]; ex[n][i] = ex[n][i - 1]; ex[n][i - 1] = te;
          const int ti = id[n][i]; id[n][i] = id[n][i - 1]; id[n][i - 1] = ti;
        }
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1)
#pragma unroll
    for (int n = 0; n < NT; ++n) sum[n] += __shfl_xor_sync(0xffffffffu, sum[n], o);
#pragma unroll 1
  for (int s = 0; s < k; ++s) {
    unsigned top[NT];
    int src[NT];
#pragma unroll
    for (int n = 0; n < NT; ++n) top[n] = __reduce_max_sync(0xffffffffu, key[n][0]);
#pragma unroll
    for (int n = 0; n < NT; ++n) {
      const unsigned holders = __ballot_sync(0xffffffffu, key[n][0] == top[n]);
      src[n] = __ffs(holders) - 1;
      if (holders & (holders - 1u))  // equal logits: the smallest id among the lanes that hold one
        src[n] = __reduce_min_sync(0xffffffffu, key[n][0] == top[n] ? id[n][0] : 0x7fffffff) & 31;
    }
#pragma unroll
    for (int n = 0; n < NT; ++n) {
      const int e = __shfl_sync(0xffffffffu, id[n][0], src[n]);
      const float x = __shfl_sync(0xffffffffu, ex[n][0], src[n]);
      if (lane == s) {
        sel_e[n] = e;
        sel_w[n] = x;
      }
      if (lane == src[n]) {
#pragma unroll
        for (int i = 0; i + 1 < EPL; ++i) {
          key[n][i] = key[n][i + 1];
          ex[n][i] = ex[n][i + 1];
          id[n][i] = id[n][i + 1];
        }
        key[n][EPL - 1] = 0u;
      }
    }
  }
  float keep[NT];
#pragma unroll
  for (int n = 0; n < NT; ++n) {
    sel_w[n] = sum[n] == 0.f ? 0.f : sel_w[n] / sum[n];  // no finite logit: 0, not 0 / 0
    keep[n] = 0.f;
  }
#pragma unroll
  for (int s = 0; s < 8; ++s)
#pragma unroll
    for (int n = 0; n < NT; ++n) {
      const float w = __shfl_sync(0xffffffffu, sel_w[n], s);
      if (s < k) keep[n] += w;
    }
#pragma unroll
  for (int n = 0; n < NT; ++n) sel_w[n] *= keep[n] > 0.f ? 1.0f / keep[n] : 0.f;
}

// The same for one token whose logits lie at lg.
__device__ __forceinline__ void warp_topk(const float *lg, int E, int k, int lane, int &sel_e, float &sel_w) {
  int e[1];
  float w[1];
  if (E <= 128) {
    float v[1][4];
    topk_load<4>(lg, E, lane, v[0]);
    warp_topk<4, 1>(v, E, k, lane, e, w);
  } else {
    float v[1][kMaxEPerLane];
    topk_load<kMaxEPerLane>(lg, E, lane, v[0]);
    warp_topk<kMaxEPerLane, 1>(v, E, k, lane, e, w);
  }
  sel_e = e[0];
  sel_w = w[0];
}

}  // namespace knj
