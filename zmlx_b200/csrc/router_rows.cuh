// Per-token-row router device functions shared by the router kernels and the fused decode-layer kernel.
// One warp owns one token row; the row's E scores live in registers (E <= 1024); top-k order is
// (score descending, expert id ascending).
#pragma once

#include <math_constants.h>

#include "common.cuh"
#include "layer_route.cuh"

namespace zmoe {

constexpr int kMaxVPL = 32;  // values per lane: E <= 1024
constexpr int kMaxK = 16;

__device__ __forceinline__ float load_logit(const void* p, int dtype, size_t i) {
  if (dtype == ZMOE_F32) return reinterpret_cast<const float*>(p)[i];
  return __bfloat162float(reinterpret_cast<const __nv_bfloat16*>(p)[i]);
}

// Top-k of the lane-strided values v[j] (expert id = lane + 32*j) in K rounds of a warp arg-max under the canonical order
// (value descending, id ascending): one redux for the largest key, one for the lowest id that holds it; the winner leaves the
// race.  Lane r < K returns the expert of slot r.  The values are left in `vals` (E floats owned by the warp) for the caller to
// look winners up.  (Ranking every value against every other one took E * VPL comparisons a lane and left the slots' arithmetic
// to one lane.  us, before -> now: top-8 of 128, 1500 rows 9.5 -> 3.1, 4096 rows 18.8 -> 4.8; of 256 in groups, 512 rows 16.9 ->
// 8.5.)
template <int VPL>
__device__ __forceinline__ int warp_topk(const float (&v)[VPL], int E, int K, int lane, float* vals) {
  // order-preserving integer keys (ld_order_key): a total order even when a row holds NaN (NaN ranks below every number)
  uint32_t kv[VPL];
  uint32_t live = 0u;
#pragma unroll
  for (int j = 0; j < VPL; ++j) {
    const int idx = lane + 32 * j;
    kv[j] = ld_order_key(v[j] + 0.0f);
    if (idx < E) {
      vals[idx] = v[j];
      live |= 1u << j;
    }
  }
  int mine = 0;
#pragma unroll 1
  for (int r = 0; r < K; ++r) {
    uint32_t bk = 0u;
    int bj = -1;
#pragma unroll
    for (int j = 0; j < VPL; ++j)
      if (((live >> j) & 1u) && (bj < 0 || kv[j] > bk)) {
        bk = kv[j];
        bj = j;
      }
    const uint32_t mx = __reduce_max_sync(0xffffffffu, bk);
    const uint32_t win = __reduce_min_sync(0xffffffffu, bj >= 0 && bk == mx ? (uint32_t)(lane + 32 * bj) : 0xffffffffu);
    if ((int)(win & 31u) == lane) live &= ~(1u << (win >> 5));  // K <= E: there always is a winner
    if (r == lane) mine = (int)win;
  }
  __syncwarp();
  return mine;
}

// One warp routes one token row (softmax family); see zmoe_router_softmax_topk.
template <int VPL>
__device__ __forceinline__ void softmax_topk_row(const void* __restrict__ logits, int dtype, int row, int E, int K,
                                                 int flavour, const float* __restrict__ bias, int renorm,
                                                 float* __restrict__ weights, uint32_t* __restrict__ indices,
                                                 int lane, float* scratch) {
  float v[VPL];
  float mx = -CUDART_INF_F;
#pragma unroll
  for (int j = 0; j < VPL; ++j) {
    int idx = lane + 32 * j;
    v[j] = (idx < E) ? load_logit(logits, dtype, (size_t)row * E + idx) : -CUDART_INF_F;
    mx = fmaxf(mx, v[j]);
  }
  // lane i < K owns slot i; sums run over the slots in order 0..K-1 (every lane repeats them)
  if (flavour == ZMOE_ROUTER_TOPK_THEN_SOFTMAX) {
    const int si = warp_topk<VPL>(v, E, K, lane, scratch);
    const float sv = scratch[si];
    const float term = expf(sv - __shfl_sync(0xffffffffu, sv, 0));
    float s = 0.0f;
    for (int i = 0; i < K; ++i) s += __shfl_sync(0xffffffffu, term, i);
    if (lane < K) {
      weights[(size_t)row * K + lane] = term / s;
      indices[(size_t)row * K + lane] = (uint32_t)si;
    }
    return;
  }
  // full softmax [+ bias] -> top-k -> optional renormalisation
  mx = warp_max(mx);
  float sum = 0.0f;
#pragma unroll
  for (int j = 0; j < VPL; ++j) {
    int idx = lane + 32 * j;
    v[j] = (idx < E) ? expf(v[j] - mx) : 0.0f;
    sum += v[j];
  }
  sum = warp_sum(sum);
#pragma unroll
  for (int j = 0; j < VPL; ++j) {
    int idx = lane + 32 * j;
    if (idx < E) {
      v[j] = v[j] / sum;
      if (bias) v[j] += bias[idx];
    }
  }
  const int si = warp_topk<VPL>(v, E, K, lane, scratch);
  const float sv = scratch[si];
  float denom = 1.0f;
  if (renorm) {
    float sk = 0.0f;
    for (int i = 0; i < K; ++i) sk += __shfl_sync(0xffffffffu, sv, i);
    denom = (renorm == 1) ? sk + 1e-20f : sk;
  }
  if (lane < K) {
    weights[(size_t)row * K + lane] = renorm ? sv / denom : sv;
    indices[(size_t)row * K + lane] = (uint32_t)si;
  }
}

// sigmoid + selection bias, optional group-limited selection.  One warp routes one token row;
// `sc` is E + 64 floats of scratch owned by the warp (scores, then group scores and keep flags).
// Groups of whole 32s are scored in registers: expert lane + 32 j belongs to group j / (per / 32).
template <int VPL>
__device__ __forceinline__ void sigmoid_topk_row(const void* __restrict__ logits, int dtype, int row, int E, int K,
                                                 const float* __restrict__ bias, int n_group, int topk_group,
                                                 float scale, float* __restrict__ weights,
                                                 uint32_t* __restrict__ indices, int lane, float* sc) {
  float* gsc = sc + E;
  float* gkeep = gsc + 32;
  float v[VPL];
#pragma unroll
  for (int j = 0; j < VPL; ++j) {
    int idx = lane + 32 * j;
    if (idx < E) {
      float aff = sigmoid_stable(load_logit(logits, dtype, (size_t)row * E + idx));
      v[j] = aff + bias[idx];
      sc[idx] = v[j];
    } else {
      v[j] = -CUDART_INF_F;
    }
  }
  if (n_group > 1) {
    __syncwarp();
    const int per = E / n_group;
    if (per % 32 == 0) {
      float t1 = -CUDART_INF_F, t2 = -CUDART_INF_F;
#pragma unroll
      for (int j = 0; j < VPL; ++j) {
        if (32 * j < E) {
          if (v[j] > t1) {  // the same comparisons as below: a NaN is nobody's best
            t2 = t1;
            t1 = v[j];
          } else if (v[j] > t2) {
            t2 = v[j];
          }
          if ((j + 1) % (per >> 5) == 0) {  // the group is complete: merge the lanes' (largest, second largest) pairs
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) {
              const float o1 = __shfl_xor_sync(0xffffffffu, t1, o);
              const float o2 = __shfl_xor_sync(0xffffffffu, t2, o);
              t2 = fmaxf(fminf(t1, o1), fmaxf(t2, o2));
              t1 = fmaxf(t1, o1);
            }
            if (lane == 0) gsc[j / (per >> 5)] = t1 + t2;
            t1 = t2 = -CUDART_INF_F;
          }
        }
      }
    } else if (lane < n_group) {
      float t1 = -CUDART_INF_F, t2 = -CUDART_INF_F;
      for (int j = 0; j < per; ++j) {
        const float x = sc[lane * per + j];
        if (x > t1) {
          t2 = t1;
          t1 = x;
        } else if (x > t2) {
          t2 = x;
        }
      }
      gsc[lane] = t1 + t2;
    }
    __syncwarp();
    if (lane < n_group) {
      float mine = gsc[lane];
      int rank = 0;
      for (int h = 0; h < n_group; ++h) {
        float o = gsc[h];
        rank += (o > mine) || (o == mine && h < lane);
      }
      gkeep[lane] = (rank < topk_group) ? 1.0f : 0.0f;
    }
    __syncwarp();
#pragma unroll
    for (int j = 0; j < VPL; ++j) {
      int idx = lane + 32 * j;
      if (idx < E && gkeep[idx / per] == 0.0f) v[j] = 0.0f;
    }
  }
  __syncwarp();
  const int si = warp_topk<VPL>(v, E, K, lane, sc);
  const float aff = sigmoid_stable(load_logit(logits, dtype, (size_t)row * E + si));
  float sum = 0.0f;
  for (int i = 0; i < K; ++i) sum += __shfl_sync(0xffffffffu, aff, i);
  const float inv = 1.0f / sum;
  float w = aff * inv;
  if (scale != 1.0f) w = w * scale;
  if (lane < K) {
    weights[(size_t)row * K + lane] = w;
    indices[(size_t)row * K + lane] = (uint32_t)si;
  }
}

}  // namespace zmoe
