// The attention side of the stacked decoder: RMSNorm with the residual add in front of it, q/k normalisation + RoPE +
// cache append, and one-token grouped-query attention over the KV cache.  Everything is float32 arithmetic on bfloat16
// storage, rounded where the model rounds (the normalised row, the rotated head, the attention output).
#include "common.cuh"

namespace zmoe {

// ------------------------------------------------------------------ residual add + RMSNorm
// One CTA per row: h += delta (rounded to bfloat16, stored back), x = bf16(h * rsqrt(mean(h^2) + eps) * w).
// Bound by latency at decode sizes (a row is 4 KB): one launch in place of the seven elementwise and reduction
// kernels of the op-by-op form.
constexpr int kNormThreads = 256;
constexpr int kNormMaxVec = 8;  // 16-byte pieces a thread keeps: d up to 16384

__global__ void __launch_bounds__(kNormThreads) add_rms_norm_kernel(__nv_bfloat16* h, const __nv_bfloat16* delta,
                                                                    const __nv_bfloat16* w, float eps, int d,
                                                                    __nv_bfloat16* x) {
  __shared__ float part[kNormThreads / 32];
  pdl_wait();
  pdl_trigger();
  const int tid = threadIdx.x, nv = d >> 3;
  const size_t row = (size_t)blockIdx.x * d;
  uint4 v[kNormMaxVec];
  float ss = 0.0f;
#pragma unroll
  for (int j = 0; j < kNormMaxVec; ++j) {
    const int i = tid + j * kNormThreads;
    if (i < nv) {
      v[j] = *(reinterpret_cast<const uint4*>(h + row) + i);
      if (delta != nullptr) {
        const uint4 a = *(reinterpret_cast<const uint4*>(delta + row) + i);
        uint32_t* q = reinterpret_cast<uint32_t*>(&v[j]);
        const uint32_t p[4] = {a.x, a.y, a.z, a.w};
#pragma unroll
        for (int k = 0; k < 4; ++k) {
          const float lo = bf16_bits_to_float(q[k] & 0xffffu) + bf16_bits_to_float(p[k] & 0xffffu);
          const float hi = bf16_bits_to_float(q[k] >> 16) + bf16_bits_to_float(p[k] >> 16);
          q[k] = (uint32_t)float_to_bf16_bits(lo) | ((uint32_t)float_to_bf16_bits(hi) << 16);
        }
        *(reinterpret_cast<uint4*>(h + row) + i) = v[j];
      }
      const uint32_t q[4] = {v[j].x, v[j].y, v[j].z, v[j].w};
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        const float lo = bf16_bits_to_float(q[k] & 0xffffu), hi = bf16_bits_to_float(q[k] >> 16);
        ss = fmaf(lo, lo, ss);
        ss = fmaf(hi, hi, ss);
      }
    }
  }
  ss = warp_sum(ss);
  if ((tid & 31) == 0) part[tid >> 5] = ss;
  __syncthreads();
  float total = 0.0f;
#pragma unroll
  for (int i = 0; i < kNormThreads / 32; ++i) total += part[i];
  const float r = rsqrtf(total / (float)d + eps);
#pragma unroll
  for (int j = 0; j < kNormMaxVec; ++j) {
    const int i = tid + j * kNormThreads;
    if (i < nv) {
      const uint4 wv = __ldg(reinterpret_cast<const uint4*>(w) + i);
      const uint32_t q[4] = {v[j].x, v[j].y, v[j].z, v[j].w}, p[4] = {wv.x, wv.y, wv.z, wv.w};
      uint32_t o[4];
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        const float lo = (bf16_bits_to_float(q[k] & 0xffffu) * r) * bf16_bits_to_float(p[k] & 0xffffu);
        const float hi = (bf16_bits_to_float(q[k] >> 16) * r) * bf16_bits_to_float(p[k] >> 16);
        o[k] = (uint32_t)float_to_bf16_bits(lo) | ((uint32_t)float_to_bf16_bits(hi) << 16);
      }
      *(reinterpret_cast<uint4*>(x + row) + i) = make_uint4(o[0], o[1], o[2], o[3]);
    }
  }
}

// ------------------------------------------------------------------ q/k norm + RoPE + cache append
struct QkvParams {
  const __nv_bfloat16 *q, *k, *v;    // (B*S, heads*hd) projections
  const __nv_bfloat16 *qn, *kn;      // (hd) norm weights
  const float *cos, *sin;            // (positions, hd/2)
  __nv_bfloat16* qo;                 // (B, Hq, S, hd)
  __nv_bfloat16 *kc, *vc;            // (B, Hk, max_seq, hd) of this layer
  const long long* pos_dev;          // position of the first of the S tokens, or NULL: pos0
  int pos0, B, S, hq, hk, hd, max_seq;
  float eps;
};

// One warp per (token, head).  A head's two halves are rotated against each other; a lane owns the pairs (i, i + hd/2).
__global__ void __launch_bounds__(256) qkv_post_kernel(const QkvParams p) {
  pdl_wait();
  pdl_trigger();
  const int lane = threadIdx.x & 31;
  const int heads = p.hq + 2 * p.hk;
  const long long unit = (long long)blockIdx.x * 8 + (threadIdx.x >> 5);
  if (unit >= (long long)p.B * p.S * heads) return;
  const int tok = (int)(unit / heads), head = (int)(unit - (long long)tok * heads);
  const int b = tok / p.S, s = tok - b * p.S;
  const int pos = (p.pos_dev != nullptr ? (int)*p.pos_dev : p.pos0) + s;
  const int hd = p.hd, h2 = hd >> 1;
  if (pos < 0 || pos >= p.max_seq) return;
  if (head >= p.hq + p.hk) {  // value heads: a copy
    const int hv = head - p.hq - p.hk;
    const __nv_bfloat16* src = p.v + ((size_t)tok * p.hk + hv) * hd;
    __nv_bfloat16* dst = p.vc + (((size_t)b * p.hk + hv) * p.max_seq + pos) * hd;
    for (int i = lane; i < h2; i += 32) reinterpret_cast<uint32_t*>(dst)[i] = reinterpret_cast<const uint32_t*>(src)[i];
    return;
  }
  const bool is_q = head < p.hq;
  const int hh = is_q ? head : head - p.hq;
  const __nv_bfloat16* src = is_q ? p.q + ((size_t)tok * p.hq + hh) * hd : p.k + ((size_t)tok * p.hk + hh) * hd;
  const __nv_bfloat16* w = is_q ? p.qn : p.kn;
  __nv_bfloat16* dst = is_q ? p.qo + (((size_t)b * p.hq + hh) * p.S + s) * hd
                            : p.kc + (((size_t)b * p.hk + hh) * p.max_seq + pos) * hd;
  float ss = 0.0f;
  for (int i = lane; i < hd; i += 32) {
    const float v = __bfloat162float(src[i]);
    ss = fmaf(v, v, ss);
  }
  const float r = rsqrtf(warp_sum(ss) / (float)hd + p.eps);
  for (int i = lane; i < h2; i += 32) {
    const float x1 = round_bf16((__bfloat162float(src[i]) * r) * __bfloat162float(w[i]));
    const float x2 = round_bf16((__bfloat162float(src[i + h2]) * r) * __bfloat162float(w[i + h2]));
    const float c = __ldg(p.cos + (size_t)pos * h2 + i), sn = __ldg(p.sin + (size_t)pos * h2 + i);
    dst[i] = __float2bfloat16_rn(__fsub_rn(__fmul_rn(x1, c), __fmul_rn(x2, sn)));
    dst[i + h2] = __float2bfloat16_rn(__fadd_rn(__fmul_rn(x2, c), __fmul_rn(x1, sn)));
  }
}

// ------------------------------------------------------------------ one-token attention over the cache
// A CTA owns one (sequence, KV head) and a slice of the positions, for all REP query heads that share the KV head: the
// cache is read once, where the op-by-op form first wrote float32 copies of it.  Per block of 64 positions: scores (a row of keys is split over HD/8 lanes, the REP sums are
// folded by halving exchanges), a running maximum, probabilities in shared memory, values (a thread owns two
// dimensions and every fourth position).  Bound by the cache's way from HBM (2 * hd * 2 bytes per position and KV
// head); slices are as many as fill the chip.  With the norm and q/k kernels above, a decode step of four sequences at
// position 3000 through four layers went from 3.31 to 0.71 ms (0.62 of it the projections, blocks and the head).
constexpr int kAttThreads = 256, kAttBlock = 64;

struct AttParams {
  const __nv_bfloat16 *q, *kc, *vc;  // (B, Hq, hd), caches (B, Hk, max_seq, hd)
  const long long* pos_dev;          // last valid position, or NULL: npos - 1
  int npos, hk, max_seq, nsplit;
  float scale;
  float* part;  // (B*Hk, nsplit, REP, hd + 2): accumulator, maximum, sum
  __nv_bfloat16* out;  // (B, Hq, hd)
};

template <int HD, int REP>
__global__ void __launch_bounds__(kAttThreads) decode_attn_kernel(const AttParams p) {
  constexpr int LPR = HD / 8;            // lanes per key row
  constexpr int RPW = 32 / LPR;          // rows a warp takes at once
  constexpr int PAIRS = HD / 2;          // value threads across the dimensions
  constexpr int GRP = kAttThreads / PAIRS;
  __shared__ float sc[kAttBlock][REP];   // scores, then probabilities
  __shared__ float red[GRP][REP][HD];
  __shared__ float run_m[REP], run_s[REP], fac[REP];
  pdl_wait();  // from here on plain loads: the non-coherent path must not run ahead of the wait
  pdl_trigger();
  const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
  const int pair = blockIdx.y, b = pair / p.hk, kh = pair - b * p.hk;
  const int P = p.pos_dev != nullptr ? min((int)*p.pos_dev + 1, p.max_seq) : p.npos;
  const int per = ((P + p.nsplit - 1) / p.nsplit + kAttBlock - 1) / kAttBlock * kAttBlock;
  const int lo = min((int)blockIdx.x * per, P), hi = min(lo + per, P);
  const __nv_bfloat16* kc = p.kc + ((size_t)b * p.hk + kh) * p.max_seq * HD;
  const __nv_bfloat16* vc = p.vc + ((size_t)b * p.hk + kh) * p.max_seq * HD;
  // this lane's eight dimensions of the REP queries, scaled
  float q[REP][8];
#pragma unroll
  for (int r = 0; r < REP; ++r) {
    const uint4 v = *(reinterpret_cast<const uint4*>(p.q + (((size_t)b * p.hk + kh) * REP + r) * HD) + lane % LPR);
    const uint32_t u[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      q[r][2 * k] = bf16_bits_to_float(u[k] & 0xffffu);
      q[r][2 * k + 1] = bf16_bits_to_float(u[k] >> 16);
    }
  }
  if (tid < REP) {
    run_m[tid] = -INFINITY;
    run_s[tid] = 0.0f;
  }
  float acc[REP][2];
#pragma unroll
  for (int r = 0; r < REP; ++r) acc[r][0] = acc[r][1] = 0.0f;
  const int dp = tid % PAIRS, grp = tid / PAIRS;

  for (int p0 = lo; p0 < hi; p0 += kAttBlock) {
    const int n = min(kAttBlock, hi - p0);
    // the block's values are requested before the scores are worked out
    uint32_t vv[kAttBlock / GRP];
#pragma unroll
    for (int j = 0; j < kAttBlock / GRP; ++j) {
      const int i = grp + j * GRP;
      vv[j] = i < n ? *(reinterpret_cast<const uint32_t*>(vc + (size_t)(p0 + i) * HD) + dp) : 0u;
    }
    __syncthreads();  // the previous block's probabilities are used up
#pragma unroll
    for (int j = 0; j < kAttBlock / (8 * RPW); ++j) {
      const int i = (j * 8 + wid) * RPW + lane / LPR;
      float s[REP];
#pragma unroll
      for (int r = 0; r < REP; ++r) s[r] = 0.0f;
      if (i < n) {
        const uint4 v = *(reinterpret_cast<const uint4*>(kc + (size_t)(p0 + i) * HD) + lane % LPR);
        const uint32_t u[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
        for (int k = 0; k < 4; ++k) {
          const float a0 = bf16_bits_to_float(u[k] & 0xffffu), a1 = bf16_bits_to_float(u[k] >> 16);
#pragma unroll
          for (int r = 0; r < REP; ++r) s[r] = fmaf(a1, q[r][2 * k + 1], fmaf(a0, q[r][2 * k], s[r]));
        }
      }
      // fold over the row's lanes: every exchange halves the heads a lane still carries, then plain butterflies
      int head = 0;
      int o = LPR >> 1;
#pragma unroll
      for (int cnt = REP; cnt > 1 && o > 0; cnt >>= 1, o >>= 1) {
        const bool up = (lane & o) != 0;
#pragma unroll
        for (int r = 0; r < cnt / 2; ++r) {
          const float give = up ? s[r] : s[r + cnt / 2], keep = up ? s[r + cnt / 2] : s[r];
          s[r] = keep + __shfl_xor_sync(0xffffffffu, give, o);
        }
        if (up) head += cnt / 2;
      }
      for (; o > 0; o >>= 1) s[0] += __shfl_xor_sync(0xffffffffu, s[0], o);
      // lanes whose low bits are zero hold one head each
      if ((lane % LPR) % (LPR / REP) == 0) sc[i][head] = i < n ? s[0] * p.scale : -INFINITY;
    }
    __syncthreads();
    if (wid < REP) {  // one warp per head: running maximum and sum
      const float s0 = sc[lane][wid], s1 = sc[lane + 32][wid];
      const float m = fmaxf(run_m[wid], warp_max(fmaxf(s0, s1)));
      const float ref = m == -INFINITY ? 0.0f : m;  // every score so far is -inf: their weights are 0, not exp(-inf + inf)
      const float e0 = expf(s0 - ref), e1 = expf(s1 - ref);
      const float sum = warp_sum(e0 + e1);
      sc[lane][wid] = e0;
      sc[lane + 32][wid] = e1;
      if (lane == 0) {
        const float f = expf(run_m[wid] - ref);
        fac[wid] = f;
        run_s[wid] = run_s[wid] * f + sum;
        run_m[wid] = m;
      }
    }
    __syncthreads();
#pragma unroll
    for (int r = 0; r < REP; ++r) {
      acc[r][0] *= fac[r];
      acc[r][1] *= fac[r];
    }
#pragma unroll
    for (int j = 0; j < kAttBlock / GRP; ++j) {
      const int i = grp + j * GRP;
      if (i < n) {
        const float v0 = bf16_bits_to_float(vv[j] & 0xffffu), v1 = bf16_bits_to_float(vv[j] >> 16);
#pragma unroll
        for (int r = 0; r < REP; ++r) {
          const float pr = sc[i][r];
          acc[r][0] = fmaf(pr, v0, acc[r][0]);
          acc[r][1] = fmaf(pr, v1, acc[r][1]);
        }
      }
    }
  }
#pragma unroll
  for (int r = 0; r < REP; ++r) *reinterpret_cast<float2*>(&red[grp][r][2 * dp]) = make_float2(acc[r][0], acc[r][1]);
  __syncthreads();
  float* part = p.part + ((size_t)pair * p.nsplit + blockIdx.x) * REP * (HD + 2);
  for (int i = tid; i < REP * HD; i += kAttThreads) {
    const int r = i / HD, c = i - r * HD;
    float t = 0.0f;
#pragma unroll
    for (int k = 0; k < GRP; ++k) t += red[k][r][c];
    part[r * (HD + 2) + c] = t;
  }
  if (tid < REP) {
    part[tid * (HD + 2) + HD] = run_m[tid];
    part[tid * (HD + 2) + HD + 1] = run_s[tid];
  }
}

// One CTA of hd threads per query head: the slices' partial results under their common maximum.
__global__ void decode_attn_join_kernel(const float* part, int nsplit, int rep, int hd, __nv_bfloat16* out) {
  pdl_wait();
  pdl_trigger();
  const int head = blockIdx.x, c = threadIdx.x;
  const int pair = head / rep, r = head - pair * rep;
  const size_t step = (size_t)rep * (hd + 2);
  const float* base = part + (size_t)pair * nsplit * step + (size_t)r * (hd + 2);
  float m = -INFINITY;
  for (int s = 0; s < nsplit; ++s) m = fmaxf(m, base[s * step + hd]);
  float num = 0.0f, den = 0.0f;
  for (int s = 0; s < nsplit; ++s) {
    const float ms = base[s * step + hd];
    const float f = ms == -INFINITY ? 0.0f : expf(ms - m);  // an empty slice
    num = fmaf(f, base[s * step + c], num);
    den = fmaf(f, base[s * step + hd + 1], den);
  }
  out[(size_t)head * hd + c] = __float2bfloat16_rn(num / den);
}

static int attn_splits(int B, int hk, int max_pos) {
  const int want = (2 * 148 + B * hk - 1) / (B * hk);  // about two CTAs per SM
  const int most = (max_pos + kAttBlock - 1) / kAttBlock;
  return want < most ? want : (most > 0 ? most : 1);
}

template <int HD>
static int launch_attn(const AttParams& p, int rep, dim3 grid, cudaStream_t st) {
  cudaError_t e;
  switch (rep) {
    case 1: e = launch_pdl(decode_attn_kernel<HD, 1>, grid, dim3(kAttThreads), 0, st, p); break;
    case 2: e = launch_pdl(decode_attn_kernel<HD, 2>, grid, dim3(kAttThreads), 0, st, p); break;
    case 4: e = launch_pdl(decode_attn_kernel<HD, 4>, grid, dim3(kAttThreads), 0, st, p); break;
    default: e = launch_pdl(decode_attn_kernel<HD, 8>, grid, dim3(kAttThreads), 0, st, p); break;
  }
  if (e != cudaSuccess) return fail(ZMOE_ERR_CUDA, "zmoe_decode_attention: %s", cudaGetErrorString(e));
  return check_launch("decode_attn_kernel");
}

}  // namespace zmoe

using namespace zmoe;

extern "C" {

int zmoe_add_rms_norm(void* h, const void* delta, const void* w, float eps, int rows, int d, void* x, void* stream) {
  ZMOE_REQUIRE(h && w && x, ZMOE_ERR_SHAPE, "zmoe_add_rms_norm: null pointer");
  ZMOE_REQUIRE(rows >= 0 && d >= 8, ZMOE_ERR_SHAPE, "zmoe_add_rms_norm: bad sizes rows=%d d=%d", rows, d);
  ZMOE_REQUIRE(d % 8 == 0 && d <= 8 * kNormThreads * kNormMaxVec, ZMOE_ERR_UNSUPPORTED,
               "zmoe_add_rms_norm: d=%d (a multiple of 8 up to %d)", d, 8 * kNormThreads * kNormMaxVec);
  ZMOE_REQUIRE((((uintptr_t)h | (uintptr_t)delta | (uintptr_t)w | (uintptr_t)x) & 15) == 0, ZMOE_ERR_ALIGN,
               "zmoe_add_rms_norm: rows must be 16-byte aligned");
  if (rows == 0) return ZMOE_OK;
  launch_pdl(add_rms_norm_kernel, dim3(rows), dim3(kNormThreads), 0, (cudaStream_t)stream, (__nv_bfloat16*)h,
             (const __nv_bfloat16*)delta, (const __nv_bfloat16*)w, eps, d, (__nv_bfloat16*)x);
  return check_launch("zmoe_add_rms_norm");
}

int zmoe_qkv_post(const void* q, const void* k, const void* v, const void* q_norm, const void* k_norm,
                  const float* cos_t, const float* sin_t, float eps, int B, int S, int hq, int hk, int hd,
                  const int64_t* pos_dev, int pos0, int max_seq, void* q_out, void* k_cache, void* v_cache,
                  void* stream) {
  ZMOE_REQUIRE(q && k && v && q_norm && k_norm && cos_t && sin_t && q_out && k_cache && v_cache, ZMOE_ERR_SHAPE,
               "zmoe_qkv_post: null pointer");
  ZMOE_REQUIRE(B >= 0 && S >= 0 && hq >= 1 && hk >= 1 && hd >= 2 && max_seq >= 1, ZMOE_ERR_SHAPE,
               "zmoe_qkv_post: bad sizes B=%d S=%d heads=%d/%d hd=%d", B, S, hq, hk, hd);
  ZMOE_REQUIRE(hd % 2 == 0, ZMOE_ERR_UNSUPPORTED, "zmoe_qkv_post: hd=%d must be even", hd);
  ZMOE_REQUIRE(pos_dev || (pos0 >= 0 && pos0 + S <= max_seq), ZMOE_ERR_SHAPE,
               "zmoe_qkv_post: positions %d..%d beyond the cache of %d", pos0, pos0 + S, max_seq);
  ZMOE_REQUIRE((((uintptr_t)v | (uintptr_t)v_cache) & 3) == 0, ZMOE_ERR_ALIGN, "zmoe_qkv_post: v must be 4-byte aligned");
  if (B == 0 || S == 0) return ZMOE_OK;
  QkvParams p;
  p.q = (const __nv_bfloat16*)q;
  p.k = (const __nv_bfloat16*)k;
  p.v = (const __nv_bfloat16*)v;
  p.qn = (const __nv_bfloat16*)q_norm;
  p.kn = (const __nv_bfloat16*)k_norm;
  p.cos = cos_t;
  p.sin = sin_t;
  p.qo = (__nv_bfloat16*)q_out;
  p.kc = (__nv_bfloat16*)k_cache;
  p.vc = (__nv_bfloat16*)v_cache;
  p.pos_dev = (const long long*)pos_dev;
  p.pos0 = pos0;
  p.B = B;
  p.S = S;
  p.hq = hq;
  p.hk = hk;
  p.hd = hd;
  p.max_seq = max_seq;
  p.eps = eps;
  const long long units = (long long)B * S * (hq + 2 * hk);
  ZMOE_REQUIRE(units < (8ll << 31), ZMOE_ERR_UNSUPPORTED, "zmoe_qkv_post: too many tokens");
  launch_pdl(qkv_post_kernel, dim3((unsigned)((units + 7) / 8)), dim3(256), 0, (cudaStream_t)stream, p);
  return check_launch("zmoe_qkv_post");
}

size_t zmoe_decode_attention_workspace_bytes(int B, int hq, int hk, int hd, int max_pos) {
  if (B < 1 || hk < 1 || hq < hk || hq % hk || max_pos < 1) return 0;
  const int rep = hq / hk;
  if ((hd != 64 && hd != 128) || (rep != 1 && rep != 2 && rep != 4 && rep != 8) || (long long)B * hk > 65535) return 0;
  return (size_t)B * hq * attn_splits(B, hk, max_pos) * (hd + 2) * sizeof(float);
}

int zmoe_decode_attention(const void* q, const void* k_cache, const void* v_cache, int B, int hq, int hk, int hd,
                          const int64_t* pos_dev, int npos, int max_seq, float scale, void* workspace,
                          size_t workspace_bytes, void* out, void* stream) {
  ZMOE_REQUIRE(q && k_cache && v_cache && out && workspace, ZMOE_ERR_SHAPE, "zmoe_decode_attention: null pointer");
  const int most = pos_dev ? max_seq : npos;
  const size_t need = zmoe_decode_attention_workspace_bytes(B, hq, hk, hd, most);
  ZMOE_REQUIRE(need > 0, ZMOE_ERR_UNSUPPORTED,
               "zmoe_decode_attention: head dimension 64 or 128 and 1, 2, 4 or 8 query heads per KV head (B=%d hq=%d "
               "hk=%d hd=%d positions=%d)", B, hq, hk, hd, most);
  ZMOE_REQUIRE(most <= max_seq, ZMOE_ERR_SHAPE, "zmoe_decode_attention: %d positions beyond the cache of %d", most, max_seq);
  ZMOE_REQUIRE(workspace_bytes >= need, ZMOE_ERR_WORKSPACE, "zmoe_decode_attention: workspace of %zu bytes, need %zu",
               workspace_bytes, need);
  ZMOE_REQUIRE((((uintptr_t)q | (uintptr_t)k_cache | (uintptr_t)v_cache) & 15) == 0, ZMOE_ERR_ALIGN,
               "zmoe_decode_attention: q and the caches must be 16-byte aligned");
  AttParams p;
  p.q = (const __nv_bfloat16*)q;
  p.kc = (const __nv_bfloat16*)k_cache;
  p.vc = (const __nv_bfloat16*)v_cache;
  p.pos_dev = (const long long*)pos_dev;
  p.npos = npos;
  p.hk = hk;
  p.max_seq = max_seq;
  p.nsplit = attn_splits(B, hk, most);
  p.scale = scale;
  p.part = (float*)workspace;
  p.out = (__nv_bfloat16*)out;
  cudaStream_t st = (cudaStream_t)stream;
  const int rep = hq / hk;
  const dim3 grid(p.nsplit, B * hk);
  const int rc = hd == 128 ? launch_attn<128>(p, rep, grid, st) : launch_attn<64>(p, rep, grid, st);
  if (rc != ZMOE_OK) return rc;
  launch_pdl(decode_attn_join_kernel, dim3(B * hq), dim3(hd), 0, st, (const float*)workspace, p.nsplit, rep, hd,
             (__nv_bfloat16*)out);
  return check_launch("decode_attn_join_kernel");
}

}  // extern "C"
