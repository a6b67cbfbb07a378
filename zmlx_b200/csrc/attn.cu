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

// The same for heads of up to 128 values, a multiple of four, on 4-byte boundaries: a warp takes four heads of a token, a lane
// the values (2 l, 2 l + 1) of both halves, every load is under way before the first is used, and the token's rotation is
// read once for the four.  The form above is bound by its chains of short loads and by instructions per byte: 1500 tokens with 40
// heads of 128 took 25.2 us, they take 14.5 now.  As long as one warp per head does not fill the chip (64 on each of some 150
// SMs) it stays the faster one: a token of four sequences 3.0 us, against 3.3 here.
constexpr int kQkvHeads = 4;

__global__ void __launch_bounds__(256) qkv_post4_kernel(const QkvParams p) {
  pdl_wait();
  pdl_trigger();
  const int lane = threadIdx.x & 31;
  const unsigned heads = p.hq + 2 * p.hk, groups = (heads + kQkvHeads - 1) / kQkvHeads;
  const unsigned unit = blockIdx.x * 8 + (threadIdx.x >> 5);
  if (unit >= (unsigned)p.B * p.S * groups) return;
  const int tok = unit / groups, head0 = (unit - tok * groups) * kQkvHeads;
  const int b = tok / p.S, s = tok - b * p.S;
  const int pos = (p.pos_dev != nullptr ? (int)*p.pos_dev : p.pos0) + s;
  if (pos < 0 || pos >= p.max_seq) return;
  const int hd = p.hd, h4 = hd >> 2;  // 32-bit words of a half
  const bool act = lane < h4;
  uint32_t lo[kQkvHeads], hi[kQkvHeads];
#pragma unroll
  for (int j = 0; j < kQkvHeads; ++j) {
    const int h = head0 + j;
    lo[j] = hi[j] = 0u;
    if (act && h < (int)heads) {
      const __nv_bfloat16* row = h < p.hq ? p.q + ((size_t)tok * p.hq + h) * hd
                                 : h < p.hq + p.hk ? p.k + ((size_t)tok * p.hk + h - p.hq) * hd
                                                   : p.v + ((size_t)tok * p.hk + h - p.hq - p.hk) * hd;
      lo[j] = reinterpret_cast<const uint32_t*>(row)[lane];
      hi[j] = reinterpret_cast<const uint32_t*>(row)[h4 + lane];
    }
  }
  float2 c = make_float2(0.0f, 0.0f), sn = c;
  uint32_t wq[2] = {0u, 0u}, wk[2] = {0u, 0u};
  if (act) {
    c = __ldg(reinterpret_cast<const float2*>(p.cos + (size_t)pos * (hd >> 1)) + lane);
    sn = __ldg(reinterpret_cast<const float2*>(p.sin + (size_t)pos * (hd >> 1)) + lane);
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      wq[i] = reinterpret_cast<const uint32_t*>(p.qn)[i * h4 + lane];
      wk[i] = reinterpret_cast<const uint32_t*>(p.kn)[i * h4 + lane];
    }
  }
#pragma unroll
  for (int j = 0; j < kQkvHeads; ++j) {
    const int h = head0 + j;
    if (h >= (int)heads) break;
    uint32_t o_lo = lo[j], o_hi = hi[j];
    if (h < p.hq + p.hk) {
      const float x0 = bf16_bits_to_float(lo[j] & 0xffffu), x1 = bf16_bits_to_float(lo[j] >> 16);
      const float y0 = bf16_bits_to_float(hi[j] & 0xffffu), y1 = bf16_bits_to_float(hi[j] >> 16);
      const float r = rsqrtf(warp_sum(fmaf(x0, x0, fmaf(x1, x1, fmaf(y0, y0, y1 * y1)))) / (float)hd + p.eps);
      const uint32_t w0 = h < p.hq ? wq[0] : wk[0], w1 = h < p.hq ? wq[1] : wk[1];
      const float a0 = round_bf16((x0 * r) * bf16_bits_to_float(w0 & 0xffffu)), a1 = round_bf16((x1 * r) * bf16_bits_to_float(w0 >> 16));
      const float b0 = round_bf16((y0 * r) * bf16_bits_to_float(w1 & 0xffffu)), b1 = round_bf16((y1 * r) * bf16_bits_to_float(w1 >> 16));
      o_lo = (uint32_t)float_to_bf16_bits(__fsub_rn(__fmul_rn(a0, c.x), __fmul_rn(b0, sn.x))) |
             (uint32_t)float_to_bf16_bits(__fsub_rn(__fmul_rn(a1, c.y), __fmul_rn(b1, sn.y))) << 16;
      o_hi = (uint32_t)float_to_bf16_bits(__fadd_rn(__fmul_rn(b0, c.x), __fmul_rn(a0, sn.x))) |
             (uint32_t)float_to_bf16_bits(__fadd_rn(__fmul_rn(b1, c.y), __fmul_rn(a1, sn.y))) << 16;
    }
    __nv_bfloat16* row = h < p.hq ? p.qo + (((size_t)b * p.hq + h) * p.S + s) * hd
                         : h < p.hq + p.hk ? p.kc + (((size_t)b * p.hk + h - p.hq) * p.max_seq + pos) * hd
                                           : p.vc + (((size_t)b * p.hk + h - p.hq - p.hk) * p.max_seq + pos) * hd;
    if (act) {
      reinterpret_cast<uint32_t*>(row)[lane] = o_lo;
      reinterpret_cast<uint32_t*>(row)[h4 + lane] = o_hi;
    }
  }
}

// ------------------------------------------------------------------ one-token attention over the cache
// A CTA owns one (sequence, KV head) and a slice of the positions, for all REP query heads that share the KV head: the
// cache is read once.  Its eight warps take tiles of 16 positions and never wait for one another: scores by mma.sync (products of
// bfloat16, exact in fp32, fp32 sums; the heads are the eight columns), a running maximum and sum per warp, probabilities in
// float32 through the warp's own corner of shared memory, values by float32 multiply-adds (a lane owns HD / 32 dimensions of all
// heads).  A tile's values and the next tile's keys are on their way while a tile is worked out.
// The slices of a (sequence, KV head) are the CTAs of a cluster, which joins their results through distributed shared memory and
// writes the output; only where eight CTAs would be too few for the positions do several clusters share them, and a second
// kernel joins theirs.  Bound by latency at a few sequences: keys and values of four sequences at position 3000 (25 MB a layer)
// take 4 us from HBM.  us in a graph, 32 query and 4 KV heads of 128, the form with barriers between scores, probabilities and
// values and always a second kernel -> now: one sequence at 3000 18.4 -> 11.7, four at 512 8.7 -> 7.5, four at 3000 30.6 -> 17.3,
// eight at 4200 63.4 -> 23.6.
constexpr int kAttThreads = 256, kAttTile = 16, kAttWarps = kAttThreads / 32;

struct AttParams {
  const __nv_bfloat16 *q, *kc, *vc;  // (B, Hq, hd), caches (B, Hk, max_seq, hd)
  const long long* pos_dev;          // last valid position, or NULL: npos - 1
  int npos, hk, max_seq, nsplit;  // nsplit: clusters per (sequence, KV head)
  float scale;
  float* part;  // (B*Hk, nsplit, REP, hd + 2): accumulator, maximum, sum; unused with one cluster
  __nv_bfloat16* out;  // (B, Hq, hd)
};

__device__ __forceinline__ void att_mma(float (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0,
                                        uint32_t b1) {
  asm volatile(
      "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
      : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
      : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}

template <int HD, int REP, int C>
__global__ void __launch_bounds__(kAttThreads, 2) decode_attn_kernel(const AttParams p) {
  constexpr int KJ = HD / 32;  // 16-byte pieces of a key row per lane
  constexpr int VD = HD / 32;  // dimensions of a lane
  __shared__ __align__(16) float prob[kAttWarps][kAttTile][8];
  __shared__ __align__(16) float fac[kAttWarps][8];
  __shared__ float red[kAttWarps][REP][HD];
  __shared__ float warp_m[kAttWarps][8], warp_s[kAttWarps][8];
  __shared__ float mine[REP][HD + 2];  // the CTA's result: accumulator, maximum, sum (read by the cluster)
  pdl_wait();  // from here on plain loads: the non-coherent path must not run ahead of the wait
  pdl_trigger();
  const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5, g = lane >> 2, tig = lane & 3;
  const int pair = blockIdx.y, b = pair / p.hk, kh = pair - b * p.hk;
  const int P = p.pos_dev != nullptr ? min((int)*p.pos_dev + 1, p.max_seq) : p.npos;
  const int slices = p.nsplit * C, per = ((P + slices - 1) / slices + kAttTile - 1) / kAttTile * kAttTile;
  const int lo = min((int)blockIdx.x * per, P), hi = min(lo + per, P);
  const __nv_bfloat16* kc = p.kc + ((size_t)b * p.hk + kh) * p.max_seq * HD;
  const __nv_bfloat16* vc = p.vc + ((size_t)b * p.hk + kh) * p.max_seq * HD;
  // head g's values as column g of the second operand, in the order in which a lane's 16 bytes serve two mma steps
  uint4 q[KJ];
#pragma unroll
  for (int j = 0; j < KJ; ++j)
    q[j] = g < REP ? *(reinterpret_cast<const uint4*>(p.q + (((size_t)b * p.hk + kh) * REP + min(g, REP - 1)) * HD) + tig + 4 * j)
                   : make_uint4(0u, 0u, 0u, 0u);
  float m[2] = {-INFINITY, -INFINITY}, sum[2] = {0.0f, 0.0f};  // of heads 2 tig and 2 tig + 1; sums: this lane's share
  float acc[REP][VD];
#pragma unroll
  for (int r = 0; r < REP; ++r)
#pragma unroll
    for (int k = 0; k < VD; ++k) acc[r][k] = 0.0f;
  uint4 ka[KJ], kb[KJ];
  auto keys = [&](int p0) {
#pragma unroll
    for (int j = 0; j < KJ; ++j) {
      const int i0 = p0 + g, i1 = p0 + g + 8;
      ka[j] = i0 < hi ? *(reinterpret_cast<const uint4*>(kc + (size_t)i0 * HD) + tig + 4 * j) : make_uint4(0u, 0u, 0u, 0u);
      kb[j] = i1 < hi ? *(reinterpret_cast<const uint4*>(kc + (size_t)i1 * HD) + tig + 4 * j) : make_uint4(0u, 0u, 0u, 0u);
    }
  };
  int p0 = lo + wid * kAttTile;
  keys(p0);
#pragma unroll 1
  for (; p0 < hi; p0 += kAttWarps * kAttTile) {
    uint32_t v[kAttTile][VD / 2];
#pragma unroll
    for (int i = 0; i < kAttTile; ++i) {
      const __nv_bfloat16* at = vc + (size_t)(p0 + i) * HD + lane * VD;
      const bool in = p0 + i < hi;
      if constexpr (VD == 4) {
        const uint2 two = in ? *reinterpret_cast<const uint2*>(at) : make_uint2(0u, 0u);
        v[i][0] = two.x;
        v[i][1] = two.y;
      } else {
        v[i][0] = in ? *reinterpret_cast<const uint32_t*>(at) : 0u;
      }
    }
    float c[2][4];
#pragma unroll
    for (int h = 0; h < 2; ++h)
#pragma unroll
      for (int k = 0; k < 4; ++k) c[h][k] = 0.0f;
#pragma unroll
    for (int j = 0; j < KJ; ++j) {
      att_mma(c[0], ka[j].x, kb[j].x, ka[j].y, kb[j].y, q[j].x, q[j].y);
      att_mma(c[1], ka[j].z, kb[j].z, ka[j].w, kb[j].w, q[j].z, q[j].w);
    }
    // ---- scores of positions g and g + 8 for heads 2 tig and 2 tig + 1
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const float s0 = p0 + g < hi ? (c[0][h] + c[1][h]) * p.scale : -INFINITY;
      const float s1 = p0 + g + 8 < hi ? (c[0][h + 2] + c[1][h + 2]) * p.scale : -INFINITY;
      float top = fmaxf(s0, s1);
#pragma unroll
      for (int o = 4; o < 32; o <<= 1) top = fmaxf(top, __shfl_xor_sync(0xffffffffu, top, o));
      top = fmaxf(m[h], top);
      const float ref = top == -INFINITY ? 0.0f : top;  // every score so far is -inf: their weights are 0, not exp(-inf + inf)
      const float e0 = expf(s0 - ref), e1 = expf(s1 - ref), f = expf(m[h] - ref);
      m[h] = top;
      sum[h] = sum[h] * f + (e0 + e1);
      prob[wid][g][2 * tig + h] = e0;
      prob[wid][g + 8][2 * tig + h] = e1;
      if (g == 0) fac[wid][2 * tig + h] = f;
    }
    __syncwarp();
    float fr[8];
    *reinterpret_cast<float4*>(fr) = *reinterpret_cast<const float4*>(&fac[wid][0]);
    *reinterpret_cast<float4*>(fr + 4) = *reinterpret_cast<const float4*>(&fac[wid][4]);
#pragma unroll
    for (int r = 0; r < REP; ++r)
#pragma unroll
      for (int k = 0; k < VD; ++k) acc[r][k] *= fr[r];
#pragma unroll
    for (int i = 0; i < kAttTile; ++i) {
      // the next tile's keys, once half of the values' registers are free
      if (i == kAttTile / 2 && p0 + kAttWarps * kAttTile < hi) keys(p0 + kAttWarps * kAttTile);
      float w[8];
      *reinterpret_cast<float4*>(w) = *reinterpret_cast<const float4*>(&prob[wid][i][0]);
      if (REP > 4) *reinterpret_cast<float4*>(w + 4) = *reinterpret_cast<const float4*>(&prob[wid][i][4]);
      float x[VD];
#pragma unroll
      for (int k = 0; k < VD; ++k) x[k] = bf16_bits_to_float((k & 1) ? v[i][k >> 1] >> 16 : v[i][k >> 1] & 0xffffu);
#pragma unroll
      for (int r = 0; r < REP; ++r)
#pragma unroll
        for (int k = 0; k < VD; ++k) acc[r][k] = fmaf(w[r], x[k], acc[r][k]);
    }
    __syncwarp();  // the probabilities are used up
  }
  // ---- the warps' results under their common maximum
#pragma unroll
  for (int h = 0; h < 2; ++h) {
#pragma unroll
    for (int o = 4; o < 32; o <<= 1) sum[h] += __shfl_xor_sync(0xffffffffu, sum[h], o);
    if (g == 0) {
      warp_m[wid][2 * tig + h] = m[h];
      warp_s[wid][2 * tig + h] = sum[h];
    }
  }
#pragma unroll
  for (int r = 0; r < REP; ++r)
#pragma unroll
    for (int k = 0; k < VD; ++k) red[wid][r][lane * VD + k] = acc[r][k];
  __syncthreads();
  for (int i = tid; i < REP * HD; i += kAttThreads) {
    const int r = i / HD, d = i - r * HD;
    float top = -INFINITY;
#pragma unroll
    for (int w = 0; w < kAttWarps; ++w) top = fmaxf(top, warp_m[w][r]);
    float num = 0.0f, den = 0.0f;
#pragma unroll
    for (int w = 0; w < kAttWarps; ++w) {
      const float f = warp_m[w][r] == -INFINITY ? 0.0f : expf(warp_m[w][r] - top);  // a warp without a position
      num = fmaf(f, red[w][r][d], num);
      den = fmaf(f, warp_s[w][r], den);
    }
    mine[r][d] = num;
    if (d == 0) {
      mine[r][HD] = top;
      mine[r][HD + 1] = den;
    }
  }
  // ---- the cluster's slices under their common maximum: CTA c takes every C-th run of kAttThreads values
  if (C > 1) {
    asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
    asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
  } else {
    __syncthreads();
  }
  auto peer = [&](const float* at, int c) -> float {
    if (C == 1) return *at;
    uint32_t addr;
    float v;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(addr) : "r"((uint32_t)__cvta_generic_to_shared(at)), "r"(c));
    asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(v) : "r"(addr) : "memory");
    return v;
  };
  const int rank = (int)blockIdx.x % C;
  for (int i = rank * kAttThreads + tid; i < REP * HD; i += C * kAttThreads) {
    const int r = i / HD, d = i - r * HD;
    float ms[C], top = -INFINITY;
#pragma unroll
    for (int k = 0; k < C; ++k) {
      ms[k] = peer(&mine[r][HD], k);
      top = fmaxf(top, ms[k]);
    }
    float num = 0.0f, den = 0.0f;
#pragma unroll
    for (int k = 0; k < C; ++k) {
      const float f = ms[k] == -INFINITY ? 0.0f : expf(ms[k] - top);  // an empty slice
      num = fmaf(f, peer(&mine[r][d], k), num);
      den = fmaf(f, peer(&mine[r][HD + 1], k), den);
    }
    if (p.nsplit == 1) {
      p.out[((size_t)pair * REP + r) * HD + d] = __float2bfloat16_rn(num / den);
    } else {
      float* part = p.part + (((size_t)pair * p.nsplit + blockIdx.x / C) * REP + r) * (HD + 2);
      part[d] = num;
      if (d == 0) {
        part[HD] = top;
        part[HD + 1] = den;
      }
    }
  }
  if (C > 1) {  // nobody reads this CTA's results any more
    asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
    asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
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

// CTAs of a cluster: as many as give every (sequence, KV head) a cluster at two CTAs per SM.
static int attn_cluster(int B, int hk) {
  const int pairs = B * hk;
  return pairs <= 32 ? 8 : pairs <= 64 ? 4 : pairs <= 128 ? 2 : 1;
}
// Clusters per (sequence, KV head): one up to 1024 positions a CTA, since a second launch costs more than it gains (four
// sequences at 4200: three clusters 28 us, one 22); above, about two CTAs per SM in all.
static int attn_splits(int B, int hk, int max_pos) {
  const int c = attn_cluster(B, hk), tile = kAttWarps * kAttTile;
  if (max_pos <= 1024 * c) return 1;
  const int want = (2 * 148 + B * hk * c - 1) / (B * hk * c);
  const int most = (max_pos + tile * c - 1) / (tile * c);
  return want < most ? want : most;
}

template <int HD, int REP>
static cudaError_t launch_attn_rep(const AttParams& p, int pairs, int cluster, cudaStream_t st) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(p.nsplit * cluster, pairs);
  cfg.blockDim = dim3(kAttThreads);
  cfg.stream = st;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  attr[1].id = cudaLaunchAttributeClusterDimension;
  attr[1].val.clusterDim.x = cluster;
  attr[1].val.clusterDim.y = attr[1].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = cluster > 1 ? 2 : 1;
  switch (cluster) {
    case 8: return cudaLaunchKernelEx(&cfg, decode_attn_kernel<HD, REP, 8>, p);
    case 4: return cudaLaunchKernelEx(&cfg, decode_attn_kernel<HD, REP, 4>, p);
    case 2: return cudaLaunchKernelEx(&cfg, decode_attn_kernel<HD, REP, 2>, p);
    default: return cudaLaunchKernelEx(&cfg, decode_attn_kernel<HD, REP, 1>, p);
  }
}

template <int HD>
static int launch_attn(const AttParams& p, int rep, int pairs, int cluster, cudaStream_t st) {
  cudaError_t e;
  switch (rep) {
    case 1: e = launch_attn_rep<HD, 1>(p, pairs, cluster, st); break;
    case 2: e = launch_attn_rep<HD, 2>(p, pairs, cluster, st); break;
    case 4: e = launch_attn_rep<HD, 4>(p, pairs, cluster, st); break;
    default: e = launch_attn_rep<HD, 8>(p, pairs, cluster, st); break;
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
  const uintptr_t rows = (uintptr_t)q | (uintptr_t)k | (uintptr_t)v | (uintptr_t)q_norm | (uintptr_t)k_norm | (uintptr_t)q_out |
                         (uintptr_t)k_cache | (uintptr_t)v_cache;
  if (units > 64 * 150 && units < (1ll << 31) && hd % 4 == 0 && hd <= 128 && (rows & 3) == 0 &&
      (((uintptr_t)cos_t | (uintptr_t)sin_t) & 7) == 0) {
    const long long warps = (long long)B * S * ((hq + 2 * hk + kQkvHeads - 1) / kQkvHeads);
    launch_pdl(qkv_post4_kernel, dim3((unsigned)((warps + 7) / 8)), dim3(256), 0, (cudaStream_t)stream, p);
    return check_launch("zmoe_qkv_post");
  }
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
  const int cluster = attn_cluster(B, hk);
  const int rc = hd == 128 ? launch_attn<128>(p, rep, B * hk, cluster, st) : launch_attn<64>(p, rep, B * hk, cluster, st);
  if (rc != ZMOE_OK || p.nsplit == 1) return rc;
  launch_pdl(decode_attn_join_kernel, dim3(B * hq), dim3(hd), 0, st, (const float*)workspace, p.nsplit, rep, hd,
             (__nv_bfloat16*)out);
  return check_launch("decode_attn_join_kernel");
}

}  // extern "C"
