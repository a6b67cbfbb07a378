// Token-grouped 4-bit expert matmul on the 5th-generation tensor cores, fed through tensor memory: the path of every
// call that brings a workspace and more than a few token rows (serving batches and prompts, affine and mxfp4 banks).
//
// What bounds it: at a few rows per expert the packed weights' way from HBM, at many rows the token tiles' way from
// L2 (one SM reads 128 weight rows x 256 codes = 18 KB against 576 B per token row for them).  So the packed codes
// must be expanded at the rate at which they arrive, and the token side must cost nothing but the copy:
//
//   prep_rows_kernel  writes, once per call, every token row in expert-sorted order as fp16 under a per-row power of
//              two, and beside it the row's group sums as three fp16 pieces.  A token tile is then a plain TMA box
//              with the 128-byte swizzle the tensor core reads, whatever the gather was.
//   qmm_tma_kernel    one persistent CTA per SM walks items (expert, 128 weight rows, a block of token rows) as one
//              unbroken stream of chunks of 256 codes:
//     weights   one thread keeps kTmRaw boxes of 128 rows x 128 packed bytes in flight;
//     tokens    one thread keeps the ring of token tiles full;
//     expanders two sets of 128 threads (one per weight row) turn every other chunk's codes into the fp16 A operand
//               and store it straight into the set's stage in TENSOR MEMORY (tcgen05.st): no shared-memory round trip,
//               no swizzle arithmetic; one set's waits and latencies lie under the other set's arithmetic;
//     issuer    one thread issues tcgen05.mma (M 128 x N 16..96 x K 16, A in tensor memory, B in shared memory);
//     finishers 256 threads fold the chunk's accumulator into fp32 registers and, at the end of an item, apply the
//               SwiGLU contract and store bf16 rows through the plan.
//
// Arithmetic.  Affine: w = q s + b = (q - 8) s + (b + 8 s).  q - 8 has three bits and a sign, s eight: their product fits
// fp16's eleven, so the scale goes into the operand and the accumulator runs over several groups.  The second term is two
// more K = 16 steps on one operand, per group (b, b, -8 s, -8 s), against the group's float32 sum X as three fp16 pieces (33
// bits): (X1, X2, -X1, -X2) and (X3, 0, -X3, 0).  The scales are first multiplied by a power of two per (row, chunk), undone
// in fp32 by the finishers, so the range of fp16 is no limit on the checkpoint's.
// (q - 8) s is exact while the four scales of a row's chunk lie within 12 binades of the largest; chunks with scales
// further apart are expanded another way (tm_expand_far), exact over 28; below, a weight is off by at most 2^-39 of the
// largest of its row's chunk.  mxfp4: e2m1 value x 2^(e - emax + 13), exact in fp16 over 36 binades, same row factor.
// Token rows carry a power of two per row: a bfloat16 of the row is exact down to 2^-26 (mxfp4: 2^-31) of its largest,
// and off by at most 2^-34 (2^-39) of it below.  Chunks are
// summed in fp32 registers rather than in the accumulator over all of K, so that no sum is longer than 160 products (mxfp4:
// 256).
//
// gate and up share one accumulator: lanes 0-15 of each warp's 32 tensor-memory lanes hold gate rows, lanes 16-31 the
// up rows of the same outputs, and the epilogue pairs them with one shuffle.
//
// Every wait is bounded by a second; one that runs out sets the plan's status word (zmoe_plan_status), everybody else
// leaves at the next wait, copies and MMAs in flight are waited for, the tensor memory is given back and the CTA's results
// become NaN.
#include <cuda.h>
#include <cuda_fp16.h>

#include "qmm_common.cuh"

namespace zmoe {

constexpr int kTmExp = 256, kTmFin = 256;
constexpr int kTmThreads = kTmExp + kTmFin + 96;  // + one warp each: issuer, weight copies, token copies
constexpr int kTmRows = 128;                      // tensor-memory lanes = weight rows of an item
constexpr int kTmChunk = 256;                     // codes per chunk
constexpr int kTmRaw = 5;                         // chunks of packed bytes in flight
constexpr int kTmRawBytes = kTmRows * kTmChunk / 2;
constexpr int kTmScRing = 4, kTmScAhead = 3;      // scales: a thread's chunks in the ring, copy distance
constexpr int kTmMaxTok = 96;                     // token rows per item, at most
constexpr int kTmMaxX = 8;                        // token stages, at most
constexpr int kTmMaxTasks = 1024;
constexpr int kTmItems = 256;                     // work items of a CTA kept in shared memory
constexpr int kTmCols = 512;
constexpr int kTmColD = 128;                      // columns between the two accumulators
constexpr int kTmSplitTok = 48;                   // up to so many token rows an accumulator is two, one per half chunk
// How a chunk is summed.  The tensor core cuts products and sums off at a fixed distance below the largest of them, so
// long sums lose.  Share of bfloat16 results that are not the float64 result's rounding, affine, K = 768 and 2048: whole
// chunks 1.7e-4, halves 1.1e-4 and 1.2e-4 (float32 sums over groups of 64 unscaled codes: 0.6e-4 and 1.0e-4).  Up to
// kTmSplitTok token rows the two halves lie side by side and are handed over together; wider items hand them over one
// after the other, which costs 6 % (c2 with 4096 rows: 828 -> 879 us a block; quarters: 1090).  Products of e2m1 codes and
// powers of two hardly lose any bits: whole chunks, 0.1e-4 to 0.6e-4.
enum TmSum { kTmWhole, kTmSplit, kTmTurns };
constexpr int kTmColA = 224, kTmAStage = 136;     // two A stages: 128 columns of codes, 8 of scales and biases

struct TmArgs {
  CUtensorMap w[2];  // packed bytes (E*N, K/2): box 128 bytes x 128 (gate and up: 64) rows
  CUtensorMap x;     // prepared rows (rows, K) fp16: box 64 x 16
  CUtensorMap xb;    // their group sums (rows, K/8) fp16: box 32 x 16
  QmmParams q;
  const float* xinv;  // (rows): 1 / the row's power of two
  int nch;            // K / 256
  int tn;             // token rows per item, at most (a multiple of 16)
  int rx;             // token stages
  int xstage;         // bytes of one
};

__device__ __forceinline__ uint32_t tm_smem(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }
__device__ __forceinline__ void tm_bar_init(uint32_t bar, int count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(count));
}
__device__ __forceinline__ void tm_arrive(uint32_t bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory");
}
__device__ __forceinline__ void tm_expect(uint32_t bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
}
// One look at a phase; the hardware may suspend the thread in it for up to `ns`, and wakes it when the phase completes.
__device__ __forceinline__ bool tm_try(uint32_t bar, uint32_t parity, uint32_t ns) {
  uint32_t ok;
  asm volatile("{ .reg .pred p; mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2, %3; selp.u32 %0, 1, 0, p; }"
               : "=r"(ok)
               : "r"(bar), "r"(parity), "r"(ns)
               : "memory");
  return ok != 0;
}
__device__ __forceinline__ unsigned long long tm_now() {
  unsigned long long t;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
  return t;
}
// Waits for the phase; false when a second passed or, unless `drain`, another thread of the CTA gave up.  Suspended
// looks rather than a spin: polling warps would take the issue slots that the expanders live on.  The patient part is
// out of line: the roles' loops share one instruction cache.
__device__ __noinline__ bool tm_wait_long(uint32_t bar, uint32_t parity, volatile int* abort_flag, bool drain) {
  const unsigned long long t0 = tm_now();
  while (true) {
    if (tm_try(bar, parity, 20000u)) return true;
    if (!drain && *abort_flag) return false;
    if (tm_now() - t0 > 1000000000ull) {
      *abort_flag = 1;
      return false;
    }
  }
}
__device__ __forceinline__ bool tm_wait(uint32_t bar, uint32_t parity, volatile int* abort_flag, bool drain = false) {
#pragma unroll 1
  for (int i = 0; i < 8; ++i)
    if (tm_try(bar, parity, 20000u)) return true;
  return tm_wait_long(bar, parity, abort_flag, drain);
}
// The same for a whole warp: all lanes leave together, as the tcgen05.ld and .st that follow need them to.
__device__ __forceinline__ bool tm_wait_warp(uint32_t bar, uint32_t parity, volatile int* abort_flag) {
  return __all_sync(0xffffffffu, tm_wait(bar, parity, abort_flag));
}
__device__ __forceinline__ void tm_load_2d(uint32_t dst, const CUtensorMap* map, int x, int y, uint32_t bar) {
  asm volatile(
      "cp.async.bulk.tensor.2d.shared::cta.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];" ::"r"(
          dst),
      "l"(map), "r"(x), "r"(y), "r"(bar)
      : "memory");
}
// Shared-memory descriptors of K-major tiles: rows of 128 (64) bytes under the 128-byte (64-byte) swizzle, eight rows
// per atom.
__device__ __forceinline__ uint64_t tm_desc128(uint32_t addr) {
  return (uint64_t)((addr & 0x3FFFFu) >> 4) | (1ull << 16) | ((uint64_t)(1024 >> 4) << 32) | (1ull << 46) | (2ull << 61);
}
__device__ __forceinline__ uint64_t tm_desc64(uint32_t addr) {
  return (uint64_t)((addr & 0x3FFFFu) >> 4) | (1ull << 16) | ((uint64_t)(512 >> 4) << 32) | (1ull << 46) | (4ull << 61);
}
// D fp32, A and B fp16, both K-major, M = 128, N = n.
__device__ __forceinline__ uint32_t tm_idesc(int n) {
  return (1u << 4) | ((uint32_t)(n >> 3) << 17) | ((uint32_t)(kTmRows >> 4) << 24);
}
__device__ __forceinline__ void tm_mma(uint32_t d, uint32_t a, uint64_t bdesc, uint32_t idesc, bool accumulate) {
  asm volatile("{ .reg .pred p; setp.ne.b32 p, %4, 0; tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p; }" ::"r"(d),
               "r"(a), "l"(bdesc), "r"(idesc), "r"((uint32_t)accumulate)
               : "memory");
}
__device__ __forceinline__ void tm_commit(uint32_t bar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar) : "memory");
}
__device__ __forceinline__ void tm_ld16(uint32_t taddr, float (&r)[16]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
      : "=f"(r[0]), "=f"(r[1]), "=f"(r[2]), "=f"(r[3]), "=f"(r[4]), "=f"(r[5]), "=f"(r[6]), "=f"(r[7]), "=f"(r[8]),
        "=f"(r[9]), "=f"(r[10]), "=f"(r[11]), "=f"(r[12]), "=f"(r[13]), "=f"(r[14]), "=f"(r[15])
      : "r"(taddr)
      : "memory");
}
__device__ __forceinline__ void tm_st16(uint32_t taddr, const uint32_t (&r)[16]) {
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16};" ::"r"(
          taddr),
      "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]), "r"(r[9]),
      "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15])
      : "memory");
}
__device__ __forceinline__ void tm_st2(uint32_t taddr, uint32_t r0, uint32_t r1) {
  asm volatile("tcgen05.st.sync.aligned.32x32b.x2.b32 [%0], {%1,%2};" ::"r"(taddr), "r"(r0), "r"(r1) : "memory");
}
// One lane of a converged warp.  The compiler knows an elected thread to be alone; behind `lane == 0` it would wrap
// every tcgen05.mma and TMA instruction in a loop over the lanes that might be active (measured: 190 cycles per MMA
// whatever its shape, 17 of them per chunk).
__device__ __forceinline__ bool tm_elect() {
  uint32_t one;
  asm volatile("{ .reg .pred p; elect.sync _|p, 0xffffffff; selp.u32 %0, 1, 0, p; }" : "=r"(one));
  return one != 0;
}
__device__ __forceinline__ uint32_t tm_bits(__half2 h) { return *reinterpret_cast<const uint32_t*>(&h); }
__device__ __forceinline__ __half2 tm_half2(uint32_t u) { return *reinterpret_cast<const __half2*>(&u); }

// Eight codes of a packed word times the group's scale, as four half2 in the order (0,4) (1,5) (2,6) (3,7) that the
// token rows are written in.  A nibble at bits 4-7 of a half IS the fp16 number q 2^-20 (subnormal or not), so one
// fused multiply-add gives q 2^-20 (s 2^20) - 8 s = (q - 8) s, exact: three shifts, four masks, four half2 operations
// per eight codes.
__device__ __forceinline__ void tm_expand_affine(uint32_t w, __half2 s20, __half2 m8s, uint32_t* out) {
  const uint32_t m = 0x00F000F0u;
  out[0] = tm_bits(__hfma2(tm_half2((w << 4) & m), s20, m8s));
  out[1] = tm_bits(__hfma2(tm_half2(w & m), s20, m8s));
  out[2] = tm_bits(__hfma2(tm_half2((w >> 4) & m), s20, m8s));
  out[3] = tm_bits(__hfma2(tm_half2((w >> 8) & m), s20, m8s));
}
// A chunk whose scales lie further apart than tm_expand_affine takes: a nibble at bits 6-9 of a half under the exponent of
// 16 is 16 + q, and (16 + q) s - 24 s = (q - 8) s is exact for s from 2^-17 to 2^11 (24 s has ten bits).  One more shift and
// four more masks per word: every chunk done this way cost 9 to 13 % (c2 with 32 rows 600 -> 657 us, c5 with 64 rows 1790
// -> 2038), so it is a call for the warps that meet such a chunk.
__device__ __noinline__ void tm_expand_far(const unsigned char* src, uint32_t swz, uint4 sc, float P, uint32_t taddr) {
  const uint32_t m = 0x03C003C0u, sixteen = 0x4C004C00u;
#pragma unroll 1
  for (int i = 0; i < 8; ++i) {  // 16 bytes: half a group
    const uint4 w4 = *reinterpret_cast<const uint4*>(src + ((i ^ swz) << 4));
    const uint32_t ws[4] = {w4.x, w4.y, w4.z, w4.w};
    const float s = __uint_as_float(sc.x << 16) * P;
    const __half2 s_op = __float2half2_rn(s), off = __float2half2_rn(-24.0f * s);
    uint32_t o[16];
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      o[4 * k] = tm_bits(__hfma2(tm_half2(((ws[k] << 6) & m) | sixteen), s_op, off));
      o[4 * k + 1] = tm_bits(__hfma2(tm_half2(((ws[k] << 2) & m) | sixteen), s_op, off));
      o[4 * k + 2] = tm_bits(__hfma2(tm_half2(((ws[k] >> 2) & m) | sixteen), s_op, off));
      o[4 * k + 3] = tm_bits(__hfma2(tm_half2(((ws[k] >> 6) & m) | sixteen), s_op, off));
    }
    tm_st16(taddr + i * 16, o);
    if (i & 1) {
      const __half2 b_op = __float2half2_rn(__uint_as_float(sc.z << 16) * P);
      tm_st2(taddr + 127 + i, tm_bits(b_op), tm_bits(__float2half2_rn(-8.0f * s)));
      sc.x = __funnelshift_r(sc.x, sc.y, 16);
      sc.y >>= 16;
      sc.z = __funnelshift_r(sc.z, sc.w, 16);
      sc.w >>= 16;
    }
  }
}
// Eight e2m1 codes in their own order, times the block's power of two.
__device__ __forceinline__ void tm_expand_mx(uint32_t w, __half2 s, uint32_t* out) {
  uint32_t a, b, c, d;
  asm("{ .reg .b8 t0, t1, t2, t3;\n"
      "mov.b32 {t0, t1, t2, t3}, %4;\n"
      "cvt.rn.f16x2.e2m1x2 %0, t0;\n"
      "cvt.rn.f16x2.e2m1x2 %1, t1;\n"
      "cvt.rn.f16x2.e2m1x2 %2, t2;\n"
      "cvt.rn.f16x2.e2m1x2 %3, t3; }"
      : "=r"(a), "=r"(b), "=r"(c), "=r"(d)
      : "r"(w));
  out[0] = tm_bits(__hmul2(tm_half2(a), s));
  out[1] = tm_bits(__hmul2(tm_half2(b), s));
  out[2] = tm_bits(__hmul2(tm_half2(c), s));
  out[3] = tm_bits(__hmul2(tm_half2(d), s));
}

// One item of the work list: token rows [p0, p0 + nt) of the sorted order against rows n0.. of expert e.
struct TmItem {
  int e, p0, nt, n0;
};
// Items are numbered task-major; inside a task the token blocks of one row tile are neighbours, so that they run at
// the same time on different SMs and share the weights through L2.  prefix[a] = token blocks of the tasks before a.
__device__ __noinline__ TmItem tm_item(const PlanView& pv, const int* prefix, int ntasks, int ntiles, int tile_rows,
                                          int w) {
  int lo = 0, hi = ntasks - 1;
  while (lo < hi) {
    const int mid = (lo + hi + 1) >> 1;
    if (ntiles * prefix[mid] <= w) lo = mid; else hi = mid - 1;
  }
  const int local = w - ntiles * prefix[lo];
  const int nblk = prefix[lo + 1] - prefix[lo];
  const int tile = local / nblk, blk = local - tile * nblk;
  const int4 task = reinterpret_cast<const int4*>(pv.tasks)[lo];  // {expert, offset, count, -}
  const int per = ((task.z + nblk - 1) / nblk + 15) & ~15;                // equal blocks, whole 16s
  TmItem it;
  it.e = task.x;
  it.p0 = task.y + blk * per;
  it.nt = min(per, task.z - blk * per);
  it.n0 = tile * tile_rows;
  return it;
}

// EPI: the SwiGLU contract of gate and up (QmmParams::epilogue).
template <bool MX, int NMAT, int EPI, TmSum SUM>
__global__ void __launch_bounds__(kTmThreads, 1) qmm_tma_kernel(const __grid_constant__ TmArgs a) {
  extern __shared__ __align__(1024) unsigned char tm_dyn[];
  __shared__ uint32_t tmem_base_s;
  // raw full / empty, token full / empty, A full, MMAs done, accumulator free, accumulator full (kTmTurns)
  __shared__ __align__(8) unsigned long long bars_s[2 * kTmRaw + 2 * kTmMaxX + 8];
  __shared__ float inv_s[4][kTmRows];
  __shared__ volatile int abort_s;
  __shared__ int prefix_s[kTmMaxTasks + 1];
  __shared__ int4 items_s[kTmItems];

  constexpr int kTile = kTmRows / NMAT;  // output rows of an item
  const QmmParams& p = a.q;
  const int tid = threadIdx.x, wid = tid >> 5, lane = tid & 31;
  const int N = p.N, nch = a.nch, tn = a.tn, rx = a.rx;
  const PlanView pv = plan_view(const_cast<int*>(p.plan), p.rows, p.E);
  unsigned char* base = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(tm_dyn) + 1023) & ~(uintptr_t)1023);
  unsigned char* raw = base;
  unsigned char* tok = raw + kTmRaw * kTmRawBytes;
  unsigned char* scr = tok + rx * a.xstage;  // [slot][expander thread][16 bytes]
  const uint32_t bars = tm_smem(bars_s);
  const uint32_t b_rawf = bars, b_rawe = bars + 8 * kTmRaw, b_tokf = bars + 16 * kTmRaw;
  const uint32_t b_toke = b_tokf + 8 * kTmMaxX, b_af = b_toke + 8 * kTmMaxX, b_done = b_af + 16, b_dfree = b_done + 16;
  const uint32_t b_acc = b_dfree + 16;

  // The plan, the prepared rows and their factors may be the work of the kernel before, still running when this one
  // starts: they are read with plain loads after the wait, never through the read-only path.
  pdl_wait();
  pdl_trigger();
  const int ntasks = min(pv.hdr[0], kTmMaxTasks);
  if (wid == 0) {  // token blocks per task, prefix-summed (lane = a contiguous run of tasks)
    const int per = (ntasks + 31) >> 5;
    int sum = 0;
    for (int i = lane * per; i < min(ntasks, (lane + 1) * per); ++i) sum += (pv.tasks[4 * i + 2] + tn - 1) / tn;
    int incl = sum;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int v = __shfl_up_sync(0xffffffffu, incl, o);
      if (lane >= o) incl += v;
    }
    int run = incl - sum;
    for (int i = lane * per; i < min(ntasks, (lane + 1) * per); ++i) {
      prefix_s[i] = run;
      run += (pv.tasks[4 * i + 2] + tn - 1) / tn;
    }
    if (lane == 31) prefix_s[ntasks] = incl;
  }
  __syncthreads();
  const int ntiles = (N + kTile - 1) / kTile;
  const int total = ntiles * prefix_s[ntasks];
  if ((int)blockIdx.x >= total) return;  // before any tensor memory is taken
  const int n_items = (total - (int)blockIdx.x + (int)gridDim.x - 1) / (int)gridDim.x;
  const int n_chunks = n_items * nch;
  // Every role walks the CTA's items: they are looked up once, by all threads (a search, two divisions and a load of
  // the task record took each role some 1500 cycles per item); a CTA with more of them looks the rest up as it goes.
  for (int i = tid; i < min(n_items, kTmItems); i += kTmThreads) {
    const TmItem it = tm_item(pv, prefix_s, ntasks, ntiles, kTile, (int)blockIdx.x + i * (int)gridDim.x);
    items_s[i] = make_int4(it.e, it.p0, it.nt, it.n0);
  }
  auto item_at = [&](int i) -> TmItem {
    if (i >= kTmItems) return tm_item(pv, prefix_s, ntasks, ntiles, kTile, (int)blockIdx.x + i * (int)gridDim.x);
    const int4 v = items_s[i];
    return TmItem{v.x, v.y, v.z, v.w};
  };

  if (tid == 0) {
    for (int i = 0; i < kTmRaw; ++i) {
      tm_bar_init(b_rawf + 8 * i, 1);
      tm_bar_init(b_rawe + 8 * i, kTmExp / 64);
    }
    for (int i = 0; i < kTmMaxX; ++i) {
      tm_bar_init(b_tokf + 8 * i, 1);
      tm_bar_init(b_toke + 8 * i, 1);
    }
    for (int i = 0; i < 2; ++i) {
      tm_bar_init(b_af + 8 * i, kTmExp / 64);
      tm_bar_init(b_done + 8 * i, 1);
      tm_bar_init(b_dfree + 8 * i, kTmFin / 32);
      tm_bar_init(b_acc + 8 * i, 1);
    }
    abort_s = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  }
  if (wid == 0) {
    __syncwarp();
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(tm_smem(&tmem_base_s)),
                 "r"(kTmCols)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t tmem = tmem_base_s;
  constexpr int kParts = SUM == kTmTurns ? 2 : 1;  // hand-overs per chunk
  volatile int* ab = &abort_s;
  bool ok = true;

  if (wid < kTmExp / 32) {
    // ================================================================== expanders: a weight row of every other chunk
    const int q4 = wid & 3, set = wid >> 2;
    const int r = q4 * 32 + lane;  // tensor-memory lane
    const int mat = NMAT == 2 ? (lane >> 4) : 0;
    const int rb = NMAT == 2 ? q4 * 16 + (lane & 15) : r;  // row inside the matrix's box
    const uint32_t at = tmem + ((uint32_t)(q4 * 32) << 16) + kTmColA + set * kTmAStage;
    const unsigned char* my_raw = raw + mat * (kTile * 128) + rb * 128;
    unsigned char* my_sc = scr + tid * 16;
    // the cursor of the scale copies runs kTmScAhead of the thread's chunks ahead
    int f_item = 0, f_c = set, f_slot = 0;
    bool f_new = true;
    const unsigned char *f_s = nullptr, *f_b = nullptr;
    auto fetch = [&] {
      while (f_c >= nch) {
        f_c -= nch;
        ++f_item;
        f_new = true;
      }
      if (f_item < n_items) {
        if (f_new) {
          f_new = false;
          const TmItem it = item_at(f_item);
          const size_t row = (size_t)it.e * N + min(it.n0 + rb, N - 1);  // clamped rows are computed, not stored
          // 8 bytes per chunk: four bfloat16 scales (biases) or eight e8m0 bytes
          f_s = reinterpret_cast<const unsigned char*>(p.s[mat]) + row * nch * 8;
          if (!MX) f_b = reinterpret_cast<const unsigned char*>(p.b[mat]) + row * nch * 8;
        }
        unsigned char* dst = my_sc + f_slot * (kTmExp * 16);
        cp_async_8(dst, f_s + f_c * 8);
        if (!MX) cp_async_8(dst + 8, f_b + f_c * 8);
      }
      asm volatile("cp.async.commit_group;" ::: "memory");
      f_c += 2;
      f_slot = (f_slot + 1) % kTmScRing;
    };
#pragma unroll 1
    for (int i = 0; i < kTmScAhead; ++i) fetch();
    int rs = set, rph = 0, slot = 0;  // raw slot and its phase, scale slot
#pragma unroll 1
    for (int c = set; c < n_chunks; c += 2) {
      fetch();
      asm volatile("cp.async.wait_group %0;" ::"n"(kTmScAhead) : "memory");
      const uint4 sc = *reinterpret_cast<const uint4*>(my_sc + slot * (kTmExp * 16));
      slot = (slot + 1) % kTmScRing;
      // ---- the chunk's power of two
      uint32_t s_lo = sc.x, s_hi = sc.y, b_lo = sc.z, b_hi = sc.w;  // shifted through, one group at a time
      float inv, P = 0.0f;
      int emax = 0;
      bool far = false;
      if (MX) {
        uint32_t v = __vmaxu4(sc.x, sc.y);
        v = __vmaxu4(v, v >> 16);
        emax = (int)max(v & 0xffu, (v >> 8) & 0xffu);
        inv = emax >= 255 ? __uint_as_float(0x7f800000u) : exp2f((float)(emax - 127 - 13));
      } else {
        // largest |s| and |b| (bits order like magnitudes), as bfloat16 bits
        uint32_t ms = __vmaxu2(sc.x & 0x7fff7fffu, sc.y & 0x7fff7fffu);
        uint32_t mb = __vmaxu2(sc.z & 0x7fff7fffu, sc.w & 0x7fff7fffu);
        ms = max(ms & 0xffffu, ms >> 16);
        mb = max(mb & 0xffffu, mb >> 16);
        // 2^(140 - e) brings |s| below 2^-4 (so that s 2^20 stays below 2^16) and |b| below 2^14; a scale that this
        // leaves below 2^-17 asks for the wider form, where |s| may reach 2^11
        const int es = (int)(ms >> 7), eb = (int)(mb >> 7);
        int e = max(es + 18, eb);
        const uint32_t least = __vminu2(sc.x & 0x7fff7fffu, sc.y & 0x7fff7fffu);
        far = __any_sync(0xffffffffu, (int)(min(least & 0xffffu, least >> 16) >> 7) + 30 < e);
        if (far) e = max(es + 3, eb);
        e = min(max(e, far ? 14 : 34), 253);
        P = __uint_as_float((uint32_t)(267 - e) << 23);
        inv = __uint_as_float((uint32_t)(e - 13) << 23);
      }
      // ---- the stage is free once the MMAs of the thread's previous chunk are done
      ok = tm_wait_warp(b_rawf + 8 * rs, rph, ab);
      if (ok && c >= 2) ok = tm_wait_warp(b_done + 8 * set, ((c >> 1) - 1) & 1, ab);
      if (!ok) break;
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      const unsigned char* src = my_raw + rs * kTmRawBytes;
      uint4 wa = *reinterpret_cast<const uint4*>(src + ((rb & 7) << 4));
      uint4 wb = *reinterpret_cast<const uint4*>(src + ((1 ^ (rb & 7)) << 4));
      if (!MX && far) tm_expand_far(src, rb & 7, sc, P, at);
#pragma unroll 1
      for (int i = !MX && far ? 4 : 0; i < 4; ++i) {  // 64 codes each: a group, or two mxfp4 blocks.  Rolled: see tm_wait_long
        const int nx = 2 * min(i + 1, 3);
        const uint4 na = *reinterpret_cast<const uint4*>(src + ((nx ^ (rb & 7)) << 4));
        const uint4 nb = *reinterpret_cast<const uint4*>(src + (((nx + 1) ^ (rb & 7)) << 4));
        const uint32_t ws[8] = {wa.x, wa.y, wa.z, wa.w, wb.x, wb.y, wb.z, wb.w};
        uint32_t o[2][16];
        if (MX) {
          // fp16 2^(e - emax + 13) in both halves, subnormal ones included
          const __half2 s0 = __float2half2_rn(__uint_as_float((uint32_t)max((int)(s_lo & 0xffu) - emax + 140, 0) << 23));
          const __half2 s1 = __float2half2_rn(__uint_as_float((uint32_t)max((int)((s_lo >> 8) & 0xffu) - emax + 140, 0) << 23));
#pragma unroll
          for (int k = 0; k < 8; ++k) tm_expand_mx(ws[k], k < 4 ? s0 : s1, o[k >> 2] + 4 * (k & 3));
        } else {
          const float s = __uint_as_float(s_lo << 16);
          const __half2 s_op = __float2half2_rn(s * (P * 1048576.0f)), s_off = __float2half2_rn(s * (-8.0f * P));
#pragma unroll
          for (int k = 0; k < 8; ++k) tm_expand_affine(ws[k], s_op, s_off, o[k >> 2] + 4 * (k & 3));
          const __half2 b_op = __float2half2_rn(__uint_as_float(b_lo << 16) * P);
          tm_st2(at + 128 + 2 * i, tm_bits(b_op), tm_bits(s_off));
          b_lo = __funnelshift_r(b_lo, b_hi, 16);
          b_hi >>= 16;
        }
        tm_st16(at + i * 32, o[0]);
        tm_st16(at + i * 32 + 16, o[1]);
        s_lo = __funnelshift_r(s_lo, s_hi, 16);
        s_hi >>= 16;
        wa = na;
        wb = nb;
      }
      inv_s[c & 3][r] = inv;
      asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
      asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
      __syncwarp();
      if (lane == 0) {
        tm_arrive(b_af + 8 * set);
        tm_arrive(b_rawe + 8 * rs);
      }
      __syncwarp();
      rs += 2;
      if (rs >= kTmRaw) {
        rs -= kTmRaw;
        rph ^= 1;
      }
    }
    asm volatile("cp.async.wait_all;" ::: "memory");
  } else if (wid < (kTmExp + kTmFin) / 32) {
    // ================================================================== finishers: weight row x every other 16 tokens
    const int q4 = wid & 3, ch = (wid - kTmExp / 32) >> 2;
    const int r = q4 * 32 + lane;
    const uint32_t lane_base = tmem + ((uint32_t)(q4 * 32) << 16);
    float acc[3][16];
    int c = 0;
#pragma unroll 1
    for (int item = 0; item < n_items && ok; ++item) {
      const TmItem it = item_at(item);
      int dst[3];     // output row and row factor of token 16 (ch + 2 j) + lane % 16
      float xin[3];
#pragma unroll
      for (int j = 0; j < 3; ++j) {
        const int t = 16 * (ch + 2 * j) + (lane & 15);
        dst[j] = t < it.nt ? pv.row_dst[it.p0 + t] : 0;
        xin[j] = t < it.nt ? a.xinv[it.p0 + t] : 0.0f;
#pragma unroll
        for (int i = 0; i < 16; ++i) acc[j][i] = 0.0f;
      }
#pragma unroll 1
      for (int cc = 0; cc < nch * kParts; ++cc, ++c) {
        const int buf = c & 1;
        ok = tm_wait_warp((SUM == kTmTurns ? b_acc : b_done) + 8 * buf, (c >> 1) & 1, ab);
        if (!ok) break;
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        const float inv = inv_s[(c / kParts) & 3][r];
        const uint32_t at = lane_base + buf * kTmColD;
#pragma unroll
        for (int j = 0; j < 3; ++j) {
          if (16 * (ch + 2 * j) < it.nt) {
            float d[16];
            tm_ld16(at + 16 * (ch + 2 * j), d);
            asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
            for (int i = 0; i < 16; ++i) acc[j][i] = fmaf(d[i], inv, acc[j][i]);
            if (SUM == kTmSplit) {
              tm_ld16(at + kTmSplitTok + 16 * (ch + 2 * j), d);
              asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
              for (int i = 0; i < 16; ++i) acc[j][i] = fmaf(d[i], inv, acc[j][i]);
            }
          }
        }
        asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
        __syncwarp();
        if (lane == 0) tm_arrive(b_dfree + 8 * buf);
      }
      if (!ok) break;
#pragma unroll
      for (int j = 0; j < 3; ++j) {
        const int t0 = 16 * (ch + 2 * j);
        if (t0 >= it.nt) break;
        // no branch between the values, so that their exponentials and divisions overlap: one after the other they held
        // both accumulators for 14,000 cycles per item of 96 rows, half of its time
        if (NMAT == 2) {
          const int n = it.n0 + q4 * 16 + (lane & 15);
          const bool hi = lane >= 16;  // the lower lanes finish the even tokens, the upper lanes the odd ones
          __nv_bfloat16* out = p.out + n;
          float gv[8], uv[8];
          int row[8];
#pragma unroll
          for (int i = 0; i < 8; ++i) {
            const float other = __shfl_xor_sync(0xffffffffu, hi ? acc[j][2 * i] : acc[j][2 * i + 1], 16);
            const float xs = __shfl_sync(0xffffffffu, xin[j], 2 * i + (hi ? 1 : 0));
            row[i] = __shfl_sync(0xffffffffu, dst[j], 2 * i + (hi ? 1 : 0));
            gv[i] = (hi ? other : acc[j][2 * i]) * xs;
            uv[i] = (hi ? acc[j][2 * i + 1] : other) * xs;
          }
#pragma unroll
          for (int i = 0; i < 8; ++i) gv[i] = swiglu_epilogue(EPI, gv[i], uv[i]);
#pragma unroll
          for (int i = 0; i < 8; ++i)
            if (t0 + 2 * i + (hi ? 1 : 0) < it.nt && n < N) out[(size_t)row[i] * p.ldo] = __float2bfloat16_rn(gv[i]);
        } else {
          const int n = it.n0 + r;
#pragma unroll
          for (int i = 0; i < 16; ++i) {
            const float xs = __shfl_sync(0xffffffffu, xin[j], i);
            const int row = __shfl_sync(0xffffffffu, dst[j], i);
            if (t0 + i < it.nt && n < N) p.out[(size_t)row * p.ldo + n] = __float2bfloat16_rn(acc[j][i] * xs);
          }
        }
      }
    }
  } else if (wid == (kTmExp + kTmFin) / 32) {
    // ================================================================== the warp that issues the MMAs (one lane does)
    int c = 0, xs = 0, xph = 0, n_first = 0;  // n_first: first halves committed (kTmTurns)
#pragma unroll 1
    for (int item = 0; item < n_items && ok; ++item) {
      const TmItem it = item_at(item);
      const uint32_t idesc = tm_idesc((it.nt + 15) & ~15);
#pragma unroll 1
      for (int cc = 0; cc < nch; ++cc, ++c) {
        const int buf = c & 1;
        ok = tm_wait_warp(b_tokf + 8 * xs, xph, ab);
        if (ok && SUM != kTmTurns && c >= 2) ok = tm_wait_warp(b_dfree + 8 * buf, ((c >> 1) - 1) & 1, ab);
        if (ok) ok = tm_wait_warp(b_af + 8 * buf, (c >> 1) & 1, ab);
        if (ok && SUM == kTmTurns && c >= 1) ok = tm_wait_warp(b_dfree, (c - 1) & 1, ab);
        if (!ok) break;
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        const uint32_t d = tmem + (SUM == kTmTurns ? 0 : buf * kTmColD), at = tmem + kTmColA + buf * kTmAStage;
        const uint32_t d2 = SUM == kTmWhole ? d : d + (SUM == kTmSplit ? kTmSplitTok : kTmColD);  // the chunk's second half
        const uint32_t bt = tm_smem(tok + xs * a.xstage);
        auto half = [&](int h) {
#pragma unroll
          for (int g = 2 * h; g < 2 * h + 2; ++g) {
            const uint64_t bd = tm_desc128(bt + g * tn * 128);
#pragma unroll
            for (int k = 0; k < 4; ++k)
              tm_mma(h ? d2 : d, at + g * 32 + k * 8, bd + 2 * k, idesc, k != 0 || (g & 1) != 0 || (h == 1 && SUM == kTmWhole));
          }
        };
        if (SUM == kTmTurns) {
          if (tm_elect()) {
            half(0);
            tm_commit(b_acc);
          }
          __syncwarp();
          ++n_first;
          if (c >= 1) ok = tm_wait_warp(b_dfree + 8, (c - 1) & 1, ab);
          if (!ok) break;
          asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        }
        if (tm_elect()) {
          if (SUM != kTmTurns) half(0);
          half(1);
          if (!MX) {  // the sums' first two pieces, and their third
            tm_mma(d2, at + 128, tm_desc64(bt + tn * 512), idesc, true);
            tm_mma(d2, at + 128, tm_desc64(bt + tn * 512) + 2, idesc, true);
          }
          if (SUM == kTmTurns) tm_commit(b_acc + 8);
          tm_commit(b_done + 8 * buf);
          tm_commit(b_toke + 8 * xs);
        }
        __syncwarp();
        if (++xs == rx) {
          xs = 0;
          xph ^= 1;
        }
      }
    }
    // MMAs in flight, and the arrivals they still owe
    if (SUM == kTmTurns) {
      if (n_first > 0) tm_wait(b_acc, (n_first - 1) & 1, ab, true);
      if (c > 0) tm_wait(b_acc + 8, (c - 1) & 1, ab, true);
    }
    for (int i = max(c - 2, 0); i < c; ++i) tm_wait(b_done + 8 * (i & 1), (i >> 1) & 1, ab, true);
    for (int i = max(c - rx, 0); i < c; ++i) tm_wait(b_toke + 8 * (i % rx), (i / rx) & 1, ab, true);
  } else if (wid == (kTmExp + kTmFin) / 32 + 1) {
    // ================================================================== the warp that copies packed weights
    int c = 0;
#pragma unroll 1
    for (int item = 0; item < n_items && ok; ++item) {
      const TmItem it = item_at(item);
      const int y = it.e * N + it.n0;  // a tile's rows beyond N are the next expert's: computed, not stored
#pragma unroll 1
      for (int cc = 0; cc < nch; ++cc, ++c) {
        const int rs = c % kTmRaw;
        if (c >= kTmRaw) ok = tm_wait_warp(b_rawe + 8 * rs, (c / kTmRaw - 1) & 1, ab);
        if (!ok) break;
        const uint32_t bar = b_rawf + 8 * rs, dst = tm_smem(raw + rs * kTmRawBytes);
        if (tm_elect()) {
          tm_expect(bar, kTmRawBytes);
#pragma unroll
          for (int m = 0; m < NMAT; ++m) tm_load_2d(dst + m * (kTile * 128), &a.w[m], cc * 128, y, bar);
        }
        __syncwarp();
      }
    }
    for (int i = max(c - kTmRaw, 0); i < c; ++i) tm_wait(b_rawf + 8 * (i % kTmRaw), (i / kTmRaw) & 1, ab, true);
  } else {
    // ================================================================== the warp that copies token tiles
    int c = 0;
#pragma unroll 1
    for (int item = 0; item < n_items && ok && !p.withhold; ++item) {
      const TmItem it = item_at(item);
      const int nb = (it.nt + 15) >> 4;
#pragma unroll 1
      for (int cc = 0; cc < nch; ++cc, ++c) {
        const int xs = c % rx;
        if (c >= rx) ok = tm_wait_warp(b_toke + 8 * xs, (c / rx - 1) & 1, ab);
        if (!ok) break;
        const uint32_t bar = b_tokf + 8 * xs, dst = tm_smem(tok + xs * a.xstage);
        if (tm_elect()) {
          tm_expect(bar, nb * (MX ? 8192 : 8192 + 1024));
          for (int b = 0; b < nb; ++b) {
#pragma unroll
            for (int g = 0; g < 4; ++g)
              tm_load_2d(dst + g * tn * 128 + b * 2048, &a.x, cc * kTmChunk + g * 64, it.p0 + 16 * b, bar);
            if (!MX) tm_load_2d(dst + tn * 512 + b * 1024, &a.xb, cc * 32, it.p0 + 16 * b, bar);
          }
        }
        __syncwarp();
      }
    }
    for (int i = max(c - rx, 0); i < c; ++i) tm_wait(b_tokf + 8 * (i % rx), (i / rx) & 1, ab, true);
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  if (abort_s) {  // a bounded wait ran out: the plan says so, and the CTA's results are NaN rather than whatever was there
    if (tid == 0) atomicExch(pv.hdr + 2, kPlanTimeout);
    for (int i = 0; i < n_items; ++i) {
      const TmItem it = item_at(i);
      for (int j = tid; j < it.nt * kTile; j += kTmThreads) {
        const int n = it.n0 + j % kTile;
        if (n < N) p.out[(size_t)pv.row_dst[it.p0 + j / kTile] * p.ldo + n] = __float2bfloat16_rn(__int_as_float(0x7fc00000));
      }
    }
  }
  if (wid == 0) {
    __syncwarp();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(kTmCols) : "memory");
  }
}

// ------------------------------------------------------------------ token rows in sorted order
// One CTA per sorted row: |x|max, then fp16 values under 2^k with |x|max 2^k in [2^14, 2^15), or for affine banks in [2^9,
// 2^10), whose group sums just fit fp16 (64 x 1020 = 65280), and the sums of its groups of 64 as (X1, X2, -X1, -X2) and
// (X3, 0, -X3, 0).  Affine rows take the order in which tm_expand_affine leaves codes.
constexpr int kPrepThreads = 128;

template <bool MX>
__global__ void __launch_bounds__(kPrepThreads) prep_rows_kernel(const __nv_bfloat16* x, int ldx, const int* plan,
                                                                 int rows, int E, int x_by_dst, int K, __half* xs,
                                                                 float* xinv) {
  __shared__ uint32_t warp_max[kPrepThreads / 32];
  pdl_wait();
  pdl_trigger();
  const PlanView pv = plan_view(const_cast<int*>(plan), rows, E);
  const int pos = blockIdx.x, tid = threadIdx.x;
  if (pos >= pv.offset[E]) return;
  const int src = x_by_dst ? pv.row_dst[pos] : pv.row_src[pos];
  const uint4* xr = reinterpret_cast<const uint4*>(x + (size_t)src * ldx);
  const int nv = K >> 3;
  uint32_t mx = 0;
  for (int i = tid; i < nv; i += kPrepThreads) {
    const uint4 v = xr[i];
    const uint32_t q[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
    for (int k = 0; k < 4; ++k) mx = max(mx, max(q[k] & 0x7fffu, (q[k] >> 16) & 0x7fffu));
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) mx = max(mx, __shfl_xor_sync(0xffffffffu, mx, o));
  if ((tid & 31) == 0) warp_max[tid >> 5] = mx;
  __syncthreads();
#pragma unroll
  for (int i = 0; i < kPrepThreads / 32; ++i) mx = max(mx, warp_max[i]);
  int ef = (MX ? 268 : 263) - (int)(mx >> 7);
  ef = (mx == 0) ? 127 : min(max(ef, 2), 252);
  const float scale = __uint_as_float((uint32_t)ef << 23);
  if (tid == 0) xinv[pos] = __uint_as_float((uint32_t)(254 - ef) << 23);
  const size_t stride = MX ? (size_t)K : (size_t)K + K / 8;
  __half* row = xs + (size_t)pos * stride;
  for (int i = tid; i < nv; i += kPrepThreads) {  // nv is a multiple of 32: a warp is whole or absent
    const uint4 v = xr[i];
    const uint32_t q[4] = {v.x, v.y, v.z, v.w};
    float f[8];
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      f[2 * k] = __uint_as_float(q[k] << 16) * scale;
      f[2 * k + 1] = __uint_as_float(q[k] & 0xffff0000u) * scale;
    }
    uint4 o;
    if (MX)
      o = make_uint4(tm_bits(__floats2half2_rn(f[0], f[1])), tm_bits(__floats2half2_rn(f[2], f[3])),
                     tm_bits(__floats2half2_rn(f[4], f[5])), tm_bits(__floats2half2_rn(f[6], f[7])));
    else
      o = make_uint4(tm_bits(__floats2half2_rn(f[0], f[4])), tm_bits(__floats2half2_rn(f[1], f[5])),
                     tm_bits(__floats2half2_rn(f[2], f[6])), tm_bits(__floats2half2_rn(f[3], f[7])));
    *reinterpret_cast<uint4*>(row + (size_t)i * 8) = o;
    if (!MX) {
      float s = ((f[0] + f[1]) + (f[2] + f[3])) + ((f[4] + f[5]) + (f[6] + f[7]));
      s += __shfl_xor_sync(0xffffffffu, s, 1);
      s += __shfl_xor_sync(0xffffffffu, s, 2);
      s += __shfl_xor_sync(0xffffffffu, s, 4);
      if ((tid & 7) == 0) {
        const __half x1 = __float2half_rn(s);
        const float s2 = s - __half2float(x1);
        const __half x2 = __float2half_rn(s2);
        const uint32_t x12 = tm_bits(__halves2half2(x1, x2));
        const uint32_t x3 = tm_bits(__floats2half2_rn(s2 - __half2float(x2), 0.0f));
        const int g = i >> 3;
        uint2* to = reinterpret_cast<uint2*>(row + K + (g >> 2) * 32 + (g & 3) * 4);  // 32 values per chunk: two K steps
        to[0] = make_uint2(x12, x12 ^ 0x80008000u);
        to[4] = make_uint2(x3, x3 ^ 0x80008000u);
      }
    }
  }
}

// ------------------------------------------------------------------ host side

size_t qmm_tma_workspace(int rows, int K, bool mx) {
  const size_t row = mx ? (size_t)K * 2 : (size_t)K * 2 + K / 4;
  return (((size_t)rows * row + 255) & ~(size_t)255) + (size_t)rows * sizeof(float);
}

// Which calls gain from the path: whole chunks along K, and more than eight rows on some expert (by the caller's
// bound).  A block of up to eight token rows is taken by the one-launch kernel or the register-fed ones, whose cost per
// expert is the same for one row as for eight (whole block, c2, T = 8: 76 us in one launch, 105 here; T = 16: 151 us in
// two launches, 121 here).
bool qmm_tma_wants(int E, int K, int rows_hint) {
  return K % kTmChunk == 0 && E <= kTmMaxTasks && rows_hint > 8;
}

// Whether this call takes it: wanted, a workspace is there, and the encoder takes the tensor maps.
bool qmm_tma_covers(const QmmParams& q, int nmat, bool mx, int rows_hint, const void* ws, size_t ws_bytes) {
  if (!ws || ((uintptr_t)ws & 255) || ws_bytes < qmm_tma_workspace(q.rows, q.K, mx)) return false;
  if (!qmm_tma_wants(q.E, q.K, rows_hint) || (long long)q.E * q.N > (1ll << 31) - kTmRows) return false;
  for (int m = 0; m < nmat; ++m)
    if ((uintptr_t)q.w[m] & 15) return false;
  return true;
}

typedef CUresult (*EncodeTiled)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                                CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

static EncodeTiled encoder() {
  static const EncodeTiled fn = [] {
    void* f = nullptr;
    cudaDriverEntryPointQueryResult res;
    if (cudaGetDriverEntryPointByVersion("cuTensorMapEncodeTiled", &f, 12000, cudaEnableDefault, &res) != cudaSuccess ||
        res != cudaDriverEntryPointSuccess)
      f = nullptr;
    return (EncodeTiled)f;
  }();
  return fn;
}

static bool map_2d(CUtensorMap* m, CUtensorMapDataType dt, const void* ptr, size_t cols, size_t nrows, size_t stride,
                   int box_cols, int box_rows, CUtensorMapSwizzle sw, CUtensorMapL2promotion prom) {
  const cuuint64_t dims[2] = {cols, nrows}, strides[1] = {stride};
  const cuuint32_t box[2] = {(cuuint32_t)box_cols, (cuuint32_t)box_rows}, es[2] = {1, 1};
  return encoder()(m, dt, 2, const_cast<void*>(ptr), dims, strides, box, es, CU_TENSOR_MAP_INTERLEAVE_NONE, sw, prom,
                   CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

template <bool MX, int NMAT, int EPI>
static int launch_tma(const TmArgs& a, int grid, size_t smem, cudaStream_t st, const char* who) {
  auto kern = a.tn <= kTmSplitTok ? qmm_tma_kernel<MX, NMAT, EPI, kTmSplit>
                                  : qmm_tma_kernel<MX, NMAT, EPI, MX ? kTmWhole : kTmTurns>;
  cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (e == cudaSuccess) e = launch_pdl(kern, dim3(grid), dim3(kTmThreads), smem, st, a);
  if (e != cudaSuccess) return fail(ZMOE_ERR_CUDA, "%s: launch failed: %s", who, cudaGetErrorString(e));
  return check_launch("qmm_tma_kernel");
}

int qmm_tma_launch(const QmmParams& q, int nmat, bool mx, int rows_hint, int max_groups, void* ws, cudaStream_t st,
                   const char* who) {
  if (!encoder()) return fail(ZMOE_ERR_CUDA, "%s: cuTensorMapEncodeTiled is not available", who);
  const size_t row = mx ? (size_t)q.K * 2 : (size_t)q.K * 2 + q.K / 4;  // bytes of a prepared row
  unsigned char* xs = reinterpret_cast<unsigned char*>(ws);
  float* xinv = reinterpret_cast<float*>(xs + (((size_t)q.rows * row + 255) & ~(size_t)255));
  TmArgs a;
  a.q = q;
  a.xinv = xinv;
  a.nch = q.K / kTmChunk;
  bool fine = true;
  for (int m = 0; m < 2; ++m)
    fine = fine && map_2d(&a.w[m], CU_TENSOR_MAP_DATA_TYPE_UINT8, q.w[m], (size_t)q.K / 2, (size_t)q.E * q.N,
                          (size_t)q.K / 2, 128, kTmRows / nmat, CU_TENSOR_MAP_SWIZZLE_128B,
                          CU_TENSOR_MAP_L2_PROMOTION_L2_256B);
  fine = fine && map_2d(&a.x, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, xs, q.K, q.rows, row, 64, 16, CU_TENSOR_MAP_SWIZZLE_128B,
                        CU_TENSOR_MAP_L2_PROMOTION_L2_256B);
  if (mx)
    a.xb = a.x;
  else
    fine = fine && map_2d(&a.xb, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, xs + (size_t)q.K * 2, q.K / 8, q.rows, row, 32, 16,
                          CU_TENSOR_MAP_SWIZZLE_64B, CU_TENSOR_MAP_L2_PROMOTION_NONE);
  if (!fine) return fail(ZMOE_ERR_CUDA, "%s: a tensor map was refused", who);
  // Token rows per item: up to twice the average task in whole 16s (a larger task takes several equal blocks); the
  // fewer rows a stage must hold, the more stages are in flight.
  long long tn = 2ll * q.rows / max_groups + 8;
  if (tn > rows_hint) tn = rows_hint;
  tn = (tn + 15) / 16 * 16;
  a.tn = tn > kTmMaxTok ? kTmMaxTok : (int)tn;
  a.xstage = (a.tn * (mx ? 512 : 576) + 1023) & ~1023;
  const int fixed = 1024 + kTmRaw * kTmRawBytes + kTmScRing * kTmExp * 16;
  const int room = 227 * 1024 - 12 * 1024 - fixed;  // 12 KB: the static part (prefix sums, items, barriers, row factors)
  a.rx = room / a.xstage > kTmMaxX ? kTmMaxX : room / a.xstage;
  const size_t smem = (size_t)fixed + (size_t)a.rx * a.xstage;
  int sms = 0, dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess ||
      cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || sms <= 0)
    return fail(ZMOE_ERR_CUDA, "%s: SM count query failed", who);
  cudaError_t e =
      mx ? launch_pdl(prep_rows_kernel<true>, dim3(q.rows), dim3(kPrepThreads), 0, st, q.x, q.ldx, q.plan, q.rows, q.E,
                      q.x_by_dst, q.K, (__half*)xs, xinv)
         : launch_pdl(prep_rows_kernel<false>, dim3(q.rows), dim3(kPrepThreads), 0, st, q.x, q.ldx, q.plan, q.rows, q.E,
                      q.x_by_dst, q.K, (__half*)xs, xinv);
  if (e != cudaSuccess) return fail(ZMOE_ERR_CUDA, "%s: launch failed: %s", who, cudaGetErrorString(e));
  // one CTA per SM, fewer when the work list is shorter
  const long long ntiles = (q.N * (long long)nmat + kTmRows - 1) / kTmRows;
  const long long items = ntiles * ((long long)q.rows / a.tn + max_groups);
  const int grid = (int)(items < sms ? items : sms);
  if (nmat == 1) return mx ? launch_tma<true, 1, 0>(a, grid, smem, st, who) : launch_tma<false, 1, 0>(a, grid, smem, st, who);
  if (mx) return q.epilogue == 2 ? launch_tma<true, 2, 2>(a, grid, smem, st, who) : launch_tma<true, 2, 1>(a, grid, smem, st, who);
  if (q.epilogue == 2) return launch_tma<false, 2, 2>(a, grid, smem, st, who);
  if (q.epilogue == 3) return launch_tma<false, 2, 3>(a, grid, smem, st, who);
  return launch_tma<false, 2, 1>(a, grid, smem, st, who);
}

}  // namespace zmoe

using namespace zmoe;

extern "C" size_t zmoe_qmm_workspace_bytes(int rows, int E, int K, int rows_hint, int qmode) {
  if (rows <= 0 || E <= 0 || K <= 0) return 0;
  if (rows_hint <= 0 || rows_hint > rows) rows_hint = rows;
  return qmm_tma_wants(E, K, rows_hint) ? qmm_tma_workspace(rows, K, qmode == ZMOE_Q_MXFP4) : 0;
}
