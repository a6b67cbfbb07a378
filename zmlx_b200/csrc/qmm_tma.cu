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
//     expanders two or three sets of 128 threads (one per weight row) take turns at the chunks, turn the codes into the fp16
//               A operand and store it straight into the set's stage in TENSOR MEMORY (tcgen05.st): no shared-memory round
//               trip, no swizzle arithmetic; one set's waits and latencies lie under the other sets' arithmetic;
//     issuer    one thread issues tcgen05.mma (M 128 x N 16..96 x K 16, A in tensor memory, B in shared memory);
//     finishers 256 threads fold the chunk's accumulator into fp32 registers and, at the end of an item, apply the
//               SwiGLU contract and store bf16 rows through the plan.
//
// What bounds a chunk (clock stamps of one CTA, c5 with 64 rows, gate/up): not the tensor pipe (8 %) nor DRAM, but the
// expanders.  A warp of theirs holds a chunk for 2000 cycles and more -- its instructions go one by one through a pipe that
// takes two cycles each (shifts, masks, conversions), satisfied waits cost 100 cycles -- while the packed bytes need 830.  So:
// five of those instructions per packed word instead of seven, scales converted once per group, the waits' looks taken
// together, and up to 16 token rows (whose accumulators leave room for a third stage) three sets of expanders, and finishers
// that take alternate ITEMS, one set's epilogue under the other's folds.  us, gate/up and down, before -> now: c2 T=32
// 80.5/48.2 -> 63.5/38.5 (2990 GB/s), c5 T=64 1107/585 -> 836/427 (4300 GB/s), c5 T=512 1369/706 -> 1209/618, c2 T=4096
// 442/294 -> 407/292, mxfp4 c3 T=300 89/49 -> 75/42.  (Alternate items above 16 rows: the finishers' registers do not
// suffice; with setmaxnreg c5 T=512 took 1595/667, c2 T=4096 485/351.  Four stages of half a chunk: twice the waits, a fifth
// slower.  Scales prepared by warps of their own: 974/468 for c5 T=64.)
//
// Arithmetic.  Affine: w = q s + b = (q - 8) s + (b + 8 s).  q - 8 has three bits and a sign, s eight: their product fits
// fp16's eleven, so the scale goes into the operand and the accumulator runs over several groups.  The second term is two
// more K = 16 steps on one operand, per group (b, b, -8 s, -8 s), against the group's float32 sum X as three fp16 pieces (33
// bits): (X1, X2, -X1, -X2) and (X3, 0, -X3, 0).  The scales are first multiplied by a power of two per (row, chunk), undone
// in fp32 by the finishers, so the range of fp16 is no limit on the checkpoint's.
// (q - 8) s and b are exact while the scales and offsets of a row's chunk (other than zero) lie within 8 binades below the
// largest scale; chunks with values further apart are expanded another way (tm_expand_far), exact over 28; below, a weight is
// off by at most 2^-39 of the largest of its row's chunk.  mxfp4: e2m1 value x 2^(e - emax + 13), exact in fp16 over 36 binades,
// same row factor.  Token rows carry a power of two per row: a bfloat16 of the row is exact down to 2^-26 (mxfp4: 2^-31) of its largest,
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
constexpr int kTmSplitTok = 48;                   // up to so many token rows an accumulator is two, one per half chunk
// How a chunk is summed.  The tensor core cuts products and sums off at a fixed distance below the largest of them, so
// long sums lose.  Share of bfloat16 results that are not the float64 result's rounding, affine, K = 768 and 2048: whole
// chunks 1.7e-4, halves 1.1e-4 and 1.2e-4 (float32 sums over groups of 64 unscaled codes: 0.6e-4 and 1.0e-4).  Up to
// kTmSplitTok token rows the two halves lie side by side and are handed over together; wider items hand them over one
// after the other, which costs 6 % (c2 with 4096 rows: 828 -> 879 us a block; quarters: 1090).  Products of e2m1 codes and
// powers of two hardly lose any bits: whole chunks, 0.1e-4 to 0.6e-4.
enum TmSum { kTmWhole, kTmSplit, kTmTurns };
constexpr int kTmAStage = 136;                    // columns of an operand stage: 128 of codes, 8 of scales and biases
constexpr int kTmInv = 8;                         // chunks whose row factors are kept

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
// The same look without a suspension: a phase that is already complete costs less this way.
__device__ __forceinline__ bool tm_test(uint32_t bar, uint32_t parity) {
  uint32_t ok;
  asm volatile("{ .reg .pred p; mbarrier.test_wait.parity.shared::cta.b64 p, [%1], %2; selp.u32 %0, 1, 0, p; }"
               : "=r"(ok)
               : "r"(bar), "r"(parity)
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
__device__ __forceinline__ bool tm_wait_long(uint32_t bar, uint32_t parity, volatile int* abort_flag, bool drain) {
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
  if (tm_test(bar, parity)) return true;
  return tm_wait_long(bar, parity, abort_flag, drain);
}
// The same for a whole warp: all lanes leave together, as the tcgen05.ld and .st that follow need them to.
__device__ __forceinline__ bool tm_wait_warp(uint32_t bar, uint32_t parity, volatile int* abort_flag) {
  return __all_sync(0xffffffffu, tm_wait(bar, parity, abort_flag));
}
// Two or three phases: both looks at once where all are complete.
__device__ __forceinline__ bool tm_wait_both(uint32_t b0, uint32_t p0, uint32_t b1, uint32_t p1, volatile int* abort_flag) {
  const bool t0 = tm_test(b0, p0), t1 = tm_test(b1, p1);
  if (__all_sync(0xffffffffu, t0 && t1)) return true;
  return tm_wait_warp(b0, p0, abort_flag) && tm_wait_warp(b1, p1, abort_flag);
}
__device__ __forceinline__ bool tm_wait_three(uint32_t b0, uint32_t p0, uint32_t b1, uint32_t p1, uint32_t b2, uint32_t p2,
                                              volatile int* abort_flag) {
  const bool t0 = tm_test(b0, p0), t1 = tm_test(b1, p1), t2 = tm_test(b2, p2);
  if (__all_sync(0xffffffffu, t0 && t1 && t2)) return true;
  return tm_wait_warp(b0, p0, abort_flag) && tm_wait_warp(b1, p1, abort_flag) && tm_wait_warp(b2, p2, abort_flag);
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
__device__ __forceinline__ void tm_st8(uint32_t taddr, uint32_t r0, uint32_t r1, uint32_t r2, uint32_t r3, uint32_t r4,
                                       uint32_t r5, uint32_t r6, uint32_t r7) {
  asm volatile("tcgen05.st.sync.aligned.32x32b.x8.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8};" ::"r"(taddr), "r"(r0), "r"(r1), "r"(r2),
               "r"(r3), "r"(r4), "r"(r5), "r"(r6), "r"(r7)
               : "memory");
}
__device__ __forceinline__ void tm_st32(uint32_t taddr, const uint32_t (&r)[32]) {
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x32.b32 [%0], "
      "{%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31,"
      "%32};" ::"r"(taddr),
      "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]), "r"(r[9]),
      "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15]), "r"(r[16]), "r"(r[17]), "r"(r[18]), "r"(r[19]),
      "r"(r[20]), "r"(r[21]), "r"(r[22]), "r"(r[23]), "r"(r[24]), "r"(r[25]), "r"(r[26]), "r"(r[27]), "r"(r[28]), "r"(r[29]),
      "r"(r[30]), "r"(r[31])
      : "memory");
}
// What the warp loaded from an accumulator is in registers: its owner may write the accumulator again.
__device__ __forceinline__ void tm_release(uint32_t bar, int lane) {
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncwarp();
  if (lane == 0) tm_arrive(bar);
}
// One lane of a converged warp.  The compiler knows an elected thread to be alone; behind `lane == 0` it would wrap
// every tcgen05.mma and TMA instruction in a loop over the lanes that might be active (measured: 190 cycles per MMA
// whatever its shape, 17 of them per chunk).
__device__ __forceinline__ bool tm_elect() {
  uint32_t one;
  asm volatile("{ .reg .pred p; elect.sync _|p, 0xffffffff; selp.u32 %0, 1, 0, p; }" : "=r"(one));
  return one != 0;
}
// Halves that are zero become the largest number.
__device__ __forceinline__ uint32_t tm_zero_as_max(uint32_t v) { return v | __vcmpeq2(v, 0u); }
__device__ __forceinline__ uint32_t tm_bits(__half2 h) { return *reinterpret_cast<const uint32_t*>(&h); }
__device__ __forceinline__ __half2 tm_half2(uint32_t u) { return *reinterpret_cast<const __half2*>(&u); }

// Eight codes of a packed word times the group's scale, as four half2 in the order (0,4) (1,5) (2,6) (3,7) that the
// token rows are written in.  A nibble at bits 0-3 (4-7) of a half IS the fp16 number q 2^-24 (q 2^-20), subnormal or not, so
// one fused multiply-add gives q 2^-24 (s 2^24) - 8 s = (q - 8) s, exact: one shift, four masks, four half2 operations per
// eight codes.
__device__ __forceinline__ void tm_expand_affine(uint32_t w, __half2 s24, __half2 s20, __half2 m8s, uint32_t* out) {
  const uint32_t m = 0x000F000Fu, m4 = 0x00F000F0u, w8 = w >> 8;
  out[0] = tm_bits(__hfma2(tm_half2(w & m), s24, m8s));
  out[1] = tm_bits(__hfma2(tm_half2(w & m4), s20, m8s));
  out[2] = tm_bits(__hfma2(tm_half2(w8 & m), s24, m8s));
  out[3] = tm_bits(__hfma2(tm_half2(w8 & m4), s20, m8s));
}
// A chunk whose scales lie further apart than tm_expand_affine takes: a nibble at bits 6-9 of a half under the exponent of
// 16 is 16 + q, and (16 + q) s - 24 s = (q - 8) s is exact for s from 2^-17 to 2^11 (24 s has ten bits).  One more shift and
// four more masks per word: every chunk done this way cost 9 to 13 % (c2 with 32 rows 600 -> 657 us, c5 with 64 rows 1790
// -> 2038), so it is a loop of its own, for the warps that meet such a chunk.
__device__ __forceinline__ void tm_expand_far(const unsigned char* src, uint32_t swz, uint4 sc, float P, uint32_t taddr) {
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
__device__ __forceinline__ TmItem tm_item(const PlanView& pv, const int* prefix, int ntasks, int ntiles, int tile_rows,
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

// Token blocks of at most tn rows before every task (the first warp computes them, the CTA waits).
__device__ __forceinline__ void tm_block_prefix(const PlanView& pv, int ntasks, int tn, int wid, int lane, int* prefix) {
  if (wid == 0) {  // lane = a contiguous run of tasks
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
      prefix[i] = run;
      run += (pv.tasks[4 * i + 2] + tn - 1) / tn;
    }
    if (lane == 31) prefix[ntasks] = incl;
  }
  __syncthreads();
}

// The sums of weight row (q4, lane) and token rows t0 .. t0 + 15 of the item, times the rows' factors, through the
// SwiGLU contract to the output.  xin, dst: row factor and output row of token t0 + lane % 16.
// No branch between the values, so that their exponentials and divisions overlap: one after the other they held
// both accumulators for 14,000 cycles per item of 96 rows, half of its time.
template <int NMAT, int EPI>
__device__ __forceinline__ void tm_store_block(const QmmParams& p, const TmItem& it, int q4, int lane, int t0,
                                               const float (&acc)[16], float xin, int dst, int N) {
  if (NMAT == 2) {
    const int n = it.n0 + q4 * 16 + (lane & 15);
    const bool hi = lane >= 16;  // the lower lanes finish the even tokens, the upper lanes the odd ones
    __nv_bfloat16* out = p.out + n;
    float gv[8], uv[8];
    int row[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      const float other = __shfl_xor_sync(0xffffffffu, hi ? acc[2 * i] : acc[2 * i + 1], 16);
      const float xs = __shfl_sync(0xffffffffu, xin, 2 * i + (hi ? 1 : 0));
      row[i] = __shfl_sync(0xffffffffu, dst, 2 * i + (hi ? 1 : 0));
      gv[i] = (hi ? other : acc[2 * i]) * xs;
      uv[i] = (hi ? acc[2 * i + 1] : other) * xs;
    }
#pragma unroll
    for (int i = 0; i < 8; ++i) gv[i] = swiglu_epilogue(EPI, gv[i], uv[i]);
#pragma unroll
    for (int i = 0; i < 8; ++i)
      if (t0 + 2 * i + (hi ? 1 : 0) < it.nt && n < N) out[(size_t)row[i] * p.ldo] = __float2bfloat16_rn(gv[i]);
  } else {
    const int n = it.n0 + q4 * 32 + lane;
#pragma unroll
    for (int i = 0; i < 16; ++i) {
      const float xs = __shfl_sync(0xffffffffu, xin, i);
      const int row = __shfl_sync(0xffffffffu, dst, i);
      if (t0 + i < it.nt && n < N) p.out[(size_t)row * p.ldo + n] = __float2bfloat16_rn(acc[i] * xs);
    }
  }
}

// Shapes of an instance.  NB: blocks of 16 token rows an item may have.  SUM: see above.  The accumulators are a ring of nD, a
// chunk takes one of them or (kTmTurns) two; kTmSplit puts a chunk's two halves side by side into one.
template <int NB, TmSum SUM>
struct TmShape {
  static constexpr int nE = NB == 1 ? 3 : 2;                               // sets of expanders, operand stages
  static constexpr bool alt = NB == 1;                                     // finisher sets take every other item, or block of it
  static constexpr int threads = 128 * nE + 256 + 128;                     // expanders, finishers, issuer and copiers
  static constexpr int parts = SUM == kTmTurns ? 2 : 1;                    // hand-overs of accumulators per chunk
  static constexpr int colD = (SUM == kTmSplit ? 2 : 1) * 16 * NB;        // columns of an accumulator
  static constexpr int colA = kTmCols - nE * kTmAStage;                    // first operand column
  static constexpr int nD = colA / colD > 4 ? 4 : colA / colD;
  static constexpr int nJ = alt ? NB : (NB + 1) / 2;                       // blocks of a finisher
  static_assert(nD >= 2 && nE + nD < kTmInv, "tensor memory, row factors in flight");
};

// EPI: the SwiGLU contract of gate and up (QmmParams::epilogue).
template <bool MX, int NMAT, int EPI, int NB, TmSum SUM>
__global__ void __launch_bounds__((TmShape<NB, SUM>::threads), 1) qmm_tma_kernel(const __grid_constant__ TmArgs a) {
  using S = TmShape<NB, SUM>;
  extern __shared__ __align__(1024) unsigned char tm_dyn[];
  __shared__ uint32_t tmem_base_s;
  // raw full / empty, token full / empty, A full, MMAs done, accumulator full (one per finisher set) / free
  __shared__ __align__(8) unsigned long long bars_s[2 * kTmRaw + 2 * kTmMaxX + 2 * S::nE + 3 * S::nD];
  __shared__ float inv_s[kTmInv][kTmRows];
  __shared__ volatile int abort_s;
  __shared__ int prefix_s[kTmMaxTasks + 1];
  __shared__ int4 items_s[kTmItems];

  constexpr int kTile = kTmRows / NMAT;  // output rows of an item
  const QmmParams& p = a.q;
  const int tid = threadIdx.x, lane = tid & 31;
  const int wid = __shfl_sync(0xffffffffu, tid >> 5, 0);
  const int N = p.N, nch = a.nch, tn = a.tn, rx = a.rx;
  const PlanView pv = plan_view(const_cast<int*>(p.plan), p.rows, p.E);
  unsigned char* base = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(tm_dyn) + 1023) & ~(uintptr_t)1023);
  unsigned char* raw = base;
  unsigned char* tok = raw + kTmRaw * kTmRawBytes;
  unsigned char* scr = tok + rx * a.xstage;  // [slot][expander thread][16 bytes]
  const uint32_t b_rawf = tm_smem(bars_s), b_rawe = b_rawf + 8 * kTmRaw, b_tokf = b_rawe + 8 * kTmRaw;
  const uint32_t b_toke = b_tokf + 8 * kTmMaxX, b_af = b_toke + 8 * kTmMaxX, b_done = b_af + 8 * S::nE;
  const uint32_t b_dfull = b_done + 8 * S::nE, b_dfree = b_dfull + 16 * S::nD;

  // The plan, the prepared rows and their factors may be the work of the kernel before, still running when this one
  // starts: they are read with plain loads after the wait, never through the read-only path.
  pdl_wait();
  pdl_trigger();
  const int ntasks = min(pv.hdr[0], kTmMaxTasks);
  tm_block_prefix(pv, ntasks, tn, wid, lane, prefix_s);
  const int ntiles = (N + kTile - 1) / kTile;
  const int total = ntiles * prefix_s[ntasks];
  if ((int)blockIdx.x >= total) return;  // before any tensor memory is taken
  const int n_items = __shfl_sync(0xffffffffu, (total - (int)blockIdx.x + (int)gridDim.x - 1) / (int)gridDim.x, 0);
  const int n_chunks = n_items * nch;
  // Every role walks the CTA's items: they are looked up once, by all threads (a search, two divisions and a load of
  // the task record took each role some 1500 cycles per item); a CTA with more of them looks the rest up as it goes.
  for (int i = tid; i < min(n_items, kTmItems); i += S::threads) {
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
      tm_bar_init(b_rawe + 8 * i, 4);
    }
    for (int i = 0; i < kTmMaxX; ++i) {
      tm_bar_init(b_tokf + 8 * i, 1);
      tm_bar_init(b_toke + 8 * i, 1);
    }
    for (int i = 0; i < S::nE; ++i) {
      tm_bar_init(b_af + 8 * i, 4);
      tm_bar_init(b_done + 8 * i, 1);
    }
    for (int i = 0; i < 2 * S::nD; ++i) tm_bar_init(b_dfull + 8 * i, 1);
    for (int i = 0; i < S::nD; ++i) tm_bar_init(b_dfree + 8 * i, S::alt ? 4 : 8);
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
  const uint32_t tmem = __shfl_sync(0xffffffffu, tmem_base_s, 0);
  volatile int* ab = &abort_s;
  bool ok = true;

  const int q4 = wid & 3;
  const int r = q4 * 32 + lane;  // tensor-memory lane
  if (wid < 4 * S::nE) {
    // ================================================================== expanders: a weight row of every other chunk
    const int set = wid >> 2;
    const int mat = NMAT == 2 ? (lane >> 4) : 0;
    const int rb = NMAT == 2 ? q4 * 16 + (lane & 15) : r;  // row inside the matrix's box
    const int swz = rb & 7;
    const uint32_t at = tmem + ((uint32_t)(q4 * 32) << 16) + S::colA + set * kTmAStage;
    const unsigned char* my_raw = raw + mat * (kTile * 128) + rb * 128;
    unsigned char* my_sc = scr + tid * 16;
    // the cursor of the scale copies runs kTmScAhead of the thread's chunks ahead
    int f_item = 0, f_c = set, f_slot = 0;
    const unsigned char *f_s = nullptr, *f_b = nullptr;
    auto fetch = [&] {
      while (f_c >= nch) {
        f_c -= nch;
        ++f_item;
        f_s = nullptr;
      }
      if (f_item < n_items) {
        if (f_s == nullptr) {
          const TmItem it = item_at(f_item);
          const size_t row = (size_t)it.e * N + min(it.n0 + rb, N - 1);  // clamped rows are computed, not stored
          // 8 bytes per chunk: four bfloat16 scales (biases) or eight e8m0 bytes
          f_s = reinterpret_cast<const unsigned char*>(p.s[mat]) + row * nch * 8;
          if (!MX) f_b = reinterpret_cast<const unsigned char*>(p.b[mat]) + row * nch * 8;
        }
        unsigned char* dst = my_sc + f_slot * (128 * S::nE * 16);
        cp_async_8(dst, f_s + f_c * 8);
        if (!MX) cp_async_8(dst + 8, f_b + f_c * 8);
      }
      asm volatile("cp.async.commit_group;" ::: "memory");
      f_c += S::nE;
      f_slot = (f_slot + 1) % kTmScRing;
    };
#pragma unroll 1
    for (int i = 0; i < kTmScAhead; ++i) fetch();
    int rs = set, rph = 0, slot = 0, aph = 1;  // raw slot and its phase, scale slot, phase of the operand stage
#pragma unroll 1
    for (int c = set; c < n_chunks; c += S::nE) {
      fetch();
      asm volatile("cp.async.wait_group %0;" ::"n"(kTmScAhead) : "memory");
      const uint4 sc = *reinterpret_cast<const uint4*>(my_sc + slot * (128 * S::nE * 16));
      slot = (slot + 1) % kTmScRing;
      // ---- the chunk's power of two
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
        const uint32_t m15 = 0x7fff7fffu;
        uint32_t ms = __vmaxu2(sc.x & m15, sc.y & m15);
        uint32_t mb = __vmaxu2(sc.z & m15, sc.w & m15);
        ms = max(ms & 0xffffu, ms >> 16);
        mb = max(mb & 0xffffu, mb >> 16);
        // 2^(140 - e) brings |s| below 2^-8 (so that s 2^24 stays below 2^16) and |b| below 2^14; a scale or an offset, other
        // than zero, that this leaves below 2^-17 asks for the wider form, where |s| may reach 2^11 (so do scales at float's
        // upper end)
        const int es = (int)(ms >> 7), eb = (int)(mb >> 7);
        int e = max(es + 22, eb);
        const uint32_t least = __vminu2(__vminu2(tm_zero_as_max(sc.x & m15), tm_zero_as_max(sc.y & m15)),
                                        __vminu2(tm_zero_as_max(sc.z & m15), tm_zero_as_max(sc.w & m15)));
        far = __any_sync(0xffffffffu, (int)(min(least & 0xffffu, least >> 16) >> 7) + 30 < e || e > 253);
        if (far) e = max(es + 3, eb);
        e = min(max(e, far ? 14 : 38), 253);
        P = __uint_as_float((uint32_t)(267 - e) << 23);
        inv = __uint_as_float((uint32_t)(e - 13) << 23);
      }
      // ---- the chunk is there, and the stage is free: the MMAs of the thread's previous chunk are done (at once the first time)
      ok = tm_wait_both(b_rawf + 8 * rs, rph, b_done + 8 * set, aph, ab);
      if (!ok) break;
      const unsigned char* src = my_raw + rs * kTmRawBytes;
      uint4 w[2];
      w[0] = *reinterpret_cast<const uint4*>(src + (swz << 4));
      w[1] = *reinterpret_cast<const uint4*>(src + ((1 ^ swz) << 4));
      aph ^= 1;
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      if (!MX && far) {
        tm_expand_far(src, swz, sc, P, at);
      } else {
        const float P24 = P * 16777216.0f;
        uint32_t bias[8];
#pragma unroll
        for (int i = 0; i < 4; ++i) {  // 64 codes each: a group, or two mxfp4 blocks
          uint32_t o[32];
          const uint32_t ws[8] = {w[0].x, w[0].y, w[0].z, w[0].w, w[1].x, w[1].y, w[1].z, w[1].w};
          if (i < 3) {
            w[0] = *reinterpret_cast<const uint4*>(src + (((2 * i + 2) ^ swz) << 4));
            w[1] = *reinterpret_cast<const uint4*>(src + (((2 * i + 3) ^ swz) << 4));
          }
          const uint32_t s2 = i < 2 ? sc.x : sc.y, b2 = i < 2 ? sc.z : sc.w;
          if (MX) {
            // fp16 2^(e - emax + 13) in both halves, subnormal ones included
            const uint32_t ee = (i & 1) ? s2 >> 16 : s2;
            const __half2 s0 = __float2half2_rn(__uint_as_float((uint32_t)max((int)(ee & 0xffu) - emax + 140, 0) << 23));
            const __half2 s1 = __float2half2_rn(__uint_as_float((uint32_t)max((int)((ee >> 8) & 0xffu) - emax + 140, 0) << 23));
#pragma unroll
            for (int k = 0; k < 8; ++k) tm_expand_mx(ws[k], k < 4 ? s0 : s1, o + 4 * k);
          } else {
            const __half2 s24 = __float2half2_rn(__uint_as_float((i & 1) ? s2 & 0xffff0000u : s2 << 16) * P24);
            const __half2 s20 = __hmul2(s24, __float2half2_rn(0x1p-4f)), s_off = __hmul2(s24, __float2half2_rn(-0x1p-21f));
#pragma unroll
            for (int k = 0; k < 8; ++k) tm_expand_affine(ws[k], s24, s20, s_off, o + 4 * k);
            const __half2 b_op = __float2half2_rn(__uint_as_float((i & 1) ? b2 & 0xffff0000u : b2 << 16) * P);
            bias[2 * i] = tm_bits(b_op);
            bias[2 * i + 1] = tm_bits(s_off);
          }
          tm_st32(at + i * 32, o);
        }
        if (!MX) tm_st8(at + 128, bias[0], bias[1], bias[2], bias[3], bias[4], bias[5], bias[6], bias[7]);
      }
      inv_s[c & (kTmInv - 1)][r] = inv;  // the finishers are at most nE + nD chunks behind: the MMAs wait for them
      asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
      asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
      __syncwarp();
      if (lane == 0) {
        tm_arrive(b_af + 8 * set);
        tm_arrive(b_rawe + 8 * rs);
      }
      __syncwarp();
      rs += S::nE;
      if (rs >= kTmRaw) {
        rs -= kTmRaw;
        rph ^= 1;
      }
    }
    asm volatile("cp.async.wait_all;" ::: "memory");
  } else if (wid < 4 * S::nE + 8) {
    // ================================================================== finishers: a weight row of every other item (or block)
    const int set = (wid >> 2) - S::nE;
    const uint32_t lane_base = tmem + ((uint32_t)(q4 * 32) << 16), b_full = b_dfull + (S::alt ? 8 * S::nD * set : 0);
    uint32_t phases = 0;  // of the set's barriers, one bit each
#pragma unroll 1
    for (int item = S::alt ? set : 0; item < n_items && ok; item += S::alt ? 2 : 1) {
      const TmItem it = item_at(item);
      float acc[S::nJ][16];  // of token block j, or set + 2 j
#pragma unroll
      for (int j = 0; j < S::nJ; ++j)
#pragma unroll
        for (int i = 0; i < 16; ++i) acc[j][i] = 0.0f;
      auto t0_of = [&](int j) { return 16 * (S::alt ? j : set + 2 * j); };
      int c = item * nch;
      int buf = (c * S::parts) % S::nD;
#pragma unroll 1
      for (int cc = 0; cc < nch * S::parts; ++cc) {
        ok = tm_wait_warp(b_full + 8 * buf, (phases >> buf) & 1, ab);
        if (!ok) break;
        phases ^= 1u << buf;
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        const float inv = inv_s[c & (kTmInv - 1)][r];
        if (S::parts == 1 || (cc & 1)) ++c;
        const uint32_t at = lane_base + buf * S::colD;
        if (NB == 1) {  // both halves at once
          float d[2][16];
          tm_ld16(at, d[0]);
          if (SUM == kTmSplit) tm_ld16(at + 16, d[1]);
          asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
          tm_release(b_dfree + 8 * buf, lane);
#pragma unroll
          for (int h = 0; h < (SUM == kTmSplit ? 2 : 1); ++h)
#pragma unroll
            for (int i = 0; i < 16; ++i) acc[0][i] = fmaf(d[h][i], inv, acc[0][i]);
        } else {
#pragma unroll
          for (int j = 0; j < S::nJ; ++j)
            if (t0_of(j) < it.nt) {
#pragma unroll
              for (int h = 0; h < (SUM == kTmSplit ? 2 : 1); ++h) {
                float d[16];
                tm_ld16(at + h * 16 * NB + t0_of(j), d);
                asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
                for (int i = 0; i < 16; ++i) acc[j][i] = fmaf(d[i], inv, acc[j][i]);
              }
            }
          tm_release(b_dfree + 8 * buf, lane);
        }
        if (++buf == S::nD) buf = 0;
      }
      if (!ok) break;
#pragma unroll
      for (int j = 0; j < S::nJ; ++j)
        if (t0_of(j) < it.nt) {
          const int t = it.p0 + min(t0_of(j) + (lane & 15), it.nt - 1);
          tm_store_block<NMAT, EPI>(p, it, q4, lane, t0_of(j), acc[j], a.xinv[t], pv.row_dst[t], N);
        }
    }
  } else {
    if (wid == 4 * S::nE + 8) {
      // ================================================================ the warp that issues the MMAs (one lane does)
      int c = 0, xs = 0, xph = 0, as = 0, aph = 0, ds = 0, dph = 1;
      uint32_t used = 0, last = 0;  // accumulator-full barriers committed to, and the parity of each one's latest phase
#pragma unroll 1
      for (int item = 0; item < n_items && ok; ++item) {
        const int nt = __shfl_sync(0xffffffffu, item_at(item).nt, 0);
        const uint32_t idesc = tm_idesc((nt + 15) & ~15);
        const int first_full = S::alt ? (item & 1) * S::nD : 0;
#pragma unroll 1
        for (int cc = 0; cc < nch; ++cc, ++c) {
          const uint32_t at = tmem + S::colA + as * kTmAStage;
          ok = tm_wait_three(b_tokf + 8 * xs, xph, b_dfree + 8 * ds, dph, b_af + 8 * as, aph, ab);  // an accumulator is free at
          if (!ok) break;                                                                          // once the first time round
          asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
          const uint32_t bt = tm_smem(tok) + xs * a.xstage;
          auto half = [&](uint32_t d, int h) {
#pragma unroll
            for (int g = 2 * h; g < 2 * h + 2; ++g) {
              const uint64_t bd = tm_desc128(bt + g * tn * 128);
#pragma unroll
              for (int k = 0; k < 4; ++k)
                tm_mma(d, at + g * 32 + k * 8, bd + 2 * k, idesc, k != 0 || (g & 1) != 0 || (h == 1 && SUM == kTmWhole));
            }
          };
          auto next = [&] {  // the ring's next accumulator
            const int full = first_full + ds;
            last = ((last ^ (used & (1u << full))) & (1u << full)) | (last & ~(1u << full));
            used |= 1u << full;
            if (++ds == S::nD) {
              ds = 0;
              dph ^= 1;
            }
          };
          if (SUM == kTmTurns) {
            if (tm_elect()) {
              half(tmem + ds * S::colD, 0);
              tm_commit(b_dfull + 8 * (first_full + ds));
            }
            __syncwarp();
            next();
            ok = tm_wait_warp(b_dfree + 8 * ds, dph, ab);
            if (!ok) break;
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
          }
          const uint32_t d = tmem + ds * S::colD, d2 = SUM == kTmSplit ? d + 16 * NB : d;
          if (tm_elect()) {
            if (SUM != kTmTurns) half(d, 0);
            half(d2, 1);
            if (!MX) {  // the sums' first two pieces, and their third
              const uint64_t bx = tm_desc64(bt + tn * 512);
              tm_mma(d2, at + 128, bx, idesc, true);
              tm_mma(d2, at + 128, bx + 2, idesc, true);
            }
            tm_commit(b_dfull + 8 * (first_full + ds));
            tm_commit(b_done + 8 * as);
            tm_commit(b_toke + 8 * xs);
          }
          __syncwarp();
          next();
          if (++as == S::nE) {
            as = 0;
            aph ^= 1;
          }
          if (++xs == rx) {
            xs = 0;
            xph ^= 1;
          }
        }
      }
      // MMAs in flight, and the arrivals they still owe
      for (int i = 0; i < 2 * S::nD; ++i)
        if ((used >> i) & 1) tm_wait(b_dfull + 8 * i, (last >> i) & 1, ab, true);
      for (int i = max(c - S::nE, 0); i < c; ++i) tm_wait(b_done + 8 * (i % S::nE), (i / S::nE) & 1, ab, true);
      for (int i = max(c - rx, 0); i < c; ++i) tm_wait(b_toke + 8 * (i % rx), (i / rx) & 1, ab, true);
    } else if (wid == 4 * S::nE + 9) {
      // ================================================================ the warp that copies packed weights
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
          const uint32_t bar = b_rawf + 8 * rs, to = tm_smem(raw + rs * kTmRawBytes);
          if (tm_elect()) {
            tm_expect(bar, kTmRawBytes);
#pragma unroll
            for (int m = 0; m < NMAT; ++m) tm_load_2d(to + m * (kTile * 128), &a.w[m], cc * 128, y, bar);
          }
          __syncwarp();
        }
      }
      for (int i = max(c - kTmRaw, 0); i < c; ++i) tm_wait(b_rawf + 8 * (i % kTmRaw), (i / kTmRaw) & 1, ab, true);
    } else if (wid == 4 * S::nE + 10) {
      // ================================================================ the warp that copies token tiles
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
          const uint32_t bar = b_tokf + 8 * xs, to = tm_smem(tok + xs * a.xstage);
          if (tm_elect()) {
            tm_expect(bar, nb * (MX ? 8192 : 8192 + 1024));
            for (int b = 0; b < nb; ++b) {
#pragma unroll
              for (int g = 0; g < 4; ++g)
                tm_load_2d(to + g * tn * 128 + b * 2048, &a.x, cc * kTmChunk + g * 64, it.p0 + 16 * b, bar);
              if (!MX) tm_load_2d(to + tn * 512 + b * 1024, &a.xb, cc * 32, it.p0 + 16 * b, bar);
            }
          }
          __syncwarp();
        }
      }
      for (int i = max(c - rx, 0); i < c; ++i) tm_wait(b_tokf + 8 * (i % rx), (i / rx) & 1, ab, true);
    }
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  if (abort_s) {  // a bounded wait ran out: the plan says so, and the CTA's results are NaN rather than whatever was there
    if (tid == 0) atomicExch(pv.hdr + 2, kPlanTimeout);
    for (int i = 0; i < n_items; ++i) {
      const TmItem it = item_at(i);
      for (int j = tid; j < it.nt * kTile; j += S::threads) {
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

template <bool MX, int R>
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
  uint4 keep[R];  // the thread's first R pieces; more are read twice
  uint32_t mx = 0;
  auto look = [&](const uint4& v) {
    const uint32_t q[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
    for (int k = 0; k < 4; ++k) mx = max(mx, max(q[k] & 0x7fffu, (q[k] >> 16) & 0x7fffu));
  };
#pragma unroll
  for (int j = 0; j < R; ++j) keep[j] = tid + j * kPrepThreads < nv ? xr[tid + j * kPrepThreads] : make_uint4(0u, 0u, 0u, 0u);
#pragma unroll
  for (int j = 0; j < R; ++j) look(keep[j]);
  for (int i = tid + R * kPrepThreads; i < nv; i += kPrepThreads) look(xr[i]);
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
  auto write = [&](int i, const uint4& v) {
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
  };
  // nv is a multiple of 32: a warp is whole or absent
#pragma unroll
  for (int j = 0; j < R; ++j)
    if (tid + j * kPrepThreads < nv) write(tid + j * kPrepThreads, keep[j]);
  for (int i = tid + R * kPrepThreads; i < nv; i += kPrepThreads) write(i, xr[i]);
}

// ------------------------------------------------------------------ host side

size_t qmm_tma_workspace(int rows, int K, bool mx) {
  const size_t row = mx ? (size_t)K * 2 : (size_t)K * 2 + K / 4;
  return (((size_t)rows * row + 255) & ~(size_t)255) + (size_t)rows * sizeof(float);
}

// Which calls gain from the path: whole chunks along K, and more than eight rows on some expert (by the caller's
// bound).  A block of up to eight token rows is taken by the one-launch kernel or the register-fed ones, whose cost per
// expert is the same for one row as for eight (whole block, called from Python: c2, T = 8 77 us in one launch, T = 9 81 here).
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
  auto kern = a.tn <= 16            ? qmm_tma_kernel<MX, NMAT, EPI, 1, kTmSplit>
              : a.tn <= kTmSplitTok ? qmm_tma_kernel<MX, NMAT, EPI, 3, kTmSplit>
                                    : qmm_tma_kernel<MX, NMAT, EPI, 6, MX ? kTmWhole : kTmTurns>;
  cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  const int threads = a.tn <= 16 ? TmShape<1, kTmSplit>::threads : TmShape<3, kTmSplit>::threads;
  if (e == cudaSuccess) e = launch_pdl(kern, dim3(grid), dim3(threads), smem, st, a);
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
  // While nearly all tasks fit 16 rows -- the average and two standard deviations of evenly routed rows -- the items do: the third
  // set of expanders is worth more than a weight tile read twice for the few larger ones (gate/up and down, us, blocks of 48 ->
  // 16: c5 T=150 1157/527 -> 941/497, c2 T=100 74/45 -> 71/42, mxfp4 c3 T=100 70/38 -> 62/36; an average of 12 to 14 is even).
  long long tn = 2ll * q.rows / max_groups + 8;
  const double avg = (double)q.rows / max_groups;
  if (avg < 16.0 && (16.0 - avg) * (16.0 - avg) >= 4.0 * avg) tn = 16;
  if (tn > rows_hint) tn = rows_hint;
  tn = (tn + 15) / 16 * 16;
  a.tn = tn > kTmMaxTok ? kTmMaxTok : (int)tn;
  a.xstage = (a.tn * (mx ? 512 : 576) + 1023) & ~1023;
  const int fixed = 1024 + kTmRaw * kTmRawBytes + kTmScRing * 128 * (a.tn <= 16 ? 3 : 2) * 16;
  const int room = 227 * 1024 - 14 * 1024 - fixed;  // 14 KB: the static part (prefix sums, items, barriers, row factors)
  a.rx = room / a.xstage > kTmMaxX ? kTmMaxX : room / a.xstage;
  const size_t smem = (size_t)fixed + (size_t)a.rx * a.xstage;
  int sms = 0, dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess ||
      cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || sms <= 0)
    return fail(ZMOE_ERR_CUDA, "%s: SM count query failed", who);
  // rows of up to 2048 (8192) values stay in registers between their largest value and their conversion
  auto prep = q.K <= 2048 ? (mx ? prep_rows_kernel<true, 2> : prep_rows_kernel<false, 2>)
                          : (mx ? prep_rows_kernel<true, 8> : prep_rows_kernel<false, 8>);
  cudaError_t e = launch_pdl(prep, dim3(q.rows), dim3(kPrepThreads), 0, st, q.x, q.ldx, q.plan, q.rows, q.E, q.x_by_dst, q.K,
                             (__half*)xs, xinv);
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
