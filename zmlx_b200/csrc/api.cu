// Error state, ABI version and the token-sorted expert plan.
#include <cstring>

#include "common.cuh"
#include "plan.cuh"

namespace zmoe {

static thread_local char g_err[512] = "";

void set_error(const char* fmt, ...) {
  va_list ap;
  va_start(ap, fmt);
  vsnprintf(g_err, sizeof(g_err), fmt, ap);
  va_end(ap);
}

int fail(int code, const char* fmt, ...) {
  va_list ap;
  va_start(ap, fmt);
  vsnprintf(g_err, sizeof(g_err), fmt, ap);
  va_end(ap);
  return code;
}

int check_launch(const char* what) {
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) return fail(ZMOE_ERR_CUDA, "%s: %s", what, cudaGetErrorString(e));
  return ZMOE_OK;
}

// The plan as a launch of its own: C CTAs, one cluster, each of which counts, and later places, its share of the pairs.  The
// counts are exchanged through distributed shared memory, every CTA scans the totals for itself.  What bounds it is the chain
// of dependent steps.  us, top-8 of 128, one CTA that scanned through shared memory -> now: 32768 pairs 40.7 -> 12.1, 12000
// pairs 17.0 -> 9.8, 4096 pairs (of 256) 8.3 -> 6.4 in one CTA, whose four pairs a thread cost less than a cluster's barriers.
// The order of rows inside an expert's segment is arbitrary, see build_plan_block.
__device__ __forceinline__ void plan_cluster_arrive() { asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory"); }
__device__ __forceinline__ void plan_cluster_wait() { asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory"); }
// A word of CTA `cta`'s shared memory, at the place where this CTA has `p`.
__device__ __forceinline__ int plan_peer(const int* p, int cta) {
  uint32_t addr;
  int v;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(addr) : "r"((uint32_t)__cvta_generic_to_shared(p)), "r"(cta));
  asm volatile("ld.shared::cluster.u32 %0, [%1];" : "=r"(v) : "r"(addr) : "memory");
  return v;
}

constexpr int kPlanThreads = 1024, kPlanCtas = 8;
constexpr int kPlanMaxE = 4096;

template <int C>
__global__ void __launch_bounds__(kPlanThreads) build_plan_kernel(const int* lhs, int lhs_div, const int* rhs, int P, int M,
                                                                  int E, int* plan_base) {
  extern __shared__ int sm[];  // counts (read by the other CTAs) and cursors, E each
  __shared__ unsigned long long warp_tot[kPlanThreads / 32];
  __shared__ int bad_s;
  pdl_wait();
  pdl_trigger();
  int *count = sm, *cursor = sm + E;
  const int rows = P * M, tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
  const int cta = C > 1 ? blockIdx.x : 0;  // the grid is one cluster
  PlanView pv = plan_view(plan_base, rows, E);
  bool timed_out = false;  // of this plan's previous build: kept
  if (tid == 0) {
    bad_s = 0;
    timed_out = cta == 0 && pv.hdr[2] == kPlanTimeout && pv.hdr[1] == rows && pv.hdr[3] == E;
  }
  for (int e = tid; e < E; e += kPlanThreads) count[e] = 0;
  __syncthreads();
  const int p0 = (int)((long long)P * cta / C), p1 = (int)((long long)P * (cta + 1) / C);
  for (int p = p0 + tid; p < p1; p += kPlanThreads) {
    const int e = rhs[p];
    if (e >= 0 && e < E)
      atomicAdd(&count[e], 1);
    else
      bad_s = 1;
  }
  if (C > 1) {
    plan_cluster_arrive();
    plan_cluster_wait();
  } else {
    __syncthreads();
  }
  int bad = 0;
  constexpr int kPer = kPlanMaxE / kPlanThreads;  // consecutive experts of a thread
  // per expert: rows in the low half, and in the high half whether there are any; before: what lower CTAs have of it
  unsigned long long v[kPer], mine = 0;
  int before[kPer];
#pragma unroll
  for (int i = 0; i < kPer; ++i) {
    const int e = tid * kPer + i;
    int sum = 0;
    before[i] = 0;
    if (e < E)
#pragma unroll
      for (int c = 0; c < C; ++c) {
        const int n = C > 1 ? plan_peer(&count[e], c) : count[e];
        if (c < cta) before[i] += n;
        sum += n;
      }
    v[i] = (unsigned long long)((unsigned)sum * (unsigned)M) | ((unsigned long long)(sum > 0) << 32);
    mine += v[i];
  }
  if (tid == 0 && cta == 0)
    for (int c = 0; c < C; ++c) bad |= C > 1 ? plan_peer(&bad_s, c) : bad_s;
  if (C > 1) plan_cluster_arrive();  // this CTA has read what it needs of the others; it may leave once all have (the wait at the end)
  // exclusive scan of both halves at once
  unsigned long long incl = mine;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const unsigned long long u = __shfl_up_sync(0xffffffffu, incl, o);
    if (lane >= o) incl += u;
  }
  if (lane == 31) warp_tot[wid] = incl;
  __syncthreads();
  unsigned long long base = 0, all = 0;
  for (int w = 0; w < kPlanThreads / 32; ++w) {
    if (w < wid) base += warp_tot[w];
    all += warp_tot[w];
  }
  unsigned long long run = base + incl - mine;
#pragma unroll
  for (int i = 0; i < kPer; ++i) {
    const int e = tid * kPer + i;
    if (e < E) {
      const int off = (int)(run & 0xFFFFFFFFull), a = (int)(run >> 32), c = (int)(v[i] & 0xFFFFFFFFull);
      cursor[e] = off + before[i] * M;
      if (cta == 0) {
        pv.offset[e] = off;
        if (c > 0) {
          pv.active[a] = e;
          reinterpret_cast<int4*>(pv.tasks)[a] = make_int4(e, off, c, 0);
        }
      }
    }
    run += v[i];
  }
  const int active = (int)(all >> 32);
  if (cta == 0) {
    for (int a = active + tid; a < E; a += kPlanThreads) reinterpret_cast<int4*>(pv.tasks)[a] = make_int4(0, 0, 0, 0);
    if (tid == 0) {
      pv.offset[E] = (int)(all & 0xFFFFFFFFull);
      pv.hdr[0] = active;
      pv.hdr[1] = rows;
      pv.hdr[2] = timed_out ? kPlanTimeout : bad;
      pv.hdr[3] = E;
    }
  }
  __syncthreads();
  for (int p = p0 + tid; p < p1; p += kPlanThreads) {
    const int e = rhs[p];
    if (e < 0 || e >= E) continue;
    const int pos = atomicAdd(&cursor[e], M);
    const int src = (lhs ? lhs[p] : p / lhs_div) * M;
    for (int m = 0; m < M; ++m) {
      pv.row_src[pos + m] = src + m;
      pv.row_dst[pos + m] = p * M + m;
    }
  }
  if (C > 1) plan_cluster_wait();  // nobody reads this CTA's counts any more
}

}  // namespace zmoe

using namespace zmoe;

extern "C" {

int zmoe_abi_version(void) { return ZMOE_ABI_VERSION; }

const char* zmoe_last_error(void) { return g_err; }

size_t zmoe_plan_bytes(int rows, int E) {
  if (rows < 0 || E <= 0) return 0;
  return plan_words(rows, E) * sizeof(int);
}

int zmoe_ep_alloc(size_t bytes, void** ptr) {
  ZMOE_REQUIRE(ptr != nullptr && bytes > 0, ZMOE_ERR_SHAPE, "zmoe_ep_alloc: bad arguments");
  cudaError_t e = cudaMalloc(ptr, bytes);
  if (e == cudaSuccess) e = cudaMemset(*ptr, 0, bytes);
  if (e == cudaSuccess) e = cudaDeviceSynchronize();
  if (e != cudaSuccess) return fail(ZMOE_ERR_CUDA, "zmoe_ep_alloc: %s", cudaGetErrorString(e));
  return ZMOE_OK;
}

int zmoe_ep_free(void* ptr) {
  cudaError_t e = cudaFree(ptr);
  if (e != cudaSuccess) return fail(ZMOE_ERR_CUDA, "zmoe_ep_free: %s", cudaGetErrorString(e));
  return ZMOE_OK;
}

int zmoe_ep_export(const void* ptr, void* handle64) {
  static_assert(sizeof(cudaIpcMemHandle_t) == 64, "the handle is 64 bytes");
  ZMOE_REQUIRE(ptr != nullptr && handle64 != nullptr, ZMOE_ERR_SHAPE, "zmoe_ep_export: null pointer");
  cudaError_t e = cudaIpcGetMemHandle(reinterpret_cast<cudaIpcMemHandle_t*>(handle64), const_cast<void*>(ptr));
  if (e != cudaSuccess) return fail(ZMOE_ERR_CUDA, "zmoe_ep_export: %s", cudaGetErrorString(e));
  return ZMOE_OK;
}

int zmoe_ep_import(const void* handle64, void** ptr) {
  ZMOE_REQUIRE(ptr != nullptr && handle64 != nullptr, ZMOE_ERR_SHAPE, "zmoe_ep_import: null pointer");
  cudaIpcMemHandle_t h;
  memcpy(&h, handle64, sizeof(h));
  cudaError_t e = cudaIpcOpenMemHandle(ptr, h, cudaIpcMemLazyEnablePeerAccess);
  if (e != cudaSuccess) return fail(ZMOE_ERR_CUDA, "zmoe_ep_import: %s", cudaGetErrorString(e));
  return ZMOE_OK;
}

int zmoe_ep_unmap(void* ptr) {
  cudaError_t e = cudaIpcCloseMemHandle(ptr);
  if (e != cudaSuccess) return fail(ZMOE_ERR_CUDA, "zmoe_ep_unmap: %s", cudaGetErrorString(e));
  return ZMOE_OK;
}

int zmoe_build_plan(const int32_t* lhs, int lhs_div, const int32_t* rhs, int P, int M, int E, void* plan,
                    size_t plan_bytes, void* stream) {
  ZMOE_REQUIRE(rhs != nullptr && plan != nullptr, ZMOE_ERR_SHAPE, "zmoe_build_plan: null pointer");
  ZMOE_REQUIRE(P >= 0 && M >= 1 && E >= 1, ZMOE_ERR_SHAPE, "zmoe_build_plan: bad sizes P=%d M=%d E=%d", P, M, E);
  ZMOE_REQUIRE(E <= 4096, ZMOE_ERR_UNSUPPORTED, "zmoe_build_plan: E=%d exceeds 4096", E);
  ZMOE_REQUIRE(lhs != nullptr || lhs_div >= 1, ZMOE_ERR_SHAPE, "zmoe_build_plan: lhs_div must be >= 1");
  ZMOE_REQUIRE((long long)P * M < (1ll << 24), ZMOE_ERR_SHAPE, "zmoe_build_plan: too many rows (limit 2^24)");
  ZMOE_REQUIRE(plan_bytes >= zmoe_plan_bytes(P * M, E), ZMOE_ERR_WORKSPACE,
               "zmoe_build_plan: plan buffer of %zu bytes, need %zu", plan_bytes, zmoe_plan_bytes(P * M, E));
  static_assert(kPlanMaxE % kPlanThreads == 0, "whole threads");
  const size_t smem = 2 * (size_t)E * sizeof(int);
  cudaError_t e;
  if (P <= 4 * kPlanThreads) {
    e = launch_pdl(build_plan_kernel<1>, dim3(1), dim3(kPlanThreads), smem, (cudaStream_t)stream, (const int*)lhs, lhs_div,
                   (const int*)rhs, P, M, E, (int*)plan);
  } else {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(kPlanCtas);
    cfg.blockDim = dim3(kPlanThreads);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = (cudaStream_t)stream;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    attr[1].id = cudaLaunchAttributeClusterDimension;
    attr[1].val.clusterDim.x = kPlanCtas;
    attr[1].val.clusterDim.y = attr[1].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 2;
    e = cudaLaunchKernelEx(&cfg, build_plan_kernel<kPlanCtas>, (const int*)lhs, lhs_div, (const int*)rhs, P, M, E, (int*)plan);
  }
  if (e != cudaSuccess) return fail(ZMOE_ERR_CUDA, "zmoe_build_plan: launch failed: %s", cudaGetErrorString(e));
  return check_launch("zmoe_build_plan");
}

int zmoe_plan_status(const void* plan, int clear, void* stream) {
  ZMOE_REQUIRE(plan != nullptr, ZMOE_ERR_SHAPE, "zmoe_plan_status: null plan");
  cudaStream_t st = (cudaStream_t)stream;
  int word = 0;
  int* dev = (int*)plan + 2;
  cudaError_t e = cudaMemcpyAsync(&word, dev, sizeof(int), cudaMemcpyDeviceToHost, st);
  if (e == cudaSuccess) e = cudaStreamSynchronize(st);
  if (e == cudaSuccess && word == kPlanTimeout && clear) e = cudaMemsetAsync(dev, 0, sizeof(int), st);
  if (e != cudaSuccess) return fail(ZMOE_ERR_CUDA, "zmoe_plan_status: %s", cudaGetErrorString(e));
  if (word != kPlanTimeout) return ZMOE_OK;
  return fail(ZMOE_ERR_TIMEOUT, "zmoe_plan_status: a bounded wait of a grouped matmul ran out; its output is NaN or void");
}

}  // extern "C"
