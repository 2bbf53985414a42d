// Building blocks of the kernels that give a probe to a cluster of CTAs: eight
// compute warps, a copy warp, shared-memory rings filled by bulk copies, and sums
// met over distributed shared memory (arnoldi_cluster.cu, gs_cluster.cu).
#pragma once

#include "common.cuh"

namespace mfg {

constexpr int kCWarps = 8;             // compute warps
constexpr int kCThreads = 32 * kCWarps;
constexpr int kCRows = 256;            // rows of a warp: 8 per lane
constexpr int kCMaxSlots = 32;
constexpr int kCMaxS = 16;
constexpr size_t kCSmem = 112 * 1024;  // dynamic shared memory of a CTA: two per SM
constexpr int kCMaxR = kCRows * kCWarps;

__device__ __forceinline__ uint32_t c_smem(const void *p) { return (uint32_t)__cvta_generic_to_shared(p); }

__device__ __forceinline__ uint32_t c_rank() {
  uint32_t r;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return r;
}

__device__ __forceinline__ uint32_t c_map(uint32_t saddr, uint32_t rank) {
  uint32_t r;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(saddr), "r"(rank));
  return r;
}

__device__ __forceinline__ double c_ld_f64(uint32_t addr) {
  double v;
  asm volatile("ld.shared::cluster.f64 %0, [%1];" : "=d"(v) : "r"(addr) : "memory");
  return v;
}

// from L2, in program order with the waits
__device__ __forceinline__ float4 c_ld_l2(const float *p) {
  float4 v;
  asm volatile("ld.global.cg.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "l"(p) : "memory");
  return v;
}

__device__ __forceinline__ void c_bulk(uint32_t dst, const void *src, uint32_t bytes, uint64_t *bar) {
  asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(dst),
               "l"(reinterpret_cast<uint64_t>(src)), "r"(bytes), "r"(c_smem(bar))
               : "memory");
}

__device__ __forceinline__ void c_expect(uint64_t *bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(c_smem(bar)), "r"(bytes) : "memory");
}

__device__ __forceinline__ void c_arrive(uint64_t *bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(c_smem(bar)) : "memory");
}

// the compute warps' barrier; the warp is converged on both sides
__device__ __forceinline__ void c_sync() {
  __syncwarp();
  asm volatile("barrier.sync 1, %0;" ::"n"(kCThreads) : "memory");
  __syncwarp();
}

// Arrival without a release: for a barrier that orders no data
__device__ __forceinline__ void c_cluster_arrive_relaxed() {
  __syncwarp();
  asm volatile("barrier.cluster.arrive.relaxed;" ::: "memory");
}

__device__ __forceinline__ void c_cluster_arrive() {
  __syncwarp();
  asm volatile("barrier.cluster.arrive.release;" ::: "memory");
}
__device__ __forceinline__ void c_cluster_wait() {
  asm volatile("barrier.cluster.wait.acquire;" ::: "memory");
  __syncwarp();
}

// The end of a CTA's work, by every warp: the cluster's CTAs have read each other's sums, and
// every role of this CTA is done.
__device__ __forceinline__ void c_done(int S) {
  if (S > 1) {
    c_cluster_arrive_relaxed();
    c_cluster_wait();
  } else {
    __syncwarp();
    asm volatile("barrier.sync 2, %0;" ::"n"(kCThreads + 32) : "memory");
  }
}

// s + e += x, exactly up to the rounding of e
__device__ __forceinline__ void two_add(float &s, float &e, float x) {
  const float t = s + x, z = t - s;
  e += (s - (t - z)) + (x - z);
  s = t;
}

// Two-float numbers x + y, |y| <= half an ulp of x: some 2^-45 of relative error per
// operation, in a few float instructions of 4 cycles each.  A float64 instruction holds
// its warp for 64 cycles here, a dependent chain of them (or one division or root)
// for thousands, on the path of every step.
__device__ __forceinline__ float2 pair(float s, float e) {
  const float t = s + e;
  return make_float2(t, e - (t - s));
}

__device__ __forceinline__ float2 pair_add(float2 a, float2 b) {
  two_add(a.x, a.y, b.x);
  return pair(a.x, a.y + b.y);
}

__device__ __forceinline__ float2 pair_neg(float2 a) { return make_float2(-a.x, -a.y); }

__device__ __forceinline__ float2 pair_mul(float2 a, float2 b) {
  const float p = a.x * b.x;
  return pair(p, fmaf(a.y, b.x, fmaf(a.x, b.y, fmaf(a.x, b.x, -p))));
}

// 1 / sqrt(a): a Newton step on the float result
__device__ __forceinline__ float2 pair_rsqrt(float2 a) {
  const float r = rsqrtf(a.x), r2 = r * r;
  const float t = fmaf(-a.y, r2, fmaf(-a.x, fmaf(r, r, -r2), fmaf(-a.x, r2, 1.0f)));
  return pair(r, 0.5f * r * t);
}

__device__ __forceinline__ float2 pair_shfl_xor(float2 a, int o) {
  return make_float2(__shfl_xor_sync(0xffffffffu, a.x, o), __shfl_xor_sync(0xffffffffu, a.y, o));
}

__device__ __forceinline__ float2 c_ld_pair(uint32_t addr) {
  float2 v;
  asm volatile("ld.shared::cluster.v2.f32 {%0, %1}, [%2];" : "=f"(v.x), "=f"(v.y) : "r"(addr) : "memory");
  return v;
}

// Sum of the lanes' two-float values (all lanes).
__device__ __forceinline__ float2 warp_pair(float s, float e) {
  float2 v = make_float2(s, e);
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    const float2 u = pair_shfl_xor(v, o);
    two_add(v.x, v.y, u.x);
    v.y += u.y;
  }
  return pair(v.x, v.y);
}

// Halving butterfly: N per-lane values to their warp sums; lane l ends with the
// sum of value idx(l), kept by the lanes of equal idx (32 / N of them).
template <int N, typename T>
__device__ __forceinline__ T c_xsum(T (&v)[N], int lane, int &idx) {
  idx = 0;
#pragma unroll
  for (int s = 0; s < 5; ++s) {
    const int o = 16 >> s, half = N >> (s + 1);
    if (half >= 1) {
      const bool up = (lane & o) != 0;
#pragma unroll
      for (int i = 0; i < half; ++i) {
        const T send = up ? v[i] : v[i + half], keep = up ? v[i + half] : v[i];
        v[i] = keep + __shfl_xor_sync(0xffffffffu, send, o);
      }
      if (up) idx += half;
    } else {
      v[0] += __shfl_xor_sync(0xffffffffu, v[0], o);
    }
  }
  return v[0];
}

// Bounded wait of a whole warp (warp-uniform result) for the phase of `bar` with
// the given parity: false, with the flag and the status raised, after the limit
// or another warp's failure.  kCluster: acquires what other CTAs wrote.
template <bool kCluster = false>
__device__ __forceinline__ bool c_wait(uint64_t *bar, uint32_t parity, volatile int *fail, int *status) {
  const uint32_t at = c_smem(bar);
  uint64_t t0 = 0;
  for (uint32_t it = 0;; ++it) {
    uint32_t ok;
    if constexpr (kCluster)
      asm volatile(
          "{\n\t.reg .pred p;\n\t"
          "mbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2;\n\t"
          "selp.u32 %0, 1, 0, p;\n\t}\n"
          : "=r"(ok)
          : "r"(at), "r"(parity)
          : "memory");
    else
      ok = mbar_try_wait_parity<false>(at, parity);
    if (__all_sync(0xffffffffu, ok)) return true;
    if ((it & 63u) == 0) {
      const uint64_t now = global_ns();
      if (it == 0) t0 = now;
      if (__any_sync(0xffffffffu, *fail != 0 || now - t0 > kMbarWaitNs)) break;
    }
  }
  if ((threadIdx.x & 31) == 0 && !*fail) {
    *fail = 1;
    if (status) atomicExch(status, (int)MFG_ERR_TIMEOUT);
  }
  __syncwarp();
  return false;
}

// This CTA has reached a meeting point of the cluster: its shared-memory writes
// before it (all warps', after a c_sync()) are released to every CTA.
__device__ __forceinline__ void c_meet_arrive(uint64_t *bar, int S) {
  if (S > 1 && (int)threadIdx.x < S)
    asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];" ::"r"(c_map(c_smem(bar), threadIdx.x))
                 : "memory");
  __syncwarp();
}

// CTAs per probe to choose from
constexpr int kCSizes = 9;
constexpr int kCSize[kCSizes] = {1, 2, 4, 6, 8, 10, 12, 14, 16};

// first distance of a butterfly over the ranks (lanes past the last hold zero)
__device__ __forceinline__ int c_half(int S) { return S > 8 ? 8 : (S > 4 ? 4 : S / 2); }

// Row warps for R rows of a CTA, and the clusters of each size that the GPU holds at a time for a kernel of kCThreads + 32 threads and kCSmem bytes.
inline int c_row_warps(int64_t R) { return R <= kCRows ? 1 : (R <= 2 * kCRows ? 2 : (R <= 4 * kCRows ? 4 : 8)); }

template <typename K>
inline bool c_prepare(K kern) {
  return cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kCSmem) == cudaSuccess &&
         cudaFuncSetAttribute(kern, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) == cudaSuccess;
}

// Clusters that the current device holds at a time, per log2 of the row warps and size
// (0: that size does not run there).
struct CSlots {
  int clusters[4][kCSizes];
};

// False if the kernel could not be prepared or asked about for another reason than a cluster size.
template <typename K>
inline bool c_count_clusters(K kern, int (&clusters)[kCSizes]) {
  bool ok = c_prepare(kern);
  for (int i = 0; i < kCSizes && ok; ++i) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(64u * kCSize[i]);
    cfg.blockDim = dim3(kCThreads + 32);
    cfg.dynamicSmemBytes = kCSmem;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = (unsigned)kCSize[i];
    attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    int c = 0;
    const cudaError_t e = cudaOccupancyMaxActiveClusters(&c, kern, &cfg);
    if (e != cudaSuccess) c = 0;
    ok = e == cudaSuccess || e == cudaErrorInvalidClusterSize || e == cudaErrorInvalidConfiguration;
    clusters[i] = c;
  }
  (void)cudaGetLastError();
  return ok;
}

// Larger clusters are not chained: placed on SMs as these come free they no longer all
// fit at once (n = 16384, k = 64, 256 probes, S = 8: 29.0 -> 35.2 ms per solve; S = 4 at n =
// 8192, 128 probes, k = 48: 17.4 -> 17.0).
constexpr int kCChainS = 4;
constexpr double kCUnchainedUs = 2.7;  // a step whose launch is not chained, in the plans' costs

template <typename K, typename A>
inline int c_launch(K kern, int S, int64_t ctas, size_t smem, const A &args, bool chained, cudaStream_t s) {
  MFG_CUDA_TRY(launch_kernel(kern, dim3((unsigned)ctas), kCThreads + 32, smem, (unsigned)S, chained && S <= kCChainS, s,
                             args));
  return MFG_LAUNCH_STATUS();
}

}  // namespace mfg
