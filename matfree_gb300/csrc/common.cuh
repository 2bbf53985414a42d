// Shared helpers of the matfree_gb300 CUDA library (sm_103a).
#pragma once

#include <cuda_runtime.h>
#include <cuda_bf16.h>
#include <stdint.h>
#include <stddef.h>

#include "../../include/matfree_gb300.h"
#include "per_device.cuh"

namespace mfg {
// Records the call site and CUDA error text of the most recent failure on
// this host thread (read back through mfg_last_error()).
void record_error(const char *where, int line, const char *what);
inline int cuda_status(cudaError_t e, const char *where, int line) {
  if (e == cudaSuccess) return MFG_OK;
  record_error(where, line, cudaGetErrorString(e));
  return MFG_ERR_CUDA;
}
}  // namespace mfg

#define MFG_CUDA_TRY(expr)                                                  \
  do {                                                                      \
    const int _s = ::mfg::cuda_status((expr), __FILE__, __LINE__);          \
    if (_s != MFG_OK) return _s;                                            \
  } while (0)

// status of the kernel launch just issued (configuration errors, and sticky
// errors of earlier kernels on the device)
#define MFG_LAUNCH_STATUS() ::mfg::cuda_status(cudaGetLastError(), __FILE__, __LINE__)

#define MFG_TRY(expr)                                       \
  do {                                                      \
    int _s = (expr);                                        \
    if (_s != MFG_OK) return _s;                            \
  } while (0)

namespace mfg {

constexpr int kThreads = 256;  // threads per CTA of the streaming kernels
constexpr int kWarps = kThreads / 32;

inline cudaStream_t as_stream(void *s) { return reinterpret_cast<cudaStream_t>(s); }

inline int64_t ceil_div(int64_t a, int64_t b) { return (a + b - 1) / b; }

inline int current_device() {
  int dev = 0;
  return cudaGetDevice(&dev) == cudaSuccess ? dev : -1;
}

// Multiprocessors of the current device (152 where it cannot be asked).
inline int sm_count() {
  static PerDevice<int> counts;
  const int dev = current_device();
  const int *sms = counts.get(dev, [&](int &n) {
    return cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev) == cudaSuccess && n > 0;
  });
  return sms ? *sms : 152;
}

// ---------------------------------------------------------------------------
// mbarrier waits, bounded in wall-clock time (%globaltimer) and given up
// early when another role raised the CTA's failure flag.  Waits on the
// critical path poll mbarrier.try_wait; waits of idle roles (an epilogue
// waiting for the whole main loop) sleep in it with a suspend-time hint, so
// they take no issue slots from the warps doing the work.
// ---------------------------------------------------------------------------

constexpr uint64_t kMbarWaitNs = 2000000000ull;  // 2 s: far beyond any copy or MMA
constexpr uint32_t kMbarSleepNs = 1000000u;      // per sleeping try_wait

__device__ __forceinline__ uint64_t global_ns() {
  uint64_t t;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
  return t;
}

template <bool kSleep>
__device__ __forceinline__ bool mbar_try_wait_parity(uint32_t bar_saddr, uint32_t parity) {
  uint32_t ok;
  if constexpr (kSleep) {
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2, %3;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}\n"
        : "=r"(ok)
        : "r"(bar_saddr), "r"(parity), "r"(kMbarSleepNs)
        : "memory");
  } else {
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}\n"
        : "=r"(ok)
        : "r"(bar_saddr), "r"(parity)
        : "memory");
  }
  return ok != 0;
}

// True once the phase of the barrier at shared address `bar_saddr` with the
// given parity has completed; false after `limit_ns` or when *fail (if given)
// becomes non-zero.
template <bool kSleep = false>
__device__ __forceinline__ bool mbar_wait_bounded(uint32_t bar_saddr, uint32_t parity,
                                                  volatile int *fail,
                                                  uint64_t limit_ns = kMbarWaitNs) {
  if (mbar_try_wait_parity<kSleep>(bar_saddr, parity)) return true;
  const uint64_t t0 = global_ns();
  for (uint32_t it = 1;; ++it) {
    if (mbar_try_wait_parity<kSleep>(bar_saddr, parity)) return true;
    if (kSleep || (it & 63u) == 0) {
      if (fail && *fail) return false;
      if (global_ns() - t0 > limit_ns) return false;
    }
  }
}

// ---------------------------------------------------------------------------
// Chained launches: inside a solve's loop a kernel may be launched while the one
// before it on the stream still runs (programmatic stream serialization), so that
// its launch, barrier set-up, TMEM allocation and first operator reads overlap that
// kernel's end.  Every thread calls chain_wait() before it touches memory that an
// earlier kernel of the loop reads or writes: it returns once the kernel before
// has completed and its writes are visible.  chain_next() afterwards lets the kernel
// after it start, so at most two kernels of a chain are resident, and all that came
// before the first of them has completed.  Only the operator, which no kernel of the
// loop writes, may be read before chain_wait(): the loop's first kernels are ordinary
// launches, behind whatever wrote the operator.
//
// What an earlier kernel of the loop wrote is not read-only while this one runs: it is read
// by plain or volatile loads through pointers without __restrict__ (which would let the
// compiler use the non-coherent path or move a load above the wait), never by __ldg.
//
// Two to three microseconds a launch: figures at chain_ok (capi.cu).
// ---------------------------------------------------------------------------

__device__ __forceinline__ void chain_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void chain_next() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }

// A launch on `s`, as clusters of `cluster` CTAs along x (0: the kernel's own) and
// chained to the kernel before it if asked.
template <typename... P, typename... A>
inline cudaError_t launch_kernel(void (*kern)(P...), dim3 grid, unsigned threads, size_t smem, unsigned cluster,
                                 bool chained, cudaStream_t s, A &&...args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = dim3(threads);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = s;
  cudaLaunchAttribute attr[2];
  unsigned na = 0;
  if (cluster) {
    attr[na].id = cudaLaunchAttributeClusterDimension;
    attr[na].val.clusterDim.x = cluster;
    attr[na].val.clusterDim.y = attr[na].val.clusterDim.z = 1;
    ++na;
  }
  if (chained) {
    attr[na].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[na].val.programmaticStreamSerializationAllowed = 1;
    ++na;
  }
  cfg.attrs = attr;
  cfg.numAttrs = na;
  return cudaLaunchKernelEx(&cfg, kern, static_cast<P>(args)...);
}

inline size_t align_up(size_t x, size_t a) { return (x + a - 1) / a * a; }

// 16-byte vector type per element type: 4 floats or 2 doubles.
template <typename T> struct Vec;
template <> struct Vec<float> {
  using type = float4;
  static constexpr int width = 4;
};
template <> struct Vec<double> {
  using type = double2;
  static constexpr int width = 2;
};

template <typename T>
__device__ __forceinline__ void vec_to_array(const typename Vec<T>::type &v, T *a);
template <>
__device__ __forceinline__ void vec_to_array<float>(const float4 &v, float *a) {
  a[0] = v.x; a[1] = v.y; a[2] = v.z; a[3] = v.w;
}
template <>
__device__ __forceinline__ void vec_to_array<double>(const double2 &v, double *a) {
  a[0] = v.x; a[1] = v.y;
}
template <typename T>
__device__ __forceinline__ typename Vec<T>::type array_to_vec(const T *a);
template <>
__device__ __forceinline__ float4 array_to_vec<float>(const float *a) {
  return make_float4(a[0], a[1], a[2], a[3]);
}
template <>
__device__ __forceinline__ double2 array_to_vec<double>(const double *a) {
  return make_double2(a[0], a[1]);
}

// Accumulator type of the per-thread partial sums: float32 for float data
// (combined in float64 across threads), float64 for double data.
template <typename T> struct Acc { using type = T; };

__device__ __forceinline__ double warp_sum(double v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

}  // namespace mfg
