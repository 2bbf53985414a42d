// Operator kernels: dense W = A V in float32 / float64, CSR
// SpMM, and builders of the dense RBF kernel matrix and its bf16 split.
#include "common.cuh"
#include "kernels.cuh"

namespace mfg {

// ---------------------------------------------------------------------------
// Dense W[b][m] = sum_k A[m][k] V[b][k] + shift V[b][m] in float32 (FMA pipes)
// and float64 (m8n8k4 MMAs).
//
// A CTA forms a tile of BM rows x BP probes over one of S equal ranges of K, a
// cluster of S CTAs covers K and adds its partial tiles over distributed shared
// memory in rank order (small operators have too few tiles for the GPU; n = 2000,
// 64 probes: 32 tiles).  Both operands are K-major; slices of BK columns go to
// shared memory as they are (cp.async, three stages, rows padded by 16 bytes so
// that 16-byte reads of neighbouring rows fall into different banks).
// ---------------------------------------------------------------------------

constexpr int kDStages = 3;
constexpr int kDMaxS = 8;

__device__ __forceinline__ uint32_t d_smem(const void *p) { return (uint32_t)__cvta_generic_to_shared(p); }

// 16 bytes to shared memory, the first `bytes` of them from global memory, the rest zero
__device__ __forceinline__ void cp_async16(void *dst, const void *src, int bytes) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(d_smem(dst)), "l"(src), "r"(bytes) : "memory");
}

__device__ __forceinline__ void d_cluster_sync() {
  __syncthreads();
  asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
  asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
}

template <typename T>
__device__ __forceinline__ T d_load_rank(const T *local, int rank) {
  uint32_t at;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(at) : "r"(d_smem(local)), "r"(rank));
  T v;
  if constexpr (sizeof(T) == 4)
    asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(v) : "r"(at) : "memory");
  else
    asm volatile("ld.shared::cluster.f64 %0, [%1];" : "=d"(v) : "r"(at) : "memory");
  return v;
}

// Slices [kb, ke) of BK columns of A's rows m0.. and V's probes b0.. through the
// stages; body(As, Vs) consumes one.  Columns past n, rows past n and probes past
// p read as zero.  A thread copies the same 16-byte column of kPer rows in every slice, by
// pointers that only advance (index arithmetic per copy cost as much as a slice's FMAs).
template <typename T, int BM, int BP, int BK, int THREADS, typename F>
__device__ __forceinline__ void d_pipeline(T *stages, const T *__restrict__ A, int64_t lda, const T *__restrict__ V,
                                           int64_t ldv, int64_t n, int64_t p, int64_t m0, int64_t b0, int64_t kb,
                                           int64_t ke, F body) {
  constexpr int VW = Vec<T>::width, LD = BK + VW, PER = BK / VW, kStage = (BM + BP) * LD;
  constexpr int kRowStep = THREADS / PER, kPer = (BM + BP + kRowStep - 1) / kRowStep;
  static_assert(THREADS % PER == 0, "a thread's column");
  const int row = threadIdx.x / PER, c = threadIdx.x % PER * VW;
  const T *src[kPer];
  bool live[kPer];
#pragma unroll
  for (int q = 0; q < kPer; ++q) {
    const int r = row + q * kRowStep;
    const bool isA = r < BM;
    const int64_t at = isA ? m0 + r : b0 + (r - BM);
    live[q] = r < BM + BP && at < (isA ? n : p);
    src[q] = live[q] ? (isA ? A + at * lda : V + at * ldv) + kb * BK + c : A;
  }
  int left = (int)(ke - kb), fill = 0;                  // slices to load; the stage they go to
  int64_t cols = n - kb * BK - c;                       // columns left at this thread's
  auto load = [&]() {
    if (left > 0) {
      T *st = stages + fill * kStage + row * LD + c;
      const int bytes = cols >= VW ? 16 : (cols > 0 ? (int)cols * (int)sizeof(T) : 0);
#pragma unroll
      for (int q = 0; q < kPer; ++q) {
        if (row + q * kRowStep < BM + BP)
          cp_async16(st + q * kRowStep * LD, live[q] && bytes ? src[q] : A, live[q] ? bytes : 0);
        src[q] += live[q] ? BK : 0;
      }
      cols -= BK;
      --left;
      if (++fill == kDStages) fill = 0;
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
#pragma unroll
  for (int s = 0; s < kDStages - 1; ++s) load();
  int use = 0;
  for (int slices = (int)(ke - kb); slices > 0; --slices) {
    asm volatile("cp.async.wait_group %0;" ::"n"(kDStages - 2) : "memory");
    __syncthreads();  // this slice has landed, and the stage loaded next is no longer read
    load();
    const T *st = stages + use * kStage;
    body(st, st + BM * LD);
    if (++use == kDStages) use = 0;
  }
  asm volatile("cp.async.wait_group 0;" ::: "memory");
  __syncthreads();
}

// The cluster's partial tiles part[BP][BM] (probes PITCH apart) into W, this CTA's
// share of the probes.
template <typename T, int BM, int BP, int PITCH, int THREADS>
__device__ __forceinline__ void d_reduce_store(const T *part, const T *__restrict__ V, int64_t ldv, T *__restrict__ W,
                                               int64_t ldw, int64_t n, int64_t p, int64_t m0, int64_t b0, int rank,
                                               int S, T shift) {
  d_cluster_sync();
  const int c0 = BP * rank / S, c1 = BP * (rank + 1) / S;
  for (int i = threadIdx.x; i < (c1 - c0) * BM; i += THREADS) {
    const int c = c0 + i / BM, r = i % BM;
    const int64_t m = m0 + r, b = b0 + c;
    if (m >= n || b >= p) continue;
    T x[kDMaxS];
#pragma unroll
    for (int q = 0; q < kDMaxS; ++q) x[q] = q < S ? d_load_rank(part + c * PITCH + r, q) : (T)0;
    T sum = x[0];
#pragma unroll
    for (int q = 1; q < kDMaxS; ++q)
      if (q < S) sum += x[q];
    W[b * ldw + m] = fma(shift, __ldg(V + b * ldv + m), sum);
  }
  // no CTA leaves while the others may read its tile; nothing waits for the stores
  __syncwarp();
  asm volatile("barrier.cluster.arrive.relaxed.aligned;" ::: "memory");
  asm volatile("barrier.cluster.wait.aligned;" ::: "memory");
}

// float32: tiles of 64 rows x BP probes by G groups of threads, each group the whole
// tile over a G-th of every slice's columns; a thread has 8 rows tx + 8 i and four probes
// ty + TY j, read 16 bytes (four columns) at a time and summed as pairs of columns by
// two-float FMAs: 12 reads for 64 of these, two CTAs an SM so that one's reads overlap
// the other's FMAs.  Bound by those reads (four cycles of shared memory each) and the FMA
// pipes.  Against 4 x 4 outputs a thread and copies indexed anew in every slice: n =
// 2000, 64 probes 27 -> 22.8 us; n = 4096, 256 279 -> 228; n = 16384, 256 4.18 -> 3.38 ms (41
// TFLOP/s).  8 x 8 outputs, one CTA an SM: 22.8, 261, 3.43; 64-column slices 24.6, 240, 3.53.
// two float FMAs in one instruction, and the sum of the two
__device__ __forceinline__ void fma2(unsigned long long &acc, unsigned long long a, unsigned long long b) {
  asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(acc) : "l"(a), "l"(b));
}
__device__ __forceinline__ float sum2(unsigned long long v) {
  return __uint_as_float((uint32_t)v) + __uint_as_float((uint32_t)(v >> 32));
}

template <int BP, int BK, int G>
__global__ void __launch_bounds__(256, 2)
dense_f32_kernel(const float *__restrict__ A, int64_t lda, const float *__restrict__ V, int64_t ldv,
                 float *__restrict__ W, int64_t ldw, int64_t n, int64_t p, float shift) {
  constexpr int BM = 64, LD = BK + 4, TY = 32 / G, TP = BP / TY, PITCH = BM + 8, KG = BK / G;
  extern __shared__ __align__(16) uint8_t d_raw[];
  float *stages = reinterpret_cast<float *>(d_raw);
  const int S = (int)gridDim.x, rank = (int)blockIdx.x;
  const int64_t m0 = (int64_t)blockIdx.y * BM, b0 = (int64_t)blockIdx.z * BP;
  const int64_t slices = (n + BK - 1) / BK;
  const int tx = threadIdx.x & 7, ty = (threadIdx.x >> 3) % TY, group = threadIdx.x / (8 * TY);
  unsigned long long acc[8][TP];
#pragma unroll
  for (int i = 0; i < 8; ++i)
#pragma unroll
    for (int j = 0; j < TP; ++j) acc[i][j] = 0;
  d_pipeline<float, BM, BP, BK, 256>(
      stages, A, lda, V, ldv, n, p, m0, b0, slices * rank / S, slices * (rank + 1) / S,
      [&](const float *As, const float *Vs) {
#pragma unroll
        for (int kk = 0; kk < KG; kk += 4) {
          const int k = group * KG + kk;
          ulonglong2 v[TP];
#pragma unroll
          for (int j = 0; j < TP; ++j) v[j] = *reinterpret_cast<const ulonglong2 *>(Vs + (ty + j * TY) * LD + k);
#pragma unroll
          for (int i = 0; i < 8; ++i) {
            const ulonglong2 a = *reinterpret_cast<const ulonglong2 *>(As + (tx + i * 8) * LD + k);
#pragma unroll
            for (int j = 0; j < TP; ++j) {
              fma2(acc[i][j], a.x, v[j].x);
              fma2(acc[i][j], a.y, v[j].y);
            }
          }
        }
      });
  // the groups' partial tiles, probes PITCH apart (no bank twice), summed in order
#pragma unroll
  for (int j = 0; j < TP; ++j)
#pragma unroll
    for (int i = 0; i < 8; ++i) stages[(group * BP + ty + j * TY) * PITCH + tx + i * 8] = sum2(acc[i][j]);
  __syncthreads();
  for (int i = threadIdx.x; i < BP * BM; i += 256) {
    const int at = i / BM * PITCH + i % BM;
    float sum = stages[at];
#pragma unroll
    for (int g = 1; g < G; ++g) sum += stages[g * BP * PITCH + at];
    stages[at] = sum;
  }
  d_reduce_store<float, BM, BP, PITCH, 256>(stages, V, ldv, W, ldw, n, p, m0, b0, rank, S, shift);
}

// float64: four warps, warp w the probes 8 w .. 8 w + 7 of the tile, its rows as M / 8
// m8n8k4 MMAs.  An SM runs 1.76 float64 FMAs a clock as MMAs and 1.68 as FMA
// instructions (measured), whatever a warp's independent chains, so tiles are small
// and many: up to five CTAs share an SM's pipe, MMAs past the last row or probe are
// left out, and no operand is reused in registers.  Against 32 x 32 tiles of FMA
// instructions on one CTA each: n = 1000, 100 probes 272 -> 234 us (0.86 TFLOP/s, 0.83 of
// that rate); n = 1500, 100 785 -> 470; n = 700, 37 193 -> 54; n = 200, 16 60 -> 11.
constexpr int kF64M = 16, kF64P = 32, kF64K = 32;

__global__ void __launch_bounds__(128)
dense_f64_kernel(const double *__restrict__ A, int64_t lda, const double *__restrict__ V, int64_t ldv,
                 double *__restrict__ W, int64_t ldw, int64_t n, int64_t p, double shift) {
  constexpr int M = kF64M, LD = kF64K + 2, kRows = M / 8;
  extern __shared__ __align__(16) uint8_t d_raw[];
  double *stages = reinterpret_cast<double *>(d_raw);
  const int S = (int)gridDim.x, rank = (int)blockIdx.x;
  const int64_t m0 = (int64_t)blockIdx.y * M, b0 = (int64_t)blockIdx.z * kF64P;
  const int64_t slices = (n + kF64K - 1) / kF64K;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int fr = lane >> 2, fk = lane & 3;  // fragment row (A) or probe (V), and column
  // warp-uniform: MMAs of 8 rows with any row and probe in range
  const int live = b0 + warp * 8 < p ? (int)(n - m0 < M ? (n - m0 + 7) / 8 : kRows) : 0;
  double c[kRows][2];
#pragma unroll
  for (int i = 0; i < kRows; ++i) c[i][0] = c[i][1] = 0.0;
  d_pipeline<double, M, kF64P, kF64K, 128>(
      stages, A, lda, V, ldv, n, p, m0, b0, slices * rank / S, slices * (rank + 1) / S,
      [&](const double *As, const double *Vs) {
        if (live == 0) return;
        const double *a = As + fr * LD + fk, *v = Vs + (warp * 8 + fr) * LD + fk;
#pragma unroll
        for (int k = 0; k < kF64K; k += 4) {
          const double vb = v[k];
#pragma unroll
          for (int i = 0; i < kRows; ++i)
            if (i < live)
              asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0, %1}, {%2}, {%3}, {%0, %1};"
                           : "+d"(c[i][0]), "+d"(c[i][1])
                           : "d"(a[i * 8 * LD + k]), "d"(vb));
        }
      });
#pragma unroll
  for (int i = 0; i < kRows; ++i)
#pragma unroll
    for (int e = 0; e < 2; ++e) stages[(warp * 8 + 2 * fk + e) * M + i * 8 + fr] = c[i][e];
  d_reduce_store<double, M, kF64P, M, 128>(stages, V, ldv, W, ldw, n, p, m0, b0, rank, S, shift);
}

// The same product by FMA instructions: a CTA of 256 threads forms a tile of 32 rows x 32
// probes over all of K, a thread 2 x 2 of it, both operands k-major in shared memory and the
// next 16 columns on their way in registers.  An SM runs 1.94 FMAs a clock so, against 1.76
// as MMAs, but a tile is a CTA: the last round of them costs as much as a full one (n =
// 1000: 278 us for up to 152 tiles, 532 for up to 304).  Bound by the float64 pipe.
constexpr int kF64Tile = 32, kF64Cols = 16;

__global__ void __launch_bounds__(256)
dense_f64_fma_kernel(const double *__restrict__ A, int64_t lda, const double *__restrict__ V, int64_t ldv,
                     double *__restrict__ W, int64_t ldw, int64_t n, int64_t p, double shift) {
  constexpr int B = kF64Tile, BK = kF64Cols;
  __shared__ __align__(16) double As[BK][B], Vs[BK][B];
  static_assert(B * BK == 2 * 256, "a 16-byte load of each operand per thread");
  const int t = threadIdx.x, tx = t % (B / 2), ty = t / (B / 2);
  const int64_t m0 = (int64_t)blockIdx.x * B, b0 = (int64_t)blockIdx.y * B;
  const int row = t / (BK / 2), kq = t % (BK / 2) * 2;  // this thread's load: two columns of a row
  double ra[2], rv[2];
  auto load = [&](const double *__restrict__ X, int64_t ldx, int64_t r, int64_t rows, int64_t k, double(&x)[2]) {
    x[0] = x[1] = 0.0;
    if (r >= rows) return;
    if (k + 2 <= n) {
      const double2 u = __ldg(reinterpret_cast<const double2 *>(X + r * ldx + k));
      x[0] = u.x;
      x[1] = u.y;
    } else if (k < n) {
      x[0] = X[r * ldx + k];
    }
  };
  double acc[2][2] = {};
  load(A, lda, m0 + row, n, kq, ra);
  load(V, ldv, b0 + row, p, kq, rv);
  for (int64_t k0 = 0; k0 < n; k0 += BK) {
    __syncthreads();
#pragma unroll
    for (int u = 0; u < 2; ++u) {
      As[kq + u][row] = ra[u];
      Vs[kq + u][row] = rv[u];
    }
    __syncthreads();
    if (k0 + BK < n) {
      load(A, lda, m0 + row, n, k0 + BK + kq, ra);
      load(V, ldv, b0 + row, p, k0 + BK + kq, rv);
    }
#pragma unroll
    for (int kk = 0; kk < BK; ++kk) {
      const double2 a = *reinterpret_cast<const double2 *>(&As[kk][tx * 2]);
      const double2 v = *reinterpret_cast<const double2 *>(&Vs[kk][ty * 2]);
      acc[0][0] = fma(a.x, v.x, acc[0][0]);
      acc[0][1] = fma(a.x, v.y, acc[0][1]);
      acc[1][0] = fma(a.y, v.x, acc[1][0]);
      acc[1][1] = fma(a.y, v.y, acc[1][1]);
    }
  }
#pragma unroll
  for (int j = 0; j < 2; ++j)
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      const int64_t m = m0 + tx * 2 + i, b = b0 + ty * 2 + j;
      if (m < n && b < p) W[b * ldw + m] = fma(shift, __ldg(V + b * ldv + m), acc[i][j]);
    }
}

template <typename K, typename T>
static int launch_dense_cluster(K kern, int bm, int bp, int threads, size_t smem, int S, const T *A, int64_t lda,
                                const T *V, int64_t ldv, T *W, int64_t ldw, int64_t n, int64_t p, T shift,
                                cudaStream_t s) {
  const int64_t gy = ceil_div(n, bm), gz = ceil_div(p, bp);
  if (gy > 65535 || gz > 65535) return MFG_ERR_UNSUPPORTED;
  MFG_CUDA_TRY(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)S, (unsigned)gy, (unsigned)gz);
  cfg.blockDim = dim3((unsigned)threads);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = s;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = (unsigned)S;
  attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  MFG_CUDA_TRY(cudaLaunchKernelEx(&cfg, kern, A, lda, V, ldv, W, ldw, n, p, shift));
  return MFG_LAUNCH_STATUS();
}

// the launch of one float32 form, with the shared memory that the form needs
template <int BP, int BK, int G>
static int launch_f32(int S, const float *A, int64_t lda, const float *V, int64_t ldv, float *W, int64_t ldw, int64_t n,
                      int64_t p, float shift, cudaStream_t s) {
  constexpr size_t kRing = (size_t)kDStages * (64 + BP) * (BK + 4) * sizeof(float);
  constexpr size_t kPart = (size_t)G * BP * 72 * sizeof(float);
  return launch_dense_cluster(dense_f32_kernel<BP, BK, G>, 64, BP, 256, kRing > kPart ? kRing : kPart, S, A, lda, V,
                              ldv, W, ldw, n, p, shift, s);
}

// SMs of 152 that clusters of S CTAs fill
constexpr int kFit[kDMaxS + 1] = {0, 152, 152, 138, 148, 140, 138, 105, 144};

template <typename T>
int launch_dense_simt(const T *A, int64_t lda, const T *V, int64_t ldv, T *W, int64_t ldw,
                      int64_t n, int64_t p, double shift, cudaStream_t s) {
  if (n <= 0 || p <= 0) return MFG_OK;
  const int sms = sm_count();
  if constexpr (sizeof(T) == 8) {
    // the K ranges of least time: an SM's CTAs one after the other on its pipe (five
    // at a time; past that a tail of two), slower with few of them to hide each
    // other's waits; clusters of three leave SMs of a GPC over
    const int64_t slices = ceil_div(n, kF64K), tiles = ceil_div(n, kF64M) * ceil_div(p, kF64P);
    int S = 1;
    double best = 1e300;
    for (int c : {1, 2, 3, 4, 8}) {
      if (c > slices) break;
      const double ctas = (double)(tiles * c) / sms;
      const double rounds = ctas <= 5.0 ? (double)ceil_div(tiles * c, sms) : ctas + 2.0;
      const double cost = rounds * (double)(ceil_div(slices, c) + 1) * (1.0 + 0.25 / ctas) * (c == 3 ? 1.1 : 1.0);
      if (cost < best) {
        best = cost;
        S = c;
      }
    }
    // FMA tiles where they fill their rounds and the MMAs' CTAs do not, both counted in the FMAs
    // of an SM at 1.76 a clock, rows and probes in MMAs of eight.  The MMAs' CTAs share an SM
    // five at a time; with a few more the first SMs to be done take five again (1.28), and many
    // even out (1.11, 1.05).  MMAs -> FMAs, us: n = 1000, 128 probes 410 -> 279 (100 probes: 239,
    // 279), 1200, 512 1642 -> 1237, 2000, 64 675 -> 546 (48: 448, 545), 4096, 256 8739 -> 7239.  Over 323
    // sizes (200 <= n <= 4096, p <= 1000) the choice is within 3 % of the faster one but for two (10 %).
    const double ctas = (double)(tiles * S * 152) / ((double)kFit[S] * sms);
    const double q = ctas <= 5.0 ? ceil(ctas) / ctas : (ctas < 10.0 ? 1.28 : (ctas < 30.0 ? 1.11 : 1.05));
    const double mma = 64.0 * (double)ceil_div(n, 8) * (double)ceil_div(p, 8) * q;
    const int64_t fx = ceil_div(n, kF64Tile), fy = ceil_div(p, kF64Tile);
    const double rounds = (double)ceil_div(fx * fy, sms);
    if (mma > (double)sms * kF64Tile * kF64Tile * (0.82 * rounds + 0.06)) {
      if (fy > 65535) return MFG_ERR_UNSUPPORTED;
      dense_f64_fma_kernel<<<dim3((unsigned)fx, (unsigned)fy), 256, 0, s>>>(A, lda, V, ldv, W, ldw, n, p, shift);
      return MFG_LAUNCH_STATUS();
    }
    const size_t smem = (size_t)kDStages * (kF64M + kF64P) * (kF64K + 2) * sizeof(double);
    return launch_dense_cluster(dense_f64_kernel, kF64M, kF64P, 128, smem, S, A, lda, V, ldv, W, ldw, n, p, shift, s);
  } else {
    // the K ranges of least time: an SM's CTAs share its pipes, so what counts is the
    // CTAs of the busiest SM (clusters of three to eight leave SMs of a GPC over) times the
    // slices of one; a range more is a tile more to add.  n = 2000, 64 probes S = 8 22.8 us (4:
    // 24.8, 5: 33.0); n = 3001, 64 S = 5 45 (4: 55, 6: 56, 8: 48); n = 4096, 256 S = 4 228 (2: 258).
    const int bp = p <= 32 ? 32 : 64;
    const int64_t tiles = ceil_div(n, 64) * ceil_div(p, bp), slices = ceil_div(n, 64);
    int S = 1;
    double best = 1e300;
    for (int c = 1; c <= kDMaxS && c <= slices; ++c) {
      const double busiest = (double)ceil_div(tiles * c * 152, (int64_t)kFit[c] * sms);
      const double cost = busiest * (double)ceil_div(slices, c) * (1.0 + 0.15 * sms / (double)(tiles * c)) + 0.15 * c;
      if (cost < best) {
        best = cost;
        S = c;
      }
    }
    if (bp == 32) return launch_f32<32, 64, 4>(S, A, lda, V, ldv, W, ldw, n, p, (float)shift, s);
    return launch_f32<64, 32, 2>(S, A, lda, V, ldv, W, ldw, n, p, (float)shift, s);
  }
}
template int launch_dense_simt<float>(const float *, int64_t, const float *, int64_t, float *,
                                      int64_t, int64_t, int64_t, double, cudaStream_t);
template int launch_dense_simt<double>(const double *, int64_t, const double *, int64_t, double *,
                                       int64_t, int64_t, int64_t, double, cudaStream_t);

// ---------------------------------------------------------------------------
// CSR SpMM: W[b][r] = sum_e val[e] V[b][col[e]] + shift V[b][r]
//
// The panels are probe-major, so the product is p sparse matrix-vector
// products that share the CSR arrays.  The rows are cut into tiles of
// kWRows; CTAs take tiles round-robin, so neighbouring tiles run at the same
// time and the vector entries they share are served from L2.  (Equal tiles
// sized to a whole number of waves measured slower on the 2-D Laplacian: the
// smaller tiles re-read more of the neighbouring rows.)  Per tile:
//   1. each row thread (4 rows per thread, rows r0 + t + 256 i) loads the
//      first RMAX entries of its rows into registers once; the tile's column
//      range [lo, hi] (including its own rows, for the shift term) follows
//      from a block reduction;
//   2. when the range is at most kWMax entries (banded matrices: stencils of
//      bandwidth up to about (kWMax - kWRows) / 2), a copy warp streams probe
//      b's window V[b][lo..hi] into a ring of shared-memory buffers with one
//      1-D bulk copy (cp.async.bulk) per probe, and the row threads form every
//      product from registers and shared memory (one shared load and one FMA
//      per entry): each probe vector is read from HBM about once, in long
//      bursts, instead of as scattered 4-byte gathers;
//   3. otherwise (wide or random column patterns) the row threads gather from
//      global memory: lane = row for short rows, and a warp walks its rows
//      one at a time with a butterfly of warp shuffles when one of them is
//      longer than kWLong entries.
// Entries beyond RMAX of a row are read from global memory in the same order.
// Every sum runs in a fixed order, so results do not depend on timing.  All
// waits are bounded (MFG_ERR_TIMEOUT in *status); after a failure the CTA
// stops at the next tile boundary and drains its copies in flight.
// ---------------------------------------------------------------------------

constexpr int kWRows = 1024;                   // rows per tile
constexpr int kWThreads = 256;                 // row threads (8 warps) + one copy warp
constexpr int kWRowWarps = kWThreads / 32;
constexpr int kWRowsPerThread = kWRows / kWThreads;
constexpr int kWMax = 4096;                    // window entries per ring buffer (16 KB)
constexpr int kWStages = 6;
constexpr int kWLong = 32;                     // longer rows take the warp-cooperative path

struct WinShared {
  uint64_t full[kWStages];
  uint64_t empty[kWStages];
  int lo, hi, fail, pad;
  int32_t rp[kWRows + 4];
  float win[kWStages][kWMax];
};

__device__ __forceinline__ uint32_t sp_smem(const void *p) {
  return (uint32_t)__cvta_generic_to_shared(p);
}

template <int RMAX>
__global__ void __launch_bounds__(kWThreads + 32, RMAX <= 6 ? 2 : 1)
csr_spmm_window_kernel(const int32_t *__restrict__ rp, const int32_t *__restrict__ ci,
                       const float *__restrict__ val, int64_t n, int tile_rows,
                       const float *__restrict__ V, int64_t ldv, float *__restrict__ W, int64_t ldw,
                       int64_t p, float shift, int *status) {
  extern __shared__ __align__(128) uint8_t sp_raw[];
  WinShared *sh = reinterpret_cast<WinShared *>(sp_raw);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const bool copier = warp == kWRowWarps;
  volatile int *fail = &sh->fail;
  if (threadIdx.x == 0) {
    for (int s = 0; s < kWStages; ++s) {
      asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(sp_smem(&sh->full[s])) : "memory");
      asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(sp_smem(&sh->empty[s])),
                   "r"(kWRowWarps)
                   : "memory");
    }
    sh->fail = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  __syncthreads();
  const int64_t ntiles = (n + tile_rows - 1) / tile_rows;
  int64_t g = 0;          // window copies issued (copy warp) / consumed (row warps) by this CTA
  int64_t issued = 0;     // copy warp: for the drain after a failure
  for (int64_t tile = blockIdx.x; tile < ntiles; tile += gridDim.x) {
    __syncthreads();  // the previous tile's shared data is no longer read
    if (*fail) break;  // uniform: read after the barrier
    const int64_t r0 = tile * tile_rows;
    const int rows = (int)(n - r0 < (int64_t)tile_rows ? n - r0 : (int64_t)tile_rows);
    for (int i = threadIdx.x; i <= rows; i += kWThreads + 32) sh->rp[i] = __ldg(rp + r0 + i);
    if (threadIdx.x == 0) {
      sh->lo = (int)r0;
      sh->hi = (int)(r0 + rows - 1);
    }
    __syncthreads();
    // this thread's rows: the first RMAX entries in registers
    int col[kWRowsPerThread][RMAX];
    float a[kWRowsPerThread][RMAX];
    int e0[kWRowsPerThread], len[kWRowsPerThread];
    if (!copier) {
      int cmin = 0x7fffffff, cmax = -1;
#pragma unroll
      for (int i = 0; i < kWRowsPerThread; ++i) {
        const int lr = threadIdx.x + i * kWThreads;
        e0[i] = lr < rows ? sh->rp[lr] : 0;
        len[i] = lr < rows ? sh->rp[lr + 1] - e0[i] : 0;
#pragma unroll
        for (int q = 0; q < RMAX; ++q) {
          col[i][q] = q < len[i] ? __ldg(ci + e0[i] + q) : (int)(r0 + (lr < rows ? lr : 0));
          a[i][q] = q < len[i] ? __ldg(val + e0[i] + q) : 0.f;
          if (q < len[i]) {
            cmin = min(cmin, col[i][q]);
            cmax = max(cmax, col[i][q]);
          }
        }
        for (int e = e0[i] + RMAX; e < e0[i] + len[i]; ++e) {
          const int c = __ldg(ci + e);
          cmin = min(cmin, c);
          cmax = max(cmax, c);
        }
      }
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) {
        cmin = min(cmin, __shfl_xor_sync(0xffffffffu, cmin, o));
        cmax = max(cmax, __shfl_xor_sync(0xffffffffu, cmax, o));
      }
      if (lane == 0) {
        atomicMin(&sh->lo, cmin);
        atomicMax(&sh->hi, cmax);
      }
    }
    __syncthreads();
    const int64_t lo = (int64_t)sh->lo & ~(int64_t)3;
    const int64_t wlen = ((int64_t)sh->hi + 1 - lo + 3) & ~(int64_t)3;  // <= ld - lo: ld % 8 == 0
    // (column indices outside [0, n) break the caller's contract; such a tile
    // never issues a bulk copy)
    const bool windowed = wlen <= kWMax && sh->lo >= 0 && sh->hi < n;

    if (windowed) {
      if (copier) {
        if (lane == 0) {
          int s = (int)(g % kWStages);
          uint32_t ph = (uint32_t)((g / kWStages) & 1);
          for (int64_t b = 0; b < p; ++b, ++g) {
            if (b > 0 && ++s == kWStages) {
              s = 0;
              ph ^= 1u;
            }
            if (g >= kWStages && !mbar_wait_bounded(sp_smem(&sh->empty[s]), ph ^ 1u, fail)) {
              *fail = 1;
              if (status) atomicExch(status, (int)MFG_ERR_TIMEOUT);
              break;
            }
            asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(
                             sp_smem(&sh->full[s])),
                         "r"((uint32_t)(wlen * 4))
                         : "memory");
            asm volatile(
                "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
                ::"r"(sp_smem(&sh->win[s][0])), "l"(reinterpret_cast<uint64_t>(V + b * ldv + lo)),
                "r"((uint32_t)(wlen * 4)), "r"(sp_smem(&sh->full[s]))
                : "memory");
            issued = g + 1;
          }
        }
        g = __shfl_sync(0xffffffffu, g, 0);
        issued = __shfl_sync(0xffffffffu, issued, 0);
      } else {
        // byte offsets into the window: the columns, and each row's own entry
        const int lo32 = (int)lo;
        int self[kWRowsPerThread];
#pragma unroll
        for (int i = 0; i < kWRowsPerThread; ++i) {
          self[i] = 4 * (int)(r0 + threadIdx.x + i * kWThreads - lo32);
#pragma unroll
          for (int q = 0; q < RMAX; ++q) col[i][q] = 4 * (col[i][q] - lo32);
        }
        int s = (int)(g % kWStages);
        uint32_t ph = (uint32_t)((g / kWStages) & 1);
        for (int64_t b = 0; b < p; ++b, ++g) {
          const bool ok = !*fail && mbar_wait_bounded(sp_smem(&sh->full[s]), ph, fail);
          if (!ok) {
            if (lane == 0) {
              *fail = 1;
              if (status) atomicExch(status, (int)MFG_ERR_TIMEOUT);
            }
            break;
          }
          const char *w = reinterpret_cast<const char *>(sh->win[s]);
          float *Wb = W + b * ldw + r0 + threadIdx.x;
#pragma unroll
          for (int i = 0; i < kWRowsPerThread; ++i) {
            if ((int)threadIdx.x + i * kWThreads < rows) {
              float acc = shift * *reinterpret_cast<const float *>(w + self[i]);
#pragma unroll
              for (int q = 0; q < RMAX; ++q)
                acc = fmaf(a[i][q], *reinterpret_cast<const float *>(w + col[i][q]), acc);
              for (int e = e0[i] + RMAX; e < e0[i] + len[i]; ++e)
                acc = fmaf(__ldg(val + e), *reinterpret_cast<const float *>(w + 4 * (__ldg(ci + e) - lo32)), acc);
              Wb[i * kWThreads] = acc;
            }
          }
          __syncwarp();
          if (lane == 0)
            asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(sp_smem(&sh->empty[s])) : "memory");
          if (++s == kWStages) {
            s = 0;
            ph ^= 1u;
          }
        }
      }
      continue;
    }

    // gather path
    if (copier) continue;
#pragma unroll 1
    for (int i = 0; i < kWRowsPerThread; ++i) {
      const int lr = threadIdx.x + i * kWThreads;
      const bool has_row = lr < rows;
      int lmax = len[i];
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) lmax = max(lmax, __shfl_xor_sync(0xffffffffu, lmax, o));
      if (lmax <= kWLong) {
        const int64_t r = r0 + lr;
        for (int64_t b = 0; b < p; ++b) {
          if (has_row) {
            const float *Vb = V + b * ldv;
            float acc = shift * __ldg(Vb + r);
            for (int e = e0[i]; e < e0[i] + len[i]; ++e) acc = fmaf(__ldg(val + e), __ldg(Vb + __ldg(ci + e)), acc);
            W[b * ldw + r] = acc;
          }
        }
        continue;
      }
      // a long row among this warp's rows: the warp walks them one at a time
      for (int j = 0; j < 32; ++j) {
        const int lj = (lr - lane) + j;
        if (lj >= rows) break;
        const int f0 = sh->rp[lj], f1 = sh->rp[lj + 1];
        const int64_t r = r0 + lj;
        for (int64_t b = 0; b < p; ++b) {
          const float *Vb = V + b * ldv;
          float acc = 0.f;
          for (int e = f0 + lane; e < f1; e += 32) acc = fmaf(__ldg(val + e), __ldg(Vb + __ldg(ci + e)), acc);
#pragma unroll
          for (int o = 16; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
          if (lane == 0) W[b * ldw + r] = fmaf(shift, __ldg(Vb + r), acc);
        }
      }
    }
  }
  // after a failure the copies in flight land before the shared memory goes away
  if (copier && lane == 0 && *fail) {
    for (int64_t t = (issued > kWStages ? issued - kWStages : 0); t < issued; ++t)
      mbar_wait_bounded(sp_smem(&sh->full[t % kWStages]), (uint32_t)((t / kWStages) & 1), nullptr,
                        kMbarWaitNs / 8);
  }
}

template <int RMAX>
static int launch_csr_spmm_t(const int32_t *row_ptr, const int32_t *col_idx, const float *val, int64_t n,
                             const float *V, int64_t ldv, float *W, int64_t ldw, int64_t p, double shift,
                             int *status, cudaStream_t s) {
  const size_t smem = sizeof(WinShared);
  static PerDevice<int> table;
  const int *per_sm = table.get(current_device(), [&](int &q) {
    return cuda_status(cudaFuncSetAttribute(csr_spmm_window_kernel<RMAX>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                            (int)smem),
                       __FILE__, __LINE__) == MFG_OK &&
           cuda_status(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&q, csr_spmm_window_kernel<RMAX>, kWThreads + 32,
                                                                     smem),
                       __FILE__, __LINE__) == MFG_OK;
  });
  if (!per_sm) return MFG_ERR_CUDA;
  if (*per_sm < 1) return MFG_ERR_UNSUPPORTED;
  const int64_t G = (int64_t)sm_count() * *per_sm;
  const int64_t tile_rows = kWRows;
  const int64_t ntiles = ceil_div(n, tile_rows);
  const int64_t grid = G < ntiles ? G : ntiles;
  csr_spmm_window_kernel<RMAX><<<(unsigned)grid, kWThreads + 32, smem, s>>>(
      row_ptr, col_idx, val, n, (int)tile_rows, V, ldv, W, ldw, p, (float)shift, status);
  return MFG_LAUNCH_STATUS();
}

int launch_csr_spmm(const int32_t *row_ptr, const int32_t *col_idx, const float *val, int64_t n,
                    int64_t nnz, const float *V, int64_t ldv, float *W, int64_t ldw, int64_t p,
                    double shift, int *status, cudaStream_t s) {
  if (n <= 0 || p <= 0) return MFG_OK;
  if (n > 0x7ffffff0 || ldv % 8 != 0 || reinterpret_cast<uintptr_t>(V) % 16 != 0) return MFG_ERR_UNSUPPORTED;
  // entries held in registers per row: 6 covers 2-D 5-point stencils, 12 the
  // 3-D 7-point ones and up to 12 entries; longer rows read the rest from
  // global memory
  if (nnz <= 6 * n)
    return launch_csr_spmm_t<6>(row_ptr, col_idx, val, n, V, ldv, W, ldw, p, shift, status, s);
  return launch_csr_spmm_t<12>(row_ptr, col_idx, val, n, V, ldv, W, ldw, p, shift, status, s);
}

// ---------------------------------------------------------------------------
// RBF kernel matrix and bf16 split
// ---------------------------------------------------------------------------

__global__ void __launch_bounds__(256)
rbf_kernel(const float *__restrict__ x, int64_t n, int dim, double s2, double inv2l2, int prec,
           int dlogell, void *__restrict__ a, void *__restrict__ a_lo, int64_t lda) {
  const int64_t i = blockIdx.y;
  const int64_t j = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (j >= lda) return;
  const int64_t o = i * lda + j;
  if (prec == MFG_PREC_FP64) {
    double v = 0.0;
    if (j < n) {
      double d2 = 0.0;
      for (int d = 0; d < dim; ++d) {
        const double df = (double)x[i * dim + d] - (double)x[j * dim + d];
        d2 += df * df;
      }
      v = s2 * exp(-d2 * inv2l2);
      if (dlogell) v *= 2.0 * d2 * inv2l2;  // d/dlog(ell) of exp(-d2/(2 ell^2))
    }
    reinterpret_cast<double *>(a)[o] = v;
    return;
  }
  float v = 0.f;
  if (j < n) {
    float d2 = 0.f;
    for (int d = 0; d < dim; ++d) {
      const float df = x[i * dim + d] - x[j * dim + d];
      d2 = fmaf(df, df, d2);
    }
    v = (float)s2 * expf(-d2 * (float)inv2l2);
    if (dlogell) v *= 2.f * d2 * (float)inv2l2;
  }
  if (prec == MFG_PREC_FP32) {
    reinterpret_cast<float *>(a)[o] = v;
  } else {
    const __nv_bfloat16 h = __float2bfloat16_rn(v);
    reinterpret_cast<__nv_bfloat16 *>(a)[o] = h;
    if (prec == MFG_PREC_BF16X3)
      reinterpret_cast<__nv_bfloat16 *>(a_lo)[o] = __float2bfloat16_rn(v - __bfloat162float(h));
  }
}

// fp32 / bf16 / bf16 hi+lo entries.  A CTA covers kRbfRows rows x 2048
// columns: the columns' points are staged in shared memory once (coalesced,
// coordinate-major) and reused for every row; each thread forms eight
// consecutive entries of a row and stores them with one 16-byte store per
// bf16 array (two for fp32).  Each entry is computed exactly as in rbf_kernel.
constexpr int kRbfRows = 16;
constexpr int kRbfCols = 256 * 8;
constexpr int kRbfMaxDim = 4;

__global__ void __launch_bounds__(256)
rbf8_kernel(const float *__restrict__ x, int64_t n, int dim, float s2, float inv2l2, int prec,
            int dlogell, void *__restrict__ a, void *__restrict__ a_lo, int64_t lda) {
  __shared__ __align__(16) float xs[kRbfMaxDim][kRbfCols];
  const int64_t c0 = (int64_t)blockIdx.x * kRbfCols;
  const int64_t r0 = (int64_t)blockIdx.y * kRbfRows;
  for (int t = threadIdx.x; t < kRbfCols * dim; t += 256) {
    const int c = t / dim, d = t - c * dim;  // x is point-major: coalesced reads
    const int64_t j = c0 + c;
    xs[d][c] = j < n ? x[j * dim + d] : 0.f;
  }
  __syncthreads();
  const int64_t j0 = c0 + (int64_t)threadIdx.x * 8;
  if (j0 >= lda) return;
  // this thread's 8 points in registers, read from shared memory once (a
  // read per row would be an 8-way bank conflict: threads are 8 floats
  // apart); dimensions past dim are zero on both sides and add nothing
  float xc[kRbfMaxDim][8];
#pragma unroll
  for (int d = 0; d < kRbfMaxDim; ++d)
#pragma unroll
    for (int e = 0; e < 8; ++e) xc[d][e] = d < dim ? xs[d][threadIdx.x * 8 + e] : 0.f;
  for (int rr = 0; rr < kRbfRows; ++rr) {
    const int64_t i = r0 + rr;
    if (i >= n) return;
    float xi[kRbfMaxDim];
#pragma unroll
    for (int d = 0; d < kRbfMaxDim; ++d) xi[d] = d < dim ? __ldg(x + i * dim + d) : 0.f;
    float v[8];
#pragma unroll
    for (int e = 0; e < 8; ++e) {
      float d2 = 0.f;
#pragma unroll
      for (int d = 0; d < kRbfMaxDim; ++d) {
        const float df = xi[d] - xc[d][e];
        d2 = fmaf(df, df, d2);
      }
      float w = s2 * expf(-d2 * inv2l2);
      if (dlogell) w *= 2.f * d2 * inv2l2;
      v[e] = (j0 + e < n) ? w : 0.f;
    }
    const int64_t o = i * lda + j0;  // 8-element aligned: lda % 8 == 0
    if (prec == MFG_PREC_FP32) {
      float4 *dst = reinterpret_cast<float4 *>(reinterpret_cast<float *>(a) + o);
      dst[0] = make_float4(v[0], v[1], v[2], v[3]);
      dst[1] = make_float4(v[4], v[5], v[6], v[7]);
      continue;
    }
    uint32_t hw[4], lw[4];
#pragma unroll
    for (int e = 0; e < 8; e += 2) {
      const __nv_bfloat16 h0 = __float2bfloat16_rn(v[e]), h1 = __float2bfloat16_rn(v[e + 1]);
      hw[e / 2] = (uint32_t)__bfloat16_as_ushort(h0) | ((uint32_t)__bfloat16_as_ushort(h1) << 16);
      const __nv_bfloat16 l0 = __float2bfloat16_rn(v[e] - __bfloat162float(h0));
      const __nv_bfloat16 l1 = __float2bfloat16_rn(v[e + 1] - __bfloat162float(h1));
      lw[e / 2] = (uint32_t)__bfloat16_as_ushort(l0) | ((uint32_t)__bfloat16_as_ushort(l1) << 16);
    }
    *reinterpret_cast<uint4 *>(reinterpret_cast<__nv_bfloat16 *>(a) + o) =
        make_uint4(hw[0], hw[1], hw[2], hw[3]);
    if (prec == MFG_PREC_BF16X3)
      *reinterpret_cast<uint4 *>(reinterpret_cast<__nv_bfloat16 *>(a_lo) + o) =
          make_uint4(lw[0], lw[1], lw[2], lw[3]);
  }
}

int launch_rbf_build(const float *x, int64_t n, int dim, double s2, double ell, int precision,
                     int dlogell, void *a, void *a_lo, int64_t lda, cudaStream_t s) {
  if (n <= 0) return MFG_OK;
  if (n > 65535) return MFG_ERR_UNSUPPORTED;
  const double inv2l2 = 1.0 / (2.0 * ell * ell);
  if (precision != MFG_PREC_FP64 && dim <= kRbfMaxDim && lda % 8 == 0 && ((uintptr_t)a & 15) == 0 &&
      (a_lo == nullptr || ((uintptr_t)a_lo & 15) == 0)) {
    rbf8_kernel<<<dim3((unsigned)ceil_div(lda, kRbfCols), (unsigned)ceil_div(n, kRbfRows)), 256, 0, s>>>(
        x, n, dim, (float)s2, (float)inv2l2, precision, dlogell, a, a_lo, lda);
    return MFG_LAUNCH_STATUS();
  }
  rbf_kernel<<<dim3((unsigned)ceil_div(lda, 256), (unsigned)n), 256, 0, s>>>(
      x, n, dim, s2, inv2l2, precision, dlogell, a, a_lo, lda);
  return MFG_LAUNCH_STATUS();
}

__global__ void split_kernel(const float *__restrict__ a, int64_t rows, int64_t cols, int64_t lda,
                             __nv_bfloat16 *__restrict__ hi, __nv_bfloat16 *__restrict__ lo,
                             int64_t ldo) {
  const int64_t i = blockIdx.y;
  const int64_t j = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= rows || j >= ldo) return;
  const float v = (j < cols) ? a[i * lda + j] : 0.f;
  const __nv_bfloat16 h = __float2bfloat16_rn(v);
  hi[i * ldo + j] = h;
  if (lo) lo[i * ldo + j] = __float2bfloat16_rn(v - __bfloat162float(h));
}

int launch_split_bf16(const float *a, int64_t rows, int64_t cols, int64_t lda, __nv_bfloat16 *hi,
                      __nv_bfloat16 *lo, int64_t ld_out, cudaStream_t s) {
  if (rows <= 0) return MFG_OK;
  if (rows > 65535) return MFG_ERR_UNSUPPORTED;
  split_kernel<<<dim3((unsigned)ceil_div(ld_out, 256), (unsigned)rows), 256, 0, s>>>(
      a, rows, cols, lda, hi, lo, ld_out);
  return MFG_LAUNCH_STATUS();
}

}  // namespace mfg
