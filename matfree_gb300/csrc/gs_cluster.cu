// Gram-Schmidt twice, and a step of the Hessenberg adjoint, as one launch: a
// cluster of CTAs per probe (building blocks in cluster.cuh; the two-sweep Arnoldi
// step in arnoldi_cluster.cu has the same organisation).
//
// Both are four passes over the same basis vectors, each needing the sums or the
// vector that the pass before completed:
//
//   Gram-Schmidt (decomp.py:454-477, 703-719)     adjoint step idx (decomp.py:560-599)
//     w -= c u_prev (bidiagonalisation)             v = gamma r - alpha lambda (+ dq)
//                                                     + Q_> Gamma[:, idx] - Lambda_> H[idx, >]
//     h = Q^T w                                     g = Q^T U
//     w -= Q h                                      v = (v + U + Q G) / beta
//     h2 = Q^T w                                    h = Q^T v
//     w -= Q h2, ||w||, q_next = w / ||w||          lambda' = v - Q (h - dH[:, idx - 1])
//
// (Q_>, Lambda_>: the vectors after idx, read once; Q: vectors 0 .. idx.)  CTA r of
// the cluster holds rows [r R, (r + 1) R) of the vector in registers.  Basis vectors
// come through per-group rings; the vectors still in a ring when a pass ends are the
// first of the next pass, so a basis that fits the rings is read once, and one
// that does not comes from HBM once and from L2 three times, as far as the probes in
// flight fit there.  As separate launches over all probes every pass came from HBM,
// with the vector written and read between them.
//
// What bounds it: for few probes the chain of loads, meetings and reductions (sums of
// floats across warps and CTAs are two-float numbers for that reason: adjoint steps of
// n = 1501, 32 probes 18.4 -> 15.8 us, n = 8192, 128 probes 87 -> 83 us), for many the reads.
// Against separate launches (four to five for Gram-Schmidt twice, twelve for an adjoint
// step): n = 8192, 128 probes, k = 32 bidiagonalisation half step 76 -> 44 us, adjoint
// k = 48 150 -> 83 us a step; float64 n = 1000, 100 probes, k = 30 62 -> 44 us a step.
#include "cluster.cuh"
#include "kernels.cuh"

namespace mfg {

constexpr int kGMaxCols = 256;

template <typename T>
struct GsArgs {
  const T *Q;  // vector i of probe b at Q + b qb + i ld, i < ncols
  int64_t qb, ld;
  int ncols;
  const T *W;  // the vector: probe stride ld
  int64_t n, p;
  int R, S, slots, passes;  // slots of a group's ring; passes 4, or 2 (one projection and update)
  int cpad, xpad;           // shared arrays: ncols, 2 nx rounded up to 8
  // Gram-Schmidt
  const T *prev;  // w -= prev_c[b prev_cs] prev, probe stride prev_b (null: none)
  int64_t prev_b;
  const double *prev_c;
  int64_t prev_cs;
  double *h;  // the first projections: h[b h_bs + i h_is]
  int64_t h_bs, h_is;
  double *norm, *norm2;  // ||w||: norm[b], norm2[b norm2_bs] (either may be null)
  int64_t norm2_bs;
  T *w_out;  // the unnormalised result, probe stride ld (null: not written)
  // adjoint (k > 0)
  int k, idx, nx;       // nx = k - 1 - idx vectors after idx
  const T *lam, *Lam;   // lambda (row idx of Lambda) and Lambda, probe stride qb
  const T *res, *dq;    // residual (probe stride ld), row idx of dQ (stride qb; null: none)
  const double *H, *Pi, *dH, *gamma, *out_scale;  // out_scale: last step, times out_scale[b]
  double *Gamma;  // GSum numbers
  // the result: q_next, lambda' or (idx 0) dv; its bf16 copies (probe stride ld)
  T *next;
  int64_t next_b;
  __nv_bfloat16 *hi, *lo;
  int *status;
};

// Sums across warps and CTAs: two-float numbers of floats, float64 of doubles.
template <typename T> struct GSum { using type = double; };
template <> struct GSum<float> { using type = float2; };
__device__ __forceinline__ double g_add(double a, double b) { return a + b; }
__device__ __forceinline__ float2 g_add(float2 a, float2 b) { return pair_add(a, b); }
__device__ __forceinline__ double g_sub(double a, double b) { return a - b; }
__device__ __forceinline__ float2 g_sub(float2 a, float2 b) { return pair_add(a, pair_neg(b)); }
__device__ __forceinline__ double g_twice(double a, double f) { return a * f; }
__device__ __forceinline__ float2 g_twice(float2 a, float f) { return make_float2(a.x * f, a.y * f); }  // f: a power of two
__device__ __forceinline__ double g_round(double a) { return a; }
__device__ __forceinline__ float g_round(float2 a) { return a.x; }
__device__ __forceinline__ double g_double(double a) { return a; }
__device__ __forceinline__ double g_double(float2 a) { return (double)a.x + (double)a.y; }
__device__ __forceinline__ double g_sum_of(double v) { return v; }
__device__ __forceinline__ float2 g_sum_of(float v) { return make_float2(v, 0.f); }
template <typename S> __device__ __forceinline__ S g_from(double v);
template <> __device__ __forceinline__ double g_from<double>(double v) { return v; }
template <> __device__ __forceinline__ float2 g_from<float2>(double v) {
  const float x = (float)v;
  return make_float2(x, (float)(v - (double)x));
}
__device__ __forceinline__ double g_load_rank(const double *p, int rank) { return c_ld_f64(c_map(c_smem(p), (uint32_t)rank)); }
__device__ __forceinline__ float2 g_load_rank(const float2 *p, int rank) { return c_ld_pair(c_map(c_smem(p), (uint32_t)rank)); }
__device__ __forceinline__ double g_xor(double v, int o) { return __shfl_xor_sync(0xffffffffu, v, o); }
__device__ __forceinline__ float2 g_xor(float2 v, int o) { return pair_shfl_xor(v, o); }
__device__ __forceinline__ double g_sqrt(double v) { return sqrt(v); }
__device__ __forceinline__ float2 g_sqrt(float2 v) {
  const float r = sqrtf(v.x);
  return r > 0.f ? pair(r, (fmaf(-r, r, v.x) + v.y) / (2.f * r)) : make_float2(r, 0.f);
}

struct GShared {
  uint64_t full[kCMaxSlots], empty[kCMaxSlots];
  uint64_t meet[3];
  // GSum numbers
  double npart[2];  // this CTA's ||w||^2, by the probe's parity
  double wred[kCWarps];
  double fin;
  int fail;
};

template <typename T>
__host__ __device__ inline size_t g_fixed(int cpad, int xpad, int R, int wr) {
  const size_t groups = kCWarps / wr;
  size_t b = (sizeof(GShared) + 15) / 16 * 16;
  b += (size_t)cpad * 8 * 6;                             // part[2][2], h_pi, dh
  b += (size_t)(wr * cpad + cpad + xpad) * sizeof(T);    // red, coef, extra coefficients
  if (groups > 1) b += groups * (size_t)R * sizeof(T);   // partial updates
  return (b + 127) / 128 * 128;
}

// a / b from r = 1 / b: a correction step makes it the rounded quotient (float64
// divisions are long here)
__device__ __forceinline__ float g_div(float a, float b, float) { return a / b; }
__device__ __forceinline__ double g_div(double a, double b, double r) {
  const double q = a * r;
  return fma(fma(-q, b, a), r, q);
}

template <typename T, int kWR, int kGC, bool kAdj>
__global__ void __launch_bounds__(kCThreads + 32, 2) gs_cluster_kernel(const GsArgs<T> a) {
  constexpr int kWC = kCWarps / kWR, VW = 16 / (int)sizeof(T), NV = 8 / VW;
  using Vt = typename Vec<T>::type;
  using Sum = typename GSum<T>::type;
  static_assert(sizeof(Sum) == 8, "shared arrays");
  extern __shared__ __align__(128) uint8_t g_raw[];
  GShared *sh = reinterpret_cast<GShared *>(g_raw);
  const int R = a.R, S = a.S, nslots = a.slots, nc = a.ncols, nx = kAdj ? a.nx : 0;
  Sum *part = reinterpret_cast<Sum *>(g_raw + (sizeof(GShared) + 15) / 16 * 16);  // [2][2][cpad]
  Sum *wred = reinterpret_cast<Sum *>(sh->wred), *npart = reinterpret_cast<Sum *>(sh->npart);
  Sum *fin = reinterpret_cast<Sum *>(&sh->fin);
  Sum *h_pi = part + 4 * a.cpad, *dh = h_pi + a.cpad;  // row idx of Pi, then the first projections; column of dH
  T *red = reinterpret_cast<T *>(dh + a.cpad);  // [kWR][cpad]
  T *coef = red + kWR * a.cpad, *xcoef = coef + a.cpad;
  T *comb = xcoef + a.xpad;  // [kWC][R]
  T *ring = reinterpret_cast<T *>(g_raw + g_fixed<T>(a.cpad, a.xpad, R, kWR));  // [kWC][nslots][kGC][R]
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int rank = S > 1 ? (int)c_rank() : 0;
  const int64_t r0 = (int64_t)rank * R;
  const int nloc = (int)(a.n - r0 < 0 ? 0 : (a.n - r0 < R ? a.n - r0 : R));
  const uint32_t col_bytes = (uint32_t)((nloc + VW - 1) / VW * 16);
  const int ns = (nc + kGC - 1) / kGC, nsx = (2 * nx + kGC - 1) / kGC;
  const int64_t cluster = blockIdx.x / S, nclusters = gridDim.x / S;
  volatile int *fail = &sh->fail;
  auto slots_of = [&](int g) { return g < ns ? (ns - g + kWC - 1) / kWC : 0; };
  auto kept_of = [&](int g) { return slots_of(g) < nslots ? slots_of(g) : nslots; };

  {
    auto init = [](uint64_t *bar, uint32_t count) {
      asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(c_smem(bar)), "r"(count) : "memory");
    };
    const int i = threadIdx.x;
    if (i < kWC * nslots) {
      init(&sh->full[i], 1);
      init(&sh->empty[i], kWR);
    } else if (i == kCMaxSlots) {
      for (int m = 0; m < 3; ++m) init(&sh->meet[m], (uint32_t)S);
      sh->fail = 0;
    }
    if (i <= kCMaxSlots) asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  __syncthreads();
  if (S > 1) c_cluster_arrive();  // waited for before the first access to another CTA
  chain_wait();
  chain_next();

  if (warp == kCWarps) {
    // copy warp: per probe the vectors after idx, then pass 1's slots, then of each
    // later pass the slots that did not stay.  Pass t takes a group's slots in the
    // order rotated by (t - 1)(slots - kept): those that stayed come first.
    int fills = 0, pos = 0;  // lane g: group g
    uint32_t par = 0;
    bool run = true;
    auto fill = [&](int g, int s, bool extra, int64_t b) {
      const int gpos = __shfl_sync(0xffffffffu, pos, g), gfills = __shfl_sync(0xffffffffu, fills, g);
      const uint32_t gpar = __shfl_sync(0xffffffffu, par, g);
      const int at = g * nslots + gpos;
      if (gfills >= nslots && !c_wait(&sh->empty[at], gpar ^ 1u, fail, a.status)) {
        run = false;
        return;
      }
      const int count = extra ? 2 * nx : nc;
      const int cols = count - s * kGC < kGC ? count - s * kGC : kGC;
      if (lane == 0) c_expect(&sh->full[at], (uint32_t)cols * col_bytes);
      __syncwarp();
      if (lane < cols && col_bytes) {
        const int c = s * kGC + lane;
        const T *src = a.Q + (int64_t)c * a.ld;
        if (extra) src = c < nx ? a.Q + (int64_t)(a.idx + 1 + c) * a.ld : a.Lam + (int64_t)(a.idx + 1 + c - nx) * a.ld;
        c_bulk(c_smem(ring + ((size_t)at * kGC + lane) * R), src + b * a.qb + r0, col_bytes, &sh->full[at]);
      }
      __syncwarp();
      if (lane == g) {
        ++fills;
        if (++pos == nslots) {
          pos = 0;
          par ^= 1u;
        }
      }
    };
    for (int64_t b = cluster; run && b < a.p; b += nclusters) {
      for (int s = 0; s < nsx && run; ++s) fill(s % kWC, s, true, b);
      for (int t = 1; t <= a.passes && run; ++t)
        for (int i = 0; i < slots_of(0) && run; ++i)
          for (int g = 0; g < kWC && run; ++g) {
            const int gs = slots_of(g), gk = kept_of(g);
            if (i >= gs || (t > 1 && i < gk)) continue;
            fill(g, (i + (t - 1) * (gs - gk)) % gs * kWC + g, false, b);
          }
    }
    if (S > 1) c_cluster_wait();
    c_done(S);
    if (*fail && lane < kWC) {
      // copies in flight land (bounded) before the shared memory goes away
      for (int f = fills > nslots ? fills - nslots : 0; f < fills; ++f)
        mbar_wait_bounded(c_smem(&sh->full[lane * nslots + f % nslots]), (uint32_t)(f / nslots) & 1u, nullptr,
                          kMbarWaitNs / 8);
    }
  } else {
    const int wr = warp % kWR, group = warp / kWR;
    int rv[NV];  // first rows of this lane's 16-byte vectors
    bool ok[NV];
#pragma unroll
    for (int q = 0; q < NV; ++q) {
      rv[q] = wr * kCRows + q * 32 * VW + lane * VW;
      ok[q] = rv[q] < nloc;
    }
    const int gs = slots_of(group), gk = kept_of(group);
    const int gsx = group < nsx ? (nsx - group + kWC - 1) / kWC : 0;
    int pos = 0;
    uint32_t sp = 0, par = 0;
    uint64_t *full = sh->full + group * nslots, *empty = sh->empty + group * nslots;
    const T *gring = ring + (size_t)group * nslots * kGC * R;
    auto next = [&]() {
      if (++pos == nslots) {
        pos = 0;
        sp ^= 1u;
      }
    };
    auto load_rows = [&](const T *src, T(&x)[8]) {  // rows past the CTA's are zero: padding is not data
#pragma unroll
      for (int q = 0; q < NV; ++q) {
        if (ok[q]) {
          vec_to_array<T>(*reinterpret_cast<const Vt *>(src + r0 + rv[q]), x + q * VW);
#pragma unroll
          for (int e = 0; e < VW; ++e)
            if (rv[q] + e >= nloc) x[q * VW + e] = (T)0;
        } else {
#pragma unroll
          for (int e = 0; e < VW; ++e) x[q * VW + e] = (T)0;
        }
      }
    };
    auto load_col = [&](const T *x, bool ready, T(&z)[8]) {
#pragma unroll
      for (int q = 0; q < NV; ++q) {
        if (ready && ok[q]) {
          vec_to_array<T>(*reinterpret_cast<const Vt *>(x + rv[q]), z + q * VW);
        } else {
#pragma unroll
          for (int e = 0; e < VW; ++e) z[q * VW + e] = (T)0;
        }
      }
    };
    // pass t over this group's slots, in that pass's order
    auto pass = [&](int t, auto body) {
      const bool last = t == a.passes;
      int u = gs > 0 ? (t - 1) * (gs - gk) % gs : 0;
      int kpos = pos;
      uint32_t ksp = sp;
      for (int i = 0; i < gs; ++i) {
        if (i == gs - gk) {
          kpos = pos;
          ksp = sp;
        }
        const bool ready = c_wait(&full[pos], sp, fail, a.status);
        body((u * kWC + group) * kGC, gring + (size_t)pos * kGC * R, ready);
        __syncwarp();
        if ((last || i < gs - gk) && lane == 0 && ready) c_arrive(&empty[pos]);
        next();
        if (++u == gs) u = 0;
      }
      if (!last) {
        pos = kpos;
        sp = ksp;
      }
    };
    auto dots = [&](int t, const T(&x)[8]) {
      pass(t, [&](int c0, const T *slot, bool ready) {
        T v[kGC];
#pragma unroll
        for (int c = 0; c < kGC; ++c) {
          T z[8];
          load_col(slot + c * R, ready, z);
          T s = z[0] * x[0];
#pragma unroll
          for (int e = 1; e < 8; ++e) s = fma(z[e], x[e], s);
          v[c] = s;
        }
        int idx;
        const T sum = c_xsum<kGC>(v, lane, idx);
        if ((lane & (32 / kGC - 1)) == 0 && c0 + idx < nc) red[wr * a.cpad + c0 + idx] = sum;
      });
    };
    auto axpy_slot = [&](const T *cf, int c0, int count, const T *slot, bool ready, T(&acc)[8]) {
#pragma unroll
      for (int c = 0; c < kGC; ++c) {
        if (c0 + c < count) {
          T z[8];
          load_col(slot + c * R, ready, z);
          const T f = cf[c0 + c];
#pragma unroll
          for (int e = 0; e < 8; ++e) acc[e] = fma(z[e], f, acc[e]);
        }
      }
    };
    bool met = S == 1;
    // the cluster's sums of red[.][0 .. nc) into tot; use(i, tot) sets coef and outputs
    auto meet_sums = [&](int which, auto use) {
      Sum *mine = part + ((size_t)which * 2 + par) * a.cpad;
      c_sync();
      const int i = threadIdx.x;  // nc <= kCThreads
      if (i < nc) {
        Sum v;
        if constexpr (sizeof(T) == 4) {
          float s0 = red[i], e0 = 0.f;
#pragma unroll
          for (int r = 1; r < kWR; ++r) two_add(s0, e0, red[r * a.cpad + i]);
          v = pair(s0, e0);
        } else {
          v = red[i];
#pragma unroll
          for (int r = 1; r < kWR; ++r) v += red[r * a.cpad + i];
        }
        mine[i] = v;
        if (S == 1) use(i, v);
      }
      c_sync();
      if (!met) {
        c_cluster_wait();
        met = true;
      }
      if (S > 1) {
        c_meet_arrive(&sh->meet[which], S);
        c_wait<true>(&sh->meet[which], par, fail, a.status);
        if (i < nc) {
          Sum v = g_sum_of((T)0);
          for (int r0 = 0; r0 < S; r0 += 4) {
            Sum x[4];
#pragma unroll
            for (int r = 0; r < 4; ++r) x[r] = r0 + r < S ? g_load_rank(mine + i, r0 + r) : g_sum_of((T)0);
#pragma unroll
            for (int r = 0; r < 4; ++r) v = g_add(v, x[r]);
          }
          use(i, v);
        }
        c_sync();
      }
    };
    // v += the groups' partial updates (all groups get the sum)
    auto combine = [&](T(&v)[8], const T(&acc)[8]) {
      if constexpr (kWC == 1) {
#pragma unroll
        for (int e = 0; e < 8; ++e) v[e] += acc[e];
      } else {
#pragma unroll
        for (int q = 0; q < NV; ++q)
          if (ok[q]) *reinterpret_cast<Vt *>(comb + (size_t)group * R + rv[q]) = array_to_vec<T>(acc + q * VW);
        c_sync();
        T sum[8];
#pragma unroll
        for (int e = 0; e < 8; ++e) sum[e] = (T)0;
#pragma unroll
        for (int g = 0; g < kWC; ++g) {
          T z[8];
          load_col(comb + (size_t)g * R, true, z);
#pragma unroll
          for (int e = 0; e < 8; ++e) sum[e] += z[e];
        }
#pragma unroll
        for (int e = 0; e < 8; ++e) v[e] += sum[e];
      }
    };

    for (int64_t b = cluster; b < a.p; b += nclusters, par ^= 1u) {
      T v[8], acc[8];
      load_rows(a.W + b * a.ld, v);
#pragma unroll
      for (int e = 0; e < 8; ++e) acc[e] = (T)0;
      const double *Hb = nullptr;
      Sum *Gb = nullptr;
      T beta = (T)1;
      if constexpr (kAdj) {
        const int64_t kk = (int64_t)a.k * a.k;
        Hb = a.H + b * kk;
        Gb = reinterpret_cast<Sum *>(a.Gamma) + b * kk;
        if ((int)threadIdx.x < nc) {
          h_pi[threadIdx.x] = g_from<Sum>(a.Pi[b * kk + (int64_t)a.idx * a.k + threadIdx.x]);
          if (a.idx > 0) dh[threadIdx.x] = g_from<Sum>(a.dH[b * kk + (int64_t)threadIdx.x * a.k + a.idx - 1]);
        }
        for (int i = threadIdx.x; i < nx; i += kCThreads) {
          xcoef[i] = g_round(Gb[(int64_t)(a.idx + 1 + i) * a.k + a.idx]);
          xcoef[nx + i] = (T)(-Hb[(int64_t)a.idx * a.k + a.idx + 1 + i]);
        }
        if (a.idx > 0) beta = (T)Hb[(int64_t)a.idx * a.k + a.idx - 1];
        if (group == 0) {
          const T alpha = (T)Hb[(int64_t)a.idx * a.k + a.idx], gam = (T)a.gamma[b * a.k + a.idx];
          T x[8];
          load_rows(a.lam + b * a.qb, x);
#pragma unroll
          for (int e = 0; e < 8; ++e) acc[e] = -alpha * x[e];
          load_rows(a.res + b * a.ld, x);
#pragma unroll
          for (int e = 0; e < 8; ++e) acc[e] = fma(gam, x[e], acc[e]);
          if (a.dq) {
            load_rows(a.dq + b * a.qb, x);
#pragma unroll
            for (int e = 0; e < 8; ++e) acc[e] += x[e];
          }
        }
        c_sync();
        for (int u = 0; u < gsx; ++u) {
          const bool ready = c_wait(&full[pos], sp, fail, a.status);
          axpy_slot(xcoef, (u * kWC + group) * kGC, 2 * nx, gring + (size_t)pos * kGC * R, ready, acc);
          __syncwarp();
          if (lane == 0 && ready) c_arrive(&empty[pos]);
          next();
        }
      } else if (a.prev) {
        T x[8];
        load_rows(a.prev + b * a.prev_b, x);
        const T c = (T)a.prev_c[b * a.prev_cs];
#pragma unroll
        for (int e = 0; e < 8; ++e) v[e] = fma(-x[e], c, v[e]);
      }

      if (nc > 0) {
        dots(1, v);
        meet_sums(0, [&](int i, Sum t) {  // i == threadIdx.x
          if constexpr (kAdj) {
            const Sum row = g_sub(h_pi[i], t);
            h_pi[i] = g_twice(row, i < a.idx ? (T)1 : (T)0.5);
            coef[i] = g_round(row);
          } else {
            h_pi[i] = t;
            coef[i] = -g_round(t);
          }
        });
        pass(2, [&](int c0, const T *slot, bool ready) { axpy_slot(coef, c0, nc, slot, ready, acc); });
        combine(v, acc);
        if constexpr (kAdj) {
          const T r = (T)1 / beta;
#pragma unroll
          for (int e = 0; e < 8; ++e) v[e] = g_div(v[e], beta, r);
        }
        if (a.passes == 4) {
          dots(3, v);
          meet_sums(1, [&](int i, Sum t) { coef[i] = kAdj ? g_round(g_sub(dh[i], t)) : -g_round(t); });
#pragma unroll
          for (int e = 0; e < 8; ++e) acc[e] = (T)0;
          pass(4, [&](int c0, const T *slot, bool ready) { axpy_slot(coef, c0, nc, slot, ready, acc); });
          combine(v, acc);
        }
      }
      T scale = (T)1, rscale = (T)1;
      bool divide = false;
      if constexpr (!kAdj) {
        if (group == 0) {
          Sum s;
          if constexpr (sizeof(T) == 4) {
            float s0 = 0.f, e0 = 0.f;
#pragma unroll
            for (int e = 0; e < 8; ++e) two_add(s0, e0, v[e] * v[e]);
            s = warp_pair(s0, e0);
          } else {
            s = v[0] * v[0];
#pragma unroll
            for (int e = 1; e < 8; ++e) s = fma(v[e], v[e], s);
            s = warp_sum(s);
          }
          if (lane == 0) wred[wr] = s;
        }
        c_sync();
        if (!met) {
          c_cluster_wait();
          met = true;
        }
        if (warp == 0) {
          if (lane == 0) {
            Sum s = wred[0];
#pragma unroll
            for (int r = 1; r < kWR; ++r) s = g_add(s, wred[r]);
            npart[par] = s;
          }
          __syncwarp();
          c_meet_arrive(&sh->meet[2], S);
          if (S > 1) c_wait<true>(&sh->meet[2], par, fail, a.status);
          Sum s = g_sum_of((T)0);
          if (lane < S) s = S > 1 ? g_load_rank(npart + par, lane) : npart[par];
          for (int o = c_half(S); o > 0; o >>= 1) s = g_add(s, g_xor(s, o));
          if (lane == 0) *fin = g_sqrt(s);
        }
        c_sync();
        scale = g_round(*fin);
        rscale = (T)1 / scale;
        divide = true;
      } else if (a.out_scale) {
        scale = (T)a.out_scale[b];
      }
      if (group == 0) {
#pragma unroll
        for (int q = 0; q < NV; ++q) {
          if (!ok[q]) continue;
          const int64_t r = r0 + rv[q];
          if (!kAdj && a.w_out) *reinterpret_cast<Vt *>(a.w_out + b * a.ld + r) = array_to_vec<T>(v + q * VW);
          if (!a.next) continue;
          T y[VW];
#pragma unroll
          for (int e = 0; e < VW; ++e) y[e] = divide ? g_div(v[q * VW + e], scale, rscale) : v[q * VW + e] * scale;
          *reinterpret_cast<Vt *>(a.next + b * a.next_b + r) = array_to_vec<T>(y);
          if constexpr (sizeof(T) == 4) {
            if (a.hi) {
              uint32_t hv[4], lv[4];
#pragma unroll
              for (int e = 0; e < 4; ++e) {
                const __nv_bfloat16 h = __float2bfloat16_rn(y[e]);
                hv[e] = __bfloat16_as_ushort(h);
                lv[e] = __bfloat16_as_ushort(__float2bfloat16_rn(y[e] - __bfloat162float(h)));
              }
              *reinterpret_cast<uint2 *>(a.hi + b * a.ld + r) = make_uint2(hv[0] | (hv[1] << 16), hv[2] | (hv[3] << 16));
              if (a.lo)
                *reinterpret_cast<uint2 *>(a.lo + b * a.ld + r) = make_uint2(lv[0] | (lv[1] << 16), lv[2] | (lv[3] << 16));
            }
          }
        }
      }
      if (rank == 0) {  // what the next step does not wait for
        if ((int)threadIdx.x < nc) {
          if constexpr (kAdj)
            Gb[(int64_t)a.idx * a.k + threadIdx.x] = h_pi[threadIdx.x];
          else
            a.h[b * a.h_bs + threadIdx.x * a.h_is] = g_double(h_pi[threadIdx.x]);
        }
        if (!kAdj && threadIdx.x == 0) {
          const double nv = g_double(*fin);
          if (a.norm) a.norm[b] = nv;
          if (a.norm2) a.norm2[b * a.norm2_bs] = nv;
        }
      }
    }
    c_done(S);
  }
}

// ---------------------------------------------------------------------------
// Host side
// ---------------------------------------------------------------------------

template <typename T> constexpr int g_gc(int wr) { return wr == 8 ? 2 : 4; }

template <typename T, bool kAdj>
static auto g_kernel(int wr) -> void (*)(const GsArgs<T>) {
  switch (wr) {
    case 1: return gs_cluster_kernel<T, 1, 4, kAdj>;
    case 2: return gs_cluster_kernel<T, 2, 4, kAdj>;
    case 4: return gs_cluster_kernel<T, 4, 4, kAdj>;
    default: return gs_cluster_kernel<T, 8, 2, kAdj>;
  }
}

// the current device's counts (its kernels prepared with them); null: not to be had
template <typename T, bool kAdj>
static const CSlots *g_slots() {
  static PerDevice<CSlots> table;
  return table.get(current_device(), [](CSlots &t) {
    for (int w = 0; w < 4; ++w)
      if (!c_count_clusters(g_kernel<T, kAdj>(1 << w), t.clusters[w])) return false;
    return true;
  });
}

struct GPlan {
  int S, R, wr, slots, clusters, cpad, xpad;
};

// CTAs per probe, as for the Arnoldi step: the fewest rounds of probes over the
// clusters the GPU holds, a round costing its meetings and the CTA's passes (40 GB/s
// from L2; float64 also its FMAs, 1.7 a clock and SM for two CTAs).  S = 0: no size
// that the GPU holds has room.
template <typename T>
static GPlan g_plan(const CSlots &slots, int64_t n, int64_t p, int passes, int ncols, int nx) {
  GPlan best{};
  best.cpad = (ncols + 7) / 8 * 8;
  best.xpad = (2 * nx + 7) / 8 * 8;
  const double cols = (double)passes * ncols + 2.0 * nx + 4.0;
  double best_us = 1e300;
  for (int i = 0; i < kCSizes; ++i) {
    const int S = kCSize[i];
    const int64_t R = ceil_div(ceil_div(n, S), 4) * 4;
    if (R > kCMaxR) continue;
    const int w = c_row_warps(R);
    int lw = 0;
    while ((1 << lw) < w) ++lw;
    const int c = slots.clusters[lw][i];
    const size_t slot = (size_t)g_gc<T>(w) * R * sizeof(T), fixed = g_fixed<T>(best.cpad, best.xpad, (int)R, w);
    const int groups = kCWarps / w;
    if (c < 1 || fixed + slot * groups > kCSmem) continue;
    double us = (S == 1 ? 6.0 : 9.0) + 0.15 * S + cols * R * sizeof(T) / 40e3;
    if (sizeof(T) == 8) us += cols * R / 1630.0;
    us = us * (double)ceil_div(p, c) + (S > kCChainS ? kCUnchainedUs : 0.0);
    if (us < best_us) {
      best_us = us;
      best.S = S;
      best.R = (int)R;
      best.wr = w;
      best.clusters = c;
      int sl = (int)((kCSmem - fixed) / slot);
      if (sl > kCMaxSlots) sl = kCMaxSlots;
      best.slots = sl / groups;
    }
  }
  return best;
}

static bool g_limits(int64_t n, int64_t ncols, int64_t nextra) {
  return n <= (int64_t)kCMaxS * kCMaxR && ncols <= kGMaxCols && nextra <= kGMaxCols;
}

// Whether Gram-Schmidt against ncols vectors, or every step of an adjoint of k, has a plan
// on the current device; the separate launches run otherwise.
template <typename T>
bool gs_cluster_applies(int64_t n, int64_t p, int64_t ncols) {
  if (!g_limits(n, ncols, 0)) return false;
  const CSlots *slots = g_slots<T, false>();
  return slots && g_plan<T>(*slots, n, p, 4, (int)ncols, 0).S > 0;
}

template <typename T>
static bool adj_has_plans(const CSlots &slots, int64_t n, int64_t p, int64_t k) {
  if (!g_limits(n, k, 2 * k)) return false;
  for (int idx = 0; idx < (int)k; ++idx)
    if (g_plan<T>(slots, n, p, idx > 0 ? 4 : 2, idx + 1, (int)k - 1 - idx).S == 0) return false;
  return true;
}

template <typename T>
bool adj_cluster_applies(int64_t n, int64_t p, int64_t k) {
  const CSlots *slots = g_slots<T, true>();
  return slots && adj_has_plans<T>(*slots, n, p, k);
}

// The plan for a table of clusters (host only): see mfg_step_plan.
template <typename T>
int gs_plan_query(const CSlots &slots, int64_t n, int64_t p, int64_t ncols, bool adj, int *out) {
  if (adj ? !adj_has_plans<T>(slots, n, p, ncols) : !g_limits(n, ncols, 0)) return 0;
  const GPlan g = adj ? g_plan<T>(slots, n, p, ncols > 1 ? 4 : 2, (int)ncols, 0) : g_plan<T>(slots, n, p, 4, (int)ncols, 0);
  out[0] = g.S;
  out[1] = g.R;
  out[2] = g.wr;
  out[3] = g.slots;
  return g.S;
}

template <typename T, bool kAdj>
static int g_run(GsArgs<T> &a, bool chained, cudaStream_t s) {
  if (a.p <= 0) return MFG_OK;
  const CSlots *slots = g_slots<T, kAdj>();
  const GPlan g = slots ? g_plan<T>(*slots, a.n, a.p, a.passes, a.ncols, kAdj ? a.nx : 0) : GPlan{};
  if (g.S == 0) return MFG_ERR_UNSUPPORTED;
  a.S = g.S;
  a.R = g.R;
  a.slots = g.slots;
  a.cpad = g.cpad;
  a.xpad = g.xpad;
  const size_t smem = g_fixed<T>(a.cpad, a.xpad, a.R, g.wr) +
                      (size_t)a.slots * (kCWarps / g.wr) * g_gc<T>(g.wr) * a.R * sizeof(T);
  return c_launch(g_kernel<T, kAdj>(g.wr), a.S, a.S * (a.p < g.clusters ? a.p : g.clusters), smem, a, chained, s);
}

// w (panel W; w -= prev_c prev first, if given) against basis vectors 0 .. ncols - 1,
// `passes` = 4 (twice) or 2 (once); see GsArgs.
template <typename T>
int launch_gs_cluster(const T *Q, int64_t qb, int64_t ld, int ncols, const T *W, int64_t n, int64_t p, int passes,
                      const T *prev, int64_t prev_b, const double *prev_c, int64_t prev_cs, double *h, int64_t h_bs,
                      int64_t h_is, double *norm, double *norm2, int64_t norm2_bs, T *w_out, T *next, int64_t next_b,
                      __nv_bfloat16 *hi, __nv_bfloat16 *lo, int *status, bool chained, cudaStream_t s) {
  GsArgs<T> a{};
  a.Q = Q;
  a.qb = qb;
  a.ld = ld;
  a.ncols = ncols;
  a.W = W;
  a.n = n;
  a.p = p;
  a.passes = passes;
  a.prev = prev;
  a.prev_b = prev_b;
  a.prev_c = prev_c;
  a.prev_cs = prev_cs;
  a.h = h;
  a.h_bs = h_bs;
  a.h_is = h_is;
  a.norm = norm;
  a.norm2 = norm2;
  a.norm2_bs = norm2_bs;
  a.w_out = w_out;
  a.next = next;
  a.next_b = next_b;
  a.hi = hi;
  a.lo = lo;
  a.status = status;
  return g_run<T, false>(a, chained, s);
}

// Step idx of the adjoint after U = A lambda: row idx of Gamma, and lambda of step
// idx - 1 (reprojected; row idx - 1 of Lambda) or, for idx 0, dv = c lambda.
template <typename T>
int launch_adj_cluster(const T *Q, int64_t qb, int64_t ld, int k, int idx, const T *U, T *Lam, const T *res,
                       const T *dq, const double *H, const double *Pi, const double *dH, const double *gamma,
                       double *Gamma, const double *c, T *dv, int64_t n, int64_t p, __nv_bfloat16 *hi,
                       __nv_bfloat16 *lo, int *status, bool chained, cudaStream_t s) {
  GsArgs<T> a{};
  a.Q = Q;
  a.qb = qb;
  a.ld = ld;
  a.ncols = idx + 1;
  a.W = U;
  a.n = n;
  a.p = p;
  a.passes = idx > 0 ? 4 : 2;
  a.k = k;
  a.idx = idx;
  a.nx = k - 1 - idx;
  a.lam = Lam + (int64_t)idx * ld;
  a.Lam = Lam;
  a.res = res;
  a.dq = dq;
  a.H = H;
  a.Pi = Pi;
  a.dH = dH;
  a.gamma = gamma;
  a.out_scale = idx > 0 ? nullptr : c;
  a.Gamma = Gamma;
  a.next = idx > 0 ? Lam + (int64_t)(idx - 1) * ld : dv;
  a.next_b = idx > 0 ? qb : ld;
  a.hi = idx > 0 ? hi : nullptr;
  a.lo = lo;
  a.status = status;
  return g_run<T, true>(a, chained, s);
}

#define MFG_INST(T)                                                                                               \
  template bool gs_cluster_applies<T>(int64_t, int64_t, int64_t);                                                  \
  template bool adj_cluster_applies<T>(int64_t, int64_t, int64_t);                                                 \
  template int gs_plan_query<T>(const CSlots &, int64_t, int64_t, int64_t, bool, int *);                           \
  template int launch_gs_cluster<T>(const T *, int64_t, int64_t, int, const T *, int64_t, int64_t, int, const T *, \
                                    int64_t, const double *, int64_t, double *, int64_t, int64_t, double *,        \
                                    double *, int64_t, T *, T *, int64_t, __nv_bfloat16 *, __nv_bfloat16 *, int *, \
                                    bool, cudaStream_t);                                                           \
  template int launch_adj_cluster<T>(const T *, int64_t, int64_t, int, int, const T *, T *, const T *, const T *,  \
                                     const double *, const double *, const double *, const double *, double *,    \
                                     const double *, T *, int64_t, int64_t, __nv_bfloat16 *, __nv_bfloat16 *,      \
                                     int *, bool, cudaStream_t);
MFG_INST(float)
MFG_INST(double)
#undef MFG_INST

}  // namespace mfg
