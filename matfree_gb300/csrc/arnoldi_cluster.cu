// One launch per two-sweep Arnoldi step: a cluster of CTAs per probe.
//
// The two-sweep step (see lanczos_kernels.cu) reads the basis twice: for the
// projections of the two vectors q~ and w = A q~, and for their updates.  As
// separate launches over all probes both reads come from HBM, and the two
// vectors, the coefficient algebra and the normalisation cost further passes
// and launches.  Here a cluster of S CTAs takes one probe at a time, CTA r the
// rows [r R, (r + 1) R), and does the whole step:
//
//   1. the copy warp streams the probe's basis rows through a shared-memory
//      ring (slots of GC vectors x R rows); q~ and w stay in registers; the
//      per-thread products go through a warp butterfly per slot;
//   2. the CTAs' float64 partial sums meet over distributed shared memory,
//      every CTA adding all of them in rank order;
//   3. q~ - Q h and w - Q g from the slots still in the ring first, then from
//      the earlier vectors read again (from L2: the probes in flight are chosen
//      to fit it), while the next probe's vectors already arrive;
//   4. the three dot products meet as in 2; every CTA forms the scalars and
//      writes its rows of q_j and of the next q~ with its bf16 copies.
//
// The basis thus crosses HBM once per step, and the two vectors once in and once
// out.  H is not formed here: the raw projections go to the places of H and Hh
// that they end up in, and arnoldi_h_kernel turns them into H once per solve.
// Two CTAs share an SM, so that one streams while the other is between passes.
//
// What bounds it: for few probes the chain of a step (about 8 us: loads, two
// float64 meetings, the scalars), for many the reads (HBM for the first pass, L2
// for the second).  Against the separate launches (projection, update,
// coefficients, finish) per solve: n = 512, k = 16, 32 probes 0.60 -> 0.22 ms;
// n = 3001, k = 32, 64 probes 1.14 -> 0.55 ms; n = 8192, k = 64, 512 probes 16.5 ->
// 11.3 ms; n = 16384, k = 64, 256 probes 15.0 -> 12.1 ms; n = 30000, k = 64, 128
// probes 14.7 -> 13.5 ms.  The separate launches remain for n > 32768, where a
// cluster's registers no longer hold the two vectors.
//
// Sums: products and a warp's sum (256 rows) in float32, warps, CTAs and the
// squared norms in float64 or its two-float equivalent, all in a fixed order.
// Waits are bounded; after a failure a CTA's warps run on without waiting or
// computing, still meeting every barrier, and the copies in flight are drained.

#include "cluster.cuh"
#include "kernels.cuh"

namespace mfg {

constexpr int kCMaxCols = kTwoSweepMaxK - 1;  // basis vectors of a step
static_assert(kCMaxCols == 128, "shared arrays");

struct CStepArgs {
  const float *Q;  // probe stride qb, vector stride ld
  int64_t qb, ld;
  const float *W;
  const float *Vin;  // q~ (first step: q_0), probe stride vb
  int64_t vb;
  float *Qj;    // row j of the basis, probe stride qb (not written in the first step)
  float *Vout;  // next q~, probe stride ld; may be null
  __nv_bfloat16 *hi, *lo;
  int64_t n, p;
  int j, k, R, S, slots;  // slots: of one group's ring
  double *H, *Hh, *nu;  // nu: (p, k + 1), nu_j at [j]
  int *status;
};

struct CShared {
  uint64_t full[kCMaxSlots], empty[kCMaxSlots];
  uint64_t wq_full, wq_empty;
  uint64_t meet[2];  // cluster barriers: the projections', the norms'
  double part[2 * kCMaxCols + 1];  // this CTA's projections [h_i, g_i] and q~ . w (read by the cluster)
  double tot[2 * kCMaxCols + 1];   // the cluster's
  double npart[3];                 // this CTA's ||b'||^2, ||z||^2, b' . z
  double wred[kCWarps][4];
  double hhg[2];  // ||Q^T q~||^2, (Q^T q~) . (Q^T w)
  float red[kCWarps][2 * kCMaxCols];
  float2 coef[kCMaxCols];
  float fin[3];
  int fail;
};

// kWR warps cover the CTA's R <= 256 kWR rows; the 8 / kWR groups of warps take
// the basis slots s in turn (group s % kWC), each group from a ring of its own
// (its warps consume every fill of it in order, so a slot's phases cannot alias).
// kFirst: step 0 (no basis: w - q_0 (q_0 . w), its norm, q~_1).
template <int kWR, int kGC, bool kFirst>
__global__ void __launch_bounds__(kCThreads + 32, 2) arnoldi_step_kernel(const CStepArgs a) {
  constexpr int kWC = kCWarps / kWR;
  extern __shared__ __align__(128) uint8_t c_raw[];
  CShared *sh = reinterpret_cast<CShared *>(c_raw);
  const int R = a.R, S = a.S, nslots = a.slots, j = kFirst ? 0 : a.j;  // slots of a group's ring
  float *wq = reinterpret_cast<float *>(c_raw + (sizeof(CShared) + 127) / 128 * 128);  // [2][R]: w, q~
  float *comb = wq + 2 * R;                                                          // [kWC - 1][2][R]
  float *ring = comb + (kWC - 1) * 2 * R;                                            // [kWC][nslots][kGC][R]
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int rank = S > 1 ? (int)c_rank() : 0;
  const int64_t r0 = (int64_t)rank * R;
  const int nloc = (int)(a.n - r0 < 0 ? 0 : (a.n - r0 < R ? a.n - r0 : R));  // this CTA's rows
  const uint32_t col_bytes = (uint32_t)((nloc + 3) / 4 * 16);
  const int ns = (j + kGC - 1) / kGC;
  const int64_t cluster = blockIdx.x / S, nclusters = gridDim.x / S;
  volatile int *fail = &sh->fail;
  // slots of group g, and how many of them stay in its ring for the second pass
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
      init(&sh->wq_full, 1);
      init(&sh->wq_empty, kCWarps);
      init(&sh->meet[0], (uint32_t)S);
      init(&sh->meet[1], (uint32_t)S);
      sh->fail = 0;
    }
    if (i <= kCMaxSlots) asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  __syncthreads();
  // waited for before the first access to another CTA; the copies start at once
  c_cluster_arrive();
  chain_wait();
  chain_next();

  if (warp == kCWarps) {
    // copy warp: per probe the two vectors, slots 0 .. ns - 1, then every group's
    // slots that did not stay in its ring again.  Lane g counts group g's fills.
    int fills = 0, pos = 0, t = 0;
    uint32_t par = 0;
    bool run = true;
    for (int64_t b = cluster; run && b < a.p; b += nclusters, ++t) {
      if (t > 0) run = c_wait(&sh->wq_empty, (uint32_t)(t - 1) & 1u, fail, a.status);
      if (!run) break;
      if (lane == 0) {
        c_expect(&sh->wq_full, 2u * col_bytes);
        if (col_bytes) {
          c_bulk(c_smem(wq), a.W + b * a.ld + r0, col_bytes, &sh->wq_full);
          c_bulk(c_smem(wq + R), a.Vin + b * a.vb + r0, col_bytes, &sh->wq_full);
        }
      }
      const float *Qb = a.Q + b * a.qb + r0;
      for (int pass = 0; pass < 2 && run; ++pass)
        for (int s = 0; s < ns; ++s) {
          const int g = s % kWC;
          if (pass == 1 && s / kWC >= slots_of(g) - kept_of(g)) continue;
          const int gpos = __shfl_sync(0xffffffffu, pos, g), gfills = __shfl_sync(0xffffffffu, fills, g);
          const uint32_t gpar = __shfl_sync(0xffffffffu, par, g);
          const int at = g * nslots + gpos;
          if (gfills >= nslots && !c_wait(&sh->empty[at], gpar ^ 1u, fail, a.status)) {
            run = false;
            break;
          }
          const int cols = j - s * kGC < kGC ? j - s * kGC : kGC;
          if (lane == 0) c_expect(&sh->full[at], (uint32_t)cols * col_bytes);
          __syncwarp();
          if (lane < cols && col_bytes)
            c_bulk(c_smem(ring + ((size_t)at * kGC + lane) * R), Qb + (int64_t)(s * kGC + lane) * a.ld, col_bytes,
                   &sh->full[at]);
          __syncwarp();
          if (lane == g) {
            ++fills;
            if (++pos == nslots) {
              pos = 0;
              par ^= 1u;
            }
          }
        }
    }
    if (*fail) {
      // copies in flight land (bounded) before the shared memory goes away
      if (lane < kWC)
        for (int f = fills > nslots ? fills - nslots : 0; f < fills; ++f)
          mbar_wait_bounded(c_smem(&sh->full[lane * nslots + f % nslots]), (uint32_t)(f / nslots) & 1u, nullptr,
                            kMbarWaitNs / 8);
      if (lane == 0 && t > 0) mbar_wait_bounded(c_smem(&sh->wq_full), (uint32_t)(t - 1) & 1u, nullptr, kMbarWaitNs / 8);
    }
    c_cluster_wait();
  } else {
    const int wr = warp % kWR, group = warp / kWR;
    const int row = wr * kCRows + lane * 4;  // rows row .. row + 3 and row + 128 .. row + 131
    const bool ok0 = row < nloc, ok1 = row + 128 < nloc;
    const float4 zero4 = make_float4(0.f, 0.f, 0.f, 0.f);
    const int gs = slots_of(group), gk = kept_of(group);
    int pos = 0;  // this group's ring
    uint32_t sp = 0, par = 0;  // parity of the ring's pass; of the probe
    uint64_t *full = sh->full + group * nslots, *empty = sh->empty + group * nslots;
    const float *gring = ring + (size_t)group * nslots * kGC * R + row;
    auto next = [&]() {
      if (++pos == nslots) {
        pos = 0;
        sp ^= 1u;
      }
    };
    bool met = false;  // the cluster's start
    for (int64_t b = cluster; b < a.p; b += nclusters, par ^= 1u) {
      float w[8], q[8];
      bool ready = c_wait(&sh->wq_full, par, fail, a.status);
      {
        auto load = [&](const float *src, float (&x)[8]) {
          const float4 u = ready && ok0 ? *reinterpret_cast<const float4 *>(src + row) : zero4;
          const float4 v = ready && ok1 ? *reinterpret_cast<const float4 *>(src + row + 128) : zero4;
          x[0] = u.x; x[1] = u.y; x[2] = u.z; x[3] = u.w;
          x[4] = v.x; x[5] = v.y; x[6] = v.z; x[7] = v.w;
#pragma unroll
          for (int e = 0; e < 8; ++e)
            if (row + (e < 4 ? e : 124 + e) >= nloc) x[e] = 0.f;  // a panel's padding is not data
        };
        load(wq, w);
        load(wq + R, q);
      }
      __syncwarp();
      if (lane == 0) c_arrive(&sh->wq_empty);

      if (group == 0) {
        float s0 = 0.f, e0 = 0.f;
#pragma unroll
        for (int e = 0; e < 8; ++e) two_add(s0, e0, w[e] * q[e]);
        const double v = warp_sum2(s0, e0);
        if (lane == 0) sh->wred[wr][3] = v;
      }

      // pass 1: q_i . q~ and q_i . w of this group's slots
      int kpos = pos;  // the first slot that stays
      uint32_t ksp = sp;
      for (int u = 0; u < gs; ++u) {
        if (u == gs - gk) {
          kpos = pos;
          ksp = sp;
        }
        ready = c_wait(&full[pos], sp, fail, a.status);
        const float *x = gring + (size_t)pos * kGC * R;
        float v[2 * kGC];
#pragma unroll
        for (int c = 0; c < kGC; ++c) {
          const float4 z = ready && ok0 ? *reinterpret_cast<const float4 *>(x + c * R) : zero4;
          const float4 y = ready && ok1 ? *reinterpret_cast<const float4 *>(x + c * R + 128) : zero4;
          float h = z.x * q[0], g = z.x * w[0];
          h = fmaf(z.y, q[1], h); g = fmaf(z.y, w[1], g);
          h = fmaf(z.z, q[2], h); g = fmaf(z.z, w[2], g);
          h = fmaf(z.w, q[3], h); g = fmaf(z.w, w[3], g);
          h = fmaf(y.x, q[4], h); g = fmaf(y.x, w[4], g);
          h = fmaf(y.y, q[5], h); g = fmaf(y.y, w[5], g);
          h = fmaf(y.z, q[6], h); g = fmaf(y.z, w[6], g);
          h = fmaf(y.w, q[7], h); g = fmaf(y.w, w[7], g);
          v[2 * c] = h;
          v[2 * c + 1] = g;
        }
        __syncwarp();
        if (u < gs - gk && lane == 0 && ready) c_arrive(&empty[pos]);
        int idx;
        const float sum = c_xsum<2 * kGC>(v, lane, idx);
        idx += (u * kWC + group) * 2 * kGC;
        if ((lane & (32 / (2 * kGC) - 1)) == 0 && idx < 2 * j) sh->red[wr][idx] = sum;
        next();
      }
      c_sync();
      double *mine = S > 1 ? sh->part : sh->tot;
      for (int i = threadIdx.x; i < 2 * j + 1; i += kCThreads) {
        if (i < 2 * j) {
          float s0 = sh->red[0][i], e0 = 0.f;
#pragma unroll
          for (int r = 1; r < kWR; ++r) two_add(s0, e0, sh->red[r][i]);
          const double v = (double)s0 + (double)e0;
          mine[i] = v;
          if (S == 1) reinterpret_cast<float *>(sh->coef)[i] = (float)v;
        } else {
          double v = sh->wred[0][3];
#pragma unroll
          for (int r = 1; r < kWR; ++r) v += sh->wred[r][3];
          mine[i] = v;
        }
      }
      c_sync();
      if (!met) {
        c_cluster_wait();
        met = true;
      }
      if (S > 1) {
        c_meet_arrive(&sh->meet[0], S);
        c_wait<true>(&sh->meet[0], par, fail, a.status);
        for (int i = threadIdx.x; i < 2 * j + 1; i += kCThreads) {
          const uint32_t at = c_smem(&sh->part[i]);
          double x[kCMaxS];
#pragma unroll
          for (int r = 0; r < kCMaxS; ++r) x[r] = r < S ? c_ld_f64(c_map(at, (uint32_t)r)) : 0.0;
          double v = x[0];
#pragma unroll
          for (int r = 1; r < kCMaxS; ++r)
            if (r < S) v += x[r];
          sh->tot[i] = v;
          if (i < 2 * j) reinterpret_cast<float *>(sh->coef)[i] = (float)v;
        }
        c_sync();
      }
      if (!kFirst && rank == 0) {
        // the raw projections, where their final values will be: Q^T q~ in column
        // j - 1 of Hh (column-major), Q^T w in column j of H
        double *hh = a.Hh + b * (int64_t)(a.k + 1) * a.k + (int64_t)(j - 1) * (a.k + 1);
        double *hc = a.H + b * (int64_t)a.k * a.k + j;
        for (int i = threadIdx.x; i < 2 * j; i += kCThreads) {
          if (i & 1)
            hc[(int64_t)(i >> 1) * a.k] = sh->tot[i];
          else
            hh[i >> 1] = sh->tot[i];
        }
      }

      // pass 2: q~ - Q h and w - Q g, even and odd vectors summed apart: the
      // slots that stayed, then the others again
      if (kFirst) {
        const float c = (float)sh->tot[0];
#pragma unroll
        for (int e = 0; e < 8; ++e) w[e] = fmaf(-q[e], c, w[e]);
      } else {
        float w1[8], q1[8];
#pragma unroll
        for (int e = 0; e < 8; ++e) {
          w1[e] = q1[e] = 0.f;
          if (group > 0) w[e] = q[e] = 0.f;
        }
        const int after_pos = pos;
        const uint32_t after_sp = sp;
        pos = kpos;
        sp = ksp;
        for (int i = 0; i < gs; ++i) {
          if (i == gk) {
            pos = after_pos;
            sp = after_sp;
          }
          const int u = i < gk ? gs - gk + i : i - gk;
          const int c0 = (u * kWC + group) * kGC;
          ready = c_wait(&full[pos], sp, fail, a.status);
          const float *x = gring + (size_t)pos * kGC * R;
#pragma unroll
          for (int c = 0; c < kGC; ++c) {
            if (c0 + c < j) {
              const float2 cf = sh->coef[c0 + c];
              const float4 z0 = ready && ok0 ? *reinterpret_cast<const float4 *>(x + c * R) : zero4;
              const float4 z1 = ready && ok1 ? *reinterpret_cast<const float4 *>(x + c * R + 128) : zero4;
              const float z[8] = {z0.x, z0.y, z0.z, z0.w, z1.x, z1.y, z1.z, z1.w};
#pragma unroll
              for (int e = 0; e < 8; ++e) {
                if (c & 1) {
                  q1[e] = fmaf(-z[e], cf.x, q1[e]);
                  w1[e] = fmaf(-z[e], cf.y, w1[e]);
                } else {
                  q[e] = fmaf(-z[e], cf.x, q[e]);
                  w[e] = fmaf(-z[e], cf.y, w[e]);
                }
              }
            }
          }
          __syncwarp();
          if (lane == 0 && ready) c_arrive(&empty[pos]);
          next();
        }
        if (gs == gk) {  // nothing was read again
          pos = after_pos;
          sp = after_sp;
        }
#pragma unroll
        for (int e = 0; e < 8; ++e) {
          w[e] += w1[e];
          q[e] += q1[e];
        }
        if (kWC > 1) {
          if (group > 0) {
            float *cw = comb + (size_t)(group - 1) * 2 * R + row;
            if (ok0) {
              *reinterpret_cast<float4 *>(cw) = make_float4(w[0], w[1], w[2], w[3]);
              *reinterpret_cast<float4 *>(cw + R) = make_float4(q[0], q[1], q[2], q[3]);
            }
            if (ok1) {
              *reinterpret_cast<float4 *>(cw + 128) = make_float4(w[4], w[5], w[6], w[7]);
              *reinterpret_cast<float4 *>(cw + R + 128) = make_float4(q[4], q[5], q[6], q[7]);
            }
          }
          c_sync();
          if (group == 0) {
#pragma unroll
            for (int g = 0; g < kWC - 1; ++g) {
              const float *cw = comb + (size_t)g * 2 * R + row;
              const float4 a0 = ok0 ? *reinterpret_cast<const float4 *>(cw) : zero4;
              const float4 b0 = ok0 ? *reinterpret_cast<const float4 *>(cw + R) : zero4;
              const float4 a1 = ok1 ? *reinterpret_cast<const float4 *>(cw + 128) : zero4;
              const float4 b1 = ok1 ? *reinterpret_cast<const float4 *>(cw + R + 128) : zero4;
              w[0] += a0.x; w[1] += a0.y; w[2] += a0.z; w[3] += a0.w;
              w[4] += a1.x; w[5] += a1.y; w[6] += a1.z; w[7] += a1.w;
              q[0] += b0.x; q[1] += b0.y; q[2] += b0.z; q[3] += b0.w;
              q[4] += b1.x; q[5] += b1.y; q[6] += b1.z; q[7] += b1.w;
            }
          }
        }
      }

      // ||b'||^2, ||z||^2, b' . z
      if (group == 0) {
        float s3[3] = {0.f, 0.f, 0.f}, e3[3] = {0.f, 0.f, 0.f};
#pragma unroll
        for (int e = 0; e < 8; ++e) {
          two_add(s3[1], e3[1], w[e] * w[e]);
          if (!kFirst) {
            two_add(s3[0], e3[0], q[e] * q[e]);
            two_add(s3[2], e3[2], q[e] * w[e]);
          }
        }
        double v3[3];
        warp_sum2x3(s3, e3, v3);
        if (lane == 0) {
          sh->wred[wr][0] = v3[0];
          sh->wred[wr][1] = v3[1];
          sh->wred[wr][2] = v3[2];
        }
      }
      if (!kFirst && warp == kCWarps - 1) {
        double hh = 0.0, hg = 0.0;
        for (int i = lane; i < j; i += 32) {
          const double h = sh->tot[2 * i];
          hh = fma(h, h, hh);
          hg = fma(h, sh->tot[2 * i + 1], hg);
        }
        hh = warp_sum(hh);
        hg = warp_sum(hg);
        if (lane == 0) {
          sh->hhg[0] = hh;
          sh->hhg[1] = hg;
        }
      }
      c_sync();
      if (warp == 0) {
        if (lane < 3) {
          double v = sh->wred[0][lane];
#pragma unroll
          for (int r = 1; r < kWR; ++r) v += sh->wred[r][lane];
          sh->npart[lane] = v;
        }
        __syncwarp();
        c_meet_arrive(&sh->meet[1], S);
        if (S > 1) c_wait<true>(&sh->meet[1], par, fail, a.status);
        // lane r holds rank r's sums; a butterfly adds them in a fixed order
        double nb = 0.0, nz = 0.0, bz = 0.0;
        if (lane < S) {
          const uint32_t at = S > 1 ? c_map(c_smem(&sh->npart[0]), (uint32_t)lane) : c_smem(&sh->npart[0]);
          nb = c_ld_f64(at);
          nz = c_ld_f64(at + 8);
          bz = c_ld_f64(at + 16);
        }
        for (int o = S / 2; o > 0; o >>= 1) {
          nz += __shfl_xor_sync(0xffffffffu, nz, o);
          if (!kFirst) {
            nb += __shfl_xor_sync(0xffffffffu, nb, o);
            bz += __shfl_xor_sync(0xffffffffu, bz, o);
          }
        }
        const double c = sh->tot[2 * j];
        if (kFirst) {
          if (lane == 0) {
            const double nu1 = sqrt(nz);
            sh->fin[0] = (float)nu1;
            if (rank == 0) {
              a.H[b * (int64_t)a.k * a.k] = c;
              a.nu[b * (a.k + 1) + 1] = nu1;
            }
          }
        } else {
          // rho = sqrt(nb) = ||w''_{j-1}|| / nu_j, qw = q_j . A q~_j = e / rho, and for
          // y = z - q_j qw:  nb ||y||^2 = nb ||z||^2 - 2 e (b' . z) + e^2 =: d.  Float64
          // divisions and roots are long here (2 FMA a clock and SM): everything
          // comes from 1 / sqrt(nb) and 1 / sqrt(nb d), taken side by side.
          nb = __shfl_sync(0xffffffffu, nb, 0);
          nz = __shfl_sync(0xffffffffu, nz, 0);
          bz = __shfl_sync(0xffffffffu, bz, 0);
          const double e = c - sh->hhg[1], zz = nb * nz;
          double d = fma(e, e, fma(-2.0 * e, bz, zz));
          if (!(d > 1e-12 * zz)) d = zz;
          const double root = rsqrt(lane == 0 ? nb : nb * d);
          const double ir = __shfl_sync(0xffffffffu, root, 0), id = __shfl_sync(0xffffffffu, root, 1);
          if (lane == 0) {
            sh->fin[0] = (float)ir;          // 1 / rho
            sh->fin[1] = (float)(nb * id);   // 1 / ||y||
            sh->fin[2] = (float)(e * id);    // qw / (rho ||y||)
            if (rank == 0) {
              const double hh = sh->hhg[0], nuj = a.nu[b * (a.k + 1) + j];
              if (hh > 0.01 * (hh + nb) && a.status) atomicExch(a.status, (int)MFG_ERR_RETRY);
              double *Hb = a.H + b * (int64_t)a.k * a.k;
              Hb[(int64_t)j * a.k + j - 1] = nuj * (nb * ir);  // beta_j
              Hb[(int64_t)j * a.k + j] = e * ir;               // raw: arnoldi_h_kernel completes it
              a.nu[b * (a.k + 1) + j + 1] = d * id * ir;       // u_{j+1} = y / rho = nu_{j+1} q~_{j+1}
            }
          }
        }
      }
      c_sync();
      if (group == 0) {
        const float f0 = sh->fin[0], f1 = kFirst ? 0.f : sh->fin[1], f2 = kFirst ? 0.f : sh->fin[2];
#pragma unroll
        for (int half = 0; half < 2; ++half) {
          if (half == 0 ? ok0 : ok1) {
            const int64_t r = r0 + row + 128 * half;
            float y[4];
#pragma unroll
            for (int e = 0; e < 4; ++e) {
              const float zz = w[4 * half + e], bb = q[4 * half + e];
              y[e] = kFirst ? zz / f0 : zz * f1 - bb * f2;
            }
            if (!kFirst)
              *reinterpret_cast<float4 *>(a.Qj + b * a.qb + r) =
                  make_float4(q[4 * half] * f0, q[4 * half + 1] * f0, q[4 * half + 2] * f0, q[4 * half + 3] * f0);
            if (a.Vout) {
              *reinterpret_cast<float4 *>(a.Vout + b * a.ld + r) = make_float4(y[0], y[1], y[2], y[3]);
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
                  *reinterpret_cast<uint2 *>(a.lo + b * a.ld + r) =
                      make_uint2(lv[0] | (lv[1] << 16), lv[2] | (lv[3] << 16));
              }
            }
          }
        }
      }
    }
  }
  // no CTA leaves while the others may read its sums or arrive on its barriers
  c_cluster_arrive();
  c_cluster_wait();
}

// ---------------------------------------------------------------------------
// H from the raw projections that the step kernels left: with hq = Q^T q~_j
// (column j - 1 of Hh), g = Q^T w (column j of H) and qw (H[j][j]),
//   Hh[:, j - 1] = H[:, j - 1] + nu_j hq (rows < j), beta_j in row j
//   H[:, j] = (nu_j [g; qw] - Hh[0 : j + 1, 0 : j] hq) / beta_j
// for j = 1 .. k - 1.  One CTA per probe keeps Hh in shared memory; a row's sum
// over the columns is cut in four.  With `band` only the tridiagonal part is
// formed (all that the quadrature reads): Hh is upper Hessenberg, so rows j - 1
// and j of the product have two terms and one, and the steps are independent.
// ---------------------------------------------------------------------------

__global__ void arnoldi_h_kernel(double *__restrict__ H, const double *__restrict__ Hh,
                                 const double *__restrict__ nu, int k, double *__restrict__ nu_last_inv) {
  extern __shared__ double hs[];  // Hh, column-major with k + 1 rows; then hq, partial sums
  const int64_t b = blockIdx.x;
  double *Hb = H + b * (int64_t)k * k;
  const double *raw = Hh + b * (int64_t)(k + 1) * k;
  const double *nub = nu + b * (k + 1);
  const int ld = k + 1, rows = blockDim.x / 4;
  double *hq = hs + (size_t)ld * k, *part = hq + k;  // part: [4][rows]
  const int i = threadIdx.x % rows, quarter = threadIdx.x / rows;
  double hlast = i == 0 ? Hb[0] : 0.0;  // H[i][j - 1] (quarter 0)
  for (int j = 1; j < k; ++j) {
    const double nuj = nub[j], beta = Hb[(int64_t)j * k + j - 1];
    if (quarter == 0 && i <= j) {
      const double h = i < j ? raw[(int64_t)(j - 1) * ld + i] : 0.0;
      if (i < j) hq[i] = h;
      hs[(size_t)(j - 1) * ld + i] = i < j ? hlast + nuj * h : beta;
    }
    const double top = (quarter == 0 && i <= j) ? Hb[(int64_t)i * k + j] : 0.0;
    __syncthreads();
    if (i <= j) {
      // columns max(i - 1, 0) .. j - 1 of row i, a quarter of them
      const int l0 = i > 0 ? i - 1 : 0, cnt = j - l0;
      const int lb = l0 + cnt * quarter / 4, le = l0 + cnt * (quarter + 1) / 4;
      double m = 0.0;
      for (int l = lb; l < le; ++l) m = fma(hs[(size_t)l * ld + i], hq[l], m);
      part[quarter * rows + i] = m;
    }
    __syncthreads();
    if (quarter == 0 && i <= j) {
      const double m = (part[i] + part[rows + i]) + (part[2 * rows + i] + part[3 * rows + i]);
      hlast = nuj * (top - m) / beta;
      Hb[(int64_t)i * k + j] = hlast;
    }
  }
  if (threadIdx.x == 0 && nu_last_inv) nu_last_inv[b] = 1.0 / nub[k];
}

__global__ void arnoldi_h_band_kernel(double *__restrict__ H, const double *__restrict__ Hh,
                                      const double *__restrict__ nu, int k) {
  const int64_t b = blockIdx.x;
  const int j = threadIdx.x + 1;
  double *Hb = H + b * (int64_t)k * k;
  const double *raw = Hh + b * (int64_t)(k + 1) * k, *nub = nu + b * (k + 1);
  double up = 0.0, diag = 0.0;
  if (j < k) {
    auto beta = [&](int i) { return Hb[(int64_t)i * k + i - 1]; };             // of step i >= 1
    auto hq = [&](int i, int r) { return raw[(int64_t)(i - 1) * (k + 1) + r]; };  // row r of Q^T q~_i
    auto diag_of = [&](int i) {
      return i == 0 ? Hb[0] : nub[i] * (Hb[(int64_t)i * k + i] - beta(i) * hq(i, i - 1)) / beta(i);
    };
    const double nuj = nub[j], bj = beta(j), h1 = hq(j, j - 1);
    double m = (diag_of(j - 1) + nuj * h1) * h1;
    if (j > 1) m = fma(beta(j - 1), hq(j, j - 2), m);
    up = nuj * (Hb[(int64_t)(j - 1) * k + j] - m) / bj;
    diag = diag_of(j);
  }
  __syncthreads();  // every raw value has been read
  if (j < k) {
    Hb[(int64_t)(j - 1) * k + j] = up;
    Hb[(int64_t)j * k + j] = diag;
  }
}

// ---------------------------------------------------------------------------
// Host side
// ---------------------------------------------------------------------------

bool arnoldi_cluster_applies(int64_t n) { return n <= (int64_t)kCMaxS * kCMaxR; }

static int c_gc(int wr) { return wr >= 4 ? 2 : 4; }

using CKernel = void (*)(const CStepArgs);

template <bool kFirst>
static CKernel c_kernel(int wr) {
  switch (wr) {
    case 1: return arnoldi_step_kernel<1, 4, kFirst>;
    case 2: return arnoldi_step_kernel<2, 4, kFirst>;
    case 4: return arnoldi_step_kernel<4, 2, kFirst>;
    default: return arnoldi_step_kernel<8, 2, kFirst>;
  }
}

static size_t c_fixed(int R, int wr) {
  return (sizeof(CShared) + 127) / 128 * 128 + (size_t)(2 * R + (kCWarps / wr - 1) * 2 * R) * 4;
}

// clusters held at a time, per log2 of the row warps
struct CSlots {
  int clusters[4][5];
  CSlots() {
    for (int w = 0; w < 4; ++w) {
      c_prepare(c_kernel<true>(1 << w));
      c_count_clusters(c_kernel<false>(1 << w), clusters[w]);
    }
  }
};

struct CPlan {
  int S, R, wr, slots, clusters;
};

// CTAs per probe: the fewest rounds of probes over the clusters the GPU holds
// (S = 1, 2, 4, 8, 16: 304, 152, 74, 36, 14 on a GB300), a round costing its
// latency (the meetings of a cluster add about 1.5 us) and the CTA's rows at
// 40 GB/s.  Measured, whole solves' steps: n = 512, 256 probes S = 1 193 us
// (2: 353, 4: 572); n = 3001, 64 probes S = 4 550 us (2: 596, 8: 788); n = 8192,
// 128 probes S = 4 2.15 ms (8: 2.87); n = 16384, 256 probes S = 8 12.1 ms (16: 18.9,
// whose clusters leave a quarter of the SMs over).
static CPlan c_plan(int64_t n, int64_t p, int j) {
  static const CSlots slots;
  CPlan best{0, 0, 0, 0, 0};
  double best_us = 1e300;
  for (int i = 0; i < 5; ++i) {
    const int S = 1 << i;
    const int64_t R = ceil_div(ceil_div(n, S), 4) * 4;
    if (R > kCMaxR) continue;
    const int wr = c_row_warps(R);
    int w = 0;
    while ((1 << w) < wr) ++w;
    const int c = slots.clusters[w][i];
    if (c < 1) continue;
    const double rounds = (double)ceil_div(p, c);
    if (c_fixed((int)R, wr) + (size_t)(kCWarps / wr) * c_gc(wr) * R * 4 > kCSmem) continue;  // no slot per group
    const double us = rounds * ((S == 1 ? 5.0 : 6.5) + 0.1 * S + (2.0 * j + 8.0) * R * 4.0 / 40e3);
    if (us < best_us) {
      best_us = us;
      int sl = (int)((kCSmem - c_fixed((int)R, wr)) / ((size_t)c_gc(wr) * R * 4));
      if (sl > kCMaxSlots) sl = kCMaxSlots;
      sl /= kCWarps / wr;  // per group of warps
      best = CPlan{S, (int)R, wr, sl, c};
    }
  }
  return best;
}

// Step j of the two-sweep iteration for every probe (j = 0: the first step).
// Q: the basis (probe stride qb, vector stride ld); W = A q~_j; Vin: q~_j with
// probe stride vb (j = 0: row 0 of Q).  Writes row j of Q (j > 0), the next q~
// into Vout with its bf16 copies (null: not formed), the raw projections into H
// and Hh, nu_{j+1}.
int launch_arnoldi_step(int j, int64_t k, int64_t n, int64_t p, float *Q, int64_t qb, int64_t ld, const float *W,
                        const float *Vin, int64_t vb, float *Vout, __nv_bfloat16 *hi, __nv_bfloat16 *lo, double *H,
                        double *Hh, double *nu, int *status, bool chained, cudaStream_t s) {
  if (p <= 0) return MFG_OK;
  const CPlan plan = c_plan(n, p, j);
  if (plan.S == 0 || j > kCMaxCols) return MFG_ERR_UNSUPPORTED;
  CStepArgs a;
  a.Q = Q;
  a.qb = qb;
  a.ld = ld;
  a.W = W;
  a.Vin = Vin;
  a.vb = vb;
  a.Qj = Q + (int64_t)j * ld;
  a.Vout = Vout;
  a.hi = hi;
  a.lo = lo;
  a.n = n;
  a.p = p;
  a.j = j;
  a.k = (int)k;
  a.R = plan.R;
  a.S = plan.S;
  a.slots = plan.slots;
  a.H = H;
  a.Hh = Hh;
  a.nu = nu;
  a.status = status;
  auto kern = j == 0 ? c_kernel<true>(plan.wr) : c_kernel<false>(plan.wr);
  const size_t smem = c_fixed(plan.R, plan.wr) + (size_t)plan.slots * (kCWarps / plan.wr) * c_gc(plan.wr) * plan.R * 4;
  return c_launch(kern, plan.S, plan.S * (p < plan.clusters ? p : plan.clusters), smem, a, chained, s);
}

// H of every probe from what the steps left (`band`: its tridiagonal part only);
// nu_last_inv (optional): 1 / nu_k.
int launch_arnoldi_h(int64_t k, int64_t p, double *H, const double *Hh, const double *nu, bool band,
                     double *nu_last_inv, cudaStream_t s) {
  if (p <= 0 || k < 2) return MFG_OK;
  const int rows = (int)ceil_div(k, 32) * 32;
  if (band) {
    arnoldi_h_band_kernel<<<(unsigned)p, rows, 0, s>>>(H, Hh, nu, (int)k);
    return MFG_LAUNCH_STATUS();
  }
  const size_t smem = ((size_t)(k + 1) * k + k + 4 * (size_t)rows) * sizeof(double);
  MFG_CUDA_TRY(cudaFuncSetAttribute(arnoldi_h_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  arnoldi_h_kernel<<<(unsigned)p, 4 * rows, smem, s>>>(H, Hh, nu, (int)k, nu_last_inv);
  return MFG_LAUNCH_STATUS();
}

}  // namespace mfg
