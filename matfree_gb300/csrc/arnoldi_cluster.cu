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
//   2. the CTAs' two-float partial sums meet over distributed shared memory,
//      every CTA adding all of them in rank order;
//   3. q~ - Q h and w - Q g from the slots still in the ring first, then from
//      the earlier vectors read again (from L2: the probes in flight are chosen
//      to fit it), while the next probe's vectors already arrive;
//   4. the three dot products meet as in 2; every CTA forms the scalars and
//      writes its rows of q_j and of the next q~ with its bf16 copies.
//
// The basis thus crosses HBM once per step, and the two vectors once in and once
// out.  H is not formed here: the raw projections go to the places of H and Hh
// that they end up in, the step's scalars to rec, and arnoldi_h_kernel turns them
// into H in float64 once per solve.
// Two CTAs share an SM, so that one streams while the other is between passes.
//
// What bounds it: for few probes the chain of a step (about 8 us: loads, two
// meetings, the scalars), for many the reads (HBM for the first pass, L2
// for the second).  Against the separate launches (projection, update,
// coefficients, finish) per solve: n = 512, k = 16, 32 probes 0.60 -> 0.22 ms;
// n = 3001, k = 32, 64 probes 1.14 -> 0.55 ms; n = 8192, k = 64, 512 probes 16.5 ->
// 11.3 ms; n = 16384, k = 64, 256 probes 15.0 -> 12.1 ms; n = 30000, k = 64, 128
// probes 14.7 -> 13.5 ms.  The separate launches remain for n > 32768, where a
// cluster's registers no longer hold the two vectors.
//
// Sums: products and a warp's sum (256 rows) in float32, warps, CTAs, the squared norms
// and the scalars formed from them as two-float numbers, all in a fixed order.
// Waits are bounded; after a failure a CTA's warps run on without waiting or
// computing, still meeting every barrier, and the copies in flight are drained.

#include "cluster.cuh"
#include "kernels.cuh"

namespace mfg {

constexpr int kCMaxCols = kTwoSweepMaxK - 1;  // basis vectors of a step
static_assert(kCMaxCols == 128, "shared arrays");

constexpr int kCRec = kTwoSweepRec;

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
  // two-float numbers: the projections where H and Hh have their places, and kCRec
  // numbers a step in rec: ||b'||^2, ||z||^2, b' . z, q~ . w, (Q^T q~) . (Q^T w)
  float2 *H, *Hh, *rec;
  int *status;
};

struct CShared {
  uint64_t full[kCMaxSlots], empty[kCMaxSlots];
  uint64_t wq_full, wq_empty;
  uint64_t meet[2];  // cluster barriers: the projections', the norms'
  float2 part[2 * kCMaxCols + 1];  // this CTA's projections [h_i, g_i] and q~ . w (read by the cluster)
  float2 tot[2 * kCMaxCols + 1];   // the cluster's
  float2 npart[3];                 // this CTA's ||b'||^2, ||z||^2, b' . z
  float2 wred[kCWarps][4];
  float2 hhg[2];  // ||Q^T q~||^2, (Q^T q~) . (Q^T w)
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
  if (S > 1) c_cluster_arrive();
  chain_wait();
  chain_next();

  if (warp == kCWarps) {
    // copy warp: per probe the two vectors (the first probe's are loaded directly),
    // slots 0 .. ns - 1, then every group's slots that did not stay in its ring
    // again.  Lane g counts group g's fills.
    int fills = 0, pos = 0, wq_fills = 0;
    uint32_t par = 0;
    bool run = true;
    for (int64_t b = cluster; run && b < a.p; b += nclusters) {
      if (b != cluster) {
        if (wq_fills > 0) run = c_wait(&sh->wq_empty, (uint32_t)(wq_fills - 1) & 1u, fail, a.status);
        if (!run) break;
        if (lane == 0) {
          c_expect(&sh->wq_full, 2u * col_bytes);
          if (col_bytes) {
            c_bulk(c_smem(wq), a.W + b * a.ld + r0, col_bytes, &sh->wq_full);
            c_bulk(c_smem(wq + R), a.Vin + b * a.vb + r0, col_bytes, &sh->wq_full);
          }
        }
        ++wq_fills;
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
    if (S > 1) c_cluster_wait();
    c_done(S);
    if (*fail) {
      // copies in flight land (bounded) before the shared memory goes away
      if (lane < kWC)
        for (int f = fills > nslots ? fills - nslots : 0; f < fills; ++f)
          mbar_wait_bounded(c_smem(&sh->full[lane * nslots + f % nslots]), (uint32_t)(f / nslots) & 1u, nullptr,
                            kMbarWaitNs / 8);
      if (lane == 0 && wq_fills > 0)
        mbar_wait_bounded(c_smem(&sh->wq_full), (uint32_t)(wq_fills - 1) & 1u, nullptr, kMbarWaitNs / 8);
    }
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
    bool met = S == 1;  // the cluster's start
    uint32_t wq_par = 0;
    for (int64_t b = cluster; b < a.p; b += nclusters, par ^= 1u) {
      float w[8], q[8];
      bool ready = true;
      {
        auto take = [&](const float4 &u, const float4 &v, float (&x)[8]) {
          x[0] = u.x; x[1] = u.y; x[2] = u.z; x[3] = u.w;
          x[4] = v.x; x[5] = v.y; x[6] = v.z; x[7] = v.w;
#pragma unroll
          for (int e = 0; e < 8; ++e)
            if (row + (e < 4 ? e : 124 + e) >= nloc) x[e] = 0.f;  // a panel's padding is not data
        };
        if (b == cluster) {  // a read of L2 is shorter than a copy's round trip
          const float *gw = a.W + b * a.ld + r0 + row, *gq = a.Vin + b * a.vb + r0 + row;
          const float4 w0 = ok0 ? c_ld_l2(gw) : zero4, q0 = ok0 ? c_ld_l2(gq) : zero4;
          const float4 w1 = ok1 ? c_ld_l2(gw + 128) : zero4, q1 = ok1 ? c_ld_l2(gq + 128) : zero4;
          take(w0, w1, w);
          take(q0, q1, q);
        } else {
          ready = c_wait(&sh->wq_full, wq_par, fail, a.status);
          wq_par ^= 1u;
          const float4 *sw = reinterpret_cast<const float4 *>(wq + row), *sq = reinterpret_cast<const float4 *>(wq + R + row);
          take(ready && ok0 ? sw[0] : zero4, ready && ok1 ? sw[32] : zero4, w);
          take(ready && ok0 ? sq[0] : zero4, ready && ok1 ? sq[32] : zero4, q);
          __syncwarp();
          if (lane == 0) c_arrive(&sh->wq_empty);
        }
      }

      if (group == 0) {
        float s0 = 0.f, e0 = 0.f;
#pragma unroll
        for (int e = 0; e < 8; ++e) two_add(s0, e0, w[e] * q[e]);
        const float2 v = warp_pair(s0, e0);
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
      float2 *mine = S > 1 ? sh->part : sh->tot;
      for (int i = threadIdx.x; i < 2 * j + 1; i += kCThreads) {
        float2 v;
        if (i < 2 * j) {
          float s0 = sh->red[0][i], e0 = 0.f;
#pragma unroll
          for (int r = 1; r < kWR; ++r) two_add(s0, e0, sh->red[r][i]);
          v = pair(s0, e0);
          if (S == 1) reinterpret_cast<float *>(sh->coef)[i] = v.x;
        } else {
          v = sh->wred[0][3];
#pragma unroll
          for (int r = 1; r < kWR; ++r) v = pair_add(v, sh->wred[r][3]);
        }
        mine[i] = v;
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
          float2 x[kCMaxS];
#pragma unroll
          for (int r = 0; r < kCMaxS; ++r)
            if (r < S) x[r] = c_ld_pair(c_map(at, (uint32_t)r));
          float2 v = x[0];
#pragma unroll
          for (int r = 1; r < kCMaxS; ++r)
            if (r < S) v = pair_add(v, x[r]);
          sh->tot[i] = v;
          if (i < 2 * j) reinterpret_cast<float *>(sh->coef)[i] = v.x;
        }
        c_sync();
      }

      // pass 2: q~ - Q h and w - Q g, even and odd vectors summed apart: the
      // slots that stayed, then the others again
      if (kFirst) {
        const float c = sh->tot[0].x;
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
#pragma unroll
        for (int o = 16; o > 0; o >>= 1)
#pragma unroll
          for (int i = 0; i < 3; ++i) {
            const float s2 = __shfl_xor_sync(0xffffffffu, s3[i], o), e2 = __shfl_xor_sync(0xffffffffu, e3[i], o);
            two_add(s3[i], e3[i], s2);
            e3[i] += e2;
          }
        if (lane == 0) {
#pragma unroll
          for (int i = 0; i < 3; ++i) sh->wred[wr][i] = pair(s3[i], e3[i]);
        }
      }
      if (!kFirst && warp == kCWarps - 1) {
        float2 hh = make_float2(0.f, 0.f), hg = hh;
        for (int i = lane; i < j; i += 32) {
          const float2 h = sh->tot[2 * i];
          hh = pair_add(hh, pair_mul(h, h));
          hg = pair_add(hg, pair_mul(h, sh->tot[2 * i + 1]));
        }
        hh = warp_pair(hh.x, hh.y);
        hg = warp_pair(hg.x, hg.y);
        if (lane == 0) {
          sh->hhg[0] = hh;
          sh->hhg[1] = hg;
        }
      }
      c_sync();
      if (warp == 0) {
        if (lane < 3) {
          float2 v = sh->wred[0][lane];
#pragma unroll
          for (int r = 1; r < kWR; ++r) v = pair_add(v, sh->wred[r][lane]);
          sh->npart[lane] = v;
        }
        __syncwarp();
        c_meet_arrive(&sh->meet[1], S);
        if (S > 1) c_wait<true>(&sh->meet[1], par, fail, a.status);
        // lane r holds rank r's sums; a butterfly adds them in a fixed order
        float2 nb = make_float2(0.f, 0.f), nz = nb, bz = nb;
        if (lane < S) {
          const uint32_t at = S > 1 ? c_map(c_smem(&sh->npart[0]), (uint32_t)lane) : c_smem(&sh->npart[0]);
          nb = c_ld_pair(at);
          nz = c_ld_pair(at + 8);
          bz = c_ld_pair(at + 16);
        }
        for (int o = c_half(S); o > 0; o >>= 1) {
          nz = pair_add(nz, pair_shfl_xor(nz, o));
          if (!kFirst) {
            nb = pair_add(nb, pair_shfl_xor(nb, o));
            bz = pair_add(bz, pair_shfl_xor(bz, o));
          }
        }
        auto first_lane = [](float2 v) {
          return make_float2(__shfl_sync(0xffffffffu, v.x, 0), __shfl_sync(0xffffffffu, v.y, 0));
        };
        nb = first_lane(nb);
        nz = first_lane(nz);
        bz = first_lane(bz);
        const float2 c = sh->tot[2 * j];
        float2 hg = make_float2(0.f, 0.f);
        if (kFirst) {
          // nu_1 = ||z||, to a float from the root's remainder
          const float r = sqrtf(nz.x);
          if (lane == 0) sh->fin[0] = r > 0.f ? r + (fmaf(-r, r, nz.x) + nz.y) / (2.f * r) : r;
        } else {
          // rho = sqrt(nb) = ||w''_{j-1}|| / nu_j, qw = q_j . A q~_j = e / rho, and for
          // y = z - q_j qw:  nb ||y||^2 = nb ||z||^2 - 2 e (b' . z) + e^2 =: d
          hg = sh->hhg[1];
          const float2 e = pair_add(c, pair_neg(hg)), zz = pair_mul(nb, nz), eb = pair_mul(e, bz);
          float2 d = pair_add(pair_add(zz, make_float2(-2.f * eb.x, -2.f * eb.y)), pair_mul(e, e));
          if (!(d.x > 1e-12f * zz.x)) d = zz;
          const float2 ir = pair_rsqrt(nb), id = pair_rsqrt(pair_mul(nb, d));
          if (lane == 0) {
            sh->fin[0] = ir.x;                  // 1 / rho
            sh->fin[1] = pair_mul(nb, id).x;    // 1 / ||y||
            sh->fin[2] = pair_mul(e, id).x;     // qw / (rho ||y||)
            const float hh = sh->hhg[0].x;
            if (rank == 0 && hh > 0.01f * (hh + nb.x) && a.status) atomicExch(a.status, (int)MFG_ERR_RETRY);
          }
        }
        if (lane < kCRec && rank == 0)
          a.rec[(b * a.k + j) * kCRec + lane] = lane == 0 ? nb : (lane == 1 ? nz : (lane == 2 ? bz : (lane == 3 ? c : hg)));
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
      if (!kFirst && rank == 0) {
        // the raw projections, where their final values will be: Q^T q~ in column
        // j - 1 of Hh (column-major), Q^T w in column j of H
        float2 *hh = a.Hh + b * (int64_t)(a.k + 1) * a.k + (int64_t)(j - 1) * (a.k + 1);
        float2 *hc = a.H + b * (int64_t)a.k * a.k + j;
        for (int i = threadIdx.x; i < 2 * j; i += kCThreads) {
          if (i & 1)
            hc[(int64_t)(i >> 1) * a.k] = sh->tot[i];
          else
            hh[i >> 1] = sh->tot[i];
        }
      }
    }
    c_done(S);
  }
}

// ---------------------------------------------------------------------------
// H from what the step kernels left as two-float numbers: hq = Q^T q~_j (column j - 1
// of Hh), g = Q^T w (column j of H), and of step j (rec) nb = ||b'||^2, nz = ||z||^2,
// bz = b' . z, c = q~ . w, hg = hq . g:
//   rho = sqrt(nb), qw = (c - hg) / rho, nu_{j+1} = ||z - qw b' / rho|| / rho,
//   Hh[:, j - 1] = H[:, j - 1] + nu_j hq (rows < j), beta_j = nu_j rho in row j
//   H[:, j] = (nu_j [g; qw] - Hh[0 : j + 1, 0 : j] hq) / beta_j
// for j = 1 .. k - 1, and H[0][0] = c, nu_1 = ||z|| of step 0.  One CTA per probe; the
// full form keeps Hh in shared memory and cuts a row's sum over the columns in
// four.  With `band` only the tridiagonal part is formed (all that the quadrature
// reads): Hh is upper Hessenberg, so rows j - 1 and j of the product have two terms
// and one, and the steps are independent.
// ---------------------------------------------------------------------------

__device__ __forceinline__ double h_raw(const double *p) {
  const float2 v = *reinterpret_cast<const float2 *>(p);
  return (double)v.x + (double)v.y;
}

// beta[1 .. k - 1], qw[0 .. k - 1] (qw[0] = H[0][0]) and nu[1 .. k] of one probe, by all threads
__device__ __forceinline__ void h_scalars(const double *rec, int k, double *beta, double *qw, double *nu) {
  for (int j = threadIdx.x; j < k; j += blockDim.x) {
    const double *r = rec + (int64_t)j * kCRec;
    const double nz = h_raw(r + 1), c = h_raw(r + 3);
    if (j == 0) {
      qw[0] = c;
      nu[1] = sqrt(nz);
    } else {
      const double nb = h_raw(r), bz = h_raw(r + 2), e = c - h_raw(r + 4), zz = nb * nz;
      double d = fma(e, e, fma(-2.0 * e, bz, zz));
      if (!(d > 1e-12 * zz)) d = zz;
      const double ir = rsqrt(nb), id = rsqrt(nb * d);
      beta[j] = nb * ir;
      qw[j] = e * ir;
      nu[j + 1] = d * id * ir;
    }
  }
  __syncthreads();
  for (int j = threadIdx.x; j < k; j += blockDim.x)
    if (j > 0) beta[j] *= nu[j];
  __syncthreads();
}

__global__ void arnoldi_h_kernel(double *H, const double *Hh, const double *rec, int k, double *__restrict__ nu_last_inv) {
  chain_wait();
  chain_next();
  extern __shared__ double hs[];  // Hh, column-major with k + 1 rows; then hq, partial sums, the steps' scalars
  const int64_t b = blockIdx.x;
  double *Hb = H + b * (int64_t)k * k;
  const double *raw = Hh + b * (int64_t)(k + 1) * k;
  const int ld = k + 1, rows = blockDim.x / 4;
  double *hq = hs + (size_t)ld * k, *part = hq + k;  // part: [4][rows]
  double *beta = part + 4 * rows, *qw = beta + k, *nu = qw + k;
  h_scalars(rec + b * k * kCRec, k, beta, qw, nu);
  const int i = threadIdx.x % rows, quarter = threadIdx.x / rows;
  double hlast = i == 0 ? qw[0] : 0.0;  // H[i][j - 1] (quarter 0)
  if (threadIdx.x == 0) Hb[0] = qw[0];
  // the raw values of step j, read a step ahead
  double hraw = 0.0, traw = 0.0;
  auto fetch = [&](int j) {
    if (quarter == 0 && i < j && j < k) {
      hraw = h_raw(raw + (int64_t)(j - 1) * ld + i);
      traw = h_raw(Hb + (int64_t)i * k + j);
    }
  };
  fetch(1);
  for (int j = 1; j < k; ++j) {
    const double nuj = nu[j], bj = beta[j];
    double top = 0.0;
    if (quarter == 0 && i <= j) {
      const double h = i < j ? hraw : 0.0;
      if (i < j) hq[i] = h;
      hs[(size_t)(j - 1) * ld + i] = i < j ? hlast + nuj * h : bj;
      top = i < j ? traw : qw[j];
    }
    fetch(j + 1);
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
      hlast = nuj * (top - m) / bj;
      Hb[(int64_t)i * k + j] = hlast;
      if (i == j) Hb[(int64_t)j * k + j - 1] = bj;
    }
  }
  if (threadIdx.x == 0 && nu_last_inv) nu_last_inv[b] = 1.0 / nu[k];
}

__global__ void arnoldi_h_band_kernel(double *H, const double *Hh, const double *rec, int k) {
  chain_wait();
  chain_next();
  __shared__ double beta[kCMaxCols + 1], qw[kCMaxCols + 1], nu[kCMaxCols + 2];
  const int64_t b = blockIdx.x;
  const int j = threadIdx.x + 1;
  double *Hb = H + b * (int64_t)k * k;
  const double *raw = Hh + b * (int64_t)(k + 1) * k;
  h_scalars(rec + b * k * kCRec, k, beta, qw, nu);
  double up = 0.0, diag = 0.0;
  if (j < k) {
    auto hq = [&](int i, int r) { return h_raw(raw + (int64_t)(i - 1) * (k + 1) + r); };  // row r of Q^T q~_i
    auto diag_of = [&](int i) { return i == 0 ? qw[0] : nu[i] * (qw[i] - beta[i] * hq(i, i - 1)) / beta[i]; };
    const double h1 = hq(j, j - 1);
    double m = (diag_of(j - 1) + nu[j] * h1) * h1;
    if (j > 1) m = fma(beta[j - 1], hq(j, j - 2), m);
    up = nu[j] * (h_raw(Hb + (int64_t)(j - 1) * k + j) - m) / beta[j];
    diag = diag_of(j);
  }
  __syncthreads();  // every raw value has been read
  if (j == 1) Hb[0] = qw[0];
  if (j < k) {
    Hb[(int64_t)(j - 1) * k + j] = up;
    Hb[(int64_t)j * k + j] = diag;
    Hb[(int64_t)j * k + j - 1] = beta[j];
  }
}

// ---------------------------------------------------------------------------
// Host side
// ---------------------------------------------------------------------------

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

// the current device's counts (its kernels prepared with them); null: not to be had
static const CSlots *c_slots() {
  static PerDevice<CSlots> table;
  return table.get(current_device(), [](CSlots &t) {
    for (int w = 0; w < 4; ++w)
      if (!c_prepare(c_kernel<true>(1 << w)) || !c_count_clusters(c_kernel<false>(1 << w), t.clusters[w])) return false;
    return true;
  });
}

struct CPlan {
  int S, R, wr, slots, clusters;
};

// CTAs per probe: the fewest rounds of probes over the clusters the GPU holds
// (S = 1, 2, 4, 8, 16: 304, 152, 74, 36, 14 on a GB300), a round costing its
// latency (the meetings of a cluster add about 1.5 us) and the CTA's rows at
// 40 GB/s.  Measured, whole solves' steps: n = 512, 256 probes S = 1 193 us
// (2: 353, 4: 572); n = 3001, 64 probes S = 4 550 us (2: 596, 8: 788); n = 8192,
// 128 probes S = 4 2.15 ms (8: 2.87); n = 16384, 256 probes S = 8 12.1 ms (16: 18.9,
// whose clusters leave a quarter of the SMs over).  Sizes between the powers of two where
// those leave rows or SMs unused: n = 23170, 96 steps, 32 probes S = 12 5.8 ms (16: 6.7), n = 18000, 64,
// 64 3.9 (16: 5.8), n = 10000, 32, 128 S = 6 1.34 (8: 1.64).  Of equal sizes the one whose launches
// are chained: n = 3001, k = 16, 40 probes 464 us per solve with S = 4, 507 with 6.  The separate
// launches, which spread any p evenly, stay behind it also where the probes are one more than
// the clusters: n = 29000, 15 probes on 14 clusters of 16 0.65, 0.65 and 0.70 of their time for
// k = 8, 32 and 100 (14 probes: 0.55, 0.52, 0.52).
static CPlan c_plan(const CSlots &slots, int64_t n, int64_t p, int j) {
  CPlan best{0, 0, 0, 0, 0};
  double best_us = 1e300;
  for (int i = 0; i < kCSizes; ++i) {
    const int S = kCSize[i];
    const int64_t R = ceil_div(ceil_div(n, S), 4) * 4;
    if (R > kCMaxR) continue;
    const int wr = c_row_warps(R);
    int w = 0;
    while ((1 << w) < wr) ++w;
    const int c = slots.clusters[w][i];
    if (c < 1) continue;
    const double rounds = (double)ceil_div(p, c);
    if (c_fixed((int)R, wr) + (size_t)(kCWarps / wr) * c_gc(wr) * R * 4 > kCSmem) continue;  // no slot per group
    const double us = rounds * ((S == 1 ? 5.0 : 6.5) + 0.1 * S + (2.0 * j + 8.0) * R * 4.0 / 40e3) + (S > kCChainS ? kCUnchainedUs : 0.0);
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

// Whether a step of n rows has a plan on the current device (which does not depend on j);
// the separate launches run otherwise.
bool arnoldi_cluster_applies(int64_t n, int64_t p) {
  if (n > (int64_t)kCMaxS * kCMaxR) return false;
  const CSlots *slots = c_slots();
  return slots && c_plan(*slots, n, p, 1).S > 0;
}

// The plan for a table of clusters (host only): see mfg_step_plan.
int arnoldi_plan_query(const CSlots &slots, int64_t n, int64_t p, int64_t j, int *out) {
  if (n > (int64_t)kCMaxS * kCMaxR || j > kCMaxCols) return 0;
  const CPlan c = c_plan(slots, n, p, (int)j);
  out[0] = c.S;
  out[1] = c.R;
  out[2] = c.wr;
  out[3] = c.slots;
  return c.S;
}

// Step j of the two-sweep iteration for every probe (j = 0: the first step).
// Q: the basis (probe stride qb, vector stride ld); W = A q~_j; Vin: q~_j with
// probe stride vb (j = 0: row 0 of Q).  Writes row j of Q (j > 0), the next q~
// into Vout with its bf16 copies (null: not formed), the raw projections into H
// and Hh, the scalars of the step into rec.
int launch_arnoldi_step(int j, int64_t k, int64_t n, int64_t p, float *Q, int64_t qb, int64_t ld, const float *W,
                        const float *Vin, int64_t vb, float *Vout, __nv_bfloat16 *hi, __nv_bfloat16 *lo, double *H,
                        double *Hh, double *rec, int *status, bool chained, cudaStream_t s) {
  if (p <= 0) return MFG_OK;
  const CSlots *slots = c_slots();
  const CPlan plan = slots ? c_plan(*slots, n, p, j) : CPlan{0, 0, 0, 0, 0};
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
  a.H = reinterpret_cast<float2 *>(H);
  a.Hh = reinterpret_cast<float2 *>(Hh);
  a.rec = reinterpret_cast<float2 *>(rec);
  a.status = status;
  auto kern = j == 0 ? c_kernel<true>(plan.wr) : c_kernel<false>(plan.wr);
  const size_t smem = c_fixed(plan.R, plan.wr) + (size_t)plan.slots * (kCWarps / plan.wr) * c_gc(plan.wr) * plan.R * 4;
  return c_launch(kern, plan.S, plan.S * (p < plan.clusters ? p : plan.clusters), smem, a, chained, s);
}

// H of every probe from what the steps left (`band`: its tridiagonal part only);
// nu_last_inv (optional): 1 / nu_k.
int launch_arnoldi_h(int64_t k, int64_t p, double *H, const double *Hh, const double *rec, bool band,
                     double *nu_last_inv, bool chained, cudaStream_t s) {
  if (p <= 0 || k < 2) return MFG_OK;
  const int rows = (int)ceil_div(k, 32) * 32;
  if (band) {
    MFG_CUDA_TRY(launch_kernel(arnoldi_h_band_kernel, dim3((unsigned)p), (unsigned)rows, 0, 0, chained, s, H, Hh, rec, (int)k));
    return MFG_LAUNCH_STATUS();
  }
  auto bytes = [](int64_t kk) {
    return ((size_t)(kk + 1) * kk + 4 * kk + 1 + 4 * (size_t)(ceil_div(kk, 32) * 32)) * sizeof(double);
  };
  const size_t smem = bytes(k);
  // the same limit in every launch: another thread's shorter solve must not lower it under this one
  MFG_CUDA_TRY(cudaFuncSetAttribute(arnoldi_h_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                    (int)bytes(kTwoSweepMaxK)));
  MFG_CUDA_TRY(launch_kernel(arnoldi_h_kernel, dim3((unsigned)p), 4u * rows, smem, 0, chained, s, H, Hh, rec, (int)k, nu_last_inv));
  return MFG_LAUNCH_STATUS();
}

}  // namespace mfg
