// Batched symmetric tridiagonal eigensolve + Gauss quadrature (float64).
//
// For each probe's k x k Hessenberg matrix H the kernel forms the symmetric
// tridiagonal T = (H + H^T)/2 (diagonal H_ii, off-diagonal (H_i,i+1 + H_i+1,i)/2),
// diagonalises it by the implicit QL method with Wilkinson shifts (Givens
// chase from the bottom of the unreduced block up to l), and tracks only the
// first row of the eigenvector matrix, as in the Golub-Welsch construction of
// Gauss rules.  The quadrature value is scale_b * sum_i f(lambda_i) s_1i^2,
// which equals e1^T V diag(f(lambda)) V^T e1 of the dense eigh route.
//
// One thread owns one problem; the three length-k work arrays live in shared
// memory with the thread index fastest, so the lanes of a warp touch
// consecutive words.  The sweep limit per eigenvalue is bounded; a problem
// that does not converge returns NaN and raises MFG_ERR_NO_CONVERGENCE.
#include <cfloat>

#include "common.cuh"
#include "kernels.cuh"

namespace mfg {

constexpr int kMaxSweeps = 64;

__global__ void tridiag_ql_kernel(int k, int64_t p, const double *__restrict__ H, int fun,
                                  double param, const double *__restrict__ scale,
                                  double *__restrict__ values, double *__restrict__ eigvals,
                                  double *__restrict__ first_sq, int *__restrict__ status) {
  extern __shared__ double sm[];
  const int TB = blockDim.x;
  const int t = threadIdx.x;
  const int64_t b = blockIdx.x * (int64_t)TB + t;
  if (b >= p) return;
  double *d = sm + t;
  double *e = sm + (size_t)TB * k + t;
  double *z = sm + (size_t)2 * TB * k + t;
#define D_(i) d[(size_t)(i) * TB]
#define E_(i) e[(size_t)(i) * TB]
#define Z_(i) z[(size_t)(i) * TB]
  const double *Hb = H + (size_t)b * k * k;
  for (int i = 0; i < k; ++i) {
    D_(i) = Hb[(size_t)i * k + i];
    E_(i) = (i + 1 < k) ? 0.5 * (Hb[(size_t)i * k + i + 1] + Hb[(size_t)(i + 1) * k + i]) : 0.0;
    Z_(i) = (i == 0) ? 1.0 : 0.0;
  }
  bool ok = true;
  for (int l = 0; l < k && ok; ++l) {
    int sweeps = 0;
    while (true) {
      int m = l;
      for (; m < k - 1; ++m) {
        const double dd = fabs(D_(m)) + fabs(D_(m + 1));
        if (fabs(E_(m)) <= DBL_EPSILON * dd) break;
      }
      if (m == l) break;
      if (++sweeps > kMaxSweeps) {
        ok = false;
        break;
      }
      // shift from the leading 2x2 block, in the numerically safe form
      double g = (D_(l + 1) - D_(l)) / (2.0 * E_(l));
      double r = hypot(g, 1.0);
      g = D_(m) - D_(l) + E_(l) / (g + copysign(r, g));
      double s = 1.0, c = 1.0, shift_acc = 0.0;
      bool deflated = false;
      // The chase reads d_i, e_i, z_i before they are written in this sweep,
      // and d_{i+1}, z_{i+1} as left by the previous rotation: those travel in
      // registers and the next rotation's inputs are loaded one step ahead, so
      // shared-memory latency stays off the float64 dependence chain.
      double d_up = D_(m), z_up = Z_(m);                // d_{i+1}, z_{i+1}
      double e_i = E_(m - 1), d_i = D_(m - 1), z_i = Z_(m - 1);
      for (int i = m - 1; i >= l; --i) {
        double e_nx = 0.0, d_nx = 0.0, z_nx = 0.0;
        if (i > l) {
          e_nx = E_(i - 1);
          d_nx = D_(i - 1);
          z_nx = Z_(i - 1);
        }
        const double f = s * e_i;
        const double bb = c * e_i;
        // Entries of Lanczos tridiagonals are far from the overflow range, so
        // the rotation uses one reciprocal square root of f^2 + g^2 (in place
        // of hypot and a division): float64 issue slots are scarce on GB300.
        const double rr = fma(f, f, g * g);
        if (rr == 0.0) {  // split: recover and restart the sweep
          E_(i + 1) = 0.0;
          D_(i + 1) = d_up - shift_acc;
          Z_(i + 1) = z_up;
          E_(m) = 0.0;
          deflated = true;
          break;
        }
        const double rinv = rsqrt(rr);
        r = rr * rinv;
        E_(i + 1) = r;
        s = f * rinv;
        c = g * rinv;
        g = d_up - shift_acc;
        r = (d_i - g) * s + 2.0 * c * bb;
        shift_acc = s * r;
        D_(i + 1) = g + shift_acc;
        g = c * r - bb;
        Z_(i + 1) = s * z_i + c * z_up;
        z_up = c * z_i - s * z_up;  // the new z_i, input of the next rotation
        d_up = d_i;
        e_i = e_nx;
        d_i = d_nx;
        z_i = z_nx;
      }
      if (deflated) continue;
      Z_(l) = z_up;
      D_(l) -= shift_acc;
      E_(l) = g;
      E_(m) = 0.0;
    }
  }
  // ascending order (insertion sort of (lambda, s_1^2) pairs), as eigh returns
  for (int i = 0; i < k; ++i) Z_(i) = Z_(i) * Z_(i);
  for (int i = 1; i < k; ++i) {
    const double dv = D_(i), zv = Z_(i);
    int j = i - 1;
    while (j >= 0 && D_(j) > dv) {
      D_(j + 1) = D_(j);
      Z_(j + 1) = Z_(j);
      --j;
    }
    D_(j + 1) = dv;
    Z_(j + 1) = zv;
  }
  double acc = 0.0;
  for (int i = 0; i < k; ++i) {
    const double lam = D_(i);
    double fl;
    if (fun == MFG_FUN_LOG)
      fl = log(lam);
    else if (fun == MFG_FUN_EXP)
      fl = exp(param * lam);
    else if (fun == MFG_FUN_POW)
      fl = pow(lam, param);
    else
      fl = 0.0;
    acc += fl * Z_(i);
    if (eigvals) eigvals[(size_t)b * k + i] = lam;
    if (first_sq) first_sq[(size_t)b * k + i] = Z_(i);
  }
  if (!ok) {
    acc = nan("");
    if (status) atomicExch(status, (int)MFG_ERR_NO_CONVERGENCE);
  }
  if (values) values[b] = (scale ? scale[b] : 1.0) * acc;
#undef D_
#undef E_
#undef Z_
}

// ------------------------------------------------- full eigenvectors, warp per problem
//
// Eigenvalues (ascending) and the full eigenvector matrix of each T, for the
// derivative of e1^T f(T) e1 (the Daleckii-Krein form needs every
// eigenvector).  Implicit QL with Wilkinson shifts as above.  Lane 0 runs
// each sweep's shift chase alone (inputs loaded one rotation ahead, as in the
// first-row kernel) and records the rotations; the warp then applies them,
// in order, to its rows of Z (rows lane, lane + 32, ...).  Z (scratch) is
// row-major k x k; the sorted eigenvectors go to S as columns
// (S[r][j] = component r of vector j).

__global__ void tridiag_eigh_full_kernel(int k, int64_t p, const double *__restrict__ H,
                                         double *__restrict__ w_out, double *__restrict__ S,
                                         double *__restrict__ Z, int *__restrict__ status) {
  extern __shared__ double smf[];
  const int lane = threadIdx.x & 31;
  const int64_t b = blockIdx.x;
  if (b >= p) return;
  double *d = smf;
  double *e = d + k;
  double *rc = e + k;   // rotation i of the current sweep: cosine
  double *rs = rc + k;  // and sine
  int *perm = reinterpret_cast<int *>(rs + k);
  const double *Hb = H + (size_t)b * k * k;
  double *Zb = Z + (size_t)b * k * k;
  for (int i = lane; i < k; i += 32) {
    d[i] = Hb[(size_t)i * k + i];
    e[i] = (i + 1 < k) ? 0.5 * (Hb[(size_t)i * k + i + 1] + Hb[(size_t)(i + 1) * k + i]) : 0.0;
  }
  for (int r = lane; r < k; r += 32)
    for (int c = 0; c < k; ++c) Zb[(size_t)r * k + c] = r == c ? 1.0 : 0.0;
  __syncwarp();
  int ok = 1;
  for (int l = 0; l < k; ++l) {
    int sweeps = 0;
    while (true) {
      // lane 0: one sweep of the chase; the rotations applied are i = hi_i
      // down to lo_i (none when l has converged, or on failure)
      int hi_i = -1, lo_i = 0, done = 0;
      if (lane == 0) {
        int m = l;
        for (; m < k - 1; ++m) {
          const double dd = fabs(d[m]) + fabs(d[m + 1]);
          if (fabs(e[m]) <= DBL_EPSILON * dd) break;
        }
        if (m == l) {
          done = 1;
        } else if (++sweeps > kMaxSweeps) {
          done = 1;
          ok = 0;
        } else {
          double g = (d[l + 1] - d[l]) / (2.0 * e[l]);
          double r = hypot(g, 1.0);
          g = d[m] - d[l] + e[l] / (g + copysign(r, g));
          double sn = 1.0, cs = 1.0, shift_acc = 0.0;
          bool deflated = false;
          double d_up = d[m];
          double e_i = e[m - 1], d_i = d[m - 1];
          hi_i = m - 1;
          lo_i = m;  // the last rotation applied so far
          for (int i = m - 1; i >= l; --i) {
            double e_nx = 0.0, d_nx = 0.0;
            if (i > l) {
              e_nx = e[i - 1];
              d_nx = d[i - 1];
            }
            const double f = sn * e_i;
            const double bb = cs * e_i;
            const double rr = fma(f, f, g * g);
            if (rr == 0.0) {  // split: recover and restart the sweep
              e[i + 1] = 0.0;
              d[i + 1] = d_up - shift_acc;
              e[m] = 0.0;
              deflated = true;
              break;
            }
            const double rinv = rsqrt(rr);
            e[i + 1] = rr * rinv;
            sn = f * rinv;
            cs = g * rinv;
            g = d_up - shift_acc;
            r = (d_i - g) * sn + 2.0 * cs * bb;
            shift_acc = sn * r;
            d[i + 1] = g + shift_acc;
            g = cs * r - bb;
            rc[i] = cs;
            rs[i] = sn;
            lo_i = i;
            d_up = d_i;
            e_i = e_nx;
            d_i = d_nx;
          }
          if (!deflated) {
            d[l] -= shift_acc;
            e[l] = g;
            e[m] = 0.0;
          }
        }
      }
      done = __shfl_sync(0xffffffffu, done, 0);
      hi_i = __shfl_sync(0xffffffffu, hi_i, 0);
      lo_i = __shfl_sync(0xffffffffu, lo_i, 0);
      __syncwarp();  // rc, rs written by lane 0
      if (done) break;
      // the sweep's rotations on columns (i, i + 1) of this lane's rows of Z
      for (int row = lane; row < k; row += 32) {
        double *zr = Zb + (size_t)row * k;
        double zu = zr[hi_i + 1];
        for (int i = hi_i; i >= lo_i; --i) {
          const double zi = zr[i];
          zr[i + 1] = rs[i] * zi + rc[i] * zu;
          zu = rc[i] * zi - rs[i] * zu;
        }
        zr[lo_i] = zu;
      }
      __syncwarp();
    }
    ok = __shfl_sync(0xffffffffu, ok, 0);
    if (!ok) break;
  }
  // ascending order: permutation by insertion sort (lane 0), then a gather of
  // the columns into S
  if (lane == 0) {
    for (int i = 0; i < k; ++i) perm[i] = i;
    for (int i = 1; i < k; ++i) {
      const int pi = perm[i];
      const double dv = d[pi];
      int j = i - 1;
      while (j >= 0 && d[perm[j]] > dv) {
        perm[j + 1] = perm[j];
        --j;
      }
      perm[j + 1] = pi;
    }
  }
  __syncwarp();
  double *Sb = S + (size_t)b * k * k;
  for (int j = lane; j < k; j += 32) w_out[(size_t)b * k + j] = ok ? d[perm[j]] : nan("");
  for (int row = lane; row < k; row += 32)
    for (int j = 0; j < k; ++j) Sb[(size_t)row * k + j] = Zb[(size_t)row * k + perm[j]];
  if (!ok && lane == 0 && status) atomicExch(status, (int)MFG_ERR_NO_CONVERGENCE);
}

static int launch_tridiag_eigh_ql(int64_t k, int64_t p, const double *H, double *w, double *S,
                                  double *Z, int *status, cudaStream_t s) {
  const size_t smem = (size_t)4 * k * sizeof(double) + (size_t)k * sizeof(int);
  if (smem > 48 * 1024) return MFG_ERR_UNSUPPORTED;
  tridiag_eigh_full_kernel<<<(unsigned)p, 32, smem, s>>>((int)k, p, H, w, S, Z, status);
  return MFG_LAUNCH_STATUS();
}

// ------------------------------------------------- divide and conquer, CTA per problem
//
// Cuppen's divide and conquer with every coupling torn: T = diag(T_1, T_2) +
// rho v v^T with v = e_{mid-1} + e_mid, so the leaves are the 1 x 1 blocks
// d_i - e_{i-1} - e_i.  Segments of width w = 1, 2, 4, ... are merged pairwise
// level by level.  A merge of (Q_1, L_1) and (Q_2, L_2) diagonalises
// D + rho z z^T with z = [last row of Q_1; first row of Q_2]; only the first
// and last rows of the eigenvector matrices are carried, because the
// quadrature needs the first row and the next merge needs the last.
//
// Per merge (D sorted, rho made positive by negating the problem):
//  * deflation (Dongarra-Sorensen): rho |z_i| <= tol drops pole i with its
//    unit vector; two kept poles closer than tol are rotated so that one of
//    them drops;
//  * secular roots of 1/rho + sum_i z_i^2 / (d_i - lambda): each root is
//    kept as an offset x from its nearer pole d_o, so that the differences
//    d_i - lambda = (d_i - d_o) - x are accurate.  The iteration interpolates
//    the two poles bounding the root with rational terms, the pole at the
//    origin with its true weight (the fixed-weight scheme of R.-C. Li,
//    "Solving secular equations stably and efficiently", 1993); the largest
//    root uses the two poles below it.  Steps outside the sign bracket fall
//    back to bisection;
//  * z is recomputed from the roots by the Loewner formula (Gu and
//    Eisenstat, 1994), which makes the eigenvectors u_j = zhat / (D - lambda_j)
//    orthogonal to working precision; the new first/last rows are
//    [f; 0]^T u_j and [0; l]^T u_j.
//
// One CTA owns one problem.  The sorted merge and the deflation run on a thread per
// element, the roots, the Loewner products and the vector rows on a group of lanes per
// root, over all merges of a level at once.  (One thread took 64000 clocks for the
// deflation of a merge of 64, and the slowest problem of a launch decides.)

constexpr int kDcMinK = 16;          // below this the QL chase is as fast
constexpr int kDcMaxK = 2048;        // shared-memory bound (about 200 KB)
constexpr int kSecularMaxIt = 128;   // bisection alone halves 2^-128 of the bracket
constexpr int kDcMaxThreads = 512;   // at ~120 registers a thread, within an SM's 64K

struct DcLayout {
  int kh;      // merges per level at most
  size_t words;  // 8-byte words per problem
};

__host__ __device__ inline DcLayout dc_layout(int k) {
  DcLayout L;
  L.kh = (k + 1) / 2;
  // LAM FR LR D Z F L X NF NL EO (k each), RH UB (kh each), O (k ints), MS (kh ints)
  L.words = (size_t)11 * k + 2 * (size_t)L.kh + ((size_t)k + L.kh + 1) / 2;
  return L;
}

// 1/x from the hardware's approximate float64 reciprocal (relative error e of
// about 2^-20) and one third-order step y (1 + e + e^2), which leaves e^3: a few
// ulp from 1/x for x in the normal range, in three dependent FMAs.  The secular
// sums, Loewner products and vector entries below carry rounding errors of that
// size anyway.
__device__ __forceinline__ double rcp_nr(double x) {
  double y;
  asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(x));
  const double e = fma(-x, y, 1.0);
  return fma(y, fma(e, e, e), y);
}

// 1/x to some 2^-20
__device__ __forceinline__ double rcp_rough(double x) {
  double y;
  asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(x));
  return y;
}

// 1 / rho of a coupling, which may be as small as the whole problem's scale
__device__ __forceinline__ double rcp_any(double x) { return x > 1e-290 ? rcp_nr(x) : 1.0 / x; }

// Square root and quotient of an iteration's step: one Newton step (relative
// error about 1e-12).  The iterate they lead to is judged by f itself.
__device__ __forceinline__ double sqrt_step(double v) {
  double y;
  asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(v));
  const double h = v * y;
  const double r = fma(0.5 * h, fma(-h, y, 1.0), h);
  return v > 1e-290 ? r : 0.0;
}
__device__ __forceinline__ double div_step(double num, double den) {
  double y;
  asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(den));
  y = fma(y, fma(-den, y, 1.0), y);
  return num * y;
}

// A double's bits as an integer of the same order (-0 sorts below +0, NaN beyond
// the infinities).
__device__ __forceinline__ long long order_key(double x) {
  const long long v = __double_as_longlong(x);
  return v ^ ((v >> 63) & 0x7fffffffffffffffll);
}
__device__ __forceinline__ bool less_than(double x, double y) { return order_key(x) < order_key(y); }
__device__ __forceinline__ bool positive(double x) { return order_key(x) > 0; }
__device__ __forceinline__ bool is_nan(double x) { return order_key(fabs(x)) > 0x7ff0000000000000ll; }

// The first failure on the stream is what the caller is told (a solve that asked to be
// repeated leaves NaN behind it).
__device__ __forceinline__ void dc_failed(int *status) {
  if (status) atomicCAS(status, 0, (int)MFG_ERR_NO_CONVERGENCE);
}

// Root of c x^2 - 2 h x + a0 with c + s0/(U - x) + s1/(V - x) = 0, U < V its poles:
// the one between them, or (right) the one above both, for c > 0.  The
// cancelling form of the quadratic formula is avoided for either sign of h;
// one square root and one quotient on every path.
__device__ __forceinline__ double dc_quadratic(double c, double h, double a0, bool right) {
  double disc = fma(h, h, -c * a0);
  disc = positive(disc) ? disc : 0.0;
  const double sq = sqrt_step(disc);
  const bool up = positive(h);
  const double t = up ? h + sq : h - sq;
  const bool small = up != right;  // the root of smaller modulus: a0 / t
  return div_step(small ? a0 : t, small ? t : c);
}

// The same in float32, for the first steps of a root.
__device__ __forceinline__ float dc_quadratic(float c, float h, float a0, bool right) {
  const float sq = sqrtf(fmaxf(fmaf(h, h, -c * a0), 0.f));
  const bool up = h > 0.f;
  const float t = up ? h + sq : h - sq;
  const bool small = up != right;
  return __fdividef(small ? a0 : t, small ? t : c);
}

// 2^e just above the largest of a merge's end poles and 2 rho, as the biased exponent
// (0: out of the range in which a float32 copy of the merge is used)
__device__ __forceinline__ int dc_exponent(double p0, double p1, double rho) {
  auto e = [](double v) { return (__double2hiint(v) >> 20) & 0x7ff; };
  int m = e(p0) > e(p1) ? e(p0) : e(p1);
  m = m > e(rho) + 1 ? m : e(rho) + 1;
  return m > 100 && m < 1900 ? m : 0;
}
__device__ __forceinline__ double dc_pow2(int biased) { return __hiloint2double(biased << 20, 0); }

// Sum (product) over the G lanes of a group (lanes G m .. G m + G - 1 of a warp).
// Every lane gets the same bits (each level adds the same two values in either
// order), so the lanes of a group take the same branches afterwards.
template <int G, typename T>
__device__ __forceinline__ T group_sum(T v, unsigned mask) {
#pragma unroll
  for (int o = 1; o < G; o <<= 1) v += __shfl_xor_sync(mask, v, o);
  return v;
}
template <int G>
__device__ __forceinline__ double group_prod(double v, unsigned mask) {
#pragma unroll
  for (int o = 1; o < G; o <<= 1) v *= __shfl_xor_sync(mask, v, o);
  return v;
}

// Root j of the secular equation of the kept poles P[0..mk) (ascending) with
// weights ZZ[i] = z_i^2 and coupling rho > 0; upper bounds the largest root.
// The G lanes of a group (sub = 0..G-1, lane mask gm) each sum every G-th term
// and take identical steps.  A warp has one float64 instruction under way at a
// time, 64 clocks each whatever its active lanes, and an SM about four warps'
// (measured), so what counts is the number of a warp's float64 instructions:
// comparisons run on integers, and a step is one chain for all its cases.
// The first steps run in float32 on copies of the poles (PF: two-float numbers, so
// that close poles keep their distance) and weights (ZF), scaled to 1: a pass over
// the poles is some 500 clocks instead of 4000 there.  They give the nearer pole and x to
// some 1e-6, from where two float64 passes reach rounding level; where they cannot
// tell (a sign within their rounding, a root closer to a pole than float32 reaches) the
// float64 midpoint decides as it would alone.  The float64 iteration is
// safeguarded by the interval of the poles either way.  Quadrature of k = 16, 32 problems
// 98 -> 61 us, k = 32, 64 146 -> 92, k = 64, 1000 1593 -> 660.
// Returns false when the iteration limit is reached, or on NaN.
template <int G>
__device__ bool dc_secular_root(const double *P, const double *ZZ, const float2 *PF, const float *ZF, int mk, int j,
                                double rho, double upper, int sub, unsigned gm, double &x_out, int &o_out) {
  o_out = j;
  if (mk == 1) {
    x_out = rho * ZZ[0];
    return !is_nan(x_out);
  }
  const double ir = rcp_any(rho);
  const bool last = j + 1 >= mk;
  // the poles of the model: (j, j + 1) inside, (j - 1, j) for the largest root
  const int m0 = last ? j - 1 : j, m1 = m0 + 1;
  const int lane0 = (int)(threadIdx.x & 31 & ~(G - 1));
  const double PU = P[m0], PV = P[m1], w0 = ZZ[m0], w1 = ZZ[m1], wh = 0.5 * (w0 + w1);
  const double lo_pole = P[j], hi_pole = last ? upper : PV;
  // one pass over the poles at base + x: the sums of all but the model's terms below
  // (negative) and above (positive) the root, their derivative, and the model's two
  double below, above, slope, t0, t1;
  auto pass = [&](double base, double x) {
    below = above = slope = t0 = t1 = 0.0;
    for (int i = sub; i < mk; i += G) {
      const double inv = rcp_nr((P[i] - base) - x);
      const double t = ZZ[i] * inv;
      if (i == m0) {
        t0 = t;
      } else if (i == m1) {
        t1 = t;
      } else {
        slope = fma(t, inv, slope);
        const double acc = (i < m0 ? below : above) + t;
        if (i < m0)
          below = acc;
        else
          above = acc;
      }
    }
    below = group_sum<G>(below, gm);
    above = group_sum<G>(above, gm);
    slope = group_sum<G>(slope, gm);
    if (G > 1) {
      t0 = __shfl_sync(gm, t0, lane0 + (m0 & (G - 1)));
      t1 = __shfl_sync(gm, t1, lane0 + (m1 & (G - 1)));
    }
  };
  int o = j;
  double x = 0.0;
  bool found = false;
  const int ex = dc_exponent(P[0], P[mk - 1], rho);
  if (ex) {
    const double sc = dc_pow2(2046 - ex);  // 2^-e
    const float irf = 1.0f / (float)(rho * sc), f0w = ZF[m0], f1w = ZF[m1];
    float2 bf = PF[j];
    const float gap = last ? (float)((upper - P[j]) * sc) : (PF[m1].x - bf.x) + (PF[m1].y - bf.y);
    float s_below, s_above, s_slope, s0, s1;
    auto passf = [&](float y) {
      s_below = s_above = s_slope = s0 = s1 = 0.f;
      for (int i = sub; i < mk; i += G) {
        const float inv = __frcp_rn(((PF[i].x - bf.x) + (PF[i].y - bf.y)) - y);
        const float v = ZF[i] * inv;
        if (i == m0) {
          s0 = v;
        } else if (i == m1) {
          s1 = v;
        } else {
          s_slope = fmaf(v, inv, s_slope);
          if (i < m0)
            s_below += v;
          else
            s_above += v;
        }
      }
      s_below = group_sum<G>(s_below, gm);
      s_above = group_sum<G>(s_above, gm);
      s_slope = group_sum<G>(s_slope, gm);
      if (G > 1) {
        s0 = __shfl_sync(gm, s0, lane0 + (m0 & (G - 1)));
        s1 = __shfl_sync(gm, s1, lane0 + (m1 & (G - 1)));
      }
    };
    float y = 0.5f * gap;
    passf(y);
    const float cm = irf + (s_below + s_above), fm = cm + (s0 + s1);
    const float mag = (irf + (s_above - s_below)) + (fabsf(s0) + fabsf(s1));
    if (fabsf(fm) > 2e-5f * mag) {
      // the guess and the steps of the float64 iteration below
      o = (!last && fm < 0.f) ? j + 1 : j;
      bf = PF[o];
      const float U = (PF[m0].x - bf.x) + (PF[m0].y - bf.y), V = (PF[m1].x - bf.x) + (PF[m1].y - bf.y);
      const float M = 0.5f * (U + V), whf = 0.5f * (f0w + f1w);
      float lo = o == j ? 0.f : -gap, hi = o == j ? gap : 0.f;
      const float ym = 0.5f * (lo + hi);
      y = dc_quadratic(cm, fmaf(cm, M, whf), fmaf(cm, U * V, fmaf(f0w, V, f1w * U)), last);
      if (!(lo < y && y < hi) || (last && !(cm > 0.f))) y = ym;
      for (int it = 0; it < 6; ++it) {
        passf(y);
        const float c0 = irf + (s_below + s_above), f = c0 + (s0 + s1);
        if (f > 0.f)
          hi = y;
        else
          lo = y;
        const float u = U - y, v = V - y;
        const float E = (last || o != j) ? u : v, se = s_slope * E;
        const float c = c0 - se;
        const float eta = dc_quadratic(c, fmaf(c, M - y, fmaf(se, 0.5f * E, whf)), u * v * f, last);
        float yn = y + eta;
        const bool done = fabsf(eta) < 1e-6f * fabsf(y);
        if (!(lo < yn && yn < hi) || (last && !(c > 0.f))) {
          if (done) break;
          yn = 0.5f * (lo + hi);
        }
        y = yn;
        if (done) break;
      }
      x = (double)y * dc_pow2(ex);
      found = fabsf(y) > 1e-30f;
    }
  }
  double base = P[o], lo = lo_pole - base, hi = hi_pole - base;
  double U = PU - base, V = PV - base;
  if (!(found && less_than(lo, x) && less_than(x, hi))) {
    // the sign at the midpoint names the nearer pole, the origin of the offsets
    const double xma = 0.5 * (lo_pole + hi_pole);
    pass(0.0, xma);
    const double cmid = ir + (below + above), fmid = cmid + (t0 + t1);
    o = (!last && !positive(fmid)) ? j + 1 : j;
    base = P[o];
    lo = lo_pole - base;
    hi = hi_pole - base;
    U = PU - base;
    V = PV - base;
    const double mid = 0.5 * (U + V), xm = 0.5 * (lo + hi);
    // first guess: the two poles of the model exact, the other terms frozen at
    // the midpoint of the interval, as an offset from the origin (a shift from the
    // midpoint loses a root that is close to its pole)
    x = dc_quadratic(cmid, fma(cmid, mid, wh), fma(cmid, U * V, fma(w0, V, w1 * U)), last);
    if (!(less_than(lo, x) && less_than(x, hi)) || (last && !positive(cmid))) x = xm;
  }
  const double M = 0.5 * (U + V);
  bool conv = false;
  const double eps_mk = DBL_EPSILON * mk;
  for (int it = 0; it < kSecularMaxIt; ++it) {
    pass(base, x);
    const double c0 = ir + (below + above);
    const double f = c0 + (t0 + t1);
    if (is_nan(f)) break;
    if (positive(f))
      hi = x;
    else
      lo = x;
    // |f| within the rounding of its terms: a Newton step is the last.  From a float32 start x
    // may still be mk times that rounding off: without the step the eigenvalues' errors were up to
    // three times those of a float64 start (k = 24: rms 2.8e-16 of the spectral radius, 8.3e-17;
    // with it 6.3e-17).  Quadrature of k = 16, 32 problems 72.4 -> 72.6 us, 100, 64 396 -> 400.
    const double mag = (ir + (above - below)) + (fabs(t0) + fabs(t1));
    if (!less_than(eps_mk * mag, fabs(f))) {
      const double fp = fma(t1 * t1, rcp_rough(w1), fma(t0 * t0, rcp_rough(w0), slope));
      const double xn = fma(-f, rcp_rough(fp), x);
      if (less_than(lo, xn) && less_than(xn, hi)) x = xn;  // not a NaN step
      conv = true;
      break;
    }
    // the rest's derivative goes to the pole E that is not the origin
    const double u = U - x, v = V - x;
    const double E = (last || o != j) ? u : v, se = slope * E;
    const double c = c0 - se;
    const double eta = dc_quadratic(c, fma(c, M - x, fma(se, 0.5 * E, wh)), u * v * f, last);
    if (!less_than(2.0 * DBL_EPSILON * fabs(x), fabs(eta))) {
      conv = true;
      break;
    }
    double xn = x + eta;
    if (!(less_than(lo, xn) && less_than(xn, hi)) || (last && !positive(c))) {  // also a NaN step
      xn = 0.5 * (lo + hi);
      if (hi - lo <= 2.0 * DBL_EPSILON * fmax(fabs(lo), fabs(hi))) {
        conv = true;
        break;
      }
    } else if (less_than(fabs(eta), 1e-10 * fabs(x))) {
      // convergence is quadratic, the other poles being no nearer than the origin:
      // what is left is below the rounding of x
      x = xn;
      conv = true;
      break;
    }
    x = xn;
  }
  x_out = x;
  o_out = o;
  return conv;
}

struct DcArrays {
  double *D, *Z, *F, *L, *X, *NF, *NL, *RH, *UB;
  int *O, *MS;
  float *ZF;  // in LAM, whose values D holds between phases A and E
};
constexpr int kFlipBit = 1 << 30;   // in MS: the merge was negated

// The next pole of positive weight behind pole r of a merge (hi: none); flags as below.
__device__ __forceinline__ int dc_next(const int *O, int r, int hi) {
  do ++r;
  while (r < hi && O[r] == 0);
  return r;
}

// Phase A of one level, on all threads: the merged position of each element of the two
// halves by binary search in the other half, its value, weight and rows written there.
// Then the deflation: poles of negligible weight, and of each run of close ones all but
// the last, whose weight is rotated onto the next one (by the thread of the run's
// first), move behind the kept poles.  MS[q]: the kept count and kFlipBit.  kVec: the
// weights come from the eigenvector columns S, CI keeps each pole's column, and a
// rotation (kept in F and L) turns two columns.  LAM, FR and LR are free once their
// values are in D, F and L.
template <bool kVec>
__device__ void dc_sorted_merge(const DcArrays &Ar, double *LAM, double *FR, double *LR, const double *EO, double *S,
                                int *CI, int k, int s, int nm, double *RH, double *UB) {
  constexpr int kLive = 1, kClose = 2, kGone = 4;  // of positive weight, close to the one before it, rotated away
  const int w = 1 << s;
  int *MS = Ar.MS, *O = Ar.O;
  for (int q = threadIdx.x; q < nm; q += blockDim.x) MS[q] = 0;
  for (int r = threadIdx.x; r < k; r += blockDim.x) {
    const int q = r >> (s + 1);
    if (q >= nm) continue;
    const int a = q * 2 * w, mid = a + w, hi = min(a + 2 * w, k);
    const bool flip = EO[mid - 1] < 0.0, first = r < mid;
    // order within the half, and in the other half the count of values below
    // (first half: strictly; equal values of the first half come first)
    const int own = flip ? (first ? mid - 1 - r : hi - 1 - r) : (first ? r - a : r - mid);
    const double v = flip ? -LAM[r] : LAM[r];
    const long long key = order_key(v);
    int lo = 0, up = first ? hi - mid : w;
    while (lo < up) {
      const int c = (lo + up) >> 1;
      const int i = first ? (flip ? hi - 1 - c : mid + c) : (flip ? mid - 1 - c : a + c);
      const long long other = order_key(flip ? -LAM[i] : LAM[i]);
      if (first ? other < key : other <= key)
        lo = c + 1;
      else
        up = c;
    }
    const int pos = a + own + lo;
    const double z = kVec ? S[(size_t)r * k + (first ? mid - 1 : mid)] : (first ? LR[r] : FR[r]);
    Ar.D[pos] = v;
    Ar.Z[pos] = z;
    Ar.NF[pos] = z * z;
    if (kVec) {
      CI[pos] = r;
    } else {
      Ar.F[pos] = first ? FR[r] : 0.0;
      Ar.L[pos] = first ? 0.0 : LR[r];
    }
  }
  __syncthreads();
  auto tol_of = [&](int a, int hi, double rho) {
    const double maxabs = fmax(fabs(Ar.D[a]), fabs(Ar.D[hi - 1]));  // of the sorted values
    return 8.0 * DBL_EPSILON * fmax(maxabs, 2.0 * rho);
  };
  // the weights are two unit rows: the largest root lies below d + 2 rho
  auto bound = [](double d, double rho) { return d + 2.0 * rho * (1.0 + 1e-12) + 16.0 * DBL_EPSILON * fabs(d); };
  int deflates = 0;
  for (int r = threadIdx.x; r < k; r += blockDim.x) {
    const int q = r >> (s + 1);
    if (q >= nm) continue;
    const int a = q * 2 * w, mid = a + w, hi = min(a + 2 * w, k);
    const double rho = fabs(EO[mid - 1]);
    const bool drop = rho * fabs(Ar.Z[r]) <= tol_of(a, hi, rho);
    O[r] = drop ? 0 : kLive;
    if (drop) MS[q] = deflates = 1;
    if (r == hi - 1) {
      RH[q] = rho;
      UB[q] = bound(Ar.D[r], rho);
    }
  }
  __syncthreads();
  int turns = 0;
  for (int r = threadIdx.x; r < k; r += blockDim.x) {
    const int q = r >> (s + 1);
    if (q >= nm || O[r] == 0) continue;
    const int a = q * 2 * w, hi = min(a + 2 * w, k);
    int prev = r - 1;
    while (prev >= a && O[prev] == 0) --prev;
    if (prev >= a && Ar.D[r] - Ar.D[prev] <= tol_of(a, hi, RH[q])) {
      O[r] = kLive | kClose;
      MS[q] = deflates = turns = 1;
    }
  }
  if (__syncthreads_or(deflates)) {
    if (__syncthreads_or(turns)) {
      for (int r = threadIdx.x; r < k; r += blockDim.x) {
        const int q = r >> (s + 1);
        if (q >= nm || (O[r] & (kLive | kClose)) != kLive) continue;
        const int hi = min(q * 2 * w + 2 * w, k);
        for (int p = r, n = dc_next(O, r, hi); n < hi && (O[n] & kClose); p = n, n = dc_next(O, n, hi)) {
          const double zp = Ar.Z[p], z = Ar.Z[n], h = hypot(zp, z), c = z / h, sn = zp / h;
          O[p] |= kGone;
          Ar.Z[n] = h;
          if (kVec) {
            Ar.F[p] = c;
            Ar.L[p] = sn;
          } else {
            const double fp = Ar.F[p], f = Ar.F[n], lp = Ar.L[p], l = Ar.L[n];
            Ar.F[p] = c * fp - sn * f;
            Ar.L[p] = c * lp - sn * l;
            Ar.F[n] = sn * fp + c * f;
            Ar.L[n] = sn * lp + c * l;
          }
        }
      }
      __syncthreads();
      if (kVec)
        for (int p = 0; p < nm * 2 * w && p < k; ++p) {
          if (!(O[p] & kGone)) continue;  // the same for all threads
          const int a = p >> (s + 1) << (s + 1), hi = min(a + 2 * w, k);
          double *vp = S + (size_t)CI[p] * k, *vc = S + (size_t)CI[dc_next(O, p, hi)] * k;
          const double c = Ar.F[p], sn = Ar.L[p];
          for (int i = a + threadIdx.x; i < hi; i += blockDim.x) {
            const double x = vp[i], y = vc[i];
            vp[i] = c * x - sn * y;
            vc[i] = sn * x + c * y;
          }
          __syncthreads();
        }
    }
    // the kept poles in front, by way of the free arrays
    int *kept_count = reinterpret_cast<int *>(Ar.NL), *ci = reinterpret_cast<int *>(FR);
    for (int r = threadIdx.x; r < k; r += blockDim.x) {
      const int q = r >> (s + 1);
      if (q >= nm || MS[q] == 0) continue;
      const int a = q * 2 * w, hi = min(a + 2 * w, k);
      int before = 0, mk = 0;
      for (int i = a; i < hi; ++i) {
        if (i == r) before = mk;
        mk += O[i] != 0 && !(O[i] & kGone);
      }
      const bool kept = O[r] != 0 && !(O[r] & kGone);
      const int pos = kept ? a + before : a + mk + (r - a - before);
      LAM[pos] = Ar.D[r];
      Ar.X[pos] = Ar.Z[r];
      if (kVec) {
        ci[pos] = CI[r];
      } else {
        FR[pos] = Ar.F[r];
        LR[pos] = Ar.L[r];
      }
      if (kept && before == mk - 1) UB[q] = bound(Ar.D[r], RH[q]);
      if (r == a) kept_count[q] = mk;
    }
    __syncthreads();
    for (int r = threadIdx.x; r < k; r += blockDim.x) {
      const int q = r >> (s + 1);
      if (q >= nm || MS[q] == 0) continue;
      Ar.D[r] = LAM[r];
      Ar.Z[r] = Ar.X[r];
      Ar.NF[r] = Ar.X[r] * Ar.X[r];
      if (kVec) {
        CI[r] = ci[r];
      } else {
        Ar.F[r] = FR[r];
        Ar.L[r] = LR[r];
      }
    }
    __syncthreads();
  }
  for (int q = threadIdx.x; q < nm; q += blockDim.x) {
    const int a = q * 2 * w, hi = min(a + 2 * w, k);
    MS[q] = (MS[q] == 0 ? hi - a : reinterpret_cast<const int *>(Ar.NL)[q]) | (EO[a + w - 1] < 0.0 ? kFlipBit : 0);
  }
  __syncthreads();
}

// Phase E: where element r (root r - a < mk or dropped pole) of a merge with dropped
// poles comes, both kinds being ascending: a dropped pole behind the roots that do not
// exceed it (counted, into C[r], by dc_drop_rank), the roots in order around them.
__device__ __forceinline__ void dc_drop_rank(const double *X, const double *D, double *C, int a, int mk, int r) {
  const long long key = order_key(D[r]);
  int c = 0;
  for (int i = a; i < a + mk; ++i) c += order_key(X[i]) <= key;
  *reinterpret_cast<int *>(C + r) = c;
}
__device__ __forceinline__ int dc_merged_place(const double *C, int a, int mk, int hi, int r) {
  const int j = r - a;
  if (j >= mk) return j - mk + *reinterpret_cast<const int *>(C + r);
  int c = 0;
  for (int i = a + mk; i < hi; ++i) c += *reinterpret_cast<const int *>(C + i) <= j;
  return j + c;
}

// Phases B-D of one level (merges of width 2^(s+1)): the secular roots, the
// Loewner zhat and the new first/last rows, G lanes per root.
// kVec: instead of new first/last rows, the normalised coefficients u of
// each root's vector in the kept poles' columns, U[r * k + i] (r the root's
// index in the problem, i < mk).
template <int G, bool kVec>
__device__ bool dc_merge_roots(const DcArrays &Ar, int k, int s, int nm, double *U) {
  double *D = Ar.D, *Z = Ar.Z, *F = Ar.F, *L = Ar.L, *X = Ar.X, *NF = Ar.NF, *NL = Ar.NL;
  const double *RH = Ar.RH, *UB = Ar.UB;
  int *O = Ar.O;
  const int *MS = Ar.MS;
  float *ZF = Ar.ZF;
  const int sub = threadIdx.x & (G - 1);
  const int grp = threadIdx.x / G, ngrp = (int)blockDim.x / G;
  const unsigned gm = (G == 1 ? 1u : (1u << G) - 1u) << (threadIdx.x & 31 & ~(G - 1));
  bool ok = true;
  // float32 copies of the kept poles (in NL) and weights (in ZF), scaled per merge
  for (int r = threadIdx.x; r < k; r += blockDim.x) {
    const int q = r >> (s + 1);
    if (q >= nm) continue;
    const int a = q << (s + 1);
    const int mk = MS[q] & (kFlipBit - 1);
    if (r - a >= mk) continue;
    const int ex = dc_exponent(D[a], D[a + mk - 1], RH[q]);
    const double d = D[r] * (ex ? dc_pow2(2046 - ex) : 0.0);
    const float h = (float)d;
    reinterpret_cast<float2 *>(NL)[r] = make_float2(h, (float)(d - (double)h));
    ZF[r] = (float)NF[r];
  }
  __syncthreads();
  // B: secular roots over all merges of the level
  for (int r = grp; r < k; r += ngrp) {
    const int q = r >> (s + 1);
    if (q >= nm) continue;
    const int a = q << (s + 1);
    const int j = r - a;
    const int mk = MS[q] & (kFlipBit - 1);
    if (j >= mk) continue;
    double x;
    int o;
    ok &= dc_secular_root<G>(D + a, NF + a, reinterpret_cast<const float2 *>(NL) + a, ZF + a, mk, j, RH[q], UB[q], sub,
                             gm, x, o);
    if (sub == 0) {
      X[r] = x;
      O[r] = o;
    }
  }
  __syncthreads();
  // C: Loewner zhat_i^2 = prod_j (lambda_j - d_i) / prod_{j != i} (d_j - d_i) / rho,
  // numerators paired with denominators to stay in range
  for (int r = grp; r < k; r += ngrp) {
    const int q = r >> (s + 1);
    if (q >= nm) continue;
    const int a = q << (s + 1);
    const int i = r - a;
    const int mk = MS[q] & (kFlipBit - 1);
    if (i >= mk) continue;
    const double *P = D + a;
    const double di = P[i];
    double prod = 1.0;
    for (int j = sub; j < mk; j += G) {
      // factor j, the last one with rho in place of a pole's distance
      const double den = j + 1 < mk ? P[j < i ? j : j + 1] - di : RH[q];
      prod *= ((P[O[a + j]] - di) + X[a + j]) * (j + 1 < mk ? rcp_nr(den) : rcp_any(den));
    }
    prod = group_prod<G>(prod, gm);
    if (sub == 0) Z[r] = copysign(sqrt(fmax(prod, 0.0)), Z[r]);
  }
  __syncthreads();
  // D: first/last rows of the merged eigenvectors
  for (int r = grp; r < k; r += ngrp) {
    const int q = r >> (s + 1);
    if (q >= nm) continue;
    const int a = q << (s + 1);
    const int j = r - a;
    const int mk = MS[q] & (kFlipBit - 1);
    if (j >= mk) continue;
    const double *P = D + a;
    const double ox = P[O[r]], x = X[r];
    double s2 = 0.0, sf = 0.0, sl = 0.0;
    for (int i = sub; i < mk; i += G) {
      const double u = Z[a + i] * rcp_nr((P[i] - ox) - x);
      s2 = fma(u, u, s2);
      if (!kVec) {
        sf = fma(F[a + i], u, sf);
        sl = fma(L[a + i], u, sl);
      }
    }
    s2 = group_sum<G>(s2, gm);
    const double rn = rsqrt(s2);
    if (kVec) {
      for (int i = sub; i < mk; i += G) U[(size_t)r * k + i] = Z[a + i] * rcp_nr((P[i] - ox) - x) * rn;
    } else {
      sf = group_sum<G>(sf, gm);
      sl = group_sum<G>(sl, gm);
    }
    if (sub == 0) {
      if (!kVec) {
        NF[r] = sf * rn;
        NL[r] = sl * rn;
      }
      X[r] = ox + x;
    }
  }
  __syncthreads();
  return ok;
}

// Lanes per root for p problems of size k: a pass over the poles costs a warp
// about 8 k / G + 3 log2 G + 29 float64 instructions of 64 clocks, and the SM's
// warps share one such instruction per 19 clocks; a warp of more roots waits for
// the slowest of more of them, which other warps hide where an SM has several
// problems.  Measured: k = 16, 32 problems 100 us with one lane per root -> 61 us
// (8); k = 32, 64: 199 -> 92 (4); k = 48, 128: 344 -> 143 (4); k = 64, 256: 671 -> 301
// (2).
static int dc_group(int64_t k, int64_t p) {
  const int sms = sm_count();
  int best = 1;
  double best_clk = 1e300;
  for (int G = 1, lg = 0; G <= 8; G *= 2, ++lg) {
    if (k * G > kDcMaxThreads && G > 1) break;
    const double per_sm = p > sms ? (double)p / sms : 1.0;
    const double share = 19.2 * (double)ceil_div(k * G, 32) * per_sm;
    const double wait = 9.0 - (per_sm > 2.0 ? 0.0 : (per_sm > 1.0 ? 0.6 : 1.0)) * lg;
    const double clk = (8.0 * k / G + 3.0 * lg + 29.0) * (share > 64.0 ? share : 64.0) * wait;
    if (clk < best_clk) {
      best_clk = clk;
      best = G;
    }
  }
  return best;
}

template <bool kVec>
__device__ bool dc_merge_level(int G, const DcArrays &Ar, int k, int s, int nm, double *U = nullptr) {
  switch (G) {
    case 8: return dc_merge_roots<8, kVec>(Ar, k, s, nm, U);
    case 4: return dc_merge_roots<4, kVec>(Ar, k, s, nm, U);
    case 2: return dc_merge_roots<2, kVec>(Ar, k, s, nm, U);
    default: return dc_merge_roots<1, kVec>(Ar, k, s, nm, U);
  }
}

__global__ void __launch_bounds__(kDcMaxThreads, 1)
    tridiag_dc_kernel(int k, int64_t p, int G, const double *H, int fun, double param,
                      const double *scale, double *__restrict__ values,
                      double *__restrict__ eigvals, double *__restrict__ first_sq,
                      int *__restrict__ status) {
  chain_wait();
  chain_next();
  extern __shared__ double sm[];
  const int tid = threadIdx.x;
  const int nt = blockDim.x;
  const int64_t b = blockIdx.x;
  const DcLayout Ly = dc_layout(k);
  double *LAM = sm;       // segment eigenvalues
  double *FR = LAM + k;   // first rows of the segment eigenvector matrices
  double *LR = FR + k;    // last rows
  double *D = LR + k;     // merge: poles (kept first, deflated after)
  double *Z = D + k;      // merge: z, then zhat
  double *F = Z + k;      // merge: first-row entries aligned with D
  double *L = F + k;      // merge: last-row entries aligned with D
  double *X = L + k;      // merge: root offsets, then roots
  double *NF = X + k;     // merge: z^2 of the kept poles, then new first rows
  double *NL = NF + k;    // merge: new last rows
  double *EO = NL + k;    // off-diagonal of T
  double *RH = EO + k;    // per merge: |rho|
  double *UB = RH + Ly.kh;  // per merge: bound of the largest root
  int *O = reinterpret_cast<int *>(UB + Ly.kh);  // per root: origin pole
  int *MS = O + k;        // per merge: kept count and kFlipBit
  const DcArrays Ar{D, Z, F, L, X, NF, NL, RH, UB, O, MS, reinterpret_cast<float *>(LAM)};

  const double *Hb = H + (size_t)b * k * k;
  for (int i = tid; i < k; i += nt)
    EO[i] = (i + 1 < k) ? 0.5 * (Hb[(size_t)i * k + i + 1] + Hb[(size_t)(i + 1) * k + i]) : 0.0;
  __syncthreads();
  int bad = 0;
  for (int i = tid; i < k; i += nt) {
    LAM[i] = Hb[(size_t)i * k + i] - (i > 0 ? EO[i - 1] : 0.0) - EO[i];
    FR[i] = 1.0;
    LR[i] = 1.0;
    bad |= is_nan(LAM[i]);
  }
  if (__syncthreads_or(bad)) {
    for (int i = tid; i < k; i += nt) {
      if (eigvals) eigvals[(size_t)b * k + i] = nan("");
      if (first_sq) first_sq[(size_t)b * k + i] = nan("");
    }
    if (tid == 0 && values) values[b] = nan("");
    if (tid == 0) dc_failed(status);
    return;
  }
  bool ok = true;
  for (int s = 0; (1 << s) < k; ++s) {
    const int w = 1 << s;
    const int nm = (k - w - 1) / (2 * w) + 1;
    // A: sorted merge of the two halves, deflation
    dc_sorted_merge<false>(Ar, LAM, FR, LR, EO, nullptr, nullptr, k, s, nm, RH, UB);
    ok &= dc_merge_level<false>(G, Ar, k, s, nm);
    // E: merge the roots [a, a+mk) with the dropped poles [a+mk, hi); a negated merge
    // is negated back and reversed
    for (int r = tid; r < k; r += nt) {
      const int q = r >> (s + 1);
      const int a = q * 2 * w, mk = q < nm ? MS[q] & (kFlipBit - 1) : 0;
      if (q < nm && r - a >= mk) dc_drop_rank(X, D, NL, a, mk, r);
    }
    __syncthreads();
    for (int r = tid; r < k; r += nt) {
      const int q = r >> (s + 1);
      if (q >= nm) continue;
      const int a = q * 2 * w, hi = min(a + 2 * w, k), mk = MS[q] & (kFlipBit - 1);
      const bool flip = (MS[q] & kFlipBit) != 0, root = r - a < mk;
      const int at = mk == hi - a ? r - a : dc_merged_place(NL, a, mk, hi, r);
      const int pos = flip ? hi - 1 - at : a + at;
      const double v = root ? X[r] : D[r];
      LAM[pos] = (flip ? -v : v) + 0.0;  // one zero: the order of the keys is that of the values
      FR[pos] = root ? NF[r] : F[r];
      LR[pos] = root ? NL[r] : L[r];
    }
    __syncthreads();
  }
  ok = __syncthreads_and(ok) != 0;
  double acc = 0.0;
  for (int i = tid; i < k; i += nt) {
    const double lam = LAM[i];
    const double w2 = FR[i] * FR[i];
    double fl;
    if (fun == MFG_FUN_LOG)
      fl = log(lam);
    else if (fun == MFG_FUN_EXP)
      fl = exp(param * lam);
    else if (fun == MFG_FUN_POW)
      fl = pow(lam, param);
    else
      fl = 0.0;
    acc = fma(fl, w2, acc);
    if (eigvals) eigvals[(size_t)b * k + i] = lam;
    if (first_sq) first_sq[(size_t)b * k + i] = w2;
  }
  // fixed-order CTA sum: warp butterflies, then warp partials in order
  __shared__ double red[32];
  acc = warp_sum(acc);
  if ((tid & 31) == 0) red[tid >> 5] = acc;
  __syncthreads();
  if (tid == 0) {
    acc = 0.0;
    for (int w = 0; w < (nt >> 5); ++w) acc += red[w];
    if (!ok) {
      acc = nan("");
      dc_failed(status);
    }
    if (values) values[b] = (scale ? scale[b] : 1.0) * acc;
  }
}

// ---------------------------------------- divide and conquer with eigenvectors
//
// The levels, deflation, secular roots and Loewner vectors of
// tridiag_dc_kernel, carrying every eigenvector column (rows a..hi-1 of its
// merge; zero elsewhere) in shared memory instead of first and last rows.
// S, S2 and U are k x k, column c of S at S[c * k].
//   A: sorted merge of the halves with deflation; each pole keeps the index CI of
//     its column in S (z is that column's entry in row mid-1 or mid), and a
//     close-pole rotation combines two columns in place;
//   B, C, D: dc_merge_roots<G, true>, which leaves each root's normalised
//     coefficients in U;
//   D' (all threads over (column, row) pairs): S2[:, a+j] = S[:, CI[a..a+mk)]
//     U[a+j, :] for the roots, and S2[:, c] = S[:, CI[c]] for the deflated
//     poles c >= a+mk;
//   E: the order of the merged eigenvalues as a column map (in O), then S
//     from S2 through that map.
// On the CPU, tests/test_dc_model.py runs the merges with a serial deflation and the float64
// iteration from the midpoint (dc_full), tests/test_dc_merge_model.py the index work of phases
// A and E element by element.
constexpr int kDcvMaxK = 64;  // S, S2, U: 3 k^2 doubles (96 KB at k = 64)

__host__ inline size_t dcv_smem_bytes(int k) {
  return (dc_layout(k).words + (size_t)3 * k * k + ((size_t)k + 1) / 2) * sizeof(double);
}

__global__ void __launch_bounds__(kDcMaxThreads, 1)
    tridiag_dcv_kernel(int k, int64_t p, int G, const double *__restrict__ H, double *__restrict__ w_out,
                       double *__restrict__ S_out, int *__restrict__ status) {
  extern __shared__ double sm[];
  const int tid = threadIdx.x;
  const int nt = blockDim.x;
  const int64_t b = blockIdx.x;
  const DcLayout Ly = dc_layout(k);
  double *LAM = sm;
  double *FR = LAM + k;  // scratch here (same layout as tridiag_dc_kernel)
  double *LR = FR + k;
  double *D = LR + k;
  double *Z = D + k;
  double *F = Z + k;
  double *L = F + k;
  double *X = L + k;
  double *NF = X + k;
  double *NL = NF + k;
  double *EO = NL + k;
  double *RH = EO + k;
  double *UB = RH + Ly.kh;
  int *O = reinterpret_cast<int *>(UB + Ly.kh);
  int *MS = O + k;
  double *S = sm + Ly.words;
  double *S2 = S + (size_t)k * k;
  double *U = S2 + (size_t)k * k;
  int *CI = reinterpret_cast<int *>(U + (size_t)k * k);
  const DcArrays Ar{D, Z, F, L, X, NF, NL, RH, UB, O, MS, reinterpret_cast<float *>(LAM)};

  const double *Hb = H + (size_t)b * k * k;
  for (int i = tid; i < k; i += nt)
    EO[i] = (i + 1 < k) ? 0.5 * (Hb[(size_t)i * k + i + 1] + Hb[(size_t)(i + 1) * k + i]) : 0.0;
  __syncthreads();
  int bad = 0;
  for (int i = tid; i < k; i += nt) {
    LAM[i] = Hb[(size_t)i * k + i] - (i > 0 ? EO[i - 1] : 0.0) - EO[i];
    CI[i] = i;  // a column at all times, also where a failure leaves the poles unordered
    bad |= is_nan(LAM[i]);
  }
  for (int idx = tid; idx < k * k; idx += nt) S[idx] = (idx / k == idx % k) ? 1.0 : 0.0;
  if (__syncthreads_or(bad)) {
    for (int i = tid; i < k; i += nt) w_out[(size_t)b * k + i] = nan("");
    for (int idx = tid; idx < k * k; idx += nt) S_out[(size_t)b * k * k + idx] = nan("");
    if (tid == 0) dc_failed(status);
    return;
  }
  bool ok = true;
  for (int s = 0; (1 << s) < k; ++s) {
    const int w = 1 << s;
    const int span = 2 * w;
    const int nm = (k - w - 1) / span + 1;
    // A
    dc_sorted_merge<true>(Ar, LAM, FR, LR, EO, S, CI, k, s, nm, RH, UB);
    ok &= dc_merge_level<true>(G, Ar, k, s, nm, U);
    // D': the merged columns into S2 (rows a..hi-1)
    for (int idx = tid; idx < nm * span * span; idx += nt) {
      const int q = idx / (span * span);
      const int rem = idx - q * span * span;
      const int j = rem / span, tt = rem - j * span;
      const int a = q * span, hi = min(a + span, k);
      const int c = a + j, t = a + tt;
      if (c >= hi || t >= hi) continue;
      const int mk = MS[q] & (kFlipBit - 1);
      if (j < mk) {
        const double *u = U + (size_t)c * k;
        double acc = 0.0;
        for (int i = 0; i < mk; ++i) acc = fma(u[i], S[(size_t)CI[a + i] * k + t], acc);
        S2[(size_t)c * k + t] = acc;
      } else {
        S2[(size_t)c * k + t] = S[(size_t)CI[c] * k + t];
      }
    }
    // E: ascending merge of the roots [a, a+mk) and the dropped poles
    // [a+mk, hi); a negated merge is negated back and reversed
    for (int r = tid; r < k; r += nt) {
      const int q = r >> (s + 1);
      const int a = q * span, mk = q < nm ? MS[q] & (kFlipBit - 1) : 0;
      if (q < nm && r - a >= mk) dc_drop_rank(X, D, NL, a, mk, r);
    }
    __syncthreads();
    for (int r = tid; r < k; r += nt) {
      const int q = r >> (s + 1);
      if (q >= nm) continue;
      const int a = q * span, hi = min(a + span, k), mk = MS[q] & (kFlipBit - 1);
      const bool flip = (MS[q] & kFlipBit) != 0, root = r - a < mk;
      const int at = mk == hi - a ? r - a : dc_merged_place(NL, a, mk, hi, r);
      const int pos = flip ? hi - 1 - at : a + at;
      const double v = root ? X[r] : D[r];
      LAM[pos] = (flip ? -v : v) + 0.0;  // one zero: the order of the keys is that of the values
      O[pos] = r;
    }
    __syncthreads();
    for (int idx = tid; idx < nm * span * span; idx += nt) {
      const int q = idx / (span * span);
      const int rem = idx - q * span * span;
      const int j = rem / span, tt = rem - j * span;
      const int a = q * span, hi = min(a + span, k);
      const int c = a + j, t = a + tt;
      if (c >= hi || t >= hi) continue;
      S[(size_t)c * k + t] = S2[(size_t)O[c] * k + t];
    }
    __syncthreads();
  }
  ok = __syncthreads_and(ok) != 0;
  for (int j = tid; j < k; j += nt) w_out[(size_t)b * k + j] = ok ? LAM[j] : nan("");
  double *Sb = S_out + (size_t)b * k * k;
  for (int idx = tid; idx < k * k; idx += nt) {
    const int row = idx / k, j = idx - row * k;
    Sb[idx] = S[(size_t)j * k + row];
  }
  if (!ok && tid == 0) dc_failed(status);
}

int launch_tridiag_quadrature(int64_t k, int64_t p, const double *H, int32_t fun, double param,
                              const double *scale, double *values, double *eigvals,
                              double *first_sq, int *status, cudaStream_t s, bool chained) {
  if (p <= 0 || k <= 0) return MFG_OK;
  if (k >= kDcMinK && k <= kDcMaxK) {
    // one problem per CTA, G lanes per root, up to 512 threads
    const size_t smem = dc_layout((int)k).words * sizeof(double);
    if (smem > 48 * 1024)
      MFG_CUDA_TRY(cudaFuncSetAttribute(tridiag_dc_kernel,
                                        cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    const int G = dc_group(k, p);
    const int64_t want = (k * G + 31) / 32 * 32;
    const int threads = (int)(want < kDcMaxThreads ? want : kDcMaxThreads);
    MFG_CUDA_TRY(launch_kernel(tridiag_dc_kernel, dim3((unsigned)p), (unsigned)threads, smem, 0, chained, s, (int)k, p, G,
                               H, fun, param, scale, values, eigvals, first_sq, status));
    return MFG_LAUNCH_STATUS();
  }
  const size_t per_thread = (size_t)3 * k * sizeof(double);
  const size_t budget = 46 * 1024;  // under the default dynamic shared-memory limit
  if (per_thread > budget) return MFG_ERR_UNSUPPORTED;
  // The solve is a serial float64 chain per problem: spread the problems over
  // all SMs (a few threads per CTA) so that no SM's float64 pipe is shared
  // by many of them.
  int sms = 152;
  int dev = 0;
  if (cudaGetDevice(&dev) == cudaSuccess)
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  int tb = 1;
  while (tb < 32 && (int64_t)tb * sms < p) tb <<= 1;
  while (tb > 1 && (size_t)tb * per_thread > budget) tb >>= 1;
  const unsigned grid = (unsigned)ceil_div(p, tb);
  tridiag_ql_kernel<<<grid, tb, (size_t)tb * per_thread, s>>>((int)k, p, H, fun, param, scale,
                                                              values, eigvals, first_sq, status);
  return MFG_LAUNCH_STATUS();
}

// mean and standard error (population std / sqrt(p)) of p values; one CTA.
__global__ void mean_sem_kernel(const double *__restrict__ v, int64_t p, double *__restrict__ out) {
  __shared__ double red[kWarps];
  __shared__ double s_mean;
  double acc = 0.0;
  for (int64_t i = threadIdx.x; i < p; i += blockDim.x) acc += v[i];
  acc = warp_sum(acc);
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = acc;
  __syncthreads();
  if (threadIdx.x == 0) {
    double t = 0.0;
    for (int q = 0; q < kWarps; ++q) t += red[q];
    s_mean = t / (double)p;
  }
  __syncthreads();
  const double mean = s_mean;
  double sq = 0.0;
  for (int64_t i = threadIdx.x; i < p; i += blockDim.x) {
    const double dv = v[i] - mean;
    sq += dv * dv;
  }
  sq = warp_sum(sq);
  __syncthreads();
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = sq;
  __syncthreads();
  if (threadIdx.x == 0) {
    double t = 0.0;
    for (int q = 0; q < kWarps; ++q) t += red[q];
    out[0] = mean;
    out[1] = sqrt(t / (double)p) / sqrt((double)p);
  }
}

int launch_mean_sem(const double *values, int64_t p, double *mean_sem, cudaStream_t s) {
  if (p <= 0) return MFG_ERR_BAD_ARG;
  mean_sem_kernel<<<1, kThreads, 0, s>>>(values, p, mean_sem);
  return MFG_LAUNCH_STATUS();
}

// Every eigenvector: divide and conquer for kDcMinK <= k <= kDcvMaxK (the
// gradient's k), implicit QL otherwise.
int launch_tridiag_eigh_full(int64_t k, int64_t p, const double *H, double *w, double *S,
                             double *Z, int *status, cudaStream_t s) {
  if (p <= 0 || k <= 0) return MFG_OK;
  if (k >= kDcMinK && k <= kDcvMaxK) {
    const size_t smem = dcv_smem_bytes((int)k);
    MFG_CUDA_TRY(cudaFuncSetAttribute(tridiag_dcv_kernel,
                                      cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    const int G = dc_group(k, p);
    const int64_t want = k * G;  // at least 4 k threads for the merged columns
    const int threads = (int)(((want > 4 * k ? want : 4 * k) + 31) / 32 * 32);
    tridiag_dcv_kernel<<<(unsigned)p, threads, smem, s>>>((int)k, p, G, H, w, S, status);
    return MFG_LAUNCH_STATUS();
  }
  return launch_tridiag_eigh_ql(k, p, H, w, S, Z, status, s);
}

}  // namespace mfg
