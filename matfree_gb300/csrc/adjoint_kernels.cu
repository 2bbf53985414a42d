// Small float64 kernels of the batched Hessenberg adjoint (reverse Arnoldi).
//
// The reverse sweep keeps, per probe b, the k x k matrices Gamma and
// Pi_gamma = H dH^T - dc c e1 e1^T and a few length-k coefficient vectors.
// These kernels update them between the n-length sweeps (projections,
// updates, operator application) that the driver issues with the forward
// kernels.  Index conventions follow the float64 restatement of
// matfree/decomp.py:480-600: step idx runs from k-1 down to 0.
#include "cluster.cuh"
#include "kernels.cuh"

namespace mfg {

// Pi[b][i][j] = sum_l H[b][i][l] dH[b][j][l]  - (i == j == 0) dc_b c_b
__global__ void pi_gamma_kernel(const double *__restrict__ H, const double *__restrict__ dH,
                                const double *__restrict__ dc, const double *__restrict__ c,
                                int k, int64_t p, double *__restrict__ Pi) {
  const int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  const int64_t kk = (int64_t)k * k;
  if (t >= p * kk) return;
  const int64_t b = t / kk;
  const int i = (int)((t % kk) / k), j = (int)(t % k);
  const double *Hb = H + b * kk, *dHb = dH + b * kk;
  double acc = 0.0;
  for (int l = 0; l < k; ++l) acc += Hb[(int64_t)i * k + l] * dHb[(int64_t)j * k + l];
  if (i == 0 && j == 0 && dc) acc -= dc[b] * c[b];
  Pi[t] = acc;
}

// gamma[b][j] = dH[b][j][k-1] - h[b][j]  (h = Q^T dr, or absent)
// coef[b][j] = -gamma[b][j]               (lambda = dr + Q gamma as an update)
__global__ void adj_init_kernel(const double *__restrict__ dH, const double *__restrict__ h, int k,
                                int64_t p, double *__restrict__ gamma, double *__restrict__ coef) {
  const int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (t >= p * k) return;
  const int64_t b = t / k;
  const int j = (int)(t % k);
  double g = dH[b * k * k + (int64_t)j * k + (k - 1)];
  if (h) g -= h[t];
  gamma[t] = g;
  coef[t] = -g;
}

// masked re-projection coefficients of step idx:
// coef[b][j] = h[b][j] - dH[b][j][idx] for j < ncols (columns 0..idx+1)
__global__ void adj_reortho_coef_kernel(const double *__restrict__ h, const double *__restrict__ dH,
                                        int k, int64_t p, int idx, int ncols,
                                        double *__restrict__ coef) {
  const int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (t >= p * ncols) return;
  const int64_t b = t / ncols;
  const int j = (int)(t % ncols);
  coef[b * k + j] = h[b * k + j] - dH[b * k * k + (int64_t)j * k + idx];
}

// Step idx after g = Q^T (A^T lambda) (g[b][j], j <= idx):
//   Gamma[idx][j] = m_j (Pi[idx][j] - g_j),  m_j = 1 (j < idx), 1/2 (j = idx), 0
//   coefG[j] = -(Gamma[idx][j] + Gamma[j][idx])   (xi adds Q (Gamma + Gamma^T)[idx, :])
//   bp[j] = H[idx][j] for j > idx, else 0        (beta_plus row of idx)
//   scal = (alpha = H[idx][idx], gamma_idx, beta_minus = H[idx][idx-1] or 1)
__global__ void adj_step_coef_kernel(const double *__restrict__ H, const double *__restrict__ Pi,
                                     const double *__restrict__ g, const double *__restrict__ gamma,
                                     int k, int64_t p, int idx, double *__restrict__ Gamma,
                                     double *__restrict__ coefG, double *__restrict__ bp,
                                     double *__restrict__ scal) {
  const int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (t >= p * k) return;
  const int64_t b = t / k;
  const int j = (int)(t % k);
  const int64_t kk = (int64_t)k * k;
  double *Gb = Gamma + b * kk;
  const double mask = j < idx ? 1.0 : (j == idx ? 0.5 : 0.0);
  const double row = (j <= idx) ? mask * (Pi[b * kk + (int64_t)idx * k + j] - g[b * k + j]) : 0.0;
  Gb[(int64_t)idx * k + j] = row;
  const double colv = (j == idx) ? row : Gb[(int64_t)j * k + idx];
  coefG[b * k + j] = -(row + colv);
  bp[b * k + j] = (j > idx) ? H[b * kk + (int64_t)idx * k + j] : 0.0;
  if (j == 0) {
    scal[b * 3 + 0] = H[b * kk + (int64_t)idx * k + idx];
    scal[b * 3 + 1] = gamma[b * k + idx];
    scal[b * 3 + 2] = idx > 0 ? H[b * kk + (int64_t)idx * k + (idx - 1)] : 1.0;
  }
}

// out[b][r] = U[b][r] - alpha_b lam[b][r] + gam_b R[b][r] (+ dq[b][r] when the
// cotangent of the basis is given: its column idx, dq_bstride apart per probe)
template <typename T>
__global__ void adj_lincomb_kernel(const T *__restrict__ U, const T *__restrict__ lam,
                                   const T *__restrict__ R, const T *__restrict__ dq, int64_t dq_bstride,
                                   const double *__restrict__ scal, int64_t n, int64_t ld, int64_t p,
                                   T *__restrict__ out) {
  const int64_t r = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  const int64_t b = blockIdx.y;
  if (r >= n || b >= p) return;
  const T alpha = (T)scal[b * 3 + 0], gam = (T)scal[b * 3 + 1];
  const int64_t o = b * ld + r;
  T v = U[o] - alpha * lam[o] + gam * R[o];
  if (dq) v += dq[b * dq_bstride + r];
  out[o] = v;
}

// y[i] += a x[i] (float64)
__global__ void axpy_f64_kernel(double a, const double *__restrict__ x, double *__restrict__ y,
                                int64_t m) {
  const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (i < m) y[i] += a * x[i];
}

// out[b][r] = sum_i coef[b][i] Q[b][i][r] for r < n, 0 for n <= r < ld: the
// back-projection Q^T (f(T) e1) of a batch of Krylov bases (p, k, ld).  The
// coefficients are staged in shared memory kCombineCoef at a time; each
// thread owns one row and sums over i in a fixed order.
constexpr int kCombineCoef = 512;

template <typename T>
__global__ void __launch_bounds__(256)
basis_combine_kernel(const T *__restrict__ Q, int64_t k, int64_t ld, int64_t n,
                     const double *__restrict__ coef, T *__restrict__ out) {
  __shared__ T sc[kCombineCoef];
  const int64_t b = blockIdx.y;
  const int64_t r = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  const T *Qb = Q + b * k * ld;
  T acc = 0;
  for (int64_t i0 = 0; i0 < k; i0 += kCombineCoef) {
    const int m = (int)(k - i0 < kCombineCoef ? k - i0 : kCombineCoef);
    __syncthreads();
    for (int t = threadIdx.x; t < m; t += blockDim.x) sc[t] = (T)coef[b * k + i0 + t];
    __syncthreads();
    if (r < n)
      for (int t = 0; t < m; ++t) acc += sc[t] * Qb[(i0 + t) * ld + r];
  }
  if (r < ld) out[b * ld + r] = r < n ? acc : (T)0;
}

// beta[b] = scal[b][2] (the divisor of step idx), for the normalise kernel
__global__ void adj_beta_kernel(const double *__restrict__ scal, int64_t p, double *__restrict__ beta) {
  const int64_t b = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (b < p) beta[b] = scal[b * 3 + 2];
}

static inline unsigned blocks(int64_t work, int tb) { return (unsigned)ceil_div(work, tb); }

int launch_pi_gamma(const double *H, const double *dH, const double *dc, const double *c, int k,
                    int64_t p, double *Pi, cudaStream_t s) {
  pi_gamma_kernel<<<blocks(p * k * k, 128), 128, 0, s>>>(H, dH, dc, c, k, p, Pi);
  return MFG_LAUNCH_STATUS();
}

int launch_adj_init(const double *dH, const double *h, int k, int64_t p, double *gamma, double *coef,
                    cudaStream_t s) {
  adj_init_kernel<<<blocks(p * k, 128), 128, 0, s>>>(dH, h, k, p, gamma, coef);
  return MFG_LAUNCH_STATUS();
}

int launch_adj_reortho_coef(const double *h, const double *dH, int k, int64_t p, int idx, int ncols,
                            double *coef, cudaStream_t s) {
  adj_reortho_coef_kernel<<<blocks(p * ncols, 128), 128, 0, s>>>(h, dH, k, p, idx, ncols, coef);
  return MFG_LAUNCH_STATUS();
}

int launch_adj_step_coef(const double *H, const double *Pi, const double *g, const double *gamma,
                         int k, int64_t p, int idx, double *Gamma, double *coefG, double *bp,
                         double *scal, double *beta, cudaStream_t s) {
  adj_step_coef_kernel<<<blocks(p * k, 128), 128, 0, s>>>(H, Pi, g, gamma, k, p, idx, Gamma, coefG,
                                                          bp, scal);
  adj_beta_kernel<<<blocks(p, 128), 128, 0, s>>>(scal, p, beta);
  return MFG_LAUNCH_STATUS();
}

template <typename T>
int launch_adj_lincomb(const T *U, const T *lam, const T *R, const T *dq, int64_t dq_bstride,
                       const double *scal, int64_t n, int64_t ld, int64_t p, T *out, cudaStream_t s) {
  if (p > 65535) return MFG_ERR_UNSUPPORTED;
  adj_lincomb_kernel<T><<<dim3(blocks(n, 256), (unsigned)p), 256, 0, s>>>(U, lam, R, dq, dq_bstride, scal,
                                                                          n, ld, p, out);
  return MFG_LAUNCH_STATUS();
}
template int launch_adj_lincomb<float>(const float *, const float *, const float *, const float *,
                                       int64_t, const double *, int64_t, int64_t, int64_t, float *,
                                       cudaStream_t);
template int launch_adj_lincomb<double>(const double *, const double *, const double *, const double *,
                                        int64_t, const double *, int64_t, int64_t, int64_t, double *,
                                        cudaStream_t);

template <typename T>
int launch_basis_combine(const T *Q, int64_t k, int64_t ld, int64_t n, int64_t p, const double *coef,
                         T *out, cudaStream_t s) {
  if (p <= 0) return MFG_OK;
  if (p > 65535) return MFG_ERR_UNSUPPORTED;
  basis_combine_kernel<T><<<dim3(blocks(ld, 256), (unsigned)p), 256, 0, s>>>(Q, k, ld, n, coef, out);
  return MFG_LAUNCH_STATUS();
}
template int launch_basis_combine<float>(const float *, int64_t, int64_t, int64_t, int64_t,
                                         const double *, float *, cudaStream_t);
template int launch_basis_combine<double>(const double *, int64_t, int64_t, int64_t, int64_t,
                                          const double *, double *, cudaStream_t);

int launch_axpy_f64(double a, const double *x, double *y, int64_t m, cudaStream_t s) {
  if (m <= 0) return MFG_OK;
  axpy_f64_kernel<<<blocks(m, 256), 256, 0, s>>>(a, x, y, m);
  return MFG_LAUNCH_STATUS();
}

// <Lam, Y> (and <Lam, Q> from the same read of Lam) over the n valid columns of
// `rows` panel rows, in float64: the parameter contractions of the reverse pass.
//
// Bound by the read of the two or three panels.  A float64 multiply-add or
// conversion costs an SM about 19 cycles a warp, several times what the load of its
// operands takes, so products of floats are kept as exact two-float pairs (product
// and fma remainder) and summed with error-free additions: ten float instructions
// an element, some 2^-45 of the sum of |lam y| against float64.  Four products
// outside [2^-90, 2^100], where a remainder could underflow or the sum overflow,
// are added in float64.  6144 rows of 8192, all of the contractions with their two
// products and the split: 4.87 ms with float64 copies of the panels and one pass per
// conversion, product and sum, 3.24 ms so (of which the products 2.6 at the GEMM's rate).
// 1024 columns a CTA step, 8 CTAs an SM; partials are summed in a fixed order.
constexpr int kDotCols = kThreads * 4;
constexpr int kDotBlocks = 152 * 8;

struct Dot2 {
  float s = 0.0f, e = 0.0f;
  double d = 0.0;
  __device__ __forceinline__ void add(const float4 &l, const float4 &y) {
    const float a[4] = {l.x, l.y, l.z, l.w}, b[4] = {y.x, y.y, y.z, y.w};
    float p[4], m = 0.0f;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      p[i] = a[i] * b[i];
      m = fmaxf(m, fabsf(p[i]));
    }
    if (m < 0x1p-90f || m > 0x1p100f) {
#pragma unroll
      for (int i = 0; i < 4; ++i) d += (double)a[i] * (double)b[i];
    } else {
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        e += fmaf(a[i], b[i], -p[i]);
        two_add(s, e, p[i]);
      }
    }
  }
  __device__ __forceinline__ double value() const { return d + ((double)s + (double)e); }
};

// the valid ones of four panel elements from column c on; padding counts as zero
__device__ __forceinline__ float4 dot_load(const float *row, int64_t c, int64_t n) {
  float4 v = __ldg(reinterpret_cast<const float4 *>(row + c));
  if (c + 4 > n) {
    if (c + 1 >= n) v.y = 0.0f;
    if (c + 2 >= n) v.z = 0.0f;
    if (c + 3 >= n) v.w = 0.0f;
  }
  return v;
}

template <typename T, bool kQ>
__global__ void __launch_bounds__(kThreads) panel_dot_kernel(const T *__restrict__ Y,
                                                             const T *__restrict__ Lam,
                                                             const T *__restrict__ Q, int64_t rows,
                                                             int64_t n, int64_t ld, int slot,
                                                             double *__restrict__ part) {
  __shared__ double sh[2][kWarps];
  const int64_t nch = (n + kDotCols - 1) / kDotCols;
  double dy = 0.0, dq = 0.0;
  Dot2 ay, aq;
  for (int64_t it = blockIdx.x; it < rows * nch; it += gridDim.x) {
    const int64_t r = it / nch, c = (it - r * nch) * kDotCols + threadIdx.x * 4;
    if (c >= n) continue;
    const int64_t o = r * ld;
    if constexpr (sizeof(T) == 4) {
      const float4 l = dot_load(Lam + o, c, n), y = dot_load(Y + o, c, n);
      if constexpr (kQ) {
        const float4 q = dot_load(Q + o, c, n);
        aq.add(l, q);
      }
      ay.add(l, y);
    } else {
#pragma unroll
      for (int i = 0; i < 4; ++i)
        if (c + i < n) {
          const double l = Lam[o + c + i];
          dy = fma(l, Y[o + c + i], dy);
          if constexpr (kQ) dq = fma(l, Q[o + c + i], dq);
        }
    }
  }
  if constexpr (sizeof(T) == 4) {
    dy = ay.value();
    dq = aq.value();
  }
  dy = warp_sum(dy);
  dq = warp_sum(dq);
  const int warp = threadIdx.x >> 5;
  if ((threadIdx.x & 31) == 0) {
    sh[0][warp] = dy;
    sh[1][warp] = dq;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    double t0 = 0.0, t1 = 0.0;
    for (int i = 0; i < kWarps; ++i) {
      t0 += sh[0][i];
      t1 += sh[1][i];
    }
    part[blockIdx.x * 3 + slot] = t0;
    if (kQ) part[blockIdx.x * 3 + 2] = t1;
  }
}

// out[i] = f_i sum_b part[b][i], f = (1, 1, scale); one warp a result
__global__ void panel_dot_sum_kernel(const double *__restrict__ part, int nb, double scale,
                                     double *__restrict__ out) {
  const int i = threadIdx.x >> 5, lane = threadIdx.x & 31;
  double t = 0.0;
  for (int b = lane; b < nb; b += 32) t += part[b * 3 + i];
  t = warp_sum(t);
  if (lane == 0) out[i] = i == 2 ? scale * t : t;
}

size_t panel_dot_bytes() { return (size_t)kDotBlocks * 3 * sizeof(double); }

static int panel_dot_blocks(int64_t rows, int64_t n) {
  const int64_t items = rows * ceil_div(n, kDotCols);
  return (int)(items < kDotBlocks ? items : kDotBlocks);
}

template <typename T>
int launch_panel_dot(const T *Y, const T *Lam, const T *Q, int64_t rows, int64_t n, int64_t ld,
                     int slot, double *part, cudaStream_t s) {
  const int nb = panel_dot_blocks(rows, n);
  if (Q)
    panel_dot_kernel<T, true><<<nb, kThreads, 0, s>>>(Y, Lam, Q, rows, n, ld, slot, part);
  else
    panel_dot_kernel<T, false><<<nb, kThreads, 0, s>>>(Y, Lam, Q, rows, n, ld, slot, part);
  return MFG_LAUNCH_STATUS();
}
template int launch_panel_dot<float>(const float *, const float *, const float *, int64_t, int64_t,
                                     int64_t, int, double *, cudaStream_t);
template int launch_panel_dot<double>(const double *, const double *, const double *, int64_t, int64_t,
                                      int64_t, int, double *, cudaStream_t);

int launch_panel_dot_sum(const double *part, int64_t rows, int64_t n, double scale, double *out,
                         cudaStream_t s) {
  panel_dot_sum_kernel<<<1, 96, 0, s>>>(part, panel_dot_blocks(rows, n), scale, out);
  return MFG_LAUNCH_STATUS();
}

// Quadrature values scale e1^T f(T) e1 and their cotangent in H from the
// eigendecomposition T = S diag(w) S^T: only the three diagonals of
// G = S (F o s1 s1^T) S^T are wanted, with s1 the first row of S and F the divided
// differences (f(w_a) - f(w_b)) / (w_a - w_b), f' at the midpoint for equal pairs.
// With u_ia = S_ia s1_a and, F being symmetric, the lower triangle
// M_i[a] = sum_{b<a} F_ab u_ib + F_aa u_ia / 2, G_ij = u_i . M_j + u_j . M_i.
//
// A CTA per probe, bound by the k^3 / 2 float64 multiply-adds (an SM takes one a
// warp every 19 cycles).  F lies in shared memory while it fits and in dH, which is
// written last, beyond; a warp takes kDhRows rows of u, so that one read of F serves
// them all.  The eigensolver and the cotangent of 32 probes of k = 24: 0.25 ms, where
// some thirty small batched operations took 0.74; 128 of k = 48: 0.50 ms, 0.73 before.
constexpr int kDhRows = 2;
constexpr int kDhThreads = 512;
constexpr size_t kDhSmem = 160 * 1024;

__global__ void __launch_bounds__(kDhThreads) quadform_dh_kernel(
    int k, const double *__restrict__ W, const double *__restrict__ S, const double *__restrict__ fW,
    const double *__restrict__ fpM, const double *__restrict__ scale, int shared_f,
    double *__restrict__ values, double *dH) {
  extern __shared__ double sh[];
  const int64_t b = blockIdx.x;
  const double *w = W + b * k, *s = S + b * k * k, *fw = fW + b * k, *fp = fpM + b * k * k;
  double *out = dH + b * k * k;
  double *gd = sh, *gy = sh + k, *gz = sh + 2 * k;  // u_i . M_i, u_{i+1} . M_i, u_{i-1} . M_i
  double *F = shared_f ? sh + 3 * k : out;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
  for (int64_t t = threadIdx.x; t < (int64_t)k * k; t += blockDim.x) {
    const int i = (int)(t / k), j = (int)(t - (int64_t)i * k);
    const double d = w[i] - w[j];
    const bool same = fabs(d) <= 1e-13 * fmax(fabs(w[i]), 1.0);
    F[t] = same ? fp[t] : (fw[i] - fw[j]) / d;
  }
  __syncthreads();
  for (int i0 = warp * kDhRows; i0 < k; i0 += nw * kDhRows) {
    double xd[kDhRows] = {}, xy[kDhRows] = {}, xz[kDhRows] = {};
    for (int a0 = 0; a0 < k; a0 += 32) {
      const int a = a0 + lane;
      const bool in = a < k;
      double M[kDhRows] = {};
      for (int b0 = 0; b0 <= a0; b0 += 32) {
        // u_i[b0 + lane], handed round by shuffles
        double u[kDhRows];
        const double s1 = b0 + lane < k ? s[b0 + lane] : 0.0;
#pragma unroll
        for (int r = 0; r < kDhRows; ++r)
          u[r] = (b0 + lane < k && i0 + r < k) ? s[(int64_t)(i0 + r) * k + b0 + lane] * s1 : 0.0;
        const int nb = k - b0 < 32 ? k - b0 : 32;
#pragma unroll 4
        for (int t = 0; t < nb; ++t) {
          const int bb = b0 + t;
          double f = (in && bb <= a) ? F[(int64_t)bb * k + a] : 0.0;
          if (bb == a) f *= 0.5;
#pragma unroll
          for (int r = 0; r < kDhRows; ++r) M[r] = fma(f, __shfl_sync(0xffffffffu, u[r], t), M[r]);
        }
      }
      if (in) {
        const double s1 = s[a];
#pragma unroll
        for (int r = 0; r < kDhRows; ++r) {
          const int i = i0 + r;
          if (i >= k) continue;
          const double m = M[r] * s1;
          xd[r] = fma(s[(int64_t)i * k + a], m, xd[r]);
          if (i + 1 < k) xy[r] = fma(s[(int64_t)(i + 1) * k + a], m, xy[r]);
          if (i > 0) xz[r] = fma(s[(int64_t)(i - 1) * k + a], m, xz[r]);
        }
      }
    }
#pragma unroll
    for (int r = 0; r < kDhRows; ++r) {
      const double d = warp_sum(xd[r]), y = warp_sum(xy[r]), z = warp_sum(xz[r]);
      if (lane == 0 && i0 + r < k) {
        gd[i0 + r] = d;
        gy[i0 + r] = y;
        gz[i0 + r] = z;
      }
    }
  }
  double v = 0.0;
  if (warp == 0) {
    for (int a = lane; a < k; a += 32) v = fma(fw[a] * s[a], s[a], v);
    v = warp_sum(v);
  }
  __syncthreads();
  const double sc = scale[b];
  if (threadIdx.x == 0) values[b] = sc * v;
  for (int64_t t = threadIdx.x; t < (int64_t)k * k; t += blockDim.x) {
    const int i = (int)(t / k), j = (int)(t - (int64_t)i * k);
    double g = 0.0;
    if (i == j)
      g = 2.0 * gd[i];
    else if (j == i + 1)
      g = gy[i] + gz[j];
    else if (i == j + 1)
      g = gy[j] + gz[i];
    out[t] = sc * g;
  }
}

int launch_quadform_dh(int64_t k, int64_t p, const double *w, const double *S, const double *fw,
                       const double *fp, const double *scale, double *values, double *dH, cudaStream_t s) {
  if (p <= 0) return MFG_OK;
  const size_t vecs = 3 * (size_t)k * 8, full = vecs + (size_t)k * k * 8;
  const bool shared_f = full <= kDhSmem;
  const size_t smem = shared_f ? full : vecs;
  if (smem > kDhSmem) return MFG_ERR_UNSUPPORTED;
  MFG_CUDA_TRY(cudaFuncSetAttribute(quadform_dh_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                    (int)kDhSmem));
  const int64_t want = 32 * ceil_div(k, kDhRows);
  quadform_dh_kernel<<<(unsigned)p, (unsigned)(want < kDhThreads ? want : kDhThreads), smem, s>>>(
      (int)k, w, S, fw, fp, scale, shared_f, values, dH);
  return MFG_LAUNCH_STATUS();
}

}  // namespace mfg
