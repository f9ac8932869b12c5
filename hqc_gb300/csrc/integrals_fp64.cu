// Analytic lattice-summed overlap / kinetic integrals and the Ewald sum (FP64).
//
// S and T follow hqc/pbc/solver.py:240-389: primitive s-s integrals summed
// over the lattice sphere, p functions obtained as derivatives with respect
// to the centres (the reference uses jacfwd).  Here those derivatives are
// closed-form Hermite derivatives of exp(-mu |R+t|^2); T = -1/2 lap_R S for
// s primitives, so every kinetic derivative is a sum of overlap derivatives.
// With forces, one more derivative gives dS/dR and dT/dR.
//
// The Ewald energy follows hqc/pbc/potential.py:6-67,103-130 (nearest-image
// real space, reciprocal sphere |G| <= Gmax, Madelung self term, Rydberg).
#include <cmath>
#include <vector>

#include "common.cuh"
#include "exp_table.cuh"
#include "kernels.h"

namespace hqcgb {

// h[n] = (d^n/dx^n e^{-mu x^2}) / e^{-mu x^2}, n = 0..5
__device__ inline void hermite6(double mu, double x, double *h) {
  h[0] = 1.0;
  h[1] = -2.0 * mu * x;
  for (int k = 1; k < 5; ++k) h[k + 1] = __fma_rn(h[1], h[k], -(2.0 * k * mu * h[k - 1]));
}

struct AOInfo {
  int l, cart;
};

// Two passes.  (1) One thread per (atom pair i, j; primitive pair a, b)
// accumulates over the lattice sphere the Hermite products
//   QS[m] = K_ab sum_t e_t h_m0(u_x) h_m1(u_y) h_m2(u_z),
//   QT[m] = K_ab sum_t e_t sum_d h_{m + 2 e_d}(u),   e_t = exp(-mu |R + t|^2),
// for every multi-index m an s/p pair needs: |m| <= 2 for S and T, |m| <= 3
// for their first derivatives (K_ab = (pi / (a + b))^(3/2)).  The exponential
// and the Hermite factors of a lattice term are computed once for all AO
// pairs.  (2) One thread per (i, j, p, q) contracts them with the
// coefficients: S_pq = sum_ab c'_pa c'_qb QS[m(p,q)], T = -1/2 (same with QT),
// and, with forces, the contribution D_pq dT/dR_i - W_pq dS/dR_i
// (R = R_i - R_j; the derivative with respect to R_j is its negative).
__constant__ int kMidx[20][3] = {{0, 0, 0}, {1, 0, 0}, {0, 1, 0}, {0, 0, 1}, {2, 0, 0},
                                 {0, 2, 0}, {0, 0, 2}, {1, 1, 0}, {1, 0, 1}, {0, 1, 1},
                                 {3, 0, 0}, {0, 3, 0}, {0, 0, 3}, {2, 1, 0}, {2, 0, 1},
                                 {1, 2, 0}, {0, 2, 1}, {1, 0, 2}, {0, 1, 2}, {1, 1, 1}};
// the same as a function, which folds in unrolled loops (registers, no constant loads)
__device__ constexpr int midx(int q, int d) {
  const int t[20][3] = {{0, 0, 0}, {1, 0, 0}, {0, 1, 0}, {0, 0, 1}, {2, 0, 0}, {0, 2, 0}, {0, 0, 2},
                        {1, 1, 0}, {1, 0, 1}, {0, 1, 1}, {3, 0, 0}, {0, 3, 0}, {0, 0, 3}, {2, 1, 0},
                        {2, 0, 1}, {1, 2, 0}, {0, 2, 1}, {1, 0, 2}, {0, 1, 2}, {1, 1, 1}};
  return t[q][d];
}
constexpr int kNq = 20;  // slots per (i, j, a, b): QS[20], QT[20]

__device__ inline int midx_of(int m0, int m1, int m2) {
  for (int k = 0; k < kNq; ++k)
    if (kMidx[k][0] == m0 && kMidx[k][1] == m1 && kMidx[k][2] == m2) return k;
  return 0;
}

// The general form, for any list of lattice vectors, one warp per sum.  The
// lanes take one vector each: they drop the images beyond exp(-60), queue the
// others in their order, and form the exponential and the Hermite products of 32
// queued vectors in shared memory; then lane s adds the s-th of the 2 NQ sums
// (4 NQ at a k-point) over the 32 vectors in that order, so that the sums are
// those of one thread going through the list (the multiply-adds are written
// out, so that no compiler choice moves them).  KPT: each lattice term also
// carries exp(-i k.t) (hqc/pbc/solver.py:257-274); the real and imaginary sums
// are stored side by side, Q[(i,j,a,b)][4][kNq] = {QS re, QT re, QS im, QT im}.
// Bound by the FP64 pipe (some 200 instructions a vector kept).  With a thread a
// sum a small molecule left most of the chip idle: H8 szv has 576 to 2,304 sums
// of 870 vectors.  Measured, S and T of one configuration, a thread -> a warp a
// sum: H8 szv (box 4.1 Bohr) 4.71 -> 0.21 ms, H8 dzv
// at a k-point 4.37 -> 0.23.
template <int NQ, bool KPT>
__global__ void __launch_bounds__(128)
    k_ovl_lattice(const double *__restrict__ xp, int n, int nprim, const double *__restrict__ alpha,
                  const double *__restrict__ lattice, int nlat, const double *__restrict__ kpt,
                  double *__restrict__ Q) {
  constexpr int NH = 2 * NQ, NS = KPT ? 2 * NH : NH, ROW = NH + (KPT ? 3 : 1);  // odd rows: no bank conflicts
  constexpr int NR = (NS + 31) / 32;
  __shared__ double val[4][32][ROW];  // a vector's products S, T; exponential (re, im)
  __shared__ int queue[4][64];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const long long idx = (long long)blockIdx.x * 4 + warp;
  const int np2 = nprim * nprim;
  if (idx >= (long long)n * n * np2) return;
  // atom pairs fastest: the warps of a block share one primitive pair (one mu),
  // so they keep about as many vectors
  const int ab = (int)(idx / ((long long)n * n)), a = ab / nprim, b = ab % nprim;
  const int ij = (int)(idx % ((long long)n * n)), i = ij / n, j = ij % n;
  double R[3];
  for (int d = 0; d < 3; ++d) R[d] = xp[i * 3 + d] - xp[j * 3 + d];
  const double asum = alpha[a] + alpha[b];
  const double mu = alpha[a] * alpha[b] / asum;
  const double K = pow(M_PI / asum, 1.5);
  int *q = queue[warp];
  auto exponent = [&](int t, double (&u)[3]) {
    double u2 = 0;
    for (int d = 0; d < 3; ++d) {
      u[d] = R[d] + lattice[t * 3 + d];
      u2 += u[d] * u[d];
    }
    return mu * u2;
  };
  double acc[NR];
#pragma unroll
  for (int r = 0; r < NR; ++r) acc[r] = 0.0;
  auto add = [&](int m) {  // the first m <= 32 queued vectors
    if (lane < m) {
      double *row = val[warp][lane];
      const int t = q[lane];
      double u[3];
      const double e0 = exponent(t, u);
      double e = K * exp(-e0);
      if (KPT) {
        double sn, cs;
        const double *tv = lattice + t * 3;
        sincos(-__fma_rn(kpt[2], tv[2], __fma_rn(kpt[0], tv[0], kpt[1] * tv[1])), &sn, &cs);
        row[NH + 1] = e * sn;
        e *= cs;
      }
      row[NH] = e;
      double hx[6], hy[6], hz[6];
      hermite6(mu, u[0], hx);
      hermite6(mu, u[1], hy);
      hermite6(mu, u[2], hz);
#pragma unroll
      for (int k = 0; k < NQ; ++k) {
        const int m0 = midx(k, 0), m1 = midx(k, 1), m2 = midx(k, 2);
        row[k] = hx[m0] * hy[m1] * hz[m2];
        row[NQ + k] = __fma_rn(hx[m0] * hy[m1], hz[m2 + 2],
                               __fma_rn(hx[m0 + 2] * hy[m1], hz[m2], hx[m0] * hy[m1 + 2] * hz[m2]));
      }
    }
    __syncwarp();
    for (int v = 0; v < m; ++v) {
#pragma unroll
      for (int r = 0; r < NR; ++r) {
        const int s = lane + 32 * r;
        if (s < NS) acc[r] = fma(val[warp][v][NH + s / NH], val[warp][v][s % NH], acc[r]);
      }
    }
    __syncwarp();
  };
  int have = 0;
  for (int t0 = 0; t0 < nlat; t0 += 32) {
    const int t = t0 + lane;
    double u[3];
    // exp(-60) times the largest Hermite factor (degree <= 5) is below 1e-18
    // of every matrix element: far images add nothing in FP64
    const bool keep = t < nlat && !(exponent(t, u) > 60.0);
    const unsigned mask = __ballot_sync(~0u, keep);
    if (keep) q[have + __popc(mask & ((1u << lane) - 1u))] = t;
    have += __popc(mask);
    __syncwarp();
    if (have >= 32) {
      add(32);
      have -= 32;
      if (lane < have) q[lane] = q[32 + lane];
      __syncwarp();
    }
  }
  if (have) add(have);
  double *out = Q + (((long long)i * n + j) * np2 + ab) * ((KPT ? 4 : 2) * kNq);
#pragma unroll
  for (int r = 0; r < NR; ++r) {
    const int s = lane + 32 * r;
    if (s < NS) out[s / NQ * kNq + s % NQ] = acc[r];
  }
}

// The lattice sums where the lattice is a sphere (or any set symmetric in
// every axis) of a cubic lattice: exp(-mu |R + t|^2) h_m0 h_m1 h_m2 is a product
// over the axes, so with x_i(t) = exp(-mu (R_x + t)^2) h_i (likewise y, z) and
// the set's rows |t_z| <= m(t_x, t_y),
//   sum = sum_{ty} y_j sum_{tx} x_i Zc_k[m(tx, ty)],  Zc_k[m] = sum_{|tz| <= m} z_k(tz):
// an exponential a translation and axis instead of one a lattice vector, and
// (KD + 1)(KD + 2) / 2 multiply-adds a row of the sphere instead of the NQ
// triple products (and their six Laplacian terms) a vector.  One thread per
// (i <= j; a, b); the pair (j, i; b, a) follows from R -> -R, t -> -t: a sign
// (-1)^|m| (and the conjugate at a k-point).  Bound by the FP64 pipe; one-warp
// blocks, so that a few atoms' pairs still spread over the chip.  Measured, S
// and T of one configuration, vector by vector -> by rows: H54 dzvp (box 8 Bohr)
// 1.99 -> 0.13 ms, H8 szv (box 4.1 Bohr, 870 vectors) 4.7 -> 0.1 ms.
template <typename Z> struct OvlZ;
template <> struct OvlZ<double> {
  static __device__ double zero() { return 0.0; }
  static __device__ double phase(double, double) { return 1.0; }
  static __device__ double conj(double a) { return a; }
};
template <> struct OvlZ<double2> {
  static __device__ double2 zero() { return make_double2(0.0, 0.0); }
  static __device__ double2 phase(double k, double t) {  // exp(-i k t)
    double s, c;
    sincos(-k * t, &s, &c);
    return make_double2(c, s);
  }
  static __device__ double2 conj(double2 a) { return make_double2(a.x, -a.y); }
};
__device__ inline double ovl_scale(double s, double z) { return s * z; }
__device__ inline double2 ovl_scale(double s, double2 z) { return make_double2(s * z.x, s * z.y); }
__device__ inline void ovl_fma(double a, double b, double &s) { s = fma(a, b, s); }
__device__ inline void ovl_fma(double2 a, double2 b, double2 &s) {
  s.x = fma(a.x, b.x, fma(-a.y, b.y, s.x));
  s.y = fma(a.x, b.y, fma(a.y, b.x, s.y));
}
__device__ inline void ovl_add(double a, double &s) { s += a; }
__device__ inline void ovl_add(double2 a, double2 &s) {
  s.x += a.x;
  s.y += a.y;
}

template <int NQ, typename Z>
__global__ void __launch_bounds__(32)
    k_ovl_rows(const double *__restrict__ xp, int n, int nprim, const double *__restrict__ alpha,
               const __grid_constant__ OvlRows rows, const double *__restrict__ kpt, double *__restrict__ Q) {
  constexpr bool KPT = sizeof(Z) > sizeof(double);
  constexpr int KD = NQ == 10 ? 4 : 5;  // Hermite orders 0..KD along an axis
  using O = OvlZ<Z>;
  __shared__ double tab[kExpTable];
  for (int k = threadIdx.x; k < kExpTable; k += 32) tab[k] = exp2(k / 64.0);
  __syncwarp();
  const long long idx = (long long)blockIdx.x * 32 + threadIdx.x;
  const int npair = n * (n + 1) / 2, np2 = nprim * nprim;
  if (idx >= (long long)npair * np2) return;
  const int ab = (int)(idx / npair), a = ab / nprim, b = ab % nprim;
  const int pr = (int)(idx % npair);  // pair i <= j at j (j + 1) / 2 + i
  int j = (int)((sqrtf(8.f * pr + 1.f) - 1.f) * 0.5f);
  while (j * (j + 1) / 2 > pr) --j;
  while ((j + 1) * (j + 2) / 2 <= pr) ++j;
  const int i = pr - j * (j + 1) / 2;
  const double asum = alpha[a] + alpha[b], mu = alpha[a] * alpha[b] / asum, s = M_PI / asum;
  const double K = s * sqrt(s);
  const int tm = rows.tmax, side = 2 * tm + 1;
  // h_k(u) exp(-mu u^2), k = 0..KD, with the phase of translation t; false (nothing) below e^-60
  auto term = [&](double R, double t, double kc, Z *out) {
    const double u = R + t, arg = mu * u * u;
    if (arg > 60.0) return false;
    const double e = exp_neg(-arg, tab), g = -2.0 * mu * u;
    const Z ph = O::phase(kc, t);
    double h0 = e, h1 = g * e;
    out[0] = ovl_scale(h0, ph);
    out[1] = ovl_scale(h1, ph);
#pragma unroll
    for (int k = 1; k < KD; ++k) {
      const double h2 = g * h1 - 2.0 * k * mu * h0;
      out[k + 1] = ovl_scale(h2, ph);
      h0 = h1;
      h1 = h2;
    }
    return true;
  };
  double R[3], kc[3] = {0, 0, 0};
  for (int d = 0; d < 3; ++d) {
    R[d] = xp[i * 3 + d] - xp[j * 3 + d];
    if (KPT) kc[d] = kpt[d];
  }
  Z X[2 * kOvlMaxT + 1][KD + 1], Zc[kOvlMaxT + 1][KD + 1], y[KD + 1], acc[KD + 1];
  int lo = side, hi = -1;  // the x translations that count
  for (int t = 0; t < side; ++t)
    if (term(R[0], (t - tm) * rows.a, kc[0], X[t])) {
      lo = min(lo, t);
      hi = t;
    }
#pragma unroll
  for (int k = 0; k <= KD; ++k) acc[k] = O::zero();
  for (int m = 0; m <= tm; ++m) {
    for (int sg = m == 0 ? 1 : -1; sg <= 1; sg += 2)
      if (term(R[2], sg * (m * rows.a), kc[2], y))
#pragma unroll
        for (int k = 0; k <= KD; ++k) ovl_add(y[k], acc[k]);
#pragma unroll
    for (int k = 0; k <= KD; ++k) Zc[m][k] = acc[k];
  }
  Z qs[NQ], qt[NQ];
#pragma unroll
  for (int k = 0; k < NQ; ++k) qs[k] = qt[k] = O::zero();
  for (int ty = 0; ty < side; ++ty) {
    if (!term(R[1], (ty - tm) * rows.a, kc[1], y)) continue;
    Z P[KD + 1][KD + 1];
#pragma unroll
    for (int p = 0; p <= KD; ++p)
#pragma unroll
      for (int k = 0; k <= KD - p; ++k) P[p][k] = O::zero();
    for (int tx = lo; tx <= hi; ++tx) {
      const int m = rows.m[tx * side + ty];
      if (m < 0) continue;
#pragma unroll
      for (int p = 0; p <= KD; ++p)
#pragma unroll
        for (int k = 0; k <= KD - p; ++k) ovl_fma(X[tx][p], Zc[m][k], P[p][k]);
    }
#pragma unroll
    for (int q = 0; q < NQ; ++q) {
      const int m0 = midx(q, 0), m1 = midx(q, 1), m2 = midx(q, 2);
      ovl_fma(y[m1], P[m0][m2], qs[q]);
      ovl_fma(y[m1], P[m0 + 2][m2], qt[q]);
      ovl_fma(y[m1 + 2], P[m0][m2], qt[q]);
      ovl_fma(y[m1], P[m0][m2 + 2], qt[q]);
    }
  }
  constexpr int W = (KPT ? 4 : 2) * kNq;
  double *out = Q + (((long long)i * n + j) * np2 + ab) * W;
  double *mir = Q + (((long long)j * n + i) * np2 + b * nprim + a) * W;
#pragma unroll
  for (int q = 0; q < NQ; ++q) {
    const double sg = (midx(q, 0) + midx(q, 1) + midx(q, 2)) & 1 ? -K : K;
    const Z vs = ovl_scale(K, qs[q]), vt = ovl_scale(K, qt[q]);
    const Z ms = ovl_scale(sg, O::conj(qs[q])), mt = ovl_scale(sg, O::conj(qt[q]));
    if constexpr (KPT) {
      out[q] = vs.x; out[kNq + q] = vt.x; out[2 * kNq + q] = vs.y; out[3 * kNq + q] = vt.y;
      if (i != j) { mir[q] = ms.x; mir[kNq + q] = mt.x; mir[2 * kNq + q] = ms.y; mir[3 * kNq + q] = mt.y; }
    } else {
      out[q] = vs; out[kNq + q] = vt;
      if (i != j) { mir[q] = ms; mir[kNq + q] = mt; }
    }
  }
}

OvlRows ovl_rows(const double *lattice, int nlat) {
  OvlRows r{};
  r.tmax = -1;
  double a = 0;
  for (int k = 0; k < 3 * nlat; ++k) {
    const double v = std::fabs(lattice[k]);
    if (!std::isfinite(v)) return r;
    if (v > 0 && (a == 0 || v < a)) a = v;
  }
  if (nlat < 1) return r;
  if (a == 0) a = 1.0;
  int tm = 0;
  for (int k = 0; k < 3 * nlat; ++k) {
    const double q = lattice[k] / a, z = std::rint(q);
    if (std::fabs(z) > kOvlMaxT || std::fabs(lattice[k] - z * a) > 4e-16 * std::fabs(lattice[k])) return r;
    tm = std::max(tm, (int)std::fabs(z));
  }
  const int side = 2 * tm + 1;
  std::vector<int> seen((size_t)side * side * side, 0);
  for (int k = 0; k < nlat; ++k) {
    int c[3];
    for (int d = 0; d < 3; ++d) c[d] = (int)std::rint(lattice[3 * k + d] / a) + tm;
    if (seen[(c[0] * side + c[1]) * side + c[2]]++) return r;  // a vector twice
  }
  for (int x = 0; x < side; ++x)
    for (int y = 0; y < side; ++y) {
      const int *col = seen.data() + (x * side + y) * side;
      int m = -1;
      while (m < tm && col[tm + m + 1]) ++m;
      for (int z = 0; z < side; ++z)
        if (col[z] != (std::abs(z - tm) <= m ? 1 : 0)) return r;  // not |t_z| <= m
      r.m[x * side + y] = (signed char)m;
    }
  for (int x = 0; x < side; ++x)
    for (int y = 0; y < side; ++y)
      if (r.m[x * side + y] != r.m[(side - 1 - x) * side + side - 1 - y]) return r;
  r.a = a;
  r.tmax = tm;
  return r;
}

__global__ void k_ovl_contract(int n, int nb, int nprim, const double *__restrict__ alpha,
                               const double *__restrict__ coef, const int *__restrict__ ao_l,
                               const int *__restrict__ ao_cart, const double *__restrict__ Q,
                               double *__restrict__ S, double *__restrict__ T,
                               const double *__restrict__ D, const double *__restrict__ W,
                               double *__restrict__ gpart) {
  const long long idx = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (idx >= (long long)n * n * nb * nb) return;
  const int q = (int)(idx % nb), p = (int)((idx / nb) % nb);
  const int j = (int)((idx / ((long long)nb * nb)) % n), i = (int)(idx / ((long long)nb * nb * n));
  const int nao = n * nb, np2 = nprim * nprim;
  const int lp = ao_l[p], lq = ao_l[q];
  int mb[3] = {0, 0, 0};
  if (lp) mb[ao_cart[p]] += 1;
  if (lq) mb[ao_cart[q]] += 1;
  const bool grad = gpart != nullptr;
  const int ks = midx_of(mb[0], mb[1], mb[2]);
  int kc[3];
  for (int c = 0; c < 3; ++c) kc[c] = midx_of(mb[0] + (c == 0), mb[1] + (c == 1), mb[2] + (c == 2));
  double sS = 0, sT = 0, gS[3] = {0, 0, 0}, gT[3] = {0, 0, 0};
  const double *Qij = Q + ((long long)i * n + j) * np2 * (2 * kNq);
  for (int a = 0; a < nprim; ++a) {
    double ca = coef[p * nprim + a];
    if (ca == 0.0) continue;
    if (lp) ca *= 0.5 / alpha[a];
    for (int b = 0; b < nprim; ++b) {
      double cb = coef[q * nprim + b];
      if (cb == 0.0) continue;
      if (lq) cb *= -0.5 / alpha[b];
      const double cc = ca * cb;
      const double *qv = Qij + (long long)(a * nprim + b) * (2 * kNq);
      sS += cc * qv[ks];
      sT += cc * qv[kNq + ks];
      if (grad)
        for (int c = 0; c < 3; ++c) {
          gS[c] += cc * qv[kc[c]];
          gT[c] += cc * qv[kNq + kc[c]];
        }
    }
  }
  const long long pq = (long long)(i * nb + p) * nao + (j * nb + q);
  if (S) S[pq] = sS;
  if (T) T[pq] = -0.5 * sT;
  if (grad) {
    const double dd = D[pq], ww = W[pq];
    for (int c = 0; c < 3; ++c) gpart[idx * 3 + c] = (i == j) ? 0.0 : dd * (-0.5 * gT[c]) - ww * gS[c];
  }
}

// k-point contraction: complex S, T (interleaved) from the phase-weighted
// sums and, with gpart, Re[conj(D_pq) dT_pq - conj(W_pq) dS_pq] per (i, j, p, q)
// (Re tr(D dT) for Hermitian D: sum_pq D_qp dT_pq = sum_pq conj(D_pq) dT_pq).
__global__ void k_ovl_contract_kpt(int n, int nb, int nprim, const double *__restrict__ alpha,
                                   const double *__restrict__ coef, const int *__restrict__ ao_l,
                                   const int *__restrict__ ao_cart, const double *__restrict__ Q,
                                   double2 *__restrict__ S, double2 *__restrict__ T,
                                   const double2 *__restrict__ D, const double2 *__restrict__ W,
                                   double *__restrict__ gpart) {
  const long long idx = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (idx >= (long long)n * n * nb * nb) return;
  const int q = (int)(idx % nb), p = (int)((idx / nb) % nb);
  const int j = (int)((idx / ((long long)nb * nb)) % n), i = (int)(idx / ((long long)nb * nb * n));
  const int nao = n * nb, np2 = nprim * nprim;
  const int lp = ao_l[p], lq = ao_l[q];
  int mb[3] = {0, 0, 0};
  if (lp) mb[ao_cart[p]] += 1;
  if (lq) mb[ao_cart[q]] += 1;
  const int ks = midx_of(mb[0], mb[1], mb[2]);
  const bool grad = gpart != nullptr;
  int kc[3];
  for (int c = 0; c < 3; ++c) kc[c] = midx_of(mb[0] + (c == 0), mb[1] + (c == 1), mb[2] + (c == 2));
  double sS = 0, sT = 0, sSi = 0, sTi = 0;
  double gS[3] = {0, 0, 0}, gT[3] = {0, 0, 0}, gSi[3] = {0, 0, 0}, gTi[3] = {0, 0, 0};
  const double *Qij = Q + ((long long)i * n + j) * np2 * (4 * kNq);
  for (int a = 0; a < nprim; ++a) {
    double ca = coef[p * nprim + a];
    if (ca == 0.0) continue;
    if (lp) ca *= 0.5 / alpha[a];
    for (int b = 0; b < nprim; ++b) {
      double cb = coef[q * nprim + b];
      if (cb == 0.0) continue;
      if (lq) cb *= -0.5 / alpha[b];
      const double cc = ca * cb;
      const double *qv = Qij + (long long)(a * nprim + b) * (4 * kNq);
      sS += cc * qv[ks];
      sT += cc * qv[kNq + ks];
      sSi += cc * qv[2 * kNq + ks];
      sTi += cc * qv[3 * kNq + ks];
      if (grad)
        for (int c = 0; c < 3; ++c) {
          gS[c] += cc * qv[kc[c]];
          gT[c] += cc * qv[kNq + kc[c]];
          gSi[c] += cc * qv[2 * kNq + kc[c]];
          gTi[c] += cc * qv[3 * kNq + kc[c]];
        }
    }
  }
  const long long pq = (long long)(i * nb + p) * nao + (j * nb + q);
  if (S) S[pq] = make_double2(sS, sSi);
  if (T) T[pq] = make_double2(-0.5 * sT, -0.5 * sTi);
  if (grad) {
    const double2 dd = D[pq], ww = W[pq];
    for (int c = 0; c < 3; ++c)
      gpart[idx * 3 + c] = (i == j) ? 0.0
                                    : -0.5 * (dd.x * gT[c] + dd.y * gTi[c]) - (ww.x * gS[c] + ww.y * gSi[c]);
  }
}

size_t ovl_scratch_doubles(int n, int nprim) {
  return (size_t)n * n * nprim * nprim * 2 * kNq;
}
size_t ovl_scratch_doubles_kpt(int n, int nprim) {
  return (size_t)n * n * nprim * nprim * 4 * kNq;
}

// grad[A][c] += sum_{j,p,q} gpart(A,j,p,q) - sum_{i,p,q} gpart(i,A,p,q)
__global__ void k_reduce_pair_grad(const double *__restrict__ gpart, int n, int nb,
                                   double *__restrict__ grad) {
  __shared__ double sh[32];
  int A = blockIdx.x;
  long long per = (long long)nb * nb;
  for (int c = 0; c < 3; ++c) {
    double s = 0;
    for (long long k = threadIdx.x; k < (long long)n * per; k += blockDim.x) {
      int o = (int)(k / per);
      long long pq = k % per;
      s += gpart[(((long long)A * n + o) * per + pq) * 3 + c];
      s -= gpart[(((long long)o * n + A) * per + pq) * 3 + c];
    }
    s = block_sum(s, sh);
    if (threadIdx.x == 0) grad[A * 3 + c] += s;
    __syncthreads();
  }
}

void launch_overlap_kinetic(const double *xp, int n, int nb, int nprim, const double *alpha,
                            const double *coef, const int *ao_l, const int *ao_cart,
                            const double *lattice, int nlat, const OvlRows &rows, double *S, double *T,
                            const double *D, const double *W, double *gpart, double *grad, double *Q,
                            cudaStream_t st) {
  HQ_STAGE(ST_OVERLAP, st);
  const long long terms = (long long)n * n * nprim * nprim;
  const int blocks = ceil_div((long long)(n * (n + 1) / 2) * nprim * nprim, 32);
  if (rows.tmax >= 0 && gpart)
    k_ovl_rows<20, double><<<blocks, 32, 0, st>>>(xp, n, nprim, alpha, rows, nullptr, Q);
  else if (rows.tmax >= 0)
    k_ovl_rows<10, double><<<blocks, 32, 0, st>>>(xp, n, nprim, alpha, rows, nullptr, Q);
  else if (gpart)
    k_ovl_lattice<20, false><<<ceil_div(terms, 4), 128, 0, st>>>(xp, n, nprim, alpha, lattice, nlat,
                                                                   nullptr, Q);
  else
    k_ovl_lattice<10, false><<<ceil_div(terms, 4), 128, 0, st>>>(xp, n, nprim, alpha, lattice, nlat,
                                                                   nullptr, Q);
  HQ_LAUNCH_CHECK();
  const long long total = (long long)n * n * nb * nb;
  k_ovl_contract<<<ceil_div(total, 128), 128, 0, st>>>(n, nb, nprim, alpha, coef, ao_l, ao_cart, Q, S,
                                                      T, D, W, gpart);
  HQ_LAUNCH_CHECK();
  if (gpart) {
    k_reduce_pair_grad<<<n, 256, 0, st>>>(gpart, n, nb, grad);
    HQ_LAUNCH_CHECK();
  }
}

// S^k, T^k at k-point kpt (device, 1/Bohr): complex Hermitian, interleaved.
void launch_overlap_kinetic_kpt(const double *xp, int n, int nb, int nprim, const double *alpha,
                                const double *coef, const int *ao_l, const int *ao_cart,
                                const double *lattice, int nlat, const OvlRows &rows, const double *kpt,
                                double2 *S, double2 *T, double *Q, cudaStream_t st, const double2 *D,
                                const double2 *W, double *gpart, double *grad) {
  HQ_STAGE(ST_OVERLAP, st);
  const long long terms = (long long)n * n * nprim * nprim;
  const int blocks = ceil_div((long long)(n * (n + 1) / 2) * nprim * nprim, 32);
  if (rows.tmax >= 0 && gpart)
    k_ovl_rows<20, double2><<<blocks, 32, 0, st>>>(xp, n, nprim, alpha, rows, kpt, Q);
  else if (rows.tmax >= 0)
    k_ovl_rows<10, double2><<<blocks, 32, 0, st>>>(xp, n, nprim, alpha, rows, kpt, Q);
  else if (gpart)
    k_ovl_lattice<20, true><<<ceil_div(terms, 4), 128, 0, st>>>(xp, n, nprim, alpha, lattice, nlat,
                                                                  kpt, Q);
  else
    k_ovl_lattice<10, true><<<ceil_div(terms, 4), 128, 0, st>>>(xp, n, nprim, alpha, lattice, nlat,
                                                                  kpt, Q);
  HQ_LAUNCH_CHECK();
  const long long total = (long long)n * n * nb * nb;
  k_ovl_contract_kpt<<<ceil_div(total, 128), 128, 0, st>>>(n, nb, nprim, alpha, coef, ao_l, ao_cart,
                                                          Q, S, T, D, W, gpart);
  HQ_LAUNCH_CHECK();
  if (gpart) {
    k_reduce_pair_grad<<<n, 256, 0, st>>>(gpart, n, nb, grad);
    HQ_LAUNCH_CHECK();
  }
}

// ---------------------------------------------------------------------------
// Ewald (potential.py:103-130).  xp in rs units, L in rs units; energy in Ry,
// grad in Ry per rs unit.  psi(r) = erfc(kappa |r|)/|r| (nearest image) +
// sum_G g(G) cos(2 pi G.r) + g0 over 0 < |G|^2 <= Gmax^2 (L = 1 units).  The
// reciprocal part of sum_{i<j} psi(r_ij) is taken from the structure factor
// S(G) = sum_i exp(2 pi i G.x_i / L):  sum_{i<j} cos(2 pi G.r_ij) =
// (|S|^2 - n) / 2, and its derivative with respect to atom a is
// -2 pi G Im(conj(S) exp(2 pi i G.x_a / L)) -- n N_G phases instead of the
// pairwise n^2 N_G / 2.
// ---------------------------------------------------------------------------
constexpr int kEwThreads = 256;

__device__ inline bool ewald_g(long long k, int gmax, int &gx, int &gy, int &gz, int &G2) {
  const int side = 2 * gmax + 1;
  gx = (int)(k / ((long long)side * side)) - gmax;
  gy = (int)((k / side) % side) - gmax;
  gz = (int)(k % side) - gmax;
  G2 = gx * gx + gy * gy + gz * gz;
  return G2 != 0 && G2 <= gmax * gmax;
}

__device__ inline double ewald_gk(int G2, double kappa) {
  return exp(-M_PI * M_PI * G2 / (kappa * kappa)) / (M_PI * G2);
}

// ewald_gk of every |G|^2 <= gmax^2 in shared memory, up to kEwTable - 1: the cube's
// points share some hundred values.  Ends with a block barrier.
constexpr int kEwTable = 1024;
__device__ inline bool ewald_table(int gmax, double kappa, double *tab) {
  const bool fits = gmax * gmax < kEwTable;
  for (int k = 1 + threadIdx.x; fits && k <= gmax * gmax; k += blockDim.x) tab[k] = ewald_gk(k, kappa);
  __syncthreads();
  return fits;
}

// S(G) per cube point (0 outside the sphere) and the reciprocal energy per block
__global__ void __launch_bounds__(kEwThreads)
    k_ewald_sf(const double *__restrict__ xp, int n, double L, double kappa, int gmax,
               double2 *__restrict__ S, double *__restrict__ part_e) {
  __shared__ double sh[32];
  const int side = 2 * gmax + 1;
  const long long nG = (long long)side * side * side;
  const long long k = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  double e = 0;
  if (k < nG) {
    int gx, gy, gz, G2;
    double sr = 0, si = 0;
    if (ewald_g(k, gmax, gx, gy, gz, G2)) {
      for (int i = 0; i < n; ++i) {
        const double ph = (gx * xp[i * 3] + gy * xp[i * 3 + 1] + gz * xp[i * 3 + 2]) / L;
        double sn, cs;
        sincospi(2.0 * ph, &sn, &cs);
        sr += cs;
        si += sn;
      }
      e = ewald_gk(G2, kappa) * 0.5 * (sr * sr + si * si - n);
    }
    S[k] = make_double2(sr, si);
  }
  e = block_sum(e, sh);
  if (threadIdx.x == 0) part_e[blockIdx.x] = e;
}

// reciprocal derivative of sum_{i<j} psi with respect to r_a (L = 1 units); one block per
// atom.  Bound by the FP64 pipe (exponential and sincospi a point).  54 atoms, Gmax
// 15, the exponentials from the table: 0.51 -> 0.31 ms; k_ewald_finish, whose atoms
// also take their own pairs only, 0.54 -> 0.08.
__global__ void __launch_bounds__(kEwThreads)
    k_ewald_recip_grad(const double *__restrict__ xp, int n, double L, double kappa, int gmax,
                       const double2 *__restrict__ S, double *__restrict__ gr) {
  __shared__ double sh[32], tab[kEwTable];
  const bool fits = ewald_table(gmax, kappa, tab);
  const int a = blockIdx.x;
  const int side = 2 * gmax + 1;
  const long long nG = (long long)side * side * side;
  double g0 = 0, g1 = 0, g2 = 0;
  for (long long k = threadIdx.x; k < nG; k += blockDim.x) {
    int gx, gy, gz, G2;
    if (!ewald_g(k, gmax, gx, gy, gz, G2)) continue;
    const double ph = (gx * xp[a * 3] + gy * xp[a * 3 + 1] + gz * xp[a * 3 + 2]) / L;
    double sn, cs;
    sincospi(2.0 * ph, &sn, &cs);
    const double2 sk = S[k];
    const double f = -2.0 * M_PI * (fits ? tab[G2] : ewald_gk(G2, kappa)) * (sk.x * sn - sk.y * cs);
    g0 += f * gx;
    g1 += f * gy;
    g2 += f * gz;
  }
  g0 = block_sum(g0, sh);
  g1 = block_sum(g1, sh);
  g2 = block_sum(g2, sh);
  if (threadIdx.x == 0) {
    gr[a * 3] = g0;
    gr[a * 3 + 1] = g1;
    gr[a * 3 + 2] = g2;
  }
}

// nearest-image real-space term and its derivative, one thread per pair (i < j)
__global__ void k_ewald_real(const double *__restrict__ xp, int n, double L, double kappa,
                             double *__restrict__ pair_e, double *__restrict__ pair_g) {
  const int npair = n * (n - 1) / 2;
  const int pidx = blockIdx.x * blockDim.x + threadIdx.x;
  if (pidx >= npair) return;
  int i = 0, rem = pidx;
  while (rem >= n - 1 - i) {
    rem -= n - 1 - i;
    ++i;
  }
  const int j = i + 1 + rem;
  double r[3];
  for (int d = 0; d < 3; ++d) {
    const double a = xp[i * 3 + d] - L * floor(xp[i * 3 + d] / L);
    const double b = xp[j * 3 + d] - L * floor(xp[j * 3 + d] / L);
    const double x = (a - b) / L;
    r[d] = x - rint(x);
  }
  const double dd = sqrt(r[0] * r[0] + r[1] * r[1] + r[2] * r[2]);
  const double sr = erfc(kappa * dd) / dd;
  const double dsr = -2.0 * kappa / sqrt(M_PI) * exp(-kappa * kappa * dd * dd) / dd - sr / dd;
  pair_e[pidx] = sr;
  for (int d = 0; d < 3; ++d) pair_g[pidx * 3 + d] = dsr * r[d] / dd;
}

__global__ void k_ewald_finish(const double *__restrict__ pair_e, const double *__restrict__ pair_g,
                               const double *__restrict__ part_e, int nblk, const double *__restrict__ gr,
                               int n, double L, double rs, double kappa, int gmax,
                               double *__restrict__ energy, double *__restrict__ grad) {
  __shared__ double sh[32], tab[kEwTable];
  const bool fits = ewald_table(gmax, kappa, tab);
  const int npair = n * (n - 1) / 2;
  double s = 0;
  for (int k = threadIdx.x; k < npair; k += blockDim.x) s += pair_e[k];
  for (int k = threadIdx.x; k < nblk; k += blockDim.x) s += part_e[k];
  s = block_sum(s, sh);
  // Madelung constant of the unit simple-cubic lattice with this kappa / Gmax
  double m = 0;
  const int side = 2 * gmax + 1;
  const long long nG = (long long)side * side * side;
  for (long long k = threadIdx.x; k < nG; k += blockDim.x) {
    int gx, gy, gz, G2;
    if (ewald_g(k, gmax, gx, gy, gz, G2)) m += fits ? tab[G2] : ewald_gk(G2, kappa);
  }
  m = block_sum(m, sh);
  if (threadIdx.x == 0) {
    const double g0 = -M_PI / (kappa * kappa);
    const double mad = m + g0 - 2.0 * kappa / sqrt(M_PI);
    *energy = 2.0 * (s + npair * g0) / L / rs + n * mad / L / rs;
  }
  if (grad) {
    for (int a = threadIdx.x; a < n; a += blockDim.x) {
      double acc[3] = {gr[a * 3], gr[a * 3 + 1], gr[a * 3 + 2]};
      // the atom's pairs (i < a, a), then (a, j > a): pair (i, j) at i (2 n - i - 1) / 2 + j - i - 1
      for (int o = 0; o < n; ++o) {
        if (o == a) continue;
        const int i = min(o, a), j = max(o, a), k = i * (2 * n - i - 1) / 2 + j - i - 1;
        for (int d = 0; d < 3; ++d) acc[d] += o > a ? pair_g[k * 3 + d] : -pair_g[k * 3 + d];
      }
      for (int d = 0; d < 3; ++d) grad[a * 3 + d] = 2.0 * acc[d] / (L * L * rs);
    }
  }
}

size_t ewald_work_doubles(int n, int gmax) {
  const long long side = 2LL * gmax + 1, nG = side * side * side;
  const size_t npair = (size_t)n * (n - 1) / 2;
  return 4 * (npair + 1) + 2 * (size_t)nG + (size_t)ceil_div(nG, kEwThreads) + 3 * (size_t)n;
}

void launch_ewald(const double *xp, int n, double L, double rs, double kappa, int gmax, double *work,
                  double *energy, double *grad, cudaStream_t st) {
  HQ_STAGE(ST_EWALD, st);
  const int npair = n * (n - 1) / 2;
  const long long side = 2LL * gmax + 1, nG = side * side * side;
  const int nblk = ceil_div(nG, kEwThreads);
  double *pe = work, *pg = pe + (npair + 1), *Sd = pg + 3 * ((size_t)npair + 1);
  double *part = Sd + 2 * nG, *gr = part + nblk;
  double2 *S = reinterpret_cast<double2 *>(Sd);  // 16-byte aligned: 4 (npair + 1) doubles before it
  k_ewald_sf<<<nblk, kEwThreads, 0, st>>>(xp, n, L, kappa, gmax, S, part);
  HQ_LAUNCH_CHECK();
  if (grad) {
    k_ewald_recip_grad<<<n, kEwThreads, 0, st>>>(xp, n, L, kappa, gmax, S, gr);
    HQ_LAUNCH_CHECK();
  }
  if (npair > 0) {
    k_ewald_real<<<ceil_div(npair, 128), 128, 0, st>>>(xp, n, L, kappa, pe, pg);
    HQ_LAUNCH_CHECK();
  }
  k_ewald_finish<<<1, 256, 0, st>>>(pe, pg, part, nblk, gr, n, L, rs, kappa, gmax, energy, grad);
  HQ_LAUNCH_CHECK();
}

}  // namespace hqcgb
