// AO values at arbitrary points (electron positions), Gamma point: the
// reference's eval_pbc_ao (hqc/pbc/gto.py:326-369) -- per axis the 1D
// lattice sums  f_a^l(x) = sum_t (x - t L)^l exp(-alpha_a (x - t L)^2)  over
// t in [-tmax, tmax] (tmax = rcut // L), their product over the three axes
// and the contraction with the normalised coefficients (s: 1/sqrt(4 pi),
// p: sqrt(3 / (4 pi)) folded in).  Used by make_slater
// (hqc/pbc/slater.py:42-104) for walker batches.  FP64 throughout.  The
// k-point variant (eval_pbc_ao_kpt, gto.py:371-427) weights each lattice
// term with exp(i k_d t) and returns complex Bloch AO values.
#include <algorithm>
#include <cmath>
#include <vector>

#include "common.cuh"
#include "exp_table.cuh"
#include "zmath.cuh"
#include "kernels.h"

namespace hqcgb {

constexpr int kPtMaxPrim = 16;
constexpr int kPtMaxAo = 16;   // AOs per atom and 1D images of k_ao_cell
constexpr int kPtMaxLat = 65;

__device__ inline double2 zmul(double a, double2 b) { return make_double2(a * b.x, a * b.y); }
__device__ inline double zmul(double a, double b) { return a * b; }
__device__ inline void zfma(double w, double p, double &s) { s = fma(w, p, s); }
__device__ inline void zfma(double w, double2 p, double2 &s) {
  s.x = fma(w, p.x, s.x);
  s.y = fma(w, p.y, s.y);
}
template <typename Z> __device__ inline Z zzero();
template <> __device__ inline double zzero<double>() { return 0.0; }
template <> __device__ inline double2 zzero<double2>() { return make_double2(0.0, 0.0); }

// AO values, one thread per (point, atom), for the images lat[t] = (t - tm) a
// of a periodic box, t = 0..2 tm (Z = double2: image t weighted with phase
// ph[d][t]).  Relative to the image nearest along each axis, u = x - t0 a,
// image t0 + m contributes exp(-alpha m a (m a -+ 2 |u|)) <= 1, and the three
// nearest ones share one exponential:
//   f_x f_y f_z = exp(-alpha |u|^2) prod_d sum_m w_m,d  (l = 1: (u - m a) w).
// A nearest image scaled to 1 rounds at the worst place of the mantissa, so the other
// images are summed without it, and alpha |u|^2 is not rounded: error of the values
// against extended precision, H8 dzv / H14 dzvp / H32 szv, the plain image sums 1.8e-16 /
// 2.2e-16 / 1.7e-16, without either 2.5e-16 / 2.7e-16 / 2.0e-16, so 1.4e-16 / 2.1e-16 /
// 1.65e-16.  At a k-point 1.9e-16 / 2.2e-16 / 1.8e-16 the sums, 1.6e-16 / 2.1e-16 /
// 1.8e-16 here.
// Factors below e^-41 (1.6e-18 of the nearest image's term) are left out;
// their exponents are tested in FP32.  For sharp primitives no other image
// counts, so a point and atom take about 25 exponentials of 11 FP64
// instructions (exp_table.cuh) where the image sums of all axes and primitives
// take 105 of 30; the kernel is bound by the FP64 pipe.  Measured with 54
// atoms, dzvp, box 8 Bohr: AO values of 2048 walkers 25.4 -> 9.0 ms, of one
// walker 238 -> 167 us a call.
template <int NB, typename Z>
__global__ void __launch_bounds__(128)
    k_ao_cell(int n_atoms, int nb, int nprim, int tm, double a, const double *__restrict__ tables,
              const int *__restrict__ ao_l, const int *__restrict__ ao_cart, const double *__restrict__ xp,
              long long npts, int pts_per_group, const double *__restrict__ xe, Z *__restrict__ out) {
  constexpr bool kPhase = sizeof(Z) > sizeof(double);
  __shared__ double s_exp[kExpTable], s_alpha[kPtMaxPrim], s_ac[kPtMaxPrim], s_coef[NB * kPtMaxPrim];
  __shared__ double2 s_ph[kPhase ? 3 * kPtMaxLat : 1];
  __shared__ int s_type[NB];  // 0: s, 1 + axis: p
  const int nlat = 2 * tm + 1;
  for (int k = threadIdx.x; k < kExpTable; k += blockDim.x) s_exp[k] = tables[k];
  for (int k = threadIdx.x; k < nprim; k += blockDim.x) {
    s_alpha[k] = tables[kExpTable + k];
    s_ac[k] = s_alpha[k] * kExpInv;
  }
  for (int k = threadIdx.x; k < nb * nprim; k += blockDim.x) s_coef[k] = tables[kExpTable + nprim + k];
  if (kPhase)
    for (int k = threadIdx.x; k < 3 * nlat; k += blockDim.x) {
      const double *p = tables + kExpTable + nprim + nb * nprim + 2 * k;
      s_ph[k] = make_double2(p[0], p[1]);
    }
  for (int k = threadIdx.x; k < nb; k += blockDim.x) s_type[k] = ao_l[k] == 1 ? 1 + ao_cart[k] : 0;
  __syncthreads();
  const long long idx = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (idx >= npts * n_atoms) return;
  long long pt, grp;
  if (npts * n_atoms < (1LL << 32)) {  // 32-bit divisions
    pt = (unsigned)idx / (unsigned)n_atoms;
    grp = (unsigned)pt / (unsigned)pts_per_group;
  } else {
    pt = idx / n_atoms;
    grp = pt / pts_per_group;
  }
  const int A = (int)(idx - pt * n_atoms);
  const double *xa = xp + (grp * n_atoms + A) * 3;
  const double *r = xe + pt * 3;
  const double inv_a = 1.0 / a;
  double u[3];
  float rel[3];  // 2 u / a
  int t0[3];
#pragma unroll
  for (int d = 0; d < 3; ++d) {
    const double x = r[d] - xa[d];
    const double t = fmin(fmax(rint(x * inv_a), -(double)tm), (double)tm);
    t0[d] = (int)t;
    u[d] = __dsub_rn(x, __dmul_rn(t, a));  // the image sums' x - lat[t]
    rel[d] = 2.f * (float)(u[d] * inv_a);
  }
  double r2, r2l = 0.0;  // |u|^2 and, for the complex values with their more roundings, what its sum left out
  if (kPhase) {
    const double p = __dmul_rn(u[0], u[0]), q = __dmul_rn(u[1], u[1]), w = __dmul_rn(u[2], u[2]);
    const double s = p + q, z = s - p, z2 = (r2 = s + w) - s;
    r2l = ((p - (s - z)) + (q - z)) + ((s - (r2 - z2)) + (w - z2)) + fma(u[0], u[0], -p) + fma(u[1], u[1], -q) +
          fma(u[2], u[2], -w);
  } else {
    r2 = u[0] * u[0] + u[1] * u[1] + u[2] * u[2];
  }
  Z v[NB];
#pragma unroll
  for (int j = 0; j < NB; ++j) v[j] = zzero<Z>();
  for (int q = 0; q < nprim; ++q) {
    const double al = s_alpha[q], ala = -al * a;
    const float alf = (float)ala * (float)a;
    Z S0[3], S1[3];  // S0 without the nearest image's term, the largest, which joins last
#pragma unroll
    for (int d = 0; d < 3; ++d) {
      auto phase = [&](int m) {
        if constexpr (kPhase) return s_ph[d * nlat + t0[d] + tm + m];
        else return 1.0;
      };
      S0[d] = zzero<Z>();
      S1[d] = zmul(u[d], phase(0));
#pragma unroll
      for (int side = -1; side <= 1; side += 2) {
        // image t0 + side m lies at u - side m a
        const int most = side > 0 ? tm - t0[d] : tm + t0[d];
        if (most < 1 || !(alf * (1.f - side * rel[d]) > -41.f)) continue;
        const double w1 = exp_neg(ala * (a - 2 * side * u[d]), s_exp);
        zfma(w1, phase(side), S0[d]);
        zfma(w1 * (u[d] - side * a), phase(side), S1[d]);
        for (int m = 2; m <= most; ++m) {
          if (!(alf * m * (m - side * rel[d]) > -41.f)) break;
          const double ma = m * a, w = exp_neg(-al * ma * (ma - 2 * side * u[d]), s_exp);
          zfma(w, phase(side * m), S0[d]);
          zfma(w * (u[d] - side * ma), phase(side * m), S1[d]);
        }
      }
    }
    double e = exp_neg_product(al, s_ac[q], r2, s_exp);
    if (kPhase && e > 0.0) e = fma(e, -al * r2l, e);  // not where |u|^2 is infinite
    Z P0, P1, P2, P3;
    if constexpr (kPhase) {
#pragma unroll
      for (int d = 0; d < 3; ++d) zfma(1.0, s_ph[d * nlat + t0[d] + tm], S0[d]);
      const Z yz = zmul(S0[1], S0[2]), ex = zmul(e, S0[0]);
      P0 = zmul(ex, yz), P1 = zmul(zmul(e, S1[0]), yz), P2 = zmul(ex, zmul(S1[1], S0[2])),
      P3 = zmul(ex, zmul(S0[1], S1[2]));
    } else {  // v (1 + S0) in one rounding
      const Z ex = fma(e, S0[0], e), xy = fma(ex, S0[1], ex), px = e * S1[0], pxy = fma(px, S0[1], px), py = ex * S1[1];
      P0 = fma(xy, S0[2], xy), P1 = fma(pxy, S0[2], pxy), P2 = fma(py, S0[2], py), P3 = xy * S1[2];
    }
#pragma unroll
    for (int j = 0; j < NB; ++j) {
      if (j >= nb) break;
      const double c = s_coef[j * nprim + q];
      if (c == 0.0) continue;
      const int ty = s_type[j];
      zfma(c, ty == 0 ? P0 : ty == 1 ? P1 : ty == 2 ? P2 : P3, v[j]);
    }
  }
  const long long nao = (long long)n_atoms * nb;
#pragma unroll
  for (int j = 0; j < NB; ++j)
    if (j < nb) out[pt * nao + (long long)A * nb + j] = v[j];
}

// Whether lat[0..n) are the images (t - tm) a, t = 0..2 tm, of a box (host).
static bool box_images(int n, const double *lat, int *tm, double *a) {
  if (n % 2 == 0 || n > kPtMaxLat) return false;
  *tm = n / 2;
  *a = n > 1 ? lat[n / 2 + 1] : 1.0;
  if (!(*a > 0)) return false;
  for (int t = 0; t < n; ++t)
    if (!(std::fabs(lat[t] - (t - *tm) * *a) <= 4e-16 * std::fabs(lat[t]))) return false;
  return true;
}

// Any image list or basis size: one thread per (point, atom): out[pt][A * nb + j].
__global__ void k_ao_points(int n_atoms, int nb, int nprim, const double *__restrict__ alpha,
                            const double *__restrict__ coef, const int *__restrict__ ao_l,
                            const int *__restrict__ ao_cart, int nlat, const double *__restrict__ lat,
                            const double *__restrict__ xp, long long npts, int pts_per_group,
                            const double *__restrict__ xe, double *__restrict__ out) {
  const long long idx = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (idx >= npts * n_atoms) return;
  const int A = (int)(idx % n_atoms);
  const long long pt = idx / n_atoms;
  const long long grp = pt / pts_per_group;
  const double *xa = xp + (grp * n_atoms + A) * 3;
  const double *r = xe + pt * 3;
  // 1D factors f[d][a][l], l = 0, 1
  double f[3][kPtMaxPrim][2];
  for (int d = 0; d < 3; ++d) {
    const double x = r[d] - xa[d];
    for (int a = 0; a < nprim; ++a) {
      double s0 = 0, s1 = 0;
      for (int t = 0; t < nlat; ++t) {
        const double u = x - lat[t];
        const double g = exp(-alpha[a] * u * u);
        s0 += g;
        s1 += u * g;
      }
      f[d][a][0] = s0;
      f[d][a][1] = s1;
    }
  }
  const long long nao = (long long)n_atoms * nb;
  for (int j = 0; j < nb; ++j) {
    const int l = ao_l[j], ca = ao_cart[j];
    const int px = (l == 1 && ca == 0), py = (l == 1 && ca == 1), pz = (l == 1 && ca == 2);
    double v = 0;
    for (int a = 0; a < nprim; ++a)
      v += coef[j * nprim + a] * f[0][a][px] * f[1][a][py] * f[2][a][pz];
    out[pt * nao + (long long)A * nb + j] = v;
  }
}


// k-point AO values (complex): one thread per (point, atom), out[pt][A * nb + j].
__global__ void k_ao_points_kpt(int n_atoms, int nb, int nprim, const double *__restrict__ alpha,
                                const double *__restrict__ coef, const int *__restrict__ ao_l,
                                const int *__restrict__ ao_cart, int nlat,
                                const double *__restrict__ lat, double k0, double k1, double k2,
                                const double *__restrict__ xp, long long npts, int pts_per_group,
                                const double *__restrict__ xe, double2 *__restrict__ out) {
  const long long idx = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (idx >= npts * n_atoms) return;
  const int A = (int)(idx % n_atoms);
  const long long pt = idx / n_atoms;
  const long long grp = pt / pts_per_group;
  const double *xa = xp + (grp * n_atoms + A) * 3;
  const double *r = xe + pt * 3;
  const double kk[3] = {k0, k1, k2};
  double2 f[3][kPtMaxPrim][2];
  for (int d = 0; d < 3; ++d) {
    const double x = r[d] - xa[d];
    for (int a = 0; a < nprim; ++a) f[d][a][0] = f[d][a][1] = make_double2(0.0, 0.0);
    for (int t = 0; t < nlat; ++t) {
      const double u = x - lat[t];
      double sn, cs;
      sincos(kk[d] * lat[t], &sn, &cs);
      for (int a = 0; a < nprim; ++a) {
        const double g = exp(-alpha[a] * u * u);
        f[d][a][0].x += g * cs;
        f[d][a][0].y += g * sn;
        f[d][a][1].x += u * g * cs;
        f[d][a][1].y += u * g * sn;
      }
    }
  }
  const long long nao = (long long)n_atoms * nb;
  for (int j = 0; j < nb; ++j) {
    const int l = ao_l[j], ca = ao_cart[j];
    const int px = (l == 1 && ca == 0), py = (l == 1 && ca == 1), pz = (l == 1 && ca == 2);
    double2 v = make_double2(0.0, 0.0);
    for (int a = 0; a < nprim; ++a) {
      const double2 t = zmul(zmul(f[0][a][px], f[1][a][py]), f[2][a][pz]);
      v.x += coef[j * nprim + a] * t.x;
      v.y += coef[j * nprim + a] * t.y;
    }
    out[pt * nao + (long long)A * nb + j] = v;
  }
}

// AO values at npts points; kpt NULL: real, else complex (interleaved).  The
// tables go to the device in one copy.  k_ao_cell where the images are those
// of a box and the basis fits its registers (every basis of the package up to
// 16 AOs an atom); the image sums otherwise.
static void ao_points(int n_atoms, int nb, int nprim, const double *alpha, const double *coef, const int *ao_l,
                      const int *ao_cart, int nlat, const double *lat, const double *kpt, const double *xp,
                      long long npts, int pts_per_group, const double *xe, double *out, cudaStream_t st) {
  int tm = 0;
  double a = 0;
  const bool cell = nb <= kPtMaxAo && box_images(nlat, lat, &tm, &a);
  const size_t nc = (size_t)nb * nprim;
  std::vector<double> h((cell ? kExpTable : 0) + nprim + nc + (cell ? (kpt ? 6 * nlat : 0) : nlat) + nb);
  double *w = h.data();
  if (cell) {
    exp_table(w);
    w += kExpTable;
  }
  w = std::copy(alpha, alpha + nprim, w);
  w = std::copy(coef, coef + nc, w);
  if (!cell) w = std::copy(lat, lat + nlat, w);
  else if (kpt)
    for (int d = 0; d < 3; ++d)
      for (int t = 0; t < nlat; ++t) {
        *w++ = std::cos(kpt[d] * lat[t]);
        *w++ = std::sin(kpt[d] * lat[t]);
      }
  int *hl = reinterpret_cast<int *>(w);  // 2 nb ints in the last nb doubles
  std::copy(ao_l, ao_l + nb, hl);
  std::copy(ao_cart, ao_cart + nb, hl + nb);
  StreamBuf blk(h.size() * sizeof(double), st);
  double *d = blk.as<double>();
  const int *dl = reinterpret_cast<const int *>(d + (h.size() - nb));
  HQ_CUDA(cudaMemcpyAsync(d, h.data(), h.size() * sizeof(double), cudaMemcpyHostToDevice, st));
  const int grid = ceil_div(npts * n_atoms, 128);
  if (cell) {
    auto go = [&](auto kernel, auto *o) {
      kernel<<<grid, 128, 0, st>>>(n_atoms, nb, nprim, tm, a, d, dl, dl + nb, xp, npts, pts_per_group, xe, o);
    };
    double2 *z = reinterpret_cast<double2 *>(out);
    if (kpt) {
      if (nb <= 1) go(k_ao_cell<1, double2>, z);
      else if (nb <= 2) go(k_ao_cell<2, double2>, z);
      else if (nb <= 5) go(k_ao_cell<5, double2>, z);
      else go(k_ao_cell<kPtMaxAo, double2>, z);
    } else {
      if (nb <= 1) go(k_ao_cell<1, double>, out);
      else if (nb <= 2) go(k_ao_cell<2, double>, out);
      else if (nb <= 5) go(k_ao_cell<5, double>, out);
      else go(k_ao_cell<kPtMaxAo, double>, out);
    }
  } else if (kpt) {
    k_ao_points_kpt<<<grid, 128, 0, st>>>(n_atoms, nb, nprim, d, d + nprim, dl, dl + nb, nlat, d + nprim + nc, kpt[0],
                                          kpt[1], kpt[2], xp, npts, pts_per_group, xe,
                                          reinterpret_cast<double2 *>(out));
  } else {
    k_ao_points<<<grid, 128, 0, st>>>(n_atoms, nb, nprim, d, d + nprim, dl, dl + nb, nlat, d + nprim + nc, xp, npts,
                                      pts_per_group, xe, out);
  }
  HQ_LAUNCH_CHECK();
  // before the tables are freed: memory freed ahead of a synchronisation goes
  // back to the system there, and allocating it again costs 90 us a call
  HQ_CUDA(cudaStreamSynchronize(st));
}

}  // namespace hqcgb

// C ABI: AO values of n_atoms protons at npts points.  Basis tables as in
// the plan parameters (host pointers); xp [ngroups][n_atoms][3] and xe [npts][3]
// (device, Bohr), points grouped by pts_per_group per proton set; out
// [npts][n_atoms * nao_atom] (device).
extern "C" int hqcgb_ao_points(int n_atoms, int nao_atom, int n_prim, const double *alpha,
                               const double *coef, const int *ao_l, const int *ao_cart, int n_lat1d,
                               const double *lat1d, const double *xp, long long npts,
                               int pts_per_group, const double *xe, double *out, void *stream) {
  using namespace hqcgb;
  cudaStream_t st = (cudaStream_t)stream;
  try {
    HQ_REQUIRE(n_atoms >= 1 && nao_atom >= 1 && n_prim >= 1 && n_prim <= kPtMaxPrim && n_lat1d >= 1 &&
                   npts >= 0 && pts_per_group >= 1 && alpha && coef && ao_l && ao_cart && lat1d &&
                   xp && xe && out,
               "bad argument");
    for (int k = 0; k < nao_atom; ++k)
      HQ_REQUIRE((ao_l[k] == 0 || ao_l[k] == 1) && ao_cart[k] >= 0 && ao_cart[k] < 3,
                 "only s and p AOs are supported");
    if (npts == 0) return HQCGB_OK;
    ao_points(n_atoms, nao_atom, n_prim, alpha, coef, ao_l, ao_cart, n_lat1d, lat1d, nullptr, xp, npts, pts_per_group,
              xe, out, st);
    return HQCGB_OK;
  } catch (const Error &e) {
    set_error(e.msg);
    return e.status;
  } catch (const std::exception &e) {  // host memory
    set_error(e.what());
    return HQCGB_CUDA_ERROR;
  }
}

namespace hqcgb {
// M[p][k] = mo[p][idx[k]] for k < m (the Slater columns)
__global__ void k_gather_cols(const double *__restrict__ mo, int nao, int nmo,
                              const int *__restrict__ idx, int m, double *__restrict__ M) {
  int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= nao * m) return;
  int p = i / m, k = i % m;
  M[i] = mo[(long long)p * nmo + idx[k]];
}
}  // namespace hqcgb

// C ABI: Slater matrices of W walkers (hqc/pbc/slater.py:42-70): up[w] =
// AO(xe[w][0:n/2]) mo[:, idx[0:n/2]], dn[w] = AO(xe[w][n/2:n]) mo[:, idx[n/2:n]].
// xp [xp_groups][n][3] with xp_groups 1 (shared protons) or W; xe [W][n][3]
// (device, Bohr); mo [nao][nmo] row-major (device); state_idx [n] (host);
// up, dn [W][n/2][n/2] (device).
extern "C" int hqcgb_slater(int n, int nao_atom, int n_prim, const double *alpha,
                            const double *coef, const int *ao_l, const int *ao_cart, int n_lat1d,
                            const double *lat1d, int W, int xp_groups, const double *xp,
                            const double *xe, const double *mo, int nmo, const int *state_idx,
                            double *up, double *dn, void *stream) {
  using namespace hqcgb;
  cudaStream_t st = (cudaStream_t)stream;
  try {
    HQ_REQUIRE(n >= 2 && n % 2 == 0 && W >= 1 && (xp_groups == 1 || xp_groups == W) && mo && up &&
                   dn && state_idx,
               "bad argument");
    const int n2 = n / 2, nao = n * nao_atom;
    for (int k = 0; k < n; ++k)
      HQ_REQUIRE(state_idx[k] >= 0 && state_idx[k] < nmo, "state index out of range");
    StreamBuf ao_buf((size_t)W * n * nao * sizeof(double), st), mu_buf((size_t)2 * nao * n2 * sizeof(double), st),
        idx_buf((size_t)n * sizeof(int), st);
    double *ao = ao_buf.as<double>(), *Mu = mu_buf.as<double>();
    int *idx = idx_buf.as<int>();
    HQ_CUDA(cudaMemcpyAsync(idx, state_idx, n * sizeof(int), cudaMemcpyHostToDevice, st));
    // AO values: with shared protons every point is in group 0
    const int ppg = xp_groups == 1 ? W * n : n;
    int s = hqcgb_ao_points(n, nao_atom, n_prim, alpha, coef, ao_l, ao_cart, n_lat1d, lat1d, xp,
                            (long long)W * n, ppg, xe, ao, stream);
    if (s != HQCGB_OK) throw Error{s, hqcgb_last_error()};
    k_gather_cols<<<ceil_div(nao * n2, 256), 256, 0, st>>>(mo, nao, nmo, idx, n2, Mu);
    HQ_LAUNCH_CHECK();
    k_gather_cols<<<ceil_div(nao * n2, 256), 256, 0, st>>>(mo, nao, nmo, idx + n2, n2,
                                                           Mu + (size_t)nao * n2);
    HQ_LAUNCH_CHECK();
    gemm_batched_rowmajor(n2, n2, nao, ao, nao, (long long)n * nao, Mu, n2, 0, up, n2,
                          (long long)n2 * n2, W, st);
    gemm_batched_rowmajor(n2, n2, nao, ao + (size_t)n2 * nao, nao, (long long)n * nao,
                          Mu + (size_t)nao * n2, n2, 0, dn, n2, (long long)n2 * n2, W, st);
    HQ_CUDA(cudaStreamSynchronize(st));
    return HQCGB_OK;
  } catch (const Error &e) {
    set_error(e.msg);
    return e.status;
  } catch (const std::exception &e) {  // host memory
    set_error(e.what());
    return HQCGB_CUDA_ERROR;
  }
}

namespace hqcgb {

__global__ void k_gather_cols_z(const double2 *__restrict__ mo, int nao, int nmo,
                                const int *__restrict__ idx, int m, double2 *__restrict__ M) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= nao * m) return;
  const int p = i / m, k = i % m;
  M[i] = mo[(long long)p * nmo + idx[k]];
}

}  // namespace hqcgb

// C ABI: k-point AO values (complex, interleaved) of n_atoms protons at npts
// points; arguments as hqcgb_ao_points plus kpt [3] (1/Bohr, host).
extern "C" int hqcgb_ao_points_kpt(int n_atoms, int nao_atom, int n_prim, const double *alpha,
                                   const double *coef, const int *ao_l, const int *ao_cart,
                                   int n_lat1d, const double *lat1d, const double *kpt,
                                   const double *xp, long long npts, int pts_per_group,
                                   const double *xe, double *out, void *stream) {
  using namespace hqcgb;
  cudaStream_t st = (cudaStream_t)stream;
  try {
    HQ_REQUIRE(n_atoms >= 1 && nao_atom >= 1 && n_prim >= 1 && n_prim <= kPtMaxPrim && n_lat1d >= 1 &&
                   npts >= 0 && pts_per_group >= 1 && alpha && coef && ao_l && ao_cart && lat1d &&
                   kpt && xp && xe && out,
               "bad argument");
    for (int k = 0; k < nao_atom; ++k)
      HQ_REQUIRE((ao_l[k] == 0 || ao_l[k] == 1) && ao_cart[k] >= 0 && ao_cart[k] < 3,
                 "only s and p AOs are supported");
    if (npts == 0) return HQCGB_OK;
    ao_points(n_atoms, nao_atom, n_prim, alpha, coef, ao_l, ao_cart, n_lat1d, lat1d, kpt, xp, npts, pts_per_group, xe,
              out, st);
    return HQCGB_OK;
  } catch (const Error &e) {
    set_error(e.msg);
    return e.status;
  } catch (const std::exception &e) {  // host memory
    set_error(e.what());
    return HQCGB_CUDA_ERROR;
  }
}

// C ABI: k-point Slater matrices (hqc/pbc/slater.py:72-93): as hqcgb_slater
// with kpt [3] (host), complex mo [nao][nmo] and complex up, dn [W][n/2][n/2]
// (interleaved re, im).
extern "C" int hqcgb_slater_kpt(int n, int nao_atom, int n_prim, const double *alpha,
                                const double *coef, const int *ao_l, const int *ao_cart, int n_lat1d,
                                const double *lat1d, const double *kpt, int W, int xp_groups,
                                const double *xp, const double *xe, const double *mo, int nmo,
                                const int *state_idx, double *up, double *dn, void *stream) {
  using namespace hqcgb;
  cudaStream_t st = (cudaStream_t)stream;
  try {
    HQ_REQUIRE(n >= 2 && n % 2 == 0 && W >= 1 && (xp_groups == 1 || xp_groups == W) && mo && up &&
                   dn && state_idx && kpt,
               "bad argument");
    const int n2 = n / 2, nao = n * nao_atom;
    for (int k = 0; k < n; ++k)
      HQ_REQUIRE(state_idx[k] >= 0 && state_idx[k] < nmo, "state index out of range");
    StreamBuf ao_buf((size_t)W * n * nao * sizeof(double2), st),
        mu_buf((size_t)2 * nao * n2 * sizeof(double2), st), idx_buf((size_t)n * sizeof(int), st);
    double2 *ao = ao_buf.as<double2>(), *Mu = mu_buf.as<double2>();
    int *idx = idx_buf.as<int>();
    HQ_CUDA(cudaMemcpyAsync(idx, state_idx, n * sizeof(int), cudaMemcpyHostToDevice, st));
    const int ppg = xp_groups == 1 ? W * n : n;
    int s = hqcgb_ao_points_kpt(n, nao_atom, n_prim, alpha, coef, ao_l, ao_cart, n_lat1d, lat1d, kpt,
                                xp, (long long)W * n, ppg, xe, reinterpret_cast<double *>(ao), stream);
    if (s != HQCGB_OK) throw Error{s, hqcgb_last_error()};
    const double2 *moz = reinterpret_cast<const double2 *>(mo);
    k_gather_cols_z<<<ceil_div(nao * n2, 256), 256, 0, st>>>(moz, nao, nmo, idx, n2, Mu);
    HQ_LAUNCH_CHECK();
    k_gather_cols_z<<<ceil_div(nao * n2, 256), 256, 0, st>>>(moz, nao, nmo, idx + n2, n2,
                                                             Mu + (size_t)nao * n2);
    HQ_LAUNCH_CHECK();
    zgemm_batched_rowmajor(n2, n2, nao, ao, nao, (long long)n * nao, Mu, n2, 0,
                           reinterpret_cast<double2 *>(up), n2, (long long)n2 * n2, W, st);
    zgemm_batched_rowmajor(n2, n2, nao, ao + (size_t)n2 * nao, nao, (long long)n * nao,
                           Mu + (size_t)nao * n2, n2, 0, reinterpret_cast<double2 *>(dn), n2,
                           (long long)n2 * n2, W, st);
    HQ_CUDA(cudaStreamSynchronize(st));
    return HQCGB_OK;
  } catch (const Error &e) {
    set_error(e.msg);
    return e.status;
  } catch (const std::exception &e) {  // host memory
    set_error(e.what());
    return HQCGB_CUDA_ERROR;
  }
}
