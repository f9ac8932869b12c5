// Real-space grid kernels of the FP64 path.
//
//  * gto1d: lattice-summed 1D Gaussian-power factors and their first two
//    derivatives (hqc/pbc/gto.py:326-339, evaluated on Rmesh_1d as in
//    hqc/pbc/solver.py:212-214);
//  * phi: AO values (and gradients) on the grid, the separable product of
//    those factors contracted over primitives (hqc/pbc/gto.py:341-369);
//  * density: rho(g) = sum_p phi_p(g) (D phi)_p(g)  (hqc/pbc/solver.py:690),
//    plus grad rho for GGA;
//  * pointwise xc / energy kernels.
//
// Layouts: grid index g = (ix * n + iy) * n + iz with x_i = i L / n; AO-major
// arrays [p][g]; factor table F[A][d][i][a][s], s = 3*l + k with k = 0 value,
// 1 first, 2 second derivative of u^l exp(-alpha u^2).
#include "common.cuh"
#include "xc.cuh"
#include "kernels.h"

namespace hqcgb {

__global__ void k_gto1d(const double *__restrict__ xp, int n_atoms, int ng, double L,
                        const double *__restrict__ alpha, int nprim,
                        const double *__restrict__ lat1d, int nlat, double *__restrict__ F) {
  long long idx = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  long long total = (long long)n_atoms * 3 * ng * nprim;
  if (idx >= total) return;
  int a = idx % nprim;
  long long r = idx / nprim;
  int i = r % ng;
  r /= ng;
  int d = r % 3;
  int A = (int)(r / 3);
  double x = i * L / ng - xp[A * 3 + d];
  double al = alpha[a];
  double s[6] = {0, 0, 0, 0, 0, 0};
  for (int t = 0; t < nlat; ++t) {
    double u = x - lat1d[t];
    double e = exp(-al * u * u);
    // l = 0: value, d/dx, d2/dx2
    s[0] += e;
    s[1] += -2.0 * al * u * e;
    s[2] += (4.0 * al * al * u * u - 2.0 * al) * e;
    // l = 1
    s[3] += u * e;
    s[4] += (1.0 - 2.0 * al * u * u) * e;
    s[5] += (4.0 * al * al * u * u * u - 6.0 * al * u) * e;
  }
  double *out = F + idx * 6;
#pragma unroll
  for (int k = 0; k < 6; ++k) out[k] = s[k];
}

void launch_gto1d(const double *xp, int n_atoms, int ng, double L, const double *alpha, int nprim,
                  const double *lat1d, int nlat, double *F, cudaStream_t st) {
  HQ_STAGE(ST_GTO, st);
  long long total = (long long)n_atoms * 3 * ng * nprim;
  k_gto1d<<<ceil_div(total, 256), 256, 0, st>>>(xp, n_atoms, ng, L, alpha, nprim, lat1d, nlat, F);
  HQ_LAUNCH_CHECK();
}

// AO value (deriv_dir < 0) or its derivative along deriv_dir (0..2), or the
// second derivative d_c d_e (hess >= 0: pair index xx yy zz xy xz yz).
__device__ inline double ao_eval(const double *__restrict__ F, const double *__restrict__ coef,
                                 int nprim, int ng, int A, int l, int cart, int ix, int iy, int iz,
                                 int c1, int c2) {
  int pw[3] = {0, 0, 0};
  if (l == 1) pw[cart] = 1;
  int kd[3] = {0, 0, 0};
  if (c1 >= 0) kd[c1] += 1;
  if (c2 >= 0) kd[c2] += 1;
  const double *fx = F + ((((long long)A * 3 + 0) * ng + ix) * nprim) * 6 + 3 * pw[0] + kd[0];
  const double *fy = F + ((((long long)A * 3 + 1) * ng + iy) * nprim) * 6 + 3 * pw[1] + kd[1];
  const double *fz = F + ((((long long)A * 3 + 2) * ng + iz) * nprim) * 6 + 3 * pw[2] + kd[2];
  double v = 0.0;
  for (int a = 0; a < nprim; ++a) v += coef[a] * fx[a * 6] * fy[a * 6] * fz[a * 6];
  return v;
}

__global__ void k_phi(const double *__restrict__ F, const double *__restrict__ coef,
                      const int *__restrict__ ao_l, const int *__restrict__ ao_cart, int nao_atom,
                      int nprim, int nao, int ng, double *__restrict__ phi,
                      double *__restrict__ dphi) {
  long long N = (long long)ng * ng * ng;
  long long idx = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (idx >= (long long)nao * N) return;
  int p = (int)(idx / N);
  long long g = idx - (long long)p * N;
  int iz = g % ng, iy = (g / ng) % ng, ix = (int)(g / ((long long)ng * ng));
  int A = p / nao_atom, k = p % nao_atom;
  const double *c = coef + k * nprim;
  phi[idx] = ao_eval(F, c, nprim, ng, A, ao_l[k], ao_cart[k], ix, iy, iz, -1, -1);
  if (dphi) {
    for (int d = 0; d < 3; ++d)
      dphi[(long long)d * nao * N + idx] =
          ao_eval(F, c, nprim, ng, A, ao_l[k], ao_cart[k], ix, iy, iz, d, -1);
  }
}

void launch_phi(const double *F, const double *coef, const int *ao_l, const int *ao_cart,
                int nao_atom, int nprim, int nao, int ng, double *phi, double *dphi,
                cudaStream_t st) {
  HQ_STAGE(ST_PHI, st);
  long long total = (long long)nao * ng * ng * ng;
  k_phi<<<ceil_div(total, 256), 256, 0, st>>>(F, coef, ao_l, ao_cart, nao_atom, nprim, nao, ng, phi,
                                               dphi);
  HQ_LAUNCH_CHECK();
}

// rho(g) = sum_p phi_p X_p, X = D phi; grad rho = 2 sum_p dphi_p X_p.
// One block: 32 grid points, 8 warps; phi tile of all AOs in shared memory.
__global__ void k_density(const double *__restrict__ phi, const double *__restrict__ dphi,
                          const double *__restrict__ D, int nao, long long N,
                          double *__restrict__ rho, double *__restrict__ grho,
                          double *__restrict__ Xout) {
  extern __shared__ double sh[];  // [nao][32] + reduction [8][4][32]
  double *tile = sh;
  double *red = sh + (size_t)nao * 32;
  int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  long long g0 = (long long)blockIdx.x * 32;
  long long g = g0 + lane;
  bool ok = g < N;
  for (int p = w; p < nao; p += 8) tile[p * 32 + lane] = ok ? phi[(long long)p * N + g] : 0.0;
  __syncthreads();
  double acc = 0, ga0 = 0, ga1 = 0, ga2 = 0;
  for (int p = w; p < nao; p += 8) {
    const double *Drow = D + (long long)p * nao;
    double x = 0;
    for (int q = 0; q < nao; ++q) x += Drow[q] * tile[q * 32 + lane];
    acc += tile[p * 32 + lane] * x;
    if (ok) {
      if (Xout) Xout[(long long)p * N + g] = x;
      if (grho) {
        ga0 += dphi[(long long)p * N + g] * x;
        ga1 += dphi[(long long)(nao + p) * N + g] * x;
        ga2 += dphi[(long long)(2 * nao + p) * N + g] * x;
      }
    }
  }
  red[(w * 4 + 0) * 32 + lane] = acc;
  red[(w * 4 + 1) * 32 + lane] = ga0;
  red[(w * 4 + 2) * 32 + lane] = ga1;
  red[(w * 4 + 3) * 32 + lane] = ga2;
  __syncthreads();
  if (w < 4 && ok) {
    double s = 0;
    for (int k = 0; k < 8; ++k) s += red[(k * 4 + w) * 32 + lane];
    if (w == 0) rho[g] = s;
    else if (grho) grho[(long long)(w - 1) * N + g] = 2.0 * s;
  }
}

void launch_density(const double *phi, const double *dphi, const double *D, int nao, long long N,
                    double *rho, double *grho, double *Xout, cudaStream_t st) {
  HQ_STAGE(ST_DENSITY, st);
  size_t smem = ((size_t)nao * 32 + 8 * 4 * 32) * sizeof(double);
  HQ_REQUIRE(smem <= 227 * 1024, "too many AOs for the FP64 density tile");
  ensure_dyn_smem((const void *)k_density, smem);
  k_density<<<ceil_div(N, 32), 256, smem, st>>>(phi, dphi, D, nao, N, rho, grho, Xout);
  HQ_LAUNCH_CHECK();
}

// ---------------------------------------------------------------------------
// S~ = dV phi phi^T of a mixed Hartree-Fock plan, in FP64: chunks of 2048 points
// in sequence, then the chunks in sequence.  8 x 8 tiles of the lower triangle, one
// output a thread: the FP64 pipe bounds it, and few AOs in larger tiles leave most
// SMs idle (28 AOs at 49^3: 664 us with 32 x 32 tiles, 163 with 8 x 8; the digit form
// of the FP64 plans takes 76, with operands and tables for this one sum a geometry).
// ---------------------------------------------------------------------------
constexpr int kGramChunk = 2048, kGramT = 8;

__global__ void __launch_bounds__(kGramT * kGramT) k_gram_part(const double *__restrict__ A, int nao, long long N,
                                                               double *__restrict__ P) {
  __shared__ double As[kGramT][33], Bs[kGramT][33];
  int pt = (int)((sqrtf(8.f * blockIdx.x + 1.f) - 1.f) * 0.5f);
  while (pt * (pt + 1) / 2 > (int)blockIdx.x) --pt;
  while ((pt + 1) * (pt + 2) / 2 <= (int)blockIdx.x) ++pt;
  const int p0 = pt * kGramT, q0 = ((int)blockIdx.x - pt * (pt + 1) / 2) * kGramT;
  const int tid = threadIdx.x, p = tid / kGramT, q = tid % kGramT, tx = tid & 31;
  const long long k0 = (long long)blockIdx.y * kGramChunk, k1 = min(k0 + kGramChunk, N);
  double acc = 0;
  for (long long kb = k0; kb < k1; kb += 32) {
    const long long k = kb + tx;
#pragma unroll
    for (int r = tid >> 5; r < kGramT; r += kGramT * kGramT / 32) {
      As[r][tx] = k < k1 && p0 + r < nao ? A[(long long)(p0 + r) * N + k] : 0.0;
      Bs[r][tx] = k < k1 && q0 + r < nao ? A[(long long)(q0 + r) * N + k] : 0.0;
    }
    __syncthreads();
#pragma unroll
    for (int kk = 0; kk < 32; ++kk) acc = fma(As[p][kk], Bs[q][kk], acc);
    __syncthreads();
  }
  if (p0 + p < nao && q0 + q < nao) P[((long long)blockIdx.y * nao + p0 + p) * nao + q0 + q] = acc;
}

__global__ void k_gram_sum(const double *__restrict__ P, int nchunk, int nao, double scale, double *__restrict__ M) {
  const int idx = blockIdx.x * blockDim.x + threadIdx.x;
  if (idx >= nao * nao) return;
  const int i = idx / nao, j = idx % nao, p = max(i, j), q = min(i, j);
  double s = 0;
#pragma unroll 8
  for (int c = 0; c < nchunk; ++c) s += P[((long long)c * nao + p) * nao + q];
  M[idx] = scale * s;
}

size_t gram_scratch_doubles(int nao, long long N) { return (size_t)ceil_div(N, kGramChunk) * nao * nao; }

void launch_gram(const double *A, int nao, long long N, double scale, double *P, double *M, cudaStream_t st) {
  HQ_STAGE(ST_QUAD, st);
  const int nt = ceil_div(nao, kGramT), nchunk = ceil_div(N, kGramChunk);
  k_gram_part<<<dim3(nt * (nt + 1) / 2, nchunk), kGramT * kGramT, 0, st>>>(A, nao, N, P);
  HQ_LAUNCH_CHECK();
  k_gram_sum<<<ceil_div(nao * nao, 256), 256, 0, st>>>(P, nchunk, nao, scale, M);
  HQ_LAUNCH_CHECK();
}

// ---------------------------------------------------------------------------
// pointwise: exchange-correlation on the grid.
//   in : rho, grho (GGA), vh (Hartree potential)
//   out: w = dV (vh + v_rho) (quadrature weight), u = 2 v_sigma grad rho (GGA)
//   partial sums per block: [0] sum e_xc, [1] sum vh*rho
// F32 (mixed path): the functional and its derivatives are evaluated in FP32
// where rho > 1e-6 (FP64 below, where FP32 would lose range); per-point
// rounding of about 1e-7 averages out in the FP64 sums.
// ---------------------------------------------------------------------------
template <bool F32>
__global__ void k_xc_pointwise(int kind, const double *__restrict__ rho,
                               const double *__restrict__ grho, const double *__restrict__ vh,
                               long long N, double dV, double *__restrict__ w,
                               double *__restrict__ vxc_out, double *__restrict__ u,
                               double *__restrict__ part) {
  __shared__ double sh[32];
  long long g = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  double exc = 0, eh = 0;
  if (g < N) {
    double r = rho[g];
    double sig = 0, gx = 0, gy = 0, gz = 0;
    if (grho) {
      gx = grho[g]; gy = grho[N + g]; gz = grho[2 * N + g];
      sig = gx * gx + gy * gy + gz * gz;
    }
    double e = 0, vr = 0, vs = 0;
    if (kind >= 0) {
      if (F32 && r > 1e-6) {
        float ef, vrf, vsf;
        xc_point<float>(kind, (float)r, (float)sig, ef, vrf, vsf);
        e = ef;
        vr = vrf;
        vs = vsf;
      } else {
        xc_point<double>(kind, r, sig, e, vr, vs);
      }
    }
    double v = vh ? vh[g] : 0.0;
    if (w) w[g] = dV * (v + vr);
    if (vxc_out) vxc_out[g] = vr;
    if (u) {
      u[g] = 2.0 * vs * gx;
      u[N + g] = 2.0 * vs * gy;
      u[2 * N + g] = 2.0 * vs * gz;
    }
    exc = e;
    eh = v * r;
  }
  double s0 = block_sum(exc, sh);
  double s1 = block_sum(eh, sh);
  if (threadIdx.x == 0) {
    part[2 * blockIdx.x] = s0;
    part[2 * blockIdx.x + 1] = s1;
  }
}

int xc_blocks(long long N) { return ceil_div(N, 256); }

void launch_xc_pointwise(int kind, const double *rho, const double *grho, const double *vh,
                         long long N, double dV, double *w, double *vxc_out, double *u,
                         double *part, cudaStream_t st, bool fp32) {
  HQ_STAGE(ST_XC, st);
  if (fp32)
    k_xc_pointwise<true><<<xc_blocks(N), 256, 0, st>>>(kind, rho, grho, vh, N, dV, w, vxc_out, u, part);
  else
    k_xc_pointwise<false><<<xc_blocks(N), 256, 0, st>>>(kind, rho, grho, vh, N, dV, w, vxc_out, u, part);
  HQ_LAUNCH_CHECK();
}

// Generic sum over blocks of interleaved partial sums: out[j] = scale * sum_b part[b*stride+j].
__global__ void k_sum_partials(const double *__restrict__ part, int nblk, int stride, int nout,
                               double scale, double *__restrict__ out, int accumulate) {
  __shared__ double sh[32];
  for (int j = 0; j < nout; ++j) {
    double s = 0;
    for (int b = threadIdx.x; b < nblk; b += blockDim.x) s += part[(long long)b * stride + j];
    s = block_sum(s, sh);
    if (threadIdx.x == 0) out[j] = accumulate ? out[j] + scale * s : scale * s;
    __syncthreads();
  }
}

void launch_sum_partials(const double *part, int nblk, int stride, int nout, double scale,
                         double *out, bool accumulate, cudaStream_t st) {
  k_sum_partials<<<1, 256, 0, st>>>(part, nblk, stride, nout, scale, out, accumulate ? 1 : 0);
  HQ_LAUNCH_CHECK();
}

}  // namespace hqcgb
