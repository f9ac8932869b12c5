// Exact exchange of the Gamma-point Hartree-Fock Fock build and of its
// nuclear gradient, in the occupied-pair form with fused FFT stages.
//
// The reference builds the full ERI tensor (pr|sq) = sum_G V(G) rho_pr(G)
// rho_sq(G)* from AO pair densities in G space (hqc/pbc/solver.py:391-433) and
// contracts it with the density matrix (solver.py:604-614, 748-751):
//   K_pq = sum_rs D_rs (pr|sq),   V(G) = 4 pi / (Omega G^2), G = 0 dropped.
// With D = sum_j f_j c_j c_j^T this is, on the same odd grid and by Parseval,
//   K_pq = sum_j sum_G w(G) Re[ conj(P^_pj(G)) P^_qj(G) ],
//   P_pj(r) = phi_p(r) psi~_j(r),  psi~_j = sqrt(f_j) sum_p c_pj phi_p,
//   w(G) = dV * 4 pi / (G^2 N),  P^ = the (unnormalised) 3D DFT of P,
// (the occupied-pair-density exchange the reference sketches as exchange_rhoG,
// solver.py:631-666).  P is real, so only the half spectrum kz = 0..(n-1)/2
// is formed and the kz > 0 terms count twice.  Three stages per pair:
//
//   k_exx_plane   one x-plane of one pair: phi_p recomputed from the
//                 separable 1D GTO factors (no AO grid is read), the pair
//                 formed in shared memory, a real DFT along z (half
//                 spectrum; two real lines per complex transform) and a
//                 complex DFT along y;
//   k_exx_column  one ky-line of one pair: the DFT along x, then the
//                 frequency-stage multiply by sqrt(w(G) (1 or 2)); the store
//                 stage writes Q = sqrt(.) P^ as FP64, or as the TF32 hi/lo
//                 pieces the tensor-core Gram kernel reads (mixed path) --
//   K = Q Q^T     one symmetric Gram matrix over all pairs of a group of
//                 orbitals (tcgen05 3xTF32 on the mixed path, FP64 otherwise).
//
// Nuclear gradient (absent in the reference, doc/solver_algorithm.md:1210):
// the exchange part of dE/dR_A,c is
//   dV sum_{p in A} sum_j sum_g d_c phi_p(g) psi~_j(g) [v * (X_p psi~_j)](g),
// X = D phi, v the Coulomb kernel; by Parseval that is
//   sum_j sum_G w(G) Re[ conj(FFT(d_c phi_p psi~_j)) FFT(X_p psi~_j) ],
// which the column kernel's dot mode contracts in its store stage (no Q is
// written): four rows per AO (X_p and the three derivatives, recomputed from
// the 1D factors), three dot products per (pair, ky-line).
//
// Data: grid index g = (ix * n + iy) * n + iz (z fastest); T[pair][x][ky][kz]
// the plane-transformed pairs, n * nh complex per plane, nh = (n + 1) / 2.
#include <algorithm>

#include "dft_shared.cuh"
#include "kernels.h"

namespace hqcgb {
namespace exx {

// dV * 4 pi / (G^2 N) (0 at G = 0), doubled for kz > 0 (the half spectrum
// stands for +G and -G).
__device__ inline double pair_weight(int kx, int ky, int kz, int n, double L, double dV) {
  const int mx = kx <= n / 2 ? kx : kx - n, my = ky <= n / 2 ? ky : ky - n;
  const double m2 = (double)mx * mx + (double)my * my + (double)kz * kz;
  if (m2 == 0.0) return 0.0;
  const double g = 2.0 * M_PI / L;
  const double N = (double)n * n * n;
  return dV * 4.0 * M_PI / (g * g * m2 * N) * (kz > 0 ? 2.0 : 1.0);
}

// wsq[kx][ky][kz] = sqrt(pair_weight), once per plan
template <typename R>
__global__ void k_pair_weights(int n, double L, double dV, R *__restrict__ wsq) {
  const int nh = (n + 1) / 2;
  const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= (long long)n * n * nh) return;
  const int kz = (int)(i % nh), ky = (int)((i / nh) % n), kx = (int)(i / ((long long)n * nh));
  wsq[i] = (R)sqrt(pair_weight(kx, ky, kz, n, L, dV));
}

struct PlaneArgs {
  int n, nh, n1, nao, nb, nprim;
  int rows;                  // pair rows per orbital: nao (Fock), 4 nao (gradient)
  int xrows;                 // rows [0, xrows) read their field from X; the rest from the 1D factors
  const double2 *tw;
  const void *F1d;           // 1D factor table [atom][axis][grid][prim][6] (R)
  const double *coef;        // [nb][nprim]
  const int *ao_l, *ao_cart; // [nb]
  const double *X;           // [nao][ldx] FP64 (gradient mode), or null
  long long ldx;
  const void *psi;           // psi~ of the group's first orbital, rows ldpsi apart (R)
  long long ldpsi;
  void *T;                   // [g][rows][n][n][nh] complex R
  int g, per;                // orbitals of the group, orbitals a block
};

// grid (n x-planes, rows, ceil(g / per)).  Several orbitals a block share the row's
// field: its primitives' products cost about as much as the transforms (28 rows,
// 10 orbitals at 49^3, FP32: 320 -> 212 us).
// CTAs of 256 threads per SM: FP32 four (64 registers; the gradient's columns three:
// 957 -> 500 us for 28 rows of 4 orbitals at 49^3, where one block an SM hid no
// latency), FP64 two (H8 szv at 41^3: 7.3 -> 6.65 ms a run)
template <typename R>
constexpr int exx_min_blocks() { return sizeof(R) == 4 ? 4 : 2; }

template <typename R>
__global__ void __launch_bounds__(256, exx_min_blocks<R>()) k_exx_plane(PlaneArgs a) {
  using R2 = typename C2<R>::T;
  extern __shared__ __align__(16) unsigned char smraw[];
  const int n = a.n, nh = a.nh, x = blockIdx.x, r = blockIdx.y;
  const int jl0 = blockIdx.z * a.per, jl1 = min(jl0 + a.per, a.g);
  const size_t bufc = (size_t)n * (n + 1) / 2 + 1;  // complex slots of one plane buffer (>= n^2 reals)
  R2 *w = reinterpret_cast<R2 *>(smraw);
  R2 *B0 = w + n;                  // plane buffers: the packed pair lines, the
  R2 *B1 = B0 + bufc;              // transforms' temporaries and the z-transformed plane
  R *fyz = reinterpret_cast<R *>(B1 + bufc);  // [2][nprim][n]: y and z factors
  load_twiddles(w, a.tw, n);
  const long long plane = (long long)x * n * n;
  const int nn = n * n;
  // The pair plane goes straight into the packed layout of the z transform:
  // complex column pr of Z[z][pr] holds the real y-lines 2 pr (real part) and
  // 2 pr + 1 (imaginary part); the last column of an odd n has no partner.
  const int npair = (n + 1) / 2;
  const int sy = (int)blockDim.x / n, sz = (int)blockDim.x - sy * n;  // a step of blockDim.x points
  const int yf = (int)threadIdx.x / n, zf = (int)threadIdx.x - yf * n;
  // each(f): f(i, y, z, slot of the packed layout) for the thread's points i = y n + z
  auto each = [&](auto f) {
    int y = yf, z = zf;
    for (int i = threadIdx.x; i < nn; i += blockDim.x) {
      f(i, y, z, 2 * (z * npair + (y >> 1)) + (y & 1));
      y += sy;
      z += sz;
      if (z >= n) {
        z -= n;
        ++y;
      }
    }
  };
  R fx[8];
  if (r >= a.xrows) {
    // Fock mode: row r is phi_p, p = r (c = -1: the value); gradient mode:
    // row nao (1 + c) + p is d_c phi_p
    const int rr = r - a.xrows;
    const int p = rr % a.nao, c = a.xrows > 0 ? rr / a.nao : -1;
    // AO p (or its derivative along c) = sum_a coef_a fx_a(x) fy_a(y) fz_a(z)
    const int A = p / a.nb, k = p % a.nb, l = a.ao_l[k], ca = a.ao_cart[k];
    int e[3];
    for (int d = 0; d < 3; ++d) e[d] = 3 * ((l == 1 && ca == d) ? 1 : 0) + (d == c ? 1 : 0);
    const R *F = reinterpret_cast<const R *>(a.F1d);
    for (int i = threadIdx.x; i < 2 * a.nprim * n; i += blockDim.x) {
      const int ax = i / (a.nprim * n), rem = i - ax * a.nprim * n, pr = rem / n, t = rem - pr * n;
      fyz[i] = F[((((long long)A * 3 + 1 + ax) * n + t) * a.nprim + pr) * 6 + e[1 + ax]];
    }
    for (int pr = 0; pr < a.nprim; ++pr)
      fx[pr] = (R)a.coef[k * a.nprim + pr] * F[((((long long)A * 3 + 0) * n + x) * a.nprim + pr) * 6 + e[0]];
    __syncthreads();
  }
  const double *Xr = a.X + (long long)r * a.ldx + plane;  // read where r < xrows
  auto field = [&](int i, int y, int z) {
    if (r < a.xrows) return (R)Xr[i];
    R v = 0;
    for (int pr = 0; pr < a.nprim; ++pr) v += fx[pr] * fyz[pr * n + y] * fyz[(a.nprim + pr) * n + z];
    return v;
  };
  R *ao = fyz + 2 * a.nprim * n;  // the row's field on the plane, packed (several orbitals a block)
  if (a.per > 1) each([&](int i, int y, int z, int slot) { ao[slot] = field(i, y, z); });
  for (int jl = jl0; jl < jl1; ++jl) {
    const R *psi = reinterpret_cast<const R *>(a.psi) + (long long)jl * a.ldpsi + plane;
    R *Zr = reinterpret_cast<R *>(B0);  // Z[z][pr] as reals: [z][pr][2]
    if (n & 1)
      for (int z = threadIdx.x; z < n; z += blockDim.x) Zr[2 * (z * npair + npair - 1) + 1] = 0;
    if (a.per > 1) each([&](int i, int, int, int slot) { Zr[slot] = ao[slot] * psi[i]; });
    else each([&](int i, int y, int z, int slot) { Zr[slot] = field(i, y, z) * psi[i]; });
    __syncthreads();
    // z transform of the packed lines, then unpacked into C[y][kz], kz < nh:
    // A[k] = (Z[k] + conj Z[n-k]) / 2 (line 2 pr), B[k] = (Z[k] - conj Z[n-k]) / 2i
    R2 *Zt = dft_axis0<R, R2>(B0, B1, n, npair, a.n1, w);
    R2 *Cb = (Zt == B0) ? B1 : B0;
    for (int i = threadIdx.x; i < npair * nh; i += blockDim.x) {
      const int pr = i / nh, kz = i - pr * nh;
      const R2 zk = Zt[kz * npair + pr], zm = Zt[(kz == 0 ? 0 : n - kz) * npair + pr];
      R2 u, v;
      u.x = (R)0.5 * (zk.x + zm.x);
      u.y = (R)0.5 * (zk.y - zm.y);
      v.x = (R)0.5 * (zk.y + zm.y);
      v.y = (R)0.5 * (zm.x - zk.x);
      Cb[(2 * pr) * nh + kz] = u;
      if (2 * pr + 1 < n) Cb[(2 * pr + 1) * nh + kz] = v;
    }
    __syncthreads();
    R2 *Ct = (Cb == B0) ? B1 : B0;
    const R2 *res = dft_axis0<R, R2>(Cb, Ct, n, nh, a.n1, w);
    R2 *T = reinterpret_cast<R2 *>(a.T) + (((long long)jl * a.rows + r) * n + x) * (long long)n * nh;
    for (int i = threadIdx.x; i < n * nh; i += blockDim.x) T[i] = res[i];
    if (jl + 1 < jl1) __syncthreads();  // the next pair overwrites res
  }
}

struct ColumnArgs {
  int n, nh, n1, nao, rows;
  const double2 *tw;
  const void *wsq;           // [n][n][nh] sqrt(pair_weight) (R)
  const void *T;             // [g][rows][n][n][nh] complex R
  // Fock mode: Q rows (one per AO), K index jl * 2 N_h + 2 ((kx n + ky) nh + kz) + {re, im}
  void *Q;                   // FP64 [rows][ldq], or the TF32 pieces [2][rows][ldq] (hi, then lo)
  long long ldq;
  // gradient mode: part[((jl * nao + p) * n + ky) * 3 + c]
  double *part;
};

__device__ inline uint32_t tf32_rna_x(float x) {
  uint32_t r;
  asm("cvt.rna.tf32.f32 %0, %1;" : "=r"(r) : "f"(x));
  return r;
}

// OUT 0: FP64 Q;  OUT 1: TF32 hi/lo Q;  OUT 2: gradient dot products.
// grid (n ky-lines, AOs (OUT 2) or rows, orbitals of the group)
template <typename R, int OUT>
__global__ void __launch_bounds__(256, OUT == 2 && sizeof(R) == 4 ? 3 : exx_min_blocks<R>()) k_exx_column(ColumnArgs a) {
  using R2 = typename C2<R>::T;
  extern __shared__ __align__(16) unsigned char smraw[];
  const int n = a.n, nh = a.nh, ky = blockIdx.x, r = blockIdx.y, jl = blockIdx.z;
  const size_t line = (size_t)n * nh;
  R2 *w = reinterpret_cast<R2 *>(smraw);
  R2 *B0 = w + n, *B1 = B0 + line, *B2 = B1 + line;
  load_twiddles(w, a.tw, n);
  const R2 *Tbase = reinterpret_cast<const R2 *>(a.T);
  const R *wsq = reinterpret_cast<const R *>(a.wsq) + (long long)ky * nh;  // + kx n nh + kz
  const long long plane = (long long)n * nh;
  auto load_line = [&](int row, R2 *dst) {
    const R2 *src = Tbase + ((long long)jl * a.rows + row) * n * plane + (long long)ky * nh;
    for (int i = threadIdx.x; i < n * nh; i += blockDim.x) {
      const int x = i / nh, kz = i - x * nh;
      dst[i] = src[(long long)x * plane + kz];
    }
    __syncthreads();
  };
  if (OUT != 2) {
    load_line(r, B0);
    const R2 *res = dft_axis0<R, R2>(B0, B1, n, nh, a.n1, w);
    const long long K0 = (long long)jl * 2 * n * plane;
    for (int i = threadIdx.x; i < n * nh; i += blockDim.x) {
      const int kx = i / nh, kz = i - kx * nh;
      const R s = wsq[(long long)kx * n * nh + kz];
      const long long K = K0 + 2 * (((long long)kx * n + ky) * nh + kz);
      const R re = res[i].x * s, im = res[i].y * s;
      if (OUT == 0) {
        double *Q = reinterpret_cast<double *>(a.Q) + (long long)r * a.ldq + K;
        Q[0] = re;
        Q[1] = im;
      } else {
        float *Qh = reinterpret_cast<float *>(a.Q) + (long long)r * a.ldq + K;
        float *Ql = Qh + (long long)a.rows * a.ldq;
        const float hr = __uint_as_float(tf32_rna_x((float)re)), hi = __uint_as_float(tf32_rna_x((float)im));
        *reinterpret_cast<float2 *>(Qh) = make_float2(hr, hi);
        *reinterpret_cast<float2 *>(Ql) =
            make_float2(__uint_as_float(tf32_rna_x((float)re - hr)), __uint_as_float(tf32_rna_x((float)im - hi)));
      }
    }
  } else {
    // rows: X_p at p, d_c phi_p at nao (1 + c) + p
    const int p = r;
    __shared__ double red[3][8];
    load_line(p, B0);
    const R2 *xh = dft_axis0<R, R2>(B0, B1, n, nh, a.n1, w);  // in B0 or B1
    R2 *spare = (xh == B0) ? B1 : B0;
    double acc[3] = {0, 0, 0};
    for (int c = 0; c < 3; ++c) {
      load_line(a.nao * (1 + c) + p, B2);
      const R2 *dh = dft_axis0<R, R2>(B2, spare, n, nh, a.n1, w);
      for (int i = threadIdx.x; i < n * nh; i += blockDim.x) {
        const int kx = i / nh, kz = i - kx * nh;
        const double s = (double)wsq[(long long)kx * n * nh + kz];
        acc[c] += s * s * ((double)xh[i].x * (double)dh[i].x + (double)xh[i].y * (double)dh[i].y);
      }
      __syncthreads();
    }
    const int lane = threadIdx.x & 31, wp = threadIdx.x >> 5;
    for (int c = 0; c < 3; ++c) {
      const double v = warp_sum(acc[c]);
      if (lane == 0) red[c][wp] = v;
    }
    __syncthreads();
    if (threadIdx.x < 3) {
      double s = 0;
      for (int k = 0; k < (int)(blockDim.x >> 5); ++k) s += red[threadIdx.x][k];
      a.part[(((long long)jl * a.nao + p) * n + ky) * 3 + threadIdx.x] = s;
    }
  }
}

// psi~_k(g) = sqrt(occ_k) sum_p C[p][k] phi_p(g) for k < nuse; 16 orbitals per
// block row, one grid point per thread.
template <typename R>
__global__ void __launch_bounds__(256) k_psi_all(const double *__restrict__ C, const double *__restrict__ occ,
                                                 int nao, int nmo, int nuse, const R *__restrict__ phi,
                                                 long long ldphi, long long N, R *__restrict__ out) {
  extern __shared__ __align__(16) unsigned char smraw[];
  R *Y = reinterpret_cast<R *>(smraw);  // [nao][16]
  const int k0 = blockIdx.y * 16;
  const int nk = min(16, nuse - k0);
  for (int i = threadIdx.x; i < nao * 16; i += blockDim.x) {
    const int p = i / 16, kk = i - p * 16;
    Y[i] = kk < nk ? (R)(C[(long long)p * nmo + k0 + kk] * sqrt(fmax(occ[k0 + kk], 0.0))) : (R)0;
  }
  __syncthreads();
  const long long g = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (g >= N) return;
  R acc[16];
#pragma unroll
  for (int kk = 0; kk < 16; ++kk) acc[kk] = 0;
  for (int p = 0; p < nao; ++p) {
    const R v = phi[(long long)p * ldphi + g];
#pragma unroll
    for (int kk = 0; kk < 16; ++kk) acc[kk] += Y[p * 16 + kk] * v;
  }
  for (int kk = 0; kk < nk; ++kk) out[(long long)(k0 + kk) * N + g] = acc[kk];
}

// grad[A][c] += sum_{p in A} sum_{jl < g, ky} part[((jl nao + p) n + ky)][c]
__global__ void k_exx_force_reduce(const double *__restrict__ part, int g, int nao, int nb, int n,
                                   double *__restrict__ grad) {
  __shared__ double sh[32];
  const int A = blockIdx.x;
  for (int c = 0; c < 3; ++c) {
    double s = 0;
    const int per = nb * n;
    for (int i = threadIdx.x; i < g * per; i += blockDim.x) {
      const int jl = i / per, rem = i - jl * per, pl = rem / n, ky = rem - pl * n;
      s += part[(((long long)jl * nao + A * nb + pl) * n + ky) * 3 + c];
    }
    s = block_sum(s, sh);
    if (threadIdx.x == 0) grad[A * 3 + c] += s;
  }
}

}  // namespace exx

// ---------------------------------------------------------------------------
int exx_factor(int n) {
  int n1 = 1;
  for (int f = 2; f * f <= n; ++f)
    if (n % f == 0) n1 = f;
  return n1;
}

template <typename R>
static size_t plane_smem(int n, int nprim) {
  using R2 = typename exx::C2<R>::T;
  const size_t bufc = (size_t)n * (n + 1) / 2 + 1;
  return sizeof(R2) * ((size_t)n + 2 * bufc) + sizeof(R) * 2 * nprim * n;
}

template <typename R>
static size_t column_smem(int n) {
  using R2 = typename exx::C2<R>::T;
  return sizeof(R2) * ((size_t)n + 3 * (size_t)n * ((n + 1) / 2));
}

bool exx_fused_supported(int n, int nprim, bool fp64) {
  const size_t lim = 227 * 1024;
  if (nprim > 8) return false;
  return fp64 ? (plane_smem<double>(n, nprim) <= lim && column_smem<double>(n) <= lim)
              : (plane_smem<float>(n, nprim) <= lim && column_smem<float>(n) <= lim);
}

long long exx_pair_len(int n) { return 2LL * n * n * ((n + 1) / 2); }

template <typename R>
void launch_exx_weights(int n, double L, double dV, R *wsq, cudaStream_t st) {
  const long long tot = (long long)n * n * ((n + 1) / 2);
  exx::k_pair_weights<R><<<ceil_div(tot, 256), 256, 0, st>>>(n, L, dV, wsq);
  HQ_LAUNCH_CHECK();
}
template void launch_exx_weights<float>(int, double, double, float *, cudaStream_t);
template void launch_exx_weights<double>(int, double, double, double *, cudaStream_t);

template <typename R>
void launch_psi_all(const double *C, const double *occ, int nao, int nmo, int nuse, const R *phi,
                    long long ldphi, long long N, R *out, cudaStream_t st) {
  HQ_STAGE(ST_EXCHANGE, st);
  HQ_REQUIRE(nao <= kMaxNao, "too many AOs");
  dim3 grid(ceil_div(N, 256), ceil_div(nuse, 16));
  const size_t smem = sizeof(R) * 16 * (size_t)nao;
  ensure_dyn_smem((const void *)exx::k_psi_all<R>, smem);
  exx::k_psi_all<R><<<grid, 256, smem, st>>>(C, occ, nao, nmo, nuse, phi, ldphi, N, out);
  HQ_LAUNCH_CHECK();
}
template void launch_psi_all<float>(const double *, const double *, int, int, int, const float *,
                                    long long, long long, float *, cudaStream_t);
template void launch_psi_all<double>(const double *, const double *, int, int, int, const double *,
                                     long long, long long, double *, cudaStream_t);

// Pair planes of `g` orbitals (psi~ rows from psi, ldpsi apart): rows = nao
// (Fock: phi_p psi~_j) or 4 nao with X (gradient: X_p psi~_j, then
// d_c phi_p psi~_j for c = x, y, z).
template <typename R>
void launch_exx_plane(const ExxGeom &G, const R *F1d, const double *X, long long ldx, const R *psi,
                      long long ldpsi, int g, void *T, cudaStream_t st) {
  HQ_STAGE(ST_EXCHANGE, st);
  exx::PlaneArgs a;
  a.n = G.n;
  a.nh = (G.n + 1) / 2;
  a.n1 = exx_factor(G.n);
  a.nao = G.nao;
  a.nb = G.nb;
  a.nprim = G.nprim;
  a.rows = X ? 4 * G.nao : G.nao;
  a.xrows = X ? G.nao : 0;
  a.tw = G.tw;
  a.F1d = F1d;
  a.coef = G.coef;
  a.ao_l = G.ao_l;
  a.ao_cart = G.ao_cart;
  a.X = X;
  a.ldx = ldx;
  a.psi = psi;
  a.ldpsi = ldpsi;
  a.T = T;
  // The shared field takes n (n + 1) reals, where that leaves four (FP64: two)
  // blocks an SM; as many blocks as orbitals allow above four waves.
  size_t smem = plane_smem<R>(G.n, G.nprim);
  const size_t field = sizeof(R) * ((size_t)G.n * (G.n + 1) + 2);
  const int blocks = sizeof(R) == 4 ? 4 : 2;
  a.g = g;
  a.per = 1;
  if (g > 1 && blocks * (smem + field + 1024) <= 228 * 1024) {
    const int split = std::min(g, std::max(1, ceil_div(152 * blocks * 4, (long long)G.n * a.rows)));
    a.per = ceil_div(g, split);
    if (a.per > 1) smem += field;
  }
  ensure_dyn_smem((const void *)exx::k_exx_plane<R>, smem);
  exx::k_exx_plane<R><<<dim3(G.n, a.rows, ceil_div(g, a.per)), 256, smem, st>>>(a);
  HQ_LAUNCH_CHECK();
}

template <typename R, int OUT>
static void column(const ExxGeom &G, int rows, const void *T, int g, void *Q, long long ldq, double *part,
                   cudaStream_t st) {
  exx::ColumnArgs a;
  a.n = G.n;
  a.nh = (G.n + 1) / 2;
  a.n1 = exx_factor(G.n);
  a.nao = G.nao;
  a.rows = rows;
  a.tw = G.tw;
  a.wsq = G.wsq;
  a.T = T;
  a.Q = Q;
  a.ldq = ldq;
  a.part = part;
  const size_t smem = column_smem<R>(G.n);
  ensure_dyn_smem((const void *)exx::k_exx_column<R, OUT>, smem);
  exx::k_exx_column<R, OUT><<<dim3(G.n, OUT == 2 ? G.nao : rows, g), 256, smem, st>>>(a);
  HQ_LAUNCH_CHECK();
}

// Q rows of the Fock build: FP64 (split = false) or the TF32 hi/lo pieces.
template <typename R>
void launch_exx_column_q(const ExxGeom &G, const void *T, int g, void *Q, long long ldq, bool split,
                         cudaStream_t st) {
  HQ_STAGE(ST_EXCHANGE, st);
  if (split) column<R, 1>(G, G.nao, T, g, Q, ldq, nullptr, st);
  else column<R, 0>(G, G.nao, T, g, Q, ldq, nullptr, st);
}

// Gradient dot products of a group, reduced into grad [n_atoms][3].
template <typename R>
void launch_exx_column_grad(const ExxGeom &G, const void *T, int g, double *part, double *grad,
                            cudaStream_t st) {
  HQ_STAGE(ST_EXCHANGE, st);
  column<R, 2>(G, 4 * G.nao, T, g, nullptr, 0, part, st);
  exx::k_exx_force_reduce<<<G.nao / G.nb, 256, 0, st>>>(part, g, G.nao, G.nb, G.n, grad);
  HQ_LAUNCH_CHECK();
}

template void launch_exx_plane<float>(const ExxGeom &, const float *, const double *, long long,
                                      const float *, long long, int, void *, cudaStream_t);
template void launch_exx_plane<double>(const ExxGeom &, const double *, const double *, long long,
                                       const double *, long long, int, void *, cudaStream_t);
template void launch_exx_column_q<float>(const ExxGeom &, const void *, int, void *, long long, bool,
                                         cudaStream_t);
template void launch_exx_column_q<double>(const ExxGeom &, const void *, int, void *, long long, bool,
                                          cudaStream_t);
template void launch_exx_column_grad<float>(const ExxGeom &, const void *, int, double *, double *,
                                            cudaStream_t);
template void launch_exx_column_grad<double>(const ExxGeom &, const void *, int, double *, double *,
                                             cudaStream_t);

}  // namespace hqcgb
