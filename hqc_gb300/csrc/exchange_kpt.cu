// FP64 grid contractions of the k-point SCF (kpoint.cu): the exchange's pair
// densities and transforms, and M_pq = sum_g A_p(g) conj(B_q(g)).
//
// Exchange: three passes over the pair densities P_pj = phibar_p conj(psibar_j)
// of a group of orbitals (hqc/pbc/solver.py:509-524 by Parseval).  The z pass
// forms the pairs as it loads, the x pass multiplies by sqrt(f_j c(G)) as it
// stores, and each pass transforms a block of lines in shared memory with the
// folded two-factor transforms of dft_shared.cuh.  The lines of a plane are taken
// as one run, so that an axis of 33 points does not leave blocks of one line.
// Bound by the FP64 pipe and L2.  Measured, H8 dzv at 33^3, one orbital (16
// grids): pairs, transforms and scaling 0.43 -> 0.08 ms.
//
// Contraction: the output has few tiles and the sum is long, so the sum is split
// over the grid: a block adds its part of one 16 x 16 tile with 128 threads of
// 2 x 2 outputs (two halves of the part's points), and a second kernel adds the
// parts.  A Hermitian result takes the tiles of one triangle.  Bound by the
// FP64 pipe (four multiply-adds a point and output).  Measured, 16 AOs, 33^3: one
// contraction of the library (split over few blocks, FP64 tensor pipe) 0.39 ms,
// this one 0.07 (its sum of the parts included).
#include <algorithm>

#include "dft_shared.cuh"
#include "kernels.h"
#include "zmath.cuh"

namespace hqcgb {

using exx::dft_axis0;
using exx::load_twiddles;

constexpr int kKxThreads = 128;

struct KxArgs {
  int n, n1, nao, cols;
  long long N;
  const double2 *tw, *phi, *psi;  // z pass: phibar [nao][N], psibar of the group's orbitals [g][N]
  const double *kern;             // x pass: sqrt(c(G))
  double2 *W;                     // [g][nao][N]
  double sqf[kKxGroup];           // x pass: sqrt(f_j)
};

// One axis of all grids; grid (runs of `cols` lines, AO, orbital).  AXIS 0 = x, 1 = y, 2 = z.
template <int AXIS>
__global__ void __launch_bounds__(kKxThreads) k_kx_pass(const __grid_constant__ KxArgs a) {
  extern __shared__ __align__(16) unsigned char smraw[];
  const int n = a.n, p = blockIdx.y, j = blockIdx.z;
  const int first = blockIdx.x * a.cols, cols = min(a.cols, n * n - first);
  double2 *w = reinterpret_cast<double2 *>(smraw), *B0 = w + n, *B1 = B0 + n * a.cols;
  load_twiddles(w, a.tw, n);
  double2 *W = a.W + ((long long)j * a.nao + p) * a.N;
  if (AXIS == 2) {  // lines (x, y), contiguous
    const double2 *phi = a.phi + (long long)p * a.N + (long long)first * n;
    const double2 *psi = a.psi + (long long)j * a.N + (long long)first * n;
    for (int i = threadIdx.x; i < n * cols; i += kKxThreads) {
      const int c = i / n, z = i - c * n;
      B0[z * cols + c] = zmul(phi[i], zconj(psi[i]));
    }
  } else {
    for (int i = threadIdx.x; i < n * cols; i += kKxThreads) {
      const int t = i / cols, id = first + i - t * cols;
      // x: lines (y, z);  y: lines (x, z)
      B0[i] = AXIS == 0 ? W[(long long)t * n * n + id] : W[((long long)(id / n) * n + t) * n + id % n];
    }
  }
  __syncthreads();
  const double2 *R = dft_axis0<double, double2>(B0, B1, n, cols, a.n1, w);
  if (AXIS == 2) {
    for (int i = threadIdx.x; i < n * cols; i += kKxThreads) {
      const int c = i / n, z = i - c * n;
      W[(long long)first * n + i] = R[z * cols + c];
    }
  } else {
    const double s = AXIS == 0 ? a.sqf[j] : 1.0;
    for (int i = threadIdx.x; i < n * cols; i += kKxThreads) {
      const int t = i / cols, id = first + i - t * cols;
      if (AXIS == 0) {
        const long long g = (long long)t * n * n + id;
        const double f = s * a.kern[g];
        W[g] = make_double2(f * R[i].x, f * R[i].y);
      } else {
        W[((long long)(id / n) * n + t) * n + id % n] = R[i];
      }
    }
  }
}

static int kx_cols(int n) { return n <= 49 ? 32 : n <= 97 ? 16 : 8; }

// Orbitals a group: the pair densities within 256 MB
int kx_group(int nao, long long N) {
  return (int)std::max(1LL, std::min((long long)kKxGroup, (256LL << 20) / ((long long)nao * N * 16)));
}

void launch_kx_pairs(const double2 *phi, const double2 *psi, const double *f, int g, const double *sqcoul, int n,
                     int nao, const double2 *tw, double2 *W, cudaStream_t st) {
  HQ_STAGE(ST_FFT, st);
  HQ_REQUIRE(n % 2 == 1 && n <= kMaxGrid && g <= kKxGroup, "odd grids and groups within the limit only");
  KxArgs a{n, exx_factor(n), nao, kx_cols(n), (long long)n * n * n, tw, phi, psi, sqcoul, W, {}};
  for (int j = 0; j < g; ++j) a.sqf[j] = std::sqrt(f[j]);
  const size_t smem = ((size_t)n + 2 * (size_t)n * a.cols) * sizeof(double2);
  const dim3 grid(ceil_div((long long)n * n, a.cols), nao, g);
  auto go = [&](auto kernel) {
    ensure_dyn_smem((const void *)kernel, smem);
    kernel<<<grid, kKxThreads, smem, st>>>(a);
    HQ_LAUNCH_CHECK();
  };
  go(k_kx_pass<2>);
  go(k_kx_pass<1>);
  go(k_kx_pass<0>);
}

// ---------------------------------------------------------------------------
constexpr int kZgT = 16, kZgK = 32, kZgThreads = 128;

struct ZgArgs {
  int n, nt;            // rows, tiles a side
  int herm;             // tiles (tp >= tq) only
  long long N, part;    // points a set, points a part (a multiple of kZgK)
  int parts;            // parts a set
  const double2 *A, *B;
  long long sA, sB;     // from one set to the next
  double2 *P;           // [set, part][tile][16][16]
};

__global__ void __launch_bounds__(kZgThreads) k_zgram(ZgArgs a) {
  __shared__ double2 As[kZgT][kZgK + 1], Bs[kZgT][kZgK + 1];
  int tp, tq;
  if (a.herm) {
    tp = (int)((sqrtf(8.f * blockIdx.x + 1.f) - 1.f) * 0.5f);
    while (tp * (tp + 1) / 2 > (int)blockIdx.x) --tp;
    while ((tp + 1) * (tp + 2) / 2 <= (int)blockIdx.x) ++tp;
    tq = blockIdx.x - tp * (tp + 1) / 2;
  } else {
    tp = blockIdx.x / a.nt;
    tq = blockIdx.x - tp * a.nt;
  }
  const int set = blockIdx.y / a.parts, part = blockIdx.y - set * a.parts;
  const long long k0 = part * a.part, k1 = min(k0 + a.part, a.N);
  const double2 *A = a.A + set * a.sA, *B = a.B + set * a.sB;
  const bool same = A == B && tp == tq, lower = a.herm && tp == tq;  // no use for the quarter above the diagonal
  const int tid = threadIdx.x, half = tid >> 6, ty = (tid >> 3) & 7, tx = tid & 7;
  const double2(*Bt)[kZgK + 1] = same ? As : Bs;
  const double2 zero = make_double2(0.0, 0.0);
  constexpr int PT = kZgT * kZgK / kZgThreads;  // values a thread loads of each side
  double2 ra[PT], rb[PT];
  auto fetch = [&](long long k) {
#pragma unroll
    for (int q = 0; q < PT; ++q) {
      const int i = tid + q * kZgThreads, r = i / kZgK;
      const long long x = k + i % kZgK;
      const int p = tp * kZgT + r, qq = tq * kZgT + r;
      ra[q] = p < a.n && x < k1 ? A[(long long)p * a.N + x] : zero;
      rb[q] = !same && qq < a.n && x < k1 ? B[(long long)qq * a.N + x] : zero;
    }
  };
  double2 acc[2][2] = {{zero, zero}, {zero, zero}};
  fetch(k0);
  for (long long k = k0; k < k1; k += kZgK) {
#pragma unroll
    for (int q = 0; q < PT; ++q) {
      const int i = tid + q * kZgThreads;
      As[i / kZgK][i % kZgK] = ra[q];
      if (!same) Bs[i / kZgK][i % kZgK] = rb[q];
    }
    __syncthreads();
    if (k + kZgK < k1) fetch(k + kZgK);
#pragma unroll 4
    for (int kk = half; kk < kZgK; kk += 2) {
      const double2 u[2] = {As[ty][kk], As[ty + 8][kk]}, v[2] = {Bt[tx][kk], Bt[tx + 8][kk]};
#pragma unroll
      for (int r = 0; r < 2; ++r)
#pragma unroll
        for (int c = 0; c < 2; ++c) {  // u conj(v)
          if (c > r && lower) continue;
          acc[r][c].x = fma(u[r].x, v[c].x, fma(u[r].y, v[c].y, acc[r][c].x));
          acc[r][c].y = fma(u[r].y, v[c].x, fma(-u[r].x, v[c].y, acc[r][c].y));
        }
    }
    __syncthreads();
  }
  double2(*sum)[kZgK + 1] = As;  // [16][16] of it
  if (half)
#pragma unroll
    for (int r = 0; r < 2; ++r)
#pragma unroll
      for (int c = 0; c < 2; ++c) sum[ty + 8 * r][tx + 8 * c] = acc[r][c];
  __syncthreads();
  if (!half) {
    double2 *out = a.P + ((long long)blockIdx.y * gridDim.x + blockIdx.x) * (kZgT * kZgT);
#pragma unroll
    for (int r = 0; r < 2; ++r)
#pragma unroll
      for (int c = 0; c < 2; ++c) {
        const double2 o = sum[ty + 8 * r][tx + 8 * c];
        out[(ty + 8 * r) * kZgT + tx + 8 * c] = make_double2(acc[r][c].x + o.x, acc[r][c].y + o.y);
      }
  }
}

// M (+)= alpha sum of the parts; a warp an element
__global__ void __launch_bounds__(256) k_zgram_sum(int n, int nt, int herm, int ntile, int nparts, double alpha,
                                                   const double2 *__restrict__ P, int accumulate,
                                                   double2 *__restrict__ M) {
  const int e = blockIdx.x * 8 + (threadIdx.x >> 5), lane = threadIdx.x & 31;
  if (e >= n * n) return;
  const int p = e / n, q = e - p * n, tp = p / kZgT, tq = q / kZgT;
  const bool flip = herm && p < q;
  const int a = flip ? tq : tp, b = flip ? tp : tq;
  const int tile = herm ? a * (a + 1) / 2 + b : tp * nt + tq;
  const int r = (flip ? q : p) % kZgT, c = (flip ? p : q) % kZgT;
  double x = 0.0, y = 0.0;
  for (int s = lane; s < nparts; s += 32) {
    const double2 v = P[((long long)s * ntile + tile) * (kZgT * kZgT) + r * kZgT + c];
    x += v.x;
    y += v.y;
  }
  x = alpha * warp_sum(x);
  y = alpha * warp_sum(flip ? -y : y);
  if (lane) return;
  if (accumulate) {
    x += M[e].x;
    y += M[e].y;
  }
  M[e] = make_double2(x, y);
}

// Parts of the sum over `sets` x N points: about six blocks an SM in all, at
// least 256 points each, so that the parts stay within a few MB.
static int zg_parts(int ntile, int sets, long long N) {
  const long long want = std::max(1LL, 912LL / ((long long)ntile * sets));
  return (int)std::min(want, std::max(1LL, N / 256));
}
static int zg_tiles(int n, bool herm) {
  const int nt = ceil_div(n, kZgT);
  return herm ? nt * (nt + 1) / 2 : nt * nt;
}

size_t zgram_scratch(int n, int sets, long long N) {  // double2s, either form
  size_t most = 0;
  for (int h = 0; h < 2; ++h)
    for (int s = 1; s <= sets; ++s) {
      const int t = zg_tiles(n, h == 1);
      most = std::max(most, (size_t)t * s * zg_parts(t, s, N) * kZgT * kZgT);
    }
  return most;
}

void launch_zgram(int n, long long N, int sets, const double2 *A, long long sA, const double2 *B, long long sB,
                  bool herm, double alpha, bool accumulate, double2 *P, double2 *M, cudaStream_t st) {
  ZgArgs a;
  a.n = n;
  a.nt = ceil_div(n, kZgT);
  a.herm = herm ? 1 : 0;
  a.N = N;
  const int ntile = zg_tiles(n, herm);
  a.parts = zg_parts(ntile, sets, N);
  a.part = (ceil_div(N, (long long)a.parts) + kZgK - 1) / kZgK * kZgK;
  a.A = A;
  a.B = B;
  a.sA = sA;
  a.sB = sB;
  a.P = P;
  k_zgram<<<dim3(ntile, sets * a.parts), kZgThreads, 0, st>>>(a);
  HQ_LAUNCH_CHECK();
  k_zgram_sum<<<ceil_div((long long)n * n, 8), 256, 0, st>>>(n, a.nt, a.herm, ntile, sets * a.parts, alpha, P,
                                                            accumulate ? 1 : 0, M);
  HQ_LAUNCH_CHECK();
}

}  // namespace hqcgb
