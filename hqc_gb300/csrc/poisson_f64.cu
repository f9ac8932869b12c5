// FP64 Hartree potential on an odd grid: v = DFT^-1[4 pi / G^2 DFT[rho]]
// (hqc/pbc/solver.py:187-207, 592-629 by Parseval, as fft_fp64.cu) for a real
// density.  Only the half spectrum kz = 0 .. (n - 1) / 2 is formed: two real
// z lines make one complex transform, the y and x transforms run over half of
// the columns, the x pass multiplies by the Coulomb kernel and transforms back
// in place, and two half-spectrum lines make one complex inverse.  The
// transforms are the paired two-factor ones of the exchange (conjugate outputs
// k and n - k together).  The FP64 pipe bounds it: the complex passes with one
// output a thread took six FP64 instructions a term and both halves, these
// take four a pair of outputs and one half.  Five launches of columns in
// chunks, so that every pass fills the SMs.  Measured, one
// potential: 65^3 0.70 -> 0.12 ms, 41^3 (a prime, direct sums) 0.57 -> 0.11,
// 49^3 0.28 -> 0.09.
#include <algorithm>

#include "dft_shared.cuh"
#include "kernels.h"

namespace hqcgb {

using exx::dft_axis0;
using exx::load_twiddles;

constexpr int kPsThreads = 128;
constexpr int kPsCols = 8;  // columns a block

struct PsArgs {
  int n, nh, n1;
  const double2 *tw;
  const double *src, *kern;
  double *dst;
  double2 *T;  // [x][y][kz]
};

__device__ inline double2 conj2(double2 a) { return make_double2(a.x, -a.y); }

// z lines of rho, two a column: T[x][y][kz] = sum_z rho W^(z kz)
__global__ void __launch_bounds__(kPsThreads) k_ps_z(PsArgs a) {
  extern __shared__ __align__(16) unsigned char smraw[];
  const int n = a.n, nh = a.nh, npair = (n + 1) / 2;
  double2 *w = reinterpret_cast<double2 *>(smraw), *B0 = w + n, *B1 = B0 + n * kPsCols;
  load_twiddles(w, a.tw, n);
  const int first = blockIdx.x * kPsCols, cols = min(kPsCols, n * npair - first);
  for (int i = threadIdx.x; i < n * cols; i += kPsThreads) {
    const int c = i / n, z = i - c * n, id = first + c, x = id / npair, pr = id - x * npair;
    const double *line = a.src + ((long long)x * n + 2 * pr) * n + z;
    B0[z * cols + c] = make_double2(line[0], 2 * pr + 1 < n ? line[n] : 0.0);
  }
  __syncthreads();
  const double2 *Z = dft_axis0<double, double2>(B0, B1, n, cols, a.n1, w);
  // A[k] = (Z[k] + conj Z[n-k]) / 2 of the first line, B[k] = (Z[k] - conj Z[n-k]) / 2i of the second
  for (int i = threadIdx.x; i < nh * cols; i += kPsThreads) {
    const int c = i / nh, kz = i - c * nh, id = first + c, x = id / npair, pr = id - x * npair;
    const double2 p = Z[kz * cols + c], q = Z[(kz == 0 ? 0 : n - kz) * cols + c];
    double2 *o = a.T + ((long long)x * n + 2 * pr) * nh + kz;
    o[0] = make_double2(0.5 * (p.x + q.x), 0.5 * (p.y - q.y));
    if (2 * pr + 1 < n) o[nh] = make_double2(0.5 * (p.y + q.y), 0.5 * (q.x - p.x));
  }
}

// The y transform of every x plane, columns kz in chunks; INV: the inverse.
template <bool INV>
__global__ void __launch_bounds__(kPsThreads) k_ps_y(PsArgs a) {
  extern __shared__ __align__(16) unsigned char smraw[];
  const int n = a.n, nh = a.nh;
  double2 *w = reinterpret_cast<double2 *>(smraw), *B0 = w + n, *B1 = B0 + n * kPsCols;
  load_twiddles(w, a.tw, n);
  const int k0 = blockIdx.y * kPsCols, cols = min(kPsCols, nh - k0);
  double2 *base = a.T + (long long)blockIdx.x * n * nh + k0;
  for (int i = threadIdx.x; i < n * cols; i += kPsThreads) {
    const int y = i / cols, c = i - y * cols;
    const double2 v = base[(long long)y * nh + c];
    B0[i] = INV ? conj2(v) : v;
  }
  __syncthreads();
  const double2 *R = dft_axis0<double, double2>(B0, B1, n, cols, a.n1, w);
  for (int i = threadIdx.x; i < n * cols; i += kPsThreads) {
    const int y = i / cols, c = i - y * cols;
    base[(long long)y * nh + c] = INV ? conj2(R[i]) : R[i];
  }
}

// The x transform of a ky plane's columns, times the Coulomb kernel, and back.
__global__ void __launch_bounds__(kPsThreads) k_ps_x(PsArgs a) {
  extern __shared__ __align__(16) unsigned char smraw[];
  const int n = a.n, nh = a.nh, ky = blockIdx.x;
  double2 *w = reinterpret_cast<double2 *>(smraw), *B0 = w + n, *B1 = B0 + n * kPsCols;
  load_twiddles(w, a.tw, n);
  const int k0 = blockIdx.y * kPsCols, cols = min(kPsCols, nh - k0);
  double2 *base = a.T + (long long)ky * nh + k0;
  for (int i = threadIdx.x; i < n * cols; i += kPsThreads) {
    const int x = i / cols, c = i - x * cols;
    B0[i] = base[(long long)x * n * nh + c];
  }
  __syncthreads();
  double2 *R = dft_axis0<double, double2>(B0, B1, n, cols, a.n1, w);
  for (int i = threadIdx.x; i < n * cols; i += kPsThreads) {
    const int kx = i / cols, c = i - kx * cols;
    const double f = a.kern[((long long)kx * n + ky) * n + k0 + c];
    R[i] = make_double2(f * R[i].x, -f * R[i].y);  // conjugated: the next transform is the inverse
  }
  __syncthreads();
  double2 *spare = R == B0 ? B1 : B0;
  const double2 *S = dft_axis0<double, double2>(R, spare, n, cols, a.n1, w);
  for (int i = threadIdx.x; i < n * cols; i += kPsThreads) {
    const int x = i / cols, c = i - x * cols;
    base[(long long)x * n * nh + c] = conj2(S[i]);
  }
}

// z lines back: Z[k] = A[k] + i B[k] of two half-spectrum lines, whose inverse
// has the lines as its real and imaginary part.
__global__ void __launch_bounds__(kPsThreads) k_ps_z_inverse(PsArgs a) {
  extern __shared__ __align__(16) unsigned char smraw[];
  const int n = a.n, nh = a.nh, npair = (n + 1) / 2;
  double2 *w = reinterpret_cast<double2 *>(smraw), *B0 = w + n, *B1 = B0 + n * kPsCols;
  load_twiddles(w, a.tw, n);
  const int first = blockIdx.x * kPsCols, cols = min(kPsCols, n * npair - first);
  for (int i = threadIdx.x; i < nh * cols; i += kPsThreads) {
    const int c = i / nh, kz = i - c * nh, id = first + c, x = id / npair, pr = id - x * npair;
    const double2 *o = a.T + ((long long)x * n + 2 * pr) * nh + kz;
    const double2 A = o[0], B = 2 * pr + 1 < n ? o[nh] : make_double2(0.0, 0.0);
    // conjugated: conj(A + i B) at kz, conj(conj A + i conj B) at n - kz; kz = 0 is real in both lines
    B0[kz * cols + c] = make_double2(A.x - (kz ? B.y : 0.0), -(kz ? A.y : 0.0) - B.x);
    if (kz) B0[(n - kz) * cols + c] = make_double2(A.x + B.y, A.y - B.x);
  }
  __syncthreads();
  const double2 *Z = dft_axis0<double, double2>(B0, B1, n, cols, a.n1, w);
  for (int i = threadIdx.x; i < n * cols; i += kPsThreads) {
    const int c = i / n, z = i - c * n, id = first + c, x = id / npair, pr = id - x * npair;
    double *line = a.dst + ((long long)x * n + 2 * pr) * n + z;
    const double2 v = Z[z * cols + c];
    line[0] = v.x;
    if (2 * pr + 1 < n) line[n] = -v.y;
  }
}

bool poisson_f64_supported(int n) { return n % 2 == 1; }

void launch_poisson_f64(const double *src, double *dst, double2 *cbuf, const double *kern, int n, const double2 *tw,
                        cudaStream_t st) {
  HQ_STAGE(ST_FFT, st);
  PsArgs a{n, (n + 1) / 2, exx_factor(n), tw, src, kern, dst, cbuf};
  const size_t smem = ((size_t)n + 2 * (size_t)n * kPsCols) * sizeof(double2);
  const int lines = ceil_div((long long)n * a.nh, kPsCols);
  const dim3 columns(n, ceil_div(a.nh, kPsCols));
  auto go = [&](auto kernel, dim3 grid) {
    ensure_dyn_smem((const void *)kernel, smem);
    kernel<<<grid, kPsThreads, smem, st>>>(a);
    HQ_LAUNCH_CHECK();
  };
  go(k_ps_z, dim3(lines));
  go(k_ps_y<false>, columns);
  go(k_ps_x, columns);
  go(k_ps_y<true>, columns);
  go(k_ps_z_inverse, dim3(lines));
}

}  // namespace hqcgb
