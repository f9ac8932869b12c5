// Ewald energy of proton + electron configurations, batched over walkers:
// potential_energy of hqc/pbc/potential.py:69-101 (with psi, 35-67).  For
// each configuration x [n][dim] (rs units; the first n/2 particles are
// protons, Z = +1, the rest electrons, Z = -1) it returns
//   vpp =  2 rs / L sum_{i<j, pp} psi(r_ij),  vep = -2 rs / L sum_{ep} psi,
//   vee =  2 rs / L sum_{i<j, ee} psi,
//   psi(r) = erfc(kappa |r|) / |r|  (nearest image)  + sum_G g(G) cos(2 pi G.r) + g0,
// r_ij = (x_i - x_j) / L wrapped to the nearest image, G the caller's integer
// vectors (kpoints(dim, Gmax), potential.py:6-16).
//
// The reciprocal part is not summed pair by pair: with the species structure
// factors S_A(G) = sum_{i in A} exp(2 pi i G.x_i / L),
//   sum_{i<j in A} cos(2 pi G.r_ij) = (|S_A|^2 - n_A) / 2,
//   sum_{i in p, j in e} cos(2 pi G.r_ij) = Re(S_p conj(S_e)),
// so a configuration costs n N_G phase evaluations instead of n^2 N_G / 2
// (integer G makes the nearest-image shift irrelevant to the cosine).  The
// real-space erfc term stays pairwise (n^2 / 2, no G loop).
#include <algorithm>
#include <climits>
#include <cstdlib>
#include <vector>

#include "common.cuh"
#include "kernels.h"

namespace hqcgb {

constexpr int kCbThreads = 256;
constexpr int kCbMaxParticles = 2048;

__device__ inline double coul_gk(int dim, double G2, double kappa) {
  if (dim == 3) return exp(-M_PI * M_PI * G2 / (kappa * kappa)) / (M_PI * G2);
  const double g = sqrt(G2);
  return erfc(M_PI * g / kappa) / g;
}

// Any integer vectors: grid (B, ceil(nG / 256)); one thread per G vector of configuration b.
// part[b][blockIdx.y][3] = sum over this block's G of g(G) x {pp, ep, ee} cosine sums.
// Only for components beyond kMaxIndex, whose phase tables would not fit.
__global__ void __launch_bounds__(kCbThreads)
    k_coul_recip_any(int n, int dim, const double *__restrict__ x, double L, const int *__restrict__ G,
                 int nG, double kappa, int stride, double *__restrict__ part) {
  extern __shared__ double xs[];  // [n][dim] / L
  __shared__ double sh[32];
  const int b = blockIdx.x;
  const double *xb = x + (long long)b * n * dim;
  for (int k = threadIdx.x; k < n * dim; k += blockDim.x) xs[k] = xb[k] / L;
  __syncthreads();
  const int np = n / 2;
  const int gi = blockIdx.y * blockDim.x + threadIdx.x;
  double vpp = 0, vep = 0, vee = 0;
  if (gi < nG) {
    int g[3] = {0, 0, 0};
    double G2 = 0;
    for (int d = 0; d < dim; ++d) {
      g[d] = G[gi * dim + d];
      G2 += (double)g[d] * g[d];
    }
    double spr = 0, spi = 0, ser = 0, sei = 0;
    for (int i = 0; i < n; ++i) {
      double ph = 0;
      for (int d = 0; d < dim; ++d) ph += g[d] * xs[i * dim + d];
      double s, c;
      sincospi(2.0 * ph, &s, &c);
      if (i < np) {
        spr += c;
        spi += s;
      } else {
        ser += c;
        sei += s;
      }
    }
    const double gk = coul_gk(dim, G2, kappa);
    vpp = gk * 0.5 * (spr * spr + spi * spi - np);
    vee = gk * 0.5 * (ser * ser + sei * sei - (n - np));
    vep = gk * (spr * ser + spi * sei);
  }
  vpp = block_sum(vpp, sh);
  vep = block_sum(vep, sh);
  vee = block_sum(vee, sh);
  if (threadIdx.x == 0) {
    double *o = part + ((long long)b * stride + blockIdx.y) * 3;
    o[0] = vpp;
    o[1] = vep;
    o[2] = vee;
  }
}

// The reciprocal sums run over columns: every listed G is folded onto its
// half space (|S(-G)| = |S(G)|, and the same for Re S_p conj(S_e)), and the
// vectors (gx, gy, +-gz) of a column share
//   S(gx, gy, +-gz) = sum_i A_i (c_i +- i s_i),   A_i = e^(2 pi i (gx x + gy y)),
// through the four real sums of Ar c, Ai s, Ar s, Ai c: four multiply-adds a
// particle for two vectors, and their mirror images for nothing, where a
// phase evaluation a vector and particle cost a sincospi (about 40 FP64
// instructions).  A thread owns kRun consecutive gz of one column; the 1D
// phases of kChunk particles sit in shared memory (powers of one sincospi an
// axis and particle).  GB300 issues 2 FP64 multiply-adds a cycle and SM, so
// the kernel is bound by their count: nG (1 + 1/RUN) a particle.  Measured at
// 1024 walkers of 54 + 54 particles, Gmax 15: the whole call 109.8 ms
// with a phase a vector, 6.3 ms with columns (0.41 of the FP64 rate).
constexpr int kChunk = 32;    // particles whose phases are in shared memory at a time
constexpr int kMaxIndex = 31; // largest |G component| of the column form

struct CoulItem {
  int gx, gy, gz0, pad;  // the column and the first gz of the run
};

__device__ inline double2 cmul(double2 a, double2 b) {
  return make_double2(a.x * b.x - a.y * b.y, a.x * b.y + a.y * b.x);
}

// Multiplicities of the listed vectors to weights g(G): wt[item][r][+-].
__global__ void k_coul_weights(int dim, double kappa, const CoulItem *__restrict__ items, int n_items, int run,
                               double *__restrict__ wt) {
  const int k = blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= n_items * run) return;
  const CoulItem it = items[k / run];
  const double gz = it.gz0 + k % run;
  const double G2 = (double)it.gx * it.gx + (double)it.gy * it.gy + gz * gz;
  if (wt[2 * k] == 0.0 && wt[2 * k + 1] == 0.0) return;  // also G = 0, which is never listed
  const double g = coul_gk(dim, G2, kappa);
  wt[2 * k] *= g;
  wt[2 * k + 1] *= g;
}

// Grid (B, ceil(items / blockDim)); part[b][blockIdx.y][3] = this block's g(G) x {pp, ep, ee} cosine sums.
// In two dimensions x is particle axis 0, z is axis 1, and gy = 0.
template <int RUN>
__global__ void __launch_bounds__(128)
    k_coul_recip(int n, int dim, const double *__restrict__ x, double L, const CoulItem *__restrict__ items,
                 int n_items, int m1, const double *__restrict__ wt, int stride, double *__restrict__ part) {
  extern __shared__ double2 ph[];  // [kChunk][3][m1], m1 = largest index + 1
  __shared__ double sh[32];
  const int b = blockIdx.x, tid = threadIdx.x;
  const double *xb = x + (long long)b * n * dim;
  const int np = n / 2;
  const int item = blockIdx.y * blockDim.x + tid;
  const bool on = item < n_items;
  CoulItem it{0, 0, 0, 0};
  if (on) it = items[item];
  const int ay = it.gy < 0 ? -it.gy : it.gy;
  const double sy = it.gy < 0 ? -1.0 : 1.0;
  double2 sp[RUN][2];  // the protons' S(+-gz)
  double2 s[RUN][2];
#pragma unroll
  for (int r = 0; r < RUN; ++r) sp[r][0] = sp[r][1] = s[r][0] = s[r][1] = make_double2(0.0, 0.0);
  for (int species = 0; species < 2; ++species) {
    const int lo = species == 0 ? 0 : np, hi = species == 0 ? np : n;
    double q[RUN][4];
#pragma unroll
    for (int r = 0; r < RUN; ++r) q[r][0] = q[r][1] = q[r][2] = q[r][3] = 0.0;
    for (int i0 = lo; i0 < hi; i0 += kChunk) {
      const int cnt = min(kChunk, hi - i0);
      __syncthreads();  // the previous chunk's phases are no longer read
      for (int k = tid; k < cnt * 3; k += blockDim.x) {
        const int i = k / 3, d = k % 3;
        const int src = dim == 3 ? d : (d == 0 ? 0 : d == 2 ? 1 : -1);
        double2 e = make_double2(1.0, 0.0);
        if (src >= 0) sincospi(2.0 * (xb[(i0 + i) * dim + src] / L), &e.y, &e.x);
        double2 *t = ph + k * m1;
        t[0] = make_double2(1.0, 0.0);
        double2 cur = e;
        for (int m = 1; m < m1; ++m) {
          t[m] = cur;
          cur = cmul(cur, e);
        }
      }
      __syncthreads();
      if (on)
        for (int i = 0; i < cnt; ++i) {
          const double2 *t = ph + i * 3 * m1;
          const double2 ex = t[it.gx];
          double2 ey = t[m1 + ay];
          ey.y *= sy;
          const double2 a = cmul(ex, ey);
          const double2 *z = t + 2 * m1 + it.gz0;
#pragma unroll
          for (int r = 0; r < RUN; ++r) {
            const double2 c = z[it.gz0 + r < m1 ? r : 0];
            q[r][0] += a.x * c.x;
            q[r][1] += a.y * c.y;
            q[r][2] += a.x * c.y;
            q[r][3] += a.y * c.x;
          }
        }
    }
#pragma unroll
    for (int r = 0; r < RUN; ++r) {
      if (species == 1) {
        sp[r][0] = s[r][0];
        sp[r][1] = s[r][1];
      }
      s[r][0] = make_double2(q[r][0] - q[r][1], q[r][2] + q[r][3]);
      s[r][1] = make_double2(q[r][0] + q[r][1], q[r][3] - q[r][2]);
    }
  }
  double vpp = 0, vep = 0, vee = 0;
  if (on)
#pragma unroll
    for (int r = 0; r < RUN; ++r)
#pragma unroll
      for (int sgn = 0; sgn < 2; ++sgn) {
        const double g = wt[((long long)item * RUN + r) * 2 + sgn];  // 0 where not listed
        const double2 p = sp[r][sgn], e = s[r][sgn];
        vpp += g * 0.5 * (p.x * p.x + p.y * p.y - np);
        vee += g * 0.5 * (e.x * e.x + e.y * e.y - (n - np));
        vep += g * (p.x * e.x + p.y * e.y);
      }
  vpp = block_sum(vpp, sh);
  vep = block_sum(vep, sh);
  vee = block_sum(vee, sh);
  if (tid == 0) {
    double *o = part + ((long long)b * stride + blockIdx.y) * 3;
    o[0] = vpp;
    o[1] = vep;
    o[2] = vee;
  }
}

// The nearest-image erfc sums of one part of a configuration's pairs, grid (B, parts); part[b][first + blockIdx.y][3].
// Few walkers spread their pairs over the chip (an erfc pair costs about 100 FP64 instructions, 64 cycles a warp each).
__global__ void __launch_bounds__(kCbThreads)
    k_coul_real(int n, int dim, const double *__restrict__ x, double L, double kappa, int first, int nblk,
                double *__restrict__ part) {
  extern __shared__ double xw[];  // [n][dim], wrapped into [0, L)
  __shared__ double sh[32];
  const int b = blockIdx.x;
  const double *xb = x + (long long)b * n * dim;
  for (int k = threadIdx.x; k < n * dim; k += blockDim.x) xw[k] = xb[k] - L * floor(xb[k] / L);
  __syncthreads();
  const int np = n / 2;
  double vpp = 0, vep = 0, vee = 0;
  // pairs i < j without idle threads: n is even, so rows r and n - 1 - r of the triangle have n - 1 pairs together
  for (int k = blockIdx.y * blockDim.x + threadIdx.x; k < (n / 2) * (n - 1); k += gridDim.y * blockDim.x) {
    const int row = k / (n - 1), c = k % (n - 1);
    const bool upper = c < n - 1 - row;
    const int i = upper ? row : n - 1 - row, j = upper ? row + 1 + c : c + 1;
    double d2 = 0;
    for (int d = 0; d < dim; ++d) {
      double r = (xw[i * dim + d] - xw[j * dim + d]) / L;
      r -= rint(r);
      d2 += r * r;
    }
    const double dd = sqrt(d2);
    const double v = erfc(kappa * dd) / dd;
    if (j < np) vpp += v;
    else if (i >= np) vee += v;
    else vep += v;
  }
  vpp = block_sum(vpp, sh);
  vep = block_sum(vep, sh);
  vee = block_sum(vee, sh);
  if (threadIdx.x == 0) {
    double *o = part + ((long long)b * nblk + first + blockIdx.y) * 3;
    o[0] = vpp;
    o[1] = vep;
    o[2] = vee;
  }
}

// One warp per configuration: the sums over its parts and the constant terms.
__global__ void __launch_bounds__(32)
    k_coul_finish(int n, double L, double rs, double g0, const double *__restrict__ part, int nblk,
                  double *__restrict__ out) {
  const int b = blockIdx.x, np = n / 2;
  double vpp = 0, vep = 0, vee = 0;
  for (int k = threadIdx.x; k < nblk; k += 32) {
    const double *o = part + ((long long)b * nblk + k) * 3;
    vpp += o[0];
    vep += o[1];
    vee += o[2];
  }
  vpp = warp_sum(vpp);
  vep = warp_sum(vep);
  vee = warp_sum(vee);
  if (threadIdx.x == 0) {
    const double ne = n - np;
    const double f = 2.0 * rs / L;
    out[b * 3 + 0] = f * (vpp + 0.5 * np * (np - 1) * g0);
    out[b * 3 + 1] = -f * (vep + (double)np * ne * g0);
    out[b * 3 + 2] = f * (vee + 0.5 * ne * (ne - 1) * g0);
  }
}

}  // namespace hqcgb

// C ABI: potential_energy (hqc/pbc/potential.py:69-101) of B configurations
// x [B][n][dim] (device, rs units; first n/2 protons), box L (rs units), G
// [nG][dim] integer vectors (host), out [B][3] = (vpp, vep, vee) (device).
extern "C" int hqcgb_coulomb_energy(int B, int n, int dim, const double *x, double L, double rs,
                                    double kappa, int nG, const int *G, double *out, void *stream) {
  using namespace hqcgb;
  cudaStream_t st = (cudaStream_t)stream;
  try {
    HQ_REQUIRE(B >= 0 && n >= 2 && n % 2 == 0 && n <= kCbMaxParticles && (dim == 2 || dim == 3) &&
                   L > 0 && kappa > 0 && nG >= 0 && (nG == 0 || G) && x && out,
               "bad argument");
    int most = 0;
    for (int k = 0; k < nG; ++k) {
      int any = 0, top = 0;
      for (int d = 0; d < dim; ++d) {
        const int g = G[k * dim + d];
        any |= g;
        top = std::max(top, g < 0 ? (g == INT_MIN ? INT_MAX : -g) : g);
      }
      HQ_REQUIRE(top < 100000, "bad G");
      HQ_REQUIRE(any != 0, "G = 0 is not part of the reciprocal sum");
      most = std::max(most, top);
    }
    if (B == 0) return HQCGB_OK;
    HQ_STAGE(ST_EWALD, st);
    const bool columns = nG > 0 && most <= kMaxIndex;
    const int m1 = most + 1;
    // Runs of 8 gz a thread cost nG (1 + 1/8) multiply-adds a particle, runs
    // of 2 half as much again but four times the threads: the long runs once
    // they fill the chip.  Measured with 54 + 54 particles, nG = 14146:
    // 1 walker 389 (runs of 8) / 300 us (runs of 2), 64: 776 / 739,
    // 128: 1133 / 1223, 1024: 6314 / 7776.
    const int run = (long long)B * nG >= 1200000 ? 8 : 2;
    int n_items = 0;
    std::vector<CoulItem> items;
    std::vector<double> wt;
    if (columns) {
      // multiplicity of (gx, gy, +-|gz|) over the half space gx > 0, or gx = 0 and gy > 0, or gz > 0
      std::vector<double> cnt((size_t)m1 * (2 * m1 - 1) * m1 * 2, 0.0);
      auto slot = [&](int gx, int gy, int gz) { return (((size_t)gx * (2 * m1 - 1) + gy + most) * m1 + gz) * 2; };
      for (int k = 0; k < nG; ++k) {
        int gx = G[k * dim], gy = dim == 3 ? G[k * dim + 1] : 0, gz = G[k * dim + dim - 1];
        if (gx < 0 || (gx == 0 && (gy < 0 || (gy == 0 && gz < 0)))) gx = -gx, gy = -gy, gz = -gz;
        cnt[slot(gx, gy, std::abs(gz)) + (gz < 0)] += 1.0;
      }
      for (int gz0 = 0; gz0 < m1; gz0 += run)
        for (int gx = 0; gx < m1; ++gx)
          for (int gy = -most; gy <= most; ++gy) {
            const int end = std::min(gz0 + run, m1);
            const double *c = cnt.data() + slot(gx, gy, 0);
            if (std::all_of(c + 2 * gz0, c + 2 * end, [](double v) { return v == 0.0; })) continue;
            items.push_back({gx, gy, gz0, 0});
            wt.insert(wt.end(), c + 2 * gz0, c + 2 * end);
            wt.resize(items.size() * run * 2, 0.0);
          }
      n_items = (int)items.size();
    }
    const int nrecip = nG == 0 ? 0 : columns ? ceil_div(n_items, 128) : ceil_div(nG, kCbThreads);
    const int pairs = (n / 2) * (n - 1);
    const int nreal = std::min(ceil_div(pairs, kCbThreads), std::max(1, 152 * 8 / B)), nblk = nrecip + nreal;
    const size_t gbytes = columns ? (size_t)n_items * sizeof(CoulItem) : ((size_t)nG * dim * sizeof(int) + 15) / 16 * 16;
    StreamBuf blk(gbytes + (wt.size() + (size_t)B * nblk * 3) * sizeof(double), st);
    double *wtd = blk.as<double>(gbytes), *part = wtd + wt.size();
    const size_t smem = (size_t)n * dim * sizeof(double);
    if (columns) {
      CoulItem *it = blk.as<CoulItem>();
      HQ_CUDA(cudaMemcpyAsync(it, items.data(), items.size() * sizeof(CoulItem), cudaMemcpyHostToDevice, st));
      HQ_CUDA(cudaMemcpyAsync(wtd, wt.data(), wt.size() * sizeof(double), cudaMemcpyHostToDevice, st));
      k_coul_weights<<<ceil_div((long long)n_items * run, 128), 128, 0, st>>>(dim, kappa, it, n_items, run, wtd);
      HQ_LAUNCH_CHECK();
      const size_t tab = (size_t)kChunk * 3 * m1 * sizeof(double2);
      auto go = [&](auto kernel) {
        ensure_dyn_smem((const void *)kernel, tab);
        kernel<<<dim3(B, nrecip), 128, tab, st>>>(n, dim, x, L, it, n_items, m1, wtd, nblk, part);
        HQ_LAUNCH_CHECK();
      };
      if (run == 8) go(k_coul_recip<8>);
      else go(k_coul_recip<2>);
    } else if (nrecip > 0) {
      int *Gd = blk.as<int>();
      HQ_CUDA(cudaMemcpyAsync(Gd, G, (size_t)nG * dim * sizeof(int), cudaMemcpyHostToDevice, st));
      k_coul_recip_any<<<dim3(B, nrecip), kCbThreads, smem, st>>>(n, dim, x, L, Gd, nG, kappa, nblk, part);
      HQ_LAUNCH_CHECK();
    }
    const double g0 = dim == 3 ? -M_PI / (kappa * kappa) : -2.0 * std::sqrt(M_PI) / kappa;
    k_coul_real<<<dim3(B, nreal), kCbThreads, smem, st>>>(n, dim, x, L, kappa, nrecip, nblk, part);
    HQ_LAUNCH_CHECK();
    k_coul_finish<<<B, 32, 0, st>>>(n, L, rs, g0, part, nblk, out);
    HQ_LAUNCH_CHECK();
    HQ_CUDA(cudaStreamSynchronize(st));
    return HQCGB_OK;
  } catch (const Error &e) {
    set_error(e.msg);
    return e.status;
  } catch (const std::exception &e) {  // host memory for the columns
    set_error(e.what());
    return HQCGB_CUDA_ERROR;
  }
}
