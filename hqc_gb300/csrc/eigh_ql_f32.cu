// The FP32 Householder + implicit QL eigensolver over several SMs, for the
// refinement in eigh_mixed.cu, and the Householder reduction it shares with
// eigh_f32.cu.  The arithmetic of every element and the order of every sum are
// those of the one-block solver (eigh_fp64.cu with T = float), so the results
// are the same bits:
//
//  1. k_tridiag_cluster: a cluster of eight CTAs holds the rows of the matrix
//     in its shared memory (row r in CTA r mod 8); a step exchanges the next
//     column and the product A v through distributed shared memory, two cluster
//     barriers a step;
//  2. k_ql_rotations (one warp): the QL iteration on d and e alone, its Givens
//     rotations written down sweep by sweep by one lane (the search for a small
//     off-diagonal element over all 32);
//  3. k_ql_apply: the rotations on the eigenvector matrix, a thread per row;
//  4. k_ql_back: the reflectors, a warp per eigenvector;
//  5. k_ql_store: ascending order.
//
// What bounds it is the chain of stage 2, about 0.85 n^2 rotations of a square
// root and two divisions each; the block that generated a sweep used to wait
// for the same block to apply it.  n = 270: 25.7 -> 11.4 ms (8.9 of them stage 2;
// 11.8 where all lanes followed a sweep).
#include <cooperative_groups.h>

#include "common.cuh"
#include "eigh_tridiag.cuh"
#include "kernels.h"

namespace hqcgb {

namespace cg = cooperative_groups;

constexpr int kTcCtas = 8, kTcThreads = 512;
constexpr int kTcMax = kTcThreads;  // one element of a column a thread

bool tridiag_cluster_supported(int n) { return n <= kTcMax; }

// LOWER: only A's lower triangle is read and the matrix stays exactly
// symmetric (element (i, j), j > i, is computed as (j, i) is); otherwise both
// triangles are updated as they stand.  Outputs as k_tridiag_f32.
template <bool LOWER>
__global__ void __launch_bounds__(kTcThreads, 1)
    k_tridiag_cluster(int n, const float *__restrict__ A, float *__restrict__ dg, float *__restrict__ eg,
                      float *__restrict__ taug, float *__restrict__ hv) {
  extern __shared__ __align__(16) float csh[];
  cg::cluster_group cluster = cg::this_cluster();
  const int rank = (int)cluster.block_rank();
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  constexpr int nw = kTcThreads / 32;
  const int own = (n - rank + kTcCtas - 1) / kTcCtas;  // rows rank, rank + 8, ...
  float *x = csh, *p = x + n, *v = p + n, *rows = v + n;  // x, p: written by the whole cluster
  __shared__ float red[2][32];
  auto sum = [&](float s, int buf) {
    s = warp_sum(s);
    if (lane == 0) red[buf][warp] = s;
    __syncthreads();
    return warp_sum(lane < nw ? red[buf][lane] : 0.f);
  };
  float *xr[kTcCtas], *pr[kTcCtas];
#pragma unroll
  for (int c = 0; c < kTcCtas; ++c) {
    xr[c] = cluster.map_shared_rank(x, c);
    pr[c] = cluster.map_shared_rank(p, c);
  }
  for (int q = warp; q < own; q += nw) {
    const int r = rank + q * kTcCtas;
    for (int j = lane; j < n; j += 32) rows[q * n + j] = LOWER && j > r ? A[(long long)j * n + r] : A[(long long)r * n + j];
  }
  for (int i = tid; i + 1 < n; i += kTcThreads) x[i] = A[(long long)(i + 1) * n];
  cluster.sync();
  for (int k = 0; k < n - 2; ++k) {
    const int m = n - k - 1;  // trailing rows k+1 .. n-1
    float s2 = 0.f;
    if (1 + tid < m) s2 = x[1 + tid] * x[1 + tid];
    s2 = sum(s2, 0);
    const float x0 = x[0];
    float tk = 0.f, sc = 0.f, beta = x0;
    if (s2 != 0.f) {
      beta = -copysignf(sqrtf(x0 * x0 + s2), x0);
      tk = (beta - x0) / beta;
      sc = 1.f / (x0 - beta);
    }
    if (rank == 0 && tid == 0) {
      taug[k] = tk;
      eg[k] = beta;
    }
    if (tid < m) {
      const float vi = (tid == 0) ? 1.f : (tk == 0.f ? 0.f : x[tid] * sc);
      v[tid] = vi;
      if (rank == 0) hv[(long long)k * n + tid] = vi;
    }
    __syncthreads();
    // the first own row of the trailing block
    const int q0 = k + 1 <= rank ? 0 : (k + 1 - rank + kTcCtas - 1) / kTcCtas;
    if (tk != 0.f) {
      for (int q = q0 + warp; q < own; q += nw) {
        const float *row = rows + q * n + k + 1;
        float s = 0.f;
#pragma unroll 4
        for (int j = lane; j < m; j += 32) s += row[j] * v[j];
        s = tk * warp_sum(s);
        float *dst = pr[0];
#pragma unroll
        for (int c = 1; c < kTcCtas; ++c)
          if (lane == c) dst = pr[c];
        if (lane < kTcCtas) dst[rank + q * kTcCtas - k - 1] = s;
      }
      cluster.sync();
      float pv = 0.f;
      if (tid < m) pv = p[tid] * v[tid];
      pv = sum(pv, 1);
      const float alpha = -0.5f * tk * pv;
      if (tid < m) p[tid] += alpha * v[tid];  // p becomes w
      __syncthreads();
    } else {
      cluster.sync();  // x is read by all before the next column comes
    }
    for (int q = q0 + warp; q < own; q += nw) {
      float *row = rows + q * n + k + 1;
      const int i = rank + q * kTcCtas - k - 1;
      if (tk != 0.f) {
        const float vi = v[i], pi = p[i];
#pragma unroll 4
        for (int j = lane; j < m; j += 32) {
          const float vj = v[j], pj = p[j];
          // rounded as the one-block reductions round it
          if (LOWER && j > i) row[j] = __fsub_rn(row[j], __fmaf_rn(vj, pi, __fmul_rn(pj, vi)));
          else row[j] = __fsub_rn(row[j], __fmaf_rn(vi, pj, __fmul_rn(pi, vj)));
        }
        __syncwarp();
      }
      // element (i, 0) belongs to the next column
      if (i > 0 && lane < kTcCtas) {
        float *dst = xr[0];
#pragma unroll
        for (int c = 1; c < kTcCtas; ++c)
          if (lane == c) dst = xr[c];
        dst[i - 1] = row[0];
      }
    }
    cluster.sync();
  }
  for (int q = tid; q < own; q += kTcThreads) {
    const int r = rank + q * kTcCtas;
    dg[r] = rows[q * n + r];
  }
  if (rank == 0 && tid == 0) {
    if (n >= 2) {
      eg[n - 2] = x[0];
      taug[n - 2] = 0.f;
    }
    eg[n - 1] = 0.f;
    taug[n - 1] = 0.f;
  }
}

void tridiag_cluster(int n, bool lower, const float *A, float *dg, float *eg, float *taug, float *hv,
                     cudaStream_t st) {
  const size_t smem = ((size_t)3 * n + (size_t)ceil_div(n, kTcCtas) * n) * sizeof(float);
  auto go = [&](auto kernel) {
    ensure_dyn_smem((const void *)kernel, smem);
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3(kTcCtas);
    cfg.blockDim = dim3(kTcThreads);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim = {kTcCtas, 1, 1};
    cfg.attrs = at;
    cfg.numAttrs = 1;
    HQ_CUDA(cudaLaunchKernelEx(&cfg, kernel, n, A, dg, eg, taug, hv));
    count_launch();
  };
  if (lower) go(k_tridiag_cluster<true>);
  else go(k_tridiag_cluster<false>);
}

// Sweep s applies rotations [first, first + count) to columns m - 1 - t and
// m - t; info[0] = sweeps, info[1] = 1 when a limit was hit.
struct QlSweep {
  int m, first, count;
};
constexpr int kQlSweeps = 16, kQlRot = 4;  // capacity: sweeps per row, rotations per matrix element

__global__ void __launch_bounds__(32)
    k_ql_rotations(int n, const float *__restrict__ dg, const float *__restrict__ eg, float *__restrict__ dout,
                   float2 *__restrict__ rot, QlSweep *__restrict__ sweeps, int *__restrict__ info) {
  extern __shared__ __align__(16) float csh[];
  float *d = csh, *e = d + n;
  const int lane = threadIdx.x;
  for (int i = lane; i < n; i += 32) {
    d[i] = dg[i];
    e[i] = eg[i];
  }
  __syncwarp();
  const long long cap = (long long)kQlRot * n * n;
  int pos = 0, ns = 0, fail = 0;
  for (int l = 0; l < n && !fail; ++l) {
    int iter = 0;
    while (true) {
      int m = n - 1;
      for (int m0 = l; m0 < n - 1; m0 += 32) {
        const int q = m0 + lane;
        bool small = false;
        if (q < n - 1) {
          const float dd = fabsf(d[q]) + fabsf(d[q + 1]);
          small = fabsf(e[q]) <= EigEps<float>::v * dd;
        }
        const unsigned mask = __ballot_sync(0xffffffffu, small);
        if (mask) {
          m = m0 + __ffs(mask) - 1;
          break;
        }
      }
      if (m == l) break;
      if (iter++ >= 60 || pos + (m - l) > cap || ns >= kQlSweeps * n) {
        fail = 1;
        break;
      }
      // one sweep by the first lane alone: it reads d and e two elements ahead of
      // where it stores them, which no other lane may do unordered
      int nrot = 0;
      if (lane == 0) {
        float g = (d[l + 1] - d[l]) / (2.f * e[l]);
        float r = e_hypot(g, 1.f);
        g = d[m] - d[l] + e[l] / (g + e_copysign(r, g));
        float s = 1.f, c = 1.f, pp = 0.f;
        bool early = false;
        float ei = e[m - 1], di = d[m - 1], di1 = d[m];
        for (int i = m - 1; i >= l; --i) {
          const float en = i > l ? e[i - 1] : 0.f, dn = i > l ? d[i - 1] : 0.f;
          const float f = s * ei, b = c * ei;
          r = e_hypot(f, g);
          e[i + 1] = r;
          if (r == 0.f) {
            d[i + 1] = di1 - pp;
            e[m] = 0.f;
            early = true;
            break;
          }
          s = f / r;
          c = g / r;
          g = di1 - pp;
          r = __fmaf_rn(2.f * c, b, __fmul_rn(di - g, s));
          pp = s * r;
          d[i + 1] = g + pp;
          rot[pos + nrot] = make_float2(c, s);
          g = c * r - b;
          ++nrot;
          di1 = di;
          di = dn;
          ei = en;
        }
        if (!early) {
          d[l] = di1 - pp;
          e[l] = g;
          e[m] = 0.f;
        }
        sweeps[ns] = QlSweep{m, pos, nrot};
      }
      __syncwarp();  // d and e are read by all lanes again
      pos += __shfl_sync(0xffffffffu, nrot, 0);
      ++ns;
    }
  }
  __syncwarp();
  for (int i = lane; i < n; i += 32) dout[i] = d[i];
  if (lane == 0) {
    info[0] = ns;
    info[1] = fail;
  }
}

// Zt[c][r] = Z[r][c], Z the product of the rotations: a thread per row r, its
// row in shared memory, the rotations 32 at a time from a register a lane.
__global__ void __launch_bounds__(32)
    k_ql_apply(int n, const float2 *__restrict__ rot, const QlSweep *__restrict__ sweeps, const int *__restrict__ info,
               float *__restrict__ Zt) {
  extern __shared__ __align__(16) float csh[];  // [n][32]
  const int lane = threadIdx.x, r = blockIdx.x * 32 + lane;
  float *z = csh + lane;
  for (int c = 0; c < n; ++c) z[c * 32] = c == r ? 1.f : 0.f;
  const int ns = info[0];
  for (int q = 0; q < ns; ++q) {
    const QlSweep sw = sweeps[q];
    if (sw.count == 0) continue;
    float cur = z[sw.m * 32];
    for (int t0 = 0; t0 < sw.count; t0 += 32) {
      const float2 mine = t0 + lane < sw.count ? rot[sw.first + t0 + lane] : make_float2(1.f, 0.f);
#pragma unroll
      for (int h = 0; h < 32; h += 16) {
        float zi[16];
#pragma unroll
        for (int u = 0; u < 16; ++u)
          if (t0 + h + u < sw.count) zi[u] = z[(sw.m - 1 - t0 - h - u) * 32];
#pragma unroll
        for (int u = 0; u < 16; ++u) {
          const float c = __shfl_sync(0xffffffffu, mine.x, h + u), s = __shfl_sync(0xffffffffu, mine.y, h + u);
          if (t0 + h + u < sw.count) {
            z[(sw.m - t0 - h - u) * 32] = __fmaf_rn(c, cur, __fmul_rn(s, zi[u]));
            cur = __fmaf_rn(c, zi[u], -__fmul_rn(s, cur));
          }
        }
      }
    }
    z[(sw.m - sw.count) * 32] = cur;
  }
  if (r < n)
    for (int c = 0; c < n; ++c) Zt[(long long)c * n + r] = z[c * 32];
}

// Zt <- the reflectors H_k, k = n-3 .. 0, on every eigenvector: a warp each.
constexpr int kQlBackWarps = 8;
__global__ void __launch_bounds__(kQlBackWarps * 32)
    k_ql_back(int n, const float *__restrict__ hv, const float *__restrict__ tau, float *__restrict__ Zt) {
  extern __shared__ __align__(16) float csh[];  // [warps][n], then 2 [n]
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nt = kQlBackWarps * 32;
  const int col = blockIdx.x * kQlBackWarps + warp;
  float *z = csh + warp * n, *vb = csh + kQlBackWarps * n;
  if (col < n)
    for (int i = lane; i < n; i += 32) z[i] = Zt[(long long)col * n + i];
  for (int i = threadIdx.x; n >= 3 && i < 2; i += nt) vb[((n - 3) & 1) * n + i] = hv[(long long)(n - 3) * n + i];
  for (int k = n - 3; k >= 0; --k) {
    __syncthreads();
    constexpr int kFetch = kTcMax / (kQlBackWarps * 32);
    float next[kFetch];
    if (k > 0)
#pragma unroll
      for (int q = 0; q < kFetch; ++q)
        if (q * nt + (int)threadIdx.x < n - k) next[q] = hv[(long long)(k - 1) * n + q * nt + threadIdx.x];
    const float tk = tau[k];
    const int m = n - k - 1;
    const float *v = vb + (k & 1) * n;
    if (tk != 0.f && col < n) {
      float *zc = z + k + 1;
      float s = 0.f;
#pragma unroll 4
      for (int i = lane; i < m; i += 32) s += v[i] * zc[i];
      s = warp_sum(s);
      const float pc = tk * s;
#pragma unroll 4
      for (int i = lane; i < m; i += 32) zc[i] -= v[i] * pc;
    }
    if (k > 0)
#pragma unroll
      for (int q = 0; q < kFetch; ++q)
        if (q * nt + (int)threadIdx.x < n - k) vb[((k - 1) & 1) * n + q * nt + threadIdx.x] = next[q];
  }
  __syncwarp();
  if (col < n)
    for (int i = lane; i < n; i += 32) Zt[(long long)col * n + i] = z[i];
}

// Ascending: w, and V[r][rank] = Zt[c][r].  A block per eigenvector.
__global__ void __launch_bounds__(256)
    k_ql_store(int n, const float *__restrict__ d, const float *__restrict__ Zt, const int *__restrict__ info,
               float *__restrict__ V, float *__restrict__ w, int *__restrict__ status) {
  __shared__ int s_rank;
  const int c = blockIdx.x;
  if (threadIdx.x == 0) s_rank = 0;
  __syncthreads();
  const float lc = d[c];
  int r = 0;
  for (int j = threadIdx.x; j < n; j += 256) r += (d[j] < lc) || (d[j] == lc && j < c);
  atomicAdd(&s_rank, r);
  __syncthreads();
  const int rank = s_rank;
  if (threadIdx.x == 0) {
    w[rank] = lc;
    if (c == 0) *status = info[1] ? -1 : 0;
  }
  for (int i = threadIdx.x; i < n; i += 256) V[(long long)i * n + rank] = Zt[(long long)c * n + i];
}

size_t eigh_ql_f32_scratch_floats(int n) {
  if (!tridiag_cluster_supported(n)) return 0;
  return (size_t)n * n + 2 * (size_t)kQlRot * n * n + 3 * (size_t)kQlSweeps * n + 4 * (size_t)n + 16;
}

// A (n x n) -> w ascending, V columns; Zt: n x n scratch; status < 0 when a limit was hit.
void eigh_ql_f32(int n, const float *A, float *V, float *w, float *Zt, float *scr, int *status, cudaStream_t st) {
  HQ_STAGE(ST_JACOBI, st);
  HQ_REQUIRE((uintptr_t)scr % sizeof(float2) == 0, "QL scratch must be 8-byte aligned");
  float2 *rot = reinterpret_cast<float2 *>(scr);
  float *hv = scr + 2 * (size_t)kQlRot * n * n, *dg = hv + (size_t)n * n, *eg = dg + n, *taug = eg + n, *dout = taug + n;
  QlSweep *sweeps = reinterpret_cast<QlSweep *>(dout + n);
  int *info = reinterpret_cast<int *>(sweeps + (size_t)kQlSweeps * n);
  tridiag_cluster(n, false, A, dg, eg, taug, hv, st);
  k_ql_rotations<<<1, 32, 2 * n * sizeof(float), st>>>(n, dg, eg, dout, rot, sweeps, info);
  HQ_LAUNCH_CHECK();
  const size_t sma = (size_t)n * 32 * sizeof(float), smb = (size_t)(kQlBackWarps + 2) * n * sizeof(float);
  ensure_dyn_smem((const void *)k_ql_apply, sma);
  k_ql_apply<<<ceil_div(n, 32), 32, sma, st>>>(n, rot, sweeps, info, Zt);
  HQ_LAUNCH_CHECK();
  k_ql_back<<<ceil_div(n, kQlBackWarps), kQlBackWarps * 32, smb, st>>>(n, hv, taug, Zt);
  HQ_LAUNCH_CHECK();
  k_ql_store<<<n, 256, 0, st>>>(n, dout, Zt, info, V, w, status);
  HQ_LAUNCH_CHECK();
}

}  // namespace hqcgb
