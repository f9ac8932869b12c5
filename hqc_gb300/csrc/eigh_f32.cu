// FP32 stage of the mixed-precision eigensolver: eigenpairs of a symmetric
// n x n matrix to single precision, for the FP64 refinement in
// eigh_mixed.cu.  Three steps:
//
//  1. Householder reduction to tridiagonal T = Q^T A Q, reflectors stored
//     contiguously: up to 95 AOs one block with the lower triangle in shared
//     memory (k_tridiag_f32_smem), to 512 a cluster of eight SMs
//     (k_tridiag_cluster in eigh_ql_f32.cu), above one block on global memory
//     (k_tridiag_f32, the form of eigh_tridiag.cuh).
//  2. k_tri_values_f32 (a warp per eigenvalue): the eigenvalues of T by
//     bisection on Sturm counts (W. Barth, R. S. Martin, J. H.
//     Wilkinson, "Calculation of the eigenvalues of a symmetric tridiagonal
//     matrix by the method of bisection", Numer. Math. 9 (1967) 386-393), all
//     in parallel; k_tri_vectors_f32 (a warp per cluster): the eigenvectors of
//     T by inverse iteration with a partial-pivoting LU of T - lambda I (J. H.
//     Wilkinson, "The Algebraic Eigenvalue Problem", 1965, ch. 5), eigenvalues
//     closer than 1e-4 ||T|| treated as a cluster whose vectors one warp
//     computes in turn, orthogonalising each against the earlier ones (modified
//     Gram-Schmidt).
//  3. k_backtransform_f32 (a block per 32 columns): V = Q Z, the reflectors
//     applied in reverse order to column tiles held in shared memory.
//
// The serial QL sweep of the FP64 solver (thousands of dependent Givens
// rotations generated by one thread) is replaced by work that is parallel
// over eigenvalues; the FP64 refinement then fixes what single precision
// leaves (inaccurate vectors within clusters included).
#include <algorithm>
#include <cfloat>
#include <cstdio>
#include <cstdlib>

#include "common.cuh"
#include "eigh_tridiag.cuh"
#include "kernels.h"

namespace hqcgb {

constexpr int kTriThreads = 1024;

__global__ void __launch_bounds__(kTriThreads)
    k_tridiag_f32(int n, float *__restrict__ A, float *__restrict__ dg, float *__restrict__ eg,
                  float *__restrict__ taug, float *__restrict__ hv) {
  extern __shared__ __align__(16) float tsh[];
  float *d = tsh, *e = d + n, *tau = e + n, *v = tau + n, *p = v + n;
  __shared__ float red[32];
  __shared__ float s_dbl[4];
  householder_tridiag<float>(n, A, d, e, tau, v, p, red, s_dbl, hv);
  for (int i = threadIdx.x; i < n; i += blockDim.x) {
    dg[i] = d[i];
    eg[i] = e[i];
    taug[i] = tau[i];
  }
}

// The same reduction with the matrix held in shared memory as a packed lower
// triangle (element (i, j), i >= j, at i (i + 1) / 2 + j): the symmetric
// matrix-vector product and the rank-2 update of each step touch only shared
// memory.  Takes n with n (n + 1) / 2 + 5 n floats within the shared-memory
// budget (n <= 310).
__device__ inline int tri_ix(int i, int j) { return i * (i + 1) / 2 + j; }

// Bound by latency, not arithmetic: 270 dependent steps of one block.  So the
// block's sums take one barrier (every warp adds the warps' parts itself), the
// reflector's scalars are computed by every thread, and a warp works on four
// rows of the triangle at a time.  n = 270: 2.0 -> 1.57 ms.
constexpr int kTriSmemThreads = 1024;
constexpr int kTriRows = 4;  // rows a warp works on at a time
__global__ void __launch_bounds__(kTriSmemThreads)
    k_tridiag_f32_smem(int n, const float *__restrict__ A, float *__restrict__ dg,
                       float *__restrict__ eg, float *__restrict__ taug, float *__restrict__ hv) {
  extern __shared__ __align__(16) float tsh[];
  float *L = tsh, *d = L + n * (n + 1) / 2, *e = d + n, *tau = e + n, *v = tau + n, *p = v + n;
  __shared__ float red[2][32];
  const int tid = threadIdx.x, nt = blockDim.x, lane = tid & 31, warp = tid >> 5, nw = nt >> 5;
  // sum over the block, to every thread; `buf` alternates between calls
  auto sum = [&](float x, int buf) {
    x = warp_sum(x);
    if (lane == 0) red[buf][warp] = x;
    __syncthreads();
    return warp_sum(lane < nw ? red[buf][lane] : 0.f);
  };
  for (int i = warp; i < n; i += nw)
    for (int j = lane; j <= i; j += 32) L[tri_ix(i, j)] = A[(long long)i * n + j];
  __syncthreads();
  for (int k = 0; k < n - 2; ++k) {
    const int m = n - k - 1;  // trailing rows k+1 .. n-1
    float s2 = 0.f;
    for (int i = 1 + tid; i < m; i += nt) {
      float x = L[tri_ix(k + 1 + i, k)];
      s2 += x * x;
    }
    s2 = sum(s2, 0);
    const float x0 = L[tri_ix(k + 1, k)];
    float tk = 0.f, sc = 0.f, beta = x0;
    if (s2 != 0.f) {
      beta = -copysignf(sqrtf(x0 * x0 + s2), x0);
      tk = (beta - x0) / beta;
      sc = 1.f / (x0 - beta);
    }
    if (tid == 0) {
      tau[k] = tk;
      e[k] = beta;
    }
    for (int i = tid; i < m; i += nt) {
      v[i] = (i == 0) ? 1.f : (tk == 0.f ? 0.f : L[tri_ix(k + 1 + i, k)] * sc);
      hv[(long long)k * n + i] = v[i];
    }
    __syncthreads();
    if (tk == 0.f) continue;
    // p = tau A22 v, one warp per row i: sum over j <= i of L[i][j] v_j and
    // over j > i of L[j][i] v_j (trailing block indices)
    for (int i0 = warp; i0 < m; i0 += kTriRows * nw) {
      float acc[kTriRows];
#pragma unroll
      for (int r = 0; r < kTriRows; ++r) acc[r] = 0.f;
      for (int j = lane; j < m; j += 32) {
        const float vj = v[j];
        const int col = tri_ix(k + 1 + j, k + 1);
#pragma unroll
        for (int r = 0; r < kTriRows; ++r) {
          const int i = i0 + r * nw;
          if (i < m) acc[r] += L[j <= i ? tri_ix(k + 1 + i, k + 1) + j : col + i] * vj;
        }
      }
#pragma unroll
      for (int o = 16; o > 0; o >>= 1)
#pragma unroll
        for (int r = 0; r < kTriRows; ++r) acc[r] += __shfl_xor_sync(0xffffffffu, acc[r], o);
      if (lane == 0)
#pragma unroll
        for (int r = 0; r < kTriRows; ++r)
          if (i0 + r * nw < m) p[i0 + r * nw] = tk * acc[r];
    }
    __syncthreads();
    float pv = 0.f;
    for (int i = tid; i < m; i += nt) pv += p[i] * v[i];
    pv = sum(pv, 1);
    const float alpha = -0.5f * tk * pv;
    for (int i = tid; i < m; i += nt) p[i] += alpha * v[i];  // p becomes w
    __syncthreads();
    // rank-2 update of the trailing lower triangle
    for (int i0 = warp; i0 < m; i0 += kTriRows * nw) {
      const int last = min(m - 1, i0 + (kTriRows - 1) * nw);
      for (int j = lane; j <= last; j += 32) {
        const float vj = v[j], pj = p[j];
#pragma unroll
        for (int r = 0; r < kTriRows; ++r) {
          const int i = i0 + r * nw;
          if (i < m && j <= i) L[tri_ix(k + 1 + i, k + 1) + j] -= v[i] * pj + p[i] * vj;
        }
      }
    }
    __syncthreads();
  }
  for (int i = tid; i < n; i += nt) {
    dg[i] = L[tri_ix(i, i)];
    eg[i] = i < n - 2 ? e[i] : (i == n - 2 ? L[tri_ix(n - 1, n - 2)] : 0.f);
    taug[i] = i < n - 2 ? tau[i] : 0.f;
  }
}

// number of eigenvalues of the tridiagonal (d, e2 = e^2) below x
__device__ inline int sturm_count(int n, const float *__restrict__ d, const float *__restrict__ e2,
                                  float x, float pivmin) {
  float q = d[0] - x;
  if (fabsf(q) < pivmin) q = -pivmin;
  int c = q < 0.f;
  for (int k = 1; k < n; ++k) {
    q = (d[k] - x) - e2[k - 1] / q;
    if (fabsf(q) < pivmin) q = -pivmin;
    c += q < 0.f;
  }
  return c;
}

// Gershgorin interval [lo, hi] and the scales of the tridiagonal (d, e).
struct TriScale {
  float tnorm, pivmin, lo, hi;
};

// Eigenvalues of the tridiagonal, w ascending: a warp per eigenvalue and block
// (every block forms the interval from all of d and e).  A Sturm count is a
// chain of n divisions, so its length is what a bisection costs: speculating
// five halvings ahead takes a fifth of the chains.  n = 270: 0.47 -> 0.11 ms.
__global__ void __launch_bounds__(32)
    k_tri_values_f32(int n, const float *__restrict__ dg, const float *__restrict__ eg, float *__restrict__ w,
                     TriScale *__restrict__ scale) {
  extern __shared__ __align__(16) float ssh[];
  float *d = ssh, *e2 = d + n;
  float lo = FLT_MAX, hi = -FLT_MAX, emax2 = 0.f;
  for (int i = threadIdx.x; i < n; i += 32) {
    d[i] = dg[i];
    const float ei = i < n - 1 ? eg[i] : 0.f;
    e2[i] = ei * ei;
    float r = (i > 0 ? fabsf(eg[i - 1]) : 0.f) + (i < n - 1 ? fabsf(eg[i]) : 0.f);
    lo = fminf(lo, dg[i] - r);
    hi = fmaxf(hi, dg[i] + r);
    emax2 = fmaxf(emax2, e2[i]);
  }
  for (int o = 16; o > 0; o >>= 1) {
    lo = fminf(lo, __shfl_xor_sync(0xffffffffu, lo, o));
    hi = fmaxf(hi, __shfl_xor_sync(0xffffffffu, hi, o));
    emax2 = fmaxf(emax2, __shfl_xor_sync(0xffffffffu, emax2, o));
  }
  __syncwarp();
  const float tnorm = fmaxf(fabsf(lo), fabsf(hi));
  const float pivmin = FLT_MIN * fmaxf(1.f, emax2);
  // widen the Gershgorin interval so that both ends are strict bounds
  const float pad = 2.f * FLT_EPSILON * tnorm + 4.f * pivmin;
  lo -= pad;
  hi += pad;
  if (blockIdx.x == 0 && threadIdx.x == 0) *scale = TriScale{tnorm, pivmin, lo, hi};
  // eigenvalue i by bisection, count(lo) <= i < count(hi), five halvings a
  // round: lane l evaluates node l of the tree of midpoints (children of l: 2 l
  // below, 2 l + 1 above it), then the warp walks the path that the counts give
  const int i = blockIdx.x, lane = threadIdx.x;
  float a = lo, b = hi;
  for (int it = 0; it < 80;) {
    float la = a, lb = b;
    for (int bit = 30 - __clz(max(lane, 1)); bit >= 0; --bit) {
      const float mid = 0.5f * (la + lb);
      if ((lane >> bit) & 1) la = mid;
      else lb = mid;
    }
    const int above = sturm_count(n, d, e2, 0.5f * (la + lb), pivmin) <= i;
    const unsigned up = __ballot_sync(0xffffffffu, above);
    bool done = false;
    for (int node = 1; node < 32 && it < 80; ++it) {
      const float mid = 0.5f * (a + b);
      done = mid <= a || mid >= b || b - a <= 2.f * FLT_EPSILON * fmaxf(fabsf(a), fabsf(b)) + pivmin;
      if (done) break;
      const int right = (up >> node) & 1;
      if (right) a = mid;
      else b = mid;
      node = 2 * node + right;
    }
    if (done) break;
  }
  if (lane == 0) w[i] = 0.5f * (a + b);
}

// Eigenvectors of the tridiagonal by inverse iteration, Z[r][c] column c that
// of w[c]; the first member of each cluster computes the cluster's vectors in
// order.  A warp per leader and block: the solves are chains of dependent
// steps that every lane follows in shared memory (30 cycles a step where they
// took an L2 round trip), sums run in the same order from values that the lanes
// fetch 32 at a time, and what is independent is spread over the lanes.
// n = 270, with k_tri_values_f32: 2.15 -> 0.78 ms.
__global__ void __launch_bounds__(32)
    k_tri_vectors_f32(int n, const float *__restrict__ dg, const float *__restrict__ eg, const float *__restrict__ lam,
                      const TriScale *__restrict__ scale, float *__restrict__ Z) {
  extern __shared__ __align__(16) float ssh[];
  const int lane = threadIdx.x, i0 = blockIdx.x;
  float *d = ssh, *e = d + n, *u1 = e + n, *u2 = u1 + n, *u3 = u2 + n, *lm = u3 + n, *x = lm + n;
  unsigned *swap = reinterpret_cast<unsigned *>(x + n);  // bit k: rows k, k + 1 swapped
  const float tnorm = scale->tnorm, pivmin = scale->pivmin;
  // clusters: eigenvalues within 1e-4 ||T||; vectors of eigenvalues further
  // apart are orthogonal to FP32 eps ||T|| / gap <= 1e-3, which the FP64
  // refinement removes
  const float sep = 1e-4f * tnorm;
  const float tiny = FLT_EPSILON * tnorm + pivmin;
  if (i0 > 0 && lam[i0] - lam[i0 - 1] <= sep) return;
  for (int i = lane; i < n; i += 32) {
    d[i] = dg[i];
    e[i] = i < n - 1 ? eg[i] : 0.f;
  }
  __syncwarp();
  int i1 = i0;
  while (i1 + 1 < n && lam[i1 + 1] - lam[i1] <= sep) ++i1;
  float shift_prev = 0.f;
  for (int j = i0; j <= i1; ++j) {
    // equal eigenvalues in a cluster are separated a little so that the
    // solves differ (the Gram-Schmidt step makes the vectors orthogonal)
    float lj = lam[j];
    if (j > i0 && lj - shift_prev < 10.f * tiny) lj = shift_prev + 10.f * tiny;
    shift_prev = lj;
    // LU with partial pivoting of T - lj I (rows k, k+1 swapped when the
    // subdiagonal entry is the larger pivot); U has two superdiagonals
    float b = d[0] - lj, c = n > 1 ? e[0] : 0.f;
    unsigned bits = 0;
    for (int k = 0; k < n - 1; ++k) {
      const float a = e[k], bn = d[k + 1] - lj, cn = k + 1 < n - 1 ? e[k + 1] : 0.f;
      float p1, p2, p3, l;
      if (fabsf(b) >= fabsf(a)) {
        if (b == 0.f) b = tiny;
        l = a / b;
        p1 = b; p2 = c; p3 = 0.f;
        b = bn - l * c;
        c = cn;
      } else {
        l = b / a;
        p1 = a; p2 = bn; p3 = cn;
        b = c - l * bn;
        c = -l * cn;
        bits |= 1u << (k & 31);
      }
      if (lane == 0) {
        u1[k] = fabsf(p1) < tiny ? (p1 < 0.f ? -tiny : tiny) : p1;
        u2[k] = p2; u3[k] = p3; lm[k] = l;
        if ((k & 31) == 31 || k == n - 2) swap[k >> 5] = bits;
      }
      if ((k & 31) == 31) bits = 0;
    }
    if (lane == 0) u1[n - 1] = fabsf(b) < tiny ? (b < 0.f ? -tiny : tiny) : b;
    // start vector: deterministic, not orthogonal to any eigenvector in practice
    for (int k = lane; k < n; k += 32) x[k] = 1.f + 0.37f * __sinf(0.7f * (float)k + 1.3f * (float)j);
    __syncwarp();
    for (int it = 0; it < 3; ++it) {
      // L y = P x, by the first lane alone: it stores x[k] and reads x[k + 1]
      if (lane == 0) {
        float y = x[0];
        unsigned word = 0;
        for (int k = 0; k < n - 1; ++k) {
          if ((k & 31) == 0) word = swap[k >> 5];
          float x1 = x[k + 1];
          if ((word >> (k & 31)) & 1) {
            const float t = y;
            y = x1;
            x1 = t;
          }
          x1 -= lm[k] * y;
          x[k] = y;
          y = x1;
        }
        x[n - 1] = y;
      }
      __syncwarp();
      // U z = y
      float z1 = x[n - 1] / u1[n - 1], z2 = 0.f;
      __syncwarp();
      if (lane == 0) x[n - 1] = z1;
      if (n > 1) {
        z2 = z1;
        z1 = (x[n - 2] - u2[n - 2] * z2) / u1[n - 2];
        __syncwarp();
        if (lane == 0) x[n - 2] = z1;
      }
      for (int k = n - 3; k >= 0; --k) {
        const float z = (x[k] - u2[k] * z1 - u3[k] * z2) / u1[k];
        z2 = z1;
        z1 = z;
        __syncwarp();
        if (lane == 0) x[k] = z;
      }
      __syncwarp();
      // orthogonalise against the cluster's earlier vectors, normalise
      for (int q = i0; q < j; ++q) {
        float s = 0.f;
        for (int k0 = 0; k0 < n; k0 += 32) {
          const int k = k0 + lane;
          const float zv = k < n ? Z[(long long)k * n + q] : 0.f, xv = k < n ? x[k] : 0.f;
          const int cnt = min(32, n - k0);
          for (int l = 0; l < cnt; ++l)
            s += __shfl_sync(0xffffffffu, zv, l) * __shfl_sync(0xffffffffu, xv, l);
        }
        __syncwarp();
        for (int k = lane; k < n; k += 32) x[k] -= s * Z[(long long)k * n + q];
        __syncwarp();
      }
      float nrm = 0.f;
#pragma unroll 8
      for (int k = 0; k < n; ++k) nrm += x[k] * x[k];
      nrm = nrm > 0.f ? rsqrtf(nrm) : 0.f;
      __syncwarp();
      for (int k = lane; k < n; k += 32) x[k] *= nrm;
      __syncwarp();
    }
    for (int k = lane; k < n; k += 32) Z[(long long)k * n + j] = x[k];
    __syncwarp();
  }
}

// V = Q Z for 32 columns per block: Z tile in shared memory, reflectors
// H_k = I - tau_k v_k v_k^T (rows k+1..n-1) applied for k = n-3 .. 0; eight
// threads (one warp quarter) own a column.  The next reflector is on its way
// in registers while one is applied; rows of 36 floats keep the eight threads
// of four columns in different banks.  n = 270: 0.96 -> 0.27 ms.
constexpr int kBackLd = 36, kBackFetch = (kMaxNao + 255) / 256;
__global__ void __launch_bounds__(256)
    k_backtransform_f32(int n, const float *__restrict__ hv, const float *__restrict__ tau,
                        const float *__restrict__ Z, float *__restrict__ V) {
  extern __shared__ __align__(16) float zt[];  // [n][kBackLd], then 2 [n]
  float *vbuf = zt + n * kBackLd;
  const int c0 = blockIdx.x * 32;
  const int tid = threadIdx.x, cc = tid >> 3, part = tid & 7;
  for (int idx = tid; idx < n * 32; idx += blockDim.x) {
    int r = idx >> 5, c = idx & 31;
    zt[r * kBackLd + c] = (c0 + c < n) ? Z[(long long)r * n + c0 + c] : 0.f;
  }
  float next[kBackFetch], tnext = 0.f;
  auto fetch = [&](int k) {
#pragma unroll
    for (int q = 0; q < kBackFetch; ++q)
      if (q * 256 + tid < n - k - 1) next[q] = hv[(long long)k * n + q * 256 + tid];
    tnext = tau[k];
  };
  auto put = [&](int k) {
#pragma unroll
    for (int q = 0; q < kBackFetch; ++q)
      if (q * 256 + tid < n - k - 1) vbuf[(k & 1) * n + q * 256 + tid] = next[q];
  };
  float tk = 0.f;
  if (n >= 3) {
    fetch(n - 3);
    put(n - 3);
    tk = tnext;
  }
  for (int k = n - 3; k >= 0; --k) {
    __syncthreads();
    if (k > 0) fetch(k - 1);
    const int m = n - k - 1;
    const float *vk = vbuf + (k & 1) * n;
    float *z = zt + (k + 1) * kBackLd + cc;
    if (tk != 0.f) {
      float s = 0.f;
#pragma unroll 4
      for (int i = part; i < m; i += 8) s += vk[i] * z[i * kBackLd];
      s += __shfl_xor_sync(0xffffffffu, s, 1);
      s += __shfl_xor_sync(0xffffffffu, s, 2);
      s += __shfl_xor_sync(0xffffffffu, s, 4);
      s *= tk;
#pragma unroll 4
      for (int i = part; i < m; i += 8) z[i * kBackLd] -= s * vk[i];
    }
    if (k > 0) put(k - 1);
    tk = tnext;
  }
  __syncthreads();
  for (int idx = tid; idx < n * 32; idx += blockDim.x) {
    int r = idx >> 5, c = idx & 31;
    if (c0 + c < n) V[(long long)r * n + c0 + c] = zt[r * kBackLd + c];
  }
}

size_t eigh_f32_scratch_floats(int n) {
  return std::max((size_t)n * n + 4 * (size_t)n + 8, eigh_ql_f32_scratch_floats(n));
}

// From this size on the reduction runs on a cluster of eight SMs: below it a
// step's arithmetic takes less than its two cluster barriers, and seven SMs
// are better left to other streams.  One block / cluster, the reduction at
// n = 270: 1.57 / 0.70 ms; whole solves at 64: 0.68 / 0.67, 128: 1.25 / 1.16,
// 190: 2.40 / 2.08.
constexpr int kClusterN = 96;

// A (n x n, destroyed) -> w ascending, V columns.  scr: eigh_f32_scratch_floats(n).
void eigh_f32(int n, float *A, float *V, float *w, float *scr, cudaStream_t st) {
  HQ_STAGE(ST_JACOBI, st);
  float *hv = scr, *dg = hv + (size_t)n * n, *eg = dg + n, *taug = eg + n;
  TriScale *scale = reinterpret_cast<TriScale *>(taug + n);
  size_t sm1 = (size_t)5 * n * sizeof(float);
  size_t sm2 = (size_t)(7 * n + (n + 31) / 32) * sizeof(float);
  size_t sm3 = (size_t)n * (kBackLd + 2) * sizeof(float);
  HQ_REQUIRE(sm3 <= 200 * 1024, "matrix too large for the FP32 eigensolver");
  ensure_dyn_smem((const void *)k_backtransform_f32, sm3);
  const bool tr = std::getenv("HQCGB_TRACE") != nullptr;
  cudaEvent_t ev[4];
  if (tr)
    for (auto &x : ev) cudaEventCreate(&x);
  if (tr) cudaEventRecord(ev[0], st);
  const size_t smt = ((size_t)n * (n + 1) / 2 + 5 * (size_t)n) * sizeof(float);
  if (n >= kClusterN && tridiag_cluster_supported(n)) {
    // one block keeps the lower triangle where it fits its shared memory, both triangles in global memory above
    tridiag_cluster(n, smt <= 200 * 1024, A, dg, eg, taug, hv, st);
  } else if (smt <= 200 * 1024) {
    ensure_dyn_smem((const void *)k_tridiag_f32_smem, smt);
    k_tridiag_f32_smem<<<1, kTriSmemThreads, smt, st>>>(n, A, dg, eg, taug, hv);
  } else {
    k_tridiag_f32<<<1, kTriThreads, sm1, st>>>(n, A, dg, eg, taug, hv);
  }
  HQ_LAUNCH_CHECK();
  if (tr) cudaEventRecord(ev[1], st);
  // Z (tridiagonal eigenvectors) goes to V, then V = Q Z in place per tile
  k_tri_values_f32<<<n, 32, 2 * n * sizeof(float), st>>>(n, dg, eg, w, scale);
  HQ_LAUNCH_CHECK();
  k_tri_vectors_f32<<<n, 32, sm2, st>>>(n, dg, eg, w, scale, V);
  HQ_LAUNCH_CHECK();
  if (tr) cudaEventRecord(ev[2], st);
  k_backtransform_f32<<<ceil_div(n, 32), 256, sm3, st>>>(n, hv, taug, V, V);
  HQ_LAUNCH_CHECK();
  if (tr) {
    cudaEventRecord(ev[3], st);
    cudaEventSynchronize(ev[3]);
    float t[3];
    for (int k = 0; k < 3; ++k) cudaEventElapsedTime(&t[k], ev[k], ev[k + 1]);
    fprintf(stderr, "  fp32 tridiag %.3f ms, bisection+inverse iteration %.3f ms, back %.3f ms\n", t[0],
            t[1], t[2]);
    for (auto &x : ev) cudaEventDestroy(x);
  }
}

}  // namespace hqcgb
