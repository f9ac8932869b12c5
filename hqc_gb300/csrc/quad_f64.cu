// FP64 grid contractions M_pq = sum_g A_p(g) B_q(g) on the tensor cores (the
// Fock quadratures and the exchange Gram of the FP64 path, hqc/pbc/solver.py:
// 592-629, 680-694).
//
// GB300 issues 2 FP64 multiply-adds a cycle and SM, its tensor cores 4096 of
// bf16, so FP64 operands are cut into integers that bf16 products add exactly
// (K. Ozaki, T. Ogita, S. Oishi, S. M. Rump, "Error-free transformations of
// matrix multiplication by using fast routines of matrix multiplication and
// its applications", Numer. Algorithms 59 (2012) 95-118):
//   x = 2^e sum_s d_s 128^-(s + 1),  s = 0..7, d_s integers in [-64, 64],
// with one power of two e for a row, |x| <= 2^(e - 1): 56 bits below the row's
// largest element, where FP64 keeps 53.  A product of digits is at most 2^12,
// so 512 points of the at most 8 products s + t = d fit FP32's 24 bits and the
// sums P_d (kind::f16, FP32 accumulators in TMEM, one per d = 0..7) are exact;
// the 36 products with s + t <= 7 are formed, the others are below 2^-56 of
// the row maxima's product.  The drains add the P_d to integers of 64 bits, so
// a CTA's share of the sum has one rounding, and the result's error is that of
// the digits: a rounding of 2^-57 of a row's maximum a point, which averages
// out, against the rounding of every FP64 product and partial sum before.
//
// Operands are stored by blocks of 32 points, [block][row block][pair][row]
// [128 bytes]: a 128-byte row holds 32 points of two digits, already in the
// K-major SW128 pattern that the MMA reads, so plain bulk copies fill the
// ring.  One CTA an SM: a persistent share of the points for one 128 x 64
// destination tile, a copy thread, an MMA thread and eight drain warps.
//
// Bounds.  One 32-point stage is 72 MMAs of 128 x 64 x 16: the kernel is bound
// by the tensor pipe, at 36 products a term.  Measured, digits
// of the weighted operand and sums included, FP64 pipe -> this: 64 AOs and 65^3
// points 2.24 -> 0.24 ms, 70 AOs and 49^3 points with the gradient term 2.21 ->
// 0.31 ms, 8 AOs and 41^3 points 0.57 -> 0.12 ms.
#include <algorithm>
#include <cmath>

#include "digits.cuh"
#include "kernels.h"

namespace hqcgb {

using namespace tc;

constexpr int kQfK = 32;                                // points per stage
constexpr int kQfChain = 16;                            // stages per TMEM sum (512 points)
constexpr int kQfM = 128, kQfN = 64;
constexpr int kQfRing = 2;
constexpr uint32_t kQfPairA = kQfM * 128, kQfPairB = kQfN * 128;
constexpr uint32_t kQfOffB = kQfPairs * kQfPairA;
constexpr uint32_t kQfStage = kQfPairs * (kQfPairA + kQfPairB);
constexpr size_t kQfSmem = kQfRing * kQfStage + 1024;   // + alignment to the swizzle atom
constexpr int kQfDrainWarps = 8;
constexpr int kQfThreads = (kQfDrainWarps + 2) * 32;
constexpr int kQfMaxTiles = (kMaxNao / kQfM) * (kMaxNao / kQfN);
constexpr int kQfBlk = 512;                             // points per entry of the maxima tables
static_assert(kQfSmem <= 227 * 1024, "FP64 quadrature ring above 227 KB");

int quad64_rows(int n) { return n <= 128 ? (n + 7) / 8 * 8 : 128; }
int quad64_row_blocks(int n) { return n <= 128 ? 1 : ceil_div(n, 128); }
size_t quad64_operand_bytes(int n, long long N) {
  return (size_t)ceil_div(N, kQfK) * quad64_row_blocks(n) * quad64_rows(n) * 128 * kQfPairs;
}
long long quad64_table(long long N) { return ceil_div(N, kQfBlk); }

static int quad64_tiles(int n, bool sym, unsigned char (*t)[2] = nullptr) {
  int cnt = 0;
  for (int m = 0; m * kQfM < n; ++m)
    for (int c = 0; c * kQfN < n; ++c) {
      if (sym && (c + 1) * kQfN <= m * kQfM) continue;  // below the diagonal
      if (t) {
        t[cnt][0] = (unsigned char)m;
        t[cnt][1] = (unsigned char)c;
      }
      ++cnt;
    }
  return cnt;
}
static int quad64_groups(int n, bool sym) { return std::max(1, 152 / quad64_tiles(n, sym)); }
size_t quad64_partial_doubles(int n) {
  size_t most = 0;
  for (int sym = 0; sym < 2; ++sym)
    most = std::max(most, (size_t)quad64_groups(n, sym) * quad64_tiles(n, sym) * kQfM * kQfN);
  return most;
}

// tab[row][block] = max |X[row][g]| over the block's points, rounded up to
// FP32; NaN and infinity compare above every number by their bits.
__global__ void __launch_bounds__(128)
    k_qf_maxima(const double *__restrict__ X, long long N, float *__restrict__ tab) {
  __shared__ unsigned s[4];
  const long long g0 = (long long)blockIdx.x * kQfBlk;
  const double *row = X + (long long)blockIdx.y * N;
  unsigned v = 0;
  for (int i = threadIdx.x; i < kQfBlk; i += 128)
    if (g0 + i < N) v = max(v, __float_as_uint(__double2float_ru(fabs(row[g0 + i]))));
  v = __reduce_max_sync(0xffffffffu, v);
  if ((threadIdx.x & 31) == 0) s[threadIdx.x >> 5] = v;
  __syncthreads();
  if (threadIdx.x == 0)
    tab[(long long)blockIdx.y * gridDim.x + blockIdx.x] =
        __uint_as_float(max(max(s[0], s[1]), max(s[2], s[3])));
}

// Exponent and scale of every row: the largest |X| (w NULL), |w X| or, with
// dtab and u, |0.5 w X + dV sum_c u_c dX_c| that the tables allow.  A row that
// is not finite gets a NaN scale.
__global__ void __launch_bounds__(128)
    k_qf_exponents(const float *__restrict__ tab, const float *__restrict__ dtab, int n, int nb,
                   const float *__restrict__ w, const float *__restrict__ u, float dV, int *__restrict__ e,
                   double *__restrict__ scale) {
  __shared__ unsigned s[4];
  const int p = blockIdx.x;
  unsigned v = 0;
  for (int b = threadIdx.x; b < nb; b += 128) {
    float m = tab[(long long)p * nb + b];
    if (w) m = __fmul_ru(m, w[b]);
    if (dtab) {
      m *= 0.5f;
      for (int c = 0; c < 3; ++c)
        m = __fmaf_ru(__fmul_ru(dV, u[c * nb + b]), dtab[((long long)c * n + p) * nb + b], m);
    }
    v = max(v, __float_as_uint(m) & 0x7fffffffu);
  }
  v = __reduce_max_sync(0xffffffffu, v);
  if ((threadIdx.x & 31) == 0) s[threadIdx.x >> 5] = v;
  __syncthreads();
  if (threadIdx.x == 0) {
    const float m = __uint_as_float(max(max(s[0], s[1]), max(s[2], s[3])));
    int k = 0;
    if (m > 0.f && m < INFINITY) frexpf(m, &k);  // m < 2^k
    e[p] = k + 1;
    scale[p] = m < INFINITY ? scalbn(1.0, k + 1) : NAN;
  }
}

// Digits of X (MODE 0), w X (1) or 0.5 w X + dV u.dX (2) into the operand
// layout; blockIdx.x = block of 32 points, a warp takes 8 rows x 4 chunks of
// 8 points.  Points beyond N become zeros; rows beyond n are left alone (they
// only reach destination rows and columns that nothing reads).
template <int MODE>
__global__ void __launch_bounds__(256)
    k_qf_digits(const double *__restrict__ X, const double *__restrict__ dX, const double *__restrict__ w,
                const double *__restrict__ u, double dV, int n, long long N, int rb, int rbn,
                const int *__restrict__ e, char *__restrict__ out) {
  const int lane = threadIdx.x & 31, c = lane & 3;
  const long long kb = blockIdx.x, g0 = kb * kQfK + c * 8;
  const int cnt = (int)min(8LL, max(0LL, N - g0));
  double wv[MODE ? 8 : 1], uv[MODE == 2 ? 24 : 1];
  if (MODE)
#pragma unroll
    for (int i = 0; i < 8; ++i) wv[i] = i < cnt ? w[g0 + i] * (MODE == 2 ? 0.5 : 1.0) : 0.0;
  if (MODE == 2)
#pragma unroll
    for (int d = 0; d < 3; ++d)
#pragma unroll
      for (int i = 0; i < 8; ++i) uv[d * 8 + i] = i < cnt ? dV * u[(long long)d * N + g0 + i] : 0.0;
  for (int p = (threadIdx.x >> 5) * 8 + (lane >> 2); p < n; p += 64) {
    const int ep = e[p];
    QfPack pack;
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      double x = 0.0;
      if (i < cnt) {
        const long long at = (long long)p * N + g0 + i;
        x = X[at];
        if (MODE) x *= wv[i];
        if (MODE == 2)
#pragma unroll
          for (int d = 0; d < 3; ++d) x += uv[d * 8 + i] * dX[(long long)d * n * N + at];
      }
      pack.put(i, x, ep);
    }
    char *row = out + ((kb * rbn + p / rb) * kQfPairs * (long long)rb + p % rb) * 128;
    const int r = p % rb;
    pack.store(row, (long long)rb * 128, c, r);
  }
}

struct QfArgs {
  const char *A, *B;
  double *part;  // [group][tile][128][64]
  int *err;
  long long stages;
  int n, rb, rbn, groups, tiles;
  unsigned char tile[kQfMaxTiles][2];  // 128-row block of A, 64-row block of B
};

struct QfPipe {
  uint64_t full[kQfRing], empty[kQfRing], acc_full, acc_empty;
  uint32_t tmem_base;
};

__global__ void __launch_bounds__(kQfThreads, 1) k_qf_gemm(const __grid_constant__ QfArgs a) {
  extern __shared__ __align__(1024) char smraw[];
  char *sm = (char *)(((uintptr_t)smraw + 1023) & ~(uintptr_t)1023);
  __shared__ QfPipe P;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int tile = blockIdx.x, g = blockIdx.y;
  const int mt = a.tile[tile][0], ct = a.tile[tile][1];
  const long long s0 = a.stages * g / a.groups;
  const int nst = (int)(a.stages * (g + 1) / a.groups - s0);
  const int nchain = (nst + kQfChain - 1) / kQfChain;
  const int rows_b = min(kQfN, a.n - ct * kQfN);            // columns that are read
  const int nn = (rows_b + 15) / 16 * 16;                   // MMA N
  if (tid == 0) {
    for (int b = 0; b < kQfRing; ++b) {
      mbar_init(&P.full[b], 1);
      mbar_init(&P.empty[b], 1);
    }
    mbar_init(&P.acc_full, 1);
    mbar_init(&P.acc_empty, kQfDrainWarps * 32);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == kQfDrainWarps) tmem_alloc(&P.tmem_base, kQfDigits * kQfN);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();

  bool ok = true;
  if (warp == kQfDrainWarps + 1) {
    if (lane == 0) {
      // rows of A's block and of B's, in steps of 8 (the swizzle's period), within the stored block
      const int brow = ct * kQfN, bblk = brow / a.rb, boff = brow % a.rb;
      const uint32_t na = (uint32_t)min(a.rb, (a.n - mt * kQfM + 7) / 8 * 8) * 128u;
      const uint32_t nb = (uint32_t)min(a.rb - boff, (rows_b + 7) / 8 * 8) * 128u;
      const long long pair = (long long)a.rb * 128, blk = kQfPairs * pair;
      for (int st = 0; st < nst; ++st) {
        const int slot = st % kQfRing, use = st / kQfRing;
        if (use > 0 && !mbar_wait(&P.empty[slot], (unsigned)((use - 1) & 1), a.err, 61)) {
          ok = false;
          break;
        }
        mbar_expect_tx(&P.full[slot], kQfPairs * (na + nb));
        const uint32_t dst = smem_u32(sm + slot * kQfStage);
        const char *srcA = a.A + ((s0 + st) * a.rbn + mt) * blk;
        const char *srcB = a.B + ((s0 + st) * a.rbn + bblk) * blk + (long long)boff * 128;
        for (int q = 0; q < kQfPairs; ++q) {
          bulk_copy(dst + q * kQfPairA, srcA + q * pair, na, &P.full[slot]);
          bulk_copy(dst + kQfOffB + q * kQfPairB, srcB + q * pair, nb, &P.full[slot]);
        }
      }
    }
  } else if (warp == kQfDrainWarps) {
    if (lane == 0) {
      // kind::f16, D = F32, A = B = BF16, both K-major
      const uint32_t idesc = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(nn >> 3) << 17) |
                             ((uint32_t)(kQfM >> 4) << 24);
      for (int j = 0, st = 0; j < nchain && ok; ++j) {
        if (j > 0 && !mbar_wait(&P.acc_empty, (unsigned)((j - 1) & 1), a.err, 64)) ok = false;
        tc_fence_after();
        const int end = min(nst, (j + 1) * kQfChain);
        bool first = true;
        for (; st < end && ok; ++st) {
          const int slot = st % kQfRing, use = st / kQfRing;
          if (!mbar_wait(&P.full[slot], (unsigned)(use & 1), a.err, 62)) ok = false;
          tc_fence_after();
          if (ok) {
            const uint64_t dA = sdesc(smem_u32(sm + slot * kQfStage)), dB = dA + (kQfOffB >> 4);
#pragma unroll 1
            for (int ks = 0; ks < kQfK / 16; ++ks) {
#pragma unroll
              for (int s = 0; s < kQfDigits; ++s) {
                // digit s: pair s / 2, half a 128-byte row (4 units of 16 bytes) each, 2 units a K step
                const uint64_t da = dA + (uint32_t)((s >> 1) * (kQfPairA >> 4) + (s & 1) * 4 + 2 * ks);
#pragma unroll
                for (int t = 0; t < kQfDigits - s; ++t)
                  mma_bf16(P.tmem_base + (s + t) * kQfN, da,
                           dB + (uint32_t)((t >> 1) * (kQfPairB >> 4) + (t & 1) * 4 + 2 * ks), idesc,
                           !(first && ks == 0 && s == 0));
              }
            }
            first = false;
          }
          mma_commit(&P.empty[slot]);
        }
        mma_commit(&P.acc_full);
      }
    }
  } else {
    // warp w owns TMEM lanes 32 (w % 4) .. and columns 32 (w / 4) .. + 31 of every P_d
    const int c0 = (warp >> 2) * 32;
    const uint32_t base = P.tmem_base + ((uint32_t)((warp & 3) * 32) << 16) + c0;
    long long hi[32], lo[32];  // sum_d P_d 128^(3 - d), d < 4, and the same of d - 4
#pragma unroll
    for (int i = 0; i < 32; ++i) hi[i] = lo[i] = 0;
    for (int j = 0; j < nchain; ++j) {
      if (ok && !mbar_wait(&P.acc_full, (unsigned)(j & 1), a.err, 63)) ok = false;
      tc_fence_after();
      if (ok) {
#pragma unroll
        for (int q = 0; q < 8; ++q) {
          uint32_t v[kQfDigits][4];
#pragma unroll
          for (int d = 0; d < kQfDigits; ++d) tmem_ld4_nowait(base + d * kQfN + q * 4, v[d]);
          tmem_wait_ld();
#pragma unroll
          for (int i = 0; i < 4; ++i)
#pragma unroll
            for (int d = 0; d < 4; ++d) {
              hi[q * 4 + i] += (long long)__float2int_rn(__uint_as_float(v[d][i])) * (1 << (7 * (3 - d)));
              lo[q * 4 + i] += (long long)__float2int_rn(__uint_as_float(v[d + 4][i])) * (1 << (7 * (3 - d)));
            }
        }
      }
      tc_fence_before();
      mbar_arrive(&P.acc_empty);
    }
    const int row = (warp & 3) * 32 + lane;
    if (ok && mt * kQfM + row < a.n) {
      double *out = a.part + (((long long)g * a.tiles + tile) * kQfM + row) * kQfN + c0;
#pragma unroll
      for (int i = 0; i < 32; ++i)
        if (c0 + i < rows_b) out[i] = fma((double)lo[i], 0x1p-28, (double)hi[i]);
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == kQfDrainWarps) {
    tc_fence_after();
    tmem_dealloc(P.tmem_base, kQfDigits * kQfN);
  }
}

// M (+)= scale 2^(eA + eB) 2^-35 sum over groups; sym: (p, q) from the upper
// triangle; tr: M_pq = v_pq + v_qp.  A block takes 32 columns of a row, eight
// threads a value.
__global__ void __launch_bounds__(256)
    k_qf_reduce(const __grid_constant__ QfArgs a, int sym, int tr, double scale, const double *__restrict__ sA,
                const double *__restrict__ sB, int accumulate, double *__restrict__ M) {
  __shared__ double sh[8][33];
  const int p = blockIdx.y, q = blockIdx.x * 32 + (threadIdx.x & 31), part = threadIdx.x >> 5;
  auto value = [&](int r, int c) {
    const int mt = r / kQfM, ct = c / kQfN;
    int t = 0;
    while (t < a.tiles && (a.tile[t][0] != mt || a.tile[t][1] != ct)) ++t;
    const double *src = a.part + ((long long)t * kQfM + r % kQfM) * kQfN + c % kQfN;
    double s = 0;
    for (int g = part; g < a.groups; g += 8) s += src[(long long)g * a.tiles * kQfM * kQfN];
    return s * sA[r] * sB[c];
  };
  double s = 0;
  if (q < a.n) {
    s = sym && q < p ? value(q, p) : value(p, q);
    if (tr) s += value(q, p);
  }
  sh[part][threadIdx.x & 31] = s;
  __syncthreads();
  if (part == 0 && q < a.n) {
    for (int k = 1; k < 8; ++k) s += sh[k][threadIdx.x];
    s *= 0x1p-35 * scale;
    double *m = M + (long long)p * a.n + q;
    *m = accumulate ? *m + s : s;
  }
}

static void maxima(const double *X, int rows, long long N, float *tab, cudaStream_t st) {
  k_qf_maxima<<<dim3((unsigned)quad64_table(N), rows), 128, 0, st>>>(X, N, tab);
  HQ_LAUNCH_CHECK();
}

static void product(const Quad64 &q, const char *A, const char *B, const double *sA, const double *sB, long long N,
                    bool sym, bool tr, double scale, bool accumulate, double *M, cudaStream_t st) {
  QfArgs a{};
  a.A = A;
  a.B = B;
  a.part = q.part;
  a.err = q.err;
  a.stages = ceil_div(N, kQfK);
  a.n = q.n;
  a.rb = quad64_rows(q.n);
  a.rbn = quad64_row_blocks(q.n);
  a.tiles = quad64_tiles(q.n, sym, a.tile);
  a.groups = quad64_groups(q.n, sym);
  ensure_dyn_smem((const void *)k_qf_gemm, kQfSmem);
  k_qf_gemm<<<dim3(a.tiles, a.groups), kQfThreads, kQfSmem, st>>>(a);
  HQ_LAUNCH_CHECK();
  k_qf_reduce<<<dim3(ceil_div(q.n, 32), q.n), 256, 0, st>>>(a, sym, tr, scale, sA, sB, accumulate, M);
  HQ_LAUNCH_CHECK();
}

void quad64_basis(const Quad64 &q, const double *phi, const double *dphi, long long N, cudaStream_t st) {
  HQ_STAGE(ST_SPLIT, st);
  const int nb = (int)quad64_table(N), rb = quad64_rows(q.n), rbn = quad64_row_blocks(q.n);
  maxima(phi, q.n, N, q.tab, st);
  if (dphi) maxima(dphi, 3 * q.n, N, q.tab + (size_t)q.n * nb, st);
  k_qf_exponents<<<q.n, 128, 0, st>>>(q.tab, nullptr, q.n, nb, nullptr, nullptr, 0.f, q.eB, q.sB);
  HQ_LAUNCH_CHECK();
  k_qf_digits<0><<<ceil_div(N, kQfK), 256, 0, st>>>(phi, nullptr, nullptr, nullptr, 0.0, q.n, N, rb, rbn, q.eB, q.B);
  HQ_LAUNCH_CHECK();
}

void quad64_weighted(const Quad64 &q, const double *phi, const double *w, long long N, double scale, double *M,
                     cudaStream_t st) {
  HQ_STAGE(ST_QUAD, st);
  if (!w) {
    product(q, q.B, q.B, q.sB, q.sB, N, true, false, scale, false, M, st);
    return;
  }
  const int nb = (int)quad64_table(N), rb = quad64_rows(q.n), rbn = quad64_row_blocks(q.n);
  maxima(w, 1, N, q.wtab, st);
  k_qf_exponents<<<q.n, 128, 0, st>>>(q.tab, nullptr, q.n, nb, q.wtab, nullptr, 0.f, q.eA, q.sA);
  HQ_LAUNCH_CHECK();
  k_qf_digits<1><<<ceil_div(N, kQfK), 256, 0, st>>>(phi, nullptr, w, nullptr, 0.0, q.n, N, rb, rbn, q.eA, q.A);
  HQ_LAUNCH_CHECK();
  product(q, q.A, q.B, q.sA, q.sB, N, true, false, scale, false, M, st);
}

void quad64_gga(const Quad64 &q, const double *phi, const double *dphi, const double *w, const double *u, double dV,
                long long N, double *M, cudaStream_t st) {
  HQ_STAGE(ST_QUAD, st);
  const int nb = (int)quad64_table(N), rb = quad64_rows(q.n), rbn = quad64_row_blocks(q.n);
  maxima(w, 1, N, q.wtab, st);
  maxima(u, 3, N, q.wtab + nb, st);
  k_qf_exponents<<<q.n, 128, 0, st>>>(q.tab, q.tab + (size_t)q.n * nb, q.n, nb, q.wtab, q.wtab + nb,
                                      std::nextafter((float)dV, INFINITY), q.eA, q.sA);
  HQ_LAUNCH_CHECK();
  k_qf_digits<2><<<ceil_div(N, kQfK), 256, 0, st>>>(phi, dphi, w, u, dV, q.n, N, rb, rbn, q.eA, q.A);
  HQ_LAUNCH_CHECK();
  product(q, q.A, q.B, q.sA, q.sB, N, false, true, 1.0, false, M, st);
}

void quad64_gram(const Quad64 &q, const double *Q, long long N, bool accumulate, double *M, cudaStream_t st) {
  HQ_STAGE(ST_QUAD, st);
  const int nb = (int)quad64_table(N), rb = quad64_rows(q.n), rbn = quad64_row_blocks(q.n);
  maxima(Q, q.n, N, q.xtab, st);
  k_qf_exponents<<<q.n, 128, 0, st>>>(q.xtab, nullptr, q.n, nb, nullptr, nullptr, 0.f, q.eA, q.sA);
  HQ_LAUNCH_CHECK();
  k_qf_digits<0><<<ceil_div(N, kQfK), 256, 0, st>>>(Q, nullptr, nullptr, nullptr, 0.0, q.n, N, rb, rbn, q.eA, q.A);
  HQ_LAUNCH_CHECK();
  product(q, q.A, q.A, q.sA, q.sA, N, true, false, 1.0, accumulate, M, st);
}

void quad64_pair(const Quad64 &q, const double *phi, const double *w, const double *Y, long long N, double scale,
                 bool accumulate, double *M, cudaStream_t st) {
  HQ_STAGE(ST_QUAD, st);
  const int nb = (int)quad64_table(N), rb = quad64_rows(q.n), rbn = quad64_row_blocks(q.n);
  maxima(w, 1, N, q.wtab, st);
  k_qf_exponents<<<q.n, 128, 0, st>>>(q.tab, nullptr, q.n, nb, q.wtab, nullptr, 0.f, q.eA, q.sA);
  HQ_LAUNCH_CHECK();
  k_qf_digits<1><<<ceil_div(N, kQfK), 256, 0, st>>>(phi, nullptr, w, nullptr, 0.0, q.n, N, rb, rbn, q.eA, q.A);
  HQ_LAUNCH_CHECK();
  maxima(Y, q.n, N, q.xtab, st);
  k_qf_exponents<<<q.n, 128, 0, st>>>(q.xtab, nullptr, q.n, nb, nullptr, nullptr, 0.f, q.eX, q.sX);
  HQ_LAUNCH_CHECK();
  k_qf_digits<0><<<ceil_div(N, kQfK), 256, 0, st>>>(Y, nullptr, nullptr, nullptr, 0.0, q.n, N, rb, rbn, q.eX, q.X);
  HQ_LAUNCH_CHECK();
  product(q, q.A, q.X, q.sA, q.sX, N, false, false, scale, accumulate, M, st);
}

}  // namespace hqcgb
