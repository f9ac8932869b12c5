// FP64 density in the orbital form on the tensor cores (hqc/pbc/solver.py:
// 566-577, 690): psi_k(g) = sum_p phi_p(g) Y_pk, Y = C sqrt(f), rho = sum_k
// psi_k^2 and grad rho = 2 sum_k psi_k grad psi_k, equal to the sum over D = Y Y^T.
//
// The products are those of quad_f64.cu (eight 7-bit digits, 36 exact bf16
// products): rows are grid points, K the AOs, columns the occupied orbitals,
// with one power of two for a point and one for an orbital.  A psi comes out of
// two 64-bit integers with a single rounding; FP64 arithmetic is left for
// psi^2, three operations an orbital and point where the sum over D takes an
// operation an AO pair and point.
//
// A tile of the sum is 128 points.  Eight warps read phi (and the gradient's three
// fields) for it and form the digits in the K-major SW128 pattern of the ring, 32 AOs a
// stage, a lane a point and 16 AOs; kept in memory those digits would be 16 bytes a value
// (9.8 GB of an H54 dzvp PBE plan at 81^3), written once a geometry and read for every
// density where phi is read now.  Y^T by 64 orbitals,
// [column block][block of 32 AOs][pair][64][128], comes by bulk copies.  Persistent CTAs,
// one an SM, take tiles in turn: the forming warps, a copy thread, an MMA warp, eight
// drain warps.  Bound by the MMAs (72 a stage) and the instructions that form their digits
// (about 80 a value) together.  Measured: 64 AOs, 38 orbitals, 65^3 points 0.18 ms (sum over
// D on the FP64 pipe 1.87, digits kept in memory 0.18); 70 AOs, 7 orbitals, 49^3 with the
// gradient 0.23 (1.05, 0.18); 270 AOs, 27 orbitals, 65^3 with the gradient 1.3 (kept 1.06,
// digits of a range of tiles formed in memory before its part of the density 3.5).  With
// four forming warps 2.5; eight, whose 18 warps leave 96 registers and some spills of the
// drains' in the gradient form, but 136 registers for those by setmaxnreg were slower.
#include <algorithm>
#include <cmath>

#include "digits.cuh"
#include "kernels.h"

namespace hqcgb {

using namespace tc;

constexpr int kDfM = 128, kDfN = 64, kDfK = 32, kDfRing = 2;
constexpr uint32_t kDfPairA = kDfM * 128, kDfPairB = kDfN * 128;
constexpr uint32_t kDfOffB = kQfPairs * kDfPairA;
constexpr uint32_t kDfStage = kQfPairs * (kDfPairA + kDfPairB);
constexpr size_t kDfSmem = kDfRing * kDfStage + 1024;
constexpr int kDfDrainWarps = 8, kDfFormWarps = 8;
constexpr int kDfThreads = (kDfDrainWarps + 2 + kDfFormWarps) * 32;
constexpr int kDfHalf = kDfFormWarps * 32 / kDfM, kDfRun = kDfK / kDfHalf;  // AOs of a stage that a lane forms
constexpr int kDfMaxAo = 512;  // one TMEM sum holds 512 terms exactly

int density64_max_ao() { return kDfMaxAo; }
static int df_blocks(int nao) { return ceil_div(nao, kDfK); }
size_t density64_orbital_bytes(int nao) {
  return (size_t)ceil_div(nao, kDfN) * df_blocks(nao) * kQfPairs * kDfPairB;
}

// Scale of every grid point, the power of two 2^e above the largest |phi_p(g)|.
__global__ void __launch_bounds__(256)
    k_df_points(const double *__restrict__ phi, int nao, long long N, double *__restrict__ scale) {
  const long long g = (long long)blockIdx.x * 256 + threadIdx.x;
  if (g >= N) return;
  unsigned v = 0;
  for (int p = 0; p < nao; ++p) v = max(v, __float_as_uint(__double2float_ru(fabs(phi[(long long)p * N + g]))));
  const float m = __uint_as_float(v);
  int k = 0;
  if (m > 0.f && m < INFINITY) frexpf(m, &k);
  scale[g] = m < INFINITY ? scalbn(1.0, k + 1) : NAN;
}

// Digits of Y^T: block k = orbital, Y_pk = C_pk sqrt(f_k); eY[k] its exponent
// (kBad when it is not finite).
constexpr int kBad = 1 << 20;
__global__ void __launch_bounds__(128)
    k_df_orbitals(const double *__restrict__ C, const double *__restrict__ occ, int nao, int nkb,
                  int *__restrict__ eY, char *__restrict__ out) {
  __shared__ unsigned s[4];
  __shared__ int s_e;
  const int k = blockIdx.x;
  const double f = sqrt(occ[k]);
  unsigned v = 0;
  for (int p = threadIdx.x; p < nao; p += 128)
    v = max(v, __float_as_uint(__double2float_ru(fabs(C[(long long)p * nao + k] * f))));
  v = __reduce_max_sync(0xffffffffu, v);
  if ((threadIdx.x & 31) == 0) s[threadIdx.x >> 5] = v;
  __syncthreads();
  if (threadIdx.x == 0) {
    const float m = __uint_as_float(max(max(s[0], s[1]), max(s[2], s[3])));
    int q = 0;
    if (m > 0.f && m < INFINITY) frexpf(m, &q);
    s_e = q + 1;
    eY[k] = m < INFINITY ? q + 1 : kBad;
  }
  __syncthreads();
  const int r = k % kDfN;
  for (int ch = threadIdx.x; ch < nkb * 4; ch += 128) {
    QfPack pack;
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      const int p = ch * 8 + i;
      pack.put(i, p < nao ? C[(long long)p * nao + k] * f : 0.0, s_e);
    }
    char *row = out + (((long long)(k / kDfN) * nkb + (ch >> 2)) * kQfPairs * kDfN + r) * 128;
    pack.store(row, kDfPairB, ch & 3, r);
  }
}

struct DfArgs {
  const double *phi, *dphi;
  const char *B;
  const double *sA;  // [fields][N]
  const int *eY;
  double *rho, *grho, *psi;  // psi [nuse][N] or null
  int *err;
  long long N;
  int nao, tiles, nkb, nuse, cols, bufs;  // cols: TMEM columns of one P_d
};

struct DfPipe {
  uint64_t full[kDfRing], empty[kDfRing], acc_full[2], acc_empty[2];
  uint32_t tmem_base;
};

// FIELDS = 1 (rho) or 4 (rho and its gradient)
template <int FIELDS>
__global__ void __launch_bounds__(kDfThreads, 1) k_df_density(const DfArgs a) {
  extern __shared__ __align__(1024) char smraw[];
  char *sm = (char *)(((uintptr_t)smraw + 1023) & ~(uintptr_t)1023);
  __shared__ DfPipe P;
  __shared__ double s_sum[FIELDS][kDfM];
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int ncb = (a.nuse + kDfN - 1) / kDfN;
  auto columns = [&](int cb) { return min(kDfN, a.nuse - cb * kDfN); };
  if (tid == 0) {
    for (int b = 0; b < kDfRing; ++b) {
      mbar_init(&P.full[b], 1 + kDfFormWarps * 32);
      mbar_init(&P.empty[b], 1);
    }
    for (int b = 0; b < 2; ++b) {
      mbar_init(&P.acc_full[b], 1);
      mbar_init(&P.acc_empty[b], kDfDrainWarps * 32);
    }
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == kDfDrainWarps) tmem_alloc(&P.tmem_base, 512);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();

  const uint32_t tmem = P.tmem_base;
  bool ok = true;
  if (warp == kDfDrainWarps + 1) {
    if (lane == 0) {
      int st = 0;
      for (int tile = blockIdx.x; tile < a.tiles && ok; tile += gridDim.x)
        for (int cb = 0; cb < ncb && ok; ++cb)
          for (int f = 0; f < FIELDS && ok; ++f)
            for (int kb = 0; kb < a.nkb; ++kb, ++st) {
              const int slot = st % kDfRing, use = st / kDfRing;
              if (use > 0 && !mbar_wait(&P.empty[slot], (unsigned)((use - 1) & 1), a.err, 71)) {
                ok = false;
                break;
              }
              const uint32_t nb = (uint32_t)((columns(cb) + 7) / 8 * 8) * 128u;
              mbar_expect_tx(&P.full[slot], kQfPairs * nb);
              const uint32_t dst = smem_u32(sm + slot * kDfStage);
              const char *srcB = a.B + ((long long)cb * a.nkb + kb) * kQfPairs * kDfPairB;
              for (int q = 0; q < kQfPairs; ++q)
                bulk_copy(dst + kDfOffB + q * kDfPairB, srcB + q * kDfPairB, nb, &P.full[slot]);
            }
    }
  } else if (warp == kDfDrainWarps) {
    // the warp stays together and one elected lane issues, as in quad_f64.cu
    int st = 0, chain = 0;
    for (int tile = blockIdx.x; tile < a.tiles && ok; tile += gridDim.x)
      for (int cb = 0; cb < ncb && ok; ++cb) {
        const int nn = (columns(cb) + 15) / 16 * 16;
        // kind::f16, D = F32, A = B = BF16, both K-major
        const uint32_t idesc = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(nn >> 3) << 17) |
                               ((uint32_t)(kDfM >> 4) << 24);
        for (int f = 0; f < FIELDS && ok; ++f, ++chain) {
          const int b = chain % a.bufs, use = chain / a.bufs;
          if (use > 0 && !mbar_wait(&P.acc_empty[b], (unsigned)((use - 1) & 1), a.err, 74)) ok = false;
          ok = __all_sync(0xffffffffu, ok);
          tc_fence_after();
          const uint32_t d0 = tmem + b * kQfDigits * a.cols;
          for (int kb = 0; kb < a.nkb && ok; ++kb, ++st) {
            const int slot = st % kDfRing, su = st / kDfRing;
            if (!mbar_wait(&P.full[slot], (unsigned)(su & 1), a.err, 72)) ok = false;
            ok = __all_sync(0xffffffffu, ok);
            tc_fence_after();
            const bool el = elect();
            if (ok && el) {
              const uint64_t dA = sdesc(smem_u32(sm + slot * kDfStage)), dB = dA + (kDfOffB >> 4);
#pragma unroll 1
              for (int ks = 0; ks < kDfK / 16; ++ks)
#pragma unroll
                for (int s = 0; s < kQfDigits; ++s) {
                  const uint64_t da = dA + (uint32_t)((s >> 1) * (kDfPairA >> 4) + (s & 1) * 4 + 2 * ks);
#pragma unroll
                  for (int t = 0; t < kQfDigits - s; ++t)
                    mma_bf16(d0 + (s + t) * a.cols, da,
                             dB + (uint32_t)((t >> 1) * (kDfPairB >> 4) + (t & 1) * 4 + 2 * ks), idesc,
                             !(kb == 0 && ks == 0 && s == 0));
                }
            }
            if (el) mma_commit(&P.empty[slot]);
          }
          if (elect()) mma_commit(&P.acc_full[b]);
        }
      }
  } else if (warp > kDfDrainWarps + 1) {
    const int t = tid - (kDfDrainWarps + 2) * 32, r = t % kDfM, c0 = t / kDfM * (kDfRun / 8);
    int st = 0;
    double v[kDfRun / 8][8];  // each chunk's values are on their way while the others become digits
    const double *X = nullptr;  // the point's values of the stage that comes next, null beyond N
    int p0 = 0;
    auto next = [&](int tile, int f, int kb) {
      const long long g = (long long)tile * kDfM + r;
      X = tile < a.tiles && g < a.N ? (f == 0 ? a.phi : a.dphi + (long long)(f - 1) * a.nao * a.N) + g : nullptr;
      p0 = kb * kDfK + c0 * 8;
    };
    auto fetch = [&](int c) {
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        const int p = p0 + c * 8 + i;
        v[c][i] = X && p < a.nao ? X[(long long)p * a.N] : 0.0;
      }
    };
    next(blockIdx.x, 0, 0);
#pragma unroll
    for (int c = 0; c < kDfRun / 8; ++c) fetch(c);
    for (int tile = blockIdx.x; tile < a.tiles && ok; tile += gridDim.x) {
      const long long g = (long long)tile * kDfM + r;
      for (int cb = 0; cb < ncb && ok; ++cb)
        for (int f = 0; f < FIELDS && ok; ++f) {
          const int e = g < a.N ? ((__double2hiint(a.sA[f * a.N + g]) >> 20) & 0x7ff) - 1023 : 0;
          for (int kb = 0; kb < a.nkb; ++kb, ++st) {
            const int slot = st % kDfRing, use = st / kDfRing;
            if (kb + 1 < a.nkb) next(tile, f, kb + 1);
            else if (f + 1 < FIELDS) next(tile, f + 1, 0);
            else next(cb + 1 < ncb ? tile : tile + gridDim.x, 0, 0);
            if (use > 0 && !mbar_wait(&P.empty[slot], (unsigned)((use - 1) & 1), a.err, 75)) {
              ok = false;
              break;
            }
            char *row = sm + slot * kDfStage + r * 128;
#pragma unroll
            for (int c = 0; c < kDfRun / 8; ++c) {
              QfPack pack;
#pragma unroll
              for (int i = 0; i < 8; ++i) pack.put(i, v[c][i], e);
              fetch(c);
              pack.store(row, kDfPairA, c0 + c, r);
            }
            fence_proxy_async();
            mbar_arrive(&P.full[slot]);
          }
        }
    }
  } else {
    // warp w: TMEM lanes 32 (w % 4) .. and half w / 4 of the columns
    const int half = warp >> 2, hc = a.cols / 2, row = (warp & 3) * 32 + lane;
    const uint32_t base = tmem + ((uint32_t)((warp & 3) * 32) << 16) + half * hc;
    int chain = 0;
    for (int tile = blockIdx.x; tile < a.tiles; tile += gridDim.x) {
      const long long g = (long long)tile * kDfM + row;
      double acc[FIELDS];
#pragma unroll
      for (int f = 0; f < FIELDS; ++f) acc[f] = 0.0;
      double bad = 0.0;
      for (int cb = 0; cb < ncb; ++cb) {
        double psi[FIELDS > 1 ? kDfN / 2 : 1];
#pragma unroll
        for (int f = 0; f < FIELDS; ++f, ++chain) {
          const int b = chain % a.bufs, use = chain / a.bufs;
          if (ok && !mbar_wait(&P.acc_full[b], (unsigned)(use & 1), a.err, 73)) ok = false;
          tc_fence_after();
          if (ok) {
            const uint32_t d0 = base + b * kQfDigits * a.cols;
#pragma unroll
            for (int q = 0; q < kDfN / 8; ++q) {
              if (q * 4 >= hc) break;
              uint32_t v[kQfDigits][4];
#pragma unroll
              for (int d = 0; d < kQfDigits; ++d) tmem_ld4_nowait(d0 + d * a.cols + q * 4, v[d]);
              tmem_wait_ld();
#pragma unroll
              for (int i = 0; i < 4; ++i) {
                const int k = cb * kDfN + half * hc + q * 4 + i;
                long long hi = 0, lo = 0;
#pragma unroll
                for (int d = 0; d < 4; ++d) {
                  hi += (long long)__float2int_rn(__uint_as_float(v[d][i])) * (1 << (7 * (3 - d)));
                  lo += (long long)__float2int_rn(__uint_as_float(v[d + 4][i])) * (1 << (7 * (3 - d)));
                }
                // psi 2^(39 + 14 - eA - eY), 63 bits before the one rounding
                const int ek = k < a.nuse ? a.eY[k] : kBad;
                double x = (double)((hi << 18) + (lo >> 10));
                if (ek == kBad) {
                  x = 0.0;
                  if (k < a.nuse) bad = NAN;
                } else if (x != 0.0) {
                  x = __hiloint2double(__double2hiint(x) + (ek << 20), __double2loint(x));
                }
                if (f == 0) {
                  acc[0] = fma(x, x, acc[0]);
                  if (FIELDS > 1) psi[q * 4 + i] = x;
                  if (a.psi && k < a.nuse && g < a.N)
                    a.psi[(long long)k * a.N + g] = x * 0x1p-53 * a.sA[g] + bad;
                } else {
                  acc[f] = fma(psi[FIELDS > 1 ? q * 4 + i : 0], x, acc[f]);
                }
              }
            }
          }
          tc_fence_before();
          mbar_arrive(&P.acc_empty[b]);
        }
      }
      // the halves' sums, then rho and grad rho
      if (half == 1)
#pragma unroll
        for (int f = 0; f < FIELDS; ++f) s_sum[f][row] = acc[f] + bad;
      asm volatile("bar.sync 1, %0;" ::"n"(kDfDrainWarps * 32) : "memory");
      if (half == 0 && g < a.N && ok) {
        const double s0 = a.sA[g] * 0x1p-53;
        a.rho[g] = (acc[0] + bad + s_sum[0][row]) * s0 * s0;
#pragma unroll
        for (int f = 1; f < FIELDS; ++f)
          a.grho[(f - 1) * a.N + g] = 2.0 * ((acc[f] + bad + s_sum[f][row]) * s0 * (a.sA[f * a.N + g] * 0x1p-53));
      }
      asm volatile("bar.sync 1, %0;" ::"n"(kDfDrainWarps * 32) : "memory");
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == kDfDrainWarps) {
    tc_fence_after();
    tmem_dealloc(tmem, 512);
  }
}

void density64_basis(const Density64 &d, const double *phi, const double *dphi, long long N, cudaStream_t st) {
  HQ_STAGE(ST_SPLIT, st);
  for (int f = 0; f < (dphi ? 4 : 1); ++f) {
    k_df_points<<<ceil_div(N, 256), 256, 0, st>>>(f == 0 ? phi : dphi + (long long)(f - 1) * d.n * N, d.n, N,
                                                  d.sA + f * N);
    HQ_LAUNCH_CHECK();
  }
}

void density64(const Density64 &d, const double *phi, const double *dphi, const double *C, const double *occ, int nuse,
               long long N, double *rho, double *grho, double *psi, cudaStream_t st) {
  HQ_STAGE(ST_DENSITY, st);
  const int nkb = df_blocks(d.n);
  k_df_orbitals<<<nuse, 128, 0, st>>>(C, occ, d.n, nkb, d.eY, d.B);
  HQ_LAUNCH_CHECK();
  DfArgs a{};
  a.phi = phi;
  a.dphi = dphi;
  a.B = d.B;
  a.sA = d.sA;
  a.eY = d.eY;
  a.rho = rho;
  a.grho = grho;
  a.psi = psi;
  a.err = d.err;
  a.N = N;
  a.nao = d.n;
  a.tiles = ceil_div(N, kDfM);
  a.nkb = nkb;
  a.nuse = nuse;
  a.cols = (std::min(nuse, kDfN) + 15) / 16 * 16;
  a.bufs = kQfDigits * a.cols * 2 <= 512 ? 2 : 1;
  const int grid = std::min(152, a.tiles);
  auto go = [&](auto kernel) {
    ensure_dyn_smem((const void *)kernel, kDfSmem);
    kernel<<<grid, kDfThreads, kDfSmem, st>>>(a);
    HQ_LAUNCH_CHECK();
  };
  if (dphi) go(k_df_density<4>);
  else go(k_df_density<1>);
}

}  // namespace hqcgb
