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
// with one power of two e for a row and a block of points, |x| <= 2^(e - 1): 56
// bits below the largest element of the row in that block, where FP64 keeps 53 of
// each.  The blocks are bricks of the grid, at most 8 points a side (512
// consecutive ones where the operand is no grid field): within a brick an AO
// changes little, so an element of M made of two AOs' tails keeps the relative
// accuracy of an FP64 sum, which one power of two for a whole row would cost it.
// Error over the sum of the absolute terms, FP64 sums / a power of two a row / a
// brick, emulated, dzvp, box 9.75 Bohr, 49^3: elements of 1e-2 of the largest and
// more 3e-16 / 2e-16 / 3e-16, of 1e-6 to 1e-4 4e-16 / 1e-12 / 6e-16, of 1e-8 to 1e-6
// 4e-16 / 3e-11 / 8e-16.
//
// A product of digits is at most 2^12, so the points of a block and the at most 8
// products s + t = d fit FP32's 24 bits and the sums P_d (kind::f16, FP32
// accumulators in TMEM, one per d = 0..7) are exact; the 36 products with
// s + t <= 7 are formed, the others are below 2^-56 of the maxima's product.  The
// drains add a block's P_d to an integer of 64 bits, round it once and add it to
// the tile's FP64 sums.
//
// Operands are stored by stages of 32 points, [stage][pair][row][128 bytes]: a
// 128-byte row holds 32 points of two digits, already in the K-major SW128 pattern
// that the MMA reads, so plain bulk copies fill the ring.  One CTA an SM: a
// persistent share of the stages for one 128 x 64 destination tile, a copy thread,
// an MMA warp and eight drain warps.  The MMA warp stays together and one elected lane
// issues: with a branch on the lane number the descriptors of every MMA go through
// ordinary registers (193 -> 146 us at 64 AOs, 65^3).  The digit pass takes a brick a block and a
// row a warp, whose maximum gives the exponent of the values it holds.
//
// Bounds.  One 32-point stage is 72 MMAs of 128 x 64 x 16: the kernel is bound
// by the tensor pipe, at 36 products a term.  Measured, digits
// of the weighted operand and sums included, FP64 pipe -> this: 64 AOs and 65^3
// points 2.24 -> 0.29 ms, 70 AOs and 49^3 points with the gradient term 2.21 ->
// 0.26 ms, 8 AOs and 41^3 points 0.57 -> 0.07 ms (with a power of two a row 0.24,
// 0.32 and 0.08).
#include <algorithm>
#include <cmath>

#include "digits.cuh"
#include "kernels.h"

namespace hqcgb {

using namespace tc;

constexpr int kQfK = 32;                                // points per stage
constexpr int kQfSide = 8;                              // most points a side of a brick
constexpr int kQfBlk = 512;                             // most points of a block: what FP32 adds exactly
constexpr int kQfM = 128, kQfN = 64;
constexpr int kQfRing = 2;
constexpr uint32_t kQfPairA = kQfM * 128, kQfPairB = kQfN * 128;
constexpr uint32_t kQfOffB = kQfPairs * kQfPairA;
constexpr uint32_t kQfStage = kQfPairs * (kQfPairA + kQfPairB);
constexpr size_t kQfSmem = kQfRing * kQfStage + 1024;   // + alignment to the swizzle atom
constexpr int kQfDrainWarps = 8;
constexpr int kQfThreads = (kQfDrainWarps + 2) * 32;
constexpr int kQfMaxTiles = (kMaxNao / kQfM) * (kMaxNao / kQfN);
constexpr long long kQfSegment = 160LL << 20;           // bytes of an operand's digits formed at a time
constexpr int kQfBad = 1 << 20;                         // exponent of a block with a value that is not finite
static_assert(kQfSmem <= 227 * 1024, "FP64 quadrature ring above 227 KB");
static_assert(kQfSide * kQfSide * kQfSide <= kQfBlk, "a brick is one block");

static int quad64_rows(int n) { return (n + 7) / 8 * 8; }  // the swizzle's period
static size_t stage_bytes(int n) { return (size_t)quad64_rows(n) * 128 * kQfPairs; }
static int quad64_parts(int ng) { return ceil_div(ng, kQfSide); }
static long long quad64_linear_blocks(long long K) { return (K + kQfBlk - 1) / kQfBlk; }

// Bricks: an axis is cut into `parts` nearly equal pieces; first[b] = the first
// stage of brick b (x slowest), first[bricks] = all stages.
std::vector<int> quad64_first(int ng) {
  const int m = quad64_parts(ng);
  std::vector<int> first(1, 0);
  auto len = [&](int k) { return ng * (k + 1) / m - ng * k / m; };
  for (int x = 0; x < m; ++x)
    for (int y = 0; y < m; ++y)
      for (int z = 0; z < m; ++z) first.push_back(first.back() + ceil_div(len(x) * len(y) * len(z), kQfK));
  return first;
}
// Operands are formed and multiplied in segments of whole blocks, so that a plan's
// memory does not grow with its digits: a grid in equal segments of kQfSegment to
// twice that, rows of any length in segments of kQfSegment and a rest (a buffer for
// the longest then holds the shorter ones').  A segment more costs two launches and
// their tails (quadratures of an H32 dzv run at 65^3, 23 of them: one segment 6.3 ms,
// three 7.9, nine 13.4 with the AOs' digits formed too).
struct Segments {
  int blocks, count, size;  // size 0: equal ones
  int begin(int k) const { return size ? std::min(blocks, k * size) : (int)((long long)blocks * k / count); }
};
static Segments grid_segments(int n, int ng, int stages) {
  const int m = quad64_parts(ng);
  return {m * m * m, (int)std::max(1LL, (long long)stages * (long long)stage_bytes(n) / kQfSegment), 0};
}
static Segments linear_segments(int n, long long K) {
  const int blocks = (int)quad64_linear_blocks(K);
  const int size = (int)std::max<long long>(1, kQfSegment / (long long)(stage_bytes(n) * (kQfBlk / kQfK)));
  return {blocks, std::max(1, ceil_div(blocks, size)), size};
}
Quad64Sizes quad64_grid_sizes(int n, int ng) {
  const std::vector<int> first = quad64_first(ng);
  const Segments sg = grid_segments(n, ng, first.back());
  int stages = 0, most = 0;
  for (int k = 0; k < sg.count; ++k) {
    stages = std::max(stages, first[sg.begin(k + 1)] - first[sg.begin(k)]);
    most = std::max(most, sg.begin(k + 1) - sg.begin(k));
  }
  const size_t rows = quad64_rows(n);
  return {first.back() * stage_bytes(n), sg.blocks * rows, stages * stage_bytes(n), most * rows};
}
Quad64Sizes quad64_linear_sizes(int n, long long K) {
  const Segments sg = linear_segments(n, K);
  const size_t rows = quad64_rows(n), stage = stage_bytes(n) * (kQfBlk / kQfK), most = std::min(sg.blocks, sg.size);
  return {sg.blocks * stage, sg.blocks * rows, most * stage, most * rows};
}

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

// A form of the operand: values X (MODE 0), w X (1) or 0.5 w X + dV u . dX (2)
// at the points of a grid in bricks (first) or in their order (first null).
struct QfSource {
  const double *X, *dX, *w, *u;
  double dV;
  int n, rows, ng, parts;
  long long N;
  const int *first;
  int b0;      // the block that the output starts with
  int *e;      // [block][rows]
  char *out;
};

constexpr int kQfFormRows = 8;                                // rows a block works on, a warp each
constexpr int kQfChunk = 9, kQfRowLd = kQfBlk / 8 * kQfChunk + 4;  // doubles from a chunk of 8 points, a row to the
                                                                   // next: no bank conflicts in either phase
static size_t form_smem(int mode) {
  return sizeof(double) * (kQfFormRows * kQfRowLd + (mode == 0 ? 0 : mode == 1 ? 1 : 4) * kQfBlk) + sizeof(int) * kQfBlk;
}

// Blocks an SM that the registers leave room for: the gradient form has four fields'
// loads under way and is better off with more of them (quadratures of an H14 dzvp PBE run
// at 49^3 with 3 / 4 / 5 blocks 5.5 / 6.2 / 6.3 ms, of an H32 dzv LDA run 7.7 / 7.0 / 6.6).
constexpr int qf_form_blocks(int mode) { return mode == 2 ? 3 : 5; }

// Grid (blocks of points, row groups).  A warp loads a row, neighbouring lanes
// neighbouring points, and its maximum gives the exponent; then the warps take a
// stage of all eight rows in turn, eight points of a row a lane, so that what they
// store is 1 KB in one piece.  Points beyond a block's last become zeros; rows beyond
// n are left alone (they only reach destination rows and columns that nothing reads).
template <int MODE>
__global__ void __launch_bounds__(kQfFormRows * 32, qf_form_blocks(MODE)) k_qf_digits(const QfSource a) {
  extern __shared__ __align__(16) double s_x[];  // [rows][kQfRowLd]
  double *s_w = s_x + kQfFormRows * kQfRowLd, *s_u = s_w + kQfBlk;
  int *s_off = reinterpret_cast<int *>(s_w + (MODE == 0 ? 0 : MODE == 1 ? 1 : 4) * kQfBlk);  // the block's points
  __shared__ int s_e[kQfFormRows];
  const int b = a.b0 + blockIdx.x, tid = threadIdx.x;
  int cnt, stage0;
  long long base = 0;
  int x0 = 0, y0 = 0, z0 = 0, sy = 1, sz = 1;
  if (a.first) {
    const int bz = b % a.parts, by = b / a.parts % a.parts, bx = b / (a.parts * a.parts);
    auto cut = [&](int k) { return a.ng * k / a.parts; };
    x0 = cut(bx);
    y0 = cut(by);
    z0 = cut(bz);
    sy = cut(by + 1) - y0;
    sz = cut(bz + 1) - z0;
    cnt = (cut(bx + 1) - x0) * sy * sz;
    stage0 = a.first[b] - a.first[a.b0];
  } else {
    base = (long long)b * kQfBlk;
    cnt = (int)min((long long)kQfBlk, a.N - base);
    stage0 = blockIdx.x * (kQfBlk / kQfK);
  }
  const int stages = (cnt + kQfK - 1) / kQfK, pts = stages * kQfK;
  for (int k = tid; k < pts; k += kQfFormRows * 32) {
    const int r = min(k, cnt - 1);  // beyond the last point: the last once more, times zero below
    int off = r;
    if (a.first) {
      const int x = r / (sy * sz), q = r - x * (sy * sz), y = q / sz;
      off = ((x0 + x) * a.ng + y0 + y) * a.ng + z0 + q - y * sz;
    }
    s_off[k] = off;
    if (MODE) s_w[k] = k < cnt ? a.w[base + off] * (MODE == 2 ? 0.5 : 1.0) : 0.0;
    if (MODE == 2)
      for (int d = 0; d < 3; ++d) s_u[d * kQfBlk + k] = k < cnt ? a.dV * a.u[(long long)d * a.N + base + off] : 0.0;
  }
  __syncthreads();
  const int lane = tid & 31, warp = tid >> 5;
  for (int p0 = blockIdx.y * kQfFormRows; p0 < a.n; p0 += gridDim.y * kQfFormRows) {
    const int p = p0 + warp;
    if (p < a.n) {
      const double *X = a.X + (long long)p * a.N + base;
      const double *dX = MODE == 2 ? a.dX + (long long)p * a.N + base : nullptr;
      unsigned top = 0;
#pragma unroll 4
      for (int k = lane; k < pts; k += 32) {
        const int off = s_off[k];
        double x = X[off];
        if (MODE) x *= s_w[k];
        else if (k >= cnt) x = 0.0;
        if (MODE == 2)
#pragma unroll
          for (int d = 0; d < 3; ++d) x += s_u[d * kQfBlk + k] * dX[(long long)d * a.n * a.N + off];
        s_x[warp * kQfRowLd + (k >> 3) * kQfChunk + (k & 7)] = x;
        top = max(top, (unsigned)__double2hiint(x) & 0x7fffffffu);
      }
      top = __reduce_max_sync(0xffffffffu, top);
      const int ex = (int)(top >> 20);  // every |x| < 2^(ex - 1022)
      const int e = ex == 0x7ff ? kQfBad : ex - 1021;
      if (lane == 0) {
        s_e[warp] = e;
        a.e[(long long)blockIdx.x * a.rows + p] = e;
      }
    }
    __syncthreads();
    const int r = lane >> 2, c = lane & 3;
    if (p0 + r < a.n) {
      const int e = s_e[r];
      for (int st = warp; st < stages; st += kQfFormRows) {
        const double *x = s_x + r * kQfRowLd + (st * 4 + c) * kQfChunk;
        QfPack pack;
#pragma unroll
        for (int i = 0; i < 8; ++i) pack.put(i, x[i], e);
        char *row = a.out + ((long long)(stage0 + st) * kQfPairs * a.rows + p0 + r) * 128;
        pack.store(row, (long long)a.rows * 128, c, r);  // p0 is a multiple of 8
      }
    }
    __syncthreads();
  }
}

struct QfArgs {
  const char *A, *B;
  const int *eA, *eB;  // [block][rows]
  const int *first;    // first stage of every block, or null: 16 stages a block, `stages` in all
  double *part;        // [group][tile][128][64]
  int *err;
  int stages, b0, b1;  // the segment's blocks
  int wholeA, wholeB;  // the operand holds all blocks, not the segment's alone
  int add;             // to the sums of the segments before
  int n, rows, groups, tiles;
  unsigned char tile[kQfMaxTiles][2];  // 128-row block of A, 64-row block of B
};

// The chains of group g's share of the segment's stages, in order: stages [s, e) of
// block b, s and e counted from the segment's first stage.
struct QfChains {
  const QfArgs &a;
  int s, e, end, b, base;
  __device__ __forceinline__ int first(int k) const { return a.first ? a.first[k] : min(k * (kQfBlk / kQfK), a.stages); }
  __device__ __forceinline__ QfChains(const QfArgs &a_, int g) : a(a_) {
    base = first(a.b0);
    const long long stages = first(a.b1) - base;
    s = e = (int)(stages * g / a.groups);
    end = (int)(stages * (g + 1) / a.groups);
    b = a.b0 + s / (kQfBlk / kQfK);  // a block is at most 16 stages
    if (a.first)
      for (int hi = a.b1; hi - b > 1;) {
        const int mid = (b + hi) / 2;
        if (a.first[mid] - base <= s) b = mid;
        else hi = mid;
      }
    --b;
  }
  __device__ __forceinline__ bool next() {
    s = e;
    if (s >= end) return false;
    ++b;
    e = min(end, first(b + 1) - base);
    return true;
  }
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

  const uint32_t tmem = P.tmem_base;
  bool ok = true;
  if (warp == kQfDrainWarps + 1) {
    if (lane == 0) {
      const uint32_t na = (uint32_t)min(kQfM, a.rows - mt * kQfM) * 128u;
      const uint32_t nb = (uint32_t)min(kQfN, a.rows - ct * kQfN) * 128u;
      const long long pair = (long long)a.rows * 128;
      int it = 0;
      QfChains c(a, g);
      const char *A0 = a.A + (a.wholeA ? c.base : 0) * kQfPairs * pair + (long long)mt * kQfM * 128;
      const char *B0 = a.B + (a.wholeB ? c.base : 0) * kQfPairs * pair + (long long)ct * kQfN * 128;
      while (ok && c.next())
        for (int s = c.s; s < c.e; ++s, ++it) {
          const int slot = it % kQfRing, use = it / kQfRing;
          if (use > 0 && !mbar_wait(&P.empty[slot], (unsigned)((use - 1) & 1), a.err, 61)) {
            ok = false;
            break;
          }
          mbar_expect_tx(&P.full[slot], kQfPairs * (na + nb));
          const uint32_t dst = smem_u32(sm + slot * kQfStage);
          const char *srcA = A0 + s * kQfPairs * pair, *srcB = B0 + s * kQfPairs * pair;
          for (int q = 0; q < kQfPairs; ++q) {
            bulk_copy(dst + q * kQfPairA, srcA + q * pair, na, &P.full[slot]);
            bulk_copy(dst + kQfOffB + q * kQfPairB, srcB + q * pair, nb, &P.full[slot]);
          }
        }
    }
  } else if (warp == kQfDrainWarps) {
    {
      // kind::f16, D = F32, A = B = BF16, both K-major
      const uint32_t idesc = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(nn >> 3) << 17) |
                             ((uint32_t)(kQfM >> 4) << 24);
      QfChains c(a, g);
      for (int j = 0, it = 0; ok && c.next(); ++j) {
        if (j > 0 && !mbar_wait(&P.acc_empty, (unsigned)((j - 1) & 1), a.err, 64)) ok = false;
        ok = __all_sync(0xffffffffu, ok);
        tc_fence_after();
        const int end = it + c.e - c.s;
        bool first = true;
        for (; it < end && ok; ++it) {
          const int slot = it % kQfRing, use = it / kQfRing;
          if (!mbar_wait(&P.full[slot], (unsigned)(use & 1), a.err, 62)) ok = false;
          ok = __all_sync(0xffffffffu, ok);
          tc_fence_after();
          const bool el = elect();
          if (ok && el) {
            const uint64_t dA = sdesc(smem_u32(sm + slot * kQfStage)), dB = dA + (kQfOffB >> 4);
#pragma unroll 1
            for (int ks = 0; ks < kQfK / 16; ++ks) {
#pragma unroll
              for (int s = 0; s < kQfDigits; ++s) {
                // digit s: pair s / 2, half a 128-byte row (4 units of 16 bytes) each, 2 units a K step
                const uint64_t da = dA + (uint32_t)((s >> 1) * (kQfPairA >> 4) + (s & 1) * 4 + 2 * ks);
#pragma unroll
                for (int t = 0; t < kQfDigits - s; ++t)
                  mma_bf16(tmem + (s + t) * kQfN, da,
                           dB + (uint32_t)((t >> 1) * (kQfPairB >> 4) + (t & 1) * 4 + 2 * ks), idesc,
                           !(first && ks == 0 && s == 0));
              }
            }
          }
          first = false;
          if (el) mma_commit(&P.empty[slot]);
        }
        if (elect()) mma_commit(&P.acc_full);
      }
    }
  } else {
    // warp w owns TMEM lanes 32 (w % 4) .. and columns 32 (w / 4) .. + 31 of every P_d
    const int c0 = (warp >> 2) * 32, row = (warp & 3) * 32 + lane;
    const uint32_t base = tmem + ((uint32_t)((warp & 3) * 32) << 16) + c0;
    const int ra = min(mt * kQfM + row, a.n - 1), rb = min(ct * kQfN + c0 + lane, a.n - 1);
    const bool own = mt * kQfM + row < a.n;
    double *out = a.part + (((long long)g * a.tiles + tile) * kQfM + row) * kQfN + c0;
    double acc[32];
#pragma unroll
    for (int i = 0; i < 32; ++i) acc[i] = a.add && own && c0 + i < rows_b ? out[i] : 0.0;
    QfChains c(a, g);
    for (int j = 0; c.next(); ++j) {
      const int ea = a.eA[(long long)(c.b - (a.wholeA ? 0 : a.b0)) * a.rows + ra],
                eb = a.eB[(long long)(c.b - (a.wholeB ? 0 : a.b0)) * a.rows + rb];
      if (!mbar_wait(&P.acc_full, (unsigned)(j & 1), a.err, 63)) ok = false;
      // a warp's lanes stay together: the loads below and the shuffles are the warp's
      ok = __all_sync(0xffffffffu, ok);
      if (!ok) break;
      tc_fence_after();
      // sum_d P_d 128^(5 - d) / 2, 63 bits before the one rounding; 2^(eA + eB - 53) of it is the block's sum
      long long x[32];
#pragma unroll
      for (int q = 0; q < 8; ++q) {
        uint32_t v[kQfDigits][4];
#pragma unroll
        for (int d = 0; d < kQfDigits; ++d) tmem_ld4_nowait(base + d * kQfN + q * 4, v[d]);
        tmem_wait_ld();
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          long long hi = 0, lo = 0;
#pragma unroll
          for (int d = 0; d < 4; ++d) {
            hi += (long long)__float2int_rn(__uint_as_float(v[d][i])) * (1 << (7 * (3 - d)));
            lo += (long long)__float2int_rn(__uint_as_float(v[d + 4][i])) * (1 << (7 * (3 - d)));
          }
          x[q * 4 + i] = (hi << 18) + (lo >> 10);
        }
      }
      tc_fence_before();
      mbar_arrive(&P.acc_empty);
      // the conversions stay behind the arrival: they run beside the next block's MMAs
#pragma unroll
      for (int i = 0; i < 32; ++i) asm volatile("" : "+l"(x[i]));
#pragma unroll
      for (int i = 0; i < 32; ++i) {
        const int ei = ea + __shfl_sync(0xffffffffu, eb, i);
        const double y = (double)x[i];
        const int h = __double2hiint(y), ey = ((h >> 20) & 0x7ff) + ei - 53;
        if (ei >= kQfBad / 2) acc[i] = NAN;
        else if (ey >= 0x7ff) acc[i] += h < 0 ? -INFINITY : INFINITY;
        else if (x[i] != 0 && ey > 0) acc[i] += __hiloint2double(h + (ei - 53) * (1 << 20), __double2loint(y));
      }
    }
    if (ok && own)
#pragma unroll
      for (int i = 0; i < 32; ++i)
        if (c0 + i < rows_b) out[i] = acc[i];
  }
  tc_fence_before();
  __syncthreads();
  if (warp == kQfDrainWarps) {
    tc_fence_after();
    tmem_dealloc(tmem, kQfDigits * kQfN);
  }
}

// M (+)= scale sum over groups; sym: (p, q) from the upper triangle; tr: M_pq =
// v_pq + v_qp.  A block takes 32 columns of a row, eight threads a value.
__global__ void __launch_bounds__(256)
    k_qf_reduce(const __grid_constant__ QfArgs a, int sym, int tr, double scale, int accumulate,
                double *__restrict__ M) {
  __shared__ double sh[8][33];
  const int p = blockIdx.y, q = blockIdx.x * 32 + (threadIdx.x & 31), part = threadIdx.x >> 5;
  auto value = [&](int r, int c) {
    const int mt = r / kQfM, ct = c / kQfN;
    int t = 0;
    while (t < a.tiles && (a.tile[t][0] != mt || a.tile[t][1] != ct)) ++t;
    const double *src = a.part + ((long long)t * kQfM + r % kQfM) * kQfN + c % kQfN;
    double s = 0;
    for (int g = part; g < a.groups; g += 8) s += src[(long long)g * a.tiles * kQfM * kQfN];
    return s;
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
    s *= scale;
    double *m = M + (long long)p * a.n + q;
    *m = accumulate ? *m + s : s;
  }
}

// Digits of an operand.
struct QfForm {
  int mode = 0;
  const double *X = nullptr, *dX = nullptr, *w = nullptr, *u = nullptr;
  double dV = 0.0;
};
static void form(const Quad64 &q, const QfForm &f, long long N, bool grid, int b0, int b1, int *e, char *out,
                 cudaStream_t st) {
  QfSource a{f.X, f.dX, f.w, f.u, f.dV, q.n, quad64_rows(q.n), q.ng, quad64_parts(q.ng), N, grid ? q.first : nullptr,
             b0, e, out};
  const int blocks = b1 - b0, groups = ceil_div(q.n, kQfFormRows);
  // few bricks: the rows over several blocks, until there are eight blocks an SM
  const dim3 g(blocks, std::max(1, std::min(groups, ceil_div(8 * 152, blocks))));
  const size_t smem = form_smem(f.mode);
  auto go = [&](auto kernel) {
    ensure_dyn_smem((const void *)kernel, smem);
    kernel<<<g, kQfFormRows * 32, smem, st>>>(a);
    HQ_LAUNCH_CHECK();
  };
  if (f.mode == 0) go(k_qf_digits<0>);
  else if (f.mode == 1) go(k_qf_digits<1>);
  else go(k_qf_digits<2>);
}

// An operand of a product: digits to be formed, segment by segment, or those of the
// AOs where the plan keeps them (X null).
static QfForm kept() { return QfForm{}; }

// M (+)= scale sum over the points; same: both operands are fa.  The sums run
// segment by segment whether or not digits are kept, so the bits do not depend on that.
static void product(const Quad64 &q, const QfForm &fa, const QfForm &fb, bool same, long long N, bool grid, bool sym,
                    bool tr, double scale, bool accumulate, double *M, cudaStream_t st) {
  QfArgs a{};
  a.wholeA = !fa.X;
  a.wholeB = same ? a.wholeA : !fb.X;
  a.A = a.wholeA ? q.B : q.A;
  a.eA = a.wholeA ? q.eB : q.eA;
  a.B = same ? a.A : a.wholeB ? q.B : q.X;
  a.eB = same ? a.eA : a.wholeB ? q.eB : q.eX;
  a.first = grid ? q.first : nullptr;
  a.part = q.part;
  a.err = q.err;
  a.stages = grid ? q.stages : ceil_div(N, kQfK);
  a.n = q.n;
  a.rows = quad64_rows(q.n);
  a.tiles = quad64_tiles(q.n, sym, a.tile);
  a.groups = quad64_groups(q.n, sym);
  ensure_dyn_smem((const void *)k_qf_gemm, kQfSmem);
  const Segments sg = grid ? grid_segments(q.n, q.ng, q.stages) : linear_segments(q.n, N);
  for (int k = 0; k < sg.count; ++k) {
    a.b0 = sg.begin(k);
    a.b1 = sg.begin(k + 1);
    a.add = k > 0;
    HQ_REQUIRE((size_t)(a.b1 - a.b0) * a.rows <= q.exponents, "segment beyond the plan's digit buffers");
    if (fa.X) form(q, fa, N, grid, a.b0, a.b1, q.eA, q.A, st);
    if (!same && fb.X) form(q, fb, N, grid, a.b0, a.b1, q.eX, q.X, st);
    k_qf_gemm<<<dim3(a.tiles, a.groups), kQfThreads, kQfSmem, st>>>(a);
    HQ_LAUNCH_CHECK();
  }
  k_qf_reduce<<<dim3(ceil_div(q.n, 32), q.n), 256, 0, st>>>(a, sym, tr, scale, accumulate, M);
  HQ_LAUNCH_CHECK();
}

void quad64_basis(const Quad64 &q, const double *phi, long long N, cudaStream_t st) {
  HQ_STAGE(ST_SPLIT, st);
  if (q.B) form(q, QfForm{0, phi}, N, true, 0, grid_segments(q.n, q.ng, q.stages).blocks, q.eB, q.B, st);
}

static QfForm basis(const Quad64 &q, const double *phi) { return q.B ? kept() : QfForm{0, phi}; }

void quad64_weighted(const Quad64 &q, const double *phi, const double *w, long long N, double scale, double *M,
                     cudaStream_t st) {
  HQ_STAGE(ST_QUAD, st);
  if (w) product(q, QfForm{1, phi, nullptr, w}, basis(q, phi), false, N, true, true, false, scale, false, M, st);
  else product(q, basis(q, phi), {}, true, N, true, true, false, scale, false, M, st);
}

void quad64_gga(const Quad64 &q, const double *phi, const double *dphi, const double *w, const double *u, double dV,
                long long N, double *M, cudaStream_t st) {
  HQ_STAGE(ST_QUAD, st);
  product(q, QfForm{2, phi, dphi, w, u, dV}, basis(q, phi), false, N, true, false, true, 1.0, false, M, st);
}

void quad64_gram(const Quad64 &q, const double *Q, long long N, bool accumulate, double *M, cudaStream_t st) {
  HQ_STAGE(ST_QUAD, st);
  product(q, QfForm{0, Q}, {}, true, N, false, true, false, 1.0, accumulate, M, st);
}

void quad64_pair(const Quad64 &q, const double *phi, const double *w, const double *Y, long long N, double scale,
                 bool accumulate, double *M, cudaStream_t st) {
  HQ_STAGE(ST_QUAD, st);
  product(q, QfForm{1, phi, nullptr, w}, QfForm{0, Y}, false, N, true, false, false, scale, accumulate, M, st);
}

}  // namespace hqcgb
