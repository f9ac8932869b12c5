// FP64 values as eight signed 7-bit digits for exact bf16 products on the
// tensor cores (the scheme is described in quad_f64.cu), and the PTX that only
// its kernels use.
#pragma once
#include <cuda_bf16.h>

#include "tc_ptx.cuh"

namespace hqcgb {

constexpr int kQfDigits = 8, kQfPairs = kQfDigits / 2;

// The digits of x 2^-e as unsigned 7-bit fields, each 64 above the digit.
__device__ __forceinline__ unsigned long long qf_fields(double x, int e) {
  constexpr long long kBias = 64LL * ((1LL << 0) + (1LL << 7) + (1LL << 14) + (1LL << 21) + (1LL << 28) +
                                      (1LL << 35) + (1LL << 42) + (1LL << 49));
  const long long bits = __double_as_longlong(x);
  const int ex = (int)((bits >> 52) & 0x7ff);
  const int sh = ex - 1075 + 7 * kQfDigits - e;  // x 2^-e 128^8 = m 2^sh
  const long long m = (bits & 0xfffffffffffffLL) | (1LL << 52);
  long long I = 0;
  if (ex > 0 && sh > -54) I = sh >= 0 ? m << min(sh, 3) : (m + (1LL << (-sh - 1))) >> -sh;
  return (unsigned long long)((bits < 0 ? -I : I) + kBias);
}

// Eight consecutive K elements of one row: their digits as bf16, 16 bytes a
// digit, stored into the K-major SW128 pattern (a 128-byte row holds 32
// elements of two digits; `pair_stride` bytes from one pair of digits to the
// next).  Two elements at a time: 0x4300 | f is 128 + f in bf16 (256 for the first
// digit's f = 128), and 192 less is the digit, exactly.
struct QfPack {
  unsigned pk[kQfDigits][4];
  unsigned long long even;

  __device__ __forceinline__ void put(int i, double x, int e) {
    const unsigned long long J = qf_fields(x, e);
    if (!(i & 1)) {
      even = J;
      return;
    }
    const __nv_bfloat162 bias = __halves2bfloat162(__ushort_as_bfloat16(0x4340), __ushort_as_bfloat16(0x4340));
#pragma unroll
    for (int s = 0; s < kQfDigits; ++s) {
      const int sh = 7 * (kQfDigits - 1 - s);
      const unsigned mask = s ? 127u : 255u;
      const unsigned w = ((unsigned)(even >> sh) & mask) | (((unsigned)(J >> sh) & mask) << 16) | 0x43004300u;
      const __nv_bfloat162 v = __hsub2(*reinterpret_cast<const __nv_bfloat162 *>(&w), bias);
      pk[s][i >> 1] = *reinterpret_cast<const unsigned *>(&v);
    }
  }
  // chunk c (0..3) of row r, `row` the row's first byte in the first pair
  __device__ __forceinline__ void store(char *row, long long pair_stride, int c, int r) const {
#pragma unroll
    for (int s = 0; s < kQfDigits; ++s)
      *reinterpret_cast<uint4 *>(row + (s >> 1) * pair_stride + (((s & 1) * 4 + c) ^ (r & 7)) * 16) =
          make_uint4(pk[s][0], pk[s][1], pk[s][2], pk[s][3]);
  }
};

namespace tc {

__device__ inline void bulk_copy(uint32_t dst, const void *src, uint32_t bytes, uint64_t *bar) {
  asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(dst),
               "l"(src), "r"(bytes), "r"(smem_u32(bar))
               : "memory");
}

__device__ inline void mma_bf16(uint32_t dtmem, uint64_t a, uint64_t b, uint32_t idesc, int acc) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}"
      ::"r"(dtmem), "l"(a), "l"(b), "r"(idesc), "r"(acc));
}

__device__ inline void tmem_ld4_nowait(uint32_t taddr, uint32_t *r) {
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x4.b32 {%0,%1,%2,%3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
               : "r"(taddr));
}

}  // namespace tc
}  // namespace hqcgb
