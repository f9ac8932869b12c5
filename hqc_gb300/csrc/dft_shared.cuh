// Small DFTs of odd length on columns in shared memory (exchange.cu, poisson_f64.cu).
#pragma once
#include "common.cuh"

namespace hqcgb {
namespace exx {

template <typename R> struct C2;
template <> struct C2<float> { using T = float2; };
template <> struct C2<double> { using T = double2; };

// Twiddles w[k] = exp(-2 pi i k / n) rounded to R from the FP64 table.
template <typename R2>
__device__ inline void load_twiddles(R2 *w, const double2 *tw, int n) {
  for (int k = threadIdx.x; k < n; k += blockDim.x) {
    w[k].x = tw[k].x;
    w[k].y = tw[k].y;
  }
}

// Small DFTs in shared memory.  Every odd length pairs its outputs k and
// n - k, whose twiddles are complex conjugates: with C = sum_j x_j Re W^(jk)
// and S = sum_j x_j Im W^(jk) (complex sums),
//   X[k] = C + i S,   X[n - k] = C - i S,
// which halves the multiply-adds.  W = exp(-2 pi i / n), w[m] = W^m.
template <typename R2>
__device__ __forceinline__ R2 cmul(R2 a, R2 b) {
  R2 r;
  r.x = a.x * b.x - a.y * b.y;
  r.y = a.x * b.y + a.y * b.x;
  return r;
}

constexpr int kMaxN1 = 16, kMaxN2 = 16;  // register-blocked factor sizes

// DFT along axis 0 of `in` [n][ncol] (columns contiguous), n odd.
// n = n1 n2 with n1 <= kMaxN1, n2 <= kMaxN2 (j = n2 j1 + j2, k = k1 + n1 k2):
//   y[j2 n1 + k1] = W^(j2 k1) sum_j1 x[n2 j1 + j2] W^(n2 j1 k1)   -> tmp
//   X[k1 + n1 k2] = sum_j2 y[j2 n1 + k1] W^(n1 j2 k2)               -> out
// each thread holding one (j2, col) input group (then one (k1, col)) in
// registers; otherwise (a prime n, n1 = 1, or a larger n2) the paired direct
// sum into tmp.  Returns the buffer holding the result; `in` may alias
// `out`.  Ends with a block barrier.
template <typename R, typename R2>
__device__ R2 *dft_axis0_any(const R2 *in, R2 *tmp, R2 *out, int n, int ncol, int n1, const R2 *w) {
  const int n2 = n1 > 1 ? n / n1 : n;
  if (n1 == 1 || n1 > kMaxN1 || n2 > kMaxN2) {
    const int nh = (n + 1) / 2;
    for (int idx = threadIdx.x; idx < nh * ncol; idx += blockDim.x) {
      const int k = idx / ncol, col = idx - k * ncol;
      R2 C = in[col], S;
      S.x = 0;
      S.y = 0;
      int t = 0;
      for (int j = 1; j < n; ++j) {
        t += k;
        if (t >= n) t -= n;
        const R2 x = in[j * ncol + col], ww = w[t];
        C.x += x.x * ww.x;
        C.y += x.y * ww.x;
        S.x += x.x * ww.y;
        S.y += x.y * ww.y;
      }
      R2 a, b;
      a.x = C.x - S.y;
      a.y = C.y + S.x;
      tmp[k * ncol + col] = a;
      if (k > 0) {
        b.x = C.x + S.y;
        b.y = C.y - S.x;
        tmp[(n - k) * ncol + col] = b;
      }
    }
    __syncthreads();
    return tmp;
  }
  for (int it = threadIdx.x; it < n2 * ncol; it += blockDim.x) {
    const int j2 = it / ncol, col = it - j2 * ncol;
    R2 x[kMaxN1];
#pragma unroll
    for (int j1 = 0; j1 < kMaxN1; ++j1)
      if (j1 < n1) x[j1] = in[(n2 * j1 + j2) * ncol + col];
    R2 s0 = x[0];
#pragma unroll
    for (int j1 = 1; j1 < kMaxN1; ++j1)
      if (j1 < n1) {
        s0.x += x[j1].x;
        s0.y += x[j1].y;
      }
    tmp[(j2 * n1) * ncol + col] = s0;
    for (int k1 = 1; 2 * k1 < n1; ++k1) {
      R2 C = x[0], S;
      S.x = 0;
      S.y = 0;
      int t = 0;
#pragma unroll
      for (int j1 = 1; j1 < kMaxN1; ++j1)
        if (j1 < n1) {
          t += k1;
          if (t >= n1) t -= n1;
          const R2 ww = w[n2 * t];
          C.x += x[j1].x * ww.x;
          C.y += x[j1].y * ww.x;
          S.x += x[j1].x * ww.y;
          S.y += x[j1].y * ww.y;
        }
      R2 a, b;
      a.x = C.x - S.y;
      a.y = C.y + S.x;
      b.x = C.x + S.y;
      b.y = C.y - S.x;
      tmp[(j2 * n1 + k1) * ncol + col] = cmul(a, w[(j2 * k1) % n]);
      tmp[(j2 * n1 + n1 - k1) * ncol + col] = cmul(b, w[(j2 * (n1 - k1)) % n]);
    }
  }
  __syncthreads();
  for (int it = threadIdx.x; it < n1 * ncol; it += blockDim.x) {
    const int k1 = it / ncol, col = it - k1 * ncol;
    R2 y[kMaxN2];
#pragma unroll
    for (int j2 = 0; j2 < kMaxN2; ++j2)
      if (j2 < n2) y[j2] = tmp[(j2 * n1 + k1) * ncol + col];
    R2 s0 = y[0];
#pragma unroll
    for (int j2 = 1; j2 < kMaxN2; ++j2)
      if (j2 < n2) {
        s0.x += y[j2].x;
        s0.y += y[j2].y;
      }
    out[k1 * ncol + col] = s0;
    for (int k2 = 1; 2 * k2 < n2; ++k2) {
      R2 C = y[0], S;
      S.x = 0;
      S.y = 0;
      int t = 0;
#pragma unroll
      for (int j2 = 1; j2 < kMaxN2; ++j2)
        if (j2 < n2) {
          t += k2;
          if (t >= n2) t -= n2;
          const R2 ww = w[n1 * t];
          C.x += y[j2].x * ww.x;
          C.y += y[j2].y * ww.x;
          S.x += y[j2].x * ww.y;
          S.y += y[j2].y * ww.y;
        }
      R2 a, b;
      a.x = C.x - S.y;
      a.y = C.y + S.x;
      b.x = C.x + S.y;
      b.y = C.y - S.x;
      out[(k1 + n1 * k2) * ncol + col] = a;
      out[(k1 + n1 * (n2 - k2)) * ncol + col] = b;
    }
  }
  __syncthreads();
  return out;
}

// The same two-factor transform for the grids of the benchmark
// configurations (n = N1 N2 at compile time): the inner transforms' twiddles
// live in registers and every index is a constant, which removes most of the
// integer work of the generic routine; work items advance without divisions.
template <typename R, typename R2, int N1, int N2>
__device__ R2 *dft_axis0_fixed(const R2 *in, R2 *tmp, R2 *out, int ncol, const R2 *w) {
  constexpr int n = N1 * N2;
  R2 w1[N1], w2[N2];  // W_N1^m = W^(N2 m), W_N2^m = W^(N1 m)
#pragma unroll
  for (int m = 0; m < N1; ++m) w1[m] = w[N2 * m];
#pragma unroll
  for (int m = 0; m < N2; ++m) w2[m] = w[N1 * m];
  const int step_r = (int)blockDim.x / ncol, step_c = (int)blockDim.x - step_r * ncol;
  {
    int j2 = (int)threadIdx.x / ncol, col = (int)threadIdx.x - j2 * ncol;
    while (j2 < N2) {
      R2 x[N1];
#pragma unroll
      for (int j1 = 0; j1 < N1; ++j1) x[j1] = in[(N2 * j1 + j2) * ncol + col];
      R2 s0 = x[0];
#pragma unroll
      for (int j1 = 1; j1 < N1; ++j1) {
        s0.x += x[j1].x;
        s0.y += x[j1].y;
      }
      tmp[(j2 * N1) * ncol + col] = s0;
#pragma unroll
      for (int k1 = 1; 2 * k1 < N1; ++k1) {
        R2 C = x[0], S;
        S.x = 0;
        S.y = 0;
#pragma unroll
        for (int j1 = 1; j1 < N1; ++j1) {
          const R2 ww = w1[(j1 * k1) % N1];
          C.x += x[j1].x * ww.x;
          C.y += x[j1].y * ww.x;
          S.x += x[j1].x * ww.y;
          S.y += x[j1].y * ww.y;
        }
        R2 a, b;
        a.x = C.x - S.y;
        a.y = C.y + S.x;
        b.x = C.x + S.y;
        b.y = C.y - S.x;
        // j2 k1 < n: no reduction of the twiddle index
        tmp[(j2 * N1 + k1) * ncol + col] = cmul(a, w[j2 * k1]);
        tmp[(j2 * N1 + N1 - k1) * ncol + col] = cmul(b, w[j2 * (N1 - k1)]);
      }
      col += step_c;
      j2 += step_r;
      if (col >= ncol) {
        col -= ncol;
        ++j2;
      }
    }
  }
  __syncthreads();
  {
    int k1 = (int)threadIdx.x / ncol, col = (int)threadIdx.x - k1 * ncol;
    while (k1 < N1) {
      R2 y[N2];
#pragma unroll
      for (int j2 = 0; j2 < N2; ++j2) y[j2] = tmp[(j2 * N1 + k1) * ncol + col];
      R2 s0 = y[0];
#pragma unroll
      for (int j2 = 1; j2 < N2; ++j2) {
        s0.x += y[j2].x;
        s0.y += y[j2].y;
      }
      out[k1 * ncol + col] = s0;
#pragma unroll
      for (int k2 = 1; 2 * k2 < N2; ++k2) {
        R2 C = y[0], S;
        S.x = 0;
        S.y = 0;
#pragma unroll
        for (int j2 = 1; j2 < N2; ++j2) {
          const R2 ww = w2[(j2 * k2) % N2];
          C.x += y[j2].x * ww.x;
          C.y += y[j2].y * ww.x;
          S.x += y[j2].x * ww.y;
          S.y += y[j2].y * ww.y;
        }
        R2 a, b;
        a.x = C.x - S.y;
        a.y = C.y + S.x;
        b.x = C.x + S.y;
        b.y = C.y - S.x;
        out[(k1 + N1 * k2) * ncol + col] = a;
        out[(k1 + N1 * (N2 - k2)) * ncol + col] = b;
      }
      col += step_c;
      k1 += step_r;
      if (col >= ncol) {
        col -= ncol;
        ++k1;
      }
    }
  }
  __syncthreads();
  (void)n;
  return out;
}

// FP64: the inputs fold as well.  With e_j = x_j + x_(M-j), o_j = x_j - x_(M-j),
//   C = x_0 + sum_(j <= h) e_j Re W^(jk),   S = sum_(j <= h) o_j Im W^(jk),   h = (M - 1) / 2,
// a quarter of the plain sum's multiply-adds (the FP64 pipe bounds these
// transforms: exchange of H8 szv at 41^3 9.5 -> 7.3 ms a run, Hartree potential
// at 65^3 0.14 -> 0.12 ms), with as many roundings a term and half as many terms.
template <int M, typename Load, typename Tw, typename Emit>
__device__ __forceinline__ void fold_dft(Load load, Tw tw, Emit emit) {  // M at compile time
  constexpr int H = (M - 1) / 2;
  const double2 x0 = load(0);
  double2 e[H], o[H], s = x0;
#pragma unroll
  for (int j = 0; j < H; ++j) {
    const double2 a = load(j + 1), b = load(M - 1 - j);
    e[j] = make_double2(a.x + b.x, a.y + b.y);
    o[j] = make_double2(a.x - b.x, a.y - b.y);
    s.x += e[j].x;
    s.y += e[j].y;
  }
  emit(0, s);
#pragma unroll
  for (int k = 1; k <= H; ++k) {
    double2 C = x0, S = make_double2(0.0, 0.0);
#pragma unroll
    for (int j = 0; j < H; ++j) {
      const double2 ww = tw(((j + 1) * k) % M);
      C.x = fma(e[j].x, ww.x, C.x);
      C.y = fma(e[j].y, ww.x, C.y);
      S.x = fma(o[j].x, ww.y, S.x);
      S.y = fma(o[j].y, ww.y, S.y);
    }
    emit(k, make_double2(C.x - S.y, C.y + S.x));
    emit(M - k, make_double2(C.x + S.y, C.y - S.x));
  }
}

constexpr int kFoldMax = 25;  // largest factor held in registers

template <typename Load, typename Tw, typename Emit>
__device__ __forceinline__ void fold_dft_any(int M, Load load, Tw tw, Emit emit) {
  constexpr int HM = (kFoldMax - 1) / 2;
  const int H = (M - 1) / 2;
  const double2 x0 = load(0);
  double2 e[HM], o[HM], s = x0;
#pragma unroll
  for (int j = 0; j < HM; ++j)
    if (j < H) {
      const double2 a = load(j + 1), b = load(M - 1 - j);
      e[j] = make_double2(a.x + b.x, a.y + b.y);
      o[j] = make_double2(a.x - b.x, a.y - b.y);
      s.x += e[j].x;
      s.y += e[j].y;
    }
  emit(0, s);
  for (int k = 1; k <= H; ++k) {
    double2 C = x0, S = make_double2(0.0, 0.0);
    int t = 0;
#pragma unroll
    for (int j = 0; j < HM; ++j)
      if (j < H) {
        t += k;
        if (t >= M) t -= M;
        const double2 ww = tw(t);
        C.x = fma(e[j].x, ww.x, C.x);
        C.y = fma(e[j].y, ww.x, C.y);
        S.x = fma(o[j].x, ww.y, S.x);
        S.y = fma(o[j].y, ww.y, S.y);
      }
    emit(k, make_double2(C.x - S.y, C.y + S.x));
    emit(M - k, make_double2(C.x + S.y, C.y - S.x));
  }
}

// n = N1 N2 at compile time (as dft_axis0_fixed); the transform is in place
template <int N1, int N2>
__device__ double2 *fold_axis0_fixed(double2 *buf, double2 *tmp, int ncol, const double2 *w) {
  double2 w1[(N1 + 1) / 2], w2[(N2 + 1) / 2];  // the other halves are their conjugates
#pragma unroll
  for (int m = 0; m < (N1 + 1) / 2; ++m) w1[m] = w[N2 * m];
  for (int it = threadIdx.x; it < N2 * ncol; it += blockDim.x) {
    const int j2 = it / ncol, col = it - j2 * ncol;
    fold_dft<N1>([&](int j1) { return buf[(N2 * j1 + j2) * ncol + col]; },
                 [&](int m) { return 2 * m < N1 ? w1[m] : make_double2(w1[N1 - m].x, -w1[N1 - m].y); },
                 [&](int k1, double2 v) { tmp[(j2 * N1 + k1) * ncol + col] = k1 ? cmul(v, w[j2 * k1]) : v; });
  }
  __syncthreads();
#pragma unroll
  for (int m = 0; m < (N2 + 1) / 2; ++m) w2[m] = w[N1 * m];
  for (int it = threadIdx.x; it < N1 * ncol; it += blockDim.x) {
    const int k1 = it / ncol, col = it - k1 * ncol;
    fold_dft<N2>([&](int j2) { return tmp[(j2 * N1 + k1) * ncol + col]; },
                 [&](int m) { return 2 * m < N2 ? w2[m] : make_double2(w2[N2 - m].x, -w2[N2 - m].y); },
                 [&](int k2, double2 v) { buf[(k1 + N1 * k2) * ncol + col] = v; });
  }
  __syncthreads();
  return buf;
}

static __device__ double2 *fold_axis0_any(double2 *buf, double2 *tmp, int n, int ncol, int n1, const double2 *w) {
  const int n2 = n1 > 1 ? n / n1 : n;
  if (n1 == 1 || n2 > kFoldMax) {  // n1 <= n2
    const int h = (n - 1) / 2;
    for (int it = threadIdx.x; it < h * ncol; it += blockDim.x) {
      const int j = it / ncol + 1, col = it - (j - 1) * ncol;
      const double2 a = buf[j * ncol + col], b = buf[(n - j) * ncol + col];
      buf[j * ncol + col] = make_double2(a.x + b.x, a.y + b.y);
      buf[(n - j) * ncol + col] = make_double2(a.x - b.x, a.y - b.y);
    }
    __syncthreads();
    for (int it = threadIdx.x; it < (h + 1) * ncol; it += blockDim.x) {
      const int k = it / ncol, col = it - k * ncol;
      double2 C = buf[col], S = make_double2(0.0, 0.0);
      int t = 0;
      for (int j = 1; j <= h; ++j) {
        t += k;
        if (t >= n) t -= n;
        const double2 e = buf[j * ncol + col], o = buf[(n - j) * ncol + col], ww = w[t];
        C.x = fma(e.x, ww.x, C.x);
        C.y = fma(e.y, ww.x, C.y);
        S.x = fma(o.x, ww.y, S.x);
        S.y = fma(o.y, ww.y, S.y);
      }
      tmp[k * ncol + col] = make_double2(C.x - S.y, C.y + S.x);
      if (k > 0) tmp[(n - k) * ncol + col] = make_double2(C.x + S.y, C.y - S.x);
    }
    __syncthreads();
    return tmp;
  }
  for (int it = threadIdx.x; it < n2 * ncol; it += blockDim.x) {
    const int j2 = it / ncol, col = it - j2 * ncol;
    fold_dft_any(n1, [&](int j1) { return buf[(n2 * j1 + j2) * ncol + col]; }, [&](int m) { return w[n2 * m]; },
                 [&](int k1, double2 v) { tmp[(j2 * n1 + k1) * ncol + col] = cmul(v, w[j2 * k1]); });
  }
  __syncthreads();
  for (int it = threadIdx.x; it < n1 * ncol; it += blockDim.x) {
    const int k1 = it / ncol, col = it - k1 * ncol;
    fold_dft_any(n2, [&](int j2) { return tmp[(j2 * n1 + k1) * ncol + col]; }, [&](int m) { return w[n1 * m]; },
                 [&](int k2, double2 v) { buf[(k1 + n1 * k2) * ncol + col] = v; });
  }
  __syncthreads();
  return buf;
}

// DFT along axis 0 of buf [n][ncol], n odd, with tmp of the same size: returns
// the one of the two that holds the result.  The fixed-size transforms for 25,
// 33, 49, 65 and 81 points (the grids of the benchmark systems), the generic routine
// otherwise: two factors in loops over the largest length a factor may have, primes
// and long factors as direct sums.  What that costs, FP64 Hartree potential (five
// passes): 45 / 49 / 51 / 55 points 97 / 72 / 164 / 135 us, 61 / 63 / 65 / 69 134 / 137 /
// 106 / 215, 73 / 75 / 77 / 81 256 / 173 / 152 / 168.
template <typename R, typename R2>
__device__ R2 *dft_axis0(R2 *buf, R2 *tmp, int n, int ncol, int n1, const R2 *w) {
  if constexpr (sizeof(R) == 8) {
    switch (n) {
      case 25: return fold_axis0_fixed<5, 5>(buf, tmp, ncol, w);
      case 33: return fold_axis0_fixed<3, 11>(buf, tmp, ncol, w);
      case 49: return fold_axis0_fixed<7, 7>(buf, tmp, ncol, w);
      case 65: return fold_axis0_fixed<5, 13>(buf, tmp, ncol, w);
      case 81: return fold_axis0_fixed<9, 9>(buf, tmp, ncol, w);
      default: return fold_axis0_any(buf, tmp, n, ncol, n1, w);
    }
  } else {
    switch (n) {
      case 25: return dft_axis0_fixed<R, R2, 5, 5>(buf, tmp, buf, ncol, w);
      case 33: return dft_axis0_fixed<R, R2, 3, 11>(buf, tmp, buf, ncol, w);
      case 49: return dft_axis0_fixed<R, R2, 7, 7>(buf, tmp, buf, ncol, w);
      case 65: return dft_axis0_fixed<R, R2, 5, 13>(buf, tmp, buf, ncol, w);
      case 81: return dft_axis0_fixed<R, R2, 9, 9>(buf, tmp, buf, ncol, w);
      default: return dft_axis0_any<R, R2>(buf, tmp, buf, n, ncol, n1, w);
    }
  }
}

}  // namespace exx
}  // namespace hqcgb
