// Register-resident two-pass FFT engine for line lengths M = R1 * R2.
//
// A CTA transforms L lines at once; each thread owns one line of one stage
// and keeps its R1 or R2 points in registers. With n = R2 n1 + n2 and
// k = k1 + R1 k2 the DFT factors as (the "four-step" decomposition)
//   X[k1 + R1 k2] = sum_n2 W_R2^{n2 k2} W_M^{n2 k1} sum_n1 W_R1^{n1 k1} x[R2 n1 + n2]
// stage 1: thread (line, n2) does the R1-point DFT over n1 (stride R2);
// stage 2: thread (line, k1) does the R2-point DFT over n2 with the twiddles
// W_M^{n2 k1} merged in, leaving X[k1 + R1 k2] in its registers. The inverse
// runs the same factorisation backwards from that register layout (R2-point
// DFTs in stage A, twiddles and R1-point DFTs in stage B), so a forward transform,
// a pointwise multiply and an inverse transform cost two shared-memory round
// trips in total. The in-register DFTs are unrolled with compile-time
// twiddles (twiddles.cuh). The first N = M/2 inputs are the only nonzero
// ones in the zero-padded forward transforms (R1 is even, so they are
// n1 < R1/2), and the inverse keeps only the first M/2 outputs.
#pragma once
#include "fft.cuh"
#include "twiddles.cuh"

namespace gato {
namespace fft2 {

template <int R> struct Split;
template <> struct Split<9> { static constexpr int A = 3, B = 3; };
template <> struct Split<18> { static constexpr int A = 2, B = 9; };
template <> struct Split<6> { static constexpr int A = 2, B = 3; };
template <> struct Split<10> { static constexpr int A = 2, B = 5; };
template <> struct Split<12> { static constexpr int A = 4, B = 3; };
template <> struct Split<14> { static constexpr int A = 2, B = 7; };
template <> struct Split<16> { static constexpr int A = 4, B = 4; };
template <> struct Split<20> { static constexpr int A = 4, B = 5; };

// a * exp(DIR * 2 pi i e / R), e a compile-time constant after unrolling
template <typename T2, int R, int DIR>
__device__ __forceinline__ T2 ctw(T2 a, int e) {
  using Rt = typename CT<T2>::R;
  if (e == 0) return a;
  if ((4 * e) % R == 0) {   // a quarter-turn multiple: -1 or +-i, exact sign and swap
    const int k = 4 * e / R;
    T2 r;
    if (k == 2) {
      r.x = -a.x;
      r.y = -a.y;
    } else if ((k == 1) == (DIR > 0)) {   // * i
      r.x = -a.y;
      r.y = a.x;
    } else {                              // * -i
      r.x = a.y;
      r.y = -a.x;
    }
    return r;
  }
  const Rt c = (Rt)TwC<R>::c(e);
  const Rt s = (Rt)DIR * (Rt)TwC<R>::s(e);
  T2 r;
  r.x = a.x * c - a.y * s;
  r.y = a.x * s + a.y * c;
  return r;
}

// ---- butterflies with the twiddle fused in -------------------------------------------------
// a +- w b with w = c (1 + i t), t = Im w / Re w: p = (1 + i t) b takes two multiply-adds and a +- c p
// four, six where a rotation and a butterfly take eight. (Merging twiddles into multiply-adds: Linzer and
// Feig, IEEE Trans. Signal Process. 41, 1993; here with the cosine kept as the butterfly's own factor, so
// nothing is rescaled and a large t costs no accuracy: p's rounding error times c is that of s b.) Where
// c = 0 the tables and constants keep a c far below the rounding, so that c t = s. The twiddles of a
// radix-4 step with inputs u0, W u1, W^2 u2, W^3 u3 all sit in such butterflies (W^2 twice, W, i W): 24
// operations where three rotations and the DFT take 28. The FP64 passes are bound by that count:
// a 256-point transform with half its inputs zero takes 4928 operations instead of 5568 (FP64 energy terms
// of water at 128^3: 7839 -> 6717 us). FP32 passes, bound by memory and latency, keep separate rotations:
// merged, they measured 217 us where a 128^3 matvec takes 209, and 182 instead of 160 in the y forward of
// five 160^3 fields (registers).
template <typename T2>
constexpr bool kMergeTw = sizeof(T2) == 16;
template <typename T2>
__device__ __forceinline__ void bfly(T2 a, T2 b, typename CT<T2>::R c, typename CT<T2>::R t, T2& plus, T2& minus) {
  T2 p;
  p.x = b.x - t * b.y;
  p.y = b.y + t * b.x;
  plus.x = a.x + c * p.x;
  plus.y = a.y + c * p.y;
  minus.x = a.x - c * p.x;
  minus.y = a.y - c * p.y;
}
// a +- DIR i w b
template <typename T2, int DIR>
__device__ __forceinline__ void bfly_i(T2 a, T2 b, typename CT<T2>::R c, typename CT<T2>::R t, T2& plus, T2& minus) {
  T2 p;
  p.x = b.x - t * b.y;
  p.y = b.y + t * b.x;
  const typename CT<T2>::R d = DIR > 0 ? c : -c;
  plus.x = a.x - d * p.y;
  plus.y = a.y + d * p.x;
  minus.x = a.x + d * p.y;
  minus.y = a.y - d * p.x;
}
// a +- exp(DIR 2 pi i e / R) b, e a compile-time constant after unrolling (quarter turns exact)
template <typename T2, int R, int DIR>
__device__ __forceinline__ void bfly_k(T2 a, T2 b, int e, T2& plus, T2& minus) {
  using Rt = typename CT<T2>::R;
  e %= R;
  if ((4 * e) % R == 0) {
    const int k = 4 * e / R;
    const T2 r = k % 2 == 0 ? b : cmul_i(b, DIR);
    const T2 hi = cadd(a, r), lo = csub(a, r);
    plus = k < 2 ? hi : lo;
    minus = k < 2 ? lo : hi;
  } else {
    const double c = TwC<R>::c(e), s = DIR * TwC<R>::s(e);
    bfly(a, b, (Rt)c, (Rt)(s / c), plus, minus);
  }
}
// v0..v3 = DFT4 of (u0, w u1, w^2 u2, w^3 u3), w = exp(DIR 2 pi i e / R)
template <typename T2, int R, int DIR>
__device__ __forceinline__ void dft4_k(T2 u0, T2 u1, T2 u2, T2 u3, int e, T2& v0, T2& v1, T2& v2, T2& v3) {
  T2 t0, t1, s0, s1;
  bfly_k<T2, R, DIR>(u0, u2, 2 * e, t0, t1);
  bfly_k<T2, R, DIR>(u1, u3, 2 * e, s0, s1);
  bfly_k<T2, R, DIR>(t0, s0, e, v0, v2);
  bfly_k<T2, R, DIR>(t1, s1, e + R / 4, v1, v3);
}

template <typename T2, int R, int DIR>
__device__ __forceinline__ void rdft(T2* v);

// Second layer of an R = A B point DFT: v[k1 + A k2] from the inner transforms y[n2 * A + k1].
template <typename T2, int R, int A, int B, int DIR>
__device__ __forceinline__ void outer_layer(const T2* y, T2* v) {
#pragma unroll
  for (int k1 = 0; k1 < A; ++k1) {
    if constexpr (B == 2 && kMergeTw<T2>) {
      bfly_k<T2, R, DIR>(y[k1], y[A + k1], k1, v[k1], v[k1 + A]);
    } else if constexpr (B == 4 && kMergeTw<T2>) {
      dft4_k<T2, R, DIR>(y[k1], y[A + k1], y[2 * A + k1], y[3 * A + k1], k1, v[k1], v[k1 + A], v[k1 + 2 * A],
                         v[k1 + 3 * A]);
    } else {
      T2 u[B];
#pragma unroll
      for (int n2 = 0; n2 < B; ++n2) u[n2] = ctw<T2, R, DIR>(y[n2 * A + k1], (n2 * k1) % R);
      rdft<T2, B, DIR>(u);
#pragma unroll
      for (int k2 = 0; k2 < B; ++k2) v[k1 + A * k2] = u[k2];
    }
  }
}

// In-place R-point DFT in natural order; DIR = -1 forward, +1 inverse (unscaled).
template <typename T2, int R, int DIR>
__device__ __forceinline__ void rdft(T2* v) {
  if constexpr (R == 1) {
  } else if constexpr (R == 2) {
    dft2(v);
  } else if constexpr (R == 4) {
    dft4(v[0], v[1], v[2], v[3], DIR);
  } else if constexpr (R == 8 && !kMergeTw<T2>) {
    dft8(v, DIR);
  } else if constexpr (R == 8) {
    T2 y[8] = {v[0], v[2], v[4], v[6], v[1], v[3], v[5], v[7]};
    dft4(y[0], y[1], y[2], y[3], DIR);
    dft4(y[4], y[5], y[6], y[7], DIR);
    outer_layer<T2, 8, 4, 2, DIR>(y, v);
  } else if constexpr (R == 3 || R == 5 || R == 7) {
    dft_odd<T2, R>(v, DIR);
  } else {
    constexpr int A = Split<R>::A, B = Split<R>::B;
    T2 y[R];
#pragma unroll
    for (int n2 = 0; n2 < B; ++n2) {
      T2 u[A];
#pragma unroll
      for (int n1 = 0; n1 < A; ++n1) u[n1] = v[B * n1 + n2];
      rdft<T2, A, DIR>(u);
#pragma unroll
      for (int k1 = 0; k1 < A; ++k1) y[n2 * A + k1] = u[k1];
    }
    outer_layer<T2, R, A, B, DIR>(y, v);
  }
}

// The same DFT when only v[0 .. R/2) is nonzero (the zero-padded half of a
// Hockney transform). For R = A B with A even the zeros are the upper half of
// every inner A-point DFT, so the saving recurses down to the base radices.
template <typename T2, int R, int DIR>
__device__ __forceinline__ void rdft_half(T2* v) {
  if constexpr (R == 2) {
    v[1] = v[0];
  } else if constexpr (R == 4) {
    const T2 a = v[0], b = v[1];
    const T2 ib = cmul_i(b, DIR);
    v[0] = cadd(a, b);
    v[1] = cadd(a, ib);
    v[2] = csub(a, b);
    v[3] = csub(a, ib);
  } else if constexpr (R == 8) {
    // even/odd split: E = DFT4(v0, v2, 0, 0), O = DFT4(v1, v3, 0, 0)
    T2 e[8] = {v[0], v[2], v[0], v[0], v[1], v[3], v[1], v[1]};
    T2* o = e + 4;
    rdft_half<T2, 4, DIR>(e);
    rdft_half<T2, 4, DIR>(o);
    if constexpr (kMergeTw<T2>) {
      outer_layer<T2, 8, 4, 2, DIR>(e, v);
    } else {
      using Rt = typename CT<T2>::R;
      const Rt s = (Rt)0.70710678118654752440;
      T2 w1, w3;
      w1.x = s;
      w1.y = (Rt)DIR * s;
      w3.x = -s;
      w3.y = (Rt)DIR * s;
      o[1] = cmul(o[1], w1);
      o[2] = cmul_i(o[2], DIR);
      o[3] = cmul(o[3], w3);
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        v[q] = cadd(e[q], o[q]);
        v[q + 4] = csub(e[q], o[q]);
      }
    }
  } else {
    constexpr int A = Split<R>::A, B = Split<R>::B;
    static_assert(A % 2 == 0, "half-input DFT needs an even inner radix");
    T2 y[R];
#pragma unroll
    for (int n2 = 0; n2 < B; ++n2) {
      T2 u[A];
#pragma unroll
      for (int n1 = 0; n1 < A / 2; ++n1) u[n1] = v[B * n1 + n2];
      rdft_half<T2, A, DIR>(u);
#pragma unroll
      for (int k1 = 0; k1 < A; ++k1) y[n2 * A + k1] = u[k1];
    }
    outer_layer<T2, R, A, B, DIR>(y, v);
  }
}

template <int R1, int R2> struct Shape {
  static constexpr int M = R1 * R2;
  static constexpr int RMAX = R1 > R2 ? R1 : R2;
};

// ---- stage twiddles ---------------------------------------------------------------------
// FP32: one table for both directions, row k1 holds exp(-2 pi i n2 k1 / M) as (c, s) for n2 < R2; the
// forward multiplies before stage 2's DFT, the inverse after stage A's (twiddle_row).
// FP64: the twiddles between the stages, exp(-+2 pi i n2 k1 / M), are inputs of the second stage's DFT and
// merge into its butterflies: forward in stage 2 (R2 points, row k1 of table F), inverse in stage B (R1 points,
// row n2 of table I). With R = A B as the DFT splits it, the inner A-point DFTs (A = 2 or 4) take the
// inputs B n1' + n2' without their common factor w^n2', w = exp(-2 pi i r / M) for row r, which the outer
// layer's twiddles (w exp(-2 pi i k1' / R))^n2' then carry. A row holds, forward signs:
//   w^B and, for A = 4, w^2B, as (c, t);
//   B = 2: w W_R^k1' as (c, t), k1' < A;  B = 4: w W_R^k1' and its square as (c, t), k1' < A;
//   other B > 1: (w W_R^k1')^n2' as (c, s), n2' = 1 .. B - 1, for each k1' < A.
__host__ __device__ constexpr int tw_a(int R) { return R % 4 == 0 ? 4 : 2; }
__host__ __device__ constexpr int tw_b(int R) { return R / tw_a(R); }
__host__ __device__ constexpr int tw_inner(int R) { return tw_a(R) == 4 ? 2 : 1; }
__host__ __device__ constexpr int tw_count(int R) {
  return tw_inner(R) + (tw_b(R) == 1 ? 0 : tw_b(R) == 2 ? tw_a(R) : tw_b(R) == 4 ? 2 * tw_a(R) : tw_a(R) * (tw_b(R) - 1));
}
// Row strides in entries: FP32 rows (twiddles move in 16-byte pairs) start on 16-byte boundaries and
// neighbouring rows, which consecutive lanes of the row passes read, in different banks; FP64 rows (16-byte
// entries) have an odd stride.
__host__ __device__ constexpr int tw_row_stride(bool f32, int R) {
  return f32 ? ((R / 2) % 2 == 0 ? R + 2 : R) : tw_count(R) | 1;
}
// Table sizes of a shape. FP64: F (R1 rows of R2's twiddles) then, unless it is the same, I (R2 rows of
// R1's). FP32: the one table is both.
template <typename T2, int R1, int R2> struct TwTab {
  static constexpr bool one = sizeof(T2) == 8 || R1 == R2;
  static constexpr int SF = tw_row_stride(sizeof(T2) == 8, R2), SI = tw_row_stride(sizeof(T2) == 8, R1);
  static constexpr int NF = R1 * SF, NI = one ? NF : R2 * SI;
  static constexpr int OI = one ? 0 : NF;              // start of I in the table
  static constexpr int N = one ? NF : NF + NI;         // both
};

// a * w for w = (c, s) = exp(-2 pi i e / M) (DIR = -1) or its conjugate (DIR = +1).
template <typename T2, int DIR>
__device__ __forceinline__ T2 rtw(T2 a, typename CT<T2>::R c, typename CT<T2>::R s) {
  T2 w;
  w.x = c;
  w.y = DIR > 0 ? -s : s;
  return cmul(a, w);
}

// X[n2] *= W_M^{DIR n2 k1} for n2 = 1 .. R2-1 from row k1 of the FP32 stage table, read in 16-byte pairs
// (R2 is even and every row starts on a 16-byte boundary); n2 = 0 is the identity and skipped.
template <typename T2, int R2, int DIR>
__device__ __forceinline__ void twiddle_row(T2* X, const T2* row) {
  static_assert(sizeof(T2) == 8 && R2 % 2 == 0, "paired FP32 twiddle loads need an even R2");
  const float4* r4 = reinterpret_cast<const float4*>(row);
#pragma unroll
  for (int p = 0; p < R2 / 2; ++p) {
    const float4 w = r4[p];
    if (p > 0) X[2 * p] = rtw<T2, DIR>(X[2 * p], w.x, w.y);
    X[2 * p + 1] = rtw<T2, DIR>(X[2 * p + 1], w.z, w.w);
  }
}

// dft4_k with a table twiddle: w and w2 = w^2 as (c, t).
template <typename T2, int DIR>
__device__ __forceinline__ void dft4_t(T2 u0, T2 u1, T2 u2, T2 u3, T2 w, T2 w2, T2& v0, T2& v1, T2& v2, T2& v3) {
  if (DIR > 0) {
    w.y = -w.y;
    w2.y = -w2.y;
  }
  T2 t0, t1, s0, s1;
  bfly(u0, u2, w2.x, w2.y, t0, t1);
  bfly(u1, u3, w2.x, w2.y, s0, s1);
  bfly(t0, s0, w.x, w.y, v0, v2);
  bfly_i<T2, DIR>(t1, s1, w.x, w.y, v1, v3);
}

// In-place R-point DFT of v[n] exp(DIR 2 pi i n r / M), row = row r of the FP64 stage table.
template <typename T2, int R, int DIR>
__device__ __forceinline__ void tw_rdft(T2* v, const T2* row) {
  constexpr int A = tw_a(R), B = tw_b(R), I = tw_inner(R);
  T2 y[R];
  if constexpr (A == 4) {
    const T2 w = row[0], w2 = row[1];
#pragma unroll
    for (int n2 = 0; n2 < B; ++n2)
      dft4_t<T2, DIR>(v[n2], v[B + n2], v[2 * B + n2], v[3 * B + n2], w, w2, y[n2 * 4], y[n2 * 4 + 1], y[n2 * 4 + 2],
                      y[n2 * 4 + 3]);
  } else {
    const T2 w = row[0];
#pragma unroll
    for (int n2 = 0; n2 < B; ++n2) bfly(v[n2], v[B + n2], w.x, DIR > 0 ? -w.y : w.y, y[n2 * 2], y[n2 * 2 + 1]);
  }
#pragma unroll
  for (int k1 = 0; k1 < A; ++k1) {
    if constexpr (B == 1) {
      v[k1] = y[k1];
    } else if constexpr (B == 2) {
      const T2 w = row[I + k1];
      bfly(y[k1], y[A + k1], w.x, DIR > 0 ? -w.y : w.y, v[k1], v[k1 + A]);
    } else if constexpr (B == 4) {
      const T2 w = row[I + 2 * k1], w2 = row[I + 2 * k1 + 1];
      dft4_t<T2, DIR>(y[k1], y[A + k1], y[2 * A + k1], y[3 * A + k1], w, w2, v[k1], v[k1 + A], v[k1 + 2 * A],
                      v[k1 + 3 * A]);
    } else {
      T2 u[B];
      u[0] = y[k1];
#pragma unroll
      for (int n2 = 1; n2 < B; ++n2) {
        const T2 w = row[I + k1 * (B - 1) + n2 - 1];
        u[n2] = rtw<T2, DIR>(y[n2 * A + k1], w.x, w.y);
      }
      rdft<T2, B, DIR>(u);
#pragma unroll
      for (int k2 = 0; k2 < B; ++k2) v[k1 + A * k2] = u[k2];
    }
  }
}

// The twiddles and DFT of stage 2 (row k1) and of stage B (row n2), and stage A's DFT.
template <typename T2, int R1, int R2>
__device__ __forceinline__ void stage2_dft(T2* X, int k1, const T2* tw) {
  const T2* row = tw + k1 * TwTab<T2, R1, R2>::SF;
  if constexpr (kMergeTw<T2>) {
    tw_rdft<T2, R2, -1>(X, row);
  } else {
    twiddle_row<T2, R2, -1>(X, row);
    rdft<T2, R2, -1>(X);
  }
}
template <typename T2, int R1, int R2>
__device__ __forceinline__ void stageA_dft(T2* X, int k1, const T2* tw) {
  rdft<T2, R2, +1>(X);
  if constexpr (!kMergeTw<T2>) twiddle_row<T2, R2, +1>(X, tw + k1 * TwTab<T2, R1, R2>::SF);
}
template <typename T2, int R1, int R2>
__device__ __forceinline__ void stageB_dft(T2* w, int n2, const T2* tw) {
  if constexpr (kMergeTw<T2>) tw_rdft<T2, R1, +1>(w, tw + n2 * TwTab<T2, R1, R2>::SI);
  else rdft<T2, R1, +1>(w);
}

// Stage 1 of the forward transform for the item (line, n2): reads x[R2 n1 + n2]
// through `get` (only n1 < R1/2 when HALF), writes Y[n2][k1] to buf.
template <typename T2, int R1, int R2, bool HALF, typename Get>
__device__ __forceinline__ void fwd_stage1(T2* buf, int LP, int line, int n2, Get get) {
  T2 v[R1];
#pragma unroll
  for (int n1 = 0; n1 < R1; ++n1) {
    if (!HALF || n1 < R1 / 2) v[n1] = get(R2 * n1 + n2);
    else v[n1].x = v[n1].y = 0;
  }
  if constexpr (HALF) rdft_half<T2, R1, -1>(v);
  else rdft<T2, R1, -1>(v);
#pragma unroll
  for (int k1 = 0; k1 < R1; ++k1) buf[(n2 * R1 + k1) * LP + line] = v[k1];
}

// Stage 2 of the forward transform for (line, k1): X[k2] = spectrum at k1 + R1 k2.
// tw is stage-twiddle table F (FP32: the one table).
template <typename T2, int R1, int R2>
__device__ __forceinline__ void fwd_stage2(const T2* buf, int LP, int line, int k1, const T2* tw,
                                           T2* X) {
#pragma unroll
  for (int n2 = 0; n2 < R2; ++n2) X[n2] = buf[(n2 * R1 + k1) * LP + line];
  stage2_dft<T2, R1, R2>(X, k1, tw);
}

// Inverse stage A for (line, k1) holding X[k2] = spectrum at k1 + R1 k2: writes Z to buf.
template <typename T2, int R1, int R2>
__device__ __forceinline__ void inv_stageA(T2* buf, int LP, int line, int k1, const T2* tw, T2* X) {
  stageA_dft<T2, R1, R2>(X, k1, tw);
#pragma unroll
  for (int n2 = 0; n2 < R2; ++n2) buf[(n2 * R1 + k1) * LP + line] = X[n2];
}

// Inverse stage B for (line, n2): outputs x[n2 + R2 n1] through `put` (n1 < R1/2 when HALF); tw is table
// I (FP32: unused).
template <typename T2, int R1, int R2, bool HALF, typename Put>
__device__ __forceinline__ void inv_stageB(const T2* buf, int LP, int line, int n2, const T2* tw, Put put) {
  T2 w[R1];
#pragma unroll
  for (int k1 = 0; k1 < R1; ++k1) w[k1] = buf[(n2 * R1 + k1) * LP + line];
  stageB_dft<T2, R1, R2>(w, n2, tw);
#pragma unroll
  for (int n1 = 0; n1 < R1; ++n1)
    if (!HALF || n1 < R1 / 2) put(n2 + R2 * n1, w[n1]);
}

// ---- row passes (the contiguous z axis) ----------------------------------------
// Line `line`'s stage element (n2, k1) sits at line * LS + n2 * (R1 + 1) + k1.
// Stages 1 and B run with n2 across the lanes, stages 2 and A with k1 across
// the lanes: both orders walk the buffer with odd element strides (no bank
// conflicts), stage 2 leaves spectrum entries k1 + R1 k2 that consecutive
// lanes store to consecutive addresses, and stage B leaves outputs
// n2 + R2 n1 in the same coalesced order, so no transpose through shared
// memory is needed on either side.
template <int R1, int R2> struct RowBuf {
  static constexpr int LS = R2 * (R1 + 1);
  static __device__ __forceinline__ int at(int line, int n2, int k1) {
    return line * LS + n2 * (R1 + 1) + k1;
  }
};

// Stage 1 for (line, n2): v[n1] = x[R2 n1 + n2] (n1 < R1/2 only when HALF).
template <typename T2, int R1, int R2, bool HALF>
__device__ __forceinline__ void row_fwd_stage1(T2* buf, int line, int n2, T2* v) {
  if constexpr (HALF) {
#pragma unroll
    for (int n1 = R1 / 2; n1 < R1; ++n1) v[n1].x = v[n1].y = 0;
    rdft_half<T2, R1, -1>(v);
  } else {
    rdft<T2, R1, -1>(v);
  }
#pragma unroll
  for (int k1 = 0; k1 < R1; ++k1) buf[RowBuf<R1, R2>::at(line, n2, k1)] = v[k1];
}

// Stage 2 for (line, k1): X[k2] = spectrum at k1 + R1 k2.
template <typename T2, int R1, int R2>
__device__ __forceinline__ void row_fwd_stage2(const T2* buf, int line, int k1, const T2* tw, T2* X) {
#pragma unroll
  for (int n2 = 0; n2 < R2; ++n2) X[n2] = buf[RowBuf<R1, R2>::at(line, n2, k1)];
  stage2_dft<T2, R1, R2>(X, k1, tw);
}

// Inverse stage A for (line, k1) holding X[k2] = spectrum at k1 + R1 k2.
template <typename T2, int R1, int R2>
__device__ __forceinline__ void row_inv_stageA(T2* buf, int line, int k1, const T2* tw, T2* X) {
  stageA_dft<T2, R1, R2>(X, k1, tw);
#pragma unroll
  for (int n2 = 0; n2 < R2; ++n2) buf[RowBuf<R1, R2>::at(line, n2, k1)] = X[n2];
}

// Inverse stage B for (line, n2): w[n1] = output at z = n2 + R2 n1; tw is table I
// (FP32: unused).
template <typename T2, int R1, int R2>
__device__ __forceinline__ void row_inv_stageB(const T2* buf, int line, int n2, const T2* tw, T2* w) {
#pragma unroll
  for (int k1 = 0; k1 < R1; ++k1) w[k1] = buf[RowBuf<R1, R2>::at(line, n2, k1)];
  stageB_dft<T2, R1, R2>(w, n2, tw);
}

}  // namespace fft2
}  // namespace gato
