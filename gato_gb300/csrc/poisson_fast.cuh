// Pair-solve pipeline kernels on the register-resident two-pass FFT engine
// (fft2.cuh), one instantiation per supported doubled-grid size M.
#pragma once
#include <atomic>
#include "fft2.cuh"
#include "poisson.cuh"
#include "ptx.cuh"

namespace gato {
namespace fast {

using namespace fft2;


// The COUNT-entry stage-twiddle table split into a register prefetch at
// kernel entry and a shared-memory store placed after the kernel's own field
// loads are issued, so the two global latencies overlap instead of adding up.
template <typename T2, int COUNT, int NT>
struct TwPrefetch {
  static constexpr int K = (COUNT + NT - 1) / NT;
  T2 v[K];
  __device__ __forceinline__ explicit TwPrefetch(const T2* tw) {
#pragma unroll
    for (int k = 0; k < K; ++k) {
      const int i = threadIdx.x + k * NT;
      if (i < COUNT) v[k] = tw[i];
    }
  }
  __device__ __forceinline__ void store(T2* tws) const {
#pragma unroll
    for (int k = 0; k < K; ++k) {
      const int i = threadIdx.x + k * NT;
      if (i < COUNT) tws[i] = v[k];
    }
  }
};

// The last column of a lone real field's half spectrum (ColGeom::edge): a whole tile for it would do
// L - 1 columns' work for nothing, and the FP64 passes are bound by just that work (72 columns instead
// of 65 at N = 64; Hartree solve at 80^3 414 -> 358 us, 96^3 530 -> 497, 128^3 1163 -> 1123). So the lines of tile `edge` are L outer indices of that one
// column (past the end: the last one again, which stores the same values). True: no such index.
template <int L>
__device__ __forceinline__ bool edge_tile(const ColGeom& g, int& outer, int& col, int line) {
  if (g.edge == 0 || (int)blockIdx.y != g.edge) return false;
  if (outer * L >= (int)gridDim.x) return true;
  outer = min(outer * L + line, (int)gridDim.x - 1);
  col = g.edge * L;
  return false;
}

// Strided-line passes (y forward, x forward * kernel * x inverse, y inverse).
// FULL: every CTA has L real columns (ncols % L == 0), so no per-access guard.
template <typename T, int R1, int R2, int L, int MODE, bool FULL>
__global__ void __launch_bounds__(L * Shape<R1, R2>::RMAX)
    k_cols(const typename Cplx<T>::type* in, typename Cplx<T>::type* out, ColGeom g,
           const typename Cplx<T>::type* tw, const T* ghat, int H) {
  using T2 = typename Cplx<T>::type;
  constexpr int M = R1 * R2, LP = L + 1;
  extern __shared__ __align__(16) unsigned char smraw[];
  T2* buf = reinterpret_cast<T2*>(smraw);
  T2* tws = buf + M * LP;
  using Tab = TwTab<T2, R1, R2>;   // tws: F, I or both as the mode needs them
  constexpr int TW0 = MODE == COL_INV ? Tab::OI : 0;
  constexpr int TWN = MODE == COL_FMI ? Tab::N : (MODE == COL_FWD ? Tab::NF : Tab::NI);
  const T2* twi = tws + (Tab::OI - TW0);
  const TwPrefetch<T2, TWN, L * Shape<R1, R2>::RMAX> twp(tw + TW0);
  gdc_wait();
  const int f = blockIdx.z, t = threadIdx.x;
  const int line = t % L, q = t / L;   // q: n2 in stages 1/B, k1 in stages 2/A
  int outer = blockIdx.x, col = blockIdx.y * L + line;
  const bool live = FULL || col < g.ncols;
  if (FULL && edge_tile<L>(g, outer, col, line)) return;
  // per-thread bases: element (pos, line) of this CTA's tile is base[pos * ps]
  const T2* src = in + f * g.in_fs + outer * g.in_os + col;
  T2* dst = out + f * g.out_fs + outer * g.out_os + col;
  const int64_t ips = g.in_ps, ops = g.out_ps;
  T2 X[R2];
  if (MODE != COL_INV) {
    if (q < R2) {
      const T2* b1 = src + q * ips;
      fwd_stage1<T2, R1, R2, true>(buf, LP, line, q, [&](int pos) {
        T2 v;
        if (live) v = b1[(pos - q) * ips];   // pos - q = R2 n1: a compile-time multiple of R2
        else v.x = v.y = 0;
        return v;
      });
    }
    twp.store(tws);
    __syncthreads();
    if (q < R1) fwd_stage2<T2, R1, R2>(buf, LP, line, q, tws, X);
  } else {
    __syncthreads();
    if (q < R1) {
      const T2* b = src + q * ips;
#pragma unroll
      for (int k2 = 0; k2 < R2; ++k2) {
        if (live) X[k2] = b[(int64_t)(R1 * k2) * ips];
        else X[k2].x = X[k2].y = 0;
      }
    }
    twp.store(tws);   // FP32: first read in inv_stageA, FP64 in inv_stageB, behind the barriers below
  }
  if (MODE == COL_FWD) {
    if (q < R1 && live) {
      T2* b = dst + q * ops;
#pragma unroll
      for (int k2 = 0; k2 < R2; ++k2) b[(int64_t)(R1 * k2) * ops] = X[k2];
    }
    return;
  }
  if (MODE == COL_FMI && q < R1) {
    static_assert(R2 % 2 == 0, "the octant fold below splits k2 at R2 / 2");
    const int ky = outer, kyo = ky <= M - ky ? ky : M - ky;
    const int kz = col, kzo = kz <= M - kz ? kz : M - kz;
    const int64_t HH = (int64_t)H * H, st = (int64_t)R1 * HH;
    // kx = q + R1 k2 (q < R1): k2 < R2/2 gives kx <= M/2, read at kx; the upper
    // half folds to M - kx = (M - q) - R1 k2.
    const T* glo = ghat + (int64_t)q * HH + (int64_t)kyo * H + kzo;
    const T* ghi = ghat + (int64_t)(M - q) * HH + (int64_t)kyo * H + kzo;
#pragma unroll
    for (int k2 = 0; k2 < R2; ++k2) {
      const T gv = live ? (k2 < R2 / 2 ? glo[k2 * st] : ghi[-k2 * st]) : (T)0;
      X[k2].x *= gv;
      X[k2].y *= gv;
    }
  }
  __syncthreads();   // stage-2 reads of buf are complete
  if (q < R1) inv_stageA<T2, R1, R2>(buf, LP, line, q, tws, X);
  __syncthreads();
  if (q < R2) {
    T2* b = dst + q * ops;
    inv_stageB<T2, R1, R2, true>(buf, LP, line, q, twi, [&](int pos, T2 v) {
      if (live) b[(pos - q) * ops] = v;
    });
  }
}

// Block sums, valid in thread 0 only, of a block of NT threads: some shapes' blocks (L * RMAX threads) are
// not whole warps, and a shuffle may name only lanes that exist. A short last warp exchanges among its
// own lanes, a lane without a partner adds nothing. `sh` holds 32 doubles; NT <= 1024.
template <int NT>
__device__ __forceinline__ double block_total(double v, double* sh) {
  constexpr int TAIL = NT % 32, NW = (NT + 31) / 32;
  if constexpr (TAIL == 0) {
    return block_sum(v, sh);
  } else {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    if (warp < NW - 1) {
      v = warp_sum(v);
    } else {
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) {
        const bool has = lane + o < TAIL;
        const double x = __shfl_sync((1u << TAIL) - 1, v, has ? lane + o : lane);
        if (has) v += x;
      }
    }
    __syncthreads();   // sh may still be read from a sum before
    if (lane == 0) sh[warp] = v;
    __syncthreads();
    double t = 0.0;
    if (threadIdx.x == 0)
      for (int w = 0; w < NW; ++w) t += sh[w];
    return t;
  }
}
// Of a per-thread accumulator.
template <int NT>
__device__ __forceinline__ double block_sum0(const Acc<double>& a, double* sh) {
  return block_total<NT>(a.value(), sh);
}

// acc times a small whole number w (exact for 0, 1 and 2).
__device__ __forceinline__ Acc<double> scaled(Acc<double> a, int w) {
  a.v = w == 0 ? 0.0 : a.v * w;   // a column without weight may hold anything
  return a;
}

// Energies without the inverse passes (Parseval). The kernel spectrum is
// stored as ghat = G^ dV / M^3, so a part's epilogue energy sum_r rho J with
// J = IDFT(ghat DFT(rho)) (unnormalised) equals sum_k ghat(k) |rho^(k)|^2 over
// the doubled grid (rho is zero outside the N^3 box). For a field F = a + i b
// of two real densities, sum_k ghat |F^|^2 is the sum of both parts' values:
// ghat is real and even, so the cross terms cancel between k and -k. Both
// parts of a field therefore carry one weight and one slot. Each CTA runs the
// x forward transform of its lines of the y-transformed field (as the x pass
// does), sums ghat |X|^2 over its spectrum entries and writes the weighted sum
// to its field's slot, 0 to the other slot.
template <typename T, int R1, int R2, int L, bool FULL>
__global__ void __launch_bounds__(L * Shape<R1, R2>::RMAX)
    k_cols_fe(const typename Cplx<T>::type* in, ColGeom g, const typename Cplx<T>::type* tw,
              const T* ghat, int H, FeArgs fa) {
  using T2 = typename Cplx<T>::type;
  constexpr int M = R1 * R2, LP = L + 1;
  static_assert(R2 % 2 == 0, "the octant fold below splits k2 at R2 / 2");
  extern __shared__ __align__(16) unsigned char smraw[];
  __shared__ double sh[32];
  T2* buf = reinterpret_cast<T2*>(smraw);
  T2* tws = buf + M * LP;
  const TwPrefetch<T2, TwTab<T2, R1, R2>::NF, L * Shape<R1, R2>::RMAX> twp(tw);
  gdc_wait();
  const int f = blockIdx.z, t = threadIdx.x;
  const int line = t % L, q = t / L;
  int outer = blockIdx.x, col = blockIdx.y * L + line;
  const bool live = FULL || col < g.ncols;
  // nothing to do: no column of a lone real field's half spectrum, or no outer index left
  const bool none = fa.half && (int)blockIdx.y * L > M / 2;
  if (none || (FULL && edge_tile<L>(g, outer, col, line))) {
    if (t == 0) {
      const int64_t b = ((int64_t)(fa.f0 + f) * gridDim.y + blockIdx.y) * gridDim.x + blockIdx.x;
      fa.partials[b] = fa.partials[fa.slot_stride + b] = 0.0;
    }
    return;
  }
  const T2* src = in + f * g.in_fs + outer * g.in_os + col;
  const int64_t ips = g.in_ps;
  if (q < R2) {
    const T2* b1 = src + q * ips;
    fwd_stage1<T2, R1, R2, true>(buf, LP, line, q, [&](int pos) {
      T2 v;
      if (live) v = b1[(pos - q) * ips];
      else v.x = v.y = 0;
      return v;
    });
  }
  twp.store(tws);
  __syncthreads();
  Acc<T> acc;
  if (q < R1) {
    T2 X[R2];
    fwd_stage2<T2, R1, R2>(buf, LP, line, q, tws, X);
    // kx = q + R1 k2, folded into the kernel-spectrum octant as in the x pass
    const int ky = outer, kyo = ky <= M - ky ? ky : M - ky;
    const int kz = col, kzo = kz <= M - kz ? kz : M - kz;
    const int64_t HH = (int64_t)H * H, st = (int64_t)R1 * HH;
    const T* glo = ghat + (int64_t)q * HH + (int64_t)kyo * H + kzo;
    const T* ghi = ghat + (int64_t)(M - q) * HH + (int64_t)kyo * H + kzo;
#pragma unroll
    for (int k2 = 0; k2 < R2; ++k2) {
      const T gv = live ? (k2 < R2 / 2 ? glo[k2 * st] : ghi[-k2 * st]) : (T)0;
      acc.add_prod(gv, X[k2].x * X[k2].x + X[k2].y * X[k2].y);
    }
    // a lone real field's columns kz and M - kz carry the same power: 0 < kz < M/2 counts twice
    // (the sum is linear in the weight, so it scales the column's finished sum)
    if (fa.half) acc = scaled(acc, kz == 0 || kz == M / 2 ? 1 : (kz < M / 2 ? 2 : 0));
    if (FULL && g.edge && (int)blockIdx.y == g.edge && (int)blockIdx.x * L + line >= (int)gridDim.x)
      acc = scaled(acc, 0);   // a line past the last outer index
  }
  const double s = block_sum0<L * Shape<R1, R2>::RMAX>(acc, sh);
  if (t == 0) {
    const int fg = fa.f0 + f;
    const int64_t b = ((int64_t)fg * gridDim.y + blockIdx.y) * gridDim.x + blockIdx.x;
    const double v = fa.w[fg] * s;
    fa.partials[b] = fa.slot[fg] == 0 ? v : 0.0;
    fa.partials[fa.slot_stride + b] = fa.slot[fg] == 0 ? 0.0 : v;
  }
}

// ---- z passes (rows) ---------------------------------------------------------------
// A CTA owns L consecutive rows (x, y) of the z axis; each stage deals its
// items to the lowest threads: n2 of line l1 in stages 1 and B, k1 of line l2
// in stages 2 and A (RowMap; the RowBuf layout of fft2.cuh), so where R1 and
// R2 differ whole warps idle in the smaller stage, not lanes of every warp (an
// FP64 instruction takes its 64 cycles of the narrow pipe whatever its lanes;
// 96^3 Hartree solve, 12 x 16, 626 -> 609 us). Field rows are read and spectra written
// straight from registers with lanes on consecutive z (or kz), so every
// global access is coalesced and no shared-memory transpose is needed.

template <int R1, int R2, int L>
struct RowMap {
  int l1, n2, l2, k1;
  bool a1, a2;   // this thread has an item in stages 1/B, in stages 2/A
  __device__ __forceinline__ RowMap()
      : l1(threadIdx.x / R2), n2(threadIdx.x % R2), l2(threadIdx.x / R1), k1(threadIdx.x % R1),
        a1(R2 >= R1 || threadIdx.x < L * R2), a2(R1 >= R2 || threadIdx.x < L * R1) {}
};

// Pair density of part q of a field at element gi (0 when the part is absent).
template <typename T>
__device__ __forceinline__ T part_density(const T* a, const T* b, int64_t gi) {
  if (!a) return (T)0;
  T v = a[gi];
  if (b) v *= b[gi];
  return v;
}

// z forward with the pair-density prologue, one field per CTA (grid.y = field).
template <typename T, int R1, int R2, int L>
__global__ void __launch_bounds__(L * Shape<R1, R2>::RMAX)
    k_rows_fwd(PassArgs args, int f0, typename Cplx<T>::type* S1, const typename Cplx<T>::type* tw) {
  using T2 = typename Cplx<T>::type;
  constexpr int M = R1 * R2, N = M / 2, RM = Shape<R1, R2>::RMAX, NT = L * RM;
  extern __shared__ __align__(16) unsigned char smraw[];
  T2* buf = reinterpret_cast<T2*>(smraw);
  T2* tws = buf + L * RowBuf<R1, R2>::LS;
  const TwPrefetch<T2, TwTab<T2, R1, R2>::NF, NT> twp(tw);
  gdc_wait();
  const int p = blockIdx.y;
  const FieldDesc& fd = args.f[f0 + p];
  const int64_t nrows = (int64_t)N * N;
  const RowMap<R1, R2, L> q;
  const int64_t row0 = (int64_t)blockIdx.x * L;
  // the pair-density factors of the real and imaginary parts (null: factor absent)
  const T* a0 = reinterpret_cast<const T*>(args.in[fd.p[0].a]);
  const T* b0 = fd.p[0].b >= 0 ? reinterpret_cast<const T*>(args.in[fd.p[0].b]) : nullptr;
  const T* a1 = fd.p[1].a >= 0 ? reinterpret_cast<const T*>(args.in[fd.p[1].a]) : nullptr;
  const T* b1 = (a1 && fd.p[1].b >= 0) ? reinterpret_cast<const T*>(args.in[fd.p[1].b]) : nullptr;
  T2 v[R1];
  if (q.a1) {
    const bool live = row0 + q.l1 < nrows;
#pragma unroll
    for (int n1 = 0; n1 < R1 / 2; ++n1) {
      const int64_t gi = (row0 + q.l1) * N + R2 * n1 + q.n2;
      v[n1].x = live ? part_density(a0, b0, gi) : (T)0;
      v[n1].y = live ? part_density(a1, b1, gi) : (T)0;
    }
  }
  twp.store(tws);
  if (q.a1) row_fwd_stage1<T2, R1, R2, true>(buf, q.l1, q.n2, v);
  __syncthreads();
  if (q.a2) {
    T2 X[R2];
    row_fwd_stage2<T2, R1, R2>(buf, q.l2, q.k1, tws, X);
    if (row0 + q.l2 < nrows) {
      T2* d = S1 + (int64_t)p * nrows * M + (row0 + q.l2) * M + q.k1;
#pragma unroll
      for (int k2 = 0; k2 < R2; ++k2) d[R1 * k2] = X[k2];
    }
  }
}

// Padded length of a staged input row: N rounded up to R2 modulo 32 words.
template <int R1, int R2> struct StageRow {
  static constexpr int N = R1 * R2 / 2;
  static constexpr int NP = N + ((R2 - N % 32) % 32 + 32) % 32;
};

// The inputs a launch group of pair fields reads, staged once per CTA by
// k_rows_fwd_multi: slot_of[i] is input i's staging slot (-1: unused).
struct RowsIn {
  int nin = 0;
  int8_t idx[kMaxIn] = {};
  int8_t slot_of[kMaxIn] = {};
};

// z forward for every field of a launch group: the L rows of each distinct
// input (the orbitals, psi) are staged in shared memory once, then each field's
// pair densities are formed straight into the stage-1 registers of its FFT.
// Same transform and output as k_rows_fwd, without re-reading the inputs per
// field. Stage-1 lanes read consecutive z of R2-lane lines, so a staged row
// is padded to a multiple of 32 words plus R2 (StageRow): the lines a warp
// reads fall in disjoint bank ranges.
// BULK: one elected thread stages every row with a 1-D bulk copy
// (cp.async.bulk, one mbarrier for the whole block, a bounded wait), so the
// staging costs one round trip and no registers; used when every input is
// 16-byte aligned, a row and a padded staged row are multiples of 16 bytes
// and L divides the rows.
// Otherwise the threads stage with batches of 8 loads each.
template <typename T, int R1, int R2, int L, bool BULK>
__global__ void __launch_bounds__(L * Shape<R1, R2>::RMAX)
    k_rows_fwd_multi(PassArgs args, RowsIn ri, int f0, int nfg, typename Cplx<T>::type* S1,
                     const typename Cplx<T>::type* tw, int* err) {
  using T2 = typename Cplx<T>::type;
  constexpr int M = R1 * R2, N = M / 2, NP = StageRow<R1, R2>::NP, RM = Shape<R1, R2>::RMAX, NT = L * RM;
  extern __shared__ __align__(16) unsigned char smraw[];
  __shared__ __align__(8) uint64_t sbar;
  T2* buf = reinterpret_cast<T2*>(smraw);
  T2* tws = buf + L * RowBuf<R1, R2>::LS;
  T* stage = reinterpret_cast<T*>(tws + TwTab<T2, R1, R2>::NF);   // [slot][line][z], rows of NP
  const TwPrefetch<T2, TwTab<T2, R1, R2>::NF, NT> twp(tw);
  gdc_wait();
  const int64_t row0 = (int64_t)blockIdx.x * L;
  const int64_t nrows = (int64_t)N * N;
  if constexpr (BULK) {
    __shared__ int s_misaligned;
    if (threadIdx.x == 0) {
      mbar_init(&sbar, 1);
      fence_barrier_init();
      // the host only picks this path for 16-byte aligned rows; re-check, and
      // record an error instead of issuing a copy that would fault
      int bad_align = (int)((smem_u32(stage) | (uint32_t)(NP * sizeof(T)) | (uint32_t)(N * sizeof(T))) & 15u);
      for (int sl = 0; sl < ri.nin; ++sl)
        bad_align |= (int)(reinterpret_cast<uintptr_t>(args.in[ri.idx[sl]]) & 15u);
      s_misaligned = bad_align;
      if (bad_align && err) atomicExch(err, 110);
    }
    __syncthreads();   // the barrier is initialised before anyone waits on it
    if (s_misaligned) return;
    if (threadIdx.x == 0) {
      mbar_expect_tx(&sbar, (uint32_t)(ri.nin * L * N * sizeof(T)));
      for (int sl = 0; sl < ri.nin; ++sl) {
        const T* src = reinterpret_cast<const T*>(args.in[ri.idx[sl]]) + row0 * N;
        for (int l = 0; l < L; ++l)
          bulk_load(stage + (sl * L + l) * NP, src + (int64_t)l * N, (uint32_t)(N * sizeof(T)), &sbar);
      }
    }
    twp.store(tws);
    bool bad = false;
    if (!mbar_wait_bounded(&sbar, 0, err, 108)) bad = true;
    if (__syncthreads_or(bad)) {
      if (threadIdx.x == 0) mbar_wait_bounded(&sbar, 0, err, 109);   // the copies still land
      return;
    }
  } else {
  // staging: 8 loads in flight per thread per batch (measured faster than one
  // batch of 32 at 128^3: 53 against 69 us)
  const int nel = ri.nin * L * N;
  constexpr int B = 8;
  for (int base = 0; base < nel; base += B * NT) {
    T v[B];
#pragma unroll
    for (int k = 0; k < B; ++k) {
      const int i = base + threadIdx.x + k * NT;
      const int sl = i / (L * N), rem = i % (L * N);
      const int64_t r = row0 + rem / N;
      v[k] = (i < nel && r < nrows) ? reinterpret_cast<const T*>(args.in[ri.idx[sl]])[r * N + rem % N] : (T)0;
    }
#pragma unroll
    for (int k = 0; k < B; ++k) {
      const int i = base + threadIdx.x + k * NT;
      if (i < nel) {
        const int sl = i / (L * N), rem = i % (L * N);
        stage[(sl * L + rem / N) * NP + rem % N] = v[k];
      }
    }
  }
  twp.store(tws);
  __syncthreads();
  }
  const RowMap<R1, R2, L> q;
  const int64_t r = row0 + q.l2;
  for (int p = 0; p < nfg; ++p) {
    const FieldDesc& fd = args.f[f0 + p];
    if (q.a1) {
      const int line = q.l1, j = q.n2;
      const int a0 = ri.slot_of[fd.p[0].a];
      const int b0 = fd.p[0].b >= 0 ? ri.slot_of[fd.p[0].b] : -1;
      const int a1 = fd.p[1].a >= 0 ? ri.slot_of[fd.p[1].a] : -1;
      const int b1 = (a1 >= 0 && fd.p[1].b >= 0) ? ri.slot_of[fd.p[1].b] : -1;
      T2 v[R1];
#pragma unroll
      for (int n1 = 0; n1 < R1 / 2; ++n1) {
        const int z = R2 * n1 + j;
        T x = stage[(a0 * L + line) * NP + z];
        if (b0 >= 0) x *= stage[(b0 * L + line) * NP + z];
        T y = (T)0;
        if (a1 >= 0) {
          y = stage[(a1 * L + line) * NP + z];
          if (b1 >= 0) y *= stage[(b1 * L + line) * NP + z];
        }
        v[n1].x = x;
        v[n1].y = y;
      }
      row_fwd_stage1<T2, R1, R2, true>(buf, line, j, v);
    }
    __syncthreads();
    if (q.a2) {
      T2 X[R2];
      row_fwd_stage2<T2, R1, R2>(buf, q.l2, q.k1, tws, X);
      if (r < nrows) {
        T2* d = S1 + (int64_t)p * nrows * M + r * M + q.k1;
#pragma unroll
        for (int k2 = 0; k2 < R2; ++k2) d[R1 * k2] = X[k2];
      }
    }
    __syncthreads();   // buf is rewritten by the next field
  }
}

// The bulk-staged z forward as a persistent kernel: each CTA walks row blocks
// blockIdx.x, blockIdx.x + gridDim.x, ... with the staging buffer doubled, so
// one elected thread issues the next block's row copies (1-D bulk copies on
// that buffer's mbarrier) before the current block is transformed and the
// copies land under the transforms. Same transforms and output as
// k_rows_fwd_multi. The host guarantees 16-byte aligned rows, a padded staged
// row that is a multiple of 16 bytes and L | N^2; the kernel re-checks the
// alignment and records error 110 instead of issuing a bad copy. Waits are
// bounded (codes 113/114).
template <typename T, int R1, int R2, int L>
__global__ void __launch_bounds__(L * Shape<R1, R2>::RMAX)
    k_rows_fwd_pers(PassArgs args, RowsIn ri, int f0, int nfg, typename Cplx<T>::type* S1,
                    const typename Cplx<T>::type* tw, int* err) {
  using T2 = typename Cplx<T>::type;
  constexpr int M = R1 * R2, N = M / 2, NP = StageRow<R1, R2>::NP, RM = Shape<R1, R2>::RMAX, NT = L * RM;
  extern __shared__ __align__(16) unsigned char smraw[];
  __shared__ __align__(8) uint64_t sbar[2];
  __shared__ int s_misaligned;
  T2* buf = reinterpret_cast<T2*>(smraw);
  T2* tws = buf + L * RowBuf<R1, R2>::LS;
  T* stage0 = reinterpret_cast<T*>(tws + TwTab<T2, R1, R2>::NF);   // [slot][input][line][z], rows of NP
  const int SB = ri.nin * L * NP;                                    // floats per staging slot
  const int64_t nrows = (int64_t)N * N;
  const int nblk = (int)(nrows / L);
  if (threadIdx.x == 0) {
    mbar_init(&sbar[0], 1);
    mbar_init(&sbar[1], 1);
    fence_barrier_init();
    int bad_align = (int)((smem_u32(stage0) | (uint32_t)(SB * sizeof(T)) | (uint32_t)(NP * sizeof(T)) |
                           (uint32_t)(N * sizeof(T))) & 15u);
    for (int sl = 0; sl < ri.nin; ++sl)
      bad_align |= (int)(reinterpret_cast<uintptr_t>(args.in[ri.idx[sl]]) & 15u);
    s_misaligned = bad_align;
    if (bad_align && err) atomicExch(err, 110);
  }
  for (int i = threadIdx.x; i < TwTab<T2, R1, R2>::NF; i += NT) tws[i] = tw[i];
  gdc_wait();
  __syncthreads();
  if (s_misaligned) return;
  auto issue = [&](int blk, int slot) {
    mbar_expect_tx(&sbar[slot], (uint32_t)(ri.nin * L * N * sizeof(T)));
    T* st = stage0 + slot * SB;
    for (int sl = 0; sl < ri.nin; ++sl) {
      const T* src = reinterpret_cast<const T*>(args.in[ri.idx[sl]]) + (int64_t)blk * L * N;
      for (int l = 0; l < L; ++l)
        bulk_load(st + (sl * L + l) * NP, src + (int64_t)l * N, (uint32_t)(N * sizeof(T)), &sbar[slot]);
    }
  };
  if (threadIdx.x == 0 && (int)blockIdx.x < nblk) issue(blockIdx.x, 0);
  const RowMap<R1, R2, L> q;
  int it = 0;
  for (int blk = blockIdx.x; blk < nblk; blk += gridDim.x, ++it) {
    const int slot = it & 1;
    // the other slot was last read by the previous block, which ended at a barrier
    const bool more = blk + (int)gridDim.x < nblk;
    if (threadIdx.x == 0 && more) issue(blk + gridDim.x, slot ^ 1);
    const bool bad = !mbar_wait_bounded(&sbar[slot], (it >> 1) & 1, err, 113);
    if (__syncthreads_or(bad)) {
      if (threadIdx.x == 0) {   // copies still in flight land before the CTA goes away
        mbar_wait_bounded(&sbar[slot], (it >> 1) & 1, err, 114);
        if (more) mbar_wait_bounded(&sbar[slot ^ 1], ((it + 1) >> 1) & 1, err, 114);
      }
      return;
    }
    const T* stage = stage0 + slot * SB;
    const int64_t r = (int64_t)blk * L + q.l2;
    for (int p = 0; p < nfg; ++p) {
      const FieldDesc& fd = args.f[f0 + p];
      if (q.a1) {
        const int line = q.l1, j = q.n2;
        const int a0 = ri.slot_of[fd.p[0].a];
        const int b0 = fd.p[0].b >= 0 ? ri.slot_of[fd.p[0].b] : -1;
        const int a1 = fd.p[1].a >= 0 ? ri.slot_of[fd.p[1].a] : -1;
        const int b1 = (a1 >= 0 && fd.p[1].b >= 0) ? ri.slot_of[fd.p[1].b] : -1;
        T2 v[R1];
#pragma unroll
        for (int n1 = 0; n1 < R1 / 2; ++n1) {
          const int z = R2 * n1 + j;
          T x = stage[(a0 * L + line) * NP + z];
          if (b0 >= 0) x *= stage[(b0 * L + line) * NP + z];
          T y = (T)0;
          if (a1 >= 0) {
            y = stage[(a1 * L + line) * NP + z];
            if (b1 >= 0) y *= stage[(b1 * L + line) * NP + z];
          }
          v[n1].x = x;
          v[n1].y = y;
        }
        row_fwd_stage1<T2, R1, R2, true>(buf, line, j, v);
      }
      fence_proxy_async_smem();   // this slot's reads precede the copies issued into it next
      __syncthreads();
      if (q.a2) {
        T2 X[R2];
        row_fwd_stage2<T2, R1, R2>(buf, q.l2, q.k1, tws, X);
        T2* d = S1 + (int64_t)p * nrows * M + r * M + q.k1;
#pragma unroll
        for (int k2 = 0; k2 < R2; ++k2) d[R1 * k2] = X[k2];
      }
      __syncthreads();   // buf is rewritten by the next field; the stage slot is free after the last
    }
  }
}

// z inverse over every field of the group, then the epilogue. NO > 0: the
// accumulation terms target outputs < NO, kept in registers (each thread owns
// the R1/2 fixed elements z = j + R2 n1 of its row); NO == 0: energy mode.
// FP32, one output, M = 256 fits 64 registers without spills: four CTAs per SM.
template <typename T, int R1, int R2, int NO>
constexpr int rows_inv_min_ctas() {
  return (NO == 1 && sizeof(T) == 4 && R1 == 16 && R2 == 16) ? 4 : 1;
}

template <typename T, int R1, int R2, int L, int NO>
__global__ void __launch_bounds__(L * Shape<R1, R2>::RMAX, (rows_inv_min_ctas<T, R1, R2, NO>()))
    k_rows_inv(PassArgs args, int f0, int nfg, const typename Cplx<T>::type* S1,
               const typename Cplx<T>::type* tw, int accumulate, double* partials,
               int64_t slot_stride) {
  using T2 = typename Cplx<T>::type;
  constexpr int M = R1 * R2, N = M / 2, RM = Shape<R1, R2>::RMAX, NT = L * RM;
  constexpr int EPT = R1 / 2;
  constexpr bool ENERGY = NO == 0;
  extern __shared__ __align__(16) unsigned char smraw[];
  __shared__ double sh[32];
  T2* buf = reinterpret_cast<T2*>(smraw);
  T2* tws = buf + L * RowBuf<R1, R2>::LS;
  const TwPrefetch<T2, TwTab<T2, R1, R2>::NI, NT> twp(tw + TwTab<T2, R1, R2>::OI);
  gdc_wait();
  const int64_t nrows = (int64_t)N * N;
  const RowMap<R1, R2, L> q;
  const int j = q.n2;
  const int64_t r = (int64_t)blockIdx.x * L + q.l1;     // row of this thread's outputs
  const int64_t rk = (int64_t)blockIdx.x * L + q.l2;    // row of its spectrum entries
  const bool own = q.a1 && r < nrows;   // this thread owns elements of the output
  T acc[ENERGY ? 1 : NO][EPT];
#pragma unroll
  for (int o = 0; o < (ENERGY ? 1 : NO); ++o)
#pragma unroll
    for (int e = 0; e < EPT; ++e) acc[o][e] = (T)0;
  Acc<T> e0, e1;
  for (int p = 0; p < nfg; ++p) {
    const FieldDesc& fd = args.f[f0 + p];
    // The epilogue's first field factor of each part (in[tc] of term 0, or the
    // density in energy mode) does not depend on the transform. With several
    // outputs (or energies) it is loaded now, so its latency overlaps the FFT;
    // with one output it is loaded in the epilogue, which keeps the kernel at
    // four CTAs per SM (64 registers). A second term (block applies on the
    // generic engine only) always loads in the epilogue.
    constexpr bool PREFETCH = ENERGY || NO > 1;
    T fac[EPT][2];
    auto load_fac = [&]() {
#pragma unroll
      for (int e = 0; e < EPT; ++e) {
        const int64_t gi = r * N + j + R2 * e;
#pragma unroll
        for (int qq = 0; qq < 2; ++qq) {
          const PartDesc& d = fd.p[qq];
          if constexpr (ENERGY)
            fac[e][qq] = (own && d.a >= 0) ? dens<T>(d, args.in, gi) : (T)0;
          else
            fac[e][qq] = (own && d.a >= 0 && d.nt > 0)
                             ? (d.tc[0] >= 0 ? reinterpret_cast<const T*>(args.in[d.tc[0]])[gi] : (T)1)
                             : (T)0;
        }
      }
    };
    if constexpr (PREFETCH) load_fac();
    T2 X[R2];
    if (q.a2) {
      const T2* src = S1 + (int64_t)p * nrows * M + rk * M + q.k1;
#pragma unroll
      for (int k2 = 0; k2 < R2; ++k2) {
        if (rk < nrows) X[k2] = src[R1 * k2];
        else X[k2].x = X[k2].y = 0;
      }
    }
    if (p == 0) twp.store(tws);
    __syncthreads();   // tws is visible; the previous field's stage-B reads of buf are done
    if (q.a2) row_inv_stageA<T2, R1, R2>(buf, q.l2, q.k1, tws, X);
    __syncthreads();
    if (own) {
      if constexpr (!PREFETCH) load_fac();
      T2 w[R1];
      row_inv_stageB<T2, R1, R2>(buf, q.l1, j, tws, w);
#pragma unroll
      for (int e = 0; e < EPT; ++e) {
        const int64_t gi = r * N + j + R2 * e;
        const T2 J = w[e];
#pragma unroll
        for (int qq = 0; qq < 2; ++qq) {
          const PartDesc& d = fd.p[qq];
          if (d.a < 0) continue;
          const T val = qq == 0 ? J.x : J.y;
          if constexpr (ENERGY) {
            const T de = fac[e][qq];
            if (d.eslot == 0) e0.add_prod(de * (T)d.ew, val);
            else e1.add_prod(de * (T)d.ew, val);
          } else {
#pragma unroll
            for (int k = 0; k < 2; ++k) {
              if (k >= d.nt) break;
              T m = (T)d.coef[k];
              if (k == 0) m *= fac[e][qq];
              else if (d.tc[1] >= 0) m *= reinterpret_cast<const T*>(args.in[d.tc[1]])[gi];
              const int to = d.to[k];
#pragma unroll
              for (int o = 0; o < NO; ++o)
                if (o == to) acc[o][e] += m * val;
            }
          }
        }
      }
    }
  }
  if constexpr (ENERGY) {
    const double s0 = block_total<NT>(e0.value(), sh);
    const double s1 = block_total<NT>(e1.value(), sh);
    if (threadIdx.x == 0) {
      partials[blockIdx.x] = s0;
      partials[slot_stride + blockIdx.x] = s1;
    }
  } else {
    if (!own) return;
    const int nout = args.nout;
#pragma unroll
    for (int o = 0; o < NO; ++o) {
      if (o >= nout) break;
      T* dst = reinterpret_cast<T*>(args.out[o]) + r * N + j;
#pragma unroll
      for (int e = 0; e < EPT; ++e) dst[R2 * e] = accumulate ? dst[R2 * e] + acc[o][e] : acc[o][e];
    }
  }
}

// ---- lone real fields ------------------------------------------------------------------
// A field whose imaginary part is absent (a Hartree density, the last pair of an odd count) is
// real, so its spectrum is Hermitian and the columns kz <= N = M/2 hold all of it. Its z passes
// transform TWO rows per line, rows 2l and 2l + 1 as real and imaginary part, and the column
// passes run over the N + 1 columns alone (rounded up to whole tiles): about half the arithmetic
// and half the spectral traffic of a complex field with a zero imaginary part. The FP64 passes are
// bound by the FP64 pipe, so the arithmetic is what counts: a 96^3 Hartree solve took 1306 us with
// the zero imaginary part and takes 736 us; the helium matvec at 64^3 falls in the same ratio.

// z forward: Z = FFT(row_2l + i row_2l+1), A = (Z_k + conj Z_-k) / 2 and B = (Z_k - conj Z_-k) / 2i
// are the two rows' spectra; the halves are taken on the inputs (exact). One field per grid.y.
template <typename T, int R1, int R2, int L>
__global__ void __launch_bounds__(L * Shape<R1, R2>::RMAX)
    k_rows_fwd_real(PassArgs args, int f0, typename Cplx<T>::type* S1, const typename Cplx<T>::type* tw) {
  using T2 = typename Cplx<T>::type;
  constexpr int M = R1 * R2, N = M / 2, RM = Shape<R1, R2>::RMAX, NT = L * RM, LS = RowBuf<R1, R2>::LS;
  static_assert(N % 2 == 0 && LS >= M, "rows pair up; a line's buffer holds its whole spectrum");
  extern __shared__ __align__(16) unsigned char smraw[];
  T2* buf = reinterpret_cast<T2*>(smraw);
  T2* tws = buf + L * LS;
  const TwPrefetch<T2, TwTab<T2, R1, R2>::NF, NT> twp(tw);
  gdc_wait();
  const int p = blockIdx.y;
  const PartDesc& pd = args.f[f0 + p].p[0];
  const int64_t npair = (int64_t)N * N / 2;
  const RowMap<R1, R2, L> q;
  const int64_t l0 = (int64_t)blockIdx.x * L;
  const T* a = reinterpret_cast<const T*>(args.in[pd.a]);
  const T* b = pd.b >= 0 ? reinterpret_cast<const T*>(args.in[pd.b]) : nullptr;
  T2 v[R1];
  if (q.a1) {
    const bool live = l0 + q.l1 < npair;
#pragma unroll
    for (int n1 = 0; n1 < R1 / 2; ++n1) {
      const int64_t gi = 2 * (l0 + q.l1) * N + R2 * n1 + q.n2;
      v[n1].x = live ? (T)0.5 * part_density(a, b, gi) : (T)0;
      v[n1].y = live ? (T)0.5 * part_density(a, b, gi + N) : (T)0;
    }
  }
  twp.store(tws);
  if (q.a1) row_fwd_stage1<T2, R1, R2, true>(buf, q.l1, q.n2, v);
  __syncthreads();
  T2 X[R2];
  if (q.a2) row_fwd_stage2<T2, R1, R2>(buf, q.l2, q.k1, tws, X);
  __syncthreads();   // stage-2 reads of buf are complete
  if (q.a2) {
#pragma unroll
    for (int k2 = 0; k2 < R2; ++k2) buf[q.l2 * LS + q.k1 + R1 * k2] = X[k2];
  }
  __syncthreads();
  const int line = threadIdx.x / RM, j = threadIdx.x % RM;
  const int64_t l = l0 + line;
  if (l >= npair) return;
  T2* d = S1 + ((int64_t)p * N * N + 2 * l) * M;
  for (int k = j; k <= N; k += RM) {
    const T2 z = buf[line * LS + k], c = buf[line * LS + (k == 0 ? 0 : M - k)];
    T2 A, B;
    A.x = z.x + c.x;
    A.y = z.y - c.y;
    B.x = z.y + c.y;
    B.y = c.x - z.x;
    d[k] = A;
    d[M + k] = B;
  }
}

// z inverse of row pairs: Z_k = A_k + i B_k for k <= N and conj(A_M-k) + i conj(B_M-k) above, whose
// transform is row_2l + i row_2l+1. J: the potential goes to field 2 (f0 + p) of jbase (one field per
// grid.y); otherwise one field's terms are added to (or, not accumulating, written to) the outputs.
template <typename T, int R1, int R2, int L, bool J>
__global__ void __launch_bounds__(L * Shape<R1, R2>::RMAX)
    k_rows_inv_real(PassArgs args, int f0, const typename Cplx<T>::type* S1, const typename Cplx<T>::type* tw,
                    int accumulate) {
  using T2 = typename Cplx<T>::type;
  constexpr int M = R1 * R2, N = M / 2, RM = Shape<R1, R2>::RMAX, NT = L * RM;
  extern __shared__ __align__(16) unsigned char smraw[];
  T2* buf = reinterpret_cast<T2*>(smraw);
  T2* tws = buf + L * RowBuf<R1, R2>::LS;
  const TwPrefetch<T2, TwTab<T2, R1, R2>::NI, NT> twp(tw + TwTab<T2, R1, R2>::OI);
  gdc_wait();
  const int p = blockIdx.y;
  const int64_t npair = (int64_t)N * N / 2;
  const RowMap<R1, R2, L> q;
  const int64_t l0 = (int64_t)blockIdx.x * L;
  T2 X[R2];
  if (q.a2) {
    const bool live = l0 + q.l2 < npair;
    const T2* A = S1 + ((int64_t)p * N * N + 2 * (l0 + q.l2)) * M;
#pragma unroll
    for (int k2 = 0; k2 < R2; ++k2) {
      const int k = q.k1 + R1 * k2;
      const bool up = k > N;
      T2 a, b;
      a.x = a.y = b.x = b.y = 0;
      if (live) {
        a = A[up ? M - k : k];
        b = A[M + (up ? M - k : k)];
      }
      X[k2].x = up ? a.x + b.y : a.x - b.y;
      X[k2].y = up ? b.x - a.y : a.y + b.x;
    }
  }
  twp.store(tws);
  __syncthreads();
  if (q.a2) row_inv_stageA<T2, R1, R2>(buf, q.l2, q.k1, tws, X);
  __syncthreads();
  const int64_t l = l0 + q.l1;
  if (!q.a1 || l >= npair) return;
  T2 w[R1];
  row_inv_stageB<T2, R1, R2>(buf, q.l1, q.n2, tws, w);
  const int64_t g0 = 2 * l * N + q.n2;
  if constexpr (J) {
    T* o = reinterpret_cast<T*>(args.jbase) + (int64_t)(2 * (f0 + p)) * args.jstride + g0;
#pragma unroll
    for (int e = 0; e < R1 / 2; ++e) {
      o[R2 * e] = w[e].x;
      o[N + R2 * e] = w[e].y;
    }
  } else {
    const PartDesc& d = args.f[f0 + p].p[0];
#pragma unroll 1
    for (int k = 0; k < d.nt; ++k) {
      T* o = reinterpret_cast<T*>(args.out[d.to[k]]) + g0;
      const T* u = d.tc[k] >= 0 ? reinterpret_cast<const T*>(args.in[d.tc[k]]) + g0 : nullptr;
      const T cf = (T)d.coef[k];
#pragma unroll
      for (int e = 0; e < R1 / 2; ++e)
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          const int i = R2 * e + h * N;
          T m = cf;
          if (u) m *= u[i];
          const T val = m * (h == 0 ? w[e].x : w[e].y);
          o[i] = accumulate ? o[i] + val : val;
        }
    }
  }
}

// z inverse of one field per CTA (grid.y = field), writing J_re and J_im of
// the row block to their own real fields (the EPI_J epilogue).
template <typename T, int R1, int R2, int L>
__global__ void __launch_bounds__(L * Shape<R1, R2>::RMAX)
    k_rows_inv_j(T* jbase, int64_t jstride, int f0, const typename Cplx<T>::type* S1,
                 const typename Cplx<T>::type* tw) {
  using T2 = typename Cplx<T>::type;
  constexpr int M = R1 * R2, N = M / 2, RM = Shape<R1, R2>::RMAX, NT = L * RM;
  extern __shared__ __align__(16) unsigned char smraw[];
  T2* buf = reinterpret_cast<T2*>(smraw);
  T2* tws = buf + L * RowBuf<R1, R2>::LS;
  const TwPrefetch<T2, TwTab<T2, R1, R2>::NI, NT> twp(tw + TwTab<T2, R1, R2>::OI);
  gdc_wait();
  const int p = blockIdx.y;
  const int64_t nrows = (int64_t)N * N;
  const RowMap<R1, R2, L> q;
  const int64_t r = (int64_t)blockIdx.x * L + q.l1, rk = (int64_t)blockIdx.x * L + q.l2;
  T2 X[R2];
  if (q.a2) {
    const T2* src = S1 + (int64_t)p * nrows * M + rk * M + q.k1;
#pragma unroll
    for (int k2 = 0; k2 < R2; ++k2) {
      if (rk < nrows) X[k2] = src[R1 * k2];
      else X[k2].x = X[k2].y = 0;
    }
  }
  twp.store(tws);
  __syncthreads();
  if (q.a2) row_inv_stageA<T2, R1, R2>(buf, q.l2, q.k1, tws, X);
  __syncthreads();
  if (q.a1 && r < nrows) {
    T2 w[R1];
    row_inv_stageB<T2, R1, R2>(buf, q.l1, q.n2, tws, w);
    T* jre = jbase + (int64_t)(2 * (f0 + p)) * jstride + r * N + q.n2;
    T* jim = jre + jstride;
#pragma unroll
    for (int n1 = 0; n1 < R1 / 2; ++n1) {
      jre[R2 * n1] = w[n1].x;
      jim[R2 * n1] = w[n1].y;
    }
  }
}

template <typename K>
inline int smem_attr(K k, size_t bytes) {
  return raise_smem_limit(reinterpret_cast<const void*>(k), bytes);
}

// Launchers for one shape.
template <typename T, int R1, int R2, int L>
struct Launch {
  using T2 = typename Cplx<T>::type;
  static constexpr int M = R1 * R2, N = M / 2, NT = L * Shape<R1, R2>::RMAX;
  using Tab = TwTab<T2, R1, R2>;   // stage-twiddle table entries
  static size_t sm_cols(int mode) {
    return (size_t)(M * (L + 1) + (mode == COL_FMI ? Tab::N : (mode == COL_FWD ? Tab::NF : Tab::NI))) * sizeof(T2);
  }
  static size_t sm_rows(bool fwd) {
    return (size_t)(L * RowBuf<R1, R2>::LS + (fwd ? Tab::NF : Tab::NI)) * sizeof(T2);
  }
  // Whole tiles only where L divides the M columns (the callers pass all of them, or a multiple of L
  // that is at most M).
  static constexpr bool FULL = M % L == 0;
  static int cols(int mode, const T2* in, T2* out, const ColGeom& g, int outer, int nf, const T2* tw,
                  const T* ghat, int H, cudaStream_t s) {
    if (FULL && g.ncols % L != 0) return fail(GATO_EUNSUPPORTED, "column pass: whole tiles of %d columns", L);
    dim3 grid(outer, (g.ncols + L - 1) / L + (g.edge > 0), nf);
    const size_t sm = sm_cols(mode);
    if (mode == COL_FWD) {
      GATO_TRY(smem_attr(k_cols<T, R1, R2, L, COL_FWD, FULL>, sm));
      GATO_TRY(launch_chained(k_cols<T, R1, R2, L, COL_FWD, FULL>, grid, NT, sm, s, in, out, g, tw, ghat, H));
    } else if (mode == COL_INV) {
      GATO_TRY(smem_attr(k_cols<T, R1, R2, L, COL_INV, FULL>, sm));
      GATO_TRY(launch_chained(k_cols<T, R1, R2, L, COL_INV, FULL>, grid, NT, sm, s, in, out, g, tw, ghat, H));
    } else {
      GATO_TRY(smem_attr(k_cols<T, R1, R2, L, COL_FMI, FULL>, sm));
      GATO_TRY(launch_chained(k_cols<T, R1, R2, L, COL_FMI, FULL>, grid, NT, sm, s, in, out, g, tw, ghat, H));
    }
    return GATO_OK;
  }
  static int cols_fe(const T2* in, const ColGeom& g, int outer, int nf, const T2* tw, const T* ghat, int H,
                     const FeArgs& fa, cudaStream_t s) {
    dim3 grid(outer, (g.ncols + L - 1) / L, nf);
    const size_t sm = sm_cols(COL_FWD);
    GATO_TRY(smem_attr(k_cols_fe<T, R1, R2, L, FULL>, sm));
    GATO_TRY(launch_chained(k_cols_fe<T, R1, R2, L, FULL>, grid, NT, sm, s, in, g, tw, ghat, H, fa));
    return GATO_OK;
  }
  static int rows_fwd_real(const PassArgs& a, int f0, int nfg, T2* S1, const T2* tw, cudaStream_t s) {
    const size_t sm = sm_rows(true);
    GATO_TRY(smem_attr(k_rows_fwd_real<T, R1, R2, L>, sm));
    const unsigned nblk = (unsigned)(((int64_t)N * N / 2 + L - 1) / L);
    GATO_TRY(launch_chained(k_rows_fwd_real<T, R1, R2, L>, dim3(nblk, nfg), NT, sm, s, a, f0, S1, tw));
    return GATO_OK;
  }
  // j: potentials to the J fields (nfg fields at once), else one field's terms to the outputs
  static int rows_inv_real(const PassArgs& a, int f0, int nfg, const T2* S1, const T2* tw, int accumulate,
                           bool j, cudaStream_t s) {
    const size_t sm = sm_rows(false);
    const unsigned nblk = (unsigned)(((int64_t)N * N / 2 + L - 1) / L);
    if (j) {
      GATO_TRY(smem_attr(k_rows_inv_real<T, R1, R2, L, true>, sm));
      GATO_TRY(launch_chained(k_rows_inv_real<T, R1, R2, L, true>, dim3(nblk, nfg), NT, sm, s, a, f0, S1, tw, 0));
    } else {
      GATO_TRY(smem_attr(k_rows_inv_real<T, R1, R2, L, false>, sm));
      GATO_TRY(launch_chained(k_rows_inv_real<T, R1, R2, L, false>, dim3(nblk, 1), NT, sm, s, a, f0, S1, tw, accumulate));
    }
    return GATO_OK;
  }
  // multi: 0 per-field CTAs, 1 multi-field CTAs from three fields up, 2 from two fields up
  // (persistent, double-buffered staging where the rows allow bulk copies), 3 as 2 with one
  // staging round trip per CTA (the non-persistent kernel)
  // (the default: with bulk staging the multi-field kernel wins at two fields too, 239 against 244 us for the
  // 128^3 matvec in one strand; in two, each strand of a call of two fields has one and takes its own kernel)
  static int rows_fwd(const PassArgs& a, int f0, int nfg, T2* S1, const T2* tw, int multi, cudaStream_t s) {
    // several fields over few distinct inputs: stage the inputs once per CTA
    RowsIn ri;
    for (int i = 0; i < kMaxIn; ++i) ri.slot_of[i] = -1;
    auto use = [&](int idx) {
      if (idx < 0 || ri.slot_of[idx] >= 0) return;
      ri.slot_of[idx] = (int8_t)ri.nin;
      ri.idx[ri.nin++] = (int8_t)idx;
    };
    for (int p = 0; p < nfg; ++p)
      for (int qq = 0; qq < 2; ++qq) {
        const PartDesc& d = a.f[f0 + p].p[qq];
        if (d.a < 0) continue;
        use(d.a);
        use(d.b);
      }
    // half the rows per CTA of the other z kernels: the grid covers every
    // field at once, so smaller CTAs give more of them and a shorter last wave
    constexpr int LM = L >= 16 ? L / 2 : L;
    const size_t stage_bytes = (size_t)ri.nin * LM * StageRow<R1, R2>::NP * sizeof(T);
    if (multi > 0 && nfg >= (multi == 1 ? 3 : 2) && stage_bytes <= 48 * 1024) {
      const size_t sm = (size_t)(LM * RowBuf<R1, R2>::LS + Tab::NF) * sizeof(T2) + stage_bytes;
      const int64_t nrows = (int64_t)N * N;
      // a bulk copy needs 16-byte aligned source and destination rows and a
      // size that is a multiple of 16 bytes (the padded staged row included)
      bool bulk = nrows % LM == 0 && (N * sizeof(T)) % 16 == 0 &&
                  (StageRow<R1, R2>::NP * sizeof(T)) % 16 == 0;
      for (int i = 0; i < ri.nin; ++i) bulk = bulk && ((uintptr_t)a.in[ri.idx[i]] % 16) == 0;
      const unsigned grid = (unsigned)((nrows + LM - 1) / LM);
      if (bulk && multi != 3) {
        // persistent CTAs over the row blocks, double-buffered staging: one resident wave
        auto kern = k_rows_fwd_pers<T, R1, R2, LM>;
        const size_t smp = sm + stage_bytes;   // a second staging slot
        GATO_TRY(smem_attr(kern, smp));
        static std::atomic<int> wave[kMaxIn + 1];   // resident blocks of one wave by staged inputs (0: unknown)
        int w = wave[ri.nin].load();
        if (w == 0) {
          int dev = 0, sms = 0, ps = 0;
          GATO_CUDA_TRY(cudaGetDevice(&dev));
          GATO_CUDA_TRY(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
          GATO_CUDA_TRY(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&ps, kern, LM * Shape<R1, R2>::RMAX, smp));
          if (ps < 1) return fail(GATO_EUNSUPPORTED, "z forward: no resident CTA fits");
          w = ps * sms;
          wave[ri.nin].store(w);
        }
        const unsigned pg = (unsigned)std::min<int64_t>(grid, (int64_t)w);
        GATO_TRY(launch_chained(kern, pg, LM * Shape<R1, R2>::RMAX, smp, s, a, ri, f0, nfg, S1, tw, device_error_word()));
      } else if (bulk) {
        GATO_TRY(smem_attr(k_rows_fwd_multi<T, R1, R2, LM, true>, sm));
        GATO_TRY(launch_chained(k_rows_fwd_multi<T, R1, R2, LM, true>, grid, LM * Shape<R1, R2>::RMAX, sm, s, a, ri, f0, nfg, S1, tw, device_error_word()));
      } else {
        GATO_TRY(smem_attr(k_rows_fwd_multi<T, R1, R2, LM, false>, sm));
        GATO_TRY(launch_chained(k_rows_fwd_multi<T, R1, R2, LM, false>, grid, LM * Shape<R1, R2>::RMAX, sm, s, a, ri, f0, nfg, S1, tw, device_error_word()));
      }
      return GATO_OK;
    }
    const size_t sm = sm_rows(true);
    GATO_TRY(smem_attr(k_rows_fwd<T, R1, R2, L>, sm));
    const int64_t nrows = (int64_t)N * N;
    GATO_TRY(launch_chained(k_rows_fwd<T, R1, R2, L>, dim3((unsigned)((nrows + L - 1) / L), nfg), NT, sm, s, a, f0, S1, tw));
    return GATO_OK;
  }
  template <int NO>
  static int rows_inv_no(const PassArgs& a, int f0, int nfg, const T2* S1, const T2* tw, int accumulate,
                         double* partials, int64_t slot_stride, cudaStream_t s) {
    const size_t sm = sm_rows(false);
    const unsigned nblk = (unsigned)(((int64_t)N * N + L - 1) / L);
    GATO_TRY(smem_attr(k_rows_inv<T, R1, R2, L, NO>, sm));
    GATO_TRY(launch_chained(k_rows_inv<T, R1, R2, L, NO>, nblk, NT, sm, s, a, f0, nfg, S1, tw, accumulate, partials, slot_stride));
    return GATO_OK;
  }
  static int rows_inv_j(const PassArgs& a, int f0, int nfg, const T2* S1, const T2* tw, cudaStream_t s) {
    const size_t sm = sm_rows(false);
    const unsigned nblk = (unsigned)(((int64_t)N * N + L - 1) / L);
    GATO_TRY(smem_attr(k_rows_inv_j<T, R1, R2, L>, sm));
    GATO_TRY(launch_chained(k_rows_inv_j<T, R1, R2, L>, dim3(nblk, nfg), NT, sm, s, (T*)a.jbase, a.jstride, f0, S1, tw));
    return GATO_OK;
  }
  static int rows_inv(const PassArgs& a, int f0, int nfg, const T2* S1, const T2* tw, int accumulate,
                      bool energy, double* partials, int64_t slot_stride, cudaStream_t s) {
    if (energy) return rows_inv_no<0>(a, f0, nfg, S1, tw, accumulate, partials, slot_stride, s);
    if (a.nout <= 1) return rows_inv_no<1>(a, f0, nfg, S1, tw, accumulate, partials, slot_stride, s);
    if (a.nout <= 2) return rows_inv_no<2>(a, f0, nfg, S1, tw, accumulate, partials, slot_stride, s);
    if (a.nout <= 4) return rows_inv_no<4>(a, f0, nfg, S1, tw, accumulate, partials, slot_stride, s);
    return rows_inv_no<8>(a, f0, nfg, S1, tw, accumulate, partials, slot_stride, s);
  }
};

}  // namespace fast
}  // namespace gato
