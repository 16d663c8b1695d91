// In-shared-memory building blocks of the panel kernels (panel.cuh, trsm.cuh): the
// factor of a diagonal block, the triangular solve of rows below it, and the updates
// between them, all in 16-column sub-panels.
//
// What bounds them is latency: a pivot must be known before the next column starts, so
// the code is written around that chain, and everything that is not on it is done by
// other warps at the same time.
//   * factor16 (one warp): lane i holds row i of the sub-panel, 16 columns in registers.
//     Per pivot the chain is one warp shuffle (the pivot), the reciprocal square root,
//     one multiplication and one fused multiply-add: the next pivot d' = a' - |l|^2 needs
//     only values of its own lane.  The column itself goes through shared memory to the
//     other lanes in the shadow of the next pivot's square root.  A warp issues in order,
//     so this overlap exists only if the whole body is one basic block: no early exit on
//     a bad pivot (its column is noted, the rest computes on rubbish that is not stored)
//     and no slow path inside.
//   * solve16 (one thread per row): right-looking substitution through 16 columns.
//   * tile_update (one warp): C(32 x 16) -= P Q^H over 16 columns; FP64 on DMMA.
// The diagonal 16 x 16 block of L is kept a second time in Ld, column j at Ld[16 j], so
// that the loops read it with aligned 16-byte loads; with ROOT its diagonal holds the pivots
// (the squares of the diagonal elements).
// ROOT: the diagonal is the rounded square root of the pivot.  Without it is the pivot times its
// reciprocal root, as the columns are scaled, up to an ulp off: the factor of order 16 to 200 errs
// 6% more in FP64.  The batched kernels go without: there the root is on the chain of a block of
// 64 (10,000 matrices in FP32 28.5 against 27.6 ms), and their errors are those of the
// condition numbers.
#pragma once
#include <stdint.h>
#include <type_traits>
#include "scalar.cuh"

namespace cuchol {

// Asynchronous global -> shared copy of one element (cp.async: no register
// staging, every copy of a loop is in flight at once); valid = false writes zeros.
template <typename T>
__device__ __forceinline__ void cp_async_elem(T* dst, const T* src, bool valid) {
  const unsigned d = static_cast<unsigned>(__cvta_generic_to_shared(dst));
  const int n = valid ? (int)sizeof(T) : 0;
  if constexpr (sizeof(T) == 16) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(d), "l"(src), "r"(n) : "memory");
  } else {
    asm volatile("cp.async.ca.shared.global [%0], [%1], %2, %3;" ::"r"(d), "l"(src), "n"(sizeof(T)), "r"(n)
                 : "memory");
  }
}
// The first `bytes` (0 .. 16) of a 16-byte piece, the rest zero; both addresses 16-byte
// aligned.
__device__ __forceinline__ void cp_async_piece(void* dst, const void* src, int bytes) {
  const unsigned d = static_cast<unsigned>(__cvta_generic_to_shared(dst));
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(d), "l"(src), "r"(bytes) : "memory");
}
__device__ __forceinline__ bool aligned16(const void* p, long long stride_bytes) {
  return ((reinterpret_cast<uintptr_t>(p) | (uintptr_t)stride_bytes) & 15) == 0;
}
__device__ __forceinline__ void cp_async_wait_all() {
  asm volatile("cp.async.commit_group;\ncp.async.wait_group 0;" ::: "memory");
}

constexpr int kSub = 16;             // sub-panel columns
constexpr int kSubRows = 32;         // rows factor16 covers: the 16 x 16 block and 16 rows below

// Shared leading dimensions are = 4 (mod 16): a DMMA fragment load (8 rows x 4 k) then
// touches 16 distinct 8-byte banks per half warp.
constexpr int kLdPad = 4;

// 1 / sqrt(d) for the pivot chain, for normal positive finite d, without branches.  FP32:
// the hardware estimate.  FP64: the hardware estimate y (relative error below 2^-20)
// refined by the Taylor series of (1 - e)^(-1/2), e = 1 - d y^2, |e| < 2^-19, to second
// order (the dropped term is 5/16 e^3 < 2^-58): four dependent FP64 operations after the
// estimate.
__device__ __forceinline__ float pivot_rsqrt(float d) {
  float y;
  asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(d));
  return y;
}
__device__ __forceinline__ double pivot_rsqrt(double d) {
  double y;
  asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(d));
  const double e = fma(-d * y, y, 1.0);
  return fma(y * e, fma(0.375, e, 0.5), y);
}
// Not a normal positive finite number (one integer subtraction and comparison).
__device__ __forceinline__ bool odd_pivot(float d) { return (unsigned)(__float_as_int(d) - 0x00800000) >= 0x7f000000u; }
__device__ __forceinline__ bool odd_pivot(double d) { return (unsigned)(__double2hiint(d) - 0x00100000) >= 0x7fe00000u; }

// Elements FROM .. 15 of 16 at a 16-byte aligned shared address, in 16-byte loads.
template <int FROM, typename T>
__device__ __forceinline__ void load_row16(const T* p, T (&v)[kSub]) {
  constexpr int per = 16 / sizeof(T);
  const int4* q = reinterpret_cast<const int4*>(p);
#pragma unroll
  for (int u = FROM / per; u < kSub / per; ++u) {
    const int4 w = q[u];
    memcpy(&v[u * per], &w, 16);
  }
}

__device__ __forceinline__ void fms(float& acc, float a, float b) { acc = fmaf(-a, b, acc); }
__device__ __forceinline__ void fms(double& acc, double a, double b) { acc = fma(-a, b, acc); }
__device__ __forceinline__ void fms(cuFloatComplex& acc, cuFloatComplex a, cuFloatComplex b) {
  acc.x = fmaf(-a.x, b.x, acc.x); acc.x = fmaf(a.y, b.y, acc.x);
  acc.y = fmaf(-a.x, b.y, acc.y); acc.y = fmaf(-a.y, b.x, acc.y);
}
__device__ __forceinline__ void fms(cuDoubleComplex& acc, cuDoubleComplex a, cuDoubleComplex b) {
  acc.x = fma(-a.x, b.x, acc.x); acc.x = fma(a.y, b.y, acc.x);
  acc.y = fma(-a.x, b.y, acc.y); acc.y = fma(-a.y, b.x, acc.y);
}
__device__ __forceinline__ float minus_abs2(float a, float l) { return fmaf(-l, l, a); }
__device__ __forceinline__ double minus_abs2(double a, double l) { return fma(-l, l, a); }
__device__ __forceinline__ float minus_abs2(cuFloatComplex a, cuFloatComplex l) { return fmaf(-l.y, l.y, fmaf(-l.x, l.x, a.x)); }
__device__ __forceinline__ double minus_abs2(cuDoubleComplex a, cuDoubleComplex l) { return fma(-l.y, l.y, fma(-l.x, l.x, a.x)); }

// One warp.  S: the sub-panel's top-left element (column-major, ld), rows 0 .. 31 of it,
// of which those below nrows exist; factors the 16 columns in place, writes Ld and the
// reciprocal pivots rd[0..15].  Returns the first failing column (pivot <= 0 or NaN) or
// -1, the same in every lane; the columns before it are then done and the others as
// they were.
//
// factor16_slow: the plain loop.  factor16 leaves every sub-panel with a pivot that is
// not a normal positive number to it (non-SPD blocks, infinities, subnormals), so the
// fast code carries one integer test per pivot and no failure handling.
template <typename T>
__device__ __noinline__ int factor16_slow(T* S, int ld, int nrows, T* Ld, RealOf<T>* rd) {
  using R = RealOf<T>;
  const int i = threadIdx.x & 31;
  for (int j = 0; j < kSub; ++j) {
    __syncwarp();
    R d = re(S[j * ld + j]);
    T a = (i < nrows) ? S[j * ld + i] : zero<T>();
    for (int k = 0; k < j; ++k) {
      const T ljk = S[k * ld + j];
      d = minus_abs2(from_real<T>(d), ljk);
      if (i < nrows) fms(a, S[k * ld + i], cj(ljk));
    }
    if (!(d > R(0))) return j;
    const R r = R(1) / sqrt(d);
    const T l = (i == j) ? from_real<T>(sqrt(d)) : scale(a, r);
    __syncwarp();
    if (i < nrows && i >= j) S[j * ld + i] = l;
    if (i < kSub) Ld[j * kSub + i] = (i == j) ? from_real<T>(d) : l;
    if (i == 0) rd[j] = r;
  }
  __syncwarp();
  return -1;
}

// Step J of factor16 and the ones after it: x the row, r the reciprocal square root of
// the pivot of column J.  (On lane J the update formula makes x[J] the pivot itself.)
template <bool ROOT, int J, typename T>
__device__ __forceinline__ void factor16_steps(T (&x)[kSub], RealOf<T> r, int i, T* Ld, RealOf<T>* rd, bool& odd) {
  using R = RealOf<T>;
  if constexpr (J < kSub) {
    if (ROOT && i == J) Ld[J * kSub + J] = from_real<T>(re(x[J]));
    x[J] = scale(x[J], r);
    R rn = R(1);
    if constexpr (J + 1 < kSub) {
      const R dn = __shfl_sync(0xffffffffu, minus_abs2(x[J + 1], x[J]), J + 1);
      odd = odd || odd_pivot(dn);
      rn = pivot_rsqrt(dn);
    }
    if (i < kSub && !(ROOT && i == J)) Ld[J * kSub + i] = x[J];
    if (i == 0) rd[J] = r;
    if constexpr (J + 1 < kSub) {
      __syncwarp();
      T v[kSub];
      load_row16<J + 1>(Ld + J * kSub, v);
#pragma unroll
      for (int q = J + 1; q < kSub; ++q) fms(x[q], x[J], cj(v[q]));
      factor16_steps<ROOT, J + 1>(x, rn, i, Ld, rd, odd);
    }
  }
}

template <bool ROOT, typename T>
__device__ __forceinline__ int factor16(T* S, int ld, int nrows, T* Ld, RealOf<T>* rd) {
  using R = RealOf<T>;
  const int i = threadIdx.x & 31;
  const bool mine = i < nrows;
  T x[kSub];
#pragma unroll
  for (int q = 0; q < kSub; ++q) x[q] = mine ? S[q * ld + i] : zero<T>();
  const R d = __shfl_sync(0xffffffffu, re(x[0]), 0);
  bool odd = odd_pivot(d);
  static_assert(ROOT || !Traits<T>::complex, "the diagonal's imaginary part goes with the root");
  factor16_steps<ROOT, 0>(x, pivot_rsqrt(d), i, Ld, rd, odd);
  if (odd) return factor16_slow<T>(S, ld, nrows, Ld, rd);
#pragma unroll
  for (int q = 0; q < kSub; ++q) {
    if (mine && (ROOT ? i > q : i >= q)) S[q * ld + i] = x[q];
  }
  return -1;
}

// Step J of solve16 and the ones after it: v holds column J of the block.  The next
// column is loaded one step ahead and no further: left alone the compiler hoists all 64
// loads to the front and spills.
template <int J, typename T>
__device__ __forceinline__ void solve16_steps(T (&x)[kSub], const T (&v)[kSub], const T* Ld, const RealOf<T>* rd) {
  if constexpr (J < kSub) {
    T w[kSub];
    if constexpr (J + 2 < kSub) load_row16<J + 2>(Ld + (J + 1) * kSub, w);
    x[J] = scale(x[J], rd[J]);
    asm volatile("" ::: "memory");
#pragma unroll
    for (int q = J + 1; q < kSub; ++q) fms(x[q], x[J], cj(v[q]));
    solve16_steps<J + 1>(x, w, Ld, rd);
  }
}

// One thread: the row x of 16 columns (elements ld apart from S) solved against the
// factored block: x := x L^-H.  120 FMAs, whose chain is one multiplication and one FMA
// per column.
template <typename T>
__device__ __forceinline__ void solve16(T* S, int ld, const T* Ld, const RealOf<T>* rd) {
  T x[kSub], v[kSub];
#pragma unroll
  for (int q = 0; q < kSub; ++q) x[q] = S[q * ld];
  load_row16<1>(Ld, v);
  solve16_steps<0>(x, v, Ld, rd);
#pragma unroll
  for (int q = 0; q < kSub; ++q) S[q * ld] = x[q];
}

// The first ncols columns only (a block that failed there).
template <typename T>
__device__ __noinline__ void solve16_part(T* S, int ld, const T* Ld, const RealOf<T>* rd, int ncols) {
  for (int j = 0; j < ncols; ++j) {
    T x = S[j * ld];
    for (int k = 0; k < j; ++k) fms(x, S[k * ld], cj(Ld[k * kSub + j]));
    S[j * ld] = scale(x, rd[j]);
  }
}

// 4 elements at a 16-byte aligned shared address.
template <typename T>
__device__ __forceinline__ void load4(const T* p, T (&v)[4]) {
  const int4* q = reinterpret_cast<const int4*>(p);
#pragma unroll
  for (int u = 0; u < (int)sizeof(T) / 4; ++u) {
    const int4 w = q[u];
    memcpy(reinterpret_cast<char*>(v) + 16 * u, &w, 16);
  }
}
template <typename T>
__device__ __forceinline__ void store4(T* p, const T (&v)[4]) {
  int4* q = reinterpret_cast<int4*>(p);
#pragma unroll
  for (int u = 0; u < (int)sizeof(T) / 4; ++u) {
    int4 w;
    memcpy(&w, reinterpret_cast<const char*>(v) + 16 * u, 16);
    q[u] = w;
  }
}

__device__ __forceinline__ void dmma16n8k4(double (&d)[4], double a0, double a1, double b) {
  asm volatile(
      "mma.sync.aligned.m16n8k4.row.col.f64.f64.f64.f64 {%0,%1,%2,%3}, {%4,%5}, {%6}, {%0,%1,%2,%3};\n"
      : "+d"(d[0]), "+d"(d[1]), "+d"(d[2]), "+d"(d[3])
      : "d"(a0), "d"(a1), "d"(b));
}

// One warp: C(r, c) -= sum_{k < 16} P(r, k) conj(Q(c, k)), r < 32, c < 16, all
// column-major in shared memory.  Rows of C and P at or past nr (a multiple of 16) are
// neither read nor written.
// The tile is 32 x 16 because eight warps then cover 128 x 32 or 64 x 64 with every
// lane holding 4 x 4 outputs.  FP64 runs on DMMA: the same flop rate as DFMA, but 6
// shared loads per 4 k instead of 32.  The 16 products are summed from zero and subtracted
// once: product by product from C an FP32 factor of order 100 errs by 1.05e-7 instead of
// 0.51e-7 (against FP64), a complex one by 1.28e-7 instead of 0.58e-7, and C held from the
// start costs panel_kernel<float> 48 bytes of spills (n = 1000: 379 us instead of 345).
template <typename T>
__device__ __forceinline__ void tile_update(T* C, int ldc, const T* P, int ldp, const T* Q, int ldq, int nr) {
  const int lane = threadIdx.x & 31;
  if constexpr (std::is_same<T, double>::value) {
    const int g = lane >> 2, t = lane & 3;
    const bool hi = nr > 16;
    double acc[2][2][4];
#pragma unroll
    for (int a = 0; a < 2; ++a)
#pragma unroll
      for (int b = 0; b < 2; ++b)
#pragma unroll
        for (int e = 0; e < 4; ++e) acc[a][b][e] = 0.0;
#pragma unroll
    for (int k4 = 0; k4 < kSub; k4 += 4) {
      const double* p = P + (k4 + t) * ldp + g;
      const double* q = Q + (k4 + t) * ldq + g;
      const double b0 = q[0], b1 = q[8];
      const double a0 = p[0], a1 = p[8];
      dmma16n8k4(acc[0][0], a0, a1, b0);
      dmma16n8k4(acc[0][1], a0, a1, b1);
      if (hi) {
        const double a2 = p[16], a3 = p[24];
        dmma16n8k4(acc[1][0], a2, a3, b0);
        dmma16n8k4(acc[1][1], a2, a3, b1);
      }
    }
#pragma unroll
    for (int a = 0; a < 2; ++a) {
      if (a == 1 && !hi) break;
#pragma unroll
      for (int b = 0; b < 2; ++b)
#pragma unroll
        for (int e = 0; e < 4; ++e) C[(8 * b + 2 * t + (e & 1)) * ldc + 16 * a + g + 8 * (e >> 1)] -= acc[a][b][e];
    }
  } else {
    // lane: rows 4 lr .. + 3, columns 4 lc .. + 3, all shared accesses in 16-byte pieces
    const int lr = lane & 7, lc = lane >> 3;
    if (4 * lr >= nr) return;
    T acc[4][4];
#pragma unroll
    for (int v = 0; v < 4; ++v)
#pragma unroll
      for (int u = 0; u < 4; ++u) acc[v][u] = zero<T>();
    constexpr int U = sizeof(T) == 4 ? 16 : sizeof(T) == 8 ? 4 : 2;   // operand loads in flight
#pragma unroll U
    for (int k = 0; k < kSub; ++k) {
      T a[4], b[4];
      load4(P + k * ldp + 4 * lr, a);
      load4(Q + k * ldq + 4 * lc, b);
#pragma unroll
      for (int v = 0; v < 4; ++v)
#pragma unroll
        for (int u = 0; u < 4; ++u) mac(acc[v][u], a[u], cj(b[v]));
    }
#pragma unroll
    for (int v = 0; v < 4; ++v) {
      T c[4];
      load4(C + (4 * lc + v) * ldc + 4 * lr, c);
#pragma unroll
      for (int u = 0; u < 4; ++u) c[u] = sub(c[u], acc[v][u]);
      store4(C + (4 * lc + v) * ldc + 4 * lr, c);
    }
  }
}

// All NT threads: C(r, c) -= sum_{k < 16} P(r, k) conj(Q(c, k)), r < R (32 or 64; rows
// at or past nr, a multiple of 16, are left alone), c < 16: the step between two
// sub-panels that is on the critical path.  FP64: one 16 x 8 DMMA tile per warp and pass
// (two independent chains of two DMMAs); otherwise a warp takes two columns and a lane
// one row.
template <typename T, int R, int NT>
__device__ __forceinline__ void strip_update(T* C, int ldc, const T* P, int ldp, const T* Q, int ldq, int nr) {
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if constexpr (std::is_same<T, double>::value) {
    const int g = lane >> 2, t = lane & 3;
    for (int w = warp; w < (R / 16) * 2; w += NT / 32) {
      const int r0 = 16 * (w >> 1), n0 = 8 * (w & 1);
      if (r0 >= nr) continue;
      double acc[2][4] = {};
#pragma unroll
      for (int k4 = 0; k4 < kSub; k4 += 4) {
        const double* p = P + (k4 + t) * ldp + r0 + g;
        dmma16n8k4(acc[(k4 >> 2) & 1], p[0], p[8], Q[(k4 + t) * ldq + n0 + g]);
      }
#pragma unroll
      for (int e = 0; e < 4; ++e) C[(n0 + 2 * t + (e & 1)) * ldc + r0 + g + 8 * (e >> 1)] -= acc[0][e] + acc[1][e];
    }
  } else {
    for (int w = warp; w < (R / 32) * 8; w += NT / 32) {
      const int r = 32 * (w >> 3) + lane, c = 2 * (w & 7);
      if (r >= nr) continue;
      T a0 = zero<T>(), a1 = zero<T>();
#pragma unroll
      for (int k = 0; k < kSub; ++k) {
        const T p = P[k * ldp + r];
        mac(a0, p, cj(Q[k * ldq + c]));
        mac(a1, p, cj(Q[k * ldq + c + 1]));
      }
      C[c * ldc + r] = sub(C[c * ldc + r], a0);
      C[(c + 1) * ldc + r] = sub(C[(c + 1) * ldc + r], a1);
    }
  }
}

// Shared memory of the factor of one block of order up to NB, with R more rows below it
// that are solved along.
template <typename T, int NB, int R = 0>
struct FactorSmem {
  static constexpr int LD = NB + R + kLdPad;
  static constexpr size_t S = sizeof(T) * NB * LD;
  static constexpr size_t LDS = sizeof(T) * kSub * kSub;
  static constexpr size_t RD = sizeof(RealOf<T>) * NB;
  static constexpr size_t bytes = S + LDS + RD;
};

// Cholesky factor of the block in S (order n16, a multiple of 16 up to NB; lower part) and
// the solve of the rows below it (rows n16 .. nrow - 1; nrow a multiple of 16; none: n16),
// by the whole CTA of NT threads, NT / 32 >= 2 warps.  rd[c] = 1 / L(c, c).  done(c0, cols)
// is called by the threads of warps 1 .. (t - 32 counts them) as soon as the columns
// c0 .. c0 + cols - 1 are final, and by all warps for the last ones, with (thread, threads);
// cols is 16, or for the sub-panel that failed the columns before the failing one.
// s_fail (shared, -1 at entry) becomes the first failing column.  Starts and ends with a
// barrier.
//
// Per sub-panel: warp 0 factors the diagonal 16 x 16 (and 16 rows below); one thread per
// remaining row solves; the 32 x 16 elements warp 0 needs next are updated by all
// threads; then warp 0 goes on while the other warps update the rest of the block.
template <typename T, int NB, int R, int NT, bool ROOT = true, typename Done>
__device__ __forceinline__ void factor_block(T* S, T* Ld, RealOf<T>* rd, int n16, int nrow, int* s_fail, Done done) {
  constexpr int LD = FactorSmem<T, NB, R>::LD;
  const int t = threadIdx.x, warp = t >> 5;
  __syncthreads();
  for (int c0 = 0; c0 < n16; c0 += kSub) {
    const int c1 = c0 + kSub;
    if (warp == 0) {
      const int f = factor16<ROOT, T>(S + c0 * LD + c0, LD, nrow - c0, Ld, rd + c0);
      if (t == 0 && f >= 0) *s_fail = c0 + f;
    } else if (c0 > 0) {
      // the rest of the update by the previous sub-panel: 32 x 16 tiles of the columns
      // from c0 on, from the diagonal down (the 32 rows warp 0 works on are done already)
      const int cp = c0 - kSub;
      int w = warp - 1;
      for (int cb = c0; cb < n16; cb += kSub)
        for (int rb = (cb == c0) ? c0 + kSubRows : cb; rb < nrow; rb += 32) {
          if (w == 0)
            tile_update<T>(S + cb * LD + rb, LD, S + cp * LD + rb, LD, S + cp * LD + cb, LD, nrow - rb);
          w = (w == 0) ? NT / 32 - 2 : w - 1;
        }
      done(cp, kSub, t - 32, NT - 32);
    }
    __syncthreads();
    const int fail = *s_fail;
    if constexpr (ROOT) {
      static_assert(NB + R - kSubRows <= NT - kSub, "these threads have no row to solve");
      const int i = t - (NT - kSub);
      if (i >= 0 && (fail < 0 || c0 + i < fail)) S[(c0 + i) * LD + c0 + i] = from_real<T>(sqrt(re(Ld[i * kSub + i])));
    }
    for (int r = c0 + kSubRows + t; r < nrow; r += NT) {
      if (fail < 0) solve16<T>(S + c0 * LD + r, LD, Ld, rd + c0);
      else solve16_part<T>(S + c0 * LD + r, LD, Ld, rd + c0, fail - c0);
    }
    __syncthreads();
    if (fail >= 0 || c1 >= n16) {
      done(c0, fail < 0 ? kSub : fail - c0, t, NT);
      break;
    }
    // the 32 x 16 elements the next factor16 works on
    strip_update<T, kSubRows, NT>(S + c1 * LD + c1, LD, S + c0 * LD + c1, LD, S + c0 * LD + c1, LD, nrow - c1);
    __syncthreads();
  }
  __syncthreads();
}

// Shared memory of a block that is also inverted.
template <typename T, int NB>
struct BlockSmem {
  static constexpr size_t F = (FactorSmem<T, NB>::bytes + 15) / 16 * 16;
  static constexpr size_t RD = sizeof(T) * NB;
  static constexpr size_t TMP = sizeof(T) * (NB / 2) * (NB / 2 + 1);
  static constexpr size_t bytes = F + RD + TMP;
};

// In-place inverse of the lower triangular block in S (order n16, a multiple of 16 up to
// NB, rd[i] = 1 / L(i, i)), by the whole CTA; TMP: (NB/2) x (NB/2 + 1) elements.  The
// part above the diagonal is neither read nor written.  Starts and ends with a barrier.
//
// The 16 x 16 diagonal blocks first, a warp each (lane c: column c by substitution, in
// registers), then pairs of inverted blocks of order b = 16, 32, ..:
//   [L11 0; L21 L22]^-1 = [W11 0; -W22 L21 W11, W22],
// all pairs of a level together, 4 x 4 outputs per thread.
template <typename T, int NB, int NT>
__device__ __forceinline__ void invert_block(T* S, int n16, const T* rd, T* TMP) {
  constexpr int LD = FactorSmem<T, NB>::LD;
  const int t = threadIdx.x, warp = t >> 5, lane = t & 31;
  __syncthreads();
  for (int c0 = kSub * warp; c0 < n16; c0 += kSub * (NT / 32)) {
    T* B = S + c0 * LD + c0;
    const int c = lane & (kSub - 1);
    T x[kSub];
#pragma unroll
    for (int i = 0; i < kSub; ++i) {
      T a0 = zero<T>(), a1 = zero<T>();
#pragma unroll
      for (int k = 0; k < i; ++k) {
        const T l = B[k * LD + i];
        if (k >= c) { if (k & 1) fms(a1, l, x[k]); else fms(a0, l, x[k]); }
      }
      x[i] = (i < c) ? zero<T>() : (i == c) ? rd[c0 + i] : mul(add(a0, a1), rd[c0 + i]);
    }
    __syncwarp();
    if (lane < kSub) {
#pragma unroll
      for (int i = 0; i < kSub; ++i)
        if (i >= c) B[c * LD + i] = x[i];
    }
  }
  __syncthreads();
  for (int b = kSub; b < n16; b *= 2) {
    const int q4 = b / 4, per = q4 * q4, pairs = (n16 - b + 2 * b - 1) / (2 * b), ldt = b + 1;
    // T(r, c) = sum_{k >= c} L21(r, k) W11(k, c)
    for (int e = t; e < pairs * per; e += NT) {
      const int pr = e / per, f = e - pr * per, r = f % q4, cq = 4 * (f / q4);
      const int c0 = 2 * b * pr, r0 = c0 + b;
      const T* L = S + c0 * LD + r0;
      const T* W = S + c0 * LD + c0;
      T acc[4][4];
#pragma unroll
      for (int u = 0; u < 4; ++u)
#pragma unroll
        for (int v = 0; v < 4; ++v) acc[u][v] = zero<T>();
#pragma unroll 4
      for (int k = cq; k < b; ++k) {
        T x[4], y[4];
#pragma unroll
        for (int u = 0; u < 4; ++u) x[u] = (r0 + r + q4 * u < n16) ? L[k * LD + r + q4 * u] : zero<T>();
#pragma unroll
        for (int v = 0; v < 4; ++v) y[v] = (k >= cq + v) ? W[(cq + v) * LD + k] : zero<T>();
#pragma unroll
        for (int u = 0; u < 4; ++u)
#pragma unroll
          for (int v = 0; v < 4; ++v) mac(acc[u][v], x[u], y[v]);
      }
#pragma unroll
      for (int u = 0; u < 4; ++u)
#pragma unroll
        for (int v = 0; v < 4; ++v) TMP[pr * b * ldt + (cq + v) * ldt + r + q4 * u] = acc[u][v];
    }
    __syncthreads();
    // W21(r, c) = -sum_{k <= r} W22(r, k) T(k, c)
    for (int e = t; e < pairs * per; e += NT) {
      const int pr = e / per, f = e - pr * per, r = f % q4, cq = 4 * (f / q4);
      const int c0 = 2 * b * pr, r0 = c0 + b, nr = min(b, n16 - r0);
      const T* W = S + r0 * LD + r0;
      const T* X = TMP + pr * b * ldt;
      T acc[4][4];
#pragma unroll
      for (int u = 0; u < 4; ++u)
#pragma unroll
        for (int v = 0; v < 4; ++v) acc[u][v] = zero<T>();
      const int ke = min(nr, r + 3 * q4 + 1);
#pragma unroll 4
      for (int k = 0; k < ke; ++k) {
        T x[4], y[4];
#pragma unroll
        for (int u = 0; u < 4; ++u) x[u] = (k <= r + q4 * u && r + q4 * u < nr) ? W[k * LD + r + q4 * u] : zero<T>();
#pragma unroll
        for (int v = 0; v < 4; ++v) y[v] = X[(cq + v) * ldt + k];
#pragma unroll
        for (int u = 0; u < 4; ++u)
#pragma unroll
          for (int v = 0; v < 4; ++v) fms(acc[u][v], x[u], y[v]);
      }
#pragma unroll
      for (int u = 0; u < 4; ++u)
        if (r + q4 * u < nr) {
#pragma unroll
          for (int v = 0; v < 4; ++v) S[(c0 + cq + v) * LD + r0 + r + q4 * u] = acc[u][v];
        }
    }
    __syncthreads();
  }
}

}  // namespace cuchol
