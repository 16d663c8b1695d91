// Row-parallel panel solve of the blocked Cholesky factorisations (?potrf and the
// mixed-precision factor): the rows below a factored diagonal block are
// independent right-hand sides of L x = b, so one CTA solves 32 or 64 of them with the
// block in shared memory, with no inverse of the block and no extra pass.
#pragma once
#include <cuda_bf16.h>
#include <stdint.h>
#include "block.cuh"
#include "panel.cuh"
#include "scalar.cuh"

namespace cuchol {

__device__ __forceinline__ float round_tf32(float x) {
  uint32_t u;
  asm("cvt.rna.tf32.f32 %0, %1;" : "=r"(u) : "f"(x));
  return __uint_as_float(u);
}
// Rounding of a solved panel value to a tensor-core operand type (BF16: round to
// nearest even; TF32 held in an FP32 word: round to nearest, ties away).
template <typename Op> __device__ __forceinline__ Op to_op(float x);
template <> __device__ __forceinline__ __nv_bfloat16 to_op<__nv_bfloat16>(float x) { return __float2bfloat16_rn(x); }
template <> __device__ __forceinline__ float to_op<float>(float x) { return round_tf32(x); }

// How the panel solve writes its second copy of X (out2, and out3 for the split).
enum : int {
  OUT_COPY = 0,      // out2 = X
  OUT_ROUND = 1,     // out2 = X rounded to the tensor-core operand type O2 (BF16 or TF32)
  OUT_SPLIT = 2,     // out2 = hi = tf32(X), out3 = lo = tf32(X - hi): X = hi + lo to 2^-22
                     // (complex: the two-row form of tcgemm.cuh)
};

// A complex value into the two-row split: (re, im) at o and (-im, re) one row further.
template <typename T>
__device__ __forceinline__ void put_split(T v, float* hi, float* lo, long long o, long long row) {
  const float re = (float)v.x, im = (float)v.y, rh = round_tf32(re), ih = round_tf32(im);
  const float rl = round_tf32(re - rh), il = round_tf32(im - ih);
  *reinterpret_cast<float2*>(hi + o) = make_float2(rh, ih);
  *reinterpret_cast<float2*>(hi + o + row) = make_float2(-ih, rh);
  *reinterpret_cast<float2*>(lo + o) = make_float2(rl, il);
  *reinterpret_cast<float2*>(lo + o + row) = make_float2(-il, rl);
}

// Shared memory of the panel solve of R rows: the row tile Xs (column-major), the parts
// of L below its 16 x 16 diagonal blocks (one column-major strip per sub-panel, from the
// row below the block), the diagonal blocks and the reciprocal pivots.
template <typename T, int NB, int R>
struct SolveSmem {
  static constexpr bool dmma = std::is_same<T, double>::value;
  static constexpr int NP = NB / kSub;
  static constexpr int LDX = R + kLdPad;
  static constexpr size_t X = (sizeof(T) * NB * LDX + 15) / 16 * 16;
  // strip p: rows 16(p+1) .. NB-1, ld = NB - 16(p+1) + kLdPad, 16 columns
  __host__ __device__ static constexpr int strip_ld(int p) { return NB - kSub * (p + 1) + kLdPad; }
  __host__ __device__ static constexpr int strip_off(int p) {
    return kSub * (p * (NB - kSub + kLdPad) - kSub * (p * (p - 1) / 2));
  }
  static constexpr size_t L = sizeof(T) * strip_off(NP - 1);
  static constexpr size_t LDS = sizeof(T) * NP * kSub * kSub;
  static constexpr size_t RD = sizeof(RealOf<T>) * NB;
  static constexpr size_t bytes = X + L + LDS + RD;
};

// Panel solve X = B L^-H in place (L^-T for real types), row-parallel: B (m x jb,
// jb <= NB, logical view B(i, j) = B[i*brs + j*bcs]) is overwritten by X, and X
// also goes to out2 (out2[i*o_rs + j*o_cs]) and, for OUT_SPLIT, out3 (same strides),
// as MODE says.  L: the factored jb x jb diagonal block (view strides lrs, lcs; real
// diagonal).  One CTA of 8 warps solves R rows with the tile and the block in shared
// memory, in 16-column sub-panels: one thread per row substitutes through the 16
// columns; all warps update the next sub-panel; then the next substitution runs while
// the other warps update the columns further right (block.cuh).  Computes in T.
//
// Bound by latency on its critical path (8 sub-panels of about 1000 cycles) and, with
// many rows, by the FP64 rate.
template <typename T, typename O2, int MODE, int NB, int R>
__global__ void __launch_bounds__(256)
    trsm_rows_kernel(T* __restrict__ B, long long brs, long long bcs, int m, int jb, const T* __restrict__ L, long long lrs,
                     long long lcs, O2* __restrict__ out2, long long o_rs, long long o_cs,
                     const int* __restrict__ stop, O2* __restrict__ out3) {
  using SM = SolveSmem<T, NB, R>;
  constexpr int NT = 256, LDX = SM::LDX, SW = R / 32;   // SW warps substitute
  extern __shared__ __align__(16) unsigned char smem_raw[];
  T* Xs = reinterpret_cast<T*>(smem_raw);                       // Xs[col * LDX + row]
  T* Ls = reinterpret_cast<T*>(smem_raw + SM::X);
  T* Ld = reinterpret_cast<T*>(smem_raw + SM::X + SM::L);
  RealOf<T>* rd = reinterpret_cast<RealOf<T>*>(smem_raw + SM::X + SM::L + SM::LDS);
  if (cta_aborted(stop)) return;
  const int t = threadIdx.x, warp = t >> 5, lane = t & 31;
  const int n16 = (jb + kSub - 1) & ~(kSub - 1);
  const long long row0 = (long long)blockIdx.x * R;
  const int rows = min((long long)R, m - row0);

  RealOf<T> dl = RealOf<T>(1);
  if (t < jb) dl = re(L[(long long)t * (lrs + lcs)]);
  // Everything else comes in with cp.async, several copies in flight per thread and in
  // 16-byte pieces where the storage allows (columns contiguous in memory and aligned).
  constexpr int V = 16 / sizeof(T);
  if (V > 1 && brs == 1 && aligned16(B, bcs * (long long)sizeof(T))) {
    constexpr int PC = R / V;                    // pieces of a column of the row tile
#pragma unroll 4
    for (int e = t; e < n16 * PC; e += NT) {
      const int r = (e % PC) * V, c = e / PC;
      const int bytes = (c < jb) ? max(0, min(16, (rows - r) * (int)sizeof(T))) : 0;
      cp_async_piece(&Xs[c * LDX + r], bytes ? B + row0 + r + (long long)c * bcs : B, bytes);
    }
  } else if (brs == 1) {
#pragma unroll 4
    for (int e = t; e < n16 * R; e += NT) {
      const int r = e % R, c = e / R;
      const bool v = r < rows && c < jb;
      cp_async_elem<T>(&Xs[c * LDX + r], v ? B + row0 + r + (long long)c * bcs : B, v);
    }
  } else {                                       // 4 rows x 8 columns per warp and step
    const int dr = lane >> 3, dc = lane & 7;
    for (int r = 4 * warp + dr; r < R; r += 4 * (NT / 32)) {
      const T* src = B + (row0 + r) * brs;
#pragma unroll 4
      for (int c = dc; c < n16; c += 8) {
        const bool v = r < rows && c < jb;
        cp_async_elem<T>(&Xs[c * LDX + r], v ? src + (long long)c * bcs : B, v);
      }
    }
  }
  const bool lvec = V > 1 && lrs == 1 && aligned16(L, lcs * (long long)sizeof(T));
  // the diagonal 16 x 16 blocks: column j at Ld[16 j], row i of its block (on and above
  // the diagonal nothing reads)
  if (lvec) {
    constexpr int PC = kSub / V;
#pragma unroll 4
    for (int e = t; e < n16 * PC; e += NT) {
      const int j = e / PC, i = (j & ~(kSub - 1)) + (e % PC) * V;
      const int bytes = (j < jb) ? max(0, min(16, (jb - i) * (int)sizeof(T))) : 0;
      cp_async_piece(&Ld[e * V], bytes ? L + i + (long long)j * lcs : L, bytes);
    }
  } else {
#pragma unroll 4
    for (int e = t; e < n16 * kSub; e += NT) {
      const int j = e / kSub, i = (j & ~(kSub - 1)) + (e & (kSub - 1));
      const bool v = i > j && i < jb;
      cp_async_elem<T>(&Ld[e], v ? L + (long long)i * lrs + (long long)j * lcs : L, v);
    }
  }
  // the strips of L below them: row r0 = 16 (p + 1) on of column j in strip p
  if (lvec) {
#pragma unroll 2
    for (int j = warp; j < n16 - kSub; j += NT / 32) {
      const int p = j / kSub, r0 = kSub * (p + 1);
      T* S = Ls + SM::strip_off(p) + (j & (kSub - 1)) * SM::strip_ld(p) - r0;
      const T* src = L + (long long)j * lcs;
#pragma unroll
      for (int u = 0; u < (NB / V + 31) / 32; ++u) {
        const int r = r0 + (lane + 32 * u) * V;
        if (r < n16) {
          const int bytes = max(0, min(16, (jb - r) * (int)sizeof(T)));
          cp_async_piece(&S[r], bytes ? src + r : L, bytes);
        }
      }
    }
  } else if (lrs == 1) {
    for (int j = warp; j < n16 - kSub; j += NT / 32) {
      const int p = j / kSub, r0 = kSub * (p + 1);
      T* S = Ls + SM::strip_off(p) + (j & (kSub - 1)) * SM::strip_ld(p) - r0;
      const T* src = L + (long long)j * lcs;
#pragma unroll
      for (int u = 0; u < NB / 32; ++u) {
        const int r = r0 + lane + 32 * u;
        if (r < n16) cp_async_elem<T>(&S[r], r < jb ? src + r : L, r < jb);
      }
    }
  } else {
    const int dr = lane >> 3, dc = lane & 7;
    for (int r = kSub + 4 * warp + dr; r < n16; r += 4 * (NT / 32)) {
      const T* src = L + (long long)r * lrs;
      const int ce = r & ~(kSub - 1);
#pragma unroll 4
      for (int j = dc; j < ce; j += 8) {
        const int p = j / kSub;
        const bool v = r < jb;
        cp_async_elem<T>(&Ls[SM::strip_off(p) + (j & (kSub - 1)) * SM::strip_ld(p) + r - kSub * (p + 1)],
                         v ? src + (long long)j * lcs : L, v);
      }
    }
  }
  if (t < n16) rd[t] = (t < jb) ? RealOf<T>(1) / dl : RealOf<T>(0);
  cp_async_wait_all();
  __syncthreads();

  for (int c0 = 0; c0 < n16; c0 += kSub) {
    const int p = c0 / kSub, c1 = c0 + kSub;
    if (warp < SW) {
      solve16<T>(Xs + c0 * LDX + t, LDX, Ld + p * kSub * kSub, rd + c0);
    } else if (p > 0) {
      // columns past this sub-panel, by the previous one
      int w = warp - SW;
      for (int cb = c1; cb < n16; cb += kSub)
        for (int rb = 0; rb < R; rb += 32) {
          if (w == 0)
            tile_update<T>(Xs + cb * LDX + rb, LDX, Xs + (c0 - kSub) * LDX + rb, LDX,
                           Ls + SM::strip_off(p - 1) + (cb - c0), SM::strip_ld(p - 1), 32);
          w = (w == 0) ? NT / 32 - SW - 1 : w - 1;
        }
    }
    __syncthreads();
    if (c1 >= n16) break;
    strip_update<T, R, NT>(Xs + c1 * LDX, LDX, Xs + c0 * LDX, LDX, Ls + SM::strip_off(p), SM::strip_ld(p), R);
    __syncthreads();
  }

  // the solved tile to each output in the order that is contiguous in that output
  auto put = [&](auto* out, long long rs_, long long cs_, auto conv) {
    if (rs_ == 1) {
      for (int c = warp; c < jb; c += NT / 32) {
        auto* dst = out + row0 + (long long)c * cs_;
#pragma unroll
        for (int r = lane; r < R; r += 32)
          if (r < rows) dst[r] = conv(Xs[c * LDX + r]);
      }
    } else {                                     // 4 rows x 8 columns per warp and step
      const int dr = lane >> 3, dc = lane & 7;
      for (int r = 4 * warp + dr; r < rows; r += 4 * (NT / 32)) {
        auto* dst = out + (row0 + r) * rs_;
#pragma unroll 4
        for (int c = dc; c < jb; c += 8) dst[(long long)c * cs_] = conv(Xs[c * LDX + r]);
      }
    }
  };
  put(B, brs, bcs, [](T v) { return v; });
  if constexpr (MODE == OUT_ROUND) {
    put(out2, o_rs, o_cs, [](T v) { return to_op<O2>((float)v); });
  } else if constexpr (MODE == OUT_SPLIT && Traits<T>::complex) {
    // two rows of the split per row: (re, im) and (-im, re); o_rs floats per row of the split
    for (int r = 4 * warp + (lane >> 3); r < rows; r += 4 * (NT / 32))
    for (int c = lane & 7; c < jb; c += 8) {
      put_split(Xs[c * LDX + r], out2, out3, 2 * (row0 + r) * o_rs + 2 * c, o_rs);
    }
  } else if constexpr (MODE == OUT_SPLIT) {
    put(out2, o_rs, o_cs, [](T v) { return round_tf32((float)v); });
    put(out3, o_rs, o_cs, [](T v) {
      const float hi = round_tf32((float)v);
      return round_tf32((float)v - hi);
    });
  } else {
    put(out2, o_rs, o_cs, [](T v) { return v; });
  }
}

// The diagonal block and the rows below it in one launch, for panels of few rows: every
// CTA factors the NB x NB block for itself, with R of the m rows below it as R more rows of
// its sub-panels, so the rows are solved in the shadow of the pivots and the step has one
// launch instead of two and no pass of the factor through memory.  The block in A must stay
// as it is while CTAs still load it: CTA 0 writes the factor to D (column-major, ld NB),
// and copy_diag_kernel takes it to A later.  Outputs for the rows as trsm_rows_kernel.
// Worth it while the CTAs fit the GPU at once (each is as long as the factor).  A bad pivot: the
// columns before it are finished in all rows, the others are left as they were (the kernels that
// take two launches leave the rows below that block alone).
// T: the computing type; TA: the storage type of A and D (float under double only with rs = 1).
// (Complex double runs 256 threads; bounds of 384 make it 140 registers.  With 190 no CTA of a
// trailing update fits the SM beside this one: zpotrf n = 3000 3.52 ms in place of 3.46.)
template <typename T, typename TA, typename O2, int MODE, int NB, int R, int NT>
__global__ void __launch_bounds__(sizeof(T) == 16 ? 384 : NT)
    panel_kernel(TA* __restrict__ A, long long rs, long long cs, int m, O2* __restrict__ out2, long long o_rs,
                 long long o_cs, O2* __restrict__ out3, TA* __restrict__ D, long long info_base, int first,
                 int* __restrict__ d_info, double* __restrict__ logdet) {
  using F = FactorSmem<T, NB, R>;
  constexpr int LD = F::LD, V = 16 / sizeof(T);
  extern __shared__ __align__(16) unsigned char smem_raw[];
  T* S = reinterpret_cast<T*>(smem_raw);
  T* Ld = reinterpret_cast<T*>(smem_raw + F::S);
  RealOf<T>* rd = reinterpret_cast<RealOf<T>*>(smem_raw + F::S + F::LDS);
  __shared__ int s_fail;
  __shared__ double s_log[NT / 32];
  const int t = threadIdx.x;
  if (first) {                       // starts the words; the other CTAs do not read them
    if (blockIdx.x == 0 && t == 0) {
      *d_info = 0;
      *logdet = 0.0;
    }
  } else if (cta_aborted_before(d_info, info_base)) {
    return;
  }
  const long long row0 = (long long)blockIdx.x * R;
  const int rows = min((long long)R, m - row0);
  TA* B = A + NB * rs;               // the rows below the block
  load_lower<T, TA, NB, NT, LD>(S, A, rs, cs, NB, NB);
  if constexpr (!std::is_same<T, TA>::value) {
    load_widened<R, NB, NT, LD, false>(S + NB, B + row0, cs, rows, NB);
  } else if (V > 1 && rs == 1 && aligned16(B, cs * (long long)sizeof(T))) {
    constexpr int PC = R / V;
#pragma unroll 4
    for (int u = 0; u < NB * PC / NT; ++u) {
      const int e = t + u * NT, r = (e % PC) * V, c = e / PC;
      const int bytes = max(0, min(16, (rows - r) * (int)sizeof(T)));
      cp_async_piece(&S[c * LD + NB + r], bytes ? B + row0 + r + (long long)c * cs : B, bytes);
    }
  } else if (rs == 1) {
#pragma unroll 4
    for (int u = 0; u < NB * R / NT; ++u) {
      const int e = t + u * NT, r = e % R, c = e / R;
      cp_async_elem<T>(&S[c * LD + NB + r], r < rows ? B + row0 + r + (long long)c * cs : B, r < rows);
    }
  } else {
#pragma unroll 4
    for (int u = 0; u < NB * R / NT; ++u) {
      const int e = t + u * NT, c = (e & 7) + 8 * ((e >> 5) % (NB / 8)), r = ((e >> 3) & 3) + 4 * (e / (4 * NB));
      cp_async_elem<T>(&S[c * LD + NB + r], r < rows ? B + (row0 + r) * rs + (long long)c * cs : B, r < rows);
    }
  }
  if (t == 0) s_fail = -1;
  cp_async_wait_all();
  factor_block<T, NB, R, NT>(S, Ld, rd, NB, NB + R, &s_fail, [&](int c0, int cols, int tt, int nt) {
    const T* X = S + c0 * LD + NB;
    if (blockIdx.x == 0)
      for (int e = tt; e < NB * kSub; e += nt) {
        const int r = e % NB, c = c0 + e / NB;
        if (r >= c) D[r + c * NB] = (TA)S[c * LD + r];
      }
    auto put = [&](auto* out, long long rs_, long long cs_, auto conv) {
#pragma unroll 4
      for (int e = tt; e < R * kSub; e += nt) {
        const int r = (rs_ == 1) ? e % R : e / kSub, c = (rs_ == 1) ? e / R : e % kSub;
        if (r < rows && c < cols) out[(row0 + r) * rs_ + (long long)(c0 + c) * cs_] = conv(X[c * LD + r]);
      }
    };
    put(B, rs, cs, [](T v) { return (TA)v; });
    if constexpr (MODE == OUT_ROUND) {
      put(out2, o_rs, o_cs, [](T v) { return to_op<O2>((float)v); });
    } else if constexpr (MODE == OUT_SPLIT && Traits<T>::complex) {
#pragma unroll 2
      for (int e = tt; e < R * kSub; e += nt) {
        const int r = e / kSub, c = e % kSub;
        if (r < rows && c < cols) put_split(X[c * LD + r], out2, out3, 2 * (row0 + r) * o_rs + 2 * (c0 + c), o_rs);
      }
    } else if constexpr (MODE == OUT_SPLIT) {
      put(out2, o_rs, o_cs, [](T v) { return round_tf32((float)v); });
      put(out3, o_rs, o_cs, [](T v) {
        const float hi = round_tf32((float)v);
        return round_tf32((float)v - hi);
      });
    } else {
      put(out2, o_rs, o_cs, [](T v) { return v; });
    }
  });
  if (blockIdx.x != 0) return;
  if (s_fail >= 0) {
    if (t == 0) atomicCAS(d_info, 0, (int)(info_base + s_fail + 1));
  } else if (logdet != nullptr) {
    add_logdet<T, NB, LD>(S, NB, s_log, logdet);
  }
}

// The factored diagonal blocks first_block + blockIdx.x from D (slot 0: block slot0) to A: the lower triangle of every
// block before the one that failed, and of that one the columns before the failing one.
template <typename T, int NB>
__global__ void __launch_bounds__(256)
    copy_diag_kernel(const T* __restrict__ D, int slot0, T* __restrict__ A, long long rs, long long cs, int first_block,
                     const int* __restrict__ d_info) {
  const int b = first_block + blockIdx.x, info = *d_info;
  const int cols = (info == 0) ? NB : min(NB, info - 1 - b * NB);
  const T* d = D + (size_t)(b - slot0) * NB * NB;
  T* a = A + (long long)b * NB * (rs + cs);
  for (int e = threadIdx.x; e < NB * NB; e += 256) {
    const int r = (rs == 1) ? e % NB : e / NB, c = (rs == 1) ? e / NB : e % NB;
    if (r >= c && c < cols) a[r * rs + c * cs] = d[r + c * NB];
  }
}

}  // namespace cuchol
