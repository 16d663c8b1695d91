// Diagonal-block kernels of the blocked factor and inverse (one CTA per block), on the
// building blocks of block.cuh.
//
//   diag_factor_kernel  Cholesky factor of one diagonal block, in place; reports the
//                       first failing pivot and adds the block's log det share.
//   diag_factor_block   the same as part of a larger kernel (batched forms), and the
//                       inverse W = inv(L) with explicit zeros above the diagonal,
//                       which turns a panel solve L21 = A21 L11^-H into a product.
//   diag_invert_kernel  in-place inverse of every nb x nb diagonal block of a
//                       triangular matrix (the leaves of ?TRTRI).
//
// The diagonal block is factored on the GPU next to the trailing update; the
// reference copied it to the host for a CPU dpotrf every step
// (lapack/dpotrf.c:263-276).
#pragma once
#include "block.cuh"
#include "scalar.cuh"

namespace cuchol {

// ROWS x COLS floats A(r, c), columns contiguous (cs), -> S (column-major, ld LD) as doubles,
// zeros past rows (LOWER: only elements on and below the diagonal inside rows x cols, and
// the one above it).  Two rows per load, up to 16 loads in flight per thread before the first
// is stored: a loop of single elements took 7 of the 34 us of a 128-column block.
template <int ROWS, int COLS, int NT, int LD, bool LOWER>
__device__ __forceinline__ void load_widened(double* S, const float* __restrict__ A, long long cs, int rows, int cols) {
  constexpr int PC = ROWS / 2, N = COLS * PC / NT, U = N < 16 ? N : 16;
  static_assert(COLS * PC % NT == 0 && N % U == 0 && LD % 2 == 0, "whole rounds, 16-byte stores");
  const int t = threadIdx.x;
  const bool pairs = aligned16(A, cs * (long long)sizeof(float));
  for (int u0 = 0; u0 < N; u0 += U) {
    float2 v[U];
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const int e = t + (u0 + u) * NT, r = 2 * (e % PC), c = e / PC;
      v[u] = make_float2(0.f, 0.f);
      if (r < rows && c < cols && (!LOWER || r + 1 >= c)) {
        const float* a = A + r + c * cs;
        if (pairs && r + 1 < rows) {
          v[u] = *reinterpret_cast<const float2*>(a);
        } else {
          v[u].x = a[0];
          if (r + 1 < rows) v[u].y = a[1];
        }
      }
    }
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const int e = t + (u0 + u) * NT, r = 2 * (e % PC), c = e / PC;
      double* d = &S[c * LD + r];
      if (!LOWER || (r + 1 < rows && c < cols && r + 1 >= c)) *reinterpret_cast<double2*>(d) = make_double2(v[u].x, v[u].y);
      else if (r < rows && c < cols && r >= c) *d = v[u].x;
    }
  }
}

// Lower part of the logical block A(r, c) (strides rs, cs) -> S (column-major, ld LD),
// order jb padded to n16 with the identity.  Index arithmetic with compile-time extents
// and several copies in flight per thread: with a loop per column this load took as long
// as 60 pivots.  Aligned columns come in 16-byte pieces (the first piece of a column may
// bring elements from above the diagonal along, which nothing reads).
template <typename T, typename TA, int NB, int NT, int LD = FactorSmem<T, NB>::LD>
__device__ __forceinline__ void load_lower(T* S, const TA* __restrict__ A, long long rs, long long cs, int jb, int n16) {
  const int t = threadIdx.x;
  // the identity past jb
  for (int e = t; e < n16 * (n16 - jb); e += NT) {
    const int r = jb + e / n16, c = e % n16;
    if (r >= c) S[c * LD + r] = from_real<T>(RealOf<T>(r == c ? 1 : 0));
  }
  if constexpr (std::is_same<T, TA>::value) {
    constexpr int V = 16 / sizeof(T);
    if (V > 1 && rs == 1 && aligned16(A, cs * (long long)sizeof(T))) {
      constexpr int PC = NB / V;                 // pieces of a column
#pragma unroll 8
      for (int u = 0; u < NB * PC / NT; ++u) {
        const int e = t + u * NT, r = (e % PC) * V, c = e / PC;
        if (r + V > c && r < jb && c < jb) {
          // a piece that crosses jb would overwrite the identity's zeros with zeros
          cp_async_piece(&S[c * LD + r], A + r + c * cs, min(16, (jb - r) * (int)sizeof(T)));
        }
      }
      return;
    }
    if (rs == 1) {
#pragma unroll 8
      for (int u = 0; u < NB * NB / NT; ++u) {
        const int e = t + u * NT, r = e % NB, c = e / NB;
        if (r >= c && r < jb) cp_async_elem<T>(&S[c * LD + r], A + r + c * cs, true);
      }
    } else {
      // columns contiguous: a warp takes 8 columns of 4 rows (64-byte pieces of rows)
#pragma unroll 8
      for (int u = 0; u < NB * NB / NT; ++u) {
        const int e = t + u * NT, c = (e & 7) + 8 * ((e >> 5) % (NB / 8)), r = ((e >> 3) & 3) + 4 * (e / (4 * NB));
        if (r >= c && r < jb) cp_async_elem<T>(&S[c * LD + r], A + r * rs + c * cs, true);
      }
    }
  } else if (rs == 1) {
    load_widened<NB, NB, NT, LD, true>(S, A, cs, jb, jb);
  } else {
#pragma unroll 8
    for (int u = 0; u < NB * NB / NT; ++u) {
      const int e = t + u * NT, r = e % NB, c = e / NB;
      if (r >= c && r < jb) S[c * LD + r] = (T)A[r * rs + c * cs];
    }
  }
}

// *logdet += 2 sum log L(j,j) of the factored block, one column per thread, reduced in a
// fixed order (deterministic).
template <typename T, int NB, int LD>
__device__ __forceinline__ void add_logdet(const T* S, int jb, double* s_log, double* __restrict__ logdet) {
  const int tid = threadIdx.x;
  double s = (tid < jb) ? log((double)re(S[tid * LD + tid])) : 0.0;
  for (int o = 16; o > 0; o >>= 1) s += __shfl_down_sync(0xffffffffu, s, o);
  if ((tid & 31) == 0) s_log[tid >> 5] = s;
  __syncthreads();
  if (tid == 0) {
    for (int w = 1; w < (NB + 31) / 32; ++w) s += s_log[w];
    *logdet += 2.0 * s;
  }
}

// Cholesky factor of one jb x jb diagonal block, jb <= NB, in place, by the whole CTA;
// T: computing type, TA: storage type; smem: FactorSmem<T, NB>::bytes, which keep the
// factor (S) and the reciprocal pivots.  On failure at local column k: *d_info =
// info_base + k + 1 (if still 0), the columns before k are written back, false.
template <typename T, typename TA, int NB, int NT, bool ROOT = true>
__device__ __forceinline__ bool factor_diag(unsigned char* smem, TA* __restrict__ A, long long rs, long long cs, int jb,
                                            long long info_base, int* __restrict__ d_info, double* __restrict__ logdet) {
  using F = FactorSmem<T, NB>;
  constexpr int LD = F::LD;
  T* S = reinterpret_cast<T*>(smem);
  T* Ld = reinterpret_cast<T*>(smem + F::S);
  RealOf<T>* rd = reinterpret_cast<RealOf<T>*>(smem + F::S + F::LDS);
  __shared__ int s_fail;
  __shared__ double s_log[NT / 32];
  const int tid = threadIdx.x, n16 = (jb + kSub - 1) & ~(kSub - 1);
  load_lower<T, TA, NB, NT>(S, A, rs, cs, jb, n16);
  if (tid == 0) s_fail = -1;
  cp_async_wait_all();
  factor_block<T, NB, 0, NT, ROOT>(S, Ld, rd, n16, n16, &s_fail, [&](int c0, int cols, int t, int nt) {
    // columns c0 .. c0 + cols - 1 of the factor back to A
    const int rows = jb - c0, ce = min(jb, c0 + cols);
    if (rs == 1) {
      for (int e = t >> 5; e < 4 * kSub; e += nt >> 5) {       // a warp per column and quarter
        const int c = c0 + (e & (kSub - 1));
        const int r = c0 + 32 * (e / kSub) + (t & 31);
        if (c < ce && r < jb && r >= c) A[r * rs + c * cs] = (TA)S[c * LD + r];
      }
    } else {
      for (int e = t; e < rows * kSub; e += nt) {
        const int c = c0 + (e & (kSub - 1)), r = c0 + e / kSub;
        if (c < ce && r >= c) A[r * rs + c * cs] = (TA)S[c * LD + r];
      }
    }
  });
  if (s_fail >= 0) {
    if (tid == 0) atomicCAS(d_info, 0, (int)(info_base + s_fail + 1));
    return false;
  }
  if (logdet != nullptr) add_logdet<T, NB, LD>(S, jb, s_log, logdet);
  return true;
}

// One diagonal block.  Bound by the chain of pivots.  One block on a B200 under ncu (cold),
// column by column before, sub-panels of 16 columns now: FP64 128 columns 73 -> 27 us, FP32
// 52 -> 21, complex 75 -> 36, 64 columns of complex double 52 -> 19.
template <typename T, typename TA, int NB, int NT>
__global__ void __launch_bounds__(NT)
diag_factor_kernel(TA* __restrict__ A, long long rs, long long cs, int jb, long long info_base, int first,
                   int* __restrict__ d_info, double* __restrict__ logdet) {
  if (first) {                       // starts the words: no launch of its own clears them
    if (threadIdx.x == 0) {
      *d_info = 0;
      *logdet = 0.0;
    }
  } else if (cta_aborted(d_info)) {
    return;                          // an earlier block already failed
  }
  extern __shared__ __align__(16) unsigned char smem_raw[];
  factor_diag<T, TA, NB, NT>(smem_raw, A, rs, cs, jb, info_base, d_info, logdet);
}

// The factor, and, if W is not null, W = inv(L) as a full jb x jb matrix (ldw), zeros
// above the diagonal (not written on failure).  smem: BlockSmem<T, NB>::bytes.
template <typename T, int NB, int NT>
__device__ __forceinline__ void diag_factor_block(T* __restrict__ A, long long rs, long long cs, int jb,
                                                  T* __restrict__ W, int ldw, long long info_base,
                                                  int* __restrict__ d_info, double* __restrict__ logdet) {
  static_assert(!Traits<T>::complex, "the reciprocal pivots serve as 1 / L(i, i)");
  using F = FactorSmem<T, NB>;
  constexpr int LD = F::LD;
  if (cta_aborted(d_info)) return;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  if (!factor_diag<T, T, NB, NT, false>(smem_raw, A, rs, cs, jb, info_base, d_info, logdet) || W == nullptr) return;
  T* S = reinterpret_cast<T*>(smem_raw);
  const T* rd = reinterpret_cast<const T*>(smem_raw + F::S + F::LDS);
  T* TMP = reinterpret_cast<T*>(smem_raw + BlockSmem<T, NB>::F + BlockSmem<T, NB>::RD);
  invert_block<T, NB, NT>(S, (jb + kSub - 1) & ~(kSub - 1), rd, TMP);
  for (int e = threadIdx.x; e < NB * NB; e += NT) {
    const int r = e % NB, c = e / NB;
    if (r < jb && c < jb) W[r + (long long)c * ldw] = (r >= c) ? S[c * LD + r] : zero<T>();
  }
}

// One diagonal block of one matrix of a batch (batched factor: one CTA per task).
template <typename T>
struct DiagTask {
  T* a;               // top-left of the block, logical lower view (strides rs, cs)
  long long rs, cs;
  int jb;
  T* w;               // inverse of the factored block (ld ldw), or null
  int ldw;
  long long info_base;
  int* info;          // the matrix's info word (later steps skip once it is set)
  double* logdet;     // the matrix's log det accumulator, or null
};

template <typename T, int NB, int NT>
__global__ void __launch_bounds__(NT) diag_factor_batched_kernel(const DiagTask<T>* __restrict__ tasks) {
  const DiagTask<T> t = tasks[blockIdx.x];
  diag_factor_block<T, NB, NT>(t.a, t.rs, t.cs, t.jb, t.w, t.ldw, t.info_base, t.info, t.logdet);
}

template <typename T, int NB, int NT>
__device__ __forceinline__ void diag_invert_block(T* __restrict__ B, long long rs, long long cs, int jb,
                                                  int unit);

// In-place inverse of the diagonal blocks [b*nb, b*nb + jb) of a triangular matrix
// (blockIdx.x = b), nb <= NB.  Only the lower triangle of each block is read or
// written; unit: the diagonal is taken as 1 and left untouched.
template <typename T, int NB, int NT>
__global__ void __launch_bounds__(NT)
diag_invert_kernel(T* __restrict__ A, long long rs, long long cs, int n, int nb, int unit) {
  const int o = blockIdx.x * nb;
  diag_invert_block<T, NB, NT>(A + o * rs + o * cs, rs, cs, min(nb, n - o), unit);
}

// In-place inverse of one diagonal block of one matrix of a batch.
template <typename T>
struct InvTask {
  T* b;               // top-left of the block (strides rs, cs)
  long long rs, cs;
  int jb;
  int unit;
  const int* stop;    // skip when this word is non-zero (the matrix's factor failed)
};

template <typename T, int NB, int NT>
__global__ void __launch_bounds__(NT) diag_invert_batched_kernel(const InvTask<T>* __restrict__ tasks) {
  const InvTask<T> t = tasks[blockIdx.x];
  if (cta_aborted(t.stop)) return;
  diag_invert_block<T, NB, NT>(t.b, t.rs, t.cs, t.jb, t.unit);
}

template <typename T, int NB, int NT>
__device__ __forceinline__ void diag_invert_block(T* __restrict__ B, long long rs, long long cs, int jb,
                                                  int unit) {
  using F = FactorSmem<T, NB>;
  constexpr int LD = F::LD;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  T* S = reinterpret_cast<T*>(smem_raw);
  T* rd = reinterpret_cast<T*>(smem_raw + BlockSmem<T, NB>::F);
  T* TMP = reinterpret_cast<T*>(smem_raw + BlockSmem<T, NB>::F + BlockSmem<T, NB>::RD);
  const int n16 = (jb + kSub - 1) & ~(kSub - 1);
  load_lower<T, T, NB, NT>(S, B, rs, cs, jb, n16);
  cp_async_wait_all();
  __syncthreads();
  for (int i = threadIdx.x; i < n16; i += NT) rd[i] = unit ? from_real<T>(RealOf<T>(1)) : recip(S[i * LD + i]);
  invert_block<T, NB, NT>(S, n16, rd, TMP);
  auto put = [&](int r, int c) {
    if (r < jb && c < jb && (r > c || (r == c && !unit))) B[r * rs + c * cs] = S[c * LD + r];
  };
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (rs == 1) {
    for (int c = warp; c < jb; c += NT / 32)
      for (int r = (c & ~31) + lane; r < jb; r += 32) put(r, c);
  } else {
    for (int r = 4 * warp + (lane >> 3); r < jb; r += 4 * (NT / 32))
      for (int c = lane & 7; c <= r; c += 8) put(r, c);
  }
}

}  // namespace cuchol
