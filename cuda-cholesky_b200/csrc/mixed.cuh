// Mixed-precision SPD solve and the FP64 triangular solves under it (included at
// the end of lapack.cu; uses its launch helpers).  No counterpart in the reference
// library, which stops at ?potrf / ?potri (lapack/dpotrf.c:172, lapack/dpotri.c:25):
// the solve follows LAPACK's DSPOSV contract (low-precision factor, FP64
// refinement, FP64 fallback) on the dense SPD path of this library.
//
// Factor (cuDcholMixedCreate):
//   1. s_i = 1 / sqrt(a_ii); W = S A S + shift * I in FP32 (lower, our own buffer):
//      the symmetric diagonal scaling removes the row/column scaling part of
//      kappa(A) before any rounding to low precision.  The shift starts at u / 16 (u
//      the operand unit roundoff) and grows 8x after a breakdown.
//   2. Right-looking blocked Cholesky of W with the two-stream schedule of ?potrf
//      (outer blocks of 512 columns = four 128-column sub-panels, lookahead 1):
//        - diagonal blocks in FP64 on FP32 storage, in one launch with the rows below
//          while those fit the GPU (panel_kernel, FP64 too); otherwise the diagonal
//          kernel and the row-parallel solve in FP32 (trsm_rows_kernel); either writes
//          the rows into W and, rounded to BF16 or TF32, into the k-major operand Q,
//        - trailing updates W22 -= Q Q^T on the tcgen05 tensor cores with FP32
//          accumulation (tc.cuh).
//   3. The inverses of W's 2048-wide diagonal blocks (for the preconditioner).
// Solve (cuDcholMixedSolve): preconditioned conjugate gradients in FP64 on A x = b
// with M^-1 = S L^-T L^-1 S, in groups of 16 right-hand sides, as iterative
// refinement: the loop ends when every normwise backward error
//   |b - A x|_inf / (|A|_inf |x|_inf + |b|_inf)
// computed from a freshly formed FP64 residual is below the tolerance.
// A x uses the FP64 A in the caller's storage (symmetric product from one
// triangle, deterministic); the triangular solves are single launches in which
// row blocks are taken in ticket order and wait (bounded) for the blocks they
// depend on.

#include "tc.cuh"

namespace {
namespace mx {

constexpr int SB = 128;        // sub-panel width: FP64 diagonal blocks
constexpr int OB = 4 * SB;     // outer block: trailing updates with k = 512
constexpr int BS = 64;         // triangular-solve block
constexpr int NR = 16;         // right-hand sides per group
constexpr int SY = 256;        // symmetric-product tile
constexpr int NBT = 2048;      // preconditioner block (inverted diagonal blocks)
constexpr int kThreads = 256;

// ---- factor kernels --------------------------------------------------------------

// s_i = 1 / sqrt(A(i, i)); a diagonal that is not positive sets *bad.
__global__ void scale_kernel(const double* __restrict__ A, long long dstride, int n, double* __restrict__ s,
                             int* __restrict__ bad) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const double a = A[(long long)i * dstride];
  if (!(a > 0.0)) atomicExch(bad, 1);
  s[i] = (a > 0.0) ? 1.0 / sqrt(a) : 0.0;
}

// W(i, j) = s_i A(i, j) s_j (+ shift on the diagonal) for i >= j, FP32.  A is the
// logical lower view A(i, j) = a[i*rs + j*cs]; 32 x 32 tiles through shared memory
// so that both the read (either storage) and the write are coalesced.
__global__ void build_kernel(const double* __restrict__ a, long long rs, long long cs, int n,
                             const double* __restrict__ s, float shift, float* __restrict__ W, long long ldw) {
  __shared__ double t[32][33];
  const int i0 = blockIdx.x * 32, j0 = blockIdx.y * 32;
  if (j0 > i0 + 31) return;
  const int tx = threadIdx.x & 31, ty = threadIdx.x >> 5;   // 32 x 8
  const bool row_contig = (rs == 1);
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    const int r = ty + 8 * k;
    // element (ii, jj) of the tile read by this thread
    const int ii = row_contig ? tx : r, jj = row_contig ? r : tx;
    const int i = i0 + ii, j = j0 + jj;
    t[ii][jj] = (i < n && j < n && i >= j) ? a[(long long)i * rs + (long long)j * cs] : 0.0;
  }
  __syncthreads();
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    const int jj = ty + 8 * k, i = i0 + tx, j = j0 + jj;
    if (i < n && j < n && i >= j) {
      float w = (float)(s[i] * t[tx][jj] * s[j]);
      if (i == j) w += shift;
      W[i + (long long)j * ldw] = w;
    }
  }
}

// ---- triangular solves ------------------------------------------------------------

// Inverse of the 64 x 64 diagonal blocks of a lower-triangular L (logical view
// L(i, j) = L[i*rs + j*cs]); DI[b] is column-major 64 x 64 with zeros above the
// diagonal.  Rows past n of the last block are given a unit diagonal.  One CTA per block,
// in shared memory in 16-wide steps (block.cuh).  (A thread per column with a division
// per row: 53 us FP64.)
template <typename T>
__global__ void __launch_bounds__(kThreads) block_inverse_kernel(const T* __restrict__ L, long long rs, long long cs,
                                                                 int n, T* __restrict__ DI) {
  using BM = BlockSmem<T, BS>;
  constexpr int LD = FactorSmem<T, BS>::LD;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  T* S = reinterpret_cast<T*>(smem_raw);
  T* rd = reinterpret_cast<T*>(smem_raw + BM::F);
  T* TMP = reinterpret_cast<T*>(smem_raw + BM::F + BM::RD);
  const int b = blockIdx.x, i0 = b * BS, t = threadIdx.x;
  load_lower<T, T, BS, kThreads>(S, L + (long long)i0 * (rs + cs), rs, cs, min(BS, n - i0), BS);
  cp_async_wait_all();
  __syncthreads();
  if (t < BS) rd[t] = T(1) / S[t * LD + t];
  invert_block<T, BS, kThreads>(S, BS, rd, TMP);
  T* out = DI + (size_t)b * BS * BS;
  for (int e = t; e < BS * BS; e += kThreads) {
    const int r = e % BS, c = e / BS;
    out[e] = (r >= c) ? S[c * LD + r] : T(0);
  }
}

__device__ __forceinline__ unsigned ld_acquire(const unsigned* p) {
  unsigned v;
  asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}
__device__ __forceinline__ void st_release(unsigned* p, unsigned v) {
  asm volatile("st.release.gpu.global.u32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}

// Thread 0 waits until *ready >= need, for at most `limit` polls (limit < 0: 2^24,
// seconds); returns the value seen.  A wait that gives up sets *err and returns
// `need`, so that the solve still ends (with a wrong result the host then discards).
__device__ __forceinline__ unsigned wait_ready(const unsigned* ready, unsigned need, int* err, int limit) {
  const unsigned polls = limit < 0 ? (1u << 24) : (unsigned)limit;
  for (unsigned it = 0; it < polls; ++it) {
    const unsigned v = ld_acquire(ready);
    if (v >= need) return v;
    if (it > 64) __nanosleep(64);
  }
  atomicExch(err, 1);
  return need;
}

// Y := L^-1 (sc .* B) for up to NR right-hand sides; L lower (view strides rs, cs),
// B of type VB (ldb), Y of type T (ldy, at least 64 * ceil(n / 64) rows).  One CTA
// per 64-row block, blocks taken in ticket order; block I accumulates L(I, J) y_J
// for J < I as the y_J are published (the counter ready = number of finished
// blocks), then applies DI_I.
// Counters: ctr[0] ticket, ctr[1] ready; both zero at launch.
// How the 256 threads share a 64-row step: four row sets of 64 threads take four
// right-hand sides each and, with eight or fewer of them, a half or a quarter of the 64
// columns (one warp per scheduler then runs 16 to 32 FP64 FMAs per column set instead of
// 64, on the chain that every later block waits for).
struct TrsvSplit {
  int g, part, c0, c1, groups;
  __device__ __forceinline__ TrsvSplit(int nrhs, int set) {
    groups = nrhs <= 4 ? 1 : nrhs <= 8 ? 2 : 4;
    g = set % groups;
    part = set / groups;
    const int w = BS * groups / 4;
    c0 = part * w;
    c1 = c0 + w;
  }
};
// v of the sets with part 0 += those of the other parts, in order; by the whole CTA.
template <typename T>
__device__ __forceinline__ void trsv_combine(const TrsvSplit& sp, T (&v)[4], T* Red /* [4][BS][4] */, int r) {
  if (sp.groups == 4) return;
  const int set = sp.part * sp.groups + sp.g;
#pragma unroll
  for (int k = 0; k < 4; ++k) Red[(set * 4 + k) * BS + r] = v[k];
  __syncthreads();
  if (sp.part == 0) {
    for (int q = 1; q < 4 / sp.groups; ++q)
#pragma unroll
      for (int k = 0; k < 4; ++k) v[k] += Red[((q * sp.groups + sp.g) * 4 + k) * BS + r];
  }
}

template <typename T, typename VB>
__global__ void __launch_bounds__(kThreads)
    trsv_fwd_kernel(const T* __restrict__ L, long long rs, long long cs, int n, const T* __restrict__ DI,
                    const VB* __restrict__ B, long long ldb, const double* __restrict__ sc, T* Y, long long ldy,
                    int nrhs, unsigned* ctr, int* err, int wait_limit) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  auto Ls = reinterpret_cast<T(*)[BS + 1]>(smem_raw);           // [BS][BS + 1]
  auto Ds = reinterpret_cast<T(*)[BS + 1]>(smem_raw + sizeof(T) * BS * (BS + 1));
  auto Vs = reinterpret_cast<T(*)[NR]>(smem_raw + 2 * sizeof(T) * BS * (BS + 1));
  T* Red = reinterpret_cast<T*>(smem_raw + 2 * sizeof(T) * BS * (BS + 1)) + BS * NR;
  __shared__ unsigned s_I, s_known;
  const int t = threadIdx.x, r = t & (BS - 1);
  const TrsvSplit sp(nrhs, t >> 6);
  const int g = sp.g;                                            // right-hand sides 4g .. 4g + 3
  if (t == 0) {
    s_I = atomicAdd(&ctr[0], 1u);
    s_known = 0;
  }
  __syncthreads();
  const int I = (int)s_I, i0 = I * BS, i = i0 + r;
  {   // DI_I into shared memory first: the diagonal step then waits on no global load
    const T* D = DI + (size_t)I * BS * BS;
    for (int e = t; e < BS * BS; e += kThreads) Ds[e % BS][e / BS] = D[e];
  }
  const bool row_contig = (rs == 1);
  T acc[4];
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    const int c = g * 4 + k;
    acc[k] = (sp.part == 0 && i < n && c < nrhs) ? (T)(sc != nullptr ? sc[i] * (double)B[i + c * ldb] : (double)B[i + c * ldb])
                                 : T(0);
  }
  // prefetch of the next L block: element e = t + 256 q
  T pre[BS * BS / kThreads];
  auto fetch = [&](int J) {
#pragma unroll
    for (int q = 0; q < BS * BS / kThreads; ++q) {
      const int e = t + kThreads * q;
      const int ii = row_contig ? (e % BS) : (e / BS), jj = row_contig ? (e / BS) : (e % BS);
      pre[q] = (i0 + ii < n) ? L[(long long)(i0 + ii) * rs + (long long)(J * BS + jj) * cs] : T(0);
    }
  };
  if (I > 0) fetch(0);
  for (int J = 0; J < I; ++J) {
#pragma unroll
    for (int q = 0; q < BS * BS / kThreads; ++q) {
      const int e = t + kThreads * q;
      const int ii = row_contig ? (e % BS) : (e / BS), jj = row_contig ? (e / BS) : (e % BS);
      Ls[ii][jj] = pre[q];
    }
    if (J + 1 < I) fetch(J + 1);
    if (t == 0 && s_known < (unsigned)(J + 1)) s_known = wait_ready(&ctr[1], (unsigned)(J + 1), err, wait_limit);
    __syncthreads();
    {
      const int jj = t >> 4, c = t & 15;   // y_J into shared memory (L2 reads: written by another CTA)
      Vs[jj][c] = __ldcg(&Y[(long long)(J * BS + jj) + c * ldy]);
      const int jj2 = jj + 16;
      Vs[jj2][c] = __ldcg(&Y[(long long)(J * BS + jj2) + c * ldy]);
      Vs[jj2 + 16][c] = __ldcg(&Y[(long long)(J * BS + jj2 + 16) + c * ldy]);
      Vs[jj2 + 32][c] = __ldcg(&Y[(long long)(J * BS + jj2 + 32) + c * ldy]);
    }
    __syncthreads();
#pragma unroll 8
    for (int cc = sp.c0; cc < sp.c1; ++cc) {
      const T l = Ls[r][cc];
#pragma unroll
      for (int k = 0; k < 4; ++k) acc[k] -= l * Vs[cc][g * 4 + k];
    }
    __syncthreads();
  }
  // y_I = DI_I acc
  trsv_combine(sp, acc, Red, r);
  if (sp.part == 0) {
#pragma unroll
    for (int k = 0; k < 4; ++k) Vs[r][g * 4 + k] = acc[k];
  }
  __syncthreads();
  T y[4] = {T(0), T(0), T(0), T(0)};
#pragma unroll 8
  for (int cc = sp.c0; cc < sp.c1; ++cc) {
    const T d = Ds[r][cc];
    if (cc <= r) {
#pragma unroll
      for (int k = 0; k < 4; ++k) y[k] += d * Vs[cc][g * 4 + k];
    }
  }
  trsv_combine(sp, y, Red, r);
  if (sp.part == 0) {
#pragma unroll
    for (int k = 0; k < 4; ++k) __stcg(&Y[i + (long long)(g * 4 + k) * ldy], i < n ? y[k] : T(0));
  }
  __threadfence();
  __syncthreads();
  if (t == 0) st_release(&ctr[1], (unsigned)(I + 1));
}

// Z := sc .* (L^-T Y) (type VZ, ldz), the transposed solve of trsv_fwd_kernel:
// blocks taken from the last one; block I accumulates L(J, I)^T z_J for J > I.
// ctr[1] counts finished blocks from the end.  Y and Z may alias (in place).
template <typename T, typename VZ>
__global__ void __launch_bounds__(kThreads)
    trsv_bwd_kernel(const T* __restrict__ L, long long rs, long long cs, int n, const T* __restrict__ DI,
                    const T* Y, long long ldy, const double* __restrict__ sc, VZ* Z, long long ldz, T* Zt,
                    int nrhs, unsigned* ctr, int* err, int wait_limit) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  auto Ls = reinterpret_cast<T(*)[BS + 1]>(smem_raw);           // Ls[c][r] = L(J*BS + c, I*BS + r)
  auto Ds = reinterpret_cast<T(*)[BS + 1]>(smem_raw + sizeof(T) * BS * (BS + 1));   // Ds[r][c] = DI_I(c, r)
  auto Vs = reinterpret_cast<T(*)[NR]>(smem_raw + 2 * sizeof(T) * BS * (BS + 1));
  T* Red = reinterpret_cast<T*>(smem_raw + 2 * sizeof(T) * BS * (BS + 1)) + BS * NR;
  __shared__ unsigned s_I, s_known;
  const int nblk = (n + BS - 1) / BS;
  const int t = threadIdx.x, r = t & (BS - 1);
  const TrsvSplit sp(nrhs, t >> 6);
  const int g = sp.g;
  if (t == 0) {
    s_I = atomicAdd(&ctr[0], 1u);
    s_known = 0;
  }
  __syncthreads();
  const int I = nblk - 1 - (int)s_I, i0 = I * BS, i = i0 + r;
  {
    const T* D = DI + (size_t)I * BS * BS;
    for (int e = t; e < BS * BS; e += kThreads) Ds[e / BS][e % BS] = D[e];
  }
  const bool row_contig = (rs == 1);
  T acc[4];
#pragma unroll
  for (int k = 0; k < 4; ++k) acc[k] = (sp.part == 0 && i < n) ? Y[i + (long long)(g * 4 + k) * ldy] : T(0);
  T pre[BS * BS / kThreads];
  auto fetch = [&](int J) {
#pragma unroll
    for (int q = 0; q < BS * BS / kThreads; ++q) {
      const int e = t + kThreads * q;
      const int cc = row_contig ? (e % BS) : (e / BS), rr = row_contig ? (e / BS) : (e % BS);
      pre[q] = (J * BS + cc < n) ? L[(long long)(J * BS + cc) * rs + (long long)(i0 + rr) * cs] : T(0);
    }
  };
  if (I < nblk - 1) fetch(nblk - 1);
  for (int J = nblk - 1; J > I; --J) {
#pragma unroll
    for (int q = 0; q < BS * BS / kThreads; ++q) {
      const int e = t + kThreads * q;
      const int cc = row_contig ? (e % BS) : (e / BS), rr = row_contig ? (e / BS) : (e % BS);
      Ls[cc][rr] = pre[q];
    }
    if (J - 1 > I) fetch(J - 1);
    const unsigned need = (unsigned)(nblk - J);
    if (t == 0 && s_known < need) s_known = wait_ready(&ctr[1], need, err, wait_limit);
    __syncthreads();
    {
      const int jj = t >> 4, c = t & 15;
#pragma unroll
      for (int q = 0; q < 4; ++q) Vs[jj + 16 * q][c] = __ldcg(&Zt[(long long)(J * BS + jj + 16 * q) + c * ldy]);
    }
    __syncthreads();
#pragma unroll 8
    for (int cc = sp.c0; cc < sp.c1; ++cc) {
      const T l = Ls[cc][r];
#pragma unroll
      for (int k = 0; k < 4; ++k) acc[k] -= l * Vs[cc][g * 4 + k];
    }
    __syncthreads();
  }
  // z_I = DI_I^T acc
  trsv_combine(sp, acc, Red, r);
  if (sp.part == 0) {
#pragma unroll
    for (int k = 0; k < 4; ++k) Vs[r][g * 4 + k] = acc[k];
  }
  __syncthreads();
  T z[4] = {T(0), T(0), T(0), T(0)};
#pragma unroll 8
  for (int cc = sp.c0; cc < sp.c1; ++cc) {
    const T d = Ds[r][cc];
    if (cc >= r) {
#pragma unroll
      for (int k = 0; k < 4; ++k) z[k] += d * Vs[cc][g * 4 + k];
    }
  }
  trsv_combine(sp, z, Red, r);
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    const int c = g * 4 + k;
    if (sp.part != 0) continue;
    __stcg(&Zt[i + (long long)c * ldy], (i < n) ? z[k] : T(0));
    if (i < n && c < nrhs) Z[i + (long long)c * ldz] = (VZ)((sc != nullptr) ? sc[i] * (double)z[k] : (double)z[k]);
  }
  __threadfence();
  __syncthreads();
  if (t == 0) st_release(&ctr[1], (unsigned)(nblk - I));
}

// ---- preconditioner: blocked triangular solves with inverted diagonal blocks -------
// M^-1 r = S F^T F S r with F = the forward solve by L (the FP32 factor), done in
// NBT-wide block steps: y_I = inv(L_II) t_I, then t_below -= L(below, I) y_I (and
// the transposed sequence backwards).  inv(L_II) is formed once per factor, so each
// step is two GEMVs that spread over the whole GPU: no step waits on a chain of
// small blocks.  FP32 throughout (it is the preconditioner); 16 right-hand sides.
constexpr int GR = 64;            // rows (gemv_n) or output columns (gemv_t) per CTA
constexpr int GMP = GR + 4;       // shared row pitch of a 64 x 64 chunk
constexpr int GVP = NR + 4;       // shared row pitch of a vector chunk

__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_async_wait() {
  asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory");
}
__device__ __forceinline__ void cp_async4(void* dst, const void* src, int src_bytes) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(tc::smem_u32(dst)), "l"(src), "r"(src_bytes)
               : "memory");
}
__device__ __forceinline__ void cp_async16_(void* dst, const void* src, int src_bytes) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(tc::smem_u32(dst)), "l"(src), "r"(src_bytes)
               : "memory");
}
constexpr int GST = 4;                                  // cp.async stages
constexpr int GSTAGE = GR * GMP + GR * GVP;             // floats per stage
constexpr size_t kGemvSmem = sizeof(float) * (GST * GSTAGE + 4 * GR * NR);

// The 4 partial 4 x 4 blocks of every thread -> out (alpha, beta), rows/columns
// [o0, o0 + 64) of the output.  With a split k range (gridDim.y > 1) the raw sums go to
// part[split][block][c][o], and the last CTA of the block to arrive at count[block] adds the
// splits in order and resets the count: a second launch for this took 3.7 us and a gap of
// the 15 to 25 us of a product.
constexpr int kGemvSplits = NBT / 256;                  // at most
__device__ __forceinline__ void gemv_finish(float (&acc)[4][4], float* Red, int ig, int cg, int ks, int o0, int m,
                                            float alpha, float beta, const float* in, float* out, long long ldv,
                                            float* part, unsigned* count) {
  const int t = threadIdx.x, o = t & 63, c0 = (t >> 6) * 4, r = o0 + o;
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j) Red[(ks * GR + 4 * ig + i) * NR + 4 * cg + j] = acc[i][j];
  __syncthreads();
  float sum[4];
#pragma unroll
  for (int q = 0; q < 4; ++q) {
    const int c = c0 + q;
    sum[q] = ((Red[(0 * GR + o) * NR + c] + Red[(1 * GR + o) * NR + c]) +
              (Red[(2 * GR + o) * NR + c] + Red[(3 * GR + o) * NR + c]));
  }
  const int ns = gridDim.y;
  if (ns > 1) {
    const long long step = (long long)gridDim.x * GR * NR;
    float* mine = part + (long long)blockIdx.x * GR * NR + c0 * GR + o;
#pragma unroll
    for (int q = 0; q < 4; ++q) mine[blockIdx.y * step + q * GR] = sum[q];
    __threadfence();
    __shared__ bool s_last;
    __syncthreads();
    if (t == 0) s_last = atomicAdd(&count[blockIdx.x], 1u) == (unsigned)ns - 1;
    __syncthreads();
    if (!s_last) return;
    __threadfence();
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      float v[kGemvSplits];
#pragma unroll
      for (int u = 0; u < kGemvSplits; ++u) v[u] = u < ns ? __ldcg(mine + u * step + q * GR) : 0.f;
      sum[q] = 0.f;
#pragma unroll
      for (int u = 0; u < kGemvSplits; ++u) sum[q] += v[u];
    }
    if (t == 0) count[blockIdx.x] = 0;
  }
  if (r >= m) return;
#pragma unroll
  for (int q = 0; q < 4; ++q) {
    const long long e = r + (long long)(c0 + q) * ldv;
    float v = alpha * sum[q];
    if (beta != 0.f) v = fmaf(beta, in[e], v);
    out[e] = v;
  }
}


// 16 consecutive k of the stage: thread block (ig, cg) += A4(ig rows) x V4(cg rhs).
__device__ __forceinline__ void gemv_mac(const float* Ms, const float* Vs, int ig, int cg, int ks,
                                         float (&acc)[4][4]) {
#pragma unroll
  for (int kq = 0; kq < 16; ++kq) {
    const int k = ks * 16 + kq;
    const float4 a = *reinterpret_cast<const float4*>(&Ms[k * GMP + 4 * ig]);
    const float4 b = *reinterpret_cast<const float4*>(&Vs[k * GVP + 4 * cg]);
    const float av[4] = {a.x, a.y, a.z, a.w}, bv[4] = {b.x, b.y, b.z, b.w};
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
      for (int j = 0; j < 4; ++j) acc[i][j] = fmaf(av[i], bv[j], acc[i][j]);
  }
}

// v chunk k0.. (64 x 16) -> Vs[k][c], zero past kk
__device__ __forceinline__ void gemv_issue_v(float* Vs, const float* v, long long ldv, int kk, int k0) {
  const int t = threadIdx.x;
#pragma unroll
  for (int q = 0; q < 4; ++q) {
    const int e = t + kThreads * q, k = e & 63, c = e >> 6, gk = k0 + k;
    cp_async4(&Vs[k * GVP + c], v + (gk < kk ? gk + (long long)c * ldv : 0), gk < kk ? 4 : 0);
  }
}

// out(r, c) = alpha * sum_k M(r, k) v(k, c) + beta * in(r, c), r < m, k < kk.
// M: FP32 column-major (ldm a multiple of 4, 16-byte aligned columns); v / in / out:
// FP32 column-major with leading dimension ldv (in may alias out).  CTA: 64 rows;
// M and v stream through a 4-stage cp.async ring in 64-wide k chunks (each column
// segment of 64 rows = 16 pieces of 16 bytes, stored as Ms[k][row]); thread: 4 rows
// x 4 right-hand sides over a quarter of each chunk.
__global__ void __launch_bounds__(kThreads)
    gemv_n_kernel(const float* __restrict__ M, long long ldm, int m, int kk, const float* __restrict__ v,
                  float alpha, float beta, const float* in, float* out, long long ldv, int kc, float* part,
                  unsigned* count, int tri) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  float* ring = reinterpret_cast<float*>(smem_raw);
  float* Red = ring + GST * GSTAGE;
  const int t = threadIdx.x, ig = t & 15, cg = (t >> 4) & 3, ks = t >> 6;
  const int r0 = blockIdx.x * GR;
  // this CTA's k range [kb, ke): split blockIdx.y of width kc (a multiple of 64); of a
  // lower triangular M only the columns up to the block's last row
  const int kb = (int)blockIdx.y * kc, ke = min(tri ? min(kk, r0 + GR) : kk, kb + kc);
  const int nch = (ke - kb + GR - 1) / GR;
  auto issue = [&](int ch) {
    float* Ms = ring + (ch % GST) * GSTAGE;
    float* Vs = Ms + GR * GMP;
    const int k0 = kb + ch * GR;
#pragma unroll
    for (int q = 0; q < 4; ++q) {   // 16-byte piece f of column col: rows r0 + 4f ..
      const int e = t + kThreads * q, f = e & 15, col = e >> 4, r = r0 + 4 * f, k = k0 + col;
      const float* src = M + r + (long long)k * ldm;
      int bytes = 0;
      if (k < ke && r < m) bytes = (r + 3 < m) ? 16 : 4 * (m - r);
      cp_async16_(&Ms[col * GMP + 4 * f], bytes ? src : M, bytes);
    }
    gemv_issue_v(Vs, v, ldv, ke, k0);
  };
  float acc[4][4] = {};
  for (int ch = 0; ch < GST - 1; ++ch) {
    if (ch < nch) issue(ch);
    cp_async_commit();
  }
  for (int ch = 0; ch < nch; ++ch) {
    cp_async_wait<GST - 2>();
    __syncthreads();
    if (ch + GST - 1 < nch) issue(ch + GST - 1);
    cp_async_commit();
    const float* Ms = ring + (ch % GST) * GSTAGE;
    gemv_mac(Ms, Ms + GR * GMP, ig, cg, ks, acc);
  }
  cp_async_wait<0>();
  gemv_finish(acc, Red, ig, cg, ks, r0, m, alpha, beta, in, out, ldv, part, count);
}

// out(j, c) = alpha * sum_k M(k, j) v(k, c) + beta * in(j, c), j < m, k < kk (the
// transposed product).  CTA: 64 output columns; the chunk is transposed on its way
// into shared memory (4-byte copies, Ms[k][col]) so that a thread reads 4 columns
// with one 16-byte load.
__global__ void __launch_bounds__(kThreads)
    gemv_t_kernel(const float* __restrict__ M, long long ldm, int m, int kk, const float* __restrict__ v,
                  float alpha, float beta, const float* in, float* out, long long ldv, int kc, float* part,
                  unsigned* count, int tri) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  float* ring = reinterpret_cast<float*>(smem_raw);
  float* Red = ring + GST * GSTAGE;
  const int t = threadIdx.x, jg = t & 15, cg = (t >> 4) & 3, ks = t >> 6;
  const int j0 = blockIdx.x * GR;
  // of a lower triangular M only the rows from the block's first column on
  const int k1 = (int)blockIdx.y * kc, kb = max(k1, tri ? j0 : 0), ke = min(kk, k1 + kc);
  const int nch = (ke - kb + GR - 1) / GR;
  auto issue = [&](int ch) {
    float* Ms = ring + (ch % GST) * GSTAGE;
    float* Vs = Ms + GR * GMP;
    const int k0 = kb + ch * GR;
#pragma unroll
    for (int q = 0; q < 16; ++q) {   // element (k, col): consecutive threads, consecutive k
      const int e = t + kThreads * q, k = e & 63, col = e >> 6, gk = k0 + k, j = j0 + col;
      const bool ok = gk < ke && j < m;
      cp_async4(&Ms[k * GMP + col], ok ? M + gk + (long long)j * ldm : M, ok ? 4 : 0);
    }
    gemv_issue_v(Vs, v, ldv, ke, k0);
  };
  float acc[4][4] = {};
  for (int ch = 0; ch < GST - 1; ++ch) {
    if (ch < nch) issue(ch);
    cp_async_commit();
  }
  for (int ch = 0; ch < nch; ++ch) {
    cp_async_wait<GST - 2>();
    __syncthreads();
    if (ch + GST - 1 < nch) issue(ch + GST - 1);
    cp_async_commit();
    const float* Ms = ring + (ch % GST) * GSTAGE;
    gemv_mac(Ms, Ms + GR * GMP, jg, cg, ks, acc);
  }
  cp_async_wait<0>();
  gemv_finish(acc, Red, jg, cg, ks, j0, m, alpha, beta, in, out, ldv, part, count);
}

// t = (float)(s .* r) (NR columns)
__global__ void scale_in_kernel(const double* __restrict__ r, const double* __restrict__ s, int n, long long ld,
                                float* __restrict__ out) {
  for (long long e = blockIdx.x * (long long)blockDim.x + threadIdx.x; e < (long long)n * NR;
       e += (long long)gridDim.x * blockDim.x) {
    const int i = (int)(e % n), c = (int)(e / n);
    out[i + c * ld] = (float)(s[i] * r[i + c * ld]);
  }
}
// z = s .* (double)y
__global__ void scale_out_kernel(const float* __restrict__ y, const double* __restrict__ s, int n, long long ld,
                                 double* __restrict__ z) {
  for (long long e = blockIdx.x * (long long)blockDim.x + threadIdx.x; e < (long long)n * NR;
       e += (long long)gridDim.x * blockDim.x) {
    const int i = (int)(e % n), c = (int)(e / n);
    z[i + c * ld] = s[i] * (double)y[i + c * ld];
  }
}

// dst(i, j) = src(i, j) converted, for i >= j (lower) or all (full); others zero.
template <typename S, typename D>
__global__ void convert_kernel(const S* __restrict__ src, long long lds, D* __restrict__ dst, long long ldd, int n,
                               int lower) {
  const int i = blockIdx.x * 32 + (threadIdx.x & 31);
  for (int j = blockIdx.y * 32 + (threadIdx.x >> 5); j < min(n, blockIdx.y * 32 + 32); j += 8) {
    if (i < n) dst[i + (long long)j * ldd] = (!lower || i >= j) ? (D)src[i + (long long)j * lds] : D(0);
  }
}

// ---- symmetric product A X in FP64 ----------------------------------------------

// Tile task t <-> lower tile (I, J), J <= I, row-major: t = I (I + 1) / 2 + J.
__device__ __forceinline__ void task_tile(int t, int& I, int& J) {
  int r = (int)((sqrt(8.0 * (double)t + 1.0) - 1.0) * 0.5);
  while (r > 0 && r * (r + 1) / 2 > t) --r;
  while ((r + 1) * (r + 2) / 2 <= t) ++r;
  I = r;
  J = t - r * (r + 1) / 2;
}

// Each stored element of the triangle is read once: the CTA of lower tile (I, J)
// writes the partial products U(I,J) = A_IJ X_J (rows of block I) and
// V(I,J) = A_IJ^T X_I (rows of block J; on a diagonal tile only the strictly lower
// part), each SY x NR, row-major [row][rhs].  absval: |A| instead of A.
// The CTA reads its tile in the stored orientation (always whole columns): for
// lower storage T = A(I-rows, J-cols), for upper storage T = A(J-rows, I-cols) =
// A_IJ^T, and then T X and T^T X trade places.  Columns are streamed in 16-column
// chunks through a 3-stage cp.async ring, and both products run on the FP64 tensor
// cores (mma.sync m16n8k4): warp w computes T X for rows [32w, 32w + 32) and a
// partial T^T X over the same 32 rows; the 8 partials are summed in shared memory.
// FP64 tensor-bound at 16 right-hand sides (n^2 * NR FMAs for n^2 / 2 * 8 bytes).
constexpr int kSP = SY + 4;    // S row pitch (doubles): conflict-free fragment loads
constexpr int kXP = NR + 4;    // Xi row pitch
constexpr int kCP = 16 + 4;    // Xc row pitch (Xc[c][jj])
constexpr int kStages = 3;
constexpr size_t kSymvSmemBytes =
    sizeof(double) * (kStages * 16 * kSP + kStages * NR * kCP + SY * kXP + 8 * 16 * NR);

__device__ __forceinline__ void cp_async16(void* dst, const void* src, int src_bytes) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(tc::smem_u32(dst)), "l"(src), "r"(src_bytes)
               : "memory");
}
__device__ __forceinline__ void cp_async8(void* dst, const void* src, int src_bytes) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;" ::"r"(tc::smem_u32(dst)), "l"(src), "r"(src_bytes)
               : "memory");
}

__global__ void __launch_bounds__(kThreads, 1)
    symv_tiles_kernel(const double* __restrict__ a, long long lda, int upper, int n,
                      const double* __restrict__ X, long long ldx, int nrhs, int absval, int vec16,
                      double* __restrict__ U, double* __restrict__ V) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  double* Sr = reinterpret_cast<double*>(smem_raw);   // stage s: Sr[s][jj * kSP + ii] = T(ii, chunk col jj)
  double* Xcr = Sr + kStages * 16 * kSP;               // stage s: Xcr[s][c * kCP + jj] = X(col block + jj, c)
  double* Xi = Xcr + kStages * NR * kCP;               // Xi[ii * kXP + c] = X(row block + ii, c)
  double* Vr = Xi + SY * kXP;                          // Vr[w][jj][c]: per-warp partial T^T X
  int I, J;
  task_tile(blockIdx.x, I, J);
  const int rb = upper ? J : I, cb = upper ? I : J;   // row / column block of T
  const int i0 = rb * SY, j0 = cb * SY, t = threadIdx.x;
  const int lane = t & 31, w = t >> 5, g = lane >> 2, tq = lane & 3;
  const bool diag = (I == J);
  for (int e = t; e < SY * NR; e += kThreads) {
    const int ii = e % SY, c = e / SY, i = i0 + ii;
    Xi[ii * kXP + c] = (i < n && c < nrhs) ? X[i + (long long)c * ldx] : 0.0;
  }
  // chunk jc -> stage st: 16 columns x 256 rows of T, and the 16 x 16 block of X
  auto issue = [&](int jc, int st) {
    double* S = Sr + st * 16 * kSP;
    const int jb0 = j0 + jc * 16;
    if (vec16) {
#pragma unroll
      for (int q = 0; q < 8; ++q) {
        const int e = t + kThreads * q;            // 16-byte piece: column e / 128, rows 2 (e % 128) ..
        const int jj = e >> 7, ii = 2 * (e & 127), i = i0 + ii, j = jb0 + jj;
        const int bytes = (j < n && i < n) ? (i + 1 < n ? 16 : 8) : 0;
        cp_async16(S + jj * kSP + ii, a + (bytes ? (long long)i + (long long)j * lda : 0), bytes);
      }
    } else {
#pragma unroll 4
      for (int q = 0; q < 16; ++q) {
        const int e = t + kThreads * q;
        const int jj = e >> 8, ii = e & 255, i = i0 + ii, j = jb0 + jj;
        const int bytes = (j < n && i < n) ? 8 : 0;
        cp_async8(S + jj * kSP + ii, a + (bytes ? (long long)i + (long long)j * lda : 0), bytes);
      }
    }
    if (t < NR * 8) {   // X block: 16 columns c of 16 rows each, 16-byte pieces (2 rows)
      double* Xc = Xcr + st * NR * kCP;
      const int c = t >> 3, jj = 2 * (t & 7), j = jb0 + jj;
      if (((ldx & 1) == 0) && (((uintptr_t)X & 15) == 0)) {
        const int bytes = (c < nrhs && j < n) ? (j + 1 < n ? 16 : 8) : 0;
        cp_async16(Xc + c * kCP + jj, X + (bytes ? (long long)j + (long long)c * ldx : 0), bytes);
      } else {
        const int b0 = (c < nrhs && j < n) ? 8 : 0, b1 = (c < nrhs && j + 1 < n) ? 8 : 0;
        cp_async8(Xc + c * kCP + jj, X + (b0 ? (long long)j + (long long)c * ldx : 0), b0);
        cp_async8(Xc + c * kCP + jj + 1, X + (b1 ? (long long)j + 1 + (long long)c * ldx : 0), b1);
      }
    }
  };
  double u[2][2][4];
#pragma unroll
  for (int m = 0; m < 2; ++m)
#pragma unroll
    for (int q = 0; q < 2; ++q)
#pragma unroll
      for (int e = 0; e < 4; ++e) u[m][q][e] = 0.0;
  double* Uo = (upper ? V : U) + (size_t)blockIdx.x * SY * NR;   // T X
  double* Vo = (upper ? U : V) + (size_t)blockIdx.x * SY * NR;   // T^T X
  const int r0 = 32 * w;   // this warp's rows of the tile
  constexpr int NCH = SY / 16;
  issue(0, 0);
  cp_async_commit();
  issue(1, 1);
  cp_async_commit();
  for (int jc = 0; jc < NCH; ++jc) {
    const int st = jc % kStages;
    cp_async_wait<kStages - 2>();   // chunk jc has landed (this thread's copies)
    __syncthreads();                // ... everyone's; and stage (jc + 2) % 3 is free
    double* S = Sr + st * 16 * kSP;
    const double* Xc = Xcr + st * NR * kCP;
    if (diag || absval) {   // keep the stored triangle only (the other one may hold anything)
      for (int e = t; e < 16 * SY; e += kThreads) {
        const int jj = e >> 8, ii = e & 255, col = jc * 16 + jj;
        double v = S[jj * kSP + ii];
        if (diag && (upper ? ii > col : ii < col)) v = 0.0;
        if (absval) v = fabs(v);
        S[jj * kSP + ii] = v;
      }
      __syncthreads();
    }
    if (jc + 2 < NCH) issue(jc + 2, (jc + 2) % kStages);
    cp_async_commit();
    // T X: 2 m16 tiles x 2 n8 tiles x 4 k4 steps
#pragma unroll
    for (int ks = 0; ks < 4; ++ks) {
      const double* Sk = S + (4 * ks + tq) * kSP + r0 + g;
      const double b0 = Xc[g * kCP + 4 * ks + tq], b1 = Xc[(8 + g) * kCP + 4 * ks + tq];
#pragma unroll
      for (int m = 0; m < 2; ++m) {
        const double a0 = Sk[16 * m], a1 = Sk[16 * m + 8];
        cuchol::dmma::dmma_16x8x4(u[m][0], a0, a1, b0);
        cuchol::dmma::dmma_16x8x4(u[m][1], a0, a1, b1);
      }
    }
    // partial T^T X over rows r0..r0+31 (on a diagonal tile without the diagonal)
    double v[2][4] = {{0.0, 0.0, 0.0, 0.0}, {0.0, 0.0, 0.0, 0.0}};
#pragma unroll
    for (int ks = 0; ks < 8; ++ks) {
      const int ii = r0 + 4 * ks + tq;
      double a0 = S[g * kSP + ii], a1 = S[(g + 8) * kSP + ii];
      if (diag) {
        if (ii == jc * 16 + g) a0 = 0.0;
        if (ii == jc * 16 + g + 8) a1 = 0.0;
      }
      const double b0 = Xi[ii * kXP + g], b1 = Xi[ii * kXP + 8 + g];
      cuchol::dmma::dmma_16x8x4(v[0], a0, a1, b0);
      cuchol::dmma::dmma_16x8x4(v[1], a0, a1, b1);
    }
    // C fragment: (row g, cols 2tq, 2tq+1) and (row g + 8, same cols) of each n8 tile
    double* Vw = Vr + w * 16 * NR;
#pragma unroll
    for (int q = 0; q < 2; ++q) {
      Vw[g * NR + 8 * q + 2 * tq] = v[q][0];
      Vw[g * NR + 8 * q + 2 * tq + 1] = v[q][1];
      Vw[(g + 8) * NR + 8 * q + 2 * tq] = v[q][2];
      Vw[(g + 8) * NR + 8 * q + 2 * tq + 1] = v[q][3];
    }
    __syncthreads();
    {
      double sum = 0.0;   // thread t: output (jj = t / 16, c = t % 16), warps in order
#pragma unroll
      for (int k = 0; k < 8; ++k) sum += Vr[k * 16 * NR + t];
      Vo[(jc * 16) * NR + t] = sum;
    }
  }
  cp_async_wait<0>();
#pragma unroll
  for (int m = 0; m < 2; ++m)
#pragma unroll
    for (int q = 0; q < 2; ++q) {
      const int row = r0 + 16 * m + g, col = 8 * q + 2 * tq;
      Uo[row * NR + col] = u[m][q][0];
      Uo[row * NR + col + 1] = u[m][q][1];
      Uo[(row + 8) * NR + col] = u[m][q][2];
      Uo[(row + 8) * NR + col + 1] = u[m][q][3];
    }
}

// Y_K = alpha * (sum_{J <= K} U(K,J) + sum_{I >= K} V(I,K)) + beta * B_K, summed in
// a fixed order (deterministic).  One CTA per 16 rows, thread = (row, rhs), so a warp reads
// whole 128-byte rows of the partials and enough CTAs are in flight to cover their latency
// (a thread per row on one CTA per tile: n = 8192 75 us).
// B may alias Y; ldy/ldb columns, only the first nrhs columns are written.
__global__ void __launch_bounds__(kThreads)
    symv_reduce_kernel(const double* __restrict__ U, const double* __restrict__ V, int n, int ntile, double alpha,
                       double beta, const double* B, long long ldb, double* Y, long long ldy, int nrhs) {
  const int i = blockIdx.x * (kThreads / NR) + threadIdx.x / NR, c = threadIdx.x % NR;
  const int K = i / SY, o = (i % SY) * NR + c;
  double sum = 0.0;
  const double* u = U + (size_t)(K * (K + 1) / 2) * SY * NR + o;
#pragma unroll 8
  for (int J = 0; J <= K; ++J) sum += u[(size_t)J * SY * NR];
#pragma unroll 8
  for (int I = K; I < ntile; ++I) sum += V[(size_t)(I * (I + 1) / 2 + K) * SY * NR + o];
  if (i >= n || c >= nrhs) return;
  double y = alpha * sum;
  if (beta != 0.0) y += beta * B[i + (long long)c * ldb];
  Y[i + (long long)c * ldy] = y;
}

// ---- PCG vector kernels (n x NR, column-major, leading dimension ld) ------------------
// Deterministic reductions: each CTA writes per-RHS partials part[blockIdx.x][NR];
// the kernel that consumes them sums all partials in the same order.
constexpr int kVecBlocks = 256;

__device__ __forceinline__ void block_sum16(double (&v)[NR], double* sh /* [kThreads][NR+1] */) {
  const int t = threadIdx.x;
#pragma unroll
  for (int c = 0; c < NR; ++c) sh[t * (NR + 1) + c] = v[c];
  __syncthreads();
  for (int s = kThreads / 2; s > 0; s >>= 1) {
    if (t < s) {
#pragma unroll
      for (int c = 0; c < NR; ++c) sh[t * (NR + 1) + c] += sh[(t + s) * (NR + 1) + c];
    }
    __syncthreads();
  }
}
__device__ __forceinline__ void block_max16(double (&v)[NR], double* sh) {
  const int t = threadIdx.x;
#pragma unroll
  for (int c = 0; c < NR; ++c) sh[t * (NR + 1) + c] = v[c];
  __syncthreads();
  for (int s = kThreads / 2; s > 0; s >>= 1) {
    if (t < s) {
#pragma unroll
      for (int c = 0; c < NR; ++c) sh[t * (NR + 1) + c] = fmax(sh[t * (NR + 1) + c], sh[(t + s) * (NR + 1) + c]);
    }
    __syncthreads();
  }
}

// part[b][c] = sum over this CTA's rows of a(i, c) * b(i, c)
__global__ void __launch_bounds__(kThreads) dot_kernel(const double* __restrict__ a, const double* __restrict__ b,
                                                       int n, long long ld, double* __restrict__ part) {
  __shared__ double sh[kThreads * (NR + 1)];
  double v[NR];
#pragma unroll
  for (int c = 0; c < NR; ++c) v[c] = 0.0;
  for (int i = blockIdx.x * kThreads + threadIdx.x; i < n; i += gridDim.x * kThreads) {
#pragma unroll
    for (int c = 0; c < NR; ++c) v[c] = fma(a[i + c * ld], b[i + c * ld], v[c]);
  }
  block_sum16(v, sh);
  if (threadIdx.x < NR) part[blockIdx.x * NR + threadIdx.x] = sh[threadIdx.x];
}

// total[c] = sum of the kVecBlocks partials of right-hand side c, by the whole CTA in a
// fixed order: thread (g, c) sums 16 consecutive partials, then thread c sums the 16
// groups (one thread per c over all 256: a chain of 256 loads, 29 us).  Ends with a barrier.
__device__ __forceinline__ void sum_parts(const double* part, double* grp /* [16][NR] */, double* total) {
  static_assert(kVecBlocks == 256 && kThreads == 16 * NR, "16 groups of 16 partials");
  const int g = threadIdx.x / NR, c = threadIdx.x % NR;
  double s = 0.0;
#pragma unroll
  for (int b = 0; b < 16; ++b) s += part[(16 * g + b) * NR + c];
  grp[g * NR + c] = s;
  __syncthreads();
  if (g == 0) {
    double t = 0.0;
#pragma unroll
    for (int b = 0; b < 16; ++b) t += grp[b * NR + c];
    total[c] = t;
  }
  __syncthreads();
}

// alpha_c = rz_c / (p_c . q_c); x += alpha p; r -= alpha q; partial max |r|, max |x|
// into part_norm[b][0..NR) and [NR..2NR).
__global__ void __launch_bounds__(kThreads)
    update_xr_kernel(double* __restrict__ x, double* __restrict__ r, const double* __restrict__ p,
                     const double* __restrict__ q, int n, long long ld, const double* __restrict__ part_pq,
                     const double* __restrict__ rz, double* __restrict__ part_norm) {
  __shared__ double alpha[NR];
  __shared__ double sh[kThreads * (NR + 1)];
  __shared__ double total[NR];
  sum_parts(part_pq, sh, total);
  if (threadIdx.x < NR) {
    const int c = threadIdx.x;
    const double pq = total[c];
    alpha[c] = (pq > 0.0 && rz[c] > 0.0) ? rz[c] / pq : 0.0;
  }
  __syncthreads();
  double rm[NR], xm[NR];
#pragma unroll
  for (int c = 0; c < NR; ++c) rm[c] = xm[c] = 0.0;
  for (int i = blockIdx.x * kThreads + threadIdx.x; i < n; i += gridDim.x * kThreads) {
#pragma unroll
    for (int c = 0; c < NR; ++c) {
      const double xv = fma(alpha[c], p[i + c * ld], x[i + c * ld]);
      const double rv = fma(-alpha[c], q[i + c * ld], r[i + c * ld]);
      x[i + c * ld] = xv;
      r[i + c * ld] = rv;
      rm[c] = fmax(rm[c], fabs(rv));
      xm[c] = fmax(xm[c], fabs(xv));
    }
  }
  block_max16(rm, sh);
  if (threadIdx.x < NR) part_norm[blockIdx.x * 2 * NR + threadIdx.x] = sh[threadIdx.x];
  __syncthreads();
  block_max16(xm, sh);
  if (threadIdx.x < NR) part_norm[blockIdx.x * 2 * NR + NR + threadIdx.x] = sh[threadIdx.x];
}

// partial max |a(:, c)| and max |b(:, c)| (b may be null)
__global__ void __launch_bounds__(kThreads) norms_kernel(const double* __restrict__ a, const double* __restrict__ b,
                                                         int n, long long ld, double* __restrict__ part_norm) {
  __shared__ double sh[kThreads * (NR + 1)];
  double am[NR], bm[NR];
#pragma unroll
  for (int c = 0; c < NR; ++c) am[c] = bm[c] = 0.0;
  for (int i = blockIdx.x * kThreads + threadIdx.x; i < n; i += gridDim.x * kThreads) {
#pragma unroll
    for (int c = 0; c < NR; ++c) {
      am[c] = fmax(am[c], fabs(a[i + c * ld]));
      if (b != nullptr) bm[c] = fmax(bm[c], fabs(b[i + c * ld]));
    }
  }
  block_max16(am, sh);
  if (threadIdx.x < NR) part_norm[blockIdx.x * 2 * NR + threadIdx.x] = sh[threadIdx.x];
  __syncthreads();
  block_max16(bm, sh);
  if (threadIdx.x < NR) part_norm[blockIdx.x * 2 * NR + NR + threadIdx.x] = sh[threadIdx.x];
}

// out[0..2NR) = max over the partials (one CTA of 2 NR warps, a warp per value)
__global__ void __launch_bounds__(64 * NR) norms_final_kernel(const double* __restrict__ part_norm, int nparts,
                                                              double* __restrict__ out) {
  const int c = threadIdx.x >> 5;
  double m = 0.0;
  for (int b = threadIdx.x & 31; b < nparts; b += 32) m = fmax(m, part_norm[b * 2 * NR + c]);
  for (int o = 16; o > 0; o >>= 1) m = fmax(m, __shfl_down_sync(0xffffffffu, m, o));
  if ((threadIdx.x & 31) == 0) out[c] = m;
}

// rz_new = sum of part_rz; beta = rz_new / rz_old (0 when restart or rz_old == 0);
// p = z + beta p.  Block 0 stores rz_new.
__global__ void __launch_bounds__(kThreads)
    update_p_kernel(double* __restrict__ p, const double* __restrict__ z, int n, long long ld,
                    const double* __restrict__ part_rz, const double* __restrict__ rz_old,
                    double* __restrict__ rz_new, int restart) {
  __shared__ double beta[NR], total[NR], grp[kThreads];
  sum_parts(part_rz, grp, total);
  if (threadIdx.x < NR) {
    const int c = threadIdx.x;
    const double rn = total[c];
    beta[c] = (!restart && rz_old[c] > 0.0) ? rn / rz_old[c] : 0.0;
    if (blockIdx.x == 0) rz_new[c] = rn;
  }
  __syncthreads();
  for (int i = blockIdx.x * kThreads + threadIdx.x; i < n; i += gridDim.x * kThreads) {
#pragma unroll
    for (int c = 0; c < NR; ++c) p[i + c * ld] = fma(beta[c], p[i + c * ld], z[i + c * ld]);
  }
}

__global__ void ones_kernel(double* __restrict__ x, int n) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) x[i] = 1.0;
}

// dst (ld) = src (lds) for columns < ncols, zero for the rest of the NR columns
__global__ void load_cols_kernel(const double* __restrict__ src, long long lds, int ncols, int n,
                                 double* __restrict__ dst, long long ld) {
  for (long long e = blockIdx.x * (long long)blockDim.x + threadIdx.x; e < (long long)n * NR;
       e += (long long)gridDim.x * blockDim.x) {
    const int i = (int)(e % n), c = (int)(e / n);
    dst[i + c * ld] = (c < ncols) ? src[i + c * lds] : 0.0;
  }
}
__global__ void store_cols_kernel(const double* __restrict__ src, long long ld, int ncols, int n,
                                  double* __restrict__ dst, long long ldd) {
  for (long long e = blockIdx.x * (long long)blockDim.x + threadIdx.x; e < (long long)n * ncols;
       e += (long long)gridDim.x * blockDim.x) {
    const int i = (int)(e % n), c = (int)(e / n);
    dst[i + c * ldd] = src[i + c * ld];
  }
}

}  // namespace mx
}  // namespace

// ---- host side ------------------------------------------------------------------

struct __cucholmixed_st {
  CULAPACKhandle h;
  int precision;              // CUCHOL_MIXED_BF16 or CUCHOL_MIXED_TF32
  int n;
  const double* A;            // the caller's matrix (read by every residual)
  long long rs, cs;           // its logical lower view
  float* W;                   // FP32 factor of S A S + shift I (lower, ldw)
  long long ldw;
  double* s;                  // the scaling S
  float* Dinv;                // inverses of W's NBT x NBT diagonal blocks (ld NBT, NBT (NBT + 1) apart)
  float* gpart;               // split-k partial sums of the preconditioner GEMVs
  double anorm;               // |A|_inf
  double shift;               // shift of the factor that succeeded
  double shift_request;       // caller's shift (< 0: automatic)
  long long ld;               // rows of the work vectors
  double *x, *r, *z, *p, *q, *b;
  float *t, *y, *zf;          // preconditioner vectors (FP32)
  double *U, *V;              // symmetric-product partials
  double *part, *part_norm, *rz, *norms;
  double* h_norms;            // pinned mirror of norms (the handle's)
  char* arena;                // the one allocation behind all of the above
  unsigned* ctr;              // triangular-solve counters
  unsigned* gcount;           // arrivals per output block of a split GEMV (zero between launches)
  int* err;                   // a bounded wait gave up
};

namespace {
namespace mx {

inline int ntile_of(int n) { return (n + SY - 1) / SY; }
constexpr size_t kSymvSmem = kSymvSmemBytes;

template <typename T>
CUresult block_inverse(int device, const T* L, long long rs, long long cs, int n, T* DI, cudaStream_t s) {
  const size_t smem = BlockSmem<T, BS>::bytes;
  static DeviceOnce attr;
  if (attr.needed(device)) {
    CUCHOL_CHECK(cudaFuncSetAttribute(block_inverse_kernel<T>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                      (int)smem));
    attr.done(device);
  }
  block_inverse_kernel<T><<<(n + BS - 1) / BS, kThreads, smem, s>>>(L, rs, cs, n, DI);
  CUCHOL_CHECK(cudaGetLastError());
  return CUDA_SUCCESS;
}

// Y = alpha A X + beta B for the symmetric A (one triangle, lower view rs, cs).
CUresult symv(int device, const double* A, long long rs, long long cs, int n, const double* X, long long ldx, int nrhs,
              int absval, double alpha, double beta, const double* B, long long ldb, double* Y, long long ldy,
              double* U, double* V, cudaStream_t s) {
  static DeviceOnce attr;
  if (attr.needed(device)) {
    CUCHOL_CHECK(cudaFuncSetAttribute(symv_tiles_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                      (int)kSymvSmem));
    attr.done(device);
  }
  const int T = ntile_of(n);
  const int upper = (rs != 1);
  const long long lda = upper ? rs : cs;
  const int vec16 = ((lda & 1) == 0) && ((reinterpret_cast<uintptr_t>(A) & 15) == 0);
  symv_tiles_kernel<<<T * (T + 1) / 2, kThreads, kSymvSmem, s>>>(A, lda, upper, n, X, ldx, nrhs, absval, vec16, U,
                                                                  V);
  CUCHOL_CHECK(cudaGetLastError());
  symv_reduce_kernel<<<T * SY * NR / kThreads, kThreads, 0, s>>>(U, V, n, T, alpha, beta, B, ldb, Y, ldy, nrhs);
  CUCHOL_CHECK(cudaGetLastError());
  return CUDA_SUCCESS;
}

template <typename T>
constexpr size_t trsv_smem() { return sizeof(T) * (2 * BS * (BS + 1) + BS * NR + 16 * BS); }

// Opt in to the triangular solves' shared memory (above 48 KB for FP64).
template <typename T, typename V>
CUresult trsv_attr(int device) {
  static DeviceOnce attr;
  if (attr.needed(device)) {
    CUCHOL_CHECK(cudaFuncSetAttribute(trsv_fwd_kernel<T, V>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                      (int)trsv_smem<T>()));
    CUCHOL_CHECK(cudaFuncSetAttribute(trsv_bwd_kernel<T, V>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                      (int)trsv_smem<T>()));
    attr.done(device);
  }
  return CUDA_SUCCESS;
}

// Z = S F^T F S R (the preconditioner; F = forward solve by the FP32 factor in
// NBT-wide steps with the inverted diagonal blocks), 16 columns.
CUresult precond(CUcholMixed p, const double* R, double* Z, cudaStream_t s) {
  static DeviceOnce attr;
  if (attr.needed(p->h->device)) {
    CUCHOL_CHECK(cudaFuncSetAttribute(gemv_n_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kGemvSmem));
    CUCHOL_CHECK(cudaFuncSetAttribute(gemv_t_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kGemvSmem));
    attr.done(p->h->device);
  }
  const int n = p->n;
  const long long ld = p->ld, ldw = p->ldw;
  const int nT = (n + NBT - 1) / NBT, vb = 4 * p->h->num_sms;
  // one GEMV; with fewer than two CTAs per SM the k range is split (chunks of 256 or
  // more) and the partial sums are added in order by the last CTA of each block
  auto gemv = [&](bool trans, bool tri, const float* M, long long ldm, int m, int kk, const float* v, float alpha,
                  float beta, const float* in, float* out) -> CUresult {
    const int blocks = (m + GR - 1) / GR, want = 2 * p->h->num_sms;
    int split = 1;
    if (blocks < want) split = std::max(1, std::min((want + blocks - 1) / blocks, kk / 256));
    const int kc = (int)round_up((size_t)((kk + split - 1) / split), GR);
    split = (kk + kc - 1) / kc;
    const dim3 grid(blocks, split);
    if (trans)
      gemv_t_kernel<<<grid, kThreads, kGemvSmem, s>>>(M, ldm, m, kk, v, alpha, beta, in, out, ld, kc, p->gpart,
                                                      p->gcount, tri);
    else
      gemv_n_kernel<<<grid, kThreads, kGemvSmem, s>>>(M, ldm, m, kk, v, alpha, beta, in, out, ld, kc, p->gpart,
                                                      p->gcount, tri);
    CUCHOL_CHECK(cudaGetLastError());
    ++p->h->launches;
    return CUDA_SUCCESS;
  };
  scale_in_kernel<<<vb, 256, 0, s>>>(R, p->s, n, ld, p->t);
  CUCHOL_CHECK(cudaGetLastError());
  for (int I = 0; I < nT; ++I) {
    const int b0 = I * NBT, bI = std::min(NBT, n - b0), rest = n - b0 - bI;
    const float* D = p->Dinv + (size_t)I * NBT * (NBT + 1);
    CUCHOL_CHECK_CU(gemv(false, true, D, NBT, bI, bI, p->t + b0, 1.f, 0.f, nullptr, p->y + b0));
    if (rest > 0)
      CUCHOL_CHECK_CU(gemv(false, false, p->W + (b0 + bI) + (long long)b0 * ldw, ldw, rest, bI, p->y + b0, -1.f, 1.f,
                           p->t + b0 + bI, p->t + b0 + bI));
  }
  for (int I = nT - 1; I >= 0; --I) {
    const int b0 = I * NBT, bI = std::min(NBT, n - b0);
    const float* D = p->Dinv + (size_t)I * NBT * (NBT + 1);
    CUCHOL_CHECK_CU(gemv(true, true, D, NBT, bI, bI, p->y + b0, 1.f, 0.f, nullptr, p->zf + b0));
    if (b0 > 0) CUCHOL_CHECK_CU(gemv(true, false, p->W + b0, ldw, b0, bI, p->zf + b0, -1.f, 1.f, p->y, p->y));
  }
  scale_out_kernel<<<vb, 256, 0, s>>>(p->zf, p->s, n, ld, Z);
  CUCHOL_CHECK(cudaGetLastError());
  p->h->launches += 2;
  return CUDA_SUCCESS;
}

// C := C + alpha Q(a0 + i) Q(b0 + j)^T (alpha = -1 in the factor) on the lower tiles of an
// m x ncols FP32 region whose
// top-left element is on the diagonal; Q k-major (q_rows x k used, row pitch ldq).
template <typename Op>
CUresult tc_update(CULAPACKhandle h, const Op* q, long long ldq, int q_rows, int k, int a0, int b0, float* c,
                   long long ldc, int m, int ncols, cudaStream_t s, const int* stop, float alpha = -1.f) {
  if (m <= 0 || ncols <= 0 || k <= 0) return CUDA_SUCCESS;
  EncodeTiledFn fn = encode_tiled();
  if (fn == nullptr) return CUDA_ERROR_NOT_SUPPORTED;
  CUtensorMap mq, mc;
  const cuuint32_t es[2] = {1, 1};
  {
    const cuuint64_t dims[2] = {(cuuint64_t)k, (cuuint64_t)q_rows};
    const cuuint64_t strides[1] = {(cuuint64_t)ldq * sizeof(Op)};
    const cuuint32_t box[2] = {(cuuint32_t)tc::OpKind<Op>::BK, (cuuint32_t)tc::BM};
    const CUtensorMapDataType dt = sizeof(Op) == 2 ? CU_TENSOR_MAP_DATA_TYPE_BFLOAT16 : CU_TENSOR_MAP_DATA_TYPE_FLOAT32;
    if (fn(&mq, dt, 2, const_cast<Op*>(q), dims, strides, box, es, CU_TENSOR_MAP_INTERLEAVE_NONE,
           CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) !=
        CUDA_SUCCESS)
      return CUDA_ERROR_INVALID_VALUE;
  }
  {
    const cuuint64_t dims[2] = {(cuuint64_t)m, (cuuint64_t)ncols};
    const cuuint64_t strides[1] = {(cuuint64_t)ldc * sizeof(float)};
    const cuuint32_t box[2] = {32, 32};
    if (fn(&mc, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 2, c, dims, strides, box, es, CU_TENSOR_MAP_INTERLEAVE_NONE,
           CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_NONE, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) !=
        CUDA_SUCCESS)
      return CUDA_ERROR_INVALID_VALUE;
  }
  tc::Params prm{};
  prm.m = m;
  prm.n = ncols;
  prm.k = k;
  prm.a_row0 = a0;
  prm.b_row0 = b0;
  prm.alpha = alpha;
  prm.lower_only = 1;
  prm.tiles_m = (m + tc::BM - 1) / tc::BM;
  prm.tiles_n = (ncols + tc::BN - 1) / tc::BN;
  prm.err = h->d_words + 3;
  const int tiles = prm.tiles_n * (prm.tiles_n + 1) / 2 + (prm.tiles_m - prm.tiles_n) * prm.tiles_n;
  static DeviceOnce attr;
  if (attr.needed(h->device)) {
    CUCHOL_CHECK(cudaFuncSetAttribute(tc::update_kernel<Op>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                      tc::SMEM_BYTES));
    attr.done(h->device);
  }
  tc::update_kernel<Op><<<tiles, tc::THREADS, tc::SMEM_BYTES, s>>>(mq, mq, mc, prm, stop);
  ++h->launches;
  CUCHOL_CHECK(cudaGetLastError());
  return CUDA_SUCCESS;
}

// Blocked Cholesky of the FP32 matrix W (lower, ldw) with FP64 diagonal blocks, FP32
// panel solves and tensor-core trailing updates in Op; schedule as ?potrf.
// *info = first failing column (1-based) or 0.
// The FP32 inverse of every 128-wide diagonal block is left in dinv (the NBT-block
// store of the plan, ld NBT) at its place in its NBT-wide block.
template <typename Op>
CUresult mixed_factor(CULAPACKhandle h, int n, float* W, long long ldw, long* info) {
  cudaStream_t sp = h->s_panel, su = h->s_update;
  int* d_info = h->d_words;
  const long long ldq = OB;
  const size_t rows = round_up((size_t)n, 128) + 128;
  const size_t qbytes = round_up(sizeof(Op) * rows * ldq, 256);
  // Block and panel in one launch while its CTAs fit the GPU, as in ?potrf: there 33 us in
  // place of 34 + 14 and a gap.  Those factors wait in D, from block dfirst on.
  const int fused_rows = kFusedRows * h->num_sms;
  int dfirst = -1, dcount = 0;
  const size_t dbytes = sizeof(float) * SB * SB * (size_t)(std::min(n, fused_rows + SB) / SB + 1);
  CUCHOL_CHECK_CU(ensure_workspace(h, 2 * qbytes + dbytes));
  char* ws = static_cast<char*>(h->ws);
  Op* Q[2] = {reinterpret_cast<Op*>(ws), reinterpret_cast<Op*>(ws + qbytes)};
  float* D = reinterpret_cast<float*>(ws + 2 * qbytes);
  CUCHOL_CHECK(cudaEventRecord(h->ev_update, sp));   // (the update stream starts behind a panel event)
  auto at = [&](long long i, long long j) { return W + i + j * ldw; };

  for (int j = 0, step = 0; j < n; j += OB, ++step) {
    const int jB = std::min(OB, n - j);
    const int m = n - j - jB;
    Op* Qj = Q[step & 1];
    const int q_rows = n - j - SB;   // P / Q row r = global row j + SB + r
    for (int s0 = 0; s0 < jB; s0 += SB) {
      const int c = j + s0, jb = std::min(SB, j + jB - c), mr = n - c - jb;
      // panel rows c + jb .. n-1 solved in place; they are Q rows s0 .., columns s0 ..
      Op* Qs = Qj + (long long)s0 * ldq + s0;
      if (mr > 0 && mr <= fused_rows) {              // (rows below it: the block is a whole one)
        if (dfirst < 0) dfirst = c / SB;
        CUCHOL_CHECK_CU((panel_fused<double, float, Op, OUT_ROUND, SB>(
            h, at(c, c), mr, 1, ldw, Qs, ldq, 1, nullptr, D + (size_t)dcount++ * SB * SB, c, c == 0, h->d_logdet, sp)));
      } else {
        CUCHOL_CHECK_CU((diag_factor<double, float, SB>(h, at(c, c), 1, ldw, jb, c, c == 0, h->d_logdet, sp)));
        if (mr == 0) break;
        CUCHOL_CHECK_CU((panel_solve<float, Op, OUT_ROUND, SB>(h, at(c + jb, c), mr, jb, at(c, c), 1, ldw, Qs, ldq, 1,
                                                               nullptr, sp)));
      }
      if (s0 + SB < jB)   // the outer block's remaining columns by this sub-panel
        CUCHOL_CHECK_CU(tc_update<Op>(h, Qs, ldq, q_rows - s0, jb, 0, 0, at(c + jb, c + jb), ldw, mr,
                                      jB - s0 - SB, sp, d_info));
    }
    CUCHOL_CHECK(cudaEventRecord(h->ev_panel, sp));
    if (m == 0) break;
    // P / Q rows from global row j + OB: all sub-panels' columns (k = jB)
    const int jB2 = std::min(OB, m);
    const Op* Qt = Qj + (long long)(OB - SB) * ldq;
    const int t_rows = q_rows - (OB - SB);
    CUCHOL_CHECK(cudaStreamWaitEvent(sp, h->ev_update, 0));
    CUCHOL_CHECK_CU(tc_update<Op>(h, Qt, ldq, t_rows, jB, 0, 0, at(j + OB, j + OB), ldw, m, jB2, sp, d_info));
    CUCHOL_CHECK(cudaStreamWaitEvent(su, h->ev_panel, 0));
    if (m > jB2)
      CUCHOL_CHECK_CU(tc_update<Op>(h, Qt, ldq, t_rows, jB, jB2, jB2, at(j + OB + jB2, j + OB + jB2), ldw, m - jB2,
                                    m - jB2, su, d_info));
    CUCHOL_CHECK(cudaEventRecord(h->ev_update, su));
  }
  CUCHOL_CHECK(cudaEventRecord(h->ev_update, su));
  CUCHOL_CHECK(cudaStreamWaitEvent(sp, h->ev_update, 0));
  if (dcount > 0) CUCHOL_CHECK_CU((copy_diag<float, SB>(h, D, W, 1, ldw, dfirst, dfirst, dcount, sp)));
  CUCHOL_CHECK_CU(fetch_words(h, sp));
  *info = h->h_words[0];
  return CUDA_SUCCESS;
}

void free_mixed(CUcholMixed p) {
  if (p == nullptr) return;
  cudaFree(p->arena);
  delete p;
}

// Largest column max |v(:, c)| for c < 2 NR of the partials -> host (synchronises s).
CUresult fetch_norms(CUcholMixed p, cudaStream_t s) {
  norms_final_kernel<<<1, 64 * NR, 0, s>>>(p->part_norm, kVecBlocks, p->norms);
  CUCHOL_CHECK(cudaGetLastError());
  CUCHOL_CHECK(cudaMemcpyAsync(p->h_norms, p->norms, 2 * NR * sizeof(double), cudaMemcpyDeviceToHost, s));
  CUCHOL_CHECK(cudaStreamSynchronize(s));
  return CUDA_SUCCESS;
}

// Scale, |A|_inf and the low-precision factor of the plan's A (its current values).
template <typename Op>
CUresult mixed_refactor(CUcholMixed p, long* info) {
  CULAPACKhandle h = p->h;
  const int n = p->n;
  cudaStream_t sp = h->s_panel;
  // scaling; a non-positive diagonal entry ends the attempt (info = its row)
  int* bad = h->d_words + 4;
  CUCHOL_CHECK(cudaMemsetAsync(bad, 0, sizeof(int), sp));
  scale_kernel<<<(n + 255) / 256, 256, 0, sp>>>(p->A, p->rs + p->cs, n, p->s, bad);
  CUCHOL_CHECK(cudaGetLastError());
  CUCHOL_CHECK(cudaMemcpyAsync(h->h_words + 4, bad, sizeof(int), cudaMemcpyDeviceToHost, sp));
  CUCHOL_CHECK(cudaStreamSynchronize(sp));
  if (h->h_words[4] != 0) {
    std::vector<double> d(n);
    CUCHOL_CHECK(cudaMemcpy2D(d.data(), sizeof(double), p->A, (p->rs + p->cs) * sizeof(double), sizeof(double), n,
                              cudaMemcpyDeviceToHost));
    long k = 0;
    while (k < n && d[k] > 0.0) ++k;
    *info = k + 1;
    return CUDA_SUCCESS;
  }
  // |A|_inf = max row sum of |A| (x is zero: column 0 set to ones)
  CUCHOL_CHECK(cudaMemsetAsync(p->x, 0, sizeof(double) * p->ld * NR, sp));
  {
    ones_kernel<<<(n + 255) / 256, 256, 0, sp>>>(p->x, n);
    CUCHOL_CHECK(cudaGetLastError());
    CUCHOL_CHECK_CU(symv(p->h->device, p->A, p->rs, p->cs, n, p->x, p->ld, 1, 1, 1.0, 0.0, nullptr, 0, p->r, p->ld, p->U, p->V,
                         sp));
    CUCHOL_CHECK(cudaMemsetAsync(p->r + p->ld, 0, sizeof(double) * p->ld * (NR - 1), sp));
    norms_kernel<<<kVecBlocks, kThreads, 0, sp>>>(p->r, nullptr, n, p->ld, p->part_norm);
    CUCHOL_CHECK(cudaGetLastError());
    CUCHOL_CHECK_CU(fetch_norms(p, sp));
    p->anorm = p->h_norms[0];
  }
  // factor S A S + shift I; on a breakdown retry with 8x the shift (automatic mode)
  const double u = (sizeof(Op) == 2) ? 0x1p-8 : 0x1p-11;
  const double shift_in = p->shift_request;
  double shift = shift_in >= 0.0 ? shift_in : u / 16;
  long finfo = 0;
  const int nT = (n + NBT - 1) / NBT;
  for (int attempt = 0; attempt < (shift_in >= 0.0 ? 1 : 4); ++attempt, shift *= 8.0) {
    dim3 g((n + 31) / 32, (n + 31) / 32);
    build_kernel<<<g, 256, 0, sp>>>(p->A, p->rs, p->cs, n, p->s, (float)shift, p->W, p->ldw);
    CUCHOL_CHECK(cudaGetLastError());
    CUCHOL_CHECK_CU(mixed_factor<Op>(h, n, p->W, p->ldw, &finfo));
    p->shift = shift;
    if (finfo == 0) break;
  }
  if (finfo != 0) {
    *info = finfo;
    return CUDA_SUCCESS;
  }
  // Inverses of the NBT-wide diagonal blocks of the factor.  Block I starts at
  // I * NBT * (NBT + 1), so all of them together look like the diagonal blocks of one
  // matrix of order n and leading dimension NBT, and ?trtri's first levels (128-wide
  // leaves, then pairs up to NBT, on the TF32 tensor cores) invert them in place.
  CUCHOL_CHECK(cudaMemsetAsync(p->Dinv, 0, sizeof(float) * (size_t)nT * NBT * (NBT + 1), sp));
  for (int I = 0; I < nT; ++I) {
    const int b0 = I * NBT, bI = std::min(NBT, n - b0);
    CUCHOL_CHECK_CU(copy_view<float>(h, p->W + b0 + (long long)b0 * p->ldw, 1, p->ldw,
                                     p->Dinv + (size_t)I * NBT * (NBT + 1), 1, NBT, bI, bI, true, sp, nullptr));
  }
  CUCHOL_CHECK_CU(set_smem<float>((const void*)diag_invert_kernel<float, SB, kDiagThreads2>,
                                  BlockSmem<float, SB>::bytes));
  diag_invert_kernel<float, SB, kDiagThreads2><<<(n + SB - 1) / SB, kDiagThreads2, BlockSmem<float, SB>::bytes, sp>>>(
      p->Dinv, 1, NBT, n, SB, 0);
  ++h->launches;
  CUCHOL_CHECK(cudaGetLastError());
  // all blocks at once, or as many as there is memory for
  auto bytes = [&](int blocks) { return trtri_levels_bytes<float>(std::min(n, blocks * NBT), NBT); };
  int per = nT;
  while (per > 1 && !try_workspace(h, bytes(per))) per = (per + 1) / 2;
  CUCHOL_CHECK_CU(ensure_workspace(h, bytes(per)));
  for (int I = 0; I < nT; I += per) {
    bool done = false;
    CUCHOL_CHECK_CU(trtri_levels_tcg<float>(h, false, std::min(n - I * NBT, per * NBT),
                                            p->Dinv + (size_t)I * NBT * (NBT + 1), 1, NBT, NBT, &done));
  }
  CUCHOL_CHECK(cudaStreamSynchronize(sp));
  *info = 0;
  return CUDA_SUCCESS;
}

template <typename Op>
CUresult mixed_create(CUcholMixed* out, CULAPACKhandle h, CBlasUplo uplo, size_t n_, CUdeviceptr A, size_t lda,
                      double shift_in, long* info) {
  const int n = (int)n_;
  auto* p = new (std::nothrow) __cucholmixed_st;
  if (p == nullptr) return CUDA_ERROR_OUT_OF_MEMORY;
  memset(p, 0, sizeof(*p));
  p->h = h;
  p->precision = (sizeof(Op) == 2) ? CUCHOL_MIXED_BF16 : CUCHOL_MIXED_TF32;
  p->n = n;
  p->A = reinterpret_cast<const double*>(A);
  const bool upper = (uplo == CBlasUpper);
  p->rs = upper ? (long long)lda : 1;
  p->cs = upper ? 1 : (long long)lda;
  p->ldw = (long long)round_up((size_t)n, 32);
  p->ld = (long long)round_up((size_t)n, SY);
  const int T = ntile_of(n);
  auto fail = [&](cudaError_t e) {
    free_mixed(p);
    return ::cuchol::report(e, "cudaMalloc", __func__, __FILE__, __LINE__);
  };
  // one device block for everything (an allocation costs about as much as a refinement
  // step, and freeing one waits for the device); pieces on 256-byte boundaries
  const int nT = (n + NBT - 1) / NBT;
  // split k only when a GEMV has fewer than 2 * SMs row blocks: at most NBT / 256 splits
  const size_t gpart = (size_t)(NBT / 256) * (2 * h->num_sms + 1) * GR * NR;
  const size_t ptile = (size_t)T * (T + 1) / 2 * SY * NR;
  const size_t nred = kVecBlocks * NR + kVecBlocks * 2 * NR + 2 * NR + 2 * NR;
  size_t total = 0;
  auto carve = [&](size_t bytes) {
    const size_t at = total;
    total += round_up(bytes, 256);
    return at;
  };
  const size_t oW = carve(sizeof(float) * p->ldw * n), os = carve(sizeof(double) * n),
               oD = carve(sizeof(float) * (size_t)nT * NBT * (NBT + 1)), og = carve(sizeof(float) * gpart),
               ox = carve(sizeof(double) * 6 * p->ld * NR), ot = carve(sizeof(float) * 3 * p->ld * NR),
               oU = carve(sizeof(double) * ptile), oV = carve(sizeof(double) * ptile), op = carve(sizeof(double) * nred),
               oc = carve((16 + 2 * h->num_sms) * sizeof(unsigned));
  cudaError_t e;
  if ((e = dev_malloc(&p->arena, total)) != cudaSuccess) return fail(e);
  p->W = reinterpret_cast<float*>(p->arena + oW);
  p->s = reinterpret_cast<double*>(p->arena + os);
  p->Dinv = reinterpret_cast<float*>(p->arena + oD);
  p->gpart = reinterpret_cast<float*>(p->arena + og);
  p->x = reinterpret_cast<double*>(p->arena + ox);   // x r z p q b
  p->r = p->x + p->ld * NR;
  p->z = p->r + p->ld * NR;
  p->p = p->z + p->ld * NR;
  p->q = p->p + p->ld * NR;
  p->b = p->q + p->ld * NR;
  p->t = reinterpret_cast<float*>(p->arena + ot);
  p->y = p->t + p->ld * NR;
  p->zf = p->y + p->ld * NR;
  p->U = reinterpret_cast<double*>(p->arena + oU);
  p->V = reinterpret_cast<double*>(p->arena + oV);
  p->part = reinterpret_cast<double*>(p->arena + op);
  p->part_norm = p->part + kVecBlocks * NR;
  p->rz = p->part_norm + kVecBlocks * 2 * NR;
  p->norms = p->rz + 2 * NR;
  p->ctr = reinterpret_cast<unsigned*>(p->arena + oc);
  p->err = reinterpret_cast<int*>(p->ctr + 8);
  p->gcount = p->ctr + 16;
  if ((e = cudaMemset(p->ctr, 0, (16 + 2 * h->num_sms) * sizeof(unsigned))) != cudaSuccess) return fail(e);
  p->h_norms = h->h_norms;

  p->shift_request = shift_in;
  *out = p;
  return mixed_refactor<Op>(p, info);
}

// Preconditioned CG in FP64 on A x = b for the columns of B, 16 at a time.
CUresult mixed_solve(CUcholMixed p, int nrhs, const double* B, long long ldb, double* X, long long ldx, double tol,
                     int maxit, int* iter, double* berr) {
  cudaStream_t s = p->h->s_panel;
  const int n = p->n;
  const long long ld = p->ld;
  if (tol <= 0.0) tol = sqrt((double)n) * 0x1p-53;
  if (maxit <= 0) maxit = 100;
  int worst_it = 0;
  bool all_ok = true;
  double worst_berr = 0.0;
  CUCHOL_CHECK(cudaMemsetAsync(p->err, 0, sizeof(int), s));
  for (int g0 = 0; g0 < nrhs; g0 += NR) {
    const int nc = std::min(NR, nrhs - g0);
    load_cols_kernel<<<4 * p->h->num_sms, 256, 0, s>>>(B + (long long)g0 * ldb, ldb, nc, n, p->b, ld);
    CUCHOL_CHECK(cudaGetLastError());
    CUCHOL_CHECK(cudaMemcpyAsync(p->r, p->b, sizeof(double) * ld * NR, cudaMemcpyDeviceToDevice, s));
    CUCHOL_CHECK(cudaMemsetAsync(p->x, 0, sizeof(double) * ld * NR, s));
    norms_kernel<<<kVecBlocks, kThreads, 0, s>>>(p->b, nullptr, n, ld, p->part_norm);
    CUCHOL_CHECK(cudaGetLastError());
    CUCHOL_CHECK_CU(fetch_norms(p, s));
    double bn[NR];
    for (int c = 0; c < NR; ++c) bn[c] = p->h_norms[c];
    auto backward = [&](const double* rx, double* eta) {   // rx: [0,NR) |r|, [NR,2NR) |x|
      bool ok = true;
      for (int c = 0; c < nc; ++c) {
        const double den = p->anorm * rx[NR + c] + bn[c];
        eta[c] = den > 0.0 ? rx[c] / den : 0.0;
        if (!(eta[c] <= tol)) ok = false;
      }
      return ok;
    };
    double eta[NR] = {0};
    int it = 0, slot = 0;
    bool done = false;
    while (!done && it < maxit) {
      // (re)start from the current residual: p = z = M^-1 r
      CUCHOL_CHECK_CU(precond(p, p->r, p->z, s));
      dot_kernel<<<kVecBlocks, kThreads, 0, s>>>(p->r, p->z, n, ld, p->part);
      update_p_kernel<<<kVecBlocks, kThreads, 0, s>>>(p->p, p->z, n, ld, p->part, p->rz + slot * NR,
                                                      p->rz + (slot ^ 1) * NR, 1);
      CUCHOL_CHECK(cudaGetLastError());
      slot ^= 1;
      while (it < maxit) {
        CUCHOL_CHECK_CU(symv(p->h->device, p->A, p->rs, p->cs, n, p->p, ld, NR, 0, 1.0, 0.0, nullptr, 0, p->q, ld, p->U, p->V, s));
        dot_kernel<<<kVecBlocks, kThreads, 0, s>>>(p->p, p->q, n, ld, p->part);
        update_xr_kernel<<<kVecBlocks, kThreads, 0, s>>>(p->x, p->r, p->p, p->q, n, ld, p->part, p->rz + slot * NR,
                                                         p->part_norm);
        CUCHOL_CHECK(cudaGetLastError());
        CUCHOL_CHECK_CU(fetch_norms(p, s));
        ++it;
        if (backward(p->h_norms, eta)) break;
        CUCHOL_CHECK_CU(precond(p, p->r, p->z, s));
        dot_kernel<<<kVecBlocks, kThreads, 0, s>>>(p->r, p->z, n, ld, p->part);
        update_p_kernel<<<kVecBlocks, kThreads, 0, s>>>(p->p, p->z, n, ld, p->part, p->rz + slot * NR,
                                                        p->rz + (slot ^ 1) * NR, 0);
        CUCHOL_CHECK(cudaGetLastError());
        slot ^= 1;
      }
      // FP64 residual from scratch: r = b - A x
      CUCHOL_CHECK_CU(symv(p->h->device, p->A, p->rs, p->cs, n, p->x, ld, NR, 0, -1.0, 1.0, p->b, ld, p->r, ld, p->U, p->V, s));
      norms_kernel<<<kVecBlocks, kThreads, 0, s>>>(p->r, p->x, n, ld, p->part_norm);
      CUCHOL_CHECK(cudaGetLastError());
      CUCHOL_CHECK_CU(fetch_norms(p, s));
      done = backward(p->h_norms, eta);
    }
    store_cols_kernel<<<4 * p->h->num_sms, 256, 0, s>>>(p->x, ld, nc, n, X + (long long)g0 * ldx, ldx);
    CUCHOL_CHECK(cudaGetLastError());
    for (int c = 0; c < nc; ++c) worst_berr = std::max(worst_berr, eta[c]);
    worst_it = std::max(worst_it, it);
    if (!done) all_ok = false;
  }
  int err = 0;
  CUCHOL_CHECK(cudaMemcpyAsync(&err, p->err, sizeof(int), cudaMemcpyDeviceToHost, s));
  CUCHOL_CHECK(cudaStreamSynchronize(s));
  if (err != 0) {
    if (errorHandler != nullptr)
      errorHandler("triangular solve wait", __func__, __FILE__, __LINE__, (int)CUDA_ERROR_LAUNCH_TIMEOUT,
                   &error_string);
    return CUDA_ERROR_LAUNCH_TIMEOUT;
  }
  *iter = all_ok ? worst_it : -worst_it;
  if (berr != nullptr) *berr = worst_berr;
  return CUDA_SUCCESS;
}

// ?POTRS: B := A^-1 B from the Cholesky factor in A (lower L or upper U = L^T).
template <typename T>
CUresult potrs_run(CULAPACKhandle h, bool upper, int n, int nrhs, const T* A, long long lda, T* B, long long ldb) {
  cudaStream_t s = h->s_panel;
  const long long rs = upper ? lda : 1, cs = upper ? 1 : lda;
  const int nblk = (n + BS - 1) / BS;
  const long long ldy = (long long)nblk * BS;
  const size_t di = round_up(sizeof(T) * (size_t)nblk * BS * BS, 256);
  CUCHOL_CHECK_CU(ensure_workspace(h, di + sizeof(T) * ldy * NR));
  T* DI = static_cast<T*>(h->ws);
  T* Y = reinterpret_cast<T*>(static_cast<char*>(h->ws) + di);
  unsigned* ctr = reinterpret_cast<unsigned*>(h->d_words + 8);   // words 8..11
  int* err = h->d_words + 3;
  CUCHOL_CHECK_CU(block_inverse<T>(h->device, A, rs, cs, n, DI, s));
  CUCHOL_CHECK_CU((trsv_attr<T, T>(h->device)));
  for (int g0 = 0; g0 < nrhs; g0 += NR) {
    const int nc = std::min(NR, nrhs - g0);
    T* Bg = B + (long long)g0 * ldb;
    CUCHOL_CHECK(cudaMemsetAsync(ctr, 0, 4 * sizeof(unsigned), s));
    trsv_fwd_kernel<T, T><<<nblk, kThreads, trsv_smem<T>(), s>>>(A, rs, cs, n, DI, Bg, ldb, nullptr, Y, ldy, nc, ctr, err,
                                                                      h->wait_limit);
    CUCHOL_CHECK(cudaGetLastError());
    trsv_bwd_kernel<T, T><<<nblk, kThreads, trsv_smem<T>(), s>>>(A, rs, cs, n, DI, Y, ldy, nullptr, Bg, ldb, Y, nc, ctr + 2,
                                                    err, h->wait_limit);
    CUCHOL_CHECK(cudaGetLastError());
    h->launches += 2;
  }
  return fetch_words(h, s);
}

}  // namespace mx
}  // namespace

// ------------------------------------------------------------------------------
// C ABI (include/cucholesky_ext.h)
// ------------------------------------------------------------------------------
namespace {
template <typename T>
CUresult api_potrs(const char* name, CULAPACKhandle h, CBlasUplo uplo, size_t n, size_t nrhs, CUdeviceptr A,
                   size_t lda, CUdeviceptr B, size_t ldb, long* info) {
  if (info == nullptr) return CUDA_ERROR_INVALID_VALUE;
  *info = 0;
  if (bad_uplo(uplo)) *info = -2;
  else if (lda < std::max<size_t>(1, n)) *info = -6;
  else if (ldb < std::max<size_t>(1, n)) *info = -8;
  if (*info != 0) {
    if (xerbla != nullptr) xerbla(name, -*info);
    return CUDA_ERROR_INVALID_VALUE;
  }
  if (h == nullptr) return CUDA_ERROR_INVALID_VALUE;
  if (n == 0 || nrhs == 0) return CUDA_SUCCESS;
  return mx::potrs_run<T>(h, uplo == CBlasUpper, (int)n, (int)nrhs, reinterpret_cast<const T*>(A), (long long)lda,
                          reinterpret_cast<T*>(B), (long long)ldb);
}
}  // namespace

extern "C" CUCHOL_EXPORT CUresult cuDpotrs(CULAPACKhandle h, CBlasUplo uplo, size_t n, size_t nrhs, CUdeviceptr A,
                                           size_t lda, CUdeviceptr B, size_t ldb, long* info) {
  return api_potrs<double>("cuDpotrs", h, uplo, n, nrhs, A, lda, B, ldb, info);
}
extern "C" CUCHOL_EXPORT CUresult cuSpotrs(CULAPACKhandle h, CBlasUplo uplo, size_t n, size_t nrhs, CUdeviceptr A,
                                           size_t lda, CUdeviceptr B, size_t ldb, long* info) {
  return api_potrs<float>("cuSpotrs", h, uplo, n, nrhs, A, lda, B, ldb, info);
}

extern "C" CUCHOL_EXPORT CUresult cuDcholMixedCreate(CUcholMixed* plan, CULAPACKhandle h, CBlasUplo uplo, size_t n,
                                                     CUdeviceptr A, size_t lda, int precision, double shift,
                                                     long* info) {
  if (plan == nullptr || info == nullptr) return CUDA_ERROR_INVALID_VALUE;
  *plan = nullptr;
  *info = 0;
  if (bad_uplo(uplo)) *info = -3;
  else if (n == 0 || n > (size_t)INT_MAX / 2) *info = -4;
  else if (lda < n) *info = -6;
  else if (precision != CUCHOL_MIXED_BF16 && precision != CUCHOL_MIXED_TF32) *info = -7;
  if (*info != 0) {
    if (xerbla != nullptr) xerbla("cuDcholMixedCreate", -*info);
    return CUDA_ERROR_INVALID_VALUE;
  }
  if (h == nullptr) return CUDA_ERROR_INVALID_VALUE;
  if (precision == CUCHOL_MIXED_BF16) return mx::mixed_create<__nv_bfloat16>(plan, h, uplo, n, A, lda, shift, info);
  return mx::mixed_create<float>(plan, h, uplo, n, A, lda, shift, info);
}

// The factor's trailing-update kernel on its own: C(i, j) += alpha sum_l Q(i, l) Q(j, l)
// for i >= j, Q k-major (row i at Q + i * ldq) in BF16 or TF32 (FP32 words), C FP32
// column-major.  Queued on `stream`.
extern "C" CUCHOL_EXPORT CUresult cuSsyrkLowp(CULAPACKhandle h, int precision, size_t n, size_t k, float alpha,
                                              CUdeviceptr Q, size_t ldq, CUdeviceptr C, size_t ldc,
                                              CUstream stream) {
  long info = 0;
  const size_t esize = (precision == CUCHOL_MIXED_BF16) ? 2 : 4;
  if (precision != CUCHOL_MIXED_BF16 && precision != CUCHOL_MIXED_TF32) info = 2;
  else if (n > (size_t)INT_MAX) info = 3;
  else if (k > (size_t)INT_MAX) info = 4;
  else if (ldq < k || (ldq * esize) % 16 != 0 || (Q & 15) != 0) info = 7;
  else if (ldc < n || ldc % 4 != 0 || (C & 15) != 0) info = 9;
  if (info != 0) {
    if (xerbla != nullptr) xerbla("cuSsyrkLowp", info);
    return CUDA_ERROR_INVALID_VALUE;
  }
  if (h == nullptr) return CUDA_ERROR_INVALID_VALUE;
  if (n == 0 || k == 0) return CUDA_SUCCESS;
  cudaStream_t s = reinterpret_cast<cudaStream_t>(stream);
  int* stop = h->d_words + 5;   // never set: the update has no earlier step to depend on
  CUCHOL_CHECK(cudaMemsetAsync(stop, 0, sizeof(int), s));
  if (precision == CUCHOL_MIXED_BF16)
    return mx::tc_update<__nv_bfloat16>(h, reinterpret_cast<const __nv_bfloat16*>(Q), (long long)ldq, (int)n,
                                        (int)k, 0, 0, reinterpret_cast<float*>(C), (long long)ldc, (int)n, (int)n, s,
                                        stop, alpha);
  return mx::tc_update<float>(h, reinterpret_cast<const float*>(Q), (long long)ldq, (int)n, (int)k, 0, 0,
                              reinterpret_cast<float*>(C), (long long)ldc, (int)n, (int)n, s, stop, alpha);
}

extern "C" CUCHOL_EXPORT CUresult cuDcholMixedRefactor(CUcholMixed p, long* info) {
  if (p == nullptr || info == nullptr) return CUDA_ERROR_INVALID_VALUE;
  if (p->precision == CUCHOL_MIXED_BF16) return mx::mixed_refactor<__nv_bfloat16>(p, info);
  return mx::mixed_refactor<float>(p, info);
}

extern "C" CUCHOL_EXPORT CUresult cuDcholMixedSolve(CUcholMixed p, size_t nrhs, CUdeviceptr B, size_t ldb,
                                                    CUdeviceptr X, size_t ldx, double tol, int maxit, int* iter,
                                                    double* berr) {
  if (p == nullptr || iter == nullptr || ldb < (size_t)p->n || ldx < (size_t)p->n) return CUDA_ERROR_INVALID_VALUE;
  *iter = 0;
  if (nrhs == 0) return CUDA_SUCCESS;
  return mx::mixed_solve(p, (int)nrhs, reinterpret_cast<const double*>(B), (long long)ldb,
                         reinterpret_cast<double*>(X), (long long)ldx, tol, maxit, iter, berr);
}

extern "C" CUCHOL_EXPORT CUresult cuCholMixedGetFactor(CUcholMixed p, CUdeviceptr* W, size_t* ldw, CUdeviceptr* s,
                                                       double* anorm, double* shift) {
  if (p == nullptr) return CUDA_ERROR_INVALID_VALUE;
  if (W != nullptr) *W = reinterpret_cast<CUdeviceptr>(p->W);
  if (ldw != nullptr) *ldw = (size_t)p->ldw;
  if (s != nullptr) *s = reinterpret_cast<CUdeviceptr>(p->s);
  if (anorm != nullptr) *anorm = p->anorm;
  if (shift != nullptr) *shift = p->shift;
  return CUDA_SUCCESS;
}

extern "C" CUCHOL_EXPORT CUresult cuCholMixedDestroy(CUcholMixed p) {
  if (p == nullptr) return CUDA_ERROR_INVALID_VALUE;
  cudaDeviceSynchronize();
  mx::free_mixed(p);
  return CUDA_SUCCESS;
}

// DSPOSV contract: iter > 0 -> refined mixed-precision solution, A unchanged;
// iter < 0 -> FP64 fallback (-3: the low-precision factor broke down, -31: no
// convergence within maxit), A holds the FP64 factor and info is cuDpotrf's.
extern "C" CUCHOL_EXPORT CUresult cuDposvMixed(CULAPACKhandle h, CBlasUplo uplo, size_t n, size_t nrhs,
                                               CUdeviceptr A, size_t lda, CUdeviceptr B, size_t ldb, CUdeviceptr X,
                                               size_t ldx, int precision, int* iter, double* berr, long* info) {
  if (iter == nullptr || info == nullptr) return CUDA_ERROR_INVALID_VALUE;
  *iter = 0;
  *info = 0;
  if (bad_uplo(uplo)) *info = -2;
  else if (lda < std::max<size_t>(1, n)) *info = -6;
  else if (ldb < std::max<size_t>(1, n)) *info = -8;
  else if (ldx < std::max<size_t>(1, n)) *info = -10;
  else if (precision != CUCHOL_MIXED_BF16 && precision != CUCHOL_MIXED_TF32) *info = -11;
  if (*info != 0) {
    if (xerbla != nullptr) xerbla("cuDposvMixed", -*info);
    return CUDA_ERROR_INVALID_VALUE;
  }
  if (h == nullptr) return CUDA_ERROR_INVALID_VALUE;
  if (n == 0 || nrhs == 0) return CUDA_SUCCESS;
  CUcholMixed p = nullptr;
  long finfo = 0;
  CUresult r = cuDcholMixedCreate(&p, h, uplo, n, A, lda, precision, -1.0, &finfo);
  if (r != CUDA_SUCCESS) return r;
  int it = 0;
  if (finfo == 0) {
    r = cuDcholMixedSolve(p, nrhs, B, ldb, X, ldx, 0.0, 0, &it, berr);
    if (r != CUDA_SUCCESS) {
      cuCholMixedDestroy(p);
      return r;
    }
  }
  cuCholMixedDestroy(p);
  if (finfo == 0 && it > 0) {
    *iter = it;
    return CUDA_SUCCESS;
  }
  *iter = (finfo != 0) ? -3 : -31;
  // FP64 fallback: X = B, factor A in place, solve
  CUCHOL_CHECK(cudaMemcpy2D(reinterpret_cast<void*>(X), ldx * sizeof(double), reinterpret_cast<const void*>(B),
                            ldb * sizeof(double), n * sizeof(double), nrhs, cudaMemcpyDeviceToDevice));
  r = cuDpotrf(h, uplo, n, A, lda, info);
  if (r != CUDA_SUCCESS || *info != 0) return r;
  long pinfo = 0;
  r = cuDpotrs(h, uplo, n, nrhs, A, lda, X, ldx, &pinfo);
  if (berr != nullptr) *berr = -1.0;
  return r;
}
