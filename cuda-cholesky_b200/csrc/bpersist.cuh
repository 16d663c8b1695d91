// Persistent form of the batched plan (included at the end of lapack.cu, after
// batched.cuh): one launch factors, log-dets and inverts every matrix of the batch.
//
// Each CTA (three of four warps per SM: while one is in a diagonal step or at a barrier the
// others have tile products to run) takes whole matrices from a work queue ordered by size,
// largest first (the longest-processing-time rule: the last matrices taken are the
// cheapest, so the CTAs finish together), and runs the blocked algorithms on the
// matrix in place as a sequence of phases over 64 x 64 tiles:
//   ?potrf  for each block column k: its tiles A_ik -= sum_{l < k} L_il L_kl^T; the
//           diagonal block factored (and its inverse W formed) in shared memory; panel
//           tiles L_ik = A_ik W^T;
//   ?trtri  every diagonal tile replaced by the inverse that the factor formed for its
//           panel (kept aside until the factor has succeeded); then, block column j from the last
//           to the first, X_ij = sum_{l=j+1..i} inv(L)_il L_lj (rows from the bottom
//           up, so each row still reads the L_lj of the rows above it) and then
//           inv(L)_ij = -X_ij inv(L_jj);
//   ?lauum  C_ij = sum_{l >= i} inv(L)_li^T inv(L)_lj, block column j from the first,
//           rows from the top down: each tile reads only tiles that are rewritten
//           after it.
// The jobs of a phase are independent of each other (by the orders above), so the
// operand tiles of the next 32 k are fetched (cp.async, two-stage ring) while the
// current ones are multiplied: FP64 on the tensor cores (mma.sync m16n8k4, four warps of
// 32 x 32 outputs), FP32 with 8 x 4 outputs per thread.  Phases are separated by barriers.
// The diagonal steps are those of panel.cuh.  A matrix whose factor fails keeps its info
// word and is left as the factor left it.
#pragma once

namespace {
namespace bpk {

constexpr int NB = 64, THREADS = 128, CTAS = kPersistentCtas, LDS = 68;      // tile order; staged rows padded to 68
constexpr int KS = 32;                                // k per stage
constexpr int TILE = KS * LDS;                        // elements per staged operand tile
template <typename T> constexpr size_t ring_bytes() { return 2 * 2 * TILE * sizeof(T); }   // 2 stages x (A, B)

template <typename T>
struct MatDesc {
  T* a;
  int n, lda;
  int* info;
  double* logdet;     // or null
};

// Operand of a tile product: element (r, k) at p[r * rs + k * ks] for r < m, k < kk;
// tri: TRI_LOWER keeps k <= r, TRI_UPPER keeps k >= r (the rest reads as zero).
template <typename T>
struct Opnd {
  const T* p;
  long long rs, ks;
  int m, kk, tri;
};

// Output of a job: C(r, c) at p[r * rs + c * cs], r < m, c < n (lower: only r >= c);
// C := acc, -acc (neg), or C - acc (sub: the accumulators then start at -C, so that the sum
// runs down to the Schur complement as step-by-step updates do and does not cancel at its
// end: FP32 log dets of ill-conditioned kernels lost half a digit otherwise).
template <typename T>
struct Out {
  T* p;
  long long rs, cs;
  int m, n;
  int neg, sub;
  int lower;
};

__device__ __forceinline__ void cp_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
__device__ __forceinline__ void cp_wait1() { asm volatile("cp.async.wait_group 1;" ::: "memory"); }

// Stage k = k0 .. k0 + 31 of one operand tile into X[(k - k0) * LDS + r] (cp.async, zeros
// where not kept).  Rows contiguous in memory: consecutive lanes take consecutive rows
// (conflict-free shared stores).  k contiguous: each 8 lanes take 8 consecutive k of one
// row, 4 rows per warp, so the shared stores, 68 elements apart along k, spread over the
// banks.
template <typename T>
__device__ __forceinline__ void stage(const Opnd<T>& o, int k0, T* X) {
  const int t = threadIdx.x;
  if (o.rs == 1) {
    const int r = t & (NB - 1);
    const T* src = o.p + r + (long long)(k0 + (t >> 6)) * o.ks;
    const long long step = 2 * o.ks;
    const bool rv = r < o.m;
    // k <= hi and k >= lo are kept
    const int hi = min(o.kk - 1, o.tri == TRI_LOWER ? r : NB), lo = o.tri == TRI_UPPER ? r : 0;
#pragma unroll
    for (int u = 0; u < KS / 2; ++u, src += step) {
      const int kl = (t >> 6) + 2 * u, k = k0 + kl;
      const bool v = rv && k <= hi && k >= lo;
      cp_async_elem<T>(&X[kl * LDS + r], v ? src : o.p, v);
    }
  } else {
    const int kl0 = (t & 7) + 8 * (t >> 5), k = k0 + kl0, r0 = (t >> 3) & 3;
    const T* src = o.p + (long long)r0 * o.rs + (long long)k * o.ks;
    const long long step = 4 * o.rs;
    // rows lo <= r < hi are kept
    const int hi = (k < o.kk) ? min(o.m, o.tri == TRI_UPPER ? k + 1 : NB) : 0, lo = o.tri == TRI_LOWER ? k : 0;
#pragma unroll
    for (int u = 0; u < NB / 4; ++u, src += step) {
      const int r = r0 + 4 * u;
      const bool v = r < hi && r >= lo;
      cp_async_elem<T>(&X[kl0 * LDS + r], v ? src : o.p, v);
    }
  }
}

// 64 x 64 accumulators of the CTA.
template <typename T> struct Acc;

// FP64: warp w holds rows 32 (w & 1) .. + 31, columns 32 (w >> 1) .. + 31 as DMMA fragments
// (g, t) of lane = 4 g + t.  A lane takes rows 2g, 2g + 1 of an m16 block's half and columns
// 2g, 2g + 1 of a pair of n8 blocks, so each fragment pair is one 16-byte shared load
// (a quarter warp touches chunks 2t + g: conflict-free), four loads per eight MMAs.
template <> struct Acc<double> {
  double v[2][4][4];
  __device__ __forceinline__ void clear() {
#pragma unroll
    for (int a = 0; a < 2; ++a)
#pragma unroll
      for (int b = 0; b < 4; ++b)
#pragma unroll
        for (int c = 0; c < 4; ++c) v[a][b][c] = 0.0;
  }
  // += A B^T for the staged tiles
  __device__ __forceinline__ void mma(const double* As, const double* Bs) {
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
    const int r0 = (warp & 1) * 32, c0 = (warp >> 1) * 32;
#pragma unroll 4
    for (int k4 = 0; k4 < KS; k4 += 4) {
      const double* a = As + (k4 + t) * LDS + r0 + 2 * g;
      const double* b = Bs + (k4 + t) * LDS + c0 + 2 * g;
      const double2 a0 = *reinterpret_cast<const double2*>(a), a1 = *reinterpret_cast<const double2*>(a + 16);
      const double2 b0 = *reinterpret_cast<const double2*>(b), b1 = *reinterpret_cast<const double2*>(b + 16);
      cuchol::dmma_m16n8k4(v[0][0], a0.x, a0.y, b0.x);
      cuchol::dmma_m16n8k4(v[0][1], a0.x, a0.y, b0.y);
      cuchol::dmma_m16n8k4(v[0][2], a0.x, a0.y, b1.x);
      cuchol::dmma_m16n8k4(v[0][3], a0.x, a0.y, b1.y);
      cuchol::dmma_m16n8k4(v[1][0], a1.x, a1.y, b0.x);
      cuchol::dmma_m16n8k4(v[1][1], a1.x, a1.y, b0.y);
      cuchol::dmma_m16n8k4(v[1][2], a1.x, a1.y, b1.x);
      cuchol::dmma_m16n8k4(v[1][3], a1.x, a1.y, b1.y);
    }
  }
  // f(row, column, value): fragment element e is row 2g + (e >> 1) and MMA column
  // 2t + (e & 1), which is column 2 (2t + (e & 1)) + (block & 1) of its pair
  template <typename F>
  __device__ __forceinline__ void each(F f) {
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
    const int r0 = (warp & 1) * 32, c0 = (warp >> 1) * 32;
#pragma unroll
    for (int mb = 0; mb < 2; ++mb)
#pragma unroll
      for (int nb8 = 0; nb8 < 4; ++nb8)
#pragma unroll
        for (int e = 0; e < 4; ++e)
          f(r0 + mb * 16 + 2 * g + (e >> 1), c0 + (nb8 >> 1) * 16 + 4 * t + 2 * (e & 1) + (nb8 & 1), v[mb][nb8][e]);
  }
};

// FP32: thread (tx, ty) holds rows 4 tx .. + 3 and 32 + 4 tx .. + 3, columns 4 ty .. + 3
// (three 16-byte shared loads per 32 FMAs).
template <> struct Acc<float> {
  float v[8][4];
  __device__ __forceinline__ void clear() {
#pragma unroll
    for (int a = 0; a < 8; ++a)
#pragma unroll
      for (int b = 0; b < 4; ++b) v[a][b] = 0.f;
  }
  __device__ __forceinline__ void mma(const float* As, const float* Bs) {
    const int tx = threadIdx.x & 7, ty = threadIdx.x >> 3;
#pragma unroll 8
    for (int k = 0; k < KS; ++k) {
      const float4 a = *reinterpret_cast<const float4*>(As + k * LDS + 4 * tx);
      const float4 d = *reinterpret_cast<const float4*>(As + k * LDS + 32 + 4 * tx);
      const float4 b = *reinterpret_cast<const float4*>(Bs + k * LDS + 4 * ty);
      const float av[8] = {a.x, a.y, a.z, a.w, d.x, d.y, d.z, d.w}, bv[4] = {b.x, b.y, b.z, b.w};
#pragma unroll
      for (int i = 0; i < 8; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) v[i][j] = fmaf(av[i], bv[j], v[i][j]);
    }
  }
  template <typename F>
  __device__ __forceinline__ void each(F f) {
    const int tx = threadIdx.x & 7, ty = threadIdx.x >> 3;
#pragma unroll
    for (int j = 0; j < 4; ++j)
#pragma unroll
      for (int i = 0; i < 8; ++i) f(4 * tx + (i & 3) + 32 * (i >> 2), 4 * ty + j, v[i][j]);
  }
};

// Runs the njobs jobs of one phase: job j has nterms(j) terms term(j, t, &a, &b) and
// output out(j).  Loads run one 32-k item ahead, across term and job boundaries.
template <typename T, typename NT, typename TF, typename OF>
__device__ __forceinline__ void run_phase(int njobs, NT nterms, TF term, OF out, T* ring) {
  if (njobs <= 0) return;
  Acc<T> acc;
  auto start = [&](int j) {
    const Out<T> o = out(j);
    acc.clear();
    if (o.sub)
      acc.each([&](int r, int c, T& x) {
        if (r < o.m && c < o.n && (!o.lower || r >= c)) x = -o.p[r * o.rs + c * o.cs];
      });
  };
  int job = 0, tt = 0, k0 = 0, st = 0, jn = nterms(0);   // the item being multiplied
  Opnd<T> A, B;
  term(0, 0, A, B);
  auto issue = [&](int s, int k) {
    stage<T>(A, k, ring + s * 2 * TILE);
    stage<T>(B, k, ring + s * 2 * TILE + TILE);
  };
  issue(0, 0);
  cp_commit();
  start(0);
  while (true) {
    // the next item: 32 k further, the next term, or the next job
    int nj = job, nt = tt, nk = k0 + KS;
    bool more = true;
    if (nk >= A.kk) {
      nk = 0;
      ++nt;
      if (nt >= jn) {
        nt = 0;
        ++nj;
        more = nj < njobs;
      }
      if (more) term(nj, nt, A, B);
    }
    if (more) issue(st ^ 1, nk);
    cp_commit();
    cp_wait1();
    __syncthreads();
    acc.mma(ring + st * 2 * TILE, ring + st * 2 * TILE + TILE);
    __syncthreads();                                 // stage st is refilled next
    if (nj != job) {
      const Out<T> o = out(job);
      const bool neg = o.neg || o.sub;
      acc.each([&](int r, int c, T& x) {
        if (r < o.m && c < o.n && (!o.lower || r >= c)) o.p[r * o.rs + c * o.cs] = neg ? -x : x;
      });
      if (!more) break;
      start(nj);
      jn = nterms(nj);
    }
    job = nj;
    tt = nt;
    k0 = nk;
    st ^= 1;
  }
  asm volatile("cp.async.wait_all;" ::: "memory");
  __syncthreads();                                   // outputs visible to the next phase
}

// Factor, log det and inverse of one matrix (lower view A(i, j) = a[i * rs + j * cs]).
template <typename T>
__device__ void process(const MatDesc<T>& M, long long rs, long long cs, bool inverse, T* W, T* ring) {
  const int n = M.n, nt = (n + NB - 1) / NB;
  T* a = M.a;
  auto tl = [&](int i, int j) { return a + (long long)i * NB * rs + (long long)j * NB * cs; };
  auto ext = [&](int i) { return min(NB, n - i * NB); };

  // W + k * NB * NB: the inverse of diagonal factor block k (ld NB), kept for the panel
  // below it and, with the inverse to follow, for ?trtri
  auto Wk = [&](int k) { return W + (inverse ? (size_t)k * NB * NB : 0); };

  // ---- ?potrf, left-looking: block column k takes all its updates at once, so a tile is
  // read and written once per step and not once per earlier column ----
  for (int k = 0; k < nt; ++k) {
    const int jb = ext(k);
    const int m = nt - k - 1;                        // tiles below the diagonal one
    // A_ik -= sum_{l < k} L_il L_kl^T, i = k .. (the diagonal tile's lower part)
    if (k > 0)
      run_phase<T>(
          m + 1, [&](int) { return k; },
          [&](int q, int l, Opnd<T>& A, Opnd<T>& B) {
            const int i = k + q;
            A = Opnd<T>{tl(i, l), rs, cs, ext(i), NB, TRI_NONE};
            B = Opnd<T>{tl(k, l), rs, cs, jb, NB, TRI_NONE};
          },
          [&](int q) {
            const int i = k + q;
            return Out<T>{tl(i, k), rs, cs, ext(i), jb, 0, 1, q == 0};
          },
          ring);
    cuchol::diag_factor_block<T, NB, THREADS>(tl(k, k), rs, cs, jb, (m > 0 || inverse) ? Wk(k) : nullptr, NB,
                                              (long long)k * NB, M.info, M.logdet);
    __syncthreads();
    if (cuchol::cta_aborted(M.info)) return;         // this matrix's factor failed
    // panel: L_ik = A_ik W^T, i = k+1 ..
    run_phase<T>(
        m, [](int) { return 1; },
        [&](int j, int, Opnd<T>& A, Opnd<T>& B) {
          const int i = k + 1 + j;
          A = Opnd<T>{tl(i, k), rs, cs, ext(i), jb, TRI_NONE};
          B = Opnd<T>{Wk(k), 1, NB, jb, jb, TRI_NONE};   // B(c, kk) = W(c, kk): zeros above the diagonal
        },
        [&](int j) {
          const int i = k + 1 + j;
          return Out<T>{tl(i, k), rs, cs, ext(i), jb, 0, 0, 0};
        },
        ring);
  }
  if (!inverse) return;

  // ---- ?trtri: the diagonal tiles take the inverses formed by the factor, then the
  // block columns from the last ----
  for (int k = 0; k < nt; ++k) {
    const int jb = ext(k);
    const T* w = Wk(k);
    for (int e = threadIdx.x; e < jb * jb; e += THREADS) {
      const int r = e % jb, c = e / jb;
      if (r >= c) tl(k, k)[r * rs + c * cs] = w[r + c * NB];
    }
  }
  __syncthreads();
  for (int j = nt - 2; j >= 0; --j) {
    const int m = nt - j - 1;
    // X_ij = sum_{l = j+1 .. i} inv(L)_il L_lj, rows i from the bottom up (in place)
    run_phase<T>(
        m, [&](int q) { return m - q; },              // row i = nt-1-q has i - j terms
        [&](int q, int t, Opnd<T>& A, Opnd<T>& B) {
          const int i = nt - 1 - q, l = j + 1 + t;
          // A(r, kk) = inv(L)_il(r, kk); the diagonal tile is lower triangular
          A = Opnd<T>{tl(i, l), rs, cs, ext(i), ext(l), l == i ? TRI_LOWER : TRI_NONE};
          // B(c, kk) = L_lj(kk, c): the transposed view
          B = Opnd<T>{tl(l, j), cs, rs, ext(j), ext(l), TRI_NONE};
        },
        [&](int q) {
          const int i = nt - 1 - q;
          return Out<T>{tl(i, j), rs, cs, ext(i), ext(j), 0, 0, 0};
        },
        ring);
    // inv(L)_ij = -X_ij inv(L_jj): B(c, kk) = inv(L_jj)(kk, c), nonzero for kk >= c
    run_phase<T>(
        m, [](int) { return 1; },
        [&](int q, int, Opnd<T>& A, Opnd<T>& B) {
          const int i = j + 1 + q;
          A = Opnd<T>{tl(i, j), rs, cs, ext(i), ext(j), TRI_NONE};
          B = Opnd<T>{tl(j, j), cs, rs, ext(j), ext(j), TRI_UPPER};
        },
        [&](int q) {
          const int i = j + 1 + q;
          return Out<T>{tl(i, j), rs, cs, ext(i), ext(j), 1, 0, 0};
        },
        ring);
  }
  // ---- ?lauum: C_ij = sum_{l >= i} inv(L)_li^T inv(L)_lj, j ascending, i ascending ----
  run_phase<T>(
      nt * (nt + 1) / 2,
      [&](int q) {
        int j = 0;
        while (q >= nt - j) { q -= nt - j; ++j; }
        const int i = j + q;
        return nt - i;
      },
      [&](int q, int t, Opnd<T>& A, Opnd<T>& B) {
        int j = 0;
        while (q >= nt - j) { q -= nt - j; ++j; }
        const int i = j + q, l = i + t;
        // A(r, kk) = inv(L)_li(kk, r) (transposed view; the diagonal tile l == i is
        // lower triangular: kk >= r), B(c, kk) = inv(L)_lj(kk, c) (lower when l == j)
        A = Opnd<T>{tl(l, i), cs, rs, ext(i), ext(l), l == i ? TRI_UPPER : TRI_NONE};
        B = Opnd<T>{tl(l, j), cs, rs, ext(j), ext(l), l == j ? TRI_UPPER : TRI_NONE};
      },
      [&](int q) {
        int j = 0;
        while (q >= nt - j) { q -= nt - j; ++j; }
        const int i = j + q;
        return Out<T>{tl(i, j), rs, cs, ext(i), ext(j), 0, 0, i == j};
      },
      ring);
}

// order: matrix indices, largest first; *next: the queue head (zero at launch).
// wbuf: per CTA, ntmax inverse blocks of NB x NB (ntmax = block columns of the largest
// matrix).
template <typename T>
__global__ void __launch_bounds__(THREADS, CTAS)
    persistent_kernel(const MatDesc<T>* __restrict__ mats, const int* __restrict__ order, int batch, int* next,
                      int upper, int inverse, T* wbuf, int ntmax) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  T* ring = reinterpret_cast<T*>(smem_raw);
  T* W = wbuf + (size_t)blockIdx.x * ntmax * NB * NB;
  __shared__ int s_w;
  while (true) {
    if (threadIdx.x == 0) s_w = atomicAdd(next, 1);
    __syncthreads();
    const int w = s_w;
    __syncthreads();
    if (w >= batch) break;
    const MatDesc<T> M = mats[order[w]];
    const long long rs = upper ? M.lda : 1, cs = upper ? 1 : M.lda;
    process<T>(M, rs, cs, inverse != 0, W, ring);
    __syncthreads();
  }
}

template <typename T>
constexpr size_t smem_bytes() {
  return ring_bytes<T>() > cuchol::BlockSmem<T, NB>::bytes ? ring_bytes<T>() : cuchol::BlockSmem<T, NB>::bytes;
}

}  // namespace bpk
}  // namespace

namespace {

// The persistent form as the plan's recorded sequence: per-matrix descriptors and
// the size order uploaded once; per run, the result words and the queue head
// cleared, then one launch (three CTAs per SM, no more than matrices).
template <typename T>
CUresult record_persistent(CUcholBatched p, const BatchedShape<T>& sh, cudaStream_t s) {
  CULAPACKhandle h = p->h;
  const int B = sh.batch;
  std::vector<bpk::MatDesc<T>> mats(B);
  for (int b = 0; b < B; ++b)
    mats[b] = bpk::MatDesc<T>{sh.a[b], sh.n[b], (int)sh.lda[b], p->d_info + b,
                           (sh.flags & 2) ? p->d_logdet + b : nullptr};
  std::vector<int> order(B);
  for (int b = 0; b < B; ++b) order[b] = b;
  std::stable_sort(order.begin(), order.end(), [&](int x, int y) { return sh.n[x] > sh.n[y]; });
  CUresult rc = CUDA_SUCCESS;
  const bpk::MatDesc<T>* dm = upload(p, mats, &rc);
  if (dm == nullptr) return rc == CUDA_SUCCESS ? CUDA_ERROR_OUT_OF_MEMORY : rc;
  const int* dord = upload(p, order, &rc);
  if (dord == nullptr) return rc == CUDA_SUCCESS ? CUDA_ERROR_OUT_OF_MEMORY : rc;
  if (p->dry) return CUDA_SUCCESS;
  static DeviceOnce attr;
  if (attr.needed(h->device)) {
    CUCHOL_CHECK(cudaFuncSetAttribute(bpk::persistent_kernel<T>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                      (int)bpk::smem_bytes<T>()));
    CUCHOL_CHECK(cudaFuncSetAttribute(bpk::persistent_kernel<T>, cudaFuncAttributePreferredSharedMemoryCarveout, 100));
    attr.done(h->device);
  }
  CUCHOL_CHECK(cudaMemsetAsync(p->d_info, 0, sizeof(int) * B, s));
  CUCHOL_CHECK(cudaMemsetAsync(p->d_logdet, 0, sizeof(double) * B, s));
  CUCHOL_CHECK(cudaMemsetAsync(p->d_next, 0, sizeof(int), s));
  const int grid = persistent_grid(h, B);
  bpk::persistent_kernel<T><<<grid, bpk::THREADS, bpk::smem_bytes<T>(), s>>>(
      dm, dord, B, p->d_next, sh.upper ? 1 : 0, (sh.flags & 4) ? 1 : 0, static_cast<T*>(p->d_wp), p->wp_tiles);
  ++h->launches;
  CUCHOL_CHECK(cudaGetLastError());
  return CUDA_SUCCESS;
}

}  // namespace
