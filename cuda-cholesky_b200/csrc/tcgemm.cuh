// FP32 products on the TF32 tensor cores (tcgen05), real and complex, for ?trtri, ?lauum
// and ?potrf:
//
//     C(i, j) = beta C(i, j) + alpha * sum_k A(i, k) B(j, k)          alpha = +-1, beta = 0 or 1
//
// Operands are packed k-major ("packs"), every value x as hi = tf32(x) and lo =
// tf32(x - hi), x = hi + lo to 2^-22 |x|, and each k block issues lo hi^T + hi lo^T +
// hi hi^T (the dropped lo lo^T is below 2^-22 of the product).
//
// Accumulation.  The tensor core truncates when it adds to its FP32 accumulator, which
// biases long sums.  So an accumulator in tensor memory only runs over `chunk` k blocks of
// 32; eight epilogue warps then add it, rounded to nearest, to FP32 registers while the next
// ones run in the other accumulator.  That is blocked summation.  With one k block (four
// additions of the large products) its error is below that of one FMA chain per element at
// every order from tcg_min_order on, with two (twelve more) it is so for long sums only
// (kLongSum), and half of the reads of tensor memory, which the products share with the MMAs,
// go: strtri + slauum n = 16384 19.5 in place of 21 ms.
//
// Complex.  With a complex number stored as two adjacent k values, a complex product is
// a real one of twice the k: Re C = (ar, ai) . (br, -bi), Im C = (ar, ai) . (bi, br).
// So the A pack of an m x k complex view is m x 2k real, the B pack has two rows per
// row, 2j = (br, -bi) and 2j + 1 = (bi, br), and real columns 2j, 2j + 1 of the product
// are Re and Im of column j.  Conjugated views flip the sign of the stored imaginary
// part.  All of it is the packs' business: the kernel only knows real products.
//
// One CTA per 128 x 128 real tile: warp 8 streams operand tiles with TMA into a 3-stage
// ring, warp 9 issues the MMAs, warps 0..7 accumulate and write C.  Triangular operands
// are zero outside their triangle in the pack; k blocks that are zero for a whole tile
// are skipped.  What bounds it: operand traffic.  A k block of 32 moves 64 KB through L2
// and shared memory for 783 tensor cycles.
#pragma once
#include "tc.cuh"
#include "trsm.cuh"

namespace cuchol {
namespace tcg {

constexpr int BM = 128, BN = 128, BK = 32, STAGES = 3;
constexpr int TILE_BYTES = BM * BK * 4;                      // 16 KB: one operand part
constexpr int STAGE_BYTES = 4 * TILE_BYTES;                  // Ahi Alo Bhi Blo
constexpr int SMEM_BYTES = STAGES * STAGE_BYTES + 1024;
constexpr int EPI_WARPS = 8, EPI_COLS = 64;                  // epilogue warps, and real columns of each
constexpr int THREADS = 32 * (EPI_WARPS + 2);
constexpr int NACC = 2;                                      // accumulators (four: no faster)
constexpr int TMEM_COLS = NACC * BN;

enum : int { K_FULL = 0, K_A_LOWER = 1, K_LAUUM = 2, K_B_UPPER = 3 };

// A launch covers `nodes` equal problems (the last one with m_last rows and, for
// K_A_LOWER, k_last): node q uses pack rows from q * a_node and q * b_node and the
// output at c + q * c_node.  cx: real columns per column of C (2 for complex).
struct Params {
  int nodes, tiles_m, tiles_n;
  int m, m_last, n;             // rows, and real columns (cx * columns)
  int k, k_last;                // real k (a multiple of BK or zero-padded in the packs)
  int kmode, cx;
  int a_row0, b_row0, a_node, b_node, k0;   // k0: first k in the packs
  float* c;                     // output, in floats; element (i, col, part) at i*rs + col*cs + part;
                                // rs or cs is cx
  long long rs, cs, c_node;     // in floats
  int chunk;                    // k blocks per accumulator
  int beta, neg;                // C := (beta ? C : 0) + (neg ? -1 : 1) * acc
  int lower_only, real_diag;
  float *xhi, *xlo;             // if not null: the product goes here, split, as an A pack of row
  long long xld;                // pitch xld, from row q * a_node, instead of to C
  int* err;
};

// k range of the tile at rows i0.. and real columns j0.. (multiples of BK: tiles are 128
// wide and cx <= 2)
__device__ __forceinline__ void k_range(const Params& p, int i0, int j0, int k, int& kb, int& ke) {
  kb = 0;
  ke = k;
  if (p.kmode == K_A_LOWER) ke = min(ke, (i0 + BM) * p.cx);
  if (p.kmode == K_LAUUM) kb = i0 * p.cx;
  if (p.kmode == K_B_UPPER) kb = j0;
}

__global__ void __launch_bounds__(THREADS, 1)
    gemm_kernel(const __grid_constant__ CUtensorMap mahi, const __grid_constant__ CUtensorMap malo,
                const __grid_constant__ CUtensorMap mbhi, const __grid_constant__ CUtensorMap mblo, const Params p,
                const int* stop) {
  extern __shared__ uint8_t smem_raw[];
  __shared__ __align__(8) uint64_t full[STAGES], empty[STAGES], acc_full[NACC], acc_empty[NACC];
  __shared__ uint32_t tmem_slot;
  __shared__ int s_fail, s_issued, s_consumed;
  if (cta_aborted(stop)) return;

  // tile -> node, tile row, tile column; long k ranges first
  const int per = p.tiles_m * p.tiles_n;
  const int q = blockIdx.x / per, t = blockIdx.x - q * per;
  int ti, tj;
  if (p.kmode == K_B_UPPER) { tj = t / p.tiles_m; ti = t - tj * p.tiles_m; }
  else { ti = t / p.tiles_n; tj = t - ti * p.tiles_n; }
  if (p.kmode == K_A_LOWER) ti = p.tiles_m - 1 - ti;
  const int i0 = ti * BM, j0 = tj * BN;
  const bool last = q == p.nodes - 1;
  const int m = last ? p.m_last : p.m;
  if (i0 >= m) return;
  if (p.lower_only && j0 > (i0 + BM - 1) * p.cx + p.cx - 1) return;
  int kb, ke;
  k_range(p, i0, j0, last ? p.k_last : p.k, kb, ke);
  const int nkb = ke > kb ? (ke - kb + BK - 1) / BK : 0;
  const int nch = (nkb + p.chunk - 1) / p.chunk;

  uint8_t* base = smem_raw + ((1024u - (tc::smem_u32(smem_raw) & 1023u)) & 1023u);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (threadIdx.x == 0) {
    for (int s = 0; s < STAGES; ++s) {
      tc::mbar_init(&full[s], 1);
      tc::mbar_init(&empty[s], 1);
    }
    for (int b = 0; b < NACC; ++b) {
      tc::mbar_init(&acc_full[b], 1);
      tc::mbar_init(&acc_empty[b], EPI_WARPS);
    }
    s_fail = 0;
    s_issued = 0;
    s_consumed = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 0) tc::tmem_alloc(&tmem_slot, TMEM_COLS);
  tc::fence_before();
  __syncthreads();
  tc::fence_after();
  const uint32_t tmem = tmem_slot;

  if (warp == EPI_WARPS) {
    if (lane == 0) {                              // TMA producer
      const int ar = p.a_row0 + q * p.a_node + i0, br = p.b_row0 + q * p.b_node + j0;
      int kk = 0;
      for (; kk < nkb; ++kk) {
        const int s = kk % STAGES;
        if (kk >= STAGES && !tc::mbar_wait(&empty[s], ((kk / STAGES) & 1) ^ 1)) {
          s_fail = 1;
          break;
        }
        uint8_t* st = base + s * STAGE_BYTES;
        const int k = p.k0 + kb + kk * BK;
        tc::mbar_expect_tx(&full[s], STAGE_BYTES);
        tc::tma_load_2d(&mahi, &full[s], st, k, ar);
        tc::tma_load_2d(&malo, &full[s], st + TILE_BYTES, k, ar);
        tc::tma_load_2d(&mbhi, &full[s], st + 2 * TILE_BYTES, k, br);
        tc::tma_load_2d(&mblo, &full[s], st + 3 * TILE_BYTES, k, br);
      }
      s_issued = kk;
    }
  } else if (warp == EPI_WARPS + 1) {
    if (lane == 0) {                              // MMA issuer
      int kk = 0;
      bool ok = true;
      for (int c = 0; c < nch && ok; ++c) {
        const int b = c % NACC;
        if (c >= NACC && !tc::mbar_wait(&acc_empty[b], ((c / NACC) & 1) ^ 1)) ok = false;
        const uint32_t d = tmem + b * BN;
        for (int u = 0; u < p.chunk && kk < nkb && ok; ++u, ++kk) {
          const int s = kk % STAGES;
          if (!tc::mbar_wait(&full[s], (kk / STAGES) & 1)) {
            ok = false;
            break;
          }
          tc::fence_after();
          const uint32_t ah = tc::smem_u32(base + s * STAGE_BYTES), al = ah + TILE_BYTES, bh = al + TILE_BYTES,
                         bl = bh + TILE_BYTES;
          // the small products first: they meet a small accumulator
#pragma unroll
          for (int x = 0; x < BK * 4 / 32; ++x)
            tc::mma<float>(d, tc::smem_desc(al + 32 * x), tc::smem_desc(bh + 32 * x), (u | x) != 0 ? 1u : 0u);
#pragma unroll
          for (int x = 0; x < BK * 4 / 32; ++x) tc::mma<float>(d, tc::smem_desc(ah + 32 * x), tc::smem_desc(bl + 32 * x), 1u);
#pragma unroll
          for (int x = 0; x < BK * 4 / 32; ++x) tc::mma<float>(d, tc::smem_desc(ah + 32 * x), tc::smem_desc(bh + 32 * x), 1u);
          tc::mma_commit(&empty[s]);
        }
        tc::mma_commit(&acc_full[b]);
      }
      if (!ok) s_fail = 1;
      s_consumed = kk;
    }
  } else {
    // epilogue warps: 32 tile rows each (a row per lane), and half of their real columns in
    // registers
    const int wrow = 32 * (warp & 3), wcol = EPI_COLS * (warp >> 2);
    float acc[EPI_COLS];
#pragma unroll
    for (int j = 0; j < EPI_COLS; ++j) acc[j] = 0.f;
    bool ok = true;
#pragma unroll 1
    for (int c = 0; c < nch; ++c) {
      const int b = c % NACC;
      if (!tc::mbar_wait(&acc_full[b], (c / NACC) & 1)) {
        ok = false;
        break;
      }
      tc::fence_after();
      const uint32_t src = tmem + b * BN + wcol + ((uint32_t)wrow << 16);
#pragma unroll
      for (int g = 0; g < EPI_COLS / 32; ++g) {
        float v[32];
        tc::tmem_ld32(src + 32 * g, v);
#pragma unroll
        for (int j = 0; j < 32; ++j) acc[32 * g + j] += v[j];
      }
      tc::fence_before();
      __syncwarp();
      if (lane == 0) asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(tc::smem_u32(&acc_empty[b])) : "memory");
    }
    if (!ok) s_fail = 1;
    if (ok) {
      // The ring is idle now (every MMA has read its operands): the rows go through it, so
      // that the output loops are rolled, coalesced in either storage, and short.  Straight
      // code over 128 registers, with C read into them first, was bound by instruction
      // fetch: 26 us for a launch of one wave with k = 128.
      float* st = reinterpret_cast<float*>(base) + warp * (EPI_COLS * 33);     // st[col * 33 + row]
#pragma unroll
      for (int j = 0; j < EPI_COLS; ++j) st[j * 33 + lane] = p.neg ? -acc[j] : acc[j];
      __syncwarp();
      const int r0 = i0 + wrow, rows = min(32, m - r0), c0 = j0 + wcol, cols = min(EPI_COLS, p.n - c0);
      float* cq = p.c + (long long)q * p.c_node;
      // C(r, col) in floats: += (no load to wait for; one CTA owns the element) or =
      auto put = [&](float* o, float v) {
        if (p.beta) atomicAdd(o, v);
        else *o = v;
      };
      // (re, im) of a complex element, in one 8-byte access: as two of 4 bytes cpotrf n = 8192
      // took 8.9 ms, not 7.5
      auto put2 = [&](float* o, float re, float im, bool diag) {
        const bool real = p.real_diag && diag;
        if (p.beta) {
          asm volatile("red.global.add.v2.f32 [%0], {%1, %2};" ::"l"(o), "f"(re), "f"(real ? 0.f : im) : "memory");
          if (real) o[1] = 0.f;
        } else {
          *reinterpret_cast<float2*>(o) = make_float2(re, real ? 0.f : im);
        }
      };
      auto keep = [&](int r, int col) { return !p.lower_only || r * p.cx + p.cx - 1 >= col; };
      if (p.xhi != nullptr) {
#pragma unroll 2
        for (int r = 0; r < rows; ++r) {
          const long long o = (long long)(q * p.a_node + r0 + r) * p.xld + c0;
#pragma unroll
          for (int u = 0; u < EPI_COLS / 32; ++u) {
            const int c = lane + 32 * u;
            if (c < cols) {
              const float x = st[c * 33 + r], h = round_tf32(x);
              p.xhi[o + c] = h;
              p.xlo[o + c] = round_tf32(x - h);
            }
          }
        }
      } else if (p.rs == p.cx && p.cx == 1) {       // rows contiguous
        float* o = cq + r0 + lane + (long long)c0 * p.cs;
        const int r = r0 + lane;
#pragma unroll 4
        for (int c = 0; c < cols; ++c, o += p.cs)
          if (lane < rows && keep(r, c0 + c)) put(o, st[c * 33 + lane]);
      } else if (p.rs == p.cx) {                    // complex, rows contiguous: a row per lane
        const int r = r0 + lane;
        float* o = cq + r * p.rs + (long long)(c0 >> 1) * p.cs;
#pragma unroll 4
        for (int c = 0; c < cols; c += 2, o += p.cs)
          if (lane < rows && keep(r, c0 + c)) put2(o, st[c * 33 + lane], st[(c + 1) * 33 + lane], r == ((c0 + c) >> 1));
      } else if (p.cx == 2) {                       // complex, columns contiguous: a column per lane
#pragma unroll 2
        for (int r = 0; r < rows; ++r) {
          float* o = cq + (r0 + r) * p.rs + c0;
#pragma unroll
          for (int u = 0; u < EPI_COLS / 64; ++u) {
            const int c = 2 * lane + 64 * u, col = c0 + c;
            if (c < cols && keep(r0 + r, col)) put2(o + c, st[c * 33 + r], st[(c + 1) * 33 + r], r0 + r == (col >> 1));
          }
        }
      } else {                                      // columns contiguous
#pragma unroll 2
        for (int r = 0; r < rows; ++r) {
          float* o = cq + (r0 + r) * p.rs + c0;
#pragma unroll
          for (int u = 0; u < EPI_COLS / 32; ++u) {
            const int c = lane + 32 * u;
            if (c < cols && keep(r0 + r, c0 + c)) put(o + c, st[c * 33 + r]);
          }
        }
      }
    }
  }
  __syncthreads();
  if (s_fail != 0 && threadIdx.x == 0) {
    // a wait gave up: record it, and let the loads still in flight land before the CTA exits
    atomicExch(p.err, 1);
    for (int kk = s_consumed; kk < s_issued; ++kk) tc::mbar_wait(&full[kk % STAGES], (kk / STAGES) & 1);
  }
  tc::fence_before();
  __syncthreads();
  if (warp == 0) {
    tc::fence_after();
    tc::tmem_dealloc(tmem, TMEM_COLS);
  }
}

// ---- packs -------------------------------------------------------------------------

// One launch packs the views of all nodes of a level: for node q and row i < rows (the
// last node: rows_last), pack row q * node_rows + i (complex B packs: 2 rows per row)
// holds the view's elements v(i, k), k < kk, at [row * ld + k * cx], zero from kk to the
// next multiple of BK and outside the triangle.  View: src + q * src_node + i*rs + k*cs.
struct Pack {
  const float* src;             // in floats
  long long rs, cs, src_node;   // in floats
  int nodes, rows, rows_last, kk, kk_last, node_rows;
  int tri;                      // TRI_NONE, TRI_LOWER (k <= i), TRI_UPPER (k >= i)
  int unit;                     // the diagonal is 1
  int cx, conj, two;            // complex: conjugate; two: the B form with two rows per row
  float *hi, *lo;
  long long ld;
};

__device__ __forceinline__ void split_store(float* hi, float* lo, long long o, float x) {
  const float h = round_tf32(x);
  hi[o] = h;
  lo[o] = round_tf32(x - h);
}

struct Packs { int count; Pack p[3]; };

// 32 x 32 elements per CTA, through shared memory so that both sides are coalesced.
// blockIdx: x = k block, y = row block, z = node * count + pack.
__global__ void __launch_bounds__(256) pack_kernel(const __grid_constant__ Packs ps) {
  const Pack& p = ps.p[blockIdx.z % ps.count];
  const int q = blockIdx.z / ps.count, i0 = blockIdx.y * 32, k0 = blockIdx.x * 32;
  if (q >= p.nodes) return;
  const bool last = q == p.nodes - 1;
  const int rows = last ? p.rows_last : p.rows, kk = last ? p.kk_last : p.kk;
  const int kpad = (kk * p.cx + BK - 1) / BK * BK / p.cx;      // zero-filled up to here
  if (i0 >= rows || k0 >= kpad) return;
  // blocks the products never read: they skip k blocks that are zero for a 128-row tile
  if (p.tri == 1 && k0 >= (i0 | 127) + 1) return;
  if (p.tri == 2 && k0 + 31 < (i0 & ~127)) return;
  __shared__ float2 s[32][33];
  const int tx = threadIdx.x & 31, ty = threadIdx.x >> 5;
  const float* src = p.src + (long long)q * p.src_node;
  const bool rows_fast = p.rs == p.cx;
#pragma unroll
  for (int u = 0; u < 4; ++u) {
    const int a = rows_fast ? tx : ty + 8 * u, b = rows_fast ? ty + 8 * u : tx;   // row, k in the block
    const int i = i0 + a, k = k0 + b;
    float2 v = make_float2(0.f, 0.f);
    if (i < rows && k < kk && (p.tri == 0 || (p.tri == 1 ? k <= i : k >= i))) {
      if (p.unit && i == k) {
        v.x = 1.f;
      } else {
        const float* e = src + (long long)i * p.rs + (long long)k * p.cs;
        v.x = e[0];
        if (p.cx == 2) v.y = p.conj ? -e[1] : e[1];
      }
    }
    s[a][b] = v;
  }
  __syncthreads();
#pragma unroll
  for (int u = 0; u < 4; ++u) {
    const int a = ty + 8 * u, i = i0 + a, k = k0 + tx;
    if (i >= rows || k >= kpad) continue;
    const float2 v = s[a][tx];
    if (p.cx == 1) {
      split_store(p.hi, p.lo, (long long)(q * p.node_rows + i) * p.ld + k, v.x);
    } else {
      const long long row = (long long)(q * p.node_rows + i) * (p.two ? 2 : 1);
      const long long o = row * p.ld + 2 * k;
      split_store(p.hi, p.lo, o, v.x);
      split_store(p.hi, p.lo, o + 1, p.two ? -v.y : v.y);
      if (p.two) {
        split_store(p.hi, p.lo, o + p.ld, v.y);
        split_store(p.hi, p.lo, o + p.ld + 1, v.x);
      }
    }
  }
}

// *bad := 1 when an entry of the lower triangle (view strides in floats; unit: without
// the diagonal) is not finite or above 2^62, or a diagonal entry below 2^-62.  One CTA
// per 64 x 64 block, blocks above the diagonal exit.
__global__ void __launch_bounds__(256) range_kernel(const float* __restrict__ a, long long rs, long long cs, int n, int cx,
                                                    int unit, int* bad) {
  const int i0 = blockIdx.x * 64, j0 = blockIdx.y * 64;
  if (j0 > i0 + 63) return;
  bool ok = true;
  for (int e = threadIdx.x; e < 64 * 64; e += 256) {
    const int i = i0 + (rs == cx ? (e & 63) : (e >> 6)), j = j0 + (rs == cx ? (e >> 6) : (e & 63));
    if (i >= n || j > i || (unit && i == j)) continue;
    const float* x = a + (long long)i * rs + (long long)j * cs;
    float m = fabsf(x[0]);
    ok = ok && m <= 0x1p62f;                     // false for NaN too
    if (cx == 2) {
      const float im = fabsf(x[1]);
      ok = ok && im <= 0x1p62f;
      m = fmaxf(m, im);
    }
    if (i == j) ok = ok && m >= 0x1p-62f;
  }
  if (!ok) atomicExch(bad, 1);
}

// Range of ?potrf's split products, read off the diagonal of A: |l_ij|^2 <= a_ii, so in a
// factorization that succeeds
//   no value overflows while a_ii <= 2^126;
//   what the hi lo products and the FP32 output drop below 2^-126 is at most 2^-126 per product,
//   which for fewer than 2^20 of them stays under the FP32 rounding 2^-24 sqrt(a_ii a_jj)
//   while a_ii >= 2^-80.
// Entries that are not positive end the factorization at their column or before, whatever
// the products of their rows are.
constexpr float kDiagMin = 0x1p-80f, kDiagMax = 0x1p126f;
__host__ __device__ inline bool diag_in_range(float d) { return !(d > 0.f) || (d >= kDiagMin && d <= kDiagMax); }

// Starts a factorization's words: info := 0, or kOutOfRange (which the kernels that follow take
// for a failure, so they leave A as it is), and log det := 0.  One CTA.
constexpr int kOutOfRange = -1;
__global__ void __launch_bounds__(1024) diag_range_kernel(const float* __restrict__ a, long long stride, int n,
                                                          int* __restrict__ info, double* __restrict__ logdet) {
  bool bad = false;
#pragma unroll 8
  for (int i = threadIdx.x; i < n; i += 1024) bad |= !diag_in_range(a[i * stride]);
  const int any = __syncthreads_or(bad);
  if (threadIdx.x == 0) {
    *info = any ? kOutOfRange : 0;
    *logdet = 0.0;
  }
}

}  // namespace tcg
}  // namespace cuchol
