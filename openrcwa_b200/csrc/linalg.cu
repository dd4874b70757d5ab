// Batched complex-FP64 GEMM, LU (getrf) and LU solve (getrs).
//
// GEMM: the pipelined tile product of tile_pipe.cuh, 64x64 output tiles by four
// warps.  The trailing updates of the one-CTA-per-matrix blocked LU and of the
// blocked triangular solves use the tile routine of tile.cuh.
#include <algorithm>
#include <atomic>
#include <map>
#include <mutex>

#include <cooperative_groups.h>

#include "linalg.cuh"
#include "lu_blocked.cuh"
#include "tile.cuh"
#include "tile_pipe.cuh"

namespace {

// Output tiles of 64 x 64 by four warps of 32 x 32, two CTAs per SM; slabs of
// 8 along K in four stages (98,816 bytes).  Bound by the FP64 tensor pipe: per K-step of
// 4 a warp's 32 x 32 share issues 64 DMMAs (16 cycles each on its quarter of the
// SM) for eight 16-byte shared loads, and the cp.async stages take the global
// loads off its path.  The
// routine of tile.cuh, whose 16 x 32 share per warp waits for two barriers and
// a register-to-shared transpose per slab, reached half of the pipe: on B200
// (DMMA peak measured 36.4 TFLOP/s) 29 x 882^3 8.49 -> 5.00 ms (31.8 TFLOP/s),
// 148 x 450^3 7.54 -> 3.94 ms (27.4), 200 x 98^3 0.191 -> 0.101 ms (15.0),
// 1 x 1250^3 0.86 -> 0.59 ms (26.7), bitwise the same results.
using GemmTile = PipeTile<2, 2, 4, 4, 8, 4>;

template <bool TA, bool TB, bool kScale>
__global__ void __launch_bounds__(GemmTile::T, 2) zgemm_kernel(GemmArgs g) {
  extern __shared__ __align__(16) unsigned char gemm_smem[];
  const int b = blockIdx.z;
  const cplx* A = (g.A ? g.A[b] : g.A0 + b * g.sA) + g.offA;
  const cplx* B = (g.B ? g.B[b] : g.B0 + b * g.sB) + g.offB;
  const cplx* s = kScale ? g.s[b] : nullptr;
  const int m0 = blockIdx.y * GemmTile::BM, n0 = blockIdx.x * GemmTile::BN;
  const int K = g.triB ? min(g.K, n0 + GemmTile::BN) : g.K;
  double re[GemmTile::RT][GemmTile::CT][2], im[GemmTile::RT][GemmTile::CT][2];
  pipe_mma<GemmTile, TA, TB, kScale>(reinterpret_cast<cplx*>(gemm_smem), re, im, A, g.lda, B, g.ldb, s, g.M, g.N, K,
                                     m0, n0);
  const cplx* C = (g.beta.x != 0.0 || g.beta.y != 0.0) ? g.C[b] + g.offC : nullptr;
  pipe_store<GemmTile>(re, im, (g.D ? g.D[b] : g.D0 + b * g.sD) + g.offD, g.ldd, C, g.ldc, g.alpha, g.beta, g.gammaI,
                       g.M, g.N, m0, n0);
}

template <bool TA, bool TB, bool kScale>
cudaError_t zgemm_launch(const GemmArgs& g, cudaStream_t st) {
  static SmemAttrOnce attr;
  cudaError_t e = attr.ensure(zgemm_kernel<TA, TB, kScale>, (int)GemmTile::kSmem);
  if (e != cudaSuccess) return e;
  const dim3 grid((g.N + GemmTile::BN - 1) / GemmTile::BN, (g.M + GemmTile::BM - 1) / GemmTile::BM, g.batch);
  zgemm_kernel<TA, TB, kScale><<<grid, GemmTile::T, GemmTile::kSmem, st>>>(g);
  ++launch_counter();
  return cudaGetLastError();
}

template <bool TA, bool TB>
cudaError_t zgemm_launch(const GemmArgs& g, cudaStream_t st) {
  return g.s ? zgemm_launch<TA, TB, true>(g, st) : zgemm_launch<TA, TB, false>(g, st);
}

// Factorise panel columns kb .. kb+jb-1 of the n x n matrix A in place (rows
// kb .. n-1), LAPACK getf2 order: pivot = largest |re|+|im| in the column
// (first index on ties), the pivot rows are interchanged across all n columns,
// the column is scaled by the reciprocal pivot and the rest of the panel gets
// the rank-1 update.  The update reads the pivot row from shared memory and
// issues the loads of eight elements before their stores, so a thread keeps
// eight L2 requests in flight instead of one; it also tracks the largest
// entry of the next column, which is that column's pivot search.  Whole CTA;
// info keeps the first exactly-zero pivot.
__device__ void lu_panel(cplx* A, int n, int lda, int kb, int jb, int* ipiv, int& info, double* red_v, int* red_i,
                         int* s_piv, cplx* prow) {
  const int tid = threadIdx.x, nthr = blockDim.x;
  constexpr int kU = 8;
  double best = -1.0;
  int bi = kb;
  for (int i0 = kb + tid; i0 < n; i0 += kU * nthr) {
    double v[kU];
#pragma unroll
    for (int q = 0; q < kU; ++q) {
      const int i = i0 + q * nthr;
      v[q] = i < n ? cabs1(A[(size_t)i * lda + kb]) : -1.0;
    }
#pragma unroll
    for (int q = 0; q < kU; ++q)
      if (v[q] > best) { best = v[q]; bi = i0 + q * nthr; }
  }
  const int ce = kb + jb;  // panel end (exclusive)
  for (int j = kb; j < ce; ++j) {
    for (int off = 16; off > 0; off >>= 1) {
      const double ov = __shfl_down_sync(0xffffffffu, best, off);
      const int oi = __shfl_down_sync(0xffffffffu, bi, off);
      if (ov > best || (ov == best && oi < bi)) { best = ov; bi = oi; }
    }
    if ((tid & 31) == 0) { red_v[tid >> 5] = best; red_i[tid >> 5] = bi; }
    __syncthreads();
    if (tid == 0) {
      double bv = red_v[0];
      int bix = red_i[0];
      for (int w = 1; w < nthr / 32; ++w)
        if (red_v[w] > bv || (red_v[w] == bv && red_i[w] < bix)) { bv = red_v[w]; bix = red_i[w]; }
      *s_piv = bix;
      ipiv[j] = bix;
    }
    __syncthreads();
    const int p = *s_piv;
    if (p != j) {
      for (int c = tid; c < n; c += nthr) {
        cplx t = A[(size_t)j * lda + c];
        A[(size_t)j * lda + c] = A[(size_t)p * lda + c];
        A[(size_t)p * lda + c] = t;
      }
    }
    __syncthreads();
    for (int c = j + tid; c < ce; c += nthr) prow[c - kb] = A[(size_t)j * lda + c];
    __syncthreads();
    const cplx piv = prow[j - kb];
    if (piv.x == 0.0 && piv.y == 0.0) {
      if (info == 0) info = j + 1;
    } else {
      const cplx inv = cdiv(mkc(1.0, 0.0), piv);
      for (int i0 = j + 1 + tid; i0 < n; i0 += kU * nthr) {
        cplx v[kU];
#pragma unroll
        for (int q = 0; q < kU; ++q) {
          const int i = i0 + q * nthr;
          if (i < n) v[q] = A[(size_t)i * lda + j];
        }
#pragma unroll
        for (int q = 0; q < kU; ++q) {
          const int i = i0 + q * nthr;
          if (i < n) A[(size_t)i * lda + j] = cmul(v[q], inv);
        }
      }
    }
    __syncthreads();
    best = -1.0;
    bi = j + 1;
    const int w = ce - j - 1;
    if (w > 0) {
      const int total = (n - j - 1) * w;
      for (int base = tid; base < total; base += kU * nthr) {
        cplx l[kU], a[kU];
#pragma unroll
        for (int q = 0; q < kU; ++q) {
          const int idx = base + q * nthr;
          if (idx < total) {
            const int i = j + 1 + idx / w, c = j + 1 + idx % w;
            l[q] = A[(size_t)i * lda + j];
            a[q] = A[(size_t)i * lda + c];
          }
        }
#pragma unroll
        for (int q = 0; q < kU; ++q) {
          const int idx = base + q * nthr;
          if (idx < total) {
            const int i = j + 1 + idx / w, c = j + 1 + idx % w;
            const cplx v = cfma(cneg(l[q]), prow[c - kb], a[q]);
            A[(size_t)i * lda + c] = v;
            if (c == j + 1) {
              const double av = cabs1(v);
              if (av > best) { best = av; bi = i; }
            }
          }
        }
      }
    }
    __syncthreads();
  }
}

// U12(:, c) = L11^-1 A12(:, c) for columns c = c0 + tid (L11 unit lower,
// jb x jb at (kb, kb), staged in Lsm); threads with c >= n idle.
__device__ void lu_trsm_cols(cplx* A, int n, int lda, int kb, int jb, int c, cplx (*Lsm)[33]) {
  if (c >= n) return;
  for (int r = 1; r < jb; ++r) {
    cplx x = A[(size_t)(kb + r) * lda + c];
    for (int q = 0; q < r; ++q) x = cfma(cneg(Lsm[r][q]), A[(size_t)(kb + q) * lda + c], x);
    A[(size_t)(kb + r) * lda + c] = x;
  }
}

// One CTA per matrix: right-looking blocked LU, panel width 32; the U12 block
// row by a shared-memory triangular solve and the trailing matrix by the
// register-blocked tile GEMM.
__global__ void __launch_bounds__(kTileThreads) zgetrf_kernel(cplx* const* Aarr, int n, int lda,
                                                             int* ipiv_all, int* info_all) {
  // the triangular block and the GEMM slabs are used in separate phases
  __shared__ __align__(16) unsigned char smem_raw[sizeof(TileSmem)];
  TileSmem& sm = *reinterpret_cast<TileSmem*>(smem_raw);
  cplx (*Lsm)[33] = reinterpret_cast<cplx (*)[33]>(smem_raw);
  __shared__ double red_v[kTileThreads / 32];
  __shared__ int red_i[kTileThreads / 32];
  __shared__ int s_piv;
  __shared__ cplx prow[32];
  const int tid = threadIdx.x;
  const int b = blockIdx.x;
  cplx* A = Aarr[b];
  int* ipiv = ipiv_all + (size_t)b * n;
  int info = 0;
  for (int kb = 0; kb < n; kb += 32) {
    const int jb = min(32, n - kb);
    lu_panel(A, n, lda, kb, jb, ipiv, info, red_v, red_i, &s_piv, prow);
    if (kb + jb < n) {
      for (int idx = tid; idx < jb * jb; idx += kTileThreads) {
        const int r = idx / jb, q = idx % jb;
        Lsm[r][q] = A[(size_t)(kb + r) * lda + kb + q];
      }
      __syncthreads();
      for (int c = kb + jb + tid; c < n; c += kTileThreads) lu_trsm_cols(A, n, lda, kb, jb, c, Lsm);
      __syncthreads();
      const int m2 = n - kb - jb;
      const int tiles_m = (m2 + kTBM - 1) / kTBM, tiles_n = (m2 + kTBN - 1) / kTBN;
      const cplx* L21 = A + (size_t)(kb + jb) * lda + kb;
      const cplx* U12 = A + (size_t)kb * lda + kb + jb;
      cplx* A22 = A + (size_t)(kb + jb) * lda + kb + jb;
      for (int t = 0; t < tiles_m * tiles_n; ++t) {
        const int tm = (t / tiles_n) * kTBM, tn = (t % tiles_n) * kTBN;
        cplx acc[4][4];
        tile_zero(acc);
        tile_mma<false, false>(sm, acc, L21, lda, U12, lda, nullptr, m2, m2, jb, tm, tn);
        tile_store(acc, A22, lda, A22, lda, mkc(-1.0, 0.0), mkc(1.0, 0.0), mkc(0.0, 0.0), m2, m2, tm, tn);
      }
      __syncthreads();
    }
  }
  if (tid == 0) info_all[b] = info;
}

// ---- panel-by-panel LU ------------------------------------------------------
// A panel is kRegW columns wide and lives in registers: one thread holds one
// row's kRegW entries, so a rank-1 update is FP64 instructions only and the
// panel crosses memory once.  Up to kRegT rows fit one CTA (128 registers a
// thread); a taller panel is shared by a thread-block cluster of up to 8 CTAs
// (n <= 4096), which exchange their pivot candidates and candidate rows
// through distributed shared memory.  Bound by the latency of a column:
// the warps' arg-max (three redux steps), two barriers, the reciprocal and the
// update.  Whole factorisations (schedule 2) against 32-column panels updated
// in L2, B200: 58 x 882 16.4 -> 8.9 ms, 46 x 494 5.3 -> 2.6 ms, 148 x 450 6.1 ->
// 4.2 ms, 2 x 1250 12.3 -> 6.2 ms (5.1 in schedule 1).  Same pivot rule and the
// same operations per entry as lu_panel, so the panel's factors are the same for
// every cluster size.
constexpr int kRegW = 16;
constexpr int kRegT = 512;
constexpr int kRegMaxRows = 8 * kRegT;

// arg-max over a warp of (key, smallest row): keys are the bits of
// non-negative doubles, which order like integers; NaN maps to 0, so that it
// never wins against a number.  Every lane gets the result.
__device__ __forceinline__ void warp_argmax(unsigned long long& key, int& row) {
  const unsigned hi = (unsigned)(key >> 32), mh = __reduce_max_sync(0xffffffffu, hi);
  const unsigned lo = hi == mh ? (unsigned)key : 0u, ml = __reduce_max_sync(0xffffffffu, lo);
  row = __reduce_min_sync(0xffffffffu, hi == mh && lo == ml ? row : 0x7fffffff);
  key = ((unsigned long long)mh << 32) | ml;
}

__global__ void __launch_bounds__(kRegT) getrf_regpanel_kernel(cplx* const* Aarr, int n, int lda, int kb, int jb,
                                                              int* ipiv_all, int* info_all) {
  namespace cg = cooperative_groups;
  cg::cluster_group cl = cg::this_cluster();
  // slots alternate between columns, so that a column's values are overwritten
  // only after a barrier that follows their last read
  __shared__ unsigned long long s_key[2][kRegT / 32];
  __shared__ int s_row[2][kRegT / 32];
  __shared__ unsigned long long s_ckey[2];
  __shared__ int s_crow[2];
  __shared__ cplx s_cand[2][kRegW], s_jrow[2][kRegW];  // this CTA's candidate row; row j, in its owner's CTA
  __shared__ cplx s_p[2][kRegW], s_j[2][kRegW];        // the pivot row and row j
  const int C = (int)cl.num_blocks(), rank = (int)cl.block_rank();
  const int tid = threadIdx.x, lane = tid & 31, nw = blockDim.x >> 5;
  const int b = blockIdx.x / C;
  cplx* A = Aarr[b];
  int* ipiv = ipiv_all + (size_t)b * n;
  int info = kb == 0 ? 0 : info_all[b];
  const int i = kb + rank * (int)blockDim.x + tid;  // this thread's row
  const bool in = i < n;
  cplx a[kRegW];
  cplx* const Ai = A + (size_t)i * lda + kb;
#pragma unroll
  for (int c = 0; c < kRegW; ++c) a[c] = in && c < jb ? Ai[c] : mkc(0.0, 0.0);
#pragma unroll
  for (int jj = 0; jj < kRegW; ++jj) {
    if (jj >= jb) break;
    const int j = kb + jj, bf = jj & 1;
    const bool act = in && i >= j;
    const double v = act ? cabs1(a[jj]) : 0.0;
    unsigned long long key = v == v ? (unsigned long long)__double_as_longlong(v) : 0ull;
    int row = act ? i : 0x7fffffff;
    if (!act) key = 0ull;
    warp_argmax(key, row);
    if (lane == 0) { s_key[bf][tid >> 5] = key; s_row[bf][tid >> 5] = row; }
    if (i == j) {
#pragma unroll
      for (int c = 0; c < kRegW; ++c) s_jrow[bf][c] = a[c];
    }
    __syncthreads();
    key = lane < nw ? s_key[bf][lane] : 0ull;
    row = lane < nw ? s_row[bf][lane] : 0x7fffffff;
    warp_argmax(key, row);
    const cplx *prow = s_cand[bf], *jrow = s_jrow[bf];
    if (i == row) {
#pragma unroll
      for (int c = 0; c < kRegW; ++c) s_cand[bf][c] = a[c];
    }
    if (C > 1) {
      if (tid == 0) { s_ckey[bf] = key; s_crow[bf] = row; }
      cl.sync();
      if (tid < 32) {
        key = lane < C ? *cl.map_shared_rank(&s_ckey[bf], lane) : 0ull;
        row = lane < C ? *cl.map_shared_rank(&s_crow[bf], lane) : 0x7fffffff;
        warp_argmax(key, row);
        // row >= j always: row j itself is a candidate
        const int owner = (row - kb) / (int)blockDim.x, jowner = jj / (int)blockDim.x;
        if (lane < kRegW) s_p[bf][lane] = *cl.map_shared_rank(&s_cand[bf][lane], owner);
        else s_j[bf][lane - kRegW] = *cl.map_shared_rank(&s_jrow[bf][lane - kRegW], jowner);
        if (lane == 0) s_crow[bf ^ 1] = row;  // read below, rewritten after the next column's barrier
      }
      prow = s_p[bf];
      jrow = s_j[bf];
    }
    __syncthreads();
    const int p = C > 1 ? s_crow[bf ^ 1] : row;
    if (rank == 0 && tid == 0) ipiv[j] = p;
    if (p != j) {
      if (i == p) {
#pragma unroll
        for (int c = 0; c < kRegW; ++c) a[c] = jrow[c];
      } else if (i == j) {
#pragma unroll
        for (int c = 0; c < kRegW; ++c) a[c] = prow[c];
      }
    }
    const cplx piv = prow[jj];
    cplx inv = mkc(1.0, 0.0);
    if (piv.x == 0.0 && piv.y == 0.0) {
      if (info == 0) info = j + 1;
    } else {
      inv = cdiv(mkc(1.0, 0.0), piv);
    }
    if (in && i > j) {
      const cplx l = piv.x == 0.0 && piv.y == 0.0 ? a[jj] : cmul(a[jj], inv);
      a[jj] = l;
#pragma unroll
      for (int c = jj + 1; c < kRegW; ++c) a[c] = cfma(cneg(l), prow[c], a[c]);
    }
  }
  if (in) {
#pragma unroll
    for (int c = 0; c < kRegW; ++c)
      if (c < jb) Ai[c] = a[c];
  }
  if (rank == 0 && tid == 0) info_all[b] = info;
  // no CTA leaves while another may still read its candidate
  if (C > 1) cl.sync();
}

// Matrices of at most kSmallLuMax rows: the whole matrix in shared memory, one
// CTA each, right-looking column by column.  Every warp finds the pivot itself
// (the same data, no exchange), so a column costs two barriers; bound by their
// latency and the reciprocal.  Same pivot rule as lu_panel.
// B200, against lu_panel in global memory: 400 x 98 2.27 -> 0.98 ms, 303 x 82
// 1.64 -> 0.49 ms, one 50-row matrix 0.15 -> 0.06 ms.
constexpr int kSmallLuMax = 116;
constexpr int kSmallLuThreads = 256;
__host__ __device__ constexpr size_t small_lu_smem(int n) { return sizeof(cplx) * (size_t)n * (n | 1); }

__global__ void __launch_bounds__(kSmallLuThreads) getrf_small_kernel(cplx* const* Aarr, int n, int lda, int* ipiv_all,
                                                                     int* info_all) {
  extern __shared__ __align__(16) unsigned char small_smem[];
  constexpr int Q = (kSmallLuMax + 31) / 32;
  cplx* const S = reinterpret_cast<cplx*>(small_smem);
  const int ld = n | 1, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, nw = kSmallLuThreads / 32;
  cplx* const A = Aarr[blockIdx.x];
  int* const ipiv = ipiv_all + (size_t)blockIdx.x * n;
  int info = 0;
  for (int idx = tid; idx < n * n; idx += kSmallLuThreads) S[(idx / n) * ld + idx % n] = A[(size_t)(idx / n) * lda + idx % n];
  __syncthreads();
  for (int j = 0; j < n; ++j) {
    unsigned long long key = 0ull;
    int row = 0x7fffffff;
#pragma unroll
    for (int q = 0; q < Q; ++q) {
      const int i = j + lane + 32 * q;
      if (i < n) {
        const double v = cabs1(S[i * ld + j]);
        const unsigned long long k = v == v ? (unsigned long long)__double_as_longlong(v) : 0ull;
        if (k > key || row == 0x7fffffff) { key = k; row = i; }
      }
    }
    warp_argmax(key, row);
    const int p = row;
    if (tid == 0) ipiv[j] = p;
    __syncthreads();  // every warp has read the column
    if (p != j)
      for (int c = tid; c < n; c += kSmallLuThreads) {
        const cplx t = S[j * ld + c];
        S[j * ld + c] = S[p * ld + c];
        S[p * ld + c] = t;
      }
    __syncthreads();
    const cplx piv = S[j * ld + j];
    const bool zero = piv.x == 0.0 && piv.y == 0.0;
    if (zero && info == 0) info = j + 1;
    const cplx inv = zero ? mkc(1.0, 0.0) : cdiv(mkc(1.0, 0.0), piv);
    cplx pr[Q];
#pragma unroll
    for (int q = 0; q < Q; ++q) {
      const int c = j + 1 + lane + 32 * q;
      pr[q] = c < n ? S[j * ld + c] : mkc(0.0, 0.0);
    }
#pragma unroll 2
    for (int i = j + 1 + warp; i < n; i += nw) {
      const cplx l = cmul(S[i * ld + j], inv);
      __syncwarp();
      if (lane == 0) S[i * ld + j] = l;
#pragma unroll
      for (int q = 0; q < Q; ++q) {
        const int c = j + 1 + lane + 32 * q;
        if (c < n) S[i * ld + c] = cfma(cneg(l), pr[q], S[i * ld + c]);
      }
    }
    __syncthreads();
  }
  for (int idx = tid; idx < n * n; idx += kSmallLuThreads) A[(size_t)(idx / n) * lda + idx % n] = S[(idx / n) * ld + idx % n];
  if (tid == 0) info_all[blockIdx.x] = info;
}

// After a register panel: its row interchanges on every column outside the
// panel, and U12 = L11^-1 A12 on the columns kb+jb .. ce-1.  One thread per
// column: the interchanges are folded into one permutation of the (at most 2
// kRegW) rows they touch, so that a column's loads are all in flight at once.
__global__ void __launch_bounds__(128) getrf_swap_trsm_kernel(cplx* const* Aarr, int n, int lda, int kb, int jb, int ce,
                                                              const int* ipiv_all) {
  __shared__ int s_dst[2 * kRegW], s_src[2 * kRegW];
  __shared__ cplx L[kRegW][kRegW + 1];
  const int b = blockIdx.y, tid = threadIdx.x;
  cplx* A = Aarr[b];
  if (tid < 32) {
    // lane q < kRegW: row kb + q; lane kRegW + q: the q-th pivot row, when it
    // lies below the panel's own rows and no earlier lane has it
    const int* ipiv = ipiv_all + (size_t)b * n + kb;
    const int q0 = tid & (kRegW - 1);
    const int p = q0 < jb ? ipiv[q0] : -1;
    int at = tid < kRegW ? kb + tid : (p >= kb + kRegW ? p : -1);
    for (int q = 0; q < kRegW - 1; ++q) {
      const int o = __shfl_sync(0xffffffffu, at, kRegW + q);
      if (tid > kRegW + q && at == o) at = -1;
    }
    int src = at;  // the row whose values end up at row `at`
    for (int q = 0; q < jb; ++q) {
      const int pq = __shfl_sync(0xffffffffu, p, q);
      const unsigned m = __ballot_sync(0xffffffffu, at == pq);
      const int lp = __ffs(m) - 1;
      const int sq = __shfl_sync(0xffffffffu, src, q), sp = __shfl_sync(0xffffffffu, src, lp);
      if (tid == q) src = sp;
      if (tid == lp) src = sq;
    }
    s_dst[tid] = at == src ? -1 : at;
    s_src[tid] = at == src ? -1 : src;
  }
  for (int idx = tid; idx < kRegW * kRegW; idx += blockDim.x) {
    const int r = idx / kRegW, q = idx % kRegW;
    L[r][q] = r < jb && q < r ? A[(size_t)(kb + r) * lda + kb + q] : mkc(0.0, 0.0);
  }
  __syncthreads();
  int c = blockIdx.x * blockDim.x + tid;
  if (c >= n - jb) return;
  if (c >= kb) c += jb;  // the panel's own columns are already permuted
  const bool solve = c >= kb && c < ce;
  cplx x[2 * kRegW];
#pragma unroll
  for (int k = 0; k < 2 * kRegW; ++k) {
    const int src = s_src[k];
    if (src >= 0) x[k] = A[(size_t)src * lda + c];
    else if (k < kRegW && k < jb && solve) x[k] = A[(size_t)(kb + k) * lda + c];
  }
  if (solve) {
#pragma unroll
    for (int r = 1; r < kRegW; ++r) {
      if (r < jb)
#pragma unroll
        for (int q = 0; q < r; ++q) x[r] = cfma(cneg(L[r][q]), x[q], x[r]);
    }
  }
#pragma unroll
  for (int k = 0; k < 2 * kRegW; ++k) {
    if (s_dst[k] >= 0) A[(size_t)s_dst[k] * lda + c] = x[k];
    else if (k < kRegW && k > 0 && k < jb && solve) A[(size_t)(kb + k) * lda + c] = x[k];
  }
}

// Matrices above kRegMaxRows rows: panels of kLuPanel columns updated in L2.  A
// whole SM per panel keeps enough loads in flight for the rank-1 updates.
constexpr int kLuPanel = 32;
constexpr int kLuPanelThreads = 512;

// Panel step of the multi-launch LU: one CTA per matrix factorises columns
// kb .. kb+jb-1 (the first panel also clears info).
__global__ void __launch_bounds__(kLuPanelThreads) getrf_panel_kernel(cplx* const* Aarr, int n, int lda, int kb,
                                                                     int jb, int* ipiv_all, int* info_all) {
  __shared__ double red_v[kLuPanelThreads / 32];
  __shared__ int red_i[kLuPanelThreads / 32];
  __shared__ int s_piv;
  __shared__ cplx prow[kLuPanel];
  const int b = blockIdx.x;
  int info = kb == 0 ? 0 : info_all[b];
  lu_panel(Aarr[b], n, lda, kb, jb, ipiv_all + (size_t)b * n, info, red_v, red_i, &s_piv, prow);
  if (threadIdx.x == 0) info_all[b] = info;
}

// Panel step of the multi-launch LU for few large matrices: a thread-block
// cluster of C CTAs per matrix shares the panel.  Rows kb..n-1 are split into
// C slices; per column every CTA finds the largest |re|+|im| of its slice
// (smallest row on ties), the CTAs read each other's candidates from shared
// memory (distributed shared memory of the cluster) and take the same pivot,
// swap their share of the columns of the two rows, and after a cluster
// barrier scale and update their own rows.  Every element gets the same
// operations as in lu_panel, so the factors are identical.
__global__ void __launch_bounds__(kLuPanelThreads) getrf_panel_team_kernel(cplx* const* Aarr, int n, int lda,
                                                                          int kb, int jb, int* ipiv_all,
                                                                          int* info_all) {
  namespace cg = cooperative_groups;
  cg::cluster_group cl = cg::this_cluster();
  __shared__ double red_v[kLuPanelThreads / 32];
  __shared__ int red_i[kLuPanelThreads / 32];
  __shared__ double s_bv;  // this CTA's pivot candidate
  __shared__ int s_bi;
  __shared__ int s_piv;
  __shared__ cplx prow[kLuPanel];
  const int C = (int)cl.num_blocks(), rank = (int)cl.block_rank();
  const int b = blockIdx.x / C;
  const int tid = threadIdx.x, nthr = blockDim.x;
  constexpr int kU = 8;
  cplx* A = Aarr[b];
  int* ipiv = ipiv_all + (size_t)b * n;
  int info = kb == 0 ? 0 : __ldcg(info_all + b);
  const int per = (n - kb + C - 1) / C;
  const int lo = kb + rank * per, hi = min(n, lo + per);
  const int cper = (n + C - 1) / C;
  const int clo = rank * cper, chi = min(n, clo + cper);
  double best = -1.0;
  int bi = n;
  for (int i0 = max(lo, kb) + tid; i0 < hi; i0 += kU * nthr) {
    double v[kU];
#pragma unroll
    for (int q = 0; q < kU; ++q) {
      const int i = i0 + q * nthr;
      v[q] = i < hi ? cabs1(A[(size_t)i * lda + kb]) : -1.0;
    }
#pragma unroll
    for (int q = 0; q < kU; ++q)
      if (v[q] > best) { best = v[q]; bi = i0 + q * nthr; }
  }
  const int ce = kb + jb;
  for (int j = kb; j < ce; ++j) {
    for (int off = 16; off > 0; off >>= 1) {
      const double ov = __shfl_down_sync(0xffffffffu, best, off);
      const int oi = __shfl_down_sync(0xffffffffu, bi, off);
      if (ov > best || (ov == best && oi < bi)) { best = ov; bi = oi; }
    }
    if ((tid & 31) == 0) { red_v[tid >> 5] = best; red_i[tid >> 5] = bi; }
    __syncthreads();
    if (tid == 0) {
      double bv = red_v[0];
      int bix = red_i[0];
      for (int w = 1; w < nthr / 32; ++w)
        if (red_v[w] > bv || (red_v[w] == bv && red_i[w] < bix)) { bv = red_v[w]; bix = red_i[w]; }
      s_bv = bv;
      s_bi = bix;
    }
    cl.sync();
    if (tid == 0) {
      double bv = -1.0;
      int bix = n;
      for (int r = 0; r < C; ++r) {
        const double v = *cl.map_shared_rank(&s_bv, r);
        const int ix = *cl.map_shared_rank(&s_bi, r);
        if (v > bv || (v == bv && ix < bix)) { bv = v; bix = ix; }
      }
      // a column of zeros below the diagonal keeps its row (lu_panel's
      // candidate is row j then)
      s_piv = bix < n ? bix : j;
      if (rank == 0) ipiv[j] = s_piv;
    }
    __syncthreads();
    const int p = s_piv;
    if (p != j) {
      for (int c = clo + tid; c < chi; c += nthr) {
        cplx t = A[(size_t)j * lda + c];
        A[(size_t)j * lda + c] = A[(size_t)p * lda + c];
        A[(size_t)p * lda + c] = t;
      }
    }
    // the swap is complete everywhere, and every CTA has read the candidates
    cl.sync();
    for (int c = j + tid; c < ce; c += nthr) prow[c - kb] = __ldcg(A + (size_t)j * lda + c);
    __syncthreads();
    const cplx piv = prow[j - kb];
    const int r0 = max(lo, j + 1);
    if (piv.x == 0.0 && piv.y == 0.0) {
      if (info == 0) info = j + 1;
    } else {
      const cplx inv = cdiv(mkc(1.0, 0.0), piv);
      for (int i0 = r0 + tid; i0 < hi; i0 += kU * nthr) {
        cplx v[kU];
#pragma unroll
        for (int q = 0; q < kU; ++q) {
          const int i = i0 + q * nthr;
          if (i < hi) v[q] = A[(size_t)i * lda + j];
        }
#pragma unroll
        for (int q = 0; q < kU; ++q) {
          const int i = i0 + q * nthr;
          if (i < hi) A[(size_t)i * lda + j] = cmul(v[q], inv);
        }
      }
    }
    __syncthreads();
    best = -1.0;
    bi = n;
    const int w = ce - j - 1;
    if (w > 0 && r0 < hi) {
      const int total = (hi - r0) * w;
      for (int base = tid; base < total; base += kU * nthr) {
        cplx l[kU], a[kU];
#pragma unroll
        for (int q = 0; q < kU; ++q) {
          const int idx = base + q * nthr;
          if (idx < total) {
            const int i = r0 + idx / w, c = j + 1 + idx % w;
            l[q] = A[(size_t)i * lda + j];
            a[q] = A[(size_t)i * lda + c];
          }
        }
#pragma unroll
        for (int q = 0; q < kU; ++q) {
          const int idx = base + q * nthr;
          if (idx < total) {
            const int i = r0 + idx / w, c = j + 1 + idx % w;
            const cplx v = cfma(cneg(l[q]), prow[c - kb], a[q]);
            A[(size_t)i * lda + c] = v;
            if (c == j + 1) {
              const double av = cabs1(v);
              if (av > best || (av == best && i < bi)) { best = av; bi = i; }
            }
          }
        }
      }
    }
    __syncthreads();
  }
  if (rank == 0 && tid == 0) info_all[b] = info;
  // no CTA leaves while another may still read its candidate
  cl.sync();
}

// U12 of the multi-launch LU: one CTA per (matrix, 64 columns right of the
// panel, up to column ce), a thread per column; the unit lower L11 (jb <=
// kLuPanel) is read through the read-only path (every thread reads the same
// entry).
__global__ void __launch_bounds__(64) getrf_trsm_kernel(cplx* const* Aarr, int lda, int kb, int jb, int ce) {
  cplx* A = Aarr[blockIdx.y];
  const int c = kb + jb + blockIdx.x * 64 + threadIdx.x;
  if (c >= ce) return;
  for (int r = 1; r < jb; ++r) {
    cplx x = A[(size_t)(kb + r) * lda + c];
    const cplx* Lr = A + (size_t)(kb + r) * lda + kb;
    for (int q = 0; q < r; ++q) x = cfma(cneg(__ldg(&Lr[q])), A[(size_t)(kb + q) * lda + c], x);
    A[(size_t)(kb + r) * lda + c] = x;
  }
}

// Blocked LU solve, left-looking: one CTA per (matrix, 64-column slab of B).
// Each 64-row block of the slab first takes the contribution of all rows
// already solved as one long-K tile GEMM (L(rb:, :rb) X(:rb) forward,
// U(rb:, re:) X(re:) backward), then its diagonal block is solved in two
// 32-row halves, one thread per column with the column in registers.
__device__ __forceinline__ void load_block32(cplx (*Tsm)[33], const cplx* LU, int lda, int r0, int c0, int h, int w) {
  for (int idx = threadIdx.x; idx < h * w; idx += blockDim.x) {
    const int r = idx / w, q = idx % w;
    Tsm[r][q] = LU[(size_t)(r0 + r) * lda + c0 + q];
  }
}

// kInv (the inverse, LAPACK getri order): B starts as the identity without
// the row interchanges, so column c of L^-1 is zero above row c and the
// forward pass of the slab starting at column c0 begins at row c0 with its
// long-K products cut to K = c0 .. rb; the column interchanges follow in
// zcolperm_kernel.  This saves a third of the flops of solving against P.
template <bool kInv>
__global__ void __launch_bounds__(kTileThreads) zgetrs_kernel(const cplx* const* LUarr, int n, int lda,
                                                             const int* ipiv_all, cplx* const* Barr,
                                                             int nrhs, int ldb) {
  __shared__ __align__(16) unsigned char smem_raw[sizeof(TileSmem)];
  TileSmem& sm = *reinterpret_cast<TileSmem*>(smem_raw);
  cplx (*Tsm)[33] = reinterpret_cast<cplx (*)[33]>(smem_raw);
  const int tid = threadIdx.x;
  const int b = blockIdx.y;
  const int c0 = blockIdx.x * 64;
  const int cw = min(64, nrhs - c0);
  const cplx* LU = LUarr[b];
  const int* ipiv = ipiv_all + (size_t)b * n;
  cplx* B = Barr[b] + c0;
  if (kInv) {
    for (int idx = tid; idx < n * cw; idx += blockDim.x) {
      const int r = idx / cw, c = idx % cw;
      B[(size_t)r * ldb + c] = mkc(r == c0 + c ? 1.0 : 0.0, 0.0);
    }
  } else if (tid < cw) {
    for (int j = 0; j < n; ++j) {
      const int p = ipiv[j];
      if (p != j) {
        cplx t = B[(size_t)j * ldb + tid];
        B[(size_t)j * ldb + tid] = B[(size_t)p * ldb + tid];
        B[(size_t)p * ldb + tid] = t;
      }
    }
  }
  __syncthreads();
  // forward substitution with the unit lower factor (rows below k0 of the
  // slab are zero for the inverse)
  const int k0 = kInv ? c0 : 0;
  for (int rb = k0; rb < n; rb += 64) {
    const int rw = min(64, n - rb);
    if (rb > k0) {
      cplx acc[4][4];
      tile_zero(acc);
      tile_mma<false, false>(sm, acc, LU + (size_t)rb * lda + k0, lda, B + (size_t)k0 * ldb, ldb, nullptr, rw, cw,
                             rb - k0, 0, 0);
      tile_store(acc, B + (size_t)rb * ldb, ldb, B + (size_t)rb * ldb, ldb, mkc(-1.0, 0.0), mkc(1.0, 0.0),
                 mkc(0.0, 0.0), rw, cw, 0, 0);
      __syncthreads();
    }
    for (int h0 = rb; h0 < rb + rw; h0 += 32) {
      const int hw = min(32, rb + rw - h0);
      if (h0 > rb) {
        // the first half of the block feeds the second
        load_block32(Tsm, LU, lda, h0, rb, hw, 32);
        __syncthreads();
        if (tid < cw) {
          cplx x[32];
#pragma unroll
          for (int q = 0; q < 32; ++q) x[q] = B[(size_t)(rb + q) * ldb + tid];
          for (int r = 0; r < hw; ++r) {
            cplx acc = B[(size_t)(h0 + r) * ldb + tid];
#pragma unroll
            for (int q = 0; q < 32; ++q) acc = cfma(cneg(Tsm[r][q]), x[q], acc);
            B[(size_t)(h0 + r) * ldb + tid] = acc;
          }
        }
        __syncthreads();
      }
      load_block32(Tsm, LU, lda, h0, h0, hw, hw);
      __syncthreads();
      if (tid < cw) {
        // the column's solved entries are re-read from L1
        for (int r = 1; r < hw; ++r) {
          cplx acc = B[(size_t)(h0 + r) * ldb + tid];
          for (int q = 0; q < r; ++q) acc = cfma(cneg(Tsm[r][q]), B[(size_t)(h0 + q) * ldb + tid], acc);
          B[(size_t)(h0 + r) * ldb + tid] = acc;
        }
      }
      __syncthreads();
    }
  }
  // back substitution with the upper factor
  for (int rb = ((n - 1) / 64) * 64; rb >= 0; rb -= 64) {
    const int re = min(n, rb + 64), rw = re - rb;
    if (re < n) {
      cplx acc[4][4];
      tile_zero(acc);
      tile_mma<false, false>(sm, acc, LU + (size_t)rb * lda + re, lda, B + (size_t)re * ldb, ldb, nullptr, rw, cw,
                             n - re, 0, 0);
      tile_store(acc, B + (size_t)rb * ldb, ldb, B + (size_t)rb * ldb, ldb, mkc(-1.0, 0.0), mkc(1.0, 0.0),
                 mkc(0.0, 0.0), rw, cw, 0, 0);
      __syncthreads();
    }
    for (int h0 = (rw > 32) ? rb + 32 : rb; h0 >= rb; h0 -= 32) {
      const int hw = min(32, re - h0);
      const int tail = re - h0 - hw;  // rows of this block below the half, already solved
      if (tail > 0) {
        load_block32(Tsm, LU, lda, h0, h0 + hw, hw, tail);
        __syncthreads();
        if (tid < cw) {
          cplx x[32];
#pragma unroll
          for (int q = 0; q < 32; ++q) x[q] = q < tail ? B[(size_t)(h0 + hw + q) * ldb + tid] : mkc(0.0, 0.0);
          for (int r = 0; r < hw; ++r) {
            cplx acc = B[(size_t)(h0 + r) * ldb + tid];
#pragma unroll
            for (int q = 0; q < 32; ++q)
              if (q < tail) acc = cfma(cneg(Tsm[r][q]), x[q], acc);
            B[(size_t)(h0 + r) * ldb + tid] = acc;
          }
        }
        __syncthreads();
      }
      load_block32(Tsm, LU, lda, h0, h0, hw, hw);
      __syncthreads();
      if (tid < cw) {
        for (int r = hw - 1; r >= 0; --r) {
          cplx acc = B[(size_t)(h0 + r) * ldb + tid];
          for (int q = r + 1; q < hw; ++q) acc = cfma(cneg(Tsm[r][q]), B[(size_t)(h0 + q) * ldb + tid], acc);
          B[(size_t)(h0 + r) * ldb + tid] = cdiv(acc, Tsm[r][r]);
        }
      }
      __syncthreads();
    }
  }
}

// X <- X P for the column interchanges of getrf (ipiv, applied from the
// last to the first as LAPACK getri does): rows of X pass through shared
// memory, `rows` per CTA; the permutation is rebuilt per CTA from ipiv.
__global__ void zcolperm_kernel(cplx* const* Xarr, int n, int ldx, const int* ipiv_all, int rows) {
  extern __shared__ __align__(16) unsigned char dsm[];
  int* perm = reinterpret_cast<int*>(dsm);
  cplx* buf = reinterpret_cast<cplx*>(dsm + (((size_t)n * sizeof(int) + 15) & ~(size_t)15));
  const int b = blockIdx.y, r0 = blockIdx.x * rows;
  const int* ipiv = ipiv_all + (size_t)b * n;
  cplx* X = Xarr[b];
  const int rw = min(rows, n - r0);
  for (int c = threadIdx.x; c < n; c += blockDim.x) perm[c] = c;
  for (int idx = threadIdx.x; idx < rw * n; idx += blockDim.x)
    buf[idx] = X[(size_t)(r0 + idx / n) * ldx + idx % n];
  __syncthreads();
  if (threadIdx.x == 0)
    for (int j = n - 1; j >= 0; --j) {
      const int p = ipiv[j];
      if (p != j) { const int t = perm[j]; perm[j] = perm[p]; perm[p] = t; }
    }
  __syncthreads();
  for (int idx = threadIdx.x; idx < rw * n; idx += blockDim.x) {
    const int r = idx / n, c = idx % n;
    X[(size_t)(r0 + r) * ldx + c] = buf[(size_t)r * n + perm[c]];
  }
}

__global__ void identity_kernel(cplx* const* Barr, int n, int ldb) {
  cplx* B = Barr[blockIdx.y];
  for (size_t idx = blockIdx.x * (size_t)blockDim.x + threadIdx.x; idx < (size_t)n * n;
       idx += (size_t)gridDim.x * blockDim.x) {
    const int r = (int)(idx / n), c = (int)(idx % n);
    B[(size_t)r * ldb + c] = mkc(r == c ? 1.0 : 0.0, 0.0);
  }
}

__global__ void copy_kernel(const cplx* const* S, int lds, cplx* const* Dd, int ldd, int rows, int cols) {
  const cplx* s = S[blockIdx.y];
  cplx* d = Dd[blockIdx.y];
  for (size_t idx = blockIdx.x * (size_t)blockDim.x + threadIdx.x; idx < (size_t)rows * cols;
       idx += (size_t)gridDim.x * blockDim.x) {
    const int r = (int)(idx / cols), c = (int)(idx % cols);
    d[(size_t)r * ldd + c] = s[(size_t)r * lds + c];
  }
}

}  // namespace

cudaError_t zgemm_batched(const GemmArgs& g, cudaStream_t st) {
  if (g.batch <= 0 || g.M <= 0 || g.N <= 0) return cudaSuccess;
  if (g.transA) return g.transB ? zgemm_launch<true, true>(g, st) : zgemm_launch<true, false>(g, st);
  return g.transB ? zgemm_launch<false, true>(g, st) : zgemm_launch<false, false>(g, st);
}

int device_sm_count() {
  static int count = 0;
  if (!count) {
    int dev = 0, c = 0;
    if (cudaGetDevice(&dev) == cudaSuccess && cudaDeviceGetAttribute(&c, cudaDevAttrMultiProcessorCount, dev) ==
                                                  cudaSuccess && c > 0)
      count = c;
    else
      return 148;
  }
  return count;
}

namespace {
// CTAs per matrix of the multi-launch LU's panel step (0: automatic), set by
// rcwa_set_lu_cluster.
std::atomic<int> g_lu_team{0};

// Team of the panels above kRegMaxRows rows: the forced size, or up to 8 CTAs
// where the batch would leave half of the SMs idle.
int lu_team_size(int batch) {
  const int forced = g_lu_team.load();
  if (forced > 0) return forced;
  const int sms = device_sm_count();
  if (2 * batch > sms) return 1;
  static std::mutex mu;
  static std::map<int, int> cache;  // batch -> size
  std::lock_guard<std::mutex> lk(mu);
  auto it = cache.find(batch);
  if (it != cache.end()) return it->second;
  int pick = 1;
  for (int c = std::min(8, sms / batch); c >= 2; --c) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(c);
    cfg.blockDim = dim3(kLuPanelThreads);
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = c;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    int nc = 0;
    if (cudaOccupancyMaxActiveClusters(&nc, (void*)getrf_panel_team_kernel, &cfg) != cudaSuccess) {
      cudaGetLastError();
      continue;
    }
    if (nc >= batch) {
      pick = c;
      break;
    }
  }
  cache[batch] = pick;
  return pick;
}

cudaError_t launch_panel(cplx* const* A, int n, int lda, int kb, int jb, int* ipiv, int* info, int batch, int team,
                         cudaStream_t st) {
  if (team <= 1) {
    getrf_panel_kernel<<<batch, kLuPanelThreads, 0, st>>>(A, n, lda, kb, jb, ipiv, info);
    return cudaGetLastError();
  }
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(batch * team);
  cfg.blockDim = dim3(kLuPanelThreads);
  cfg.stream = st;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = team;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, getrf_panel_team_kernel, A, n, lda, kb, jb, ipiv, info);
}
}  // namespace

namespace {
// Threads of a register panel of `rows` rows (one per row), and its CTAs: what
// its rows need, or the forced cluster size if that is larger.
int regpanel_threads(int rows) { return rows <= 128 ? 128 : rows <= 256 ? 256 : kRegT; }
int regpanel_team(int rows) {
  const int threads = regpanel_threads(rows);
  return std::max((rows + threads - 1) / threads, g_lu_team.load());
}

cudaError_t launch_regpanel(cplx* const* A, int n, int lda, int kb, int jb, int* ipiv, int* info, int batch,
                            cudaStream_t st) {
  const int threads = regpanel_threads(n - kb), team = regpanel_team(n - kb);
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(batch * team);
  cfg.blockDim = dim3(threads);
  cfg.stream = st;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = team;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, getrf_regpanel_kernel, A, n, lda, kb, jb, ipiv, info);
}

// A22 -= L21 U12 on the columns kb+jb .. ce-1
cudaError_t panel_update(cplx* const* A, int n, int lda, int kb, int jb, int ce, int batch, cudaStream_t st) {
  GemmArgs g{};
  g.A = A; g.B = A; g.C = A; g.D = A;
  g.offA = (size_t)(kb + jb) * lda + kb;
  g.offB = (size_t)kb * lda + kb + jb;
  g.offC = g.offD = (size_t)(kb + jb) * lda + kb + jb;
  g.M = n - kb - jb; g.N = ce - kb - jb; g.K = jb;
  g.lda = g.ldb = g.ldc = g.ldd = lda;
  g.alpha = mkc(-1.0, 0.0); g.beta = mkc(1.0, 0.0); g.gammaI = mkc(0.0, 0.0);
  g.batch = batch;
  return zgemm_batched(g, st);
}
}  // namespace

extern "C" int rcwa_set_lu_cluster(int ctas) {
  if (ctas < 0 || ctas > 8) return RCWA_ERR_INVALID;
  g_lu_team.store(ctas);
  return RCWA_OK;
}

extern "C" int rcwa_lu_cluster_size(int n, int batch) {
  if (batch <= 0 || n <= 0 || zgetrf_default_schedule(n, batch) == 0) return 1;
  return n <= kRegMaxRows ? regpanel_team(n) : lu_team_size(batch);
}

int zgetrf_default_schedule(int n, int batch, int sms) {
  if (sms <= 0) sms = device_sm_count();
  // The lines were drawn with the 32-column panels in L2 and hold for full
  // batches (B200, schedules 1 / 2: 58 x 882 13.6 / 9.0 ms, 148 x 450 5.4 / 4.2,
  // 148 x 256 1.35 / 1.25; 0 / 1: 148 x 98 0.17 / 0.30).  With the register
  // panels schedule 1 is faster for few matrices (1 x 300 0.85 against 1.12 ms,
  // 2 x 1250 5.1 against 6.2), for n = 117..128 (148 x 122 0.38 against 0.50) and,
  // like schedule 2, for four waves and more (600 x 98 0.67 against 0.81, 600 x
  // 198 2.6 against 5.9, 600 x 450 19.6 and 15.2 against 37.1); the tuner finds
  // these.
  if (n <= 128 || batch >= 4 * sms) return 0;
  return n >= 256 ? 2 : 1;
}

cudaError_t zgetrf_batched(cplx* const* A, int n, int lda, int* ipiv, int* info, int batch,
                           cudaStream_t st, int schedule) {
  if (batch <= 0 || n <= 0) return cudaSuccess;
  if (schedule < 0) schedule = zgetrf_default_schedule(n, batch);
  if (schedule == 0 && n <= kSmallLuMax) {
    static SmemAttrOnce attr;
    const cudaError_t e = attr.ensure(getrf_small_kernel, (int)small_lu_smem(kSmallLuMax));
    if (e != cudaSuccess) return e;
    getrf_small_kernel<<<batch, kSmallLuThreads, small_lu_smem(n), st>>>(A, n, lda, ipiv, info);
    ++launch_counter();
    return cudaGetLastError();
  }
  if (schedule == 0) {
    zgetrf_kernel<<<batch, kTileThreads, 0, st>>>(A, n, lda, ipiv, info);
    ++launch_counter();
    return cudaGetLastError();
  }
  if (schedule == 2) return zgetrf_blocked_batched(A, n, lda, ipiv, info, batch, nullptr, st);
  return zgetrf_columns(A, n, lda, 0, n, ipiv, info, batch, st);
}

cudaError_t zgetrf_columns(cplx* const* A, int n, int lda, int k0, int ce, int* ipiv, int* info, int batch,
                           cudaStream_t st) {
  if (batch <= 0 || k0 < 0 || ce > n || k0 >= ce) return cudaErrorInvalidValue;
  if (n <= kRegMaxRows) {
    for (int kb = k0; kb < ce; kb += kRegW) {
      const int jb = min(kRegW, ce - kb);
      cudaError_t e = launch_regpanel(A, n, lda, kb, jb, ipiv, info, batch, st);
      if (e != cudaSuccess) return e;
      ++launch_counter();
      if (n == jb) break;  // nothing beside the panel
      getrf_swap_trsm_kernel<<<dim3((n - jb + 127) / 128, batch), 128, 0, st>>>(A, n, lda, kb, jb, ce, ipiv);
      ++launch_counter();
      if ((e = cudaGetLastError()) != cudaSuccess) return e;
      if ((e = panel_update(A, n, lda, kb, jb, ce, batch, st)) != cudaSuccess) return e;
    }
    return cudaSuccess;
  }
  // a cluster of CTAs per matrix shares each panel when the batch leaves SMs idle
  const int team = lu_team_size(batch);
  for (int kb = k0; kb < ce; kb += kLuPanel) {
    const int jb = min(kLuPanel, ce - kb);
    cudaError_t pe = launch_panel(A, n, lda, kb, jb, ipiv, info, batch, team, st);
    if (pe != cudaSuccess) return pe;
    ++launch_counter();
    const int m2 = n - kb - jb, w = ce - kb - jb;
    if (m2 <= 0 || w <= 0) break;
    getrf_trsm_kernel<<<dim3((w + 63) / 64, batch), 64, 0, st>>>(A, lda, kb, jb, ce);
    ++launch_counter();
    const cudaError_t err = panel_update(A, n, lda, kb, jb, ce, batch, st);
    if (err != cudaSuccess) return err;
  }
  return cudaGetLastError();
}

// Whether a solve runs blocked (lu_blocked.cu: 128-row triangles with a thread
// per right-hand side and the entries of 32 rows in registers, plus batched
// GEMM updates over the whole grid) or on one CTA per 64-column slab, whose
// triangles wait for a dependent load per entry.  Callers have 1, 2 or at least
// n right-hand sides; for 1 or 2 most of a blocked CTA would be idle.  With more
// slabs than SMs the blocked route is faster at every order from 16 on (B200,
// solves of 300 x 16 1.7x, 1200 x 22 4.2x, 148 x 98 1.6x, 300 x 126 1.9x).  One
// wave of slabs costs the slab kernel its n rows and the blocked one triangles
// padded to 32 rows, so it keeps the orders with the most padding (slab kernel's
// time over the blocked one's, one to 74 matrices with n right-hand sides:
// 0.63-0.68 at order 16, 0.88-0.92 at 22, 0.94-1.03 at 24, 1.13-1.22 at 28,
// 0.92-0.99 at 34, 0.98-1.04 at 38, 1.2-1.26 at 50, 1.0-1.09 at 66, 0.96-1.04 at
// 98, 1.14-1.23 at 128).  Above 128 right-hand sides the blocked route needs a
// second CTA per matrix: with 2 n or 3 n of them 1.16 at 50, 0.93-0.97 at 66-82,
// 1.1 at 86, 0.89-0.92 at 98-116, 0.95-1.07 at 122, 1.03-1.07 at 128.
constexpr int kBlockedSolveMin = 16;

bool solve_blocked(int n, int nrhs, int batch) {
  if (n < kBlockedSolveMin || nrhs < kBlockedSolveMin) return false;
  if ((long long)batch * ((nrhs + 63) / 64) > device_sm_count()) return true;
  if (n < 24) return false;
  return nrhs <= 128 ? n <= 32 || n >= 38 : n <= 64 || (n > 82 && n <= 96) || n > 122;
}

cudaError_t zgetrs_batched(const cplx* const* LU, int n, int lda, const int* ipiv, cplx* const* B,
                           int nrhs, int ldb, int batch, cudaStream_t st) {
  if (batch <= 0 || n <= 0 || nrhs <= 0) return cudaSuccess;
  if (solve_blocked(n, nrhs, batch))
    return zgetrs_blocked_batched(LU, n, lda, ipiv, B, nrhs, ldb, batch, false, nullptr, st);
  dim3 grid((nrhs + 63) / 64, batch);
  zgetrs_kernel<false><<<grid, kTileThreads, 0, st>>>(LU, n, lda, ipiv, B, nrhs, ldb);
  ++launch_counter();
  return cudaGetLastError();
}

cudaError_t zgetri_batched(const cplx* const* LU, int n, int lda, const int* ipiv, cplx* const* X, int ldx,
                           int batch, cudaStream_t st) {
  if (batch <= 0 || n <= 0) return cudaSuccess;
  if (solve_blocked(n, n, batch)) return zgetrs_blocked_batched(LU, n, lda, ipiv, X, n, ldx, batch, true, nullptr, st);
  dim3 grid((n + 63) / 64, batch);
  zgetrs_kernel<true><<<grid, kTileThreads, 0, st>>>(LU, n, lda, ipiv, X, n, ldx);
  ++launch_counter();
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) return e;
  return zcolperm_batched(X, n, ldx, ipiv, batch, st);
}

cudaError_t zcolperm_batched(cplx* const* X, int n, int ldx, const int* ipiv, int batch, cudaStream_t st) {
  cudaError_t e;
  // rows per CTA: as many as fit in 64 KB next to the permutation
  const size_t perm_bytes = ((size_t)n * sizeof(int) + 15) & ~(size_t)15;
  const int rows = (int)std::max<size_t>(1, std::min<size_t>(8, (64u << 10) / ((size_t)n * sizeof(cplx))));
  const size_t smem = perm_bytes + (size_t)rows * n * sizeof(cplx);
  if (smem > (size_t)(227u << 10)) return cudaErrorInvalidValue;
  static SmemAttrOnce attr;
  if ((e = attr.ensure(zcolperm_kernel, (int)(227u << 10))) != cudaSuccess) return e;
  zcolperm_kernel<<<dim3((n + rows - 1) / rows, batch), 256, smem, st>>>(X, n, ldx, ipiv, rows);
  ++launch_counter();
  return cudaGetLastError();
}

cudaError_t zset_identity_batched(cplx* const* B, int n, int ldb, int batch, cudaStream_t st) {
  if (batch <= 0 || n <= 0) return cudaSuccess;
  dim3 grid(min(1024, (n * n + 255) / 256), batch);
  identity_kernel<<<grid, 256, 0, st>>>(B, n, ldb);
  ++launch_counter();
  return cudaGetLastError();
}

cudaError_t zcopy_batched(const cplx* const* src, int lds, cplx* const* dst, int ldd, int rows, int cols,
                          int batch, cudaStream_t st) {
  if (batch <= 0 || rows <= 0 || cols <= 0) return cudaSuccess;
  dim3 grid(min(1024, (rows * cols + 255) / 256), batch);
  copy_kernel<<<grid, 256, 0, st>>>(src, lds, dst, ldd, rows, cols);
  ++launch_counter();
  return cudaGetLastError();
}
