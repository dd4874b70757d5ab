// Pipelined complex-FP64 tile product on the FP64 tensor path (DMMA).
//
// A CTA of WR x WC warps computes a (WR*RT*8) x (WC*CT*8) output tile, each
// warp RT x CT blocks of 8 x 8 with a real and an imaginary accumulator
// fragment (mma.sync m8n8k4 f64, four real products per complex block).
// Operand slabs of BK along K move into ST shared-memory stages with cp.async
// (16 bytes = one complex number, zero-filled outside the matrix), so ST - 1
// slabs are in flight while one is multiplied and one barrier per slab is
// enough.  Numbers stay interleaved (re, im): a fragment element is one
// 16-byte shared load.  The row pitch is 4 (mod 8) elements for an operand
// staged with K contiguous and 2 (mod 8) for one staged with M or N
// contiguous, so the eight lanes of a load phase (two rows g, four k) touch
// the eight 16-byte bank groups once.
#pragma once
#include "tile.cuh"

__device__ __forceinline__ void cp_async16_zfill(void* smem_dst, const void* gmem_src, bool in) {
  const unsigned s = (unsigned)__cvta_generic_to_shared(smem_dst);
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(s), "l"(gmem_src), "r"(in ? 16 : 0) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;\n" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_async_wait_group() { asm volatile("cp.async.wait_group %0;\n" ::"n"(N) : "memory"); }

template <int kWR, int kWC, int kRT, int kCT, int kBK, int kST>
struct PipeTile {
  static constexpr int WR = kWR, WC = kWC, RT = kRT, CT = kCT, BK = kBK, ST = kST;
  static constexpr int BM = WR * RT * 8, BN = WC * CT * 8, T = WR * WC * 32;
  static constexpr int PK = BK + 4;                                 // pitch, K contiguous
  static constexpr int PM = BM + 2, PN = BN + 2;                    // pitch, M / N contiguous
  static constexpr int EA = BM * PK > BK * PM ? BM * PK : BK * PM;  // elements of one A stage
  static constexpr int EB = BN * PK > BK * PN ? BN * PK : BK * PN;
  static constexpr int kLoadsA = BM * BK / T, kLoadsB = BN * BK / T;
  static constexpr size_t kSmem = sizeof(cplx) * (size_t)ST * (EA + EB + BK);
  static_assert(BK % 8 == 0 && BM % 8 == 0 && BN % 8 == 0, "pitch residues");
  static_assert(BM * BK % T == 0 && BN * BK % T == 0 && T % BK == 0 && T % BM == 0 && T % BN == 0, "whole loads");
};

// One slab [k0, k0 + BK) of op(A) rows m0.., op(B) columns n0.. (and of the
// diagonal s between them) into stage `st`.  The out-of-range elements are
// written as zeros.
template <class C, bool TA, bool TB, bool kScale>
__device__ __forceinline__ void pipe_load(cplx* sm, int st, const cplx* __restrict__ A, int lda,
                                          const cplx* __restrict__ B, int ldb, const cplx* __restrict__ s, int M,
                                          int N, int K, int m0, int n0, int k0) {
  const int tid = threadIdx.x;
  cplx* a = sm + (size_t)st * (C::EA + C::EB + C::BK);
  cplx* b = a + C::EA;
#pragma unroll
  for (int r = 0; r < C::kLoadsA; ++r) {
    const int idx = tid + r * C::T;
    const int kk = TA ? idx / C::BM : idx % C::BK, mm = TA ? idx % C::BM : idx / C::BK;
    const int gm = m0 + mm, gk = k0 + kk;
    const bool in = gm < M && gk < K;
    const cplx* src = TA ? A + (size_t)gk * lda + gm : A + (size_t)gm * lda + gk;
    cp_async16_zfill(TA ? a + kk * C::PM + mm : a + mm * C::PK + kk, in ? src : A, in);
  }
#pragma unroll
  for (int r = 0; r < C::kLoadsB; ++r) {
    const int idx = tid + r * C::T;
    const int kk = TB ? idx % C::BK : idx / C::BN, nn = TB ? idx / C::BK : idx % C::BN;
    const int gn = n0 + nn, gk = k0 + kk;
    const bool in = gn < N && gk < K;
    const cplx* src = TB ? B + (size_t)gn * ldb + gk : B + (size_t)gk * ldb + gn;
    cp_async16_zfill(TB ? b + nn * C::PK + kk : b + kk * C::PN + nn, in ? src : B, in);
  }
  if (kScale && tid < C::BK) cp_async16_zfill(b + C::EB + tid, k0 + tid < K ? s + k0 + tid : s, k0 + tid < K);
}

// acc = op(A)[m0.., :K] diag(s) op(B)[:K, n0..].  Accumulator layout: re/im
// [rt][ct][e] is element (8*(RT*wr + rt) + lane/4, 8*(CT*wc + ct) +
// 2*(lane%4) + e) of the tile.  Every thread of the CTA takes part; sm holds
// C::kSmem bytes and is free again after the caller's next barrier.  Blocks of
// 8 rows or columns that lie outside the matrix are skipped (a warp-uniform
// test), so an edge tile costs what it holds.  The products of an element are
// added in the order of k, the four real products of a k-step of 4 in the
// order of tile_mma, so both routines round alike.
template <class C, bool TA, bool TB, bool kScale>
__device__ __forceinline__ void pipe_mma(cplx* sm, double (&re)[C::RT][C::CT][2], double (&im)[C::RT][C::CT][2],
                                         const cplx* __restrict__ A, int lda, const cplx* __restrict__ B, int ldb,
                                         const cplx* __restrict__ s, int M, int N, int K, int m0, int n0) {
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const int g = lane >> 2, t = lane & 3;
  const int wm = (w % C::WR) * C::RT * 8, wn = (w / C::WR) * C::CT * 8;
  const int nrt = min(C::RT, (M - m0 - wm + 7) >> 3), nct = min(C::CT, (N - n0 - wn + 7) >> 3);
#pragma unroll
  for (int i = 0; i < C::RT; ++i)
#pragma unroll
    for (int j = 0; j < C::CT; ++j) re[i][j][0] = re[i][j][1] = im[i][j][0] = im[i][j][1] = 0.0;
  const int nk = (K + C::BK - 1) / C::BK;
#pragma unroll
  for (int p = 0; p < C::ST - 1; ++p) {
    if (p < nk) pipe_load<C, TA, TB, kScale>(sm, p, A, lda, B, ldb, s, M, N, K, m0, n0, p * C::BK);
    cp_async_commit();
  }
  int st = 0;
  for (int it = 0; it < nk; ++it) {
    cp_async_wait_group<C::ST - 2>();
    __syncthreads();
    {
      const int nx = it + C::ST - 1;
      int ls = st + C::ST - 1;
      if (ls >= C::ST) ls -= C::ST;
      if (nx < nk) pipe_load<C, TA, TB, kScale>(sm, ls, A, lda, B, ldb, s, M, N, K, m0, n0, nx * C::BK);
      cp_async_commit();
    }
    const cplx* a = sm + (size_t)st * (C::EA + C::EB + C::BK);
    const cplx* b = a + C::EA;
    const cplx* sc = b + C::EB;
    if (++st == C::ST) st = 0;
    if (nrt <= 0 || nct <= 0) continue;
#pragma unroll
    for (int k4 = 0; k4 < C::BK; k4 += 4) {
      cplx fa[C::RT], fb[C::CT];
#pragma unroll
      for (int i = 0; i < C::RT; ++i)
        fa[i] = TA ? a[(k4 + t) * C::PM + wm + 8 * i + g] : a[(wm + 8 * i + g) * C::PK + k4 + t];
#pragma unroll
      for (int j = 0; j < C::CT; ++j) {
        fb[j] = TB ? b[(wn + 8 * j + g) * C::PK + k4 + t] : b[(k4 + t) * C::PN + wn + 8 * j + g];
        if (kScale) fb[j] = cmul(sc[k4 + t], fb[j]);
      }
#pragma unroll
      for (int i = 0; i < C::RT; ++i) {
        if (i >= nrt) break;
        const double an = -fa[i].y;
#pragma unroll
        for (int j = 0; j < C::CT; ++j) {
          if (j < nct) {
            dmma_8x8x4(re[i][j][0], re[i][j][1], fa[i].x, fb[j].x);
            dmma_8x8x4(re[i][j][0], re[i][j][1], an, fb[j].y);
            dmma_8x8x4(im[i][j][0], im[i][j][1], fa[i].x, fb[j].y);
            dmma_8x8x4(im[i][j][0], im[i][j][1], fa[i].y, fb[j].x);
          }
        }
      }
    }
  }
  cp_async_wait_group<0>();
}

// D = alpha*acc + beta*C + gammaI*(m == n) (no C when beta is zero; C may
// alias D), in tile_store's order of operations.
template <class C>
__device__ __forceinline__ void pipe_store(const double (&re)[C::RT][C::CT][2], const double (&im)[C::RT][C::CT][2],
                                           cplx* D, int ldd, const cplx* Cm, int ldc, cplx alpha, cplx beta,
                                           cplx gammaI, int M, int N, int m0, int n0) {
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const int g = lane >> 2, t = lane & 3;
  const int wm = (w % C::WR) * C::RT * 8, wn = (w / C::WR) * C::CT * 8;
#pragma unroll
  for (int i = 0; i < C::RT; ++i) {
    const int m = m0 + wm + 8 * i + g;
    if (m >= M) continue;
    cplx c[C::CT][2];
    if (Cm) {
#pragma unroll
      for (int j = 0; j < C::CT; ++j)
#pragma unroll
        for (int e = 0; e < 2; ++e) {
          const int n = n0 + wn + 8 * j + 2 * t + e;
          if (n < N) c[j][e] = Cm[(size_t)m * ldc + n];
        }
    }
#pragma unroll
    for (int j = 0; j < C::CT; ++j)
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        const int n = n0 + wn + 8 * j + 2 * t + e;
        if (n >= N) continue;
        cplx v = cmul(alpha, mkc(re[i][j][e], im[i][j][e]));
        if (Cm) v = cfma(beta, c[j][e], v);
        if (m == n) v = cadd(v, gammaI);
        D[(size_t)m * ldd + n] = v;
      }
  }
}
