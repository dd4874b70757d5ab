// Batched complex eigensolver, one CTA per matrix or (above 116 rows, where the
// batch leaves SMs idle) a cluster of up to 8, FP64 throughout:
//   1. Householder reduction to upper Hessenberg form, Q accumulated backwards;
//   2. small-bulge multishift QR (Ahues-Tisseur deflation test, exceptional
//      shifts after 10 sweeps) producing the Schur form T with Schur vectors Z:
//      matrices of at most kBlkMax rows entirely in shared memory
//      (schur_block), larger ones through a chase window in shared memory with
//      aggressive early deflation (schur_ms);
//   3. eigenvectors of T by back-substitution (protected small divisors),
//      back-transformed with Z by the tile GEMM and normalised to unit 2-norm.
// This replaces LAPACK zgeev('N','V') behind MKLEigenSolver
// (rcwa/MKLEigenSolver.hpp:102-179).  Balancing is not applied.
#include <algorithm>
#include <atomic>
#include <map>
#include <mutex>
#include <tuple>

#include "eig.cuh"
#include "linalg.cuh"
#include "tile.cuh"

namespace {

constexpr int kEigThreads = kTileThreads;  // 256
constexpr int kWin = 32;

constexpr int kHb = kEigPanel;

__host__ __device__ inline size_t workspace_bytes(int n) { return zgeev_workspace_bytes(n); }

struct Scratch {
  cplx* Z;     // n*n, column-major: Z(r, c) = Z[c*n + r]
  cplx* X;     // n*n, row-major upper-triangular eigenvector matrix of T
  cplx* v;     // n: current Householder vector / work column
  double* scale; // what the eigenvalues are to be multiplied with (n complex)
  cplx* uv;    // n
  cplx* v0;    // n: leading element of each stored reflector
  cplx* Vb;    // n x kHb  panel reflectors, explicit (row-major)
  cplx* VH;    // kHb x n  their conjugate transposes (or n x kHb conj(V))
  cplx* Yb;    // n x kHb  A V T  (also kHb x n work)
  cplx* Wb;    // kHb x n  (also n x kHb work)
  cplx* Vt;    // kHb x n  V^T (first kHb x kHb: T^H / T^T)
  cplx* Tall;  // (ceil(n/kHb)+1) x kHb x kHb  triangular factors of all panels
  double* tau; // n
};

#ifdef RCWA_EIG_STATS
// counters: 0 ms sweeps, 1 ss sweeps, 2 passes, 3 chase cycles, 4 replay cycles, 5 window-Schur cycles,
// 6 reordering and re-Hessenberg cycles, 7 early-deflation update cycles, 8 early-deflation cycles,
// 9 single-shift cycles, 10 Schur cycles, 11 early deflations, 12 deflated by them
__device__ unsigned long long g_eig_stats[32];
#define STAT_ADD(i, v) do { if (threadIdx.x == 0) atomicAdd(&g_eig_stats[i], (unsigned long long)(v)); } while (0)
#else
#define STAT_ADD(i, v) do { } while (0)
#endif

__device__ Scratch scratch_for(void* work, int n, int b) {
  const size_t nn = (size_t)n * n;
  const size_t nk = (size_t)n * kHb;
  char* base = (char*)work + (size_t)b * workspace_bytes(n);
  Scratch s;
  s.Z = (cplx*)base;
  s.X = s.Z + nn;
  s.v = s.X + nn;
  s.scale = reinterpret_cast<double*>(s.v + n);
  s.uv = s.v + 2 * (size_t)n;
  s.v0 = s.uv + n;
  s.Vb = s.v0 + n;
  s.VH = s.Vb + nk;
  s.Yb = s.VH + nk;
  s.Wb = s.Yb + nk;
  s.Vt = s.Wb + nk;
  s.Tall = s.Vt + (size_t)(n > kHb ? n : kHb) * kHb;
  s.tau = (double*)(s.Tall + ((size_t)(n + kHb - 1) / kHb + 1) * kHb * kHb);
  return s;
}

// The CTAs that work on one matrix: a thread-block cluster of `size` CTAs
// (size 1: the CTA alone).  sync() is the cluster barrier, whose release and
// acquire make every CTA's global writes before it visible to all CTAs of the
// cluster after it; a lone CTA uses __syncthreads.  Every thread of every
// CTA of the team must reach each sync().
struct Team {
  int rank, size;
  __device__ void sync() const {
    if (size > 1) {
      asm volatile("barrier.cluster.arrive.release.aligned;\n" ::: "memory");
      asm volatile("barrier.cluster.wait.acquire.aligned;\n" ::: "memory");
    } else {
      __syncthreads();
    }
  }
};

__device__ __forceinline__ Team cluster_team() {
  unsigned r, s;
  asm volatile("mov.u32 %0, %%cluster_ctarank;\n" : "=r"(r));
  asm volatile("mov.u32 %0, %%cluster_nctarank;\n" : "=r"(s));
  return Team{(int)r, (int)s};
}

__device__ double block_sum(double v, double* red) {
  for (int off = 16; off > 0; off >>= 1) v += __shfl_down_sync(0xffffffffu, v, off);
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  __syncthreads();
  if (lane == 0) red[wid] = v;
  __syncthreads();
  double t = 0.0;
  for (int w = 0; w < (int)(blockDim.x >> 5); ++w) t += red[w];
  return t;
}


__device__ int block_max_int(int v, int* red) {
  for (int off = 16; off > 0; off >>= 1) v = max(v, __shfl_down_sync(0xffffffffu, v, off));
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  __syncthreads();
  if (lane == 0) red[wid] = v;
  __syncthreads();
  int t = red[0];
  for (int w = 1; w < (int)(blockDim.x >> 5); ++w) t = max(t, red[w]);
  return t;
}


// In-CTA GEMM over 64x64 tiles: D = alpha*op(A)*op(B) + beta*C (C may alias D).
// A CTA of a team takes the tiles t = rank, rank + size, ...; kL2 loads the
// operands from L2 (they may come from other CTAs of the team).
template <bool TA, bool TB, bool kL2 = false>
__device__ void cta_gemm(TileSmem& sm, int M, int N, int K, const cplx* A, int lda, const cplx* B, int ldb,
                         cplx* D, int ldd, const cplx* C, int ldc, cplx alpha, cplx beta, int rank = 0,
                         int size = 1) {
  if (M <= 0 || N <= 0) return;
  const int tm = (M + kTBM - 1) / kTBM, tn = (N + kTBN - 1) / kTBN;
  for (int t = rank; t < tm * tn; t += size) {
    const int m0 = (t / tn) * kTBM, n0 = (t % tn) * kTBN;
    cplx acc[4][4];
    tile_zero(acc);
    if (K > 0) tile_mma<TA, TB, kL2>(sm, acc, A, lda, B, ldb, nullptr, M, N, K, m0, n0);
    tile_store(acc, D, ldd, C, ldc, alpha, beta, mkc(0.0, 0.0), M, N, m0, n0);
  }
  tile_barrier();
}

// cta_gemm by the first kTileThreads threads of every CTA of a team (the
// Hessenberg kernel runs more warps than the tile routines use), the tiles
// split over the team, then a barrier over the team.
template <bool TA, bool TB, bool kTeam>
__device__ void cta_gemm_part(const Team& tm, TileSmem& sm, int M, int N, int K, const cplx* A, int lda,
                              const cplx* B, int ldb, cplx* D, int ldd, const cplx* C, int ldc, cplx alpha,
                              cplx beta) {
  if (threadIdx.x < kTileThreads) {
    if (kTeam)
      cta_gemm<TA, TB, true>(sm, M, N, K, A, lda, B, ldb, D, ldd, C, ldc, alpha, beta, tm.rank, tm.size);
    else
      cta_gemm<TA, TB>(sm, M, N, K, A, lda, B, ldb, D, ldd, C, ldc, alpha, beta);
  }
  tm.sync();
}

// Blocked Householder reduction to Hessenberg form in compact WY form, the
// scheme of LAPACK's gehrd/lahr2 (Quintana-Orti and van de Geijn, ACM TOMS
// 32(2), 2006).  For panel columns k..k+jb-1 the reflectors are generated one
// column at a time from A0 (the matrix at the panel start) corrected by
// Y = A0 V T; each column needs one product A0(:, j+1:) v_j, the only O(n^2)
// memory traffic per column.  The trailing matrix is then updated by
// A <- (I - V T^H V^H)(A - Y V^H) with tile GEMMs, and Q = prod(I - V T V^H)
// is formed backwards with tile GEMMs.  Reflectors H = I - tau v v^H are
// Hermitian with real tau; column j stores beta at (j+1, j) and the tail of
// v_j below it, v_j(j+1) = v0[j].
// A team of several CTAs (a cluster) shares the work of one matrix: the
// first CTA forms each reflector, every CTA then takes a slice of the rows of
// A0 v_j and Y, and the tiles of every GEMM are split over the team.  Each
// element is computed by the same operations as with one CTA, so the result
// does not depend on the team size.  kTeam: compiled for teams of more than
// one CTA (operands of the tile GEMMs then come from L2).
template <bool kTeam>
__device__ void hessenberg_blocked(cplx* A, int n, int lda, const Scratch& s, double* red, TileSmem& tsm,
                                   const Team& tm) {
  const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5, nw = blockDim.x >> 5;
  const int nb = kHb;
  const bool lead = tm.rank == 0;
  // this CTA's rows of the matrix-vector products (an even split point)
  const int per = ((n + tm.size - 1) / tm.size + 1) & ~1;
  const int r0 = min(n, tm.rank * per), r1 = min(n, r0 + per);
  cplx* a = s.v;    // work column, then v_j
  __shared__ cplx z[2 * kHb];
  cplx* u = s.uv;   // n
  // the panel's reflectors V and Y = A0 V T column-major (column q at q*n),
  // so that every sweep over the rows is coalesced
  cplx* Vc = s.Vb;
  cplx* Yc = s.Yb;
  // v_j in shared memory during the panel (aliases the tile buffer)
  cplx* vs = reinterpret_cast<cplx*>(&tsm);
  const bool vs_ok = (size_t)n * sizeof(cplx) <= sizeof(TileSmem);
  for (int k = 0; k + 2 < n; k += nb) {
#ifdef RCWA_EIG_STATS
    const long long c_p0 = clock64();
#endif
    const int jb = min(nb, n - 2 - k);
    cplx* T = s.Tall + (size_t)(k / nb) * nb * nb;
    if (lead)
      for (int idx = tid; idx < nb * nb; idx += blockDim.x) T[idx] = mkc(0.0, 0.0);
    for (int jj = 0; jj < jb; ++jj) {
      const int j = k + jj;
#ifdef RCWA_EIG_STATS
      long long h_t = clock64();
#define HMARK(i) do { if (tid == 0 && lead) { const long long t_ = clock64(); atomicAdd(&g_eig_stats[i], (unsigned long long)(t_ - h_t)); h_t = t_; } } while (0)
#else
#define HMARK(i) do {} while (0)
#endif
      double tau = 0.0;
      if (lead) {
        // a = A0(:, j) - Y(:, :jj) conj(V(j, :jj))
        for (int i = tid; i < n; i += blockDim.x) {
          cplx acc = A[(size_t)i * lda + j];
          for (int q = 0; q < jj; ++q) acc = cfma(cneg(Yc[(size_t)q * n + i]), cconj(Vc[(size_t)q * n + j]), acc);
          a[i] = acc;
        }
        __syncthreads();
        HMARK(16);
        if (jj > 0) {
          // a(k+1:) <- (I - V T^H V^H) a(k+1:):  z = V^H a, z = T^H z, a -= V z
          for (int q = wid; q < jj; q += nw) {
            cplx acc = mkc(0.0, 0.0);
            for (int i = k + 1 + q + lane; i < n; i += 32) acc = cfmaconj(Vc[(size_t)q * n + i], a[i], acc);
            for (int off = 16; off > 0; off >>= 1) {
              acc.x += __shfl_xor_sync(0xffffffffu, acc.x, off);
              acc.y += __shfl_xor_sync(0xffffffffu, acc.y, off);
            }
            if (lane == 0) z[q] = acc;
          }
          __syncthreads();
          if (tid < jj) {
            cplx acc = mkc(0.0, 0.0);
            for (int q = 0; q <= tid; ++q) acc = cfmaconj(T[q * nb + tid], z[q], acc);  // (T^H z)_tid
            z[nb + tid] = acc;
          }
          __syncthreads();
          for (int i = k + 1 + tid; i < n; i += blockDim.x) {
            cplx acc = a[i];
            for (int q = 0; q < jj; ++q) acc = cfma(cneg(Vc[(size_t)q * n + i]), z[nb + q], acc);
            a[i] = acc;
          }
          __syncthreads();
        }
        HMARK(17);
        // reflector from a(j+1:)
        double sig = 0.0;
        for (int i = j + 2 + tid; i < n; i += blockDim.x) sig += cnorm2(a[i]);
        sig = block_sum(sig, red);
        const cplx alpha = a[j + 1];
        cplx beta = alpha, v0 = mkc(1.0, 0.0);
        if (sig != 0.0) {
          const double aa = cabs(alpha);
          const double xnorm = sqrt(aa * aa + sig);
          const cplx ph = aa > 0.0 ? cscale(alpha, 1.0 / aa) : mkc(1.0, 0.0);
          beta = cscale(ph, -xnorm);
          v0 = cscale(ph, aa + xnorm);
          tau = 2.0 / (cnorm2(v0) + sig);
        }
        // column j of the result; explicit v_j in V(:, jj) and V^H(jj, :),
        // and in shared memory for the matrix-vector product (the tile
        // buffer is free during the panel)
        for (int i = tid; i < n; i += blockDim.x) {
          cplx vi = mkc(0.0, 0.0);
          if (i <= j) A[(size_t)i * lda + j] = a[i];
          else if (i == j + 1) { A[(size_t)i * lda + j] = beta; vi = v0; }
          else { A[(size_t)i * lda + j] = a[i]; vi = a[i]; }
          if (tau == 0.0) vi = mkc(0.0, 0.0);
          Vc[(size_t)jj * n + i] = vi;
          s.VH[(size_t)jj * n + i] = cconj(vi);
          a[i] = vi;
          if (vs_ok) vs[i] = vi;
        }
        if (tid == 0) { s.tau[j] = tau; s.v0[j] = v0; }
      }
      tm.sync();
      if (!lead) {
        // the other CTAs of the team take v_j and tau from the first
        tau = __ldcg(s.tau + j);
        if (vs_ok) {
          for (int i = tid; i < n; i += blockDim.x) vs[i] = __ldcg(a + i);
          __syncthreads();
        }
      }
      HMARK(18);
      // u = A0(:, j+1:) v_j (one pass over the trailing columns), z = V(:, :jj)^H v_j.
      // The pass is bound by the loads in flight (the trailing matrix mostly
      // comes from L2): a warp takes two rows at a time and issues all eight
      // loads of a 128-column step at once, predicated at the row end rather
      // than finished by a serial tail loop; v_j comes from shared memory.
      const cplx* vj = vs_ok ? vs : a;
      for (int i0 = r0 + 2 * wid; i0 < r1; i0 += 2 * nw) {
        const bool two = i0 + 1 < r1;
        const cplx* row0 = A + (size_t)i0 * lda;
        const cplx* row1 = two ? row0 + lda : row0;
        cplx acc0 = mkc(0.0, 0.0), acc1 = mkc(0.0, 0.0);
        for (int c = j + 1 + lane; c < n; c += 128) {
          cplx r0v[4], r1v[4], w[4];
#pragma unroll
          for (int q = 0; q < 4; ++q) {
            const int cc = c + 32 * q;
            const bool in = cc < n;
            r0v[q] = in ? row0[cc] : mkc(0.0, 0.0);
            r1v[q] = in ? row1[cc] : mkc(0.0, 0.0);
            w[q] = in ? vj[cc] : mkc(0.0, 0.0);
          }
#pragma unroll
          for (int q = 0; q < 4; ++q) {
            acc0 = cfma(r0v[q], w[q], acc0);
            acc1 = cfma(r1v[q], w[q], acc1);
          }
        }
        for (int off = 16; off > 0; off >>= 1) {
          acc0.x += __shfl_xor_sync(0xffffffffu, acc0.x, off);
          acc0.y += __shfl_xor_sync(0xffffffffu, acc0.y, off);
          acc1.x += __shfl_xor_sync(0xffffffffu, acc1.x, off);
          acc1.y += __shfl_xor_sync(0xffffffffu, acc1.y, off);
        }
        if (lane == 0) {
          u[i0] = acc0;
          if (two) u[i0 + 1] = acc1;
        }
      }
      HMARK(19);
      for (int q = wid; q < jj; q += nw) {
        cplx acc = mkc(0.0, 0.0);
        for (int i = j + 1 + lane; i < n; i += 32) acc = cfmaconj(Vc[(size_t)q * n + i], Vc[(size_t)jj * n + i], acc);
        for (int off = 16; off > 0; off >>= 1) {
          acc.x += __shfl_xor_sync(0xffffffffu, acc.x, off);
          acc.y += __shfl_xor_sync(0xffffffffu, acc.y, off);
        }
        if (lane == 0) z[q] = acc;
      }
      __syncthreads();
      HMARK(20);
      // Y(:, jj) = tau (u - Y(:, :jj) z); T(:jj, jj) = -tau T(:jj, :jj) z; T(jj, jj) = tau
      for (int i = r0 + tid; i < r1; i += blockDim.x) {
        cplx acc = u[i];
        for (int q = 0; q < jj; ++q) acc = cfma(cneg(Yc[(size_t)q * n + i]), z[q], acc);
        Yc[(size_t)jj * n + i] = cscale(acc, tau);
      }
      if (lead) {
        if (tid < jj) {
          cplx acc = mkc(0.0, 0.0);
          for (int q = tid; q < jj; ++q) acc = cfma(T[tid * nb + q], z[q], acc);
          T[tid * nb + jj] = cscale(acc, -tau);
        }
        if (tid == 0) T[jj * nb + jj] = mkc(tau, 0.0);
      }
      tm.sync();
      HMARK(21);
#undef HMARK
    }
#ifdef RCWA_EIG_STATS
    const long long c_p1 = clock64();
    if (lead) STAT_ADD(13, c_p1 - c_p0);
#endif
    // trailing columns c0..n-1
    const int c0 = k + jb;
    const int m2 = n - c0;
    if (m2 > 0) {
      // A(:, c0:) -= Y V(c0:, :)^H
      cta_gemm_part<true, false, kTeam>(tm, tsm, n, m2, jb, Yc, n, s.VH + c0, n, A + c0, lda, A + c0, lda,
                                        mkc(-1.0, 0.0), mkc(1.0, 0.0));
      // W = V(k+1:, :)^H A(k+1:, c0:)  (jb x m2), W2 = T^H W, A(k+1:, c0:) -= V(k+1:, :) W2
      cta_gemm_part<false, false, kTeam>(tm, tsm, jb, m2, n - k - 1, s.VH + k + 1, n,
                                         A + (size_t)(k + 1) * lda + c0, lda, s.Wb + c0, n, nullptr, 0,
                                         mkc(1.0, 0.0), mkc(0.0, 0.0));
      if (lead)
        for (int idx = tid; idx < nb * nb; idx += blockDim.x) {
          const int r = idx / nb, c = idx % nb;
          s.Vt[idx] = (r < jb && c < jb) ? cconj(T[c * nb + r]) : mkc(0.0, 0.0);  // T^H in Vt
        }
      tm.sync();
      cta_gemm_part<false, false, kTeam>(tm, tsm, jb, m2, jb, s.Vt, nb, s.Wb + c0, n, s.Yb + c0, n, nullptr, 0,
                                         mkc(1.0, 0.0), mkc(0.0, 0.0));
      cta_gemm_part<true, false, kTeam>(tm, tsm, n - k - 1, m2, jb, Vc + k + 1, n, s.Yb + c0, n,
                                        A + (size_t)(k + 1) * lda + c0, lda, A + (size_t)(k + 1) * lda + c0, lda,
                                        mkc(-1.0, 0.0), mkc(1.0, 0.0));
    }
#ifdef RCWA_EIG_STATS
    if (lead) STAT_ADD(14, clock64() - c_p1);
#endif
  }
#ifdef RCWA_EIG_STATS
  const long long c_q0 = clock64();
#endif
  // Z (column-major, i.e. Zt = Z^T row-major) = Q, accumulated backwards:
  // Zt(k+1:, k+1:) -= (Zt conj(V)) T^T V^T
  for (size_t idx = (size_t)r0 * n + tid; idx < (size_t)r1 * n; idx += blockDim.x)
    s.Z[idx] = mkc((idx / n) == (idx % n) ? 1.0 : 0.0, 0.0);
  tm.sync();
  const int npan = (n >= 3) ? (n - 3) / nb + 1 : 0;
  for (int pnl = npan - 1; pnl >= 0; --pnl) {
    const int k = pnl * nb;
    const int jb = min(nb, n - 2 - k);
    const cplx* T = s.Tall + (size_t)pnl * nb * nb;
    // conj(V) (n x nb, in Wb) and V^T (nb x n, in VH) from the stored reflectors
    for (int i = r0 + tid; i < r1; i += blockDim.x) {
      for (int q = 0; q < nb; ++q) {
        const int j = k + q;
        cplx vi = mkc(0.0, 0.0);
        if (q < jb && s.tau[j] != 0.0) {
          if (i == j + 1) vi = s.v0[j];
          else if (i > j + 1) vi = A[(size_t)i * lda + j];
        }
        s.Wb[(size_t)i * nb + q] = cconj(vi);
        s.VH[(size_t)q * n + i] = vi;
      }
    }
    if (lead)
      for (int idx = tid; idx < nb * nb; idx += blockDim.x) {
        const int r = idx / nb, c = idx % nb;
        s.Vt[idx] = T[c * nb + r];  // T^T
      }
    tm.sync();
    const int m = n - k - 1;
    cplx* Zs = s.Z + (size_t)(k + 1) * n + (k + 1);
    cta_gemm_part<false, false, kTeam>(tm, tsm, m, jb, m, Zs, n, s.Wb + (size_t)(k + 1) * nb, nb, s.Yb, nb,
                                       nullptr, 0, mkc(1.0, 0.0), mkc(0.0, 0.0));
    cta_gemm_part<false, false, kTeam>(tm, tsm, m, jb, jb, s.Yb, nb, s.Vt, nb, s.Vb, nb, nullptr, 0,
                                       mkc(1.0, 0.0), mkc(0.0, 0.0));
    cta_gemm_part<false, false, kTeam>(tm, tsm, m, m, jb, s.Vb, nb, s.VH + k + 1, n, Zs, n, Zs, n,
                                       mkc(-1.0, 0.0), mkc(1.0, 0.0));
  }
  for (size_t idx = (size_t)r0 * n + tid; idx < (size_t)r1 * n; idx += blockDim.x) {
    const int i = (int)(idx / n), j = (int)(idx % n);
    if (i > j + 1) A[(size_t)i * lda + j] = mkc(0.0, 0.0);
  }
  tm.sync();
#ifdef RCWA_EIG_STATS
  if (lead) STAT_ADD(15, clock64() - c_q0);
#endif
}

// ---------------------------------------------------------------- QR
// Rotation [c s; -conj(s) c] (c real) with G [x; y] = [r; 0]:
// c = |x| / |(x, y)|, s = x conj(y) / (|x| |(x, y)|), from one reciprocal
// square root of |x|^2 |(x, y)|^2 and a Newton step towards c^2 + |s|^2 = 1
// (with it the residuals of the eigenpairs are 2-4% below, without it 9% above
// those of two reciprocal square roots; random matrices of order 40-450).
// Inputs whose squares could leave the normal range are scaled by a power of
// two first (exact), out of line: the scaling alone (frexp, ldexp) takes as
// many cycles as the rest of the rotation, which is the serial step of every
// QR sweep.
__device__ __noinline__ void givens_scaled(cplx x, cplx y, double& c, cplx& s) {
  if (y.x == 0.0 && y.y == 0.0) { c = 1.0; s = mkc(0.0, 0.0); return; }
  const double m = fmax(fmax(fabs(x.x), fabs(x.y)), fmax(fabs(y.x), fabs(y.y)));
  int e;
  frexp(m, &e);
  const double sc = ldexp(1.0, -e);
  x = cscale(x, sc);
  y = cscale(y, sc);
  const double ax2 = cnorm2(x);
  if (ax2 == 0.0) { c = 0.0; s = mkc(1.0, 0.0); return; }
  const double ra = rsqrt(ax2), rr = rsqrt(ax2 + cnorm2(y));
  c = ax2 * ra * rr;
  s = cscale(cmul(x, cconj(y)), ra * rr);
}
__device__ __forceinline__ void givens_fast(cplx x, cplx y, double& c, cplx& s) {
  const double ax2 = cnorm2(x), r2 = ax2 + cnorm2(y);
  if (ax2 > 0x1p-400 && r2 < 0x1p400) {
    const double q = rsqrt(ax2 * r2);
    c = ax2 * q;
    s = cscale(cmul(x, cconj(y)), q);
    // one Newton step towards c^2 + |s|^2 = 1
    const double h = 0.5 * fma(-s.y, s.y, fma(-s.x, s.x, fma(-c, c, 1.0)));
    c = fma(c, h, c);
    s = mkc(fma(s.x, h, s.x), fma(s.y, h, s.y));
  } else {
    givens_scaled(x, y, c, s);
  }
}

// Negligible subdiagonal T(k,k-1) inside the active block [l, i]:
// the standard relative test refined by the criterion of Ahues and Tisseur
// (LAPACK Working Note 122, 1997).
__device__ bool negligible(const cplx* T, int ldt, int k, int l, int i, double ulp, double smlnum) {
  const cplx h = T[(size_t)k * ldt + k - 1];
  const double ah = cabs1(h);
  if (ah <= smlnum) return true;
  const cplx hkk = T[(size_t)k * ldt + k], hk1 = T[(size_t)(k - 1) * ldt + k - 1];
  double tst = cabs1(hk1) + cabs1(hkk);
  if (tst == 0.0) {
    if (k - 2 >= l) tst += cabs1(T[(size_t)(k - 1) * ldt + k - 2]);
    if (k + 1 <= i) tst += cabs1(T[(size_t)(k + 1) * ldt + k]);
  }
  if (ah <= ulp * tst) {
    const double up = cabs1(T[(size_t)(k - 1) * ldt + k]);
    const double ab = fmax(ah, up), ba = fmin(ah, up);
    const double d1 = cabs1(hkk), d2 = cabs1(csub(hk1, hkk));
    const double aa = fmax(d1, d2), bb = fmin(d1, d2);
    const double sc = aa + ab;
    if (ba * (ab / sc) <= fmax(smlnum, ulp * (bb * (aa / sc)))) return true;
  }
  return false;
}

// Eigenvalue of the trailing 2x2 [[a, b], [c, d]] closest to d:
// d - b*c / (delta + r), delta = (a - d)/2, r = sqrt(delta^2 + b*c) taken on
// the side of delta so that the denominator does not cancel.
__device__ cplx wilkinson_shift(cplx a, cplx b, cplx c, cplx d) {
  const cplx bc = cmul(b, c);
  const double sbc = cabs1(bc);
  if (sbc == 0.0) return d;
  const cplx delta = cscale(csub(a, d), 0.5);
  const double sc = fmax(cabs1(delta), sqrt(sbc));
  const cplx ds = cscale(delta, 1.0 / sc);
  cplx r = csqrt_principal(cadd(cmul(ds, ds), cscale(bc, 1.0 / (sc * sc))));
  r = cscale(r, sc);
  if (delta.x * r.x + delta.y * r.y < 0.0) r = cneg(r);
  const cplx den = cadd(delta, r);
  if (den.x == 0.0 && den.y == 0.0) return d;
  return csub(d, cdiv(bc, den));
}

__device__ void qr_sweep(cplx* T, int ldt, cplx* Z, int n, int l, int i, cplx shift,
                         cplx (*Wt)[kWin + 1], double* rc, cplx* rs) {
  const int tid = threadIdx.x;
  int k = l, ws = l;
  while (k <= i - 1) {
    const int we = min(ws + kWin - 1, i);
    const int ke = (we == i) ? i - 1 : we - 2;
    const int w = we - ws + 1;
    for (int idx = tid; idx < w * w; idx += blockDim.x)
      Wt[idx / w][idx % w] = T[(size_t)(ws + idx / w) * ldt + ws + idx % w];
    __syncthreads();
    if (tid < 32) {
      const int lane = tid;
      for (int r = k; r <= ke; ++r) {
        cplx x, y;
        if (r == l) {
          x = csub(Wt[r - ws][r - ws], shift);
          y = Wt[r + 1 - ws][r - ws];
        } else {
          x = Wt[r - ws][r - 1 - ws];
          y = Wt[r + 1 - ws][r - 1 - ws];
        }
        double c;
        cplx sn;
        givens_fast(x, y, c, sn);
        const int j0 = (r == l) ? r : r - 1;
        const int jj = j0 - ws + lane;
        if (jj < w) {
          const cplx a = Wt[r - ws][jj], b = Wt[r + 1 - ws][jj];
          Wt[r - ws][jj] = cfma(sn, b, cscale(a, c));
          Wt[r + 1 - ws][jj] = cfma(cneg(cconj(sn)), a, cscale(b, c));
        }
        __syncwarp();
        if (lane == 0 && r > l) Wt[r + 1 - ws][r - 1 - ws] = mkc(0.0, 0.0);
        const int iend = min(r + 2, i) - ws;
        if (lane <= iend) {
          const cplx a = Wt[lane][r - ws], b = Wt[lane][r + 1 - ws];
          Wt[lane][r - ws] = cfma(cconj(sn), b, cscale(a, c));
          Wt[lane][r + 1 - ws] = cfma(cneg(sn), a, cscale(b, c));
        }
        __syncwarp();
        if (lane == 0) { rc[r - k] = c; rs[r - k] = sn; }
      }
    }
    __syncthreads();
    for (int idx = tid; idx < w * w; idx += blockDim.x)
      T[(size_t)(ws + idx / w) * ldt + ws + idx % w] = Wt[idx / w][idx % w];
    // deferred application of rotations k..ke outside the window
    const int nrot = ke - k + 1;
    const int nright = n - 1 - we;
    const int nup = ws;
    const int ntask = nright + nup + n;
    for (int t = tid; t < ntask; t += blockDim.x) {
      if (t < nright) {
        const int j = we + 1 + t;
        cplx x = T[(size_t)k * ldt + j];
        for (int q = 0; q < nrot; ++q) {
          const cplx y = T[(size_t)(k + q + 1) * ldt + j];
          const double c = rc[q];
          const cplx sn = rs[q];
          T[(size_t)(k + q) * ldt + j] = cfma(sn, y, cscale(x, c));
          x = cfma(cneg(cconj(sn)), x, cscale(y, c));
        }
        T[(size_t)(k + nrot) * ldt + j] = x;
      } else if (t < nright + nup) {
        const int ii = t - nright;
        cplx* row = T + (size_t)ii * ldt;
        cplx x = row[k];
        for (int q = 0; q < nrot; ++q) {
          const cplx y = row[k + q + 1];
          const double c = rc[q];
          const cplx sn = rs[q];
          row[k + q] = cfma(cconj(sn), y, cscale(x, c));
          x = cfma(cneg(sn), x, cscale(y, c));
        }
        row[k + nrot] = x;
      } else {
        const int ii = t - nright - nup;
        cplx x = Z[(size_t)k * n + ii];
        for (int q = 0; q < nrot; ++q) {
          const cplx y = Z[(size_t)(k + q + 1) * n + ii];
          const double c = rc[q];
          const cplx sn = rs[q];
          Z[(size_t)(k + q) * n + ii] = cfma(cconj(sn), y, cscale(x, c));
          x = cfma(cneg(sn), x, cscale(y, c));
        }
        Z[(size_t)(k + nrot) * n + ii] = x;
      }
    }
    __syncthreads();
    ws = ke;
    k = ke + 1;
  }
}

// ---------------------------------------------------------------- Schur form of a small matrix
// Matrices of at most kBlkMax rows: the whole matrix in shared memory, small-
// bulge multishift sweeps of up to kBlkShifts bulges three rows apart, two
// warps per bulge.  The first evaluates the rotation (every lane the same
// arithmetic on a broadcast read) and updates the bulge's rows of T, then
// after a barrier its columns, while the second applies the previous barrier's
// rotation to the Schur vectors: a chain passes column p + 1 from one rotation
// to the next in registers and fetches column p + 2 a step ahead, so Z stays
// in global memory (L1/L2) and leaves the shared memory to T (5 CTAs per SM at
// order 50).  The shifts are the two eigenvalues of the trailing 2 x 2 block; a
// sweep of four uses each twice (near convergence the second pair still gains
// a factor of the error, and it costs no extra steps).
//
// Bound by the serial latency of a chain step (the rotation, two barriers),
// which this pays once for up to kBlkShifts rotations and without memory in
// the chain; single-shift sweeps over a 32-row window with the rest of T and
// Z updated in global memory took 2.58 ms for one matrix of order 50 (B200).
constexpr int kBlkMax = 116;
constexpr int kBlkShifts = 4;
constexpr int kBlkThreads = 64 * kBlkShifts;

__host__ __device__ constexpr int blk_ld(int n) { return n | 1; }  // odd pitch: conflict-free columns
constexpr size_t blk_smem(int n) { return sizeof(cplx) * (size_t)n * blk_ld(n); }
static_assert(blk_smem(kBlkMax) <= 230000, "the block must fit beside the kernel's static shared memory");

// T: n x n upper Hessenberg in shared memory, pitch ld; Z: column-major in
// global memory (Z(r, c) = Z[c*n + r]); n <= 32 Q.  Whole CTA; every warp takes
// the same decisions from the same data.  Returns 0 or RCWA_ERR_NOCONV.
template <int Q>
__device__ int schur_block(cplx* T, int ld, cplx* Z, int n, int sweep_cap) {
  __shared__ cplx s_sn[kBlkShifts];
  __shared__ double s_c[kBlkShifts];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int b = warp >> 1;            // this warp's bulge
  const bool lead = (warp & 1) == 0;  // rotation and T; else Z
  const double ulp = 2.0 * RCWA_DBL_EPS;
  const double smlnum = RCWA_DBL_MIN * ((double)n / ulp);
  const int budget = sweep_cap > 0 ? min(30 * max(10, n), sweep_cap) : 30 * max(10, n);
  int hi = n - 1, its = 0;
  for (int total = 0; hi >= 0;) {
    __syncthreads();
    int lo = 0;
#pragma unroll
    for (int q = 0; q < Q; ++q) {
      const int k = lane + 32 * q;
      const unsigned m = __ballot_sync(0xffffffffu, k >= 1 && k <= hi && negligible(T, ld, k, 0, hi, ulp, smlnum));
      if (m) lo = 32 * q + 31 - __clz(m);
    }
    // every warp has read the subdiagonal before one thread clears an entry
    __syncthreads();
    if (lo > 0 && threadIdx.x == 0) T[lo * ld + lo - 1] = mkc(0.0, 0.0);
    if (lo == hi) {
      --hi;
      its = 0;
      continue;
    }
    if (++total > budget) return RCWA_ERR_NOCONV;
    const int m = hi - lo + 1;
    const int s = m < 4 ? 1 : m < 8 ? 2 : kBlkShifts;
    cplx sh;
    if (its == 10 || its == 30) {
      sh = cadd(T[lo * ld + lo], mkc(0.75 * cabs1(T[(lo + 1) * ld + lo]), 0.0));
    } else if (its == 20 || its == 40) {
      sh = cadd(T[hi * ld + hi], mkc(0.75 * cabs1(T[hi * ld + hi - 1]), 0.0));
    } else {
      const cplx ta = T[(hi - 1) * ld + hi - 1], td = T[hi * ld + hi];
      sh = wilkinson_shift(ta, T[(hi - 1) * ld + hi], T[hi * ld + hi - 1], td);
      if (b & 1) sh = csub(cadd(ta, td), sh);  // the other eigenvalue
    }
    ++its;
    __syncthreads();
    const int tend = (hi - lo) + 3 * (s - 1);
    cplx zx[Q], zy[Q];  // Z warps: columns p and p + 1
#pragma unroll
    for (int q = 0; q < Q; ++q) zx[q] = zy[q] = mkc(0.0, 0.0);
    for (int t = 0; t < tend; ++t) {
      const int p = lo + t - 3 * b;
      const bool on = b < s && p >= lo && p <= hi - 1;
      double c = 1.0;
      cplx sn = mkc(0.0, 0.0);
      if (lead) {
        if (on) {
          cplx* const r0 = T + p * ld;
          cplx* const r1 = r0 + ld;
          const int j0 = (p == lo ? p : p - 1) + lane;
          cplx x, y, ra[Q], rb[Q];
          if (p == lo) { x = csub(r0[p], sh); y = r1[p]; }
          else { x = r0[p - 1]; y = r1[p - 1]; }
#pragma unroll
          for (int q = 0; q < Q; ++q)
            if (j0 + 32 * q < n) { ra[q] = r0[j0 + 32 * q]; rb[q] = r1[j0 + 32 * q]; }
          givens_fast(x, y, c, sn);
          __syncwarp();
#pragma unroll
          for (int q = 0; q < Q; ++q) {
            const int j = j0 + 32 * q;
            if (j < n) {
              r0[j] = cfma(sn, rb[q], cscale(ra[q], c));
              r1[j] = j < p ? mkc(0.0, 0.0) : cfma(cneg(cconj(sn)), ra[q], cscale(rb[q], c));
            }
          }
          if (lane == 0) { s_c[b] = c; s_sn[b] = sn; }
        }
      } else if (b < s && p == lo) {
        // the bulge behind left these columns two and three steps ago
#pragma unroll
        for (int q = 0; q < Q; ++q)
          if (lane + 32 * q < n) {
            zx[q] = Z[(size_t)p * n + lane + 32 * q];
            zy[q] = Z[(size_t)(p + 1) * n + lane + 32 * q];
          }
      }
      __syncthreads();
      if (on) {
        if (lead) {
          cplx* const col = T + p;
          const int rn = min(p + 2, hi);
#pragma unroll
          for (int q = 0; q < Q; ++q) {
            const int r = lane + 32 * q;
            if (r <= rn) {
              const cplx x = col[r * ld], y = col[r * ld + 1];
              col[r * ld] = cfma(cconj(sn), y, cscale(x, c));
              col[r * ld + 1] = cfma(cneg(sn), x, cscale(y, c));
            }
          }
        } else {
          c = s_c[b];
          sn = s_sn[b];
          const bool last = p == hi - 1;
#pragma unroll
          for (int q = 0; q < Q; ++q) {
            const int r = lane + 32 * q;
            if (r < n) {
              Z[(size_t)p * n + r] = cfma(cconj(sn), zy[q], cscale(zx[q], c));
              zx[q] = cfma(cneg(sn), zx[q], cscale(zy[q], c));
              if (last) Z[(size_t)(p + 1) * n + r] = zx[q];
              else zy[q] = Z[(size_t)(p + 2) * n + r];
            }
          }
        }
      }
      __syncthreads();
    }
  }
  __syncthreads();
  return 0;
}

// ---------------------------------------------------------------- multishift QR
// Small-bulge multishift QR (the scheme of Braman, Byers and Mathias, SIAM J.
// Matrix Anal. Appl. 23(4), 2002) for complex Hessenberg matrices.  A sweep
// chases a chain of s single-shift bulges, three rows apart, from the top to
// the bottom of the active block.  The chain advances inside a W x W window
// held in shared memory, one warp per bulge (their row pairs and column pairs
// are disjoint), so a chain step costs two barriers.  Every rotation is
// logged; after a window pass the log is applied to the rest of T (the rows
// right of the window, the columns above it) and to Z, one line of 32 per
// warp task, with the part of each line the chain spans held in registers
// (replay_frame), so an element of T or Z crosses memory once per pass
// instead of once per rotation.
//
// What bounds it (order 882, one matrix per SM, cycle counters of a lone
// matrix, 64-row window and 16-row early deflation): the replay 191 of 298 ms,
// at 7.0 cycles per rotation of 32 lines and SM against 6 of its eight
// FP64 instructions alone; then the serial latency of the chase (51 ms) and of
// the early deflation (54 ms).  With every rotation at 12 FP64 instructions, a
// register shift per step and the chase's rotations on ten threads the same
// matrix took 404 ms.  Schur stage of whole batches (window 64 / 72 / 100, early
// deflation 16): 145 x 882 335 / 325 / 372 ms, 148 x 450 80 / 78 / 89 ms; ten
// shifts (the frame spills) 537 ms, six 468 ms at 145 x 882.  As built (window
// 72, early deflation 12) 330 and 77 ms.
#ifndef RCWA_MS_WINDOW
#define RCWA_MS_WINDOW 72
#endif
constexpr int kMsW = RCWA_MS_WINDOW;  // window order (a build-time parameter)
#ifndef RCWA_MS_SHIFTS
#define RCWA_MS_SHIFTS 8
#endif
constexpr int kMsShifts = RCWA_MS_SHIFTS;  // bulges per sweep (a build-time parameter)
constexpr int kMsMin = kSchurCrossover;  // smallest crossover
constexpr int kMsThreads = 32 * kMsShifts;  // a warp per bulge in the chase, all of them in the replay
constexpr int kMsLd = kMsW + 1;
constexpr int kMsFrame = 3 * (kMsShifts - 1) + 2;  // indices the chain spans
constexpr int kMsPre = 4;                          // replay steps per unrolled group
// chain steps of one window pass, rounded up to whole replay groups
constexpr int kMsMaxSteps = (kMsW + 3 * kMsShifts + kMsPre - 1) / kMsPre * kMsPre;
static_assert(kMsW % 2 == 0, "an odd window pitch keeps column accesses conflict free");

struct MsSmem {
  cplx* Wt;      // [kMsW][kMsLd]  the chase window
  cplx* work;    // early deflation's window, vectors and reflector; the small shift problem
  cplx* log;     // [kMsMaxSteps][kMsShifts][2]  replay coefficients per chain step and bulge
  double* lc;    // [kMsMaxSteps][kMsShifts]  rotation cosines
  double* dfin;  // [kMsW]  scale of every window index after the pass
  cplx* shifts;  // [kMsShifts]
  int* redi;     // [kMsThreads / 32]
  int* aed;      // [4] early-deflation results: converged flag, undeflated count, shift count
};

// the window is only used by the chase, the work area only by the early
// deflation and the shift computation between sweeps: they share one region
constexpr size_t kMsRegion = sizeof(cplx) * kMsW * kMsLd;
constexpr size_t kMsSmemBytes = kMsRegion + 2 * sizeof(cplx) * kMsMaxSteps * kMsShifts +
                                sizeof(double) * (kMsMaxSteps * kMsShifts + kMsW) + sizeof(cplx) * kMsShifts +
                                sizeof(int) * (kMsThreads / 32 + 4);
static_assert(kMsSmemBytes <= 232448, "multishift shared memory exceeds the per-block limit");

__device__ MsSmem carve_ms_smem(unsigned char* base) {
  MsSmem sm;
  sm.Wt = (cplx*)base;
  sm.work = (cplx*)base;
  sm.log = (cplx*)(base + kMsRegion);
  sm.shifts = sm.log + 2 * kMsMaxSteps * kMsShifts;
  sm.lc = (double*)(sm.shifts + kMsShifts);
  sm.dfin = sm.lc + kMsMaxSteps * kMsShifts;
  sm.redi = (int*)(sm.dfin + kMsW);
  sm.aed = sm.redi + kMsThreads / 32;
  return sm;
}

// the multishift kernel's dynamic shared memory (the replay is a function of
// its own, so that its frame has the registers to itself)
extern __shared__ __align__(16) unsigned char ms_dsm[];

#define MSW(r, c) sm.Wt[(r) * kMsLd + (c)]

// Eigenvalues of the s x s upper Hessenberg matrix B (row stride ldb) by
// single-shift QR without vectors; one warp.  Unconverged remainders after
// the iteration budget are returned as their diagonal entries.
__device__ void small_eigs_warp(cplx* B, int ldb, int s, cplx* out) {
  const int lane = threadIdx.x & 31;
  const double ulp = 2.0 * RCWA_DBL_EPS;
  int hi = s - 1, its = 0;
  while (hi >= 0) {
    int lo = 0;
    for (int k = hi; k >= 1; --k) {
      const double h = cabs1(B[k * ldb + k - 1]);
      if (h <= ulp * (cabs1(B[(k - 1) * ldb + k - 1]) + cabs1(B[k * ldb + k])) || h < RCWA_DBL_MIN) {
        lo = k;
        break;
      }
    }
    if (lo == hi || its > 60) {
      for (int k = lo + lane; k <= hi; k += 32) out[k] = B[k * ldb + k];
      __syncwarp();
      hi = lo - 1;
      its = 0;
      continue;
    }
    cplx sh;
    if (its == 10 || its == 20) sh = cadd(B[hi * ldb + hi], mkc(0.75 * cabs1(B[hi * ldb + hi - 1]), 0.0));
    else sh = wilkinson_shift(B[(hi - 1) * ldb + hi - 1], B[(hi - 1) * ldb + hi], B[hi * ldb + hi - 1], B[hi * ldb + hi]);
    for (int r = lo; r < hi; ++r) {
      cplx x, y;
      if (r == lo) { x = csub(B[lo * ldb + lo], sh); y = B[(lo + 1) * ldb + lo]; }
      else { x = B[r * ldb + r - 1]; y = B[(r + 1) * ldb + r - 1]; }
      double c;
      cplx sn;
      givens_fast(x, y, c, sn);
      __syncwarp();
      const int j = ((r == lo) ? r : r - 1) + lane;
      if (j <= hi) {
        const cplx a = B[r * ldb + j], b = B[(r + 1) * ldb + j];
        B[r * ldb + j] = cfma(sn, b, cscale(a, c));
        B[(r + 1) * ldb + j] = cfma(cneg(cconj(sn)), a, cscale(b, c));
      }
      __syncwarp();
      if (r > lo && lane == 0) B[(r + 1) * ldb + r - 1] = mkc(0.0, 0.0);
      const int row = lo + lane;
      if (row <= min(r + 2, hi)) {
        const cplx a = B[row * ldb + r], b = B[row * ldb + r + 1];
        B[row * ldb + r] = cfma(cconj(sn), b, cscale(a, c));
        B[row * ldb + r + 1] = cfma(cneg(sn), a, cscale(b, c));
      }
      __syncwarp();
    }
    ++its;
  }
}

// ---------------------------------------------------------------- aggressive early deflation
// Aggressive early deflation (Braman, Byers and Mathias, SIAM J. Matrix Anal.
// Appl. 23(4), 2002; the complex variant of LAPACK's zlaqr3): the trailing
// kAedW x kAedW window of the active block is brought to Schur form with its
// unitary V; the spike s*conj(V(0,:)) that couples it to the rest tells which
// window eigenvalues have converged.  Converged ones at the bottom are
// deflated, the others are moved to the top by adjacent swaps and serve as
// shifts; the spike of the undeflated part is reflected onto its first entry
// and that part is returned to Hessenberg form by Householder reflectors.
// The window's one-warp Schur form is serial, so a smaller window is cheaper
// per call and deflates less: Schur stage with windows of 16 / 14 / 12 (64-row
// chase window) 145 x 882 335 / 346 / 342 ms, 148 x 450 80 / 81 / 75 ms, 74 x
// 198 19.6 / 18.8 / 16.3 ms; one size serves all orders, and 12 costs order 882
// 2%.  A 32-row window on all warps cut the sweeps by 20% but cost 60 + 35 ms for
// its Schur form and reordering at order 882.
#ifndef RCWA_AED_WINDOW
#define RCWA_AED_WINDOW 12
#endif
constexpr int kAedW = RCWA_AED_WINDOW;  // window order (a build-time parameter)
static_assert(kAedW <= 16 && kAedW >= kMsShifts + 2, "a half warp per row of the early-deflation window and of V");
constexpr int kAedLd = kAedW + 1;
constexpr int kAedNibble = 14;   // percent of the window deflated that skips the sweep
static_assert(sizeof(cplx) * (2 * kAedW * kAedLd + kAedW) <= kMsRegion &&
                  sizeof(cplx) * kMsShifts * (kMsShifts + 1) <= kMsRegion && sizeof(cplx) * kWin * (kWin + 1) <= kMsRegion,
              "the work areas must fit in the chase window's region");

#define AW(r, c) W[(r) * kAedLd + (c)]
#define AV(r, c) V[(r) * kAedLd + (c)]

// Schur form of the Hessenberg window W (nw x nw) with V <- V G^H for every
// rotation G; single-shift QR by one warp, lanes 0-15 on W and lanes 16-31 on
// V.  Returns false when the iteration budget runs out.
__device__ bool aed_window_schur(cplx* W, cplx* V, int nw) {
  const int lane = threadIdx.x & 31, idx = lane & 15;
  const bool wl = lane < 16;
  const double ulp = 2.0 * RCWA_DBL_EPS;
  cplx* const col = wl ? W : V;  // this lane's row of W or V in the column updates
  int hi = nw - 1, its = 0, total = 0;
  while (hi >= 0) {
    __syncwarp();
    bool defl = false;
    if (lane >= 1 && lane <= hi) {
      const double h = cabs1(AW(lane, lane - 1));
      defl = h <= ulp * (cabs1(AW(lane - 1, lane - 1)) + cabs1(AW(lane, lane))) || h < RCWA_DBL_MIN;
    }
    const unsigned mask = __ballot_sync(0xffffffffu, defl);
    const int lo = mask ? 31 - __clz(mask) : 0;
    __syncwarp();
    if (lo == hi) {
      if (hi > 0 && lane == 0) AW(hi, hi - 1) = mkc(0.0, 0.0);
      --hi;
      its = 0;
      continue;
    }
    if (lo > 0 && lane == 0) AW(lo, lo - 1) = mkc(0.0, 0.0);
    if (++total > 30 * nw) return false;
    cplx sh;
    if (its == 10) sh = cadd(AW(lo, lo), mkc(0.75 * cabs1(AW(lo + 1, lo)), 0.0));
    else if (its == 20) sh = cadd(AW(hi, hi), mkc(0.75 * cabs1(AW(hi, hi - 1)), 0.0));
    else sh = wilkinson_shift(AW(hi - 1, hi - 1), AW(hi - 1, hi), AW(hi, hi - 1), AW(hi, hi));
    __syncwarp();
    for (int p = lo; p < hi; ++p) {
      cplx x, y;
      if (p == lo) { x = csub(AW(lo, lo), sh); y = AW(lo + 1, lo); }
      else { x = AW(p, p - 1); y = AW(p + 1, p - 1); }
      const bool row = wl && idx >= (p == lo ? p : p - 1) && idx < nw;
      cplx a = mkc(0.0, 0.0), b = mkc(0.0, 0.0);
      if (row) { a = AW(p, idx); b = AW(p + 1, idx); }
      double c;
      cplx sn;
      givens_fast(x, y, c, sn);
      __syncwarp();
      if (row) {
        AW(p, idx) = cfma(sn, b, cscale(a, c));
        AW(p + 1, idx) = idx < p ? mkc(0.0, 0.0) : cfma(cneg(cconj(sn)), a, cscale(b, c));
      }
      __syncwarp();
      if (idx <= (wl ? min(p + 2, hi) : nw - 1)) {
        a = col[idx * kAedLd + p];
        b = col[idx * kAedLd + p + 1];
        col[idx * kAedLd + p] = cfma(cconj(sn), b, cscale(a, c));
        col[idx * kAedLd + p + 1] = cfma(cneg(sn), a, cscale(b, c));
      }
      __syncwarp();
    }
    ++its;
  }
  __syncwarp();
  return true;
}

// Swap the adjacent eigenvalues k, k+1 of the upper triangular W (LAPACK
// ztrexc step): G from (W(k,k+1), W(k+1,k+1) - W(k,k)) applied to rows
// k, k+1 right of the pair, to columns k, k+1 above it and to V; the
// diagonal entries trade places and W(k,k+1) keeps its value.  One warp: the
// three updates touch disjoint entries, lanes 0-15 take those of W and lanes
// 16-31 those of V.
__device__ void aed_swap(cplx* W, cplx* V, int nw, int k) {
  const int lane = threadIdx.x & 31, idx = lane & 15;
  const bool wl = lane < 16, row = wl && idx >= k + 2 && idx < nw, cl = wl ? idx < k : idx < nw;
  cplx* const pa = row ? &AW(k, idx) : wl ? &AW(idx, k) : &AV(idx, k);
  cplx* const pb = row ? &AW(k + 1, idx) : pa + 1;
  const cplx t11 = AW(k, k), t22 = AW(k + 1, k + 1);
  cplx a = mkc(0.0, 0.0), b = mkc(0.0, 0.0);
  if (row || cl) { a = *pa; b = *pb; }
  double c;
  cplx sn;
  givens_fast(AW(k, k + 1), csub(t22, t11), c, sn);
  __syncwarp();
  if (!row) sn = cconj(sn);
  if (row || cl) {
    *pa = cfma(sn, b, cscale(a, c));
    *pb = cfma(cneg(cconj(sn)), a, cscale(b, c));
  }
  if (lane == 0) { AW(k, k) = t22; AW(k + 1, k + 1) = t11; }
  __syncwarp();
}

// Householder reflector H = I - tau v v^H with H^H x = beta e1 for the
// vector x[0..len) in shared memory (LAPACK zlarfg convention: v[0] = 1,
// tau = (beta - alpha)/beta, beta = -sign(Re alpha) ||x||); v overwrites x.
// One warp; returns tau (zero when x is already beta e1).
__device__ cplx aed_house(cplx* x, int len) {
  const int lane = threadIdx.x & 31;
  double part = (lane >= 1 && lane < len) ? cnorm2(x[lane]) : 0.0;
  for (int off = 16; off > 0; off >>= 1) part += __shfl_xor_sync(0xffffffffu, part, off);
  const cplx alpha = x[0];
  __syncwarp();
  if (part == 0.0 && alpha.y == 0.0) return mkc(0.0, 0.0);
  const double beta = -copysign(sqrt(cnorm2(alpha) + part), alpha.x);
  const cplx tau = mkc((beta - alpha.x) / beta, -alpha.y / beta);
  const cplx scal = cdiv(mkc(1.0, 0.0), csub(alpha, mkc(beta, 0.0)));
  if (lane >= 1 && lane < len) x[lane] = cmul(x[lane], scal);
  if (lane == 0) x[0] = mkc(beta, 0.0);  // beta kept in x[0]; v[0] = 1 implied
  __syncwarp();
  return tau;
}

// M(r0 + r, c) -= conj(tau) v[r] (v^H M(r0.., c)) for columns c in [c0, nw):
// the left product H^H M on rows r0 .. r0+len-1; v[0] = 1.  One warp.
__device__ void aed_left(cplx* M, const cplx* v, int len, cplx tau, int r0, int c0, int nw) {
  const int lane = threadIdx.x & 31;
  if (lane >= c0 && lane < nw) {
    cplx w = M[r0 * kAedLd + lane];
    for (int r = 1; r < len; ++r) w = cfmaconj(v[r], M[(r0 + r) * kAedLd + lane], w);
    const cplx f = cmul(cconj(tau), w);
    M[r0 * kAedLd + lane] = csub(M[r0 * kAedLd + lane], f);
    for (int r = 1; r < len; ++r) M[(r0 + r) * kAedLd + lane] = csub(M[(r0 + r) * kAedLd + lane], cmul(v[r], f));
  }
  __syncwarp();
}

// M(r, c0 + c) -= tau (M(r, c0..) v) conj(v[c]) for rows r < rows: the right
// product M H on columns c0 .. c0+len-1; v[0] = 1.  One warp.
__device__ void aed_right(cplx* M, const cplx* v, int len, cplx tau, int rows, int c0) {
  const int lane = threadIdx.x & 31;
  if (lane < rows) {
    cplx w = M[lane * kAedLd + c0];
    for (int c = 1; c < len; ++c) w = cfma(M[lane * kAedLd + c0 + c], v[c], w);
    const cplx f = cmul(tau, w);
    M[lane * kAedLd + c0] = csub(M[lane * kAedLd + c0], f);
    for (int c = 1; c < len; ++c)
      M[lane * kAedLd + c0 + c] = csub(M[lane * kAedLd + c0 + c], cmul(f, cconj(v[c])));
  }
  __syncwarp();
}

// Aggressive early deflation on the active block [l, i].  A block of at most
// kAedW rows is the window itself: it has no spike, so its Schur form deflates
// all of it.  Returns the number of deflated eigenvalues (0 when none, -1 when the window
// did not converge and nothing was changed).  On return sm.shifts[0..cnt)
// hold the bottom undeflated window eigenvalues, cnt <= kMsShifts, in
// sm.aed[2].  Whole CTA.
// With a team of several CTAs every CTA computes the window's Schur form
// (the same operations on the same data), the first CTA's outcome is taken
// by all (ctrl[2..4]), the first CTA writes the window back and the
// off-window updates are split over the team.  *shift_count receives the
// number of shifts left in sm.shifts.
__device__ int aed(cplx* T, int ldt, cplx* Z, int n, int l, int i, const MsSmem& sm, const Team& tm, int* ctrl,
                   int* shift_count) {
  const int tid = threadIdx.x, nthr = blockDim.x;
  const bool lead = tm.rank == 0;
  const int stride = nthr * tm.size, off0 = tid + nthr * tm.rank;
  const int nw = min(kAedW, i - l + 1);
  const int kw = i - nw + 1;
  cplx* W = sm.work;
  cplx* V = W + kAedW * kAedLd;
  cplx* hv = V + kAedW * kAedLd;
  const double ulp = 2.0 * RCWA_DBL_EPS;
  const double smlnum = RCWA_DBL_MIN * ((double)n / ulp);
  for (int idx = tid; idx < kAedW * kAedW; idx += nthr) {
    const int r = idx / kAedW, c = idx % kAedW;
    if (r < nw && c < nw) AW(r, c) = T[(size_t)(kw + r) * ldt + kw + c];
    AV(r, c) = mkc(r == c && r < nw ? 1.0 : 0.0, 0.0);
  }
  const cplx s = kw > l ? T[(size_t)kw * ldt + kw - 1] : mkc(0.0, 0.0);
  __syncthreads();
  // every CTA holds the window before the first one writes it back
  if (tm.size > 1) tm.sync();
  if (tid < 32) {
    const int lane = tid;
#ifdef RCWA_EIG_STATS
    long long c_w0 = clock64();
#endif
    const bool ok = aed_window_schur(W, V, nw);
#ifdef RCWA_EIG_STATS
    if (lane == 0) { const long long c_w1 = clock64(); atomicAdd(&g_eig_stats[5], (unsigned long long)(c_w1 - c_w0)); c_w0 = c_w1; }
#endif
    int ns = nw;
    if (ok) {
      // deflation test from the bottom, undeflatable eigenvalues moved up
      int ilst = 0;
      const double as = cabs1(s);
      for (int knt = 0; knt < nw && ns > ilst; ++knt) {
        double foo = cabs1(AW(ns - 1, ns - 1));
        if (foo == 0.0) foo = as;
        if (as * cabs1(AV(0, ns - 1)) <= fmax(smlnum, ulp * foo)) {
          --ns;
        } else {
          for (int k = ns - 2; k >= ilst; --k) aed_swap(W, V, nw, k);
          ++ilst;
        }
      }
      // shifts: the bottom undeflated eigenvalues, before the reflection
      const int cnt = min(ns, kMsShifts);
      if (lane < cnt) sm.shifts[lane] = AW(ns - cnt + lane, ns - cnt + lane);
      if (lane == 0) sm.aed[2] = cnt;
      __syncwarp();
      if (ns < nw && ns > 1 && (s.x != 0.0 || s.y != 0.0)) {
        // reflect the spike onto its first entry
        if (lane < ns) hv[lane] = cmul(s, cconj(AV(0, lane)));
        __syncwarp();
        const cplx tau = aed_house(hv, ns);
        if (tau.x != 0.0 || tau.y != 0.0) {
          aed_left(W, hv, ns, tau, 0, 0, nw);
          aed_right(W, hv, ns, tau, ns, 0);
          aed_right(V, hv, ns, tau, nw, 0);
        }
        // back to Hessenberg form
        for (int j = 0; j + 2 < ns; ++j) {
          const int len = ns - j - 1;
          if (lane < len) hv[lane] = AW(j + 1 + lane, j);
          __syncwarp();
          const cplx tj = aed_house(hv, len);
          if (tj.x != 0.0 || tj.y != 0.0) {
            if (lane < len) AW(j + 1 + lane, j) = lane == 0 ? hv[0] : mkc(0.0, 0.0);
            __syncwarp();
            aed_left(W, hv, len, tj, j + 1, j + 1, nw);
            aed_right(W, hv, len, tj, ns, j + 1);
            aed_right(V, hv, len, tj, nw, j + 1);
          }
        }
      }
    }
    if (lane == 0) { sm.aed[0] = ok ? 1 : 0; sm.aed[1] = ns; }
#ifdef RCWA_EIG_STATS
    if (lane == 0) atomicAdd(&g_eig_stats[6], (unsigned long long)(clock64() - c_w0));
#endif
  }
  __syncthreads();
  bool ok = sm.aed[0] != 0;
  int ns = sm.aed[1];
  bool spike = s.x != 0.0 || s.y != 0.0;
  *shift_count = sm.aed[2];
  if (tm.size > 1) {
    if (lead && tid == 0) {
      ctrl[2] = ok ? ns : -1;
      ctrl[3] = sm.aed[2];
      ctrl[4] = spike ? 1 : 0;
    }
    tm.sync();
    const int c2 = __ldcg(ctrl + 2);
    ok = c2 >= 0;
    ns = ok ? c2 : ns;
    *shift_count = __ldcg(ctrl + 3);
    spike = __ldcg(ctrl + 4) != 0;
  }
  if (!ok) return -1;
  if (ns == nw && spike) return 0;
#ifdef RCWA_EIG_STATS
  const long long c_off = clock64();
#endif
  // window, spike and the off-window blocks
  if (lead) {
    for (int idx = tid; idx < kAedW * kAedW; idx += nthr) {
      const int r = idx / kAedW, c = idx % kAedW;
      if (r < nw && c < nw) T[(size_t)(kw + r) * ldt + kw + c] = AW(r, c);
    }
    if (tid == 0 && kw > l) T[(size_t)kw * ldt + kw - 1] = cmul(s, cconj(AV(0, 0)));
  }
  // rows kw..i right of the window: Vh * T
  for (int j = i + 1 + off0; j < n; j += stride) {
    cplx x[kAedW];
#pragma unroll
    for (int r = 0; r < kAedW; ++r) x[r] = r < nw ? T[(size_t)(kw + r) * ldt + j] : mkc(0.0, 0.0);
#pragma unroll 2
    for (int r = 0; r < nw; ++r) {
      cplx acc = mkc(0.0, 0.0);
#pragma unroll
      for (int c = 0; c < kAedW; ++c) acc = cfmaconj(AV(c, r), x[c], acc);
      T[(size_t)(kw + r) * ldt + j] = acc;
    }
  }
  // columns kw..i above the window: T * V
  for (int r = off0; r < kw; r += stride) {
    cplx x[kAedW];
#pragma unroll
    for (int c = 0; c < kAedW; ++c) x[c] = c < nw ? T[(size_t)r * ldt + kw + c] : mkc(0.0, 0.0);
#pragma unroll 2
    for (int c = 0; c < nw; ++c) {
      cplx acc = mkc(0.0, 0.0);
#pragma unroll
      for (int k = 0; k < kAedW; ++k) acc = cfma(x[k], AV(k, c), acc);
      T[(size_t)r * ldt + kw + c] = acc;
    }
  }
  // Schur vectors (column-major): Z(:, kw..i) * V
  for (int r = off0; r < n; r += stride) {
    cplx x[kAedW];
#pragma unroll
    for (int c = 0; c < kAedW; ++c) x[c] = c < nw ? Z[(size_t)(kw + c) * n + r] : mkc(0.0, 0.0);
#pragma unroll 2
    for (int c = 0; c < nw; ++c) {
      cplx acc = mkc(0.0, 0.0);
#pragma unroll
      for (int k = 0; k < kAedW; ++k) acc = cfma(x[k], AV(k, c), acc);
      Z[(size_t)(kw + c) * n + r] = acc;
    }
  }
  tm.sync();
#ifdef RCWA_EIG_STATS
  STAT_ADD(7, clock64() - c_off);
#endif
  return nw - ns;
}

#undef AW
#undef AV

// Off-window update of one window pass for one lane: the rotations of every
// bulge, in chain order, on one line of T or Z (a column of T right of the
// window, a row of T above it, a row of Z), read and written through
// base + r * stride for index r in [rlo, rhi].  At pass step sg bulge b acts
// on the pair (p, p+1), p = top0 + sg + 3 (kMsShifts - 1 - b), so the chain
// spans kMsFrame consecutive indices that slide by one per step.  That span
// is held in registers: each step takes in the index entering at the bottom
// (loaded kMsPre steps ahead), applies the kMsShifts rotations and stores the
// index leaving at the top, so every element crosses memory once per pass.
// kMsPre steps are unrolled into one group over a frame of kMsFrame + kMsPre -
// 1 registers, which then moves down by kMsPre in one go (a shift per step
// cost as many moves as the rotations cost FP64 instructions).  nsteps is a
// multiple of kMsPre (the log is padded with identities).
//
// Rows: [x; y] <- [c x + s y; -conj(s) x + c y]; columns: the conjugate
// transpose [c x + conj(s) y; -s x + c y].  kScaled: the cosines are taken out
// of the rotations (fast Givens rotations, W. M. Gentleman, J. Inst. Math.
// Appl. 12, 1973): a register holds X with the true value x = d X, and with t
// = s / c the pair becomes X + (t dy/dx) Y, Y - (conj(t) dx/dy) X with both
// scales multiplied by c.  The two coefficients and the final scale of every
// index are common to all lines and come from the log, so a rotation takes 8
// FP64 instructions instead of 12; an element is scaled once, on leaving.
template <bool kRows, bool kScaled>
__device__ __noinline__ void replay_frame(cplx* base, int stride, int top0, int nsteps, int ws, int rlo, int rhi) {
  cplx f[kMsFrame + kMsPre - 1];
  const int lo = rlo - top0, hi = rhi - top0;  // [lo, hi]: the touched indices relative to top0
  // walking pointers of the next entering and the next leaving element
  cplx* out = base + (ptrdiff_t)top0 * stride;
  const cplx* in = out;
#pragma unroll
  for (int k = 0; k < kMsFrame - 1; ++k) {
    f[k] = (k >= lo && k <= hi) ? *in : mkc(0.0, 0.0);
    in += stride;
  }
  cplx pre[kMsPre];
#pragma unroll
  for (int d = 0; d < kMsPre; ++d) {
    const int k = d + kMsFrame - 1;
    pre[d] = (k >= lo && k <= hi) ? *in : mkc(0.0, 0.0);
    in += stride;
  }
  const MsSmem sm = carve_ms_smem(ms_dsm);
  const cplx* e = sm.log;
  const double* df = sm.dfin + (top0 - ws);
#pragma unroll 1
  for (int sg0 = 0; sg0 < nsteps; sg0 += kMsPre) {
#pragma unroll
    for (int d = 0; d < kMsPre; ++d) {
      f[kMsFrame - 1 + d] = pre[d];
      const int k = sg0 + kMsPre + d + kMsFrame - 1;
      pre[d] = (sg0 + kMsPre < nsteps && k >= lo && k <= hi) ? *in : mkc(0.0, 0.0);
      in += stride;
    }
#pragma unroll
    for (int d = 0; d < kMsPre; ++d) {
#pragma unroll
      for (int b = 0; b < kMsShifts; ++b) {
        const cplx e0 = e[2 * b], e1 = e[2 * b + 1];
        const int kb = d + 3 * (kMsShifts - 1 - b);
        const cplx x = f[kb], y = f[kb + 1];
        if (kScaled) {
          f[kb] = kRows ? cfma(e0, y, x) : cfmaconj(e0, y, x);
          f[kb + 1] = kRows ? cfma(e1, x, y) : cfmaconj(e1, x, y);
        } else {  // e0 = s, e1.x = c
          f[kb] = kRows ? cfma(e0, y, cscale(x, e1.x)) : cfmaconj(e0, y, cscale(x, e1.x));
          f[kb + 1] = cfma(cneg(kRows ? cconj(e0) : e0), x, cscale(y, e1.x));
        }
      }
      e += 2 * kMsShifts;
      const int k = sg0 + d;
      if (k >= lo && k <= hi) *out = kScaled ? cscale(f[d], df[k]) : f[d];
      out += stride;
    }
#pragma unroll
    for (int k = 0; k < kMsFrame - 1; ++k) f[k] = f[k + kMsPre];
  }
#pragma unroll
  for (int k0 = 0; k0 < kMsFrame - 1; ++k0) {
    const int k = nsteps + k0;
    if (k >= lo && k <= hi) *out = kScaled ? cscale(f[k0], df[k]) : f[k0];
    out += stride;
  }
}

// The lines a window pass leaves to the replay: columns of T right of the
// window, rows of T above it, rows of Z, 32 lines per warp task, dealt over
// the team's warps.
template <bool kScaled>
__device__ __forceinline__ void replay_lines(cplx* T, int ldt, cplx* Z, int n, int ws, int we, int top0, int nsteps,
                                             int rlo, int rhi, const Team& tm) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nwarp = blockDim.x >> 5;
  const int nR = (n - 1 - we + 31) / 32, nU = (ws + 31) / 32, nZ = (n + 31) / 32;
  for (int task = warp + nwarp * tm.rank; task < nR + nU + nZ; task += nwarp * tm.size) {
    if (task < nR) {
      // T(rlo..rhi, j), j right of the window: row rotations, lane = column
      const int j = we + 1 + 32 * task + lane;
      if (j < n) replay_frame<true, kScaled>(T + j, ldt, top0, nsteps, ws, rlo, rhi);
    } else {
      // T(r, rlo..rhi), r above the window (lane = row), or Z(r, rlo..rhi)
      // (column-major, lane = row): column rotations
      const bool up = task < nR + nU;
      const int r = 32 * (up ? task - nR : task - nR - nU) + lane;
      if (r < (up ? ws : n))
        replay_frame<false, kScaled>(up ? T + (size_t)r * ldt : Z + r, up ? 1 : n, top0, nsteps, ws,
                                     rlo, rhi);
    }
  }
}

// Cosines below this keep a pass on the unscaled replay (the scaled one
// divides by them; an index takes at most 2 kMsShifts rotations per pass, so
// its scale stays above 2^-400).
constexpr double kMsMinCos = 9.5367431640625e-07;  // 2^-20

// The replay coefficients of a pass from its rotation log (cosines in lc,
// sines in log[..][0]).  Index r takes, per bulge, the rotation at p = r - 1
// as its second and the one at p = r as its first element; bulge b is at p
// three steps after bulge b - 1.  So before bulge b's rotation at p (step sg)
// the scales are products of the cosines of the earlier bulges at p - 1, p
// and p + 1, all read from the log, and every entry is computed
// independently.  Returns whether the scaled replay can be used.
__device__ bool replay_coefficients(const MsSmem& sm, int top0, int ws, int nsteps) {
  const int tid = threadIdx.x, nthr = blockDim.x;
  bool small = false;
  for (int idx = tid; idx < nsteps * kMsShifts; idx += nthr) small |= sm.lc[idx] < kMsMinCos;
  const bool scaled = !__syncthreads_or(small);
  if (!scaled) {
    for (int idx = tid; idx < nsteps * kMsShifts; idx += nthr) sm.log[2 * idx + 1] = mkc(sm.lc[idx], 0.0);
    return false;
  }
  auto cosine = [&](int sg, int b) { return sg >= 0 && sg < nsteps ? sm.lc[sg * kMsShifts + b] : 1.0; };
  for (int idx = tid; idx < nsteps * kMsShifts; idx += nthr) {
    const int sg = idx / kMsShifts, b = idx % kMsShifts;
    double dx = cosine(sg - 1, b), dy = 1.0;
    for (int q = 1; q <= b; ++q) {
      const double c = cosine(sg - 3 * q, b - q);
      dx *= cosine(sg - 3 * q - 1, b - q) * c;
      dy *= cosine(sg - 3 * q + 1, b - q) * c;
    }
    const cplx s = sm.log[2 * idx];
    const double c = sm.lc[idx], r = dy / (c * dx), q = dx / (c * dy);
    sm.log[2 * idx] = cscale(s, r);
    sm.log[2 * idx + 1] = mkc(-s.x * q, s.y * q);
  }
  // index r is at p = r at step r - top0 - 3 (kMsShifts - 1 - b) of bulge b
  for (int r = tid; r < kMsW; r += nthr) {
    double d = 1.0;
    for (int b = 0; b < kMsShifts; ++b) {
      const int sg = ws + r - top0 - 3 * (kMsShifts - 1 - b);
      d *= cosine(sg - 1, b) * cosine(sg, b);
    }
    sm.dfin[r] = d;
  }
  return true;
}

// One multishift sweep over the active block [l, i] with sm.shifts[0..s).
// Bulge b sits at position p = l + t - 3b at chain step t; it is active while
// l <= p <= i-1 and its rotation acts on rows/columns (p, p+1).  Warp b chases
// bulge b: every lane evaluates the rotation (a broadcast read and the same
// arithmetic, no exchange), then the warp updates the bulge's two rows, and
// after a barrier its two columns.
// With a team of several CTAs every CTA chases the bulges through its own
// copy of the window (the same operations on the same data), the first CTA
// writes the window back, and the off-window lines are split over the team.
__device__ void ms_sweep(cplx* T, int ldt, cplx* Z, int n, int l, int i, int s, const MsSmem& sm, const Team& tm) {
  const int tid = threadIdx.x, nthr = blockDim.x, lane = tid & 31, b = tid >> 5;
  const int tend = (i - l) + 3 * (s - 1);
  int t = 0;
  while (t < tend) {
    const int bmax0 = min(s - 1, t / 3);
    const int pmin = l + t - 3 * bmax0;
    // while bulges are still being introduced at l the window starts at l
    const int ws = (t < 3 * (s - 1) || pmin == l) ? l : pmin - 1;
    const int we = min(i, ws + kMsW - 1);
    const int w = we - ws + 1;
    int t1 = t;
    while (t1 < tend) {
      const int over = l + t1 - (i - 1);
      const int b0 = over > 0 ? (over + 2) / 3 : 0;
      if (we != i && l + t1 - 3 * b0 + 2 > we) break;
      ++t1;
    }
    STAT_ADD(2, 1);
#ifdef RCWA_EIG_STATS
    const long long c_start = clock64();
#endif
    for (int idx = tid; idx < w * w; idx += nthr)
      cp_async16(&MSW(idx / w, idx % w), &T[(size_t)(ws + idx / w) * ldt + ws + idx % w]);
    cp_async_wait_all();
    __syncthreads();
    // every CTA holds its window before the first one writes it back
    if (tm.size > 1) tm.sync();
    const int nsteps = t1 - t;
    for (int sg = 0; sg < nsteps; ++sg) {
      const int p = l + t + sg - 3 * b;
      const bool on = b < s && p >= l && p <= i - 1;
      double c = 1.0;
      cplx sn = mkc(0.0, 0.0);
      if (on) {
        cplx* const r0 = &MSW(p - ws, 0);
        cplx* const r1 = r0 + kMsLd;
        const int j0 = ((p == l) ? l : p - 1) - ws, jn = we - ws;
        cplx x, y, ra[(kMsW + 31) / 32], rb[(kMsW + 31) / 32];
        if (p == l) { x = csub(r0[p - ws], sm.shifts[b]); y = r1[p - ws]; }
        else { x = r0[p - 1 - ws]; y = r1[p - 1 - ws]; }
        // row operations: rows (p, p+1), columns max(p-1, l) .. we
#pragma unroll
        for (int q = 0; q < (kMsW + 31) / 32; ++q) {
          const int j = j0 + lane + 32 * q;
          if (j <= jn) { ra[q] = r0[j]; rb[q] = r1[j]; }
        }
        givens_fast(x, y, c, sn);
        __syncwarp();
#pragma unroll
        for (int q = 0; q < (kMsW + 31) / 32; ++q) {
          const int j = j0 + lane + 32 * q;
          if (j <= jn) {
            r0[j] = cfma(sn, rb[q], cscale(ra[q], c));
            r1[j] = j < p - ws ? mkc(0.0, 0.0) : cfma(cneg(cconj(sn)), ra[q], cscale(rb[q], c));
          }
        }
      }
      if (lane == 0 && b < kMsShifts) {
        sm.lc[sg * kMsShifts + b] = c;
        sm.log[2 * (sg * kMsShifts + b)] = sn;
      }
      __syncthreads();
      if (on) {
        // column operations: columns (p, p+1), rows ws .. min(p+2, i)
        const int rn = min(p + 2, i) - ws;
#pragma unroll
        for (int q = 0; q < (kMsW + 31) / 32; ++q) {
          const int r = lane + 32 * q;
          if (r <= rn) {
            const cplx a = MSW(r, p - ws), bb = MSW(r, p + 1 - ws);
            MSW(r, p - ws) = cfma(cconj(sn), bb, cscale(a, c));
            MSW(r, p + 1 - ws) = cfma(cneg(sn), a, cscale(bb, c));
          }
        }
      }
      __syncthreads();
    }
    // identity steps up to a whole replay group
    const int npad = (nsteps + kMsPre - 1) / kMsPre * kMsPre;
    for (int idx = nsteps * kMsShifts + tid; idx < npad * kMsShifts; idx += nthr) {
      sm.lc[idx] = 1.0;
      sm.log[2 * idx] = mkc(0.0, 0.0);
    }
#ifdef RCWA_EIG_STATS
    const long long c_mid = clock64();
    STAT_ADD(3, c_mid - c_start);
#endif
    if (tm.rank == 0)
      for (int idx = tid; idx < w * w; idx += nthr) T[(size_t)(ws + idx / w) * ldt + ws + idx % w] = MSW(idx / w, idx % w);
    __syncthreads();
    const int top0 = l + t - 3 * (kMsShifts - 1);
    const bool scaled = replay_coefficients(sm, top0, ws, npad);
    __syncthreads();
    // indices touched in this pass
    const int rlo = max(l, l + t - 3 * (s - 1)), rhi = min(i, l + t1);
    if (scaled) replay_lines<true>(T, ldt, Z, n, ws, we, top0, npad, rlo, rhi, tm);
    else replay_lines<false>(T, ldt, Z, n, ws, we, top0, npad, rlo, rhi, tm);
    tm.sync();
#ifdef RCWA_EIG_STATS
    STAT_ADD(4, clock64() - c_mid);
#endif
    t = t1;
  }
}

// Schur form by early deflation and multishift sweeps; an active block that
// fits the early-deflation window is finished there, in shared memory (single
// shifts take over if the window's iteration runs out).  Returns 0 or
// RCWA_ERR_NOCONV.  With a team of several CTAs the first CTA finds each
// split point and runs the single-shift sweeps, and every decision that
// steers the team's barriers comes from the first CTA through ctrl (global
// scratch of at least 8 ints), so all CTAs take the same path.
__device__ int schur_ms(cplx* T, int ldt, cplx* Z, int n, const MsSmem& sm, int sweep_cap, const Team& tm,
                        int* ctrl) {
  const double ulp = 2.0 * RCWA_DBL_EPS;
  const double smlnum = RCWA_DBL_MIN * ((double)n / ulp);
  const int tid = threadIdx.x;
  int i = n - 1;
  long long sweeps = 0;
  const long long budget = sweep_cap > 0 ? min(30LL * max(10, n), (long long)sweep_cap) : 30LL * max(10, n);
  int stall = 0, last_i = -1, last_l = -1;
  const bool lead = tm.rank == 0;
  int it = 0;
  while (i >= 0) {
    int l = 0;
    if (lead) {
      int best = 0;
      for (int k = 1 + tid; k <= i; k += blockDim.x)
        if (negligible(T, ldt, k, 0, i, ulp, smlnum)) best = max(best, k);
      l = block_max_int(best, sm.redi);
      if (l > 0 && tid == 0) T[(size_t)l * ldt + l - 1] = mkc(0.0, 0.0);
      if (tm.size > 1 && tid == 0) ctrl[it & 1] = l;
    }
    tm.sync();
    if (tm.size > 1) l = __ldcg(ctrl + (it & 1));  // two slots: the first CTA may run one split ahead
    ++it;
    if (l >= i) {
      --i;
      stall = 0;
      continue;
    }
    stall = (i == last_i && l == last_l) ? stall + 1 : 0;
    last_i = i;
    last_l = l;
    const int m = i - l + 1;
    // aggressive early deflation on the trailing window; its undeflated
    // eigenvalues are the next sweep's shifts
    int s = kMsShifts, cnt = 0;
    bool have_shifts = false;
#ifdef RCWA_EIG_STATS
    const long long c_aed = clock64();
#endif
    const int nd = aed(T, ldt, Z, n, l, i, sm, tm, ctrl, &cnt);
#ifdef RCWA_EIG_STATS
    STAT_ADD(8, clock64() - c_aed);
    STAT_ADD(11, 1);
    STAT_ADD(12, nd > 0 ? nd : 0);
#endif
    if (nd > 0) {
      stall = 0;
      i -= nd;
      if (100 * nd > kAedNibble * kAedW || i - l < kAedW) {
        if (++sweeps > budget) return RCWA_ERR_NOCONV;
        continue;
      }
    } else if (m <= kAedW) {
      // the window's iteration ran out: a single-shift sweep
      cplx shift;
      if (stall == 10 || stall == 30)
        shift = cadd(T[(size_t)l * ldt + l], mkc(0.75 * cabs1(T[(size_t)(l + 1) * ldt + l]), 0.0));
      else if (stall == 20 || stall == 40)
        shift = cadd(T[(size_t)i * ldt + i], mkc(0.75 * cabs1(T[(size_t)i * ldt + i - 1]), 0.0));
      else
        shift = wilkinson_shift(T[(size_t)(i - 1) * ldt + i - 1], T[(size_t)(i - 1) * ldt + i],
                                T[(size_t)i * ldt + i - 1], T[(size_t)i * ldt + i]);
      __syncthreads();
      STAT_ADD(1, 1);
      if (lead) qr_sweep(T, ldt, Z, n, l, i, shift, reinterpret_cast<cplx(*)[kWin + 1]>(sm.Wt), sm.lc, sm.log);
      if (++sweeps > budget) return RCWA_ERR_NOCONV;
      continue;
    }
    if (nd >= 0 && cnt >= kMsShifts / 2) {
      s = cnt;
      have_shifts = true;
    }
    __syncthreads();
    {
      STAT_ADD(0, 1);
      if (tid < 32) {
        cplx* B = sm.work;  // s x s, stride s + 1
        const int o = i - s + 1;
        if (stall > 0 && stall % 6 == 0) {
          for (int k = tid; k < s; k += 32)
            sm.shifts[k] = cadd(T[(size_t)(o + k) * ldt + o + k],
                                mkc(0.75 * cabs1(T[(size_t)(o + k) * ldt + o + k - 1]), 0.0));
        } else if (!have_shifts) {
          for (int idx = tid; idx < s * s; idx += 32)
            B[(idx / s) * (s + 1) + idx % s] = T[(size_t)(o + idx / s) * ldt + o + idx % s];
          __syncwarp();
          small_eigs_warp(B, s + 1, s, sm.shifts);
        }
      }
    }
    __syncthreads();
    ms_sweep(T, ldt, Z, n, l, i, s, sm, tm);
    if (++sweeps > budget) return RCWA_ERR_NOCONV;
  }
  return 0;
}

// True when every entry of the Hessenberg matrix is finite (whole CTA).  A
// NaN or Inf never passes the deflation tests, so such a matrix would only
// burn the sweep budget; it is reported as RCWA_ERR_NONFINITE instead.
__device__ bool hessenberg_finite(const cplx* T, int ldt, int n, int* redi) {
  int bad = 0;
  for (int idx = threadIdx.x; idx < n * n; idx += blockDim.x) {
    const int r = idx / n, c = idx % n;
    if (r <= c + 1) {
      const cplx v = T[(size_t)r * ldt + c];
      if (!isfinite(v.x) || !isfinite(v.y)) bad = 1;
    }
  }
  return block_max_int(bad, redi) == 0;
}

__global__ void __launch_bounds__(kMsThreads) schur_ms_kernel(cplx* const* Aarr, int n, int lda, cplx* w_all,
                                                             void* work, int* info_all, int sweep_cap) {
  const MsSmem sm = carve_ms_smem(ms_dsm);
  // one matrix per team (cluster) of CTAs
  const Team tm = cluster_team();
  const int mb = blockIdx.x / tm.size;
  cplx* A = Aarr[mb];
  const Scratch s = scratch_for(work, n, mb);
  // the team's decisions go through the reflector scalars' storage, dead
  // after the Hessenberg reduction (n >= 64 doubles)
  int* ctrl = reinterpret_cast<int*>(s.tau);
#ifdef RCWA_EIG_STATS
  const long long c_schur = clock64();
#endif
  bool fin = false;
  if (tm.rank == 0) {
    fin = hessenberg_finite(A, lda, n, sm.redi);
    if (tm.size > 1 && threadIdx.x == 0) ctrl[5] = fin ? 1 : 0;
  }
  if (tm.size > 1) {
    tm.sync();
    fin = __ldcg(ctrl + 5) != 0;
  }
  const int status = fin ? schur_ms(A, lda, s.Z, n, sm, sweep_cap, tm, ctrl) : RCWA_ERR_NONFINITE;
#ifdef RCWA_EIG_STATS
  STAT_ADD(10, clock64() - c_schur);
#endif
  if (tm.rank == 0) {
    const double f = s.scale[0];
    cplx* w = w_all + (size_t)mb * n;
    for (int k = threadIdx.x; k < n; k += blockDim.x) w[k] = cscale(A[(size_t)k * lda + k], f);
    if (threadIdx.x == 0) info_all[mb] = status;
  }
}

// ---------------------------------------------------------------- eigenvectors
// Eigenvectors of the upper triangular T (LAPACK ztrevc, right vectors, back
// substitution with protected divisors): column k of X solves
// (T - t_kk I) x = 0 with x_k = 1 and x_j = 0 for j > k.  Blocked bottom-up
// over 64-row blocks [r0, r1): the coupling to the rows already solved,
// B = T(r0:r1, r1:) X(r1:, k), is a tile GEMM over the upper triangle of X
// (column tile by column tile, K cut at the tile's last column); the block
// itself is solved by one thread per column in two 32-row halves held in
// registers.
constexpr int kTrBlk = 64;

template <int R>
__device__ __forceinline__ void trevc_half(const cplx* T, int ldt, cplx* X, int n, int k, int h0, int hend,
                                           cplx tkk, double ulp, double smlnum, cplx (&x)[R]) {
  // rows h0 .. h0+R-1 (those < hend); X(i, k) holds the right-hand side
  const double smin = fmax(ulp * cabs1(tkk), smlnum);
#pragma unroll
  for (int ii = R - 1; ii >= 0; --ii) {
    const int i = h0 + ii;
    cplx xi = mkc(0.0, 0.0);
    if (i < hend) {
      if (i == k) {
        xi = mkc(1.0, 0.0);
      } else if (i < k) {
        cplx acc = X[(size_t)i * n + k];
#pragma unroll
        for (int jj = ii + 1; jj < R; ++jj) acc = cfma(__ldg(&T[(size_t)i * ldt + h0 + jj]), x[jj], acc);
        cplx d = csub(__ldg(&T[(size_t)i * ldt + i]), tkk);
        if (cabs1(d) < smin) d = mkc(smin, 0.0);
        xi = cneg(cdiv(acc, d));
      }
      X[(size_t)i * n + k] = xi;
    }
    x[ii] = xi;
  }
}

__device__ void trevc_blocked(const cplx* T, int ldt, cplx* X, int n, TileSmem& tsm) {
  const double ulp = 2.0 * RCWA_DBL_EPS;
  const double smlnum = RCWA_DBL_MIN * ((double)n / ulp);
  // X = 0 everywhere but the unit diagonal; rows are overwritten block by block
  for (size_t idx = threadIdx.x; idx < (size_t)n * n; idx += blockDim.x)
    X[idx] = mkc((idx / n) == (idx % n) ? 1.0 : 0.0, 0.0);
  __syncthreads();
  const int nblk = (n + kTrBlk - 1) / kTrBlk;
  for (int bi = nblk - 1; bi >= 0; --bi) {
    const int r0 = bi * kTrBlk, r1 = min(n, r0 + kTrBlk);
    // B(r0:r1, c) = sum_{j >= r1} T(r0:r1, j) X(j, c) for columns c >= r1;
    // X(j, c) = 0 for j > c, so the tile of columns [c0, c0+64) needs j < c0+64
    for (int c0 = r1; c0 < n; c0 += kTBN) {
      const int nc = min(kTBN, n - c0);
      const int K = min(n, c0 + nc) - r1;
      cta_gemm<false, false>(tsm, r1 - r0, nc, K, T + (size_t)r0 * ldt + r1, ldt, X + (size_t)r1 * n + c0, n,
                             X + (size_t)r0 * n + c0, n, nullptr, 0, mkc(1.0, 0.0), mkc(0.0, 0.0));
    }
    // columns k > r0 solve the block rows; columns inside the block start
    // from a zero right-hand side (X(i, k) = 0 for i < k there)
    for (int k = r0 + 1 + threadIdx.x; k < n; k += blockDim.x) {
      const cplx tkk = __ldg(&T[(size_t)k * ldt + k]);
      cplx xl[32], xh[32];
      // lower half [r0+32, r1)
      trevc_half<32>(T, ldt, X, n, k, r0 + 32, r1, tkk, ulp, smlnum, xh);
      // the lower half's contribution to the upper half's right-hand side
      if (k > r0) {
        for (int ii = 0; ii < 32 && r0 + ii < min(k, r1); ++ii) {
          const int i = r0 + ii;
          cplx acc = X[(size_t)i * n + k];
#pragma unroll
          for (int jj = 0; jj < 32; ++jj)
            if (r0 + 32 + jj < r1) acc = cfma(__ldg(&T[(size_t)i * ldt + r0 + 32 + jj]), xh[jj], acc);
          X[(size_t)i * n + k] = acc;
        }
      }
      trevc_half<32>(T, ldt, X, n, k, r0, min(r1, r0 + 32), tkk, ulp, smlnum, xl);
    }
    __syncthreads();
  }
}

// The Hessenberg reduction runs 512 threads: its per-column sweeps and
// matrix-vector products stream from L2/DRAM and need the loads in flight;
// the first 256 threads also run the tile products.
constexpr int kHessThreads = 512;

template <bool kTeam>
__global__ void __launch_bounds__(kHessThreads) hessenberg_kernel(cplx* const* Aarr, int n, int lda, void* work) {
  __shared__ double red[kHessThreads / 32];
  __shared__ int redi[kHessThreads / 32];
  __shared__ TileSmem tsm;
  // one matrix per team (cluster) of CTAs
  const Team tm = kTeam ? cluster_team() : Team{0, 1};
  const int mb = blockIdx.x / tm.size;
  const Scratch s = scratch_for(work, n, mb);
  cplx* A = Aarr[mb];
  // a matrix whose products could leave the normal range is reduced, iterated
  // and back-substituted at a power of two of its size (exact; a scaled-back
  // Schur form could overflow, or lie below the smallest divisor that the back
  // substitution allows); only the eigenvalues are scaled back
  int ex = 0;
  for (int i = threadIdx.x >> 5; i < n; i += blockDim.x >> 5) {
    int e4 = 0;
#pragma unroll 4
    for (int j = threadIdx.x & 31; j < n; j += 32) {
      const cplx v = A[(size_t)i * lda + j];
      e4 = max(e4, max(__double2hiint(v.x) & 0x7fffffff, __double2hiint(v.y) & 0x7fffffff));
    }
    ex = max(ex, e4 >> 20);
  }
  ex = block_max_int(ex, redi) - 1023;
  const int sh = ex > 100 ? min(ex, 1000) : ex < -100 ? max(ex, -1000) : 0;
  // no CTA writes the matrix before every CTA of the team has read all of it:
  // the reduction's first column can cross the bound that the scan tests, and
  // the CTAs must agree on the branch below, which holds a barrier
  if (kTeam) tm.sync();
  if (sh != 0) {
    const double f = scalbn(1.0, -sh);
    const int per = (n + tm.size - 1) / tm.size;
    for (int i = tm.rank * per; i < min(n, (tm.rank + 1) * per); ++i)
      for (int j = threadIdx.x; j < n; j += blockDim.x) A[(size_t)i * lda + j] = cscale(A[(size_t)i * lda + j], f);
    tm.sync();
  }
  if (tm.rank == 0 && threadIdx.x == 0) s.scale[0] = scalbn(1.0, sh);
  hessenberg_blocked<kTeam>(A, n, lda, s, red, tsm, tm);
}

template <int Q>
__global__ void __launch_bounds__(kBlkThreads) schur_block_kernel(cplx* const* Aarr, int n, int lda, cplx* w_all,
                                                                 void* work, int* info_all, int sweep_cap) {
  extern __shared__ __align__(16) unsigned char blk_dsm[];
  __shared__ int redi[kBlkThreads / 32];
  cplx* A = Aarr[blockIdx.x];
  cplx* T = reinterpret_cast<cplx*>(blk_dsm);
  const Scratch s = scratch_for(work, n, blockIdx.x);
  const int ld = blk_ld(n);
  int status = RCWA_ERR_NONFINITE;
  if (hessenberg_finite(A, lda, n, redi)) {
    for (int idx = threadIdx.x; idx < n * n; idx += blockDim.x) {
      const int r = idx / n, c = idx % n;
      T[r * ld + c] = r <= c + 1 ? A[(size_t)r * lda + c] : mkc(0.0, 0.0);
    }
    __syncthreads();
    status = schur_block<Q>(T, ld, s.Z, n, sweep_cap);
    __syncthreads();
    for (int idx = threadIdx.x; idx < n * n; idx += blockDim.x)
      A[(size_t)(idx / n) * lda + idx % n] = T[(idx / n) * ld + idx % n];
    __syncthreads();
  }
  const double f = s.scale[0];
  cplx* w = w_all + (size_t)blockIdx.x * n;
  for (int k = threadIdx.x; k < n; k += blockDim.x) w[k] = cscale(A[(size_t)k * lda + k], f);
  if (threadIdx.x == 0) info_all[blockIdx.x] = status;
}

__global__ void __launch_bounds__(kEigThreads) trevc_kernel(cplx* const* Aarr, int n, int lda, void* work) {
  __shared__ TileSmem tsm;
  const Scratch s = scratch_for(work, n, blockIdx.x);
  trevc_blocked(Aarr[blockIdx.x], lda, s.X, n, tsm);
}

// unit 2-norm columns; non-finite eigenpairs flag the matrix
__global__ void normalize_kernel(cplx* const* VRarr, int n, int ldv, const cplx* w_all, int* info_all) {
  cplx* VR = VRarr[blockIdx.y];
  const cplx* w = w_all + (size_t)blockIdx.y * n;
  const int j = blockIdx.x * blockDim.x + threadIdx.x;
  if (j >= n) return;
  double ss = 0.0;
  for (int i = 0; i < n; ++i) ss += cnorm2(VR[(size_t)i * ldv + j]);
  const double sc = ss > 0.0 ? 1.0 / sqrt(ss) : 1.0;
  for (int i = 0; i < n; ++i) VR[(size_t)i * ldv + j] = cscale(VR[(size_t)i * ldv + j], sc);
  if (!isfinite(sc) || !isfinite(ss) || !isfinite(w[j].x) || !isfinite(w[j].y))
    atomicCAS(&info_all[blockIdx.y], 0, RCWA_ERR_NONFINITE);
}


}  // namespace


namespace {
// QR sweep cap of every later eigensolve (0: the built-in budget), set by
// rcwa_set_qr_sweep_limit; read when the Schur kernels are launched.
std::atomic<int> g_qr_sweep_cap{0};
// CTAs per matrix of the Hessenberg and multishift Schur kernels (0: the
// automatic choice), set by rcwa_set_eig_cluster.
std::atomic<int> g_eig_team{0};

// Clusters of `size` CTAs of `kernel` that fit on the device at once.
template <class K>
int active_clusters(K kernel, int threads, size_t smem, int size) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(size);
  cfg.blockDim = dim3(threads);
  cfg.dynamicSmemBytes = smem;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = size;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  int nc = 0;
  if (cudaOccupancyMaxActiveClusters(&nc, (void*)kernel, &cfg) != cudaSuccess) {
    cudaGetLastError();
    return 0;
  }
  return nc;
}

// Allows the multishift kernel its dynamic shared memory on this device.
cudaError_t schur_ms_ready() {
  static SmemAttrOnce attr;
  return attr.ensure(schur_ms_kernel, (int)kMsSmemBytes);
}

// Team size for a batch of order-n matrices: the largest (up to 8, and a CTA
// per 64 rows) whose clusters of both kernels all fit on the device in one
// wave, when the batch alone would leave at least half of the SMs idle; 1
// otherwise.
int eig_team_auto(int n, int batch) {
  int dev = 0, sms = 0;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  // the occupancy of the Schur kernel needs its shared memory allowed first
  if (batch <= 0 || 2 * batch > sms || schur_ms_ready() != cudaSuccess) return 1;
  const int most = std::min(std::min(8, sms / batch), std::max(1, n / 64));
  static std::mutex mu;
  static std::map<std::tuple<int, int, int>, int> cache;  // (device, batch, largest size) -> size
  std::lock_guard<std::mutex> lk(mu);
  const auto key = std::make_tuple(dev, batch, most);
  auto it = cache.find(key);
  if (it != cache.end()) return it->second;
  int pick = 1;
  for (int c = most; c >= 2; --c)
    if (active_clusters(hessenberg_kernel<true>, kHessThreads, 0, c) >= batch &&
        active_clusters(schur_ms_kernel, kMsThreads, kMsSmemBytes, c) >= batch) {
      pick = c;
      break;
    }
  cache[key] = pick;
  return pick;
}

// CTAs per matrix of a batch of order-n matrices: one where the matrix is held
// in shared memory, else the forced or the automatic team.
int eig_team(int n, int batch, int ms_min) {
  if (zgeev_in_shared_memory(n, ms_min)) return 1;
  const int forced = g_eig_team.load();
  return forced > 0 ? forced : eig_team_auto(n, batch);
}

// launch of kernel over batch * team CTAs in clusters of `team`
template <class K, class... Args>
cudaError_t launch_team(K kernel, int batch, int team, int threads, size_t smem, cudaStream_t st, Args... args) {
  if (team <= 1) {
    kernel<<<batch, threads, smem, st>>>(args...);
    return cudaGetLastError();
  }
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(batch * team);
  cfg.blockDim = dim3(threads);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = team;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, kernel, args...);
}

template <int Q>
cudaError_t launch_block(cplx* const* A, int n, int lda, cplx* w, void* work, int* info, int sweep_cap, int batch,
                         cudaStream_t st) {
  static SmemAttrOnce attr;
  const cudaError_t e = attr.ensure(schur_block_kernel<Q>, (int)blk_smem(std::min(32 * Q, kBlkMax)));
  if (e != cudaSuccess) return e;
  schur_block_kernel<Q><<<batch, kBlkThreads, blk_smem(n), st>>>(A, n, lda, w, work, info, sweep_cap);
  return cudaGetLastError();
}

}  // namespace

bool zgeev_in_shared_memory(int n, int ms_min) {
  return n <= kBlkMax && (ms_min <= 0 || n < std::max(ms_min, kMsMin));
}

extern "C" int rcwa_set_qr_sweep_limit(int sweeps) {
  if (sweeps < 0) return RCWA_ERR_INVALID;
  g_qr_sweep_cap.store(sweeps);
  return RCWA_OK;
}

extern "C" int rcwa_set_eig_cluster(int ctas) {
  if (ctas < 0 || ctas > 8) return RCWA_ERR_INVALID;
  g_eig_team.store(ctas);
  return RCWA_OK;
}

extern "C" int rcwa_eig_cluster_size(int n, int batch) {
  return n <= 0 || batch <= 0 ? 1 : eig_team(n, batch, 0);
}

cudaError_t zgeev_batched(cplx* const* A, int n, int lda, cplx* w, cplx* const* VR, int ldv, void* work,
                          int* info, int batch, cudaStream_t st, StageProf* prof, int ms_min) {
  if (batch <= 0 || n <= 0) return cudaSuccess;
  const int sweep_cap = g_qr_sweep_cap.load();
  StageProf none;
  StageProf& P = prof ? *prof : none;
  cudaError_t e = schur_ms_ready();
  if (e != cudaSuccess) return e;
  const bool block = zgeev_in_shared_memory(n, ms_min);
  const int team = eig_team(n, batch, ms_min);
  e = team > 1 ? launch_team(hessenberg_kernel<true>, batch, team, kHessThreads, 0, st, A, n, lda, work)
               : launch_team(hessenberg_kernel<false>, batch, 1, kHessThreads, 0, st, A, n, lda, work);
  if (e != cudaSuccess) return e;
  ++launch_counter();
  P.mark(st, kStHessenberg);
  if (block) {
    e = n <= 32 ? launch_block<1>(A, n, lda, w, work, info, sweep_cap, batch, st)
        : n <= 64 ? launch_block<2>(A, n, lda, w, work, info, sweep_cap, batch, st)
                  : launch_block<4>(A, n, lda, w, work, info, sweep_cap, batch, st);
  } else {
    e = launch_team(schur_ms_kernel, batch, team, kMsThreads, kMsSmemBytes, st, A, n, lda, w, work, info, sweep_cap);
  }
  if (e != cudaSuccess) return e;
  ++launch_counter();
  P.mark(st, kStSchur);
  trevc_kernel<<<batch, kEigThreads, 0, st>>>(A, n, lda, work);
  ++launch_counter();
  P.mark(st, kStTrevc);
  // VR = Z X for every matrix (Z column-major == transposed operand)
  GemmArgs g{};
  g.A = nullptr;
  g.A0 = (const cplx*)work;
  g.sA = workspace_bytes(n) / sizeof(cplx);
  g.B = nullptr;
  g.B0 = (const cplx*)work + (size_t)n * n;
  g.sB = g.sA;
  g.D = VR;
  g.M = n; g.N = n; g.K = n;
  g.lda = n; g.ldb = n; g.ldd = ldv; g.ldc = ldv;
  g.transA = 1; g.transB = 0;
  g.triB = 1;  // X is upper triangular
  g.alpha = mkc(1.0, 0.0); g.beta = mkc(0.0, 0.0); g.gammaI = mkc(0.0, 0.0);
  g.batch = batch;
  cudaError_t err = zgemm_batched(g, st);
  if (err != cudaSuccess) return err;
  P.mark(st, kStBackTransform);
  dim3 grid((n + 127) / 128, batch);
  normalize_kernel<<<grid, 128, 0, st>>>(VR, n, ldv, w, info);
  ++launch_counter();
  P.mark(st, kStNormalize);
  return cudaGetLastError();
}

#ifdef RCWA_EIG_STATS
extern "C" int rcwa_debug_eig_stats(unsigned long long* out, int reset) {
  unsigned long long h[32];
  if (cudaMemcpyFromSymbol(h, g_eig_stats, sizeof(h)) != cudaSuccess) return 2;
  for (int i = 0; i < 32; ++i) out[i] = h[i];
  if (reset) {
    unsigned long long z[32] = {};
    cudaMemcpyToSymbol(g_eig_stats, z, sizeof(z));
  }
  return 0;
}
#endif
