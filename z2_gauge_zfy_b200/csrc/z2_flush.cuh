// z2_flush.cuh -- the rank-2k flush G -= X Yt^T of the delayed updates
// (LocalK_metro, src/localK.f90:45-173) as DMMA tiles.
#pragma once
#include "z2_dmma.cuh"

// The delayed-update factors X and Yt (N x k2 each) keep their columns in
// interleaved pairs: element (i, q) sits at (q / 2) 2 ldx + 2 i + q % 2, so
// the two columns an accepted flip adds are one 16-byte word per row (one
// load in the ratio evaluation and in the column phase, one store), and a
// DMMA fragment (rows r + 0..7, columns l + 0..3) still hits 16 distinct
// bank pairs per half-warp for ldx = 4 (mod 16).
__device__ __forceinline__ size_t xy_at(int i, int q, int ldx) {
  return (size_t)(q >> 1) * (2 * ldx) + 2 * i + (q & 1);
}

// G <- G - X Yt^T over the m queued columns (paired layout) when 8 TR and 8 TC
// divide N: each warp owns (8 TR) x (8 TC) blocks of G, loads their old
// values straight into the DMMA accumulators and adds (-X) Yt^T to them in
// chunks of 4 columns, reusing each X fragment TC times and each Yt fragment
// TR times.
template <bool GS, int TR, int TC>
static __device__ __noinline__ void flush_tiles(double *G, int ldg, const double *X, const double *Yt,
                                         int N, int ldx, int m) {
  if (GS) G = as_shared(G);
  X = as_shared(X);
  Yt = as_shared(Yt);
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int lr = lane >> 2, lc = lane & 3;
  const int gr = N / (8 * TR), gcn = N / (8 * TC);
  const int m4 = m & ~3;
  const size_t s4 = (size_t)4 * ldx;
  for (int g = warp; g < gr * gcn; g += Z2_WARPS) {
    const int r0 = (g % gr) * 8 * TR, c0 = (g / gr) * 8 * TC;
    double *cp = G + r0 + lr + (size_t)(c0 + 2 * lc) * ldg;
    double acc[TR][TC][2];
#pragma unroll
    for (int a = 0; a < TR; ++a)
#pragma unroll
      for (int b = 0; b < TC; ++b)
#pragma unroll
        for (int e = 0; e < 2; ++e) acc[a][b][e] = cp[8 * a + (size_t)(8 * b + e) * ldg];
    const double *pa = X + xy_at(r0 + lr, lc, ldx);
    const double *pb = Yt + xy_at(c0 + lr, lc, ldx);
#pragma unroll 2
    for (int l0 = 0; l0 < m4; l0 += 4) {
      double fa[TR], fb[TC];
#pragma unroll
      for (int u = 0; u < TR; ++u) fa[u] = -pa[16 * u];
#pragma unroll
      for (int v = 0; v < TC; ++v) fb[v] = pb[16 * v];
      pa += s4; pb += s4;
#pragma unroll
      for (int u = 0; u < TR; ++u)
#pragma unroll
        for (int v = 0; v < TC; ++v) dmma884(acc[u][v][0], acc[u][v][1], fa[u], fb[v]);
    }
    if (m4 < m) {
      // two trailing columns: lanes lc >= m - m4 feed zeros
      const bool ok = lc < m - m4;
      double fa[TR], fb[TC];
#pragma unroll
      for (int u = 0; u < TR; ++u) fa[u] = ok ? -pa[16 * u] : 0.0;
#pragma unroll
      for (int v = 0; v < TC; ++v) fb[v] = ok ? pb[16 * v] : 0.0;
#pragma unroll
      for (int u = 0; u < TR; ++u)
#pragma unroll
        for (int v = 0; v < TC; ++v) dmma884(acc[u][v][0], acc[u][v][1], fa[u], fb[v]);
    }
#pragma unroll
    for (int a = 0; a < TR; ++a)
#pragma unroll
      for (int b = 0; b < TC; ++b)
#pragma unroll
        for (int e = 0; e < 2; ++e) cp[8 * a + (size_t)(8 * b + e) * ldg] = acc[a][b][e];
  }
  __syncthreads();
}

// The same update for any N: (8 GS) x (8 GS) groups with bounds checks.
template <bool SH, int GS>
static __device__ __noinline__ void flush_generic(double *G, int ldg, const double *X, const double *Yt,
                                           int N, int ldx, int m) {
  if (SH) G = as_shared(G);
  X = as_shared(X);
  Yt = as_shared(Yt);
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int lr = lane >> 2, lc = lane & 3;
  const int gm = (N + 8 * GS - 1) / (8 * GS);
  for (int g = warp; g < gm * gm; g += Z2_WARPS) {
    const int r0 = (g % gm) * 8 * GS, c0 = (g / gm) * 8 * GS;
    double acc[GS][GS][2];
#pragma unroll
    for (int a = 0; a < GS; ++a)
#pragma unroll
      for (int b = 0; b < GS; ++b)
#pragma unroll
        for (int e = 0; e < 2; ++e) {
          const int row = r0 + 8 * a + lr, col = c0 + 8 * b + 2 * lc + e;
          acc[a][b][e] = (row < N && col < N) ? G[row + (size_t)col * ldg] : 0.0;
        }
    for (int l0 = 0; l0 < m; l0 += 4) {
      const int l = l0 + lc;
      const bool lk = l < m;
      double fa[GS], fb[GS];
#pragma unroll
      for (int u = 0; u < GS; ++u) {
        const int ra = r0 + 8 * u + lr, cb = c0 + 8 * u + lr;
        fa[u] = (lk && ra < N) ? -X[xy_at(ra, l, ldx)] : 0.0;
        fb[u] = (lk && cb < N) ? Yt[xy_at(cb, l, ldx)] : 0.0;
      }
#pragma unroll
      for (int u = 0; u < GS; ++u)
#pragma unroll
        for (int v = 0; v < GS; ++v) dmma884(acc[u][v][0], acc[u][v][1], fa[u], fb[v]);
    }
#pragma unroll
    for (int a = 0; a < GS; ++a)
#pragma unroll
      for (int b = 0; b < GS; ++b)
#pragma unroll
        for (int e = 0; e < 2; ++e) {
          const int row = r0 + 8 * a + lr, col = c0 + 8 * b + 2 * lc + e;
          if (row < N && col < N) G[row + (size_t)col * ldg] = acc[a][b][e];
        }
  }
  __syncthreads();
}

// Tile shapes of the rank-2k flush (z2_options.flush_shape_chain).  Every
// shape forms each element of G from its old value with the same k chunks,
// so they give the same bits; they differ in how the N x N update
// is cut into warp blocks (load balance over the 8 warps against fragment
// reuse).  0 picks by divisibility: 24 x 24 blocks when 24 | N, 16 x 16 when
// 16 | N, else the bounded 16 x 16 groups.
enum {
  FS_DEFAULT = 0, FS_GEN16 = 1, FS_GEN8 = 2, FS_T11 = 3, FS_T22 = 4, FS_T33 = 5, FS_T21 = 6,
  FS_T32 = 7, FS_COUNT = 8
};
__host__ __device__ __forceinline__ bool flush_shape_ok(int shape, int N) {
  switch (shape) {
    case FS_DEFAULT: case FS_GEN16: case FS_GEN8: return true;
    case FS_T11: return N % 8 == 0;
    case FS_T22: case FS_T21: return N % 16 == 0;
    case FS_T33: return N % 24 == 0;
    case FS_T32: return N % 48 == 0;
    default: return false;
  }
}

// G <- G - X Yt^T over the m queued columns: one DMMA rank-m update.
// GS: G is in shared memory (X and Yt always are).
template <bool GS>
__device__ __forceinline__ void rank_update(double *G, int ldg, const double *X, const double *Yt,
                                            int N, int ldx, int m, int shape = FS_DEFAULT) {
  switch (shape) {
    case FS_GEN16: flush_generic<GS, 2>(G, ldg, X, Yt, N, ldx, m); return;
    case FS_GEN8: flush_generic<GS, 1>(G, ldg, X, Yt, N, ldx, m); return;
    case FS_T11: flush_tiles<GS, 1, 1>(G, ldg, X, Yt, N, ldx, m); return;
    case FS_T22: flush_tiles<GS, 2, 2>(G, ldg, X, Yt, N, ldx, m); return;
    case FS_T33: flush_tiles<GS, 3, 3>(G, ldg, X, Yt, N, ldx, m); return;
    case FS_T21: flush_tiles<GS, 2, 1>(G, ldg, X, Yt, N, ldx, m); return;
    case FS_T32: flush_tiles<GS, 3, 2>(G, ldg, X, Yt, N, ldx, m); return;
    default: break;
  }
  if (N % 24 == 0) flush_tiles<GS, 3, 3>(G, ldg, X, Yt, N, ldx, m);
  else if (N % 16 == 0) flush_tiles<GS, 2, 2>(G, ldg, X, Yt, N, ldx, m);
  else flush_generic<GS, 2>(G, ldg, X, Yt, N, ldx, m);
}
