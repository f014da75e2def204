// z2_stab.cuh -- UDV stabilization (src/stabilization.f90:42-200) on the
// DMMA GEMM, the blocked panel kernels and the register-resident pivoted QR.
#pragma once
#include "z2_gemm.cuh"
#include "z2_qrp.cuh"

// C = A B with the options of gemm_nnn; any n (the unit kernel takes n a
// multiple of 4, which every lattice has).
__device__ __forceinline__ void mul_nn(int n, MatRef A, bool a_upper, MatRef B, bool b_lower, double *C,
                                       int ldc) {
  if ((n & 3) == 0) gemm_nnn(n, A, nullptr, a_upper, B, b_lower, GemmOut{C, ldc});
  else blk_dmma(n, n, n, 1.0, A, a_upper, B, b_lower, 0.0, C, ldc);
}

// The orthogonal factor of reflectors with coefficients tau (the pivoted QR),
// in place; vd: n doubles of shared memory.
static __device__ __noinline__ void form_q(double *A, int lda, int n, const double *tau, double *vd,
                                    double *work, int wd) {
  if (wd < wy_work(n)) {
    blk_org2r_tc(A, lda, n, n, tau);
  } else if (__isShared(A)) {
    blk_wy_t<true>(A, lda, n, tau, vd, work);
    blk_form_q<true>(A, lda, n, vd, work);
  } else {
    blk_wy_t<false>(A, lda, n, tau, vd, work);
    blk_form_q<false>(A, lda, n, vd, work);
  }
}

// stab_UR (left = false) / stab_UL (left = true), src/stabilization.f90:70-120.
// On entry A (lda; shared arena or global) holds the propagated U (UR, or
// UL^T).  U, D, V are the factors in global memory (U = UR or UL^T); W0 is an
// N x N global workspace.
static __device__ __noinline__ void dev_stab_U(const Smem &s, int N, double *A, int lda, double *U,
                                        double *D, double *V, double *W0, bool left) {
  double *tau = s.vec, *vn1 = s.vec + N, *vn2 = s.vec + 2 * N, *Dn = s.vec + 3 * N;
  int *jpvt = s.ivec;
  blk_scale_cols(A, lda, N, N, D);                 // matUDV(:,i) *= D(i)
  blk_geqp3_fast(A, lda, N, jpvt, tau, vn1, vn2, s.tile, s.tile_doubles, s.red);   // ZGEQP3
  blk_qdrp_scale(A, lda, N, Dn, vn2);              // D = |R_ii|, R rows /= D
  for (int i = threadIdx.x; i < N; i += Z2_NT) D[i] = Dn[i];
  if (!left) {
    // VR <- R (P^T VR)     (ZLAPMR(.true.) + ZTRMM('L','U','N','N'))
    blk_perm_rows(W0, N, V, N, N, N, jpvt, true);
    mul_nn(N, MatRef{A, 1, lda}, true, MatRef{W0, 1, N}, false, V, N);
  } else {
    // VL <- (VL P) R^T     (ZLAPMT(.true.) + ZTRMM('R','U','C','N'))
    blk_perm_cols(W0, N, V, N, N, N, jpvt, true);
    mul_nn(N, MatRef{W0, 1, N}, false, MatRef{A, lda, 1}, true, V, N);
  }
  form_q(A, lda, N, tau, s.vec + 4 * N, s.tile, s.tile_doubles);   // ZUNGQR
  blk_copy(U, N, A, lda, N, N);                    // UR = Q, or UL^T = Q
}

// stab_green (src/stabilization.f90:122-200): G = (I + UR DR VR VL DL UL)^-1
// into Gout (global, ld N).  The reference applies Q^H with ZUNMQR; here Q is
// formed (ZUNGQR) and applied by a DMMA GEMM, then D^-1, the triangular solve
// (DMMA-blocked) and the permutation follow in the reference's order.
// M (ldm) is the QR work matrix (shared arena when it fits); W1, W2, W3 are
// N x N global workspaces (W3 keeps the scaled R).
static __device__ __noinline__ void dev_stab_green(const Smem &s, int N, int nt, int Ltrot,
                                            const double *UR, const double *DR,
                                            const double *VR, const double *ULT,
                                            const double *DL, const double *VL, double *M,
                                            int ldm, double *W1, double *W2, double *W3,
                                            double *Gout) {
  double *tau = s.vec, *vn1 = s.vec + N, *vn2 = s.vec + 2 * N, *Dn = s.vec + 3 * N;
  int *jpvt = s.ivec;
  // invULUR = UR^T UL^T -> M ; VRVL = VR VL -> W1
  mul_nn(N, MatRef{UR, N, 1}, false, MatRef{ULT, 1, N}, false, M, ldm);
  mul_nn(N, MatRef{VR, 1, N}, false, MatRef{VL, 1, N}, false, W1, N);
  // matUDV = invULUR + DR (VRVL DL)   (src/stabilization.f90:138-146)
  for (int j = threadIdx.x / 32; j < N; j += Z2_WARPS) {
    const double dl = DL[j];
    for (int i = threadIdx.x & 31; i < N; i += 32) {
      const double t = W1[i + (size_t)j * N] * dl;
      const double u = DR[i] * t;
      M[i + (size_t)j * ldm] = M[i + (size_t)j * ldm] + u;
    }
  }
  __syncthreads();
  const int half = Ltrot / 2;
  if (nt > half) {   // matUDV = matUDV^dagger
    for (int j = threadIdx.x / 32; j < N; j += Z2_WARPS)
      for (int i = threadIdx.x & 31; i < j; i += 32) {
        const double a = M[i + (size_t)j * ldm], b = M[j + (size_t)i * ldm];
        M[i + (size_t)j * ldm] = b;
        M[j + (size_t)i * ldm] = a;
      }
    __syncthreads();
  }
  blk_geqp3_fast(M, ldm, N, jpvt, tau, vn1, vn2, s.tile, s.tile_doubles, s.red);
  blk_qdrp_scale(M, ldm, N, Dn, vn2);   // vn2 keeps 1/D for the D^-1 scalings below
  // keep the scaled R (upper triangle) for the triangular solve
  for (int j = threadIdx.x / 32; j < N; j += Z2_WARPS)
    for (int i = threadIdx.x & 31; i <= j; i += 32) W3[i + (size_t)j * N] = M[i + (size_t)j * ldm];
  __syncthreads();
  form_q(M, ldm, N, tau, s.vec + 4 * N, s.tile, s.tile_doubles);   // Q in M
  if (nt < half + 1) {
    // G = UL^T P R^-1 D^-1 Q^T UR^T
    mul_nn(N, MatRef{M, ldm, 1}, false, MatRef{UR, N, 1}, false, W2, N);
    // Y = D^-1 (Q^T UR^T) back into the arena (Q is no longer needed)
    for (int j = threadIdx.x / 32; j < N; j += Z2_WARPS)
      for (int i = threadIdx.x & 31; i < N; i += 32)
        M[i + (size_t)j * ldm] = W2[i + (size_t)j * N] * vn2[i];
    __syncthreads();
    blk_trsm_lun_blocked(W3, N, N, M, ldm, N);     // R_s^-1 Y
    blk_perm_rows(W1, N, M, ldm, N, N, jpvt, false);   // ZLAPMR(.false.)
    mul_nn(N, MatRef{ULT, 1, N}, false, MatRef{W1, 1, N}, false, Gout, N);
  } else {
    // G = UL^T Q D^-1 R^-T P^T UR^T, solved transposed: X^T = R_s^-1 D^-1 (UL^T Q)^T
    mul_nn(N, MatRef{ULT, 1, N}, false, MatRef{M, 1, ldm}, false, W2, N);
    for (int j = threadIdx.x / 32; j < N; j += Z2_WARPS)
      for (int i = threadIdx.x & 31; i < N; i += 32)
        M[i + (size_t)j * ldm] = W2[j + (size_t)i * N] * vn2[i];
    __syncthreads();
    blk_trsm_lun_blocked(W3, N, N, M, ldm, N);     // X^T
    blk_perm_rows(W1, N, M, ldm, N, N, jpvt, false);   // (X P^T)^T
    mul_nn(N, MatRef{W1, N, 1}, false, MatRef{UR, N, 1}, false, Gout, N);
  }
}

// ---------------------------------------------------------------------------
// Pre-pivoted stabilization (the chain's default).  The reference factors with
// column-pivoted QR (ZGEQP3), a column step of which waits on the norm
// downdate and the arg-max of the previous one.  Here the columns are put in
// decreasing norm order once ("pre-pivoting", Bai, Lee, Li and Xu, Linear
// Algebra Appl. 435 (2011) 659) and factored by the blocked Householder QR
// without pivoting; the Green's function is formed from the scale-split
// middle matrix (Loh and Gubernatis; the same construction as QUEST's
// stabilized G):
//   M  = UR^T UL^T + DR (VR VL) DL
//      = DRb (DRb^-1 UR^T UL^T DLb^-1 + DRs VR VL DLs) DLb = DRb M' DLb,
//   DRb = max(DR, 1), DRs = min(DR, 1) (DLb, DLs likewise),
//   G  = UL^T M^-1 UR^T = UL^T DLb^-1 M'^-1 DRb^-1 UR^T,
// where M' has entries of order one and is inverted by Gauss-Jordan
// elimination with partial pivoting.  U, D, V and G are the same as the
// reference's up to rounding (the UDV factors of a product are not unique: the
// column order of D may differ).
//
// Every step is a panel kernel of z2_blocked.cuh or a product of z2_gemm.cuh.
// At N = 144 (cycles, one SM): QR 175 K, Q 95 K, inverse 170 K, a product 90 K;
// the register-resident kernels they replace (one column per step over the
// whole tile) took 393 K, 188 K, 298 K and 103 K.
// ---------------------------------------------------------------------------
// Sizes the panel kernels take with wd doubles of shared work space.
__device__ __forceinline__ bool wy_ok(int n, int wd) {
  return n >= 4 && n <= 256 && (n & 3) == 0 && wd >= wy_work(n);
}

__device__ __forceinline__ void qr_panels_any(double *A, int lda, int n, double *vd, double *work) {
  if constexpr (Z2_NMAX <= 64) blk_qr_panels<true, 2>(A, lda, n, vd, work);
  else if (__isShared(A) && n <= 160) blk_qr_panels<true, 5>(A, lda, n, vd, work);
  else blk_qr_panels<false, 8>(A, lda, n, vd, work);
}
__device__ __forceinline__ void form_q_any(double *A, int lda, int n, const double *vd, double *work) {
  if (__isShared(A)) blk_form_q<true>(A, lda, n, vd, work);
  else blk_form_q<false>(A, lda, n, vd, work);
}
__device__ __forceinline__ void gj_any(double *M, int ldm, int n, int *piv, double *work) {
  if constexpr (Z2_NMAX <= 64) {
    if (n <= 32) blk_gj_panels<true, 1>(M, ldm, n, piv, work);
    else blk_gj_panels<true, 2>(M, ldm, n, piv, work);
  } else if (__isShared(M) && n <= 160) {
    if (n <= 32) blk_gj_panels<true, 1>(M, ldm, n, piv, work);
    else if (n <= 64) blk_gj_panels<true, 2>(M, ldm, n, piv, work);
    else if (n <= 96) blk_gj_panels<true, 3>(M, ldm, n, piv, work);
    else if (n <= 128) blk_gj_panels<true, 4>(M, ldm, n, piv, work);
    else blk_gj_panels<true, 5>(M, ldm, n, piv, work);
  } else {
    blk_gj_panels<false, 8>(M, ldm, n, piv, work);
  }
}

// A <- A P S, column j of it being sc[j] (null: 1) times column perm[j] of A, in
// shared memory through registers (n <= 32 T).
template <int T>
static __device__ __noinline__ void permute_cols_reg(double *A, int lda, int n, const int *perm, const double *sc) {
  A = as_shared(A);
  constexpr int C = 32 * T / Z2_WARPS;    // columns per warp
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  double v[C][T];
#pragma unroll
  for (int c = 0; c < C; ++c) {
    const int j = warp + Z2_WARPS * c;
    const double *src = A + (j < n ? perm[j] : 0) * lda;
#pragma unroll
    for (int t = 0; t < T; ++t) v[c][t] = (j < n && lane + 32 * t < n) ? src[lane + 32 * t] : 0.0;
  }
  __syncthreads();
#pragma unroll
  for (int c = 0; c < C; ++c) {
    const int j = warp + Z2_WARPS * c;
    const double x = (sc && j < n) ? sc[j] : 1.0;
#pragma unroll
    for (int t = 0; t < T; ++t)
      if (j < n && lane + 32 * t < n) A[lane + 32 * t + j * lda] = v[c][t] * x;
  }
  __syncthreads();
}
// The same for any A; W: an n x n global workspace.
__device__ __forceinline__ void permute_cols(double *A, int lda, int n, const int *perm, const double *sc,
                                             double *W) {
  if constexpr (Z2_NMAX <= 64) {
    if (n <= 32) permute_cols_reg<1>(A, lda, n, perm, sc);
    else permute_cols_reg<2>(A, lda, n, perm, sc);
    return;
  } else if (__isShared(A) && n <= 160) {
    if (n <= 32) permute_cols_reg<1>(A, lda, n, perm, sc);
    else if (n <= 64) permute_cols_reg<2>(A, lda, n, perm, sc);
    else if (n <= 96) permute_cols_reg<3>(A, lda, n, perm, sc);
    else if (n <= 128) permute_cols_reg<4>(A, lda, n, perm, sc);
    else permute_cols_reg<5>(A, lda, n, perm, sc);
    return;
  }
  blk_copy(W, n, A, lda, n, n);
  blk_walk<8, double>(
      n, n, [&](int i, int j) { return W[i + (size_t)perm[j] * n]; },
      [&](double v, int i, int j) { A[i + (size_t)j * lda] = sc ? v * sc[j] : v; });
  __syncthreads();
}

// sqrt(sum A(:, j)^2) D(j) of every column, a NaN as -1; R(i, j) <- R(i, j)
// cj(j) ri(i) on the upper triangle.
template <bool SH>
__device__ __forceinline__ void col_norms(const double *A, int lda, int n, const double *D, double *nrm) {
  if (SH) A = as_shared(const_cast<double *>(A));
  const int lane = threadIdx.x & 31;
  for (int j = 2 * (threadIdx.x >> 5); j < n; j += 2 * Z2_WARPS) {   // n is even
    double s0 = 0.0, s1 = 0.0;
#pragma unroll 5
    for (int i = lane; i < n; i += 32) {
      const double a = A[i + j * lda], b = A[i + (j + 1) * lda];
      s0 = fma(a, a, s0);
      s1 = fma(b, b, s1);
    }
    s0 = warp_sum(s0);
    s1 = warp_sum(s1);
    if (lane < 2) {
      const double x = sqrt(lane ? s1 : s0) * D[j + lane];
      nrm[j + lane] = (x == x) ? x : -1.0;         // a NaN column sorts last
    }
  }
  __syncthreads();
}
template <bool SH>
__device__ __forceinline__ void scale_upper(double *A, int lda, int n, const double *cj, const double *ri) {
  if (SH) A = as_shared(A);
  const int lane = threadIdx.x & 31;
  for (int j = threadIdx.x >> 5; j < n; j += Z2_WARPS) {
    const double dj = cj[j];
#pragma unroll 5
    for (int i = lane; i <= j; i += 32) A[i + j * lda] *= dj * ri[i];
  }
  __syncthreads();
}

// stab_UR / stab_UL with the pre-pivoted QR; arguments as dev_stab_U.  D scales
// the columns of A, which leaves Q as it is and scales R's columns, so A itself
// is factored and D meets only the column order and R.
static __device__ __noinline__ void dev_stab_U_fast(const Smem &s, int N, double *A, int lda, double *U,
                                             double *D, double *V, double *W0, bool left) {
  if (!wy_ok(N, s.tile_doubles)) {
    dev_stab_U(s, N, A, lda, U, D, V, W0, left);
    return;
  }
  double *vd = s.vec, *nrm = s.vec + N, *Dp = s.vec + 2 * N, *rd = s.vec + 3 * N;
  int *perm = s.ivec;
  const bool sh = __isShared(A);
  if (sh) col_norms<true>(A, lda, N, D, nrm);
  else col_norms<false>(A, lda, N, D, nrm);
  // decreasing norm, ties in column order: a permutation for any input
  for (int j = threadIdx.x; j < N; j += Z2_NT) {
    const double x = nrm[j];
    int r = 0;
#pragma unroll 4
    for (int i = 0; i < N; ++i) {
      const double y = nrm[i];
      r += (y > x || (y == x && i < j)) ? 1 : 0;
    }
    perm[r] = j;
  }
  __syncthreads();
  permute_cols(A, lda, N, perm, nullptr, W0);
  qr_panels_any(A, lda, N, vd, s.tile);            // A P = Q R
  // D = |R_ii| D_p(i), R(i, j) <- R(i, j) D_p(j) / D(i)
  for (int i = threadIdx.x; i < N; i += Z2_NT) {
    const double dp = D[perm[i]];
    Dp[i] = dp;
    rd[i] = fabs(A[i + (size_t)i * lda]) * dp;
  }
  __syncthreads();
  for (int i = threadIdx.x; i < N; i += Z2_NT) {
    D[i] = rd[i];
    rd[i] = 1.0 / rd[i];
  }
  __syncthreads();
  if (sh) scale_upper<true>(A, lda, N, Dp, rd);
  else scale_upper<false>(A, lda, N, Dp, rd);
  if (!left) {
    blk_walk<8, double>(                           // VR <- R (P^T VR)
        N, N, [&](int i, int j) { return V[perm[i] + (size_t)j * N]; },
        [&](double v, int i, int j) { W0[i + (size_t)j * N] = v; });
    __syncthreads();
    gemm_nnn(N, MatRef{A, 1, lda}, nullptr, true, MatRef{W0, 1, N}, false, GemmOut{V, N});
  } else {
    blk_walk<8, double>(                           // VL <- (VL P) R^T
        N, N, [&](int i, int j) { return V[i + (size_t)perm[j] * N]; },
        [&](double v, int i, int j) { W0[i + (size_t)j * N] = v; });
    __syncthreads();
    gemm_nnn(N, MatRef{W0, 1, N}, nullptr, false, MatRef{A, lda, 1}, true, GemmOut{V, N});
  }
  form_q_any(A, lda, N, vd, s.tile);
  blk_copy(U, N, A, lda, N, N);
}

// M <- (M')^-1 of the scale-split middle matrix, up to a row order: with piv[j]
// the pivot row of column j, M'^-1(j, piv[m]) = M(piv[j], m).  rRb, rLb, Rs, Ls
// receive DRb^-1, DLb^-1, DRs, DLs (N doubles of shared memory each).  N a
// multiple of 4; above the panel kernels' range the inverse comes from a
// blocked LU through the N x N global workspaces W0, W1.
static __device__ __noinline__ void middle_inverse(const Smem &s, int N, const double *UR, const double *DR,
                                            const double *VR, const double *ULT, const double *DL,
                                            const double *VL, double *M, int ldm, double *rRb,
                                            double *rLb, double *Rs, double *Ls, int *piv, double *W0,
                                            double *W1) {
  for (int i = threadIdx.x; i < N; i += Z2_NT) {
    rRb[i] = 1.0 / fmax(DR[i], 1.0);
    rLb[i] = 1.0 / fmax(DL[i], 1.0);
    Rs[i] = fmin(DR[i], 1.0);
    Ls[i] = fmin(DL[i], 1.0);
  }
  // M' = DRb^-1 (UR^T UL^T) DLb^-1 + DRs (VR VL) DLs
  gemm_nnn(N, MatRef{UR, N, 1}, nullptr, false, MatRef{ULT, 1, N}, false, GemmOut{M, ldm});
  gemm_nnn(N, MatRef{VR, 1, N}, nullptr, false, MatRef{VL, 1, N}, false,
           GemmOut{M, ldm, rRb, rLb, Rs, Ls});
  if (wy_ok(N, s.tile_doubles)) {
    gj_any(M, ldm, N, piv, s.tile);
  } else {
    blk_inverse_blocked(M, ldm, N, W0, N, piv, s.red, s.flag, s.tile);
    for (int i = threadIdx.x; i < N; i += Z2_NT) piv[i] = i;
    __syncthreads();
  }
}

// stab_green with the scale-split middle matrix; arguments as dev_stab_green
// (W1 and W2 are N x N scratch).
static __device__ __noinline__ void dev_stab_green_fast(const Smem &s, int N, int nt, int Ltrot,
                                                 const double *UR, const double *DR,
                                                 const double *VR, const double *ULT,
                                                 const double *DL, const double *VL, double *M,
                                                 int ldm, double *W1, double *W2, double *W3,
                                                 double *Gout) {
  if (!wy_ok(N, s.tile_doubles)) {
    dev_stab_green(s, N, nt, Ltrot, UR, DR, VR, ULT, DL, VL, M, ldm, W1, W2, W3, Gout);
    return;
  }
  double *rRb = s.vec + N, *rLb = s.vec + 2 * N;
  int *piv = s.ivec;
  middle_inverse(s, N, UR, DR, VR, ULT, DL, VL, M, ldm, rRb, rLb, s.vec + 3 * N, s.vec + 4 * N, piv,
                 W1, W2);
  // columns of M into M'^-1's order, times DRb^-1: W1 = DLb^-1 M'^-1 DRb^-1 UR^T,
  // G = UL^T W1
  int *inv = piv + N;
  for (int m = threadIdx.x; m < N; m += Z2_NT) inv[piv[m]] = m;
  __syncthreads();
  permute_cols(M, ldm, N, inv, rRb, W2);
  gemm_nnn(N, MatRef{M, 1, ldm}, piv, false, MatRef{UR, N, 1}, false, GemmOut{W1, N, rLb});
  gemm_nnn(N, MatRef{ULT, 1, N}, nullptr, false, MatRef{W1, 1, N}, false, GemmOut{Gout, N});
}
