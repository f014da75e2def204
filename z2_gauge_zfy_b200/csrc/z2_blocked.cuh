// z2_blocked.cuh -- blocked Householder QR, the orthogonal factor it encodes,
// and the Gauss-Jordan inverse, all in panels of 8 columns.
//
// A panel is factored by warp 0 with its columns in registers (lane l holds
// rows l + 32 t), where a column step needs only warp shuffles; the other
// columns are updated in tiles of 8 columns, each tile by one warp from top to
// bottom with DMMA (the products with V and T, or with the pivot rows, never
// leave the warp).  Warp 0 updates the next panel's tile first and factors it
// while the other seven warps finish the rest, so a panel costs one block
// barrier and the chain of column steps overlaps the updates.
//
// Matrices are column-major; SH: the matrix is in shared memory.
#pragma once
#include "z2_dmma.cuh"

#define WY_NB 8

// Leading dimension of the panel buffers: = 4 (mod 16), so both orientations of
// a DMMA fragment (row + 4 column, column + 4 row) hit 16 distinct bank
// pairs per half-warp; rows up to the next multiple of 8 are stored (zeros).
__host__ __device__ __forceinline__ int wy_ldv(int n) {
  return ((((n + 7) & ~7) + 11) & ~15) + 4;
}
__host__ __device__ __forceinline__ int wy_panels(int n) { return (n + WY_NB - 1) / WY_NB; }
// Shared work space (doubles): two panel buffers, every panel's T, and 64 more.
__host__ __device__ __forceinline__ int wy_work(int n) {
  return 2 * WY_NB * wy_ldv(n) + WY_NB * WY_NB * (wy_panels(n) + 1);
}

template <int I>
struct WyIdx { static constexpr int v = I; };

// 1 / x to rounding (error < 1.01 2^-53) for 2^-1022 <= |x| <= 2^1022: the
// hardware's approximation and two Newton steps r <- r (2 - x r) (no special
// cases, so it schedules beside other work, unlike the division).  Outside, 0
// and subnormals give NaN and larger values 0: the determinant of an accepted
// proposal and the pivots of a matrix of order one do not get there.
__device__ __forceinline__ double rcp_newton(double x) {
  double r;
  asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(r) : "d"(x));
  r = fma(r, fma(-x, r, 1.0), r);
  return fma(r, fma(-x, r, 1.0), r);
}

// nb = sqrt(q) and g = 1 / (q + al nb) for al >= 0, al^2 <= q and 2^-959 <= q <=
// 2^960, to rounding (errors < 1.55 and 3 times 2^-53; outside, y or r may be 0
// or infinite and the result NaN: warp_qr_panel_scaled).
// y ~ 1 / sqrt(q) and r ~ 1 / (q + al sqrt(q)) are the hardware's
// approximations (2^-20), each corrected by one third-order Newton step:
// with t = q y, e = 1 - t y:  sqrt(q) = t (1 + e / 2 + 3 e^2 / 8 + O(e^3)), and
// with f = 1 - d r:  1 / d = r (1 + f + f^2 + O(f^3)).  r starts from t, so the
// two chains overlap.
__device__ __forceinline__ void sqrt_rcp(double q, double al, double &nb, double &g) {
  double y, r;
  asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(q));
  const double t = q * y;
  const double d0 = fma(al, t, q);
  asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(r) : "d"(d0));
  const double e = fma(-t, y, 1.0);
  nb = fma(t, e * fma(0.375, e, 0.5), t);
  const double f = fma(-fma(al, nb, q), r, 1.0);
  g = fma(r, fma(f, f, f), r);
}

// The exponent field of x (x = m 2^(exp_of - 1023), 1 <= m < 2).
__device__ __forceinline__ unsigned exp_of(double x) { return ((unsigned)__double2hiint(x) >> 20) & 0x7ffu; }

// An 8 x 8 accumulator (row lane / 4, columns 2 (lane % 4) + {0, 1}) as the two
// B fragments of a product over its rows: b[s] = X(4 s + lane % 4, lane / 4).
__device__ __forceinline__ void acc_to_b(double x0, double x1, double (&b)[2], int lane) {
  const int lr = lane >> 2, lc = lane & 3;
#pragma unroll
  for (int s = 0; s < 2; ++s) {
    const int src = (4 * s + lc) * 4 + (lr >> 1);
    const double y0 = __shfl_sync(Z2_FULL, x0, src), y1 = __shfl_sync(Z2_FULL, x1, src);
    b[s] = (lr & 1) ? y1 : y0;
  }
}

// C += Z X for NT tiles of 8 columns (c0[i]..) of A, rows j0..n: Z (rows at 1,
// columns at ldv) from the panel buffer, X as B fragments, by one warp, four row
// tiles at a time.  Two tiles share the loads of Z and overlap each other's
// latency.  (Prefetching the next four row tiles behind the products measured
// slower: the warp's shared-memory instructions fill the time.)
template <int NT>
__device__ __forceinline__ void panel_update(double *A, int lda, int n, int j0, const int (&c0)[NT],
                                             const double *Zb, int ldv, const double (&b)[NT][2]) {
  const int lane = threadIdx.x & 31, lr = lane >> 2, lc = lane & 3;
  const double *qv = Zb + lc * ldv + lr;
  double *qc[NT];
  int st[NT];
  bool k0[NT], k1[NT];
#pragma unroll
  for (int i = 0; i < NT; ++i) {
    const int col = c0[i] + 2 * lc;
    k0[i] = col < n;
    k1[i] = col + 1 < n;
    qc[i] = A + (k0[i] ? col : n - 1) * lda + lr;
    st[i] = k1[i] ? lda : 0;
  }
  int r0 = j0;
  for (; r0 + 32 <= n; r0 += 32) {
    double c[NT][4][2], x[4][2];
#pragma unroll
    for (int u = 0; u < 4; ++u) {
#pragma unroll
      for (int i = 0; i < NT; ++i) {
        c[i][u][0] = qc[i][r0 + 8 * u];
        c[i][u][1] = qc[i][r0 + 8 * u + st[i]];
      }
      x[u][0] = qv[r0 + 8 * u]; x[u][1] = qv[r0 + 8 * u + 4 * ldv];
    }
#pragma unroll
    for (int s = 0; s < 2; ++s)
#pragma unroll
      for (int u = 0; u < 4; ++u)
#pragma unroll
        for (int i = 0; i < NT; ++i) dmma884(c[i][u][0], c[i][u][1], x[u][s], b[i][s]);
#pragma unroll
    for (int u = 0; u < 4; ++u)
#pragma unroll
      for (int i = 0; i < NT; ++i) {
        if (k0[i]) qc[i][r0 + 8 * u] = c[i][u][0];
        if (k1[i]) qc[i][r0 + 8 * u + st[i]] = c[i][u][1];
      }
  }
  for (; r0 < n; r0 += 8) {
    const bool ok = r0 + lr < n;
    const double x0 = qv[r0], x1 = qv[r0 + 4 * ldv];
    double c[NT][2];
#pragma unroll
    for (int i = 0; i < NT; ++i) {
      c[i][0] = ok ? qc[i][r0] : 0.0;
      c[i][1] = ok ? qc[i][r0 + st[i]] : 0.0;
    }
#pragma unroll
    for (int i = 0; i < NT; ++i) {
      dmma884(c[i][0], c[i][1], x0, b[i][0]);
      dmma884(c[i][0], c[i][1], x1, b[i][1]);
      if (ok && k0[i]) qc[i][r0] = c[i][0];
      if (ok && k1[i]) qc[i][r0 + st[i]] = c[i][1];
    }
  }
  __syncwarp();
}

// ---------------------------------------------------------------------------
// Householder QR
// ---------------------------------------------------------------------------
// DGEQR2 on the panel A(j0:n, j0:j0+8) by one warp, n - j0 <= 8 R: lane
// (lr, lc) = (lane / 4, lane % 4) holds rows lr + 8 i of columns 2 lc and
// 2 lc + 1, so a column's products with its neighbours are sums over eight
// lanes, and the column reaches the other lanes by R shuffles within groups of
// four.  The reflectors are left unscaled: H = I - g v v^T, v(j) = alpha - beta,
// v(r) = A(r, j) below, g = 1 / (beta (beta - alpha)) (DLARFG divides v by
// v(j); here nothing on the column's chain waits for that division).  R and
// the reflectors below it go back into A, v(j) into vd, the reflectors clean
// (zeros above) into Vb (column c at c ldv), and the block's T (DLARFT forward /
// columnwise with g for tau, column-major 8 x 8) into Tb; the products
// v_q^T v_k it needs come with the same sums, through the 64 doubles zs.
// Returns false with nothing written (unless any) where a diagonal entry of R is
// outside [2^-100, 2^100) (or NaN: the squares left the range): then squares, or
// products of an unscaled reflector with a column, may over- or underflow.
// (Scaling a column at its step, in the column's chain, cost 1 to 3 % of a bin.)
template <int R>
__device__ __forceinline__ bool warp_qr_panel(double *A, int lda, int n, int j0, double *Vb, int ldv,
                                              double *Tb, double *vd, double *zs, bool any) {
  const int lane = threadIdx.x & 31, lr = lane >> 2, lc = lane & 3;
  const int mp = n - j0, ib = mp < WY_NB ? mp : WY_NB;
  double *Ap = A + j0 + (j0 + 2 * lc) * lda + lr;
  double a[R][2];
#pragma unroll
  for (int i = 0; i < R; ++i)
#pragma unroll
    for (int e = 0; e < 2; ++e)
      a[i][e] = (lr + 8 * i < mp && 2 * lc + e < ib) ? Ap[8 * i + e * lda] : 0.0;
  double gl = 0.0, vl = 1.0;    // lane k < 8: g and v(j) of column k
  // one column; e = k % 2 is static, so that the panel is a loop over column
  // pairs (unrolled over all eight, the panels alone filled the instruction
  // cache)
  const auto column = [&](int k, auto E) {
    constexpr int e = decltype(E)::v;
    const int own = k >> 1;
    double x[R];
#pragma unroll
    for (int i = 0; i < R; ++i) x[i] = __shfl_sync(Z2_FULL, a[i][e], own, 4);
    const double alpha = __shfl_sync(Z2_FULL, x[0], 4 * k);
    const double r0 = __shfl_sync(Z2_FULL, a[0][0], 4 * k + lc);
    const double r1 = __shfl_sync(Z2_FULL, a[0][1], 4 * k + lc);
    x[0] = lr > k ? x[0] : 0.0;                     // rows below the diagonal
    double d0 = x[0] * a[0][0], d1 = x[0] * a[0][1], f0 = 0.0, f1 = 0.0;
#pragma unroll
    for (int i = 1; i < R; ++i) {
      if (i & 1) { f0 = fma(x[i], a[i][0], f0); f1 = fma(x[i], a[i][1], f1); }
      else { d0 = fma(x[i], a[i][0], d0); d1 = fma(x[i], a[i][1], d1); }
    }
    d0 += f0; d1 += f1;
#pragma unroll
    for (int o = 4; o <= 16; o <<= 1) {
      d0 += __shfl_xor_sync(Z2_FULL, d0, o);
      d1 += __shfl_xor_sync(Z2_FULL, d1, o);
    }
    const double ss = __shfl_sync(Z2_FULL, e ? d1 : d0, own, 4);
    // beta = -sign(alpha) sqrt(alpha^2 + |x|^2); a zero column: H = I
    const bool refl = ss != 0.0;
    const double q = refl ? fma(alpha, alpha, ss) : 1.0;
    double nb, gq;
    sqrt_rcp(q, fabs(alpha), nb, gq);
    const double beta = refl ? -copysign(nb, alpha) : alpha;
    const double hv = alpha - beta;
    const double g = refl ? gq : 0.0;
    // v_c^T v_k for the earlier columns, H_j on the later ones:
    // A(:, c) -= g (v(j) A(j, c) + x^T A(j+1:, c)) v
    const double p0 = fma(hv, r0, d0), p1 = fma(hv, r1, d1);
    if (lr == 0) { zs[8 * k + 2 * lc] = p0; zs[8 * k + 2 * lc + 1] = p1; }
    const double w0 = 2 * lc > k ? -g * p0 : 0.0, w1 = 2 * lc + 1 > k ? -g * p1 : 0.0;
    x[0] = lr == k ? hv : x[0];
#pragma unroll
    for (int i = 0; i < R; ++i) {
      a[i][0] = fma(w0, x[i], a[i][0]);
      a[i][1] = fma(w1, x[i], a[i][1]);
    }
    if (lr == k && lc == own) a[0][e] = beta;
    if (lane == k) { gl = g; vl = hv; }
  };
#pragma unroll 1
  for (int k = 0; k < ib; k += 2) {
    column(k, WyIdx<0>{});
    if (k + 1 < ib) column(k + 1, WyIdx<1>{});
  }
  // row r's lane of column r: R(r, r), the column's norm at its step
  const double rr = (lr & 1) ? a[0][1] : a[0][0];
  const bool far = (lr >> 1) == lc && lr < ib && exp_of(rr) - 923u >= 200u;
  if (__any_sync(Z2_FULL, far) && !any) return false;
  for (int t = 8 * ib + lane; t < 64; t += 32) zs[t] = 0.0;   // columns past the matrix
  __syncwarp();
  const int m8 = (mp + 7) & ~7;
#pragma unroll
  for (int i = 0; i < R; ++i) {
    const int r = lr + 8 * i;
#pragma unroll
    for (int e = 0; e < 2; ++e) {
      const int c = 2 * lc + e;
      double v = 0.0;
      if (c < ib) {
        if (r < mp) Ap[8 * i + e * lda] = a[i][e];
        if (r > c) v = a[i][e];
      }
      if (r < m8 && (i > 0 || r != c)) Vb[j0 + r + c * ldv] = v;
    }
  }
  if (lane < 8) {
    Vb[j0 + lane + lane * ldv] = lane < ib ? vl : 0.0;
    if (lane < ib) vd[j0 + lane] = vl;
  }
  // T row by row in lane i < 8: T(i, k) = -g_k sum_{q < k} T(i, q) z_q(k)
  double tr[8];
#pragma unroll
  for (int k = 0; k < 8; ++k) {
    double s = 0.0;
#pragma unroll
    for (int q = 0; q < k; ++q) s = fma(tr[q], zs[8 * k + q], s);
    const double g = __shfl_sync(Z2_FULL, gl, k);
    tr[k] = lane == k ? g : (lane < k ? -g * s : 0.0);
  }
  if (lane < 8) {
#pragma unroll
    for (int c = 0; c < 8; ++c) Tb[c * 8 + lane] = tr[c];
  }
  __syncwarp();
  return true;
}

// The panel with the smallest R that holds its n - j0 <= 32 T rows.
template <bool SH, int T>
static __device__ __noinline__ bool warp_qr_panel_any(double *A, int lda, int n, int j0, double *Vb, int ldv,
                                               double *Tb, double *vd, double *zs, bool any) {
  if (SH) A = as_shared(A);
  zs = as_shared(zs);
  Vb = as_shared(Vb);
  Tb = as_shared(Tb);
  vd = as_shared(vd);
  const int mp = n - j0;
  if (T > 5 && mp > 160) return warp_qr_panel<32>(A, lda, n, j0, Vb, ldv, Tb, vd, zs, any);
  if (T > 4 && mp > 144) return warp_qr_panel<20>(A, lda, n, j0, Vb, ldv, Tb, vd, zs, any);
  if (T > 3 && mp > 104) return warp_qr_panel<18>(A, lda, n, j0, Vb, ldv, Tb, vd, zs, any);
  if (T > 2 && mp > 64) return warp_qr_panel<13>(A, lda, n, j0, Vb, ldv, Tb, vd, zs, any);
  if (T > 1 && mp > 32) return warp_qr_panel<8>(A, lda, n, j0, Vb, ldv, Tb, vd, zs, any);
  if (mp > 16) return warp_qr_panel<4>(A, lda, n, j0, Vb, ldv, Tb, vd, zs, any);
  return warp_qr_panel<2>(A, lda, n, j0, Vb, ldv, Tb, vd, zs, any);
}

// Panel j0 by one warp; where the plain one gives up, on scaled columns: every
// column of the panel times a power of two that brings its largest entry into
// [1, 2).  The reflectors, v(j) and g of the scaled columns give the same H; R is
// scaled back.  Lane l looks after column l / 4, rows l % 4 + 4 i.
template <bool SH, int T>
static __device__ __noinline__ void warp_qr_panel_scaled(double *A, int lda, int n, int j0, double *Vb, int ldv,
                                                  double *Tb, double *vd, double *zs) {
  const int lane = threadIdx.x & 31, c = lane >> 2, r0 = lane & 3, mp = n - j0;
  double *Ac = A + j0 + (j0 + c) * lda;
  const int m = c < mp ? mp : 0;
  double mx = 0.0, un = 1.0;
  for (int r = r0; r < m; r += 4) mx = fmax(mx, fabs(Ac[r]));
  mx = fmax(mx, __shfl_xor_sync(Z2_FULL, mx, 1));
  mx = fmax(mx, __shfl_xor_sync(Z2_FULL, mx, 2));
  if (mx > 0.0) {
    const int b = min(max(2046 - (int)exp_of(mx), 1), 2045);      // times 2^(b - 1023)
    for (int r = r0; r < m; r += 4) Ac[r] *= __hiloint2double(b << 20, 0);
    un = __hiloint2double((2046 - b) << 20, 0);
  }
  __syncwarp();
  warp_qr_panel_any<SH, T>(A, lda, n, j0, Vb, ldv, Tb, vd, zs, true);
  for (int r = r0; r < min(c + 1, m); r += 4) Ac[r] *= un;
  __syncwarp();
}
template <bool SH, int T>
__device__ __forceinline__ void warp_qr_panel_safe(double *A, int lda, int n, int j0, double *Vb, int ldv,
                                                   double *Tb, double *vd, double *zs) {
  if (!warp_qr_panel_any<SH, T>(A, lda, n, j0, Vb, ldv, Tb, vd, zs, false))
    warp_qr_panel_scaled<SH, T>(A, lda, n, j0, Vb, ldv, Tb, vd, zs);
}

// C <- C - V (op(T) (V^T C)) for NT tiles of 8 columns of A, rows j0..n, by one
// warp; op(T) = T^T (TT: Q^T C, the factorization) or T (Q C).
template <bool TT, int NT>
__device__ __forceinline__ void wy_tile(double *A, int lda, int n, int j0, const int (&c0)[NT],
                                        const double *Vb, int ldv, const double *Tb) {
  const int lane = threadIdx.x & 31, lr = lane >> 2, lc = lane & 3;
  // W = V^T C in 4 / NT chains per tile
  constexpr int CH = 4 / NT;
  const double *pv = Vb + lr * ldv + lc;
  const double *pc[NT];
#pragma unroll
  for (int i = 0; i < NT; ++i) pc[i] = A + min(c0[i] + lr, n - 1) * lda + lc;
  double w[NT][CH][2] = {};
  int l = j0;
  for (; l + 16 <= n; l += 16) {
    double x[4], y[NT][4];
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      x[u] = pv[l + 4 * u];
#pragma unroll
      for (int i = 0; i < NT; ++i) y[i][u] = pc[i][l + 4 * u];
    }
#pragma unroll
    for (int u = 0; u < 4; ++u)
#pragma unroll
      for (int i = 0; i < NT; ++i) dmma884(w[i][u % CH][0], w[i][u % CH][1], x[u], y[i][u]);
  }
#pragma unroll
  for (int u = 0; u < 4; ++u) {
    const int r = l + 4 * u;
    if (r < n) {                                    // uniform
      const bool ok = r + lc < n;
      const double x = ok ? pv[r] : 0.0;
#pragma unroll
      for (int i = 0; i < NT; ++i) dmma884(w[i][u % CH][0], w[i][u % CH][1], x, ok ? pc[i][r] : 0.0);
    }
  }
  double b[NT][2];
#pragma unroll
  for (int i = 0; i < NT; ++i) {
#pragma unroll
    for (int h = 1; h < CH; ++h) { w[i][0][0] += w[i][h][0]; w[i][0][1] += w[i][h][1]; }
    acc_to_b(w[i][0][0], w[i][0][1], b[i], lane);
  }
  double t[2];
#pragma unroll
  for (int s = 0; s < 2; ++s) t[s] = TT ? Tb[lr * 8 + 4 * s + lc] : Tb[(4 * s + lc) * 8 + lr];
#pragma unroll
  for (int i = 0; i < NT; ++i) {
    double y0 = 0.0, y1 = 0.0;
    dmma884(y0, y1, t[0], b[i][0]);
    dmma884(y0, y1, t[1], b[i][1]);
    acc_to_b(-y0, -y1, b[i], lane);
  }
  panel_update<NT>(A, lda, n, j0, c0, Vb, ldv, b);   // C += V (-op(T) W)
}

// Column tiles first, first + step, ... < np by the calling warp, in pairs.
template <bool TT>
__device__ __forceinline__ void wy_tiles(double *A, int lda, int n, int j0, int first, int step, int np,
                                         const double *Vb, int ldv, const double *Tb) {
  int ct = first;
  for (; ct + step < np; ct += 2 * step) {
    const int c[2] = {ct * WY_NB, (ct + step) * WY_NB};
    wy_tile<TT, 2>(A, lda, n, j0, c, Vb, ldv, Tb);
  }
  if (ct < np) {
    const int c[1] = {ct * WY_NB};
    wy_tile<TT, 1>(A, lda, n, j0, c, Vb, ldv, Tb);
  }
}

// Householder QR without pivoting of the n x n matrix A, n <= 32 T: R and the
// reflectors in A, their diagonals in vd (n doubles of shared memory), every
// panel's T in work (wy_work(n) doubles of it): what blk_form_q takes.
template <bool SH, int T>
static __device__ __noinline__ void blk_qr_panels(double *A, int lda, int n, double *vd, double *work) {
  if (SH) A = as_shared(A);
  work = as_shared(work);
  const int warp = threadIdx.x >> 5;
  const int ldv = wy_ldv(n), np = wy_panels(n);
  double *Tall = work + 2 * WY_NB * ldv, *zs = Tall + 64 * np;
  if (warp == 0) warp_qr_panel_safe<SH, T>(A, lda, n, 0, work, ldv, Tall, vd, zs);
  __syncthreads();
  for (int p = 0; p + 1 < np; ++p) {
    const int j0 = p * WY_NB;
    const double *Vb = work + (p & 1) * WY_NB * ldv, *Tb = Tall + p * 64;
    // warp 0: the next panel's tile, then that panel; the others the rest
    wy_tiles<true>(A, lda, n, j0, p + 1 + warp, warp == 0 ? np : Z2_WARPS - 1, np, Vb, ldv, Tb);
    if (warp == 0)
      warp_qr_panel_safe<SH, T>(A, lda, n, j0 + WY_NB, work + ((p + 1) & 1) * WY_NB * ldv, ldv,
                                Tall + (p + 1) * 64, vd, zs);
    __syncthreads();
  }
}

// The T factors of reflectors that came without them (the pivoted QR: v(j) = 1,
// coefficients tau): one panel per warp, S = V^T V by DMMA, T by the recurrence
// of warp_qr_panel; vd = 1.
template <bool SH>
static __device__ __noinline__ void blk_wy_t(const double *A, int lda, int n, const double *tau, double *vd,
                                      double *work) {
  if (SH) A = as_shared(const_cast<double *>(A));
  double *Tall = as_shared(work) + 2 * WY_NB * wy_ldv(n);
  const int lane = threadIdx.x & 31, lr = lane >> 2, lc = lane & 3;
  for (int i = threadIdx.x; i < n; i += Z2_NT) vd[i] = 1.0;
  for (int p = threadIdx.x >> 5; p < wy_panels(n); p += Z2_WARPS) {
    const int j0 = p * WY_NB, mp = n - j0, ib = mp < WY_NB ? mp : WY_NB;
    const double *Ap = A + j0 + (size_t)j0 * lda;
    double w[4][2] = {};
    for (int l = 0; l < mp; l += 16) {
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        const int r = l + 4 * u + lc;
        const double v = (r < mp && lr < ib && r >= lr) ? (r == lr ? 1.0 : Ap[r + (size_t)lr * lda]) : 0.0;
        dmma884(w[u][0], w[u][1], v, v);
      }
    }
    // lane i: row i of S (columns > i are used) and of T
    const double s0 = (w[0][0] + w[1][0]) + (w[2][0] + w[3][0]);
    const double s1 = (w[0][1] + w[1][1]) + (w[2][1] + w[3][1]);
    double tr[8];
#pragma unroll
    for (int k = 0; k < 8; ++k) {
      double s = 0.0;
#pragma unroll
      for (int q = 0; q < k; ++q)
        s = fma(tr[q], __shfl_sync(Z2_FULL, (k & 1) ? s1 : s0, 4 * q + (k >> 1)), s);
      const double tk = k < ib ? tau[j0 + k] : 0.0;
      tr[k] = lane == k ? tk : (lane < k ? -tk * s : 0.0);
    }
    if (lane < 8) {
#pragma unroll
      for (int c = 0; c < 8; ++c) Tall[p * 64 + c * 8 + lane] = tr[c];
    }
  }
  __syncthreads();
}

// Reflectors of panel p clean into Vb, and the panel's columns of A set to
// those of the unit matrix.
__device__ __forceinline__ void wy_load_v(double *A, int lda, int n, int p, const double *vd, double *Vb,
                                          int ldv, int w, int nw) {
  const int j0 = p * WY_NB, ib = (n - j0) < WY_NB ? (n - j0) : WY_NB;
  const int n8 = (n + 7) & ~7;
  for (int c = w; c < WY_NB; c += nw) {
    double *Ac = A + (size_t)(j0 + c) * lda;
    for (int r = threadIdx.x & 31; r < n8; r += 32) {
      if (c < ib && r < n) {
        const double x = Ac[r];
        if (r >= j0) Vb[r + c * ldv] = r == j0 + c ? vd[r] : (r > j0 + c ? x : 0.0);
        Ac[r] = r == j0 + c ? 1.0 : 0.0;
      } else if (r >= j0) {
        Vb[r + c * ldv] = 0.0;
      }
    }
  }
}

// DORGQR: Q = H_0 H_1 ... H_{n-1} over the reflectors in A, from the last panel
// to the first, with the T factors in work (blk_qr_panels or blk_wy_t).  The
// next panel's reflectors are taken out of A while the current one is
// applied: one block barrier per panel.
template <bool SH>
static __device__ __noinline__ void blk_form_q(double *A, int lda, int n, const double *vd, double *work) {
  if (SH) A = as_shared(A);
  work = as_shared(work);
  const int warp = threadIdx.x >> 5;
  const int ldv = wy_ldv(n), np = wy_panels(n);
  const double *Tall = work + 2 * WY_NB * ldv;
  wy_load_v(A, lda, n, np - 1, vd, work + ((np - 1) & 1) * WY_NB * ldv, ldv, warp, Z2_WARPS);
  __syncthreads();
  for (int p = np - 1; p >= 0; --p) {
    const double *Vb = work + (p & 1) * WY_NB * ldv;
    if (p > 0)
      wy_load_v(A, lda, n, p - 1, vd, work + ((p - 1) & 1) * WY_NB * ldv, ldv, Z2_WARPS - 1 - warp, Z2_WARPS);
    wy_tiles<false>(A, lda, n, p * WY_NB, p + warp, Z2_WARPS, np, Vb, ldv, Tall + p * 64);
    __syncthreads();
  }
}

// ---------------------------------------------------------------------------
// Gauss-Jordan inverse with partial pivoting
// ---------------------------------------------------------------------------
// u = a[i] for the warp-uniform i in [LO, HI), by halving.
template <int LO, int HI, int T>
__device__ __forceinline__ void pick_row(int i, const double (&a)[T][8], double (&u)[8]) {
  if constexpr (HI - LO == 1) {
#pragma unroll
    for (int c = 0; c < 8; ++c) u[c] = a[LO][c];
  } else {
    constexpr int MID = (LO + HI) / 2;
    if (i < MID) pick_row<LO, MID>(i, a, u);
    else pick_row<MID, HI>(i, a, u);
  }
}

// Eight exchange steps on the panel M(:, j0:j0+8) by one warp, n <= 32 T: step
// k picks the largest entry of column k among the rows not yet used (to
// within 2^-12 relative: the high word of |a|, which orders like the value,
// with its low byte replaced by 255 - row, ties to the smaller row),
// p with pivot d and l_r = a(r, k):
//   a(p, :) /= d, a(r, c) -= l_r a(p, c), a(r, k) = -l_r / d, a(p, k) = 1 / d.
// On exit the panel (in M and in Zb, rows up to the next multiple of 8) holds
// Z: the columns outside the panel become C(r, :) + Z(r, :) C(P, :) with
// C(P, :) read as zero on the left.  A picked row is kept times its pivot
// until the end (its multiplier at its own step is 0).
template <int T>
__device__ __forceinline__ unsigned warp_gj_panel(double *M, int ldm, int n, int j0, double *Zb, int ldv,
                                                  int *piv, unsigned used) {
  const int lane = threadIdx.x & 31;
  const int ib = (n - j0) < WY_NB ? (n - j0) : WY_NB;
  double *Mp = M + j0 * ldm;
  double a[T][8], scl[T];
#pragma unroll
  for (int t = 0; t < T; ++t) {
    const int r = lane + 32 * t;
    scl[t] = 1.0;
#pragma unroll
    for (int c = 0; c < 8; ++c) a[t][c] = (r < n && c < ib) ? Mp[r + c * ldm] : 0.0;
  }
  // one step: the panel's column k, in the registers' column 0
  const auto step = [&](int k) {
    unsigned key = 0;
#pragma unroll
    for (int t = 0; t < T; ++t) {
      const unsigned h = ((unsigned)__double2hiint(fabs(a[t][0])) & 0xFFFFFF00u) |
                         (unsigned)(255 - (lane + 32 * t));
      if (!((used >> t) & 1u)) key = max(key, h);
    }
    key = __reduce_max_sync(Z2_FULL, key);
    const int br = 255 - (int)(key & 0xFFu), ol = br & 31, ot = br >> 5;
    double u[8];
    pick_row<0, T>(ot, a, u);                       // uniform branches
#pragma unroll
    for (int c = 0; c < 8; ++c) u[c] = __shfl_sync(Z2_FULL, u[c], ol);
    const double rd = rcp_newton(u[0]);
    if (lane == 0) piv[j0 + k] = br;
#pragma unroll
    for (int c = 0; c < 8; ++c) u[c] *= rd;
#pragma unroll
    for (int t = 0; t < T; ++t) {
      const bool isp = t == ot && lane == ol;
      const double l = isp ? 0.0 : a[t][0];
#pragma unroll
      for (int c = 1; c < 8; ++c) a[t][c] = fma(-l, u[c], a[t][c]);
      a[t][0] = isp ? 1.0 : -l * rd;
      if (isp) { scl[t] = rd; used |= 1u << t; }
    }
  };
  // a loop over the columns, the current one rotated to the front: 8 T moves a
  // step for an eighth of the code (unrolled, alone on an SM: the same within 1 %
  // at N = 36 ... 144; the SM's instruction cache is shared by several blocks in
  // the 128-thread build)
#pragma unroll 1
  for (int k = 0; k < 8; ++k) {
    if (k < ib) step(k);
#pragma unroll
    for (int t = 0; t < T; ++t) {
      const double f = a[t][0];
#pragma unroll
      for (int c = 0; c < 7; ++c) a[t][c] = a[t][c + 1];
      a[t][7] = f;
    }
  }
  const int n8 = (n + 7) & ~7;
#pragma unroll
  for (int t = 0; t < T; ++t) {
    const int r = lane + 32 * t;
    if (r < n8) {
#pragma unroll
      for (int c = 0; c < 8; ++c) {
        const double z = a[t][c] * scl[t];
        if (r < n && c < ib) Mp[r + c * ldm] = z;
        Zb[r + c * ldv] = z;
      }
    }
  }
  __syncwarp();
  return used;
}

// C <- (C with the panel's pivot rows zeroed) + Z C(P, :) for NT tiles of 8
// columns of M by one warp.
template <int NT>
__device__ __forceinline__ void gj_tile(double *M, int ldm, int n, const int (&c0)[NT], const double *Zb,
                                        int ldv, const int *piv, int ib) {
  const int lane = threadIdx.x & 31, lr = lane >> 2, lc = lane & 3;
  double b[NT][2];
#pragma unroll
  for (int s = 0; s < 2; ++s) {
    const int k = 4 * s + lc, pr = k < ib ? piv[k] : 0;
#pragma unroll
    for (int i = 0; i < NT; ++i) {
      const int cb = c0[i] + lr;
      const bool ok = k < ib && cb < n;
      double *e = M + (ok ? pr + cb * ldm : 0);
      b[i][s] = ok ? *e : 0.0;
      if (ok) *e = 0.0;
    }
  }
  __syncwarp();
  panel_update<NT>(M, ldm, n, 0, c0, Zb, ldv, b);
}

// The panel's update of column tiles number first, first + step, ... < count
// (tile number i is column tile map(i)) by the calling warp, in pairs.
template <class Map>
__device__ __forceinline__ void gj_tiles(double *M, int ldm, int n, int first, int step, int count, Map map,
                                         const double *Zb, int ldv, const int *piv, int ib) {
  int i = first;
  for (; i + step < count; i += 2 * step) {
    const int c[2] = {map(i) * WY_NB, map(i + step) * WY_NB};
    gj_tile<2>(M, ldm, n, c, Zb, ldv, piv, ib);
  }
  if (i < count) {
    const int c[1] = {map(i) * WY_NB};
    gj_tile<1>(M, ldm, n, c, Zb, ldv, piv, ib);
  }
}

// Inverse of the n x n matrix M in place by blocked Gauss-Jordan, n <= 32 T <=
// 256, rows not swapped: with piv[j] the pivot row of column j,
//   M^-1(j, piv[m]) = (M on exit)(piv[j], m).
// work: 2 WY_NB wy_ldv(n) doubles of shared memory, piv n ints of it.
template <bool SH, int T>
static __device__ __noinline__ void blk_gj_panels(double *M, int ldm, int n, int *piv, double *work) {
  if (SH) M = as_shared(M);
  work = as_shared(work);
  piv = as_shared(piv);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int ldv = wy_ldv(n), np = wy_panels(n);
  unsigned used = 0;                                // warp 0: bit t, row lane + 32 t
#pragma unroll
  for (int t = 0; t < T; ++t)
    if (lane + 32 * t >= n) used |= 1u << t;
  if (warp == 0) used = warp_gj_panel<T>(M, ldm, n, 0, work, ldv, piv, used);
  __syncthreads();
  for (int p = 0; p < np; ++p) {
    const int j0 = p * WY_NB, ib = (n - j0) < WY_NB ? (n - j0) : WY_NB;
    const double *Zb = work + (p & 1) * WY_NB * ldv;
    if (p + 1 < np) {
      // warp 0: the next panel's tile, then that panel; the others the rest
      if (warp == 0) {
        const int c[1] = {j0 + WY_NB};
        gj_tile<1>(M, ldm, n, c, Zb, ldv, piv + j0, ib);
        used = warp_gj_panel<T>(M, ldm, n, j0 + WY_NB, work + ((p + 1) & 1) * WY_NB * ldv, ldv, piv, used);
      } else {
        gj_tiles(M, ldm, n, warp - 1, Z2_WARPS - 1, np - 2, [p](int i) { return i < p ? i : i + 2; }, Zb, ldv,
                 piv + j0, ib);
      }
    } else {
      gj_tiles(M, ldm, n, warp, Z2_WARPS, p, [](int i) { return i; }, Zb, ldv, piv + j0, ib);
    }
    __syncthreads();
  }
}
