// z2_linalg.cuh -- CTA-cooperative dense FP64 linear algebra.
//
// Every routine is called by all Z2_NT threads of a block, operates on
// column-major matrices through generic pointers (shared or global memory)
// and ends with the block synchronised.  The routines restate the LAPACK /
// BLAS operations the reference's stabilization calls (ZGEQP3, ZUNGQR,
// ZUNMQR, ZTRMM, ZTRSM, ZLAPMR, ZLAPMT, ZGEMM; src/stabilization.f90:42-200)
// for real matrices, with the same algorithms (Householder reflectors of
// DLARFG, partial column-norm downdating of DLAQP2, column-oriented
// triangular solves of DTRSM).
#pragma once
#include "z2_common.cuh"

__device__ __forceinline__ double dlapy2(double x, double y) {
  double xa = fabs(x), ya = fabs(y);
  double w = fmax(xa, ya), z = fmin(xa, ya);
  if (z == 0.0) return w;
  double q = z / w;
  return w * sqrt(1.0 + q * q);
}

// Element walk over an m x n column-major block whose operands sit in L2 or
// HBM: the elements are dealt to the threads in column-major order
// (consecutive threads take consecutive rows, so accesses stay coalesced), B
// per thread at a time, and every batch issues its B loads before any use.  ld(i, j) returns
// the element's operands, use(v, i, j) consumes them.
template <int B, class T, class Ld, class Use>
__device__ __forceinline__ void blk_walk(int m, int n, Ld ld, Use use) {
  if (m <= 0 || n <= 0) return;
  const int dj = Z2_NT / m, di = Z2_NT % m;
  int i = threadIdx.x % m, j = threadIdx.x / m;
  const long long total = (long long)m * n;
  for (long long e0 = 0; e0 < total; e0 += (long long)B * Z2_NT) {
    int ii[B], jj[B];
    T v[B];
#pragma unroll
    for (int b = 0; b < B; ++b) {
      ii[b] = i;
      jj[b] = j;
      if (j < n) v[b] = ld(i, j);
      i += di;
      j += dj;
      if (i >= m) { i -= m; ++j; }
    }
#pragma unroll
    for (int b = 0; b < B; ++b)
      if (jj[b] < n) use(v[b], ii[b], jj[b]);
  }
}

// dst = src.  Pairs of rows move as 16-byte words, eight per thread in flight
// (m, both leading dimensions even and both pointers 16-byte aligned), dealt
// out flat over the block: the copies wait on L2, 144 x 144 took 20 K cycles as
// one column per warp with four loads in flight.
static __device__ __noinline__ void blk_copy(double *dst, int ldd, const double *src, int lds, int m, int n) {
  if (!((m | ldd | lds) & 1) && !(((size_t)dst | (size_t)src) & 15)) {
    double2 *d = reinterpret_cast<double2 *>(dst);
    const double2 *s = reinterpret_cast<const double2 *>(src);
    const int hd = ldd >> 1, hs = lds >> 1;
    blk_walk<8, double2>(
        m >> 1, n, [&](int i, int j) { return s[i + j * hs]; },
        [&](double2 v, int i, int j) { d[i + j * hd] = v; });
    __syncthreads();
    return;
  }
  const int lane = threadIdx.x & 31;
  for (int j = threadIdx.x / 32; j < n; j += Z2_WARPS)
    for (int i = lane; i < m; i += 32) dst[i + (size_t)j * ldd] = src[i + (size_t)j * lds];
  __syncthreads();
}
// dst = src^T (src m x n -> dst n x m)
static __device__ __noinline__ void blk_transpose(double *dst, int ldd, const double *src, int lds, int m, int n) {
  for (int j = threadIdx.x / 32; j < m; j += Z2_WARPS)
    for (int i = threadIdx.x & 31; i < n; i += 32) dst[i + (size_t)j * ldd] = src[j + (size_t)i * lds];
  __syncthreads();
}
static __device__ __noinline__ void blk_identity(double *A, int lda, int n) {
  for (int j = threadIdx.x / 32; j < n; j += Z2_WARPS)
    for (int i = threadIdx.x & 31; i < n; i += 32) A[i + (size_t)j * lda] = (i == j) ? 1.0 : 0.0;
  __syncthreads();
}
static __device__ __noinline__ void blk_fill(double *v, int n, double x) {
  for (int i = threadIdx.x; i < n; i += Z2_NT) v[i] = x;
  __syncthreads();
}
static __device__ __noinline__ void blk_scale(double *A, int lda, int m, int n, double a) {
  for (int j = threadIdx.x / 32; j < n; j += Z2_WARPS)
    for (int i = threadIdx.x & 31; i < m; i += 32) A[i + (size_t)j * lda] *= a;
  __syncthreads();
}
// A(:, j) *= d(j)
static __device__ __noinline__ void blk_scale_cols(double *A, int lda, int m, int n, const double *d) {
  for (int j = threadIdx.x / 32; j < n; j += Z2_WARPS) {
    double dj = d[j];
    for (int i = threadIdx.x & 31; i < m; i += 32) A[i + (size_t)j * lda] *= dj;
  }
  __syncthreads();
}

// ---------------------------------------------------------------------------
// Pivoted Householder QR (DGEQP3 -> DLAQP2 semantics, all columns free).
// On exit A holds R and the reflectors, tau the scalar factors, jpvt the
// 1-based pivots (column j of A*P is column jpvt(j) of A).
// ---------------------------------------------------------------------------
static __device__ __noinline__ void blk_geqp3(double *A, int lda, int n, int *jpvt, double *tau, double *vn1,
                          double *vn2) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const double tol3z = 1.0536712127723509e-08;   // sqrt(dlamch('E')) = sqrt(2^-53)
  for (int j = warp; j < n; j += Z2_WARPS) {
    double s = 0.0;
    for (int i = lane; i < n; i += 32) { double a = A[i + (size_t)j * lda]; s += a * a; }
    s = warp_sum(s);
    if (lane == 0) { double nr = sqrt(s); vn1[j] = nr; vn2[j] = nr; jpvt[j] = j + 1; }
  }
  __syncthreads();
  for (int j = 0; j < n; ++j) {
    // IDAMAX over vn1(j:n): first index of the largest value
    double bv = -1.0; int bi = n;
    for (int k = j + lane; k < n; k += 32) { double v = vn1[k]; if (v > bv) { bv = v; bi = k; } }
#pragma unroll
    for (int o = 16; o; o >>= 1) {
      double ov = __shfl_xor_sync(Z2_FULL, bv, o);
      int oi = __shfl_xor_sync(Z2_FULL, bi, o);
      if (ov > bv || (ov == bv && oi < bi)) { bv = ov; bi = oi; }
    }
    const int pvt = bi < n ? bi : j;   // no candidate: a column of NaNs
    __syncthreads();
    if (warp == 0) {
      double *Aj = A + (size_t)j * lda;
      if (pvt != j) {
        double *Ap = A + (size_t)pvt * lda;
        for (int i = lane; i < n; i += 32) { double t = Ap[i]; Ap[i] = Aj[i]; Aj[i] = t; }
        if (lane == 0) {
          int t = jpvt[pvt]; jpvt[pvt] = jpvt[j]; jpvt[j] = t;
          vn1[pvt] = vn1[j]; vn2[pvt] = vn2[j];
        }
      }
      __syncwarp();
      // DLARFG on A(j:n, j)
      double s = 0.0;
      for (int i = j + 1 + lane; i < n; i += 32) { double a = Aj[i]; s += a * a; }
      s = warp_sum(s);
      double alpha = Aj[j];
      double t = 0.0, beta = alpha;
      if (j < n - 1 && s != 0.0) {
        double xnorm = sqrt(s);
        beta = -copysign(dlapy2(alpha, xnorm), alpha);
        t = (beta - alpha) / beta;
        double sc = 1.0 / (alpha - beta);
        for (int i = j + 1 + lane; i < n; i += 32) Aj[i] *= sc;
      }
      __syncwarp();
      if (lane == 0) { tau[j] = t; Aj[j] = beta; }
    }
    __syncthreads();
    // DLARF('Left') on the trailing columns + norm downdate, one warp per column
    const double tj = tau[j];
    const double *v = A + (size_t)j * lda;
    for (int k = j + 1 + warp; k < n; k += Z2_WARPS) {
      double *Ak = A + (size_t)k * lda;
      if (tj != 0.0) {
        double w = 0.0;
        for (int i = j + 1 + lane; i < n; i += 32) w += v[i] * Ak[i];
        w = warp_sum(w) + Ak[j];
        double tw = tj * w;
        __syncwarp();
        if (lane == 0) Ak[j] -= tw;
        for (int i = j + 1 + lane; i < n; i += 32) Ak[i] -= v[i] * tw;
      }
      __syncwarp();
      double v1 = vn1[k];
      if (v1 != 0.0) {
        double r = fabs(Ak[j]) / v1;
        double temp = fmax(1.0 - r * r, 0.0);
        double q = v1 / vn2[k];
        double temp2 = temp * q * q;
        if (temp2 <= tol3z) {
          double nv = 0.0;
          if (j < n - 1) {
            double s2 = 0.0;
            for (int i = j + 1 + lane; i < n; i += 32) { double a = Ak[i]; s2 += a * a; }
            nv = sqrt(warp_sum(s2));
          }
          if (lane == 0) { vn1[k] = nv; vn2[k] = nv; }
        } else if (lane == 0) {
          vn1[k] = v1 * sqrt(temp);
        }
      }
    }
    __syncthreads();
  }
}

// QDRP_decompose's split (src/stabilization.f90:61-66): D(i) = |R(i,i)|,
// R(i, i:n) /= D(i).
// The rows are scaled by the reciprocal of D (one division per row instead
// of one per element; rd: n doubles of scratch, left holding 1/D).
static __device__ __noinline__ void blk_qdrp_scale(double *A, int lda, int n, double *D, double *rd) {
  for (int i = threadIdx.x; i < n; i += Z2_NT) {
    const double d = fabs(A[i + (size_t)i * lda]);
    D[i] = d;
    rd[i] = 1.0 / d;
  }
  __syncthreads();
  for (int j = threadIdx.x / 32; j < n; j += Z2_WARPS)
    for (int i = threadIdx.x & 31; i <= j; i += 32) A[i + (size_t)j * lda] = A[i + (size_t)j * lda] * rd[i];
  __syncthreads();
}

// Row / column permutations with 1-based pivots (ZLAPMR, ZLAPMT).
// forward row: dst(i,:) = src(jpvt(i),:) ; backward row: dst(jpvt(i),:) = src(i,:)
static __device__ __noinline__ void blk_perm_rows(double *dst, int ldd, const double *src, int lds, int n, int nc,
                              const int *jpvt, bool forward) {
  for (int j = threadIdx.x / 32; j < nc; j += Z2_WARPS)
    for (int i = threadIdx.x & 31; i < n; i += 32) {
      int p = jpvt[i] - 1;
      if (forward) dst[i + (size_t)j * ldd] = src[p + (size_t)j * lds];
      else dst[p + (size_t)j * ldd] = src[i + (size_t)j * lds];
    }
  __syncthreads();
}
// forward col: dst(:,j) = src(:,jpvt(j)) ; backward col: dst(:,jpvt(j)) = src(:,j)
static __device__ __noinline__ void blk_perm_cols(double *dst, int ldd, const double *src, int lds, int nr, int n,
                              const int *jpvt, bool forward) {
  for (int j = threadIdx.x / 32; j < n; j += Z2_WARPS) {
    int p = jpvt[j] - 1;
    for (int i = threadIdx.x & 31; i < nr; i += 32) {
      if (forward) dst[i + (size_t)j * ldd] = src[i + (size_t)p * lds];
      else dst[i + (size_t)p * ldd] = src[i + (size_t)j * lds];
    }
  }
  __syncthreads();
}
