// z2_gemm.cuh -- the square N x N x N products of the stabilization on DMMA.
//
// Each warp forms units of (8 RT) x (8 CT) entries over the whole k range,
// straight from global or shared memory: an operand fragment is used for RT or
// CT products.  (Loading the next eight k values ahead of the products in the
// middle units: 0.5 % slower bins at N = 64, 1 % at N = 100.)
#pragma once
#include "z2_blocked.cuh"

// C = op(A B) of a product: C(i, j) = rs[i] v (rs null: v) for plain products,
// and with rs2: C(i, j) = C(i, j) rs[i] cs[j] + rs2[i] v cs2[j].
struct GemmOut {
  double *C;
  int ldc;
  const double *rs = nullptr, *cs = nullptr, *rs2 = nullptr, *cs2 = nullptr;
};

// The k loop of a unit: VA / VB: 16-byte loads of that operand (k contiguous,
// aligned, the other stride even); TRI 1: A(i, l) reads as 0 for i > l, TRI 2:
// B(l, j) reads as 0 for l < j (the loop starts at the unit's first row / column).
// Lane lc takes k = l0 + 2 lc and l0 + 2 lc + 1 of every eight.
template <int RT, int CT, bool VA, bool VB, int TRI>
__device__ __forceinline__ void gemm_unit(int n, MatRef A, MatRef B, int r0, int c0, const int (&oa)[RT],
                                          const int (&ob)[CT], double (&acc)[RT][CT][2]) {
  const int lane = threadIdx.x & 31, lr = lane >> 2, lc = lane & 3;
  const int n8 = n & ~7;
  const int lb = TRI == 1 ? r0 : (TRI == 2 ? c0 : 0);
  const double *pa = A.p + (lb + 2 * lc) * A.cs, *pb = B.p + (lb + 2 * lc) * B.rs;
  const int sa = 8 * A.cs, sb = 8 * B.rs;
  const auto load = [&](double2 (&fa)[RT], double2 (&fb)[CT]) {
#pragma unroll
    for (int a = 0; a < RT; ++a)
      fa[a] = VA ? *reinterpret_cast<const double2 *>(pa + oa[a]) : make_double2(pa[oa[a]], pa[oa[a] + A.cs]);
#pragma unroll
    for (int b = 0; b < CT; ++b)
      fb[b] = VB ? *reinterpret_cast<const double2 *>(pb + ob[b]) : make_double2(pb[ob[b]], pb[ob[b] + B.rs]);
    pa += sa;
    pb += sb;
  };
  const auto mul = [&](int l, double2 (&fa)[RT], double2 (&fb)[CT]) {
    if (TRI == 1) {
#pragma unroll
      for (int a = 0; a < RT; ++a) {
        const int r = r0 + 8 * a + lr;
        if (r > l) fa[a].x = 0.0;
        if (r > l + 1) fa[a].y = 0.0;
      }
    }
    if (TRI == 2) {
#pragma unroll
      for (int b = 0; b < CT; ++b) {
        const int c = c0 + 8 * b + lr;
        if (l < c) fb[b].x = 0.0;
        if (l + 1 < c) fb[b].y = 0.0;
      }
    }
#pragma unroll
    for (int a = 0; a < RT; ++a)
#pragma unroll
      for (int b = 0; b < CT; ++b) dmma884(acc[a][b][0], acc[a][b][1], fa[a].x, fb[b].x);
#pragma unroll
    for (int a = 0; a < RT; ++a)
#pragma unroll
      for (int b = 0; b < CT; ++b) dmma884(acc[a][b][0], acc[a][b][1], fa[a].y, fb[b].y);
  };
#pragma unroll 1
  for (int l = lb + 2 * lc; l < n8; l += 8) {
    double2 fa[RT], fb[CT];
    load(fa, fb);
    mul(l, fa, fb);
  }
  if (n8 < n) {              // four trailing k values
    const int l = n8 + lc;
    double fa[RT], fb[CT];
#pragma unroll
    for (int a = 0; a < RT; ++a) {
      const double x = A.p[l * A.cs + oa[a]];
      fa[a] = (TRI == 1 && r0 + 8 * a + lr > l) ? 0.0 : x;
    }
#pragma unroll
    for (int b = 0; b < CT; ++b) {
      const double x = B.p[l * B.rs + ob[b]];
      fb[b] = (TRI == 2 && l < c0 + 8 * b + lr) ? 0.0 : x;
    }
#pragma unroll
    for (int a = 0; a < RT; ++a)
#pragma unroll
      for (int b = 0; b < CT; ++b) dmma884(acc[a][b][0], acc[a][b][1], fa[a], fb[b]);
  }
}

// C = A B (out), n % 4 == 0; rowmap (optional): row i of A is its row rowmap[i].
template <int RT, int CT, bool VA, bool VB, int TRI>
static __device__ __noinline__ void gemm_units(int n, MatRef A, const int *rowmap, MatRef B, const GemmOut &out) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int lr = lane >> 2, lc = lane & 3;
  const int tiles = (n + 7) >> 3;
  const int ur = (tiles + RT - 1) / RT, uc = (tiles + CT - 1) / CT;
  for (int g = warp; g < ur * uc; g += Z2_WARPS) {
    const int r0 = (g % ur) * 8 * RT, c0 = (g / ur) * 8 * CT;
    int oa[RT], ob[CT];      // element offsets of this lane's rows and columns (k = 0)
#pragma unroll
    for (int a = 0; a < RT; ++a) {
      const int r = min(r0 + 8 * a + lr, n - 1);
      oa[a] = (rowmap ? rowmap[r] : r) * A.rs;
    }
#pragma unroll
    for (int b = 0; b < CT; ++b) ob[b] = min(c0 + 8 * b + lr, n - 1) * B.cs;
    double acc[RT][CT][2];
#pragma unroll
    for (int a = 0; a < RT; ++a)
#pragma unroll
      for (int b = 0; b < CT; ++b) acc[a][b][0] = acc[a][b][1] = 0.0;
    gemm_unit<RT, CT, VA, VB, TRI>(n, A, B, r0, c0, oa, ob, acc);
    double *C = out.C;
    const int ldc = out.ldc;
    const bool comb = out.rs2 != nullptr;
#pragma unroll
    for (int a = 0; a < RT; ++a) {
      const int r = r0 + 8 * a + lr;
      if (r < n) {
        const double s = out.rs ? out.rs[r] : 1.0, s2 = comb ? out.rs2[r] : 0.0;
#pragma unroll
        for (int b = 0; b < CT; ++b)
#pragma unroll
          for (int e = 0; e < 2; ++e) {
            const int c = c0 + 8 * b + 2 * lc + e;
            if (c < n) {
              double *p = C + r + c * ldc;
              *p = comb ? fma(s2 * acc[a][b][e], out.cs2[c], *p * s * out.cs[c]) : s * acc[a][b][e];
            }
          }
      }
    }
  }
  __syncthreads();
}

template <bool VA, bool VB, int TRI>
__device__ __forceinline__ void gemm_sized(int n, MatRef A, const int *rowmap, MatRef B, const GemmOut &out) {
  const int t = (n + 7) >> 3;
  if (t <= 5) gemm_units<1, 2, VA, VB, TRI>(n, A, rowmap, B, out);
  else if (Z2_NMAX <= 64 || t <= 8) gemm_units<2, Z2_NT == 256 ? 4 : 2, VA, VB, TRI>(n, A, rowmap, B, out);
  else if constexpr (Z2_NMAX > 64) {
    if (t <= 12) gemm_units<3, 3, VA, VB, TRI>(n, A, rowmap, B, out);
    else if (t <= 14) gemm_units<2, 7, VA, VB, TRI>(n, A, rowmap, B, out);
    else gemm_units<3, 9, VA, VB, TRI>(n, A, rowmap, B, out);
  }
}

// The product in units that cut the (N / 8)^2 tiles into a multiple of the four
// sub-partitions' tensor pipes where they can (18 x 18 tiles: 12 units of 3 x 9,
// three per sub-partition), with as many products per fragment as registers
// allow: N = 144 takes 90 K cycles against 103 K for 16 x 16 groups (47 K at the
// SM's DMMA rate; the fragment loads' trips to L2 are the rest).  a_upper: A(i, l)
// reads as 0 for i > l; b_lower: B(l, j) reads as 0 for l < j.
static __device__ __noinline__ void gemm_nnn(int n, MatRef A, const int *rowmap, bool a_upper, MatRef B,
                                      bool b_lower, GemmOut out) {
  const bool va = A.cs == 1 && (A.rs & 1) == 0 && ((uintptr_t)A.p & 15) == 0;
  const bool vb = B.rs == 1 && (B.cs & 1) == 0 && ((uintptr_t)B.p & 15) == 0;
  if (a_upper) gemm_sized<false, false, 1>(n, A, rowmap, B, out);
  else if (b_lower) gemm_sized<false, false, 2>(n, A, rowmap, B, out);
  else if (va && vb) gemm_sized<true, true, 0>(n, A, rowmap, B, out);
  else if (vb) gemm_sized<false, true, 0>(n, A, rowmap, B, out);
  else gemm_sized<false, false, 0>(n, A, rowmap, B, out);
}
