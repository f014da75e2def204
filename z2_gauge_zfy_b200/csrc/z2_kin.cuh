// z2_kin.cuh -- the checkerboard kinetic propagator (src/operator_kin.f90:61-179).
//
// B = E0 E1 E2 E3 E3 E2 E1 E0, E_g the product of group g's disjoint bond
// rotations [a, b] <- [[C, S], [S, C]] [a, b], S = sigma sinh.  On an Lx x Ly
// lattice with periodic boundaries (sites y Lx + x) the four groups are the x
// bonds from odd x (group 0) and from even x (group 1), and the y bonds from
// odd y (group 2) and from even y (group 3), each listed row by row
// (HostLattice, src/lattice.f90:72-102):
//   group 0: bond (y Lx + x, y Lx + x+1 mod Lx), x = 2m+1, table slot y Lx/2 + m
//   group 1: x = 2m, same slots;  group 2: (y Lx + x, (y+1 mod Ly) Lx + x),
//   y = 2m+1, slot m Lx + x;  group 3: y = 2m, same slots.
// Groups 0 and 1 only mix the sites of one lattice row and groups 2 and 3
// only those of one lattice column, so the passes 0 1 | 2 3 3 2 | 1 0 run as
// three sweeps over lines: a thread loads one line (or two neighbouring ones)
// of a matrix column (or of two neighbouring matrix rows) into registers as
// 16-byte words, applies its passes (E3 E3 as one rotation) and stores it, so
// the matrix crosses shared memory three times per product.
//
// Bound: shared-memory bandwidth.  N = 144: the two products of a slice move
// 2 MB, 15.5 K cycles at 128 B/clk; the previous sweeps (generic addresses,
// two coefficient loads per rotation) took 41 K.
#pragma once
#include "z2_linalg.cuh"

// Checkerboard group of pass p = 0..7 of one B (src/operator_kin.f90:74-85).
__device__ __forceinline__ int kin_pass_group(int p) { return p < 4 ? p : 7 - p; }

// The part of the slice table that does not change: position q = g half + k
// holds bond groups[q]: its sites, C, sinh (in S's place) and, in gid, the bond
// with the sign of sinh on top.  Once per launch and chain.
static __device__ __noinline__ void kin_init(const ChainDesc &c, const Smem &s) {
  for (int q = threadIdx.x; q < c.nb; q += Z2_NT) {
    const int b = c.groups[q];
    const double sh = c.chsh[2 * b + 1];
    s.tp[2 * q] = c.bonds[2 * b];
    s.tp[2 * q + 1] = c.bonds[2 * b + 1];
    s.cs[q] = make_double2(c.chsh[2 * b], sh);
    s.gid[q] = (short)(b | (sh < 0.0 ? 0x4000 : 0));
    s.bond[2 * q] = c.bonds[2 * q];
    s.bond[2 * q + 1] = c.bonds[2 * q + 1];
  }
  __syncthreads();
}

// S of slice nt: sigma sinh(alpha).
__device__ __forceinline__ void build_table_on(const signed char *sg, int nb, double2 *cs, const short *gid) {
  for (int q = threadIdx.x; q < nb; q += Z2_NT) {
    const int g = gid[q];
    const int neg = (sg[g & 0x3fff] < 0) ^ ((g >> 14) & 1);
    const double a = fabs(cs[q].y);
    cs[q].y = neg ? -a : a;
  }
  __syncthreads();
}

static __device__ __noinline__ void build_table(const ChainDesc &c, const Smem &s, int nt) {
  build_table_on(c.sigma + (size_t)(nt - 1) * c.nb, c.nb, as_shared(s.cs), as_shared(s.gid));
}

// One bond (process_group): one product, one FMA per output.
__device__ __forceinline__ void kin_rot(double &a, double &b, double2 k) {
  const double na = __fma_rn(k.x, a, __dmul_rn(k.y, b));
  const double nb = __fma_rn(k.y, a, __dmul_rn(k.x, b));
  a = na;
  b = nb;
}
__device__ __forceinline__ double2 kin_coef(const double2 *cs, int q, double fl) {
  const double2 k = cs[q];
  return make_double2(k.x, fl * k.y);
}
// E E: cosh and sinh of the doubled angle.
__device__ __forceinline__ double2 kin_twice(double2 k) {
  return make_double2(fma(k.x, k.x, k.y * k.y), 2.0 * k.x * k.y);
}

// The passes of one line of L sites: x lines: odd (before), even, odd (after)
// bonds; y lines (Y): odd, even twice, odd.  co, ce: the coefficients of the odd
// (2m+1, 2m+2) and even (2m, 2m+1) bonds, st slots apart.
template <int L, bool Y>
__device__ __forceinline__ void kin_line(double (&v)[L], const double2 *co, const double2 *ce, int st, double fl,
                                         bool before, bool after) {
  if (Y || before) {      // uniform
#pragma unroll
    for (int m = 0; m < L / 2; ++m) kin_rot(v[2 * m + 1], v[(2 * m + 2) % L], kin_coef(co, m * st, fl));
  }
#pragma unroll
  for (int m = 0; m < L / 2; ++m) {
    const double2 k = kin_coef(ce, m * st, fl);
    kin_rot(v[2 * m], v[2 * m + 1], Y ? kin_twice(k) : k);
  }
  if (Y || after) {
#pragma unroll
    for (int m = 0; m < L / 2; ++m) kin_rot(v[2 * m + 1], v[(2 * m + 2) % L], kin_coef(co, m * st, fl));
  }
}

// One sweep of M <- B^fl M (ROWS: vectors are the columns of M, sites contiguous)
// or M <- M B^fl (vectors are pairs of rows, sites ld apart) for n vectors: x
// lines (Y false) or y lines (Y) of L sites.  A thread takes one (line, vector)
// item at a time, vector fastest: ROWS y lines two neighbouring lattice columns
// (16-byte words), the others one line, of two neighbouring matrix rows if
// !ROWS.  (Keeping a line's coefficients in registers over a warp's share of
// the vectors spilled and measured slower than reading them.)  M in shared
// memory, 16-byte aligned, ld and n even.
template <bool ROWS, bool Y, int L>
__device__ __forceinline__ void kin_sweep_on(const double2 *cs, double *M, int ld, int n, int Lx, int Ly,
                                             double fl, bool before, bool after) {
  const int half = (Lx * Ly) >> 1;
  constexpr bool PAIR = ROWS && Y;
  const int nv = ROWS ? n : n >> 1;
  const int items = nv * (Y ? (PAIR ? Lx >> 1 : Lx) : Ly);
  const int dl = Z2_NT / nv, di = Z2_NT - dl * nv;
  int line = threadIdx.x / nv, i = threadIdx.x - line * nv;
  for (int e = threadIdx.x; e < items; e += Z2_NT) {
    const int q = Y ? (PAIR ? 2 * line : line) : line * (L >> 1);   // first slot of the line
    const double2 *co = cs + (Y ? 2 * half : 0) + q, *ce = co + half;
    const int qs = Y ? Lx : 1;
    if constexpr (ROWS && !PAIR) {
      double2 *p = reinterpret_cast<double2 *>(M + i * ld) + line * (L >> 1);
      double v[L];
#pragma unroll
      for (int x = 0; x < L / 2; ++x) {
        const double2 w = p[x];
        v[2 * x] = w.x;
        v[2 * x + 1] = w.y;
      }
      kin_line<L, Y>(v, co, ce, qs, fl, before, after);
#pragma unroll
      for (int x = 0; x < L / 2; ++x) p[x] = make_double2(v[2 * x], v[2 * x + 1]);
    } else {
      double2 *p;
      int st;      // in 16-byte words
      if (ROWS) {
        p = reinterpret_cast<double2 *>(M + i * ld) + line;
        st = Lx >> 1;
      } else {
        p = reinterpret_cast<double2 *>(M + 2 * i + (Y ? line : line * L) * ld);
        st = (Y ? Lx * ld : ld) >> 1;
      }
      double v[L], w[L];
#pragma unroll
      for (int x = 0; x < L; ++x) {
        const double2 u = p[x * st];
        v[x] = u.x;
        w[x] = u.y;
      }
      kin_line<L, Y>(v, co, ce, qs, fl, before, after);
      kin_line<L, Y>(w, PAIR ? co + 1 : co, PAIR ? ce + 1 : ce, qs, fl, before, after);
#pragma unroll
      for (int x = 0; x < L; ++x) p[x * st] = make_double2(v[x], w[x]);
    }
    i += di;
    line += dl;
    if (i >= nv) { i -= nv; ++line; }
  }
  __syncthreads();
}

template <bool ROWS, bool Y, int L, bool SH>
static __device__ __noinline__ void kin_sweep(const double2 *cs, double *M, int ld, int n, int Lx, int Ly, double fl,
                                       bool before, bool after) {
  kin_sweep_on<ROWS, Y, L>(as_shared(const_cast<double2 *>(cs)), SH ? as_shared(M) : M, ld, n, Lx, Ly, fl, before,
                           after);
}

template <bool ROWS, bool Y, bool SH>
__device__ __forceinline__ void kin_sweep_any(const Smem &s, double *M, int ld, int n, int Lx, int Ly, double fl,
                                              bool before, bool after) {
  switch (Y ? Ly : Lx) {
    case 4: kin_sweep<ROWS, Y, 4, SH>(s.cs, M, ld, n, Lx, Ly, fl, before, after); return;
    case 6: kin_sweep<ROWS, Y, 6, SH>(s.cs, M, ld, n, Lx, Ly, fl, before, after); return;
    case 8: kin_sweep<ROWS, Y, 8, SH>(s.cs, M, ld, n, Lx, Ly, fl, before, after); return;
    case 10: kin_sweep<ROWS, Y, 10, SH>(s.cs, M, ld, n, Lx, Ly, fl, before, after); return;
    case 12: kin_sweep<ROWS, Y, 12, SH>(s.cs, M, ld, n, Lx, Ly, fl, before, after); return;
    case 14: kin_sweep<ROWS, Y, 14, SH>(s.cs, M, ld, n, Lx, Ly, fl, before, after); return;
    case 16: kin_sweep<ROWS, Y, 16, SH>(s.cs, M, ld, n, Lx, Ly, fl, before, after); return;
    default: return;
  }
}

// Lines of 2 sites or more than 16: group by group, one thread per vector (column of M
// at stride 1, or row at stride ld), eight disjoint rotations at a time loaded,
// rotated and stored as a whole.
__device__ __forceinline__ void kin_group_vec(const Smem &s, double *base, size_t stride, int g0, int half,
                                              double fl) {
  const int2 *__restrict__ tp2 = reinterpret_cast<const int2 *>(as_shared(s.tp));
  const double2 *__restrict__ cs = as_shared(s.cs);
  int kq = 0;
  for (; kq + 7 < half; kq += 8) {
    int2 pp[8];
    double2 k[8];
    double a[8], b[8];
#pragma unroll
    for (int q = 0; q < 8; ++q) {
      pp[q] = tp2[g0 + kq + q];
      k[q] = kin_coef(cs, g0 + kq + q, fl);
    }
#pragma unroll
    for (int q = 0; q < 8; ++q) { a[q] = base[pp[q].x * stride]; b[q] = base[pp[q].y * stride]; }
#pragma unroll
    for (int q = 0; q < 8; ++q) {
      kin_rot(a[q], b[q], k[q]);
      base[pp[q].x * stride] = a[q];
      base[pp[q].y * stride] = b[q];
    }
  }
  for (; kq < half; ++kq) {
    const int2 pp = tp2[g0 + kq];
    double a = base[pp.x * stride], b = base[pp.y * stride];
    kin_rot(a, b, kin_coef(cs, g0 + kq, fl));
    base[pp.x * stride] = a;
    base[pp.y * stride] = b;
  }
}

// Sweep K (0: groups 0 1; 1: groups 2 3 3 2; 2: groups 1 0) of M <- B^nflag M
// (rows) or M <- M B^nflag, M in shared memory and fit for the line sweeps.
template <bool ROWS, bool SH>
__device__ __forceinline__ void kin_lines(const ChainDesc &c, const Smem &s, double *M, int ld, int n, double fl,
                                          int K) {
  if (K == 1) kin_sweep_any<ROWS, true, SH>(s, M, ld, n, c.Lx, c.Ly, fl, true, true);
  else kin_sweep_any<ROWS, false, SH>(s, M, ld, n, c.Lx, c.Ly, fl, K == 0, K == 2);
}
template <bool ROWS>
__device__ __forceinline__ void kin_groups(const ChainDesc &c, const Smem &s, double *M, int ld, int n, double fl,
                                           int p0, int p1) {
  for (int i = threadIdx.x; i < n; i += Z2_NT)
    for (int p = p0; p < p1; ++p)
      kin_group_vec(s, ROWS ? M + (size_t)i * ld : M + i, ROWS ? 1 : (size_t)ld, kin_pass_group(p) * c.half, c.half, fl);
  __syncthreads();
}
// Sweeps k0 <= K < k1 of M <- B^nflag M for n columns (ROWS) or M <- M B^nflag for
// n rows.  In global memory (N > 144; the arena is free whenever this is called
// then) B M passes through shared memory in slabs of columns, one read and one
// write instead of one of each per sweep; M B, whose loads are whole lines of row
// pairs, sweeps in place (16x16: B M 207 us in place, 96 in slabs; M B 53 and 104).
template <bool ROWS>
static __device__ __noinline__ void kin_apply(const ChainDesc &c, const Smem &s, double *M, int ld, int n, int nflag,
                                       int k0, int k1) {
  const double fl = (double)nflag;
  const int N = c.N;
  if (c.kin_lines && ((ld | n) & 1) == 0 && ((size_t)M & 15) == 0) {
    if (__isShared(M)) {
      for (int k = k0; k < k1; ++k) kin_lines<ROWS, true>(c, s, M, ld, n, fl, k);
      return;
    }
    if constexpr (Z2_NMAX > 64 && !ROWS) {
      for (int k = k0; k < k1; ++k) kin_lines<false, false>(c, s, M, ld, n, fl, k);
      return;
    }
    const int w = (s.tile_doubles / (N + 2) - 2) & ~1;      // columns of a slab
    if (Z2_NMAX > 64 && !c.g_in_smem && w >= 16) {
      for (int i = 0; i < n; i += w) {
        const int m = min(w, n - i);
        double *src = M + (size_t)i * ld;
        blk_copy(s.tile, N + 2, src, ld, N, m);
        for (int k = k0; k < k1; ++k) kin_lines<ROWS, true>(c, s, s.tile, N + 2, m, fl, k);
        blk_copy(src, ld, s.tile, N + 2, N, m);
      }
      return;
    }
  }
  const int p[4] = {0, 2, 6, 8};
  kin_groups<ROWS>(c, s, M, ld, n, fl, p[k0], p[k1]);
}

// M <- B^nflag M (row rotations) for n columns; M <- M B^nflag for n rows.
__device__ __forceinline__ void kin_rows(const ChainDesc &c, const Smem &s, double *M, int ld, int n, int nflag) {
  kin_apply<true>(c, s, M, ld, n, nflag, 0, 3);
}
__device__ __forceinline__ void kin_cols(const ChainDesc &c, const Smem &s, double *M, int ld, int n, int nflag) {
  kin_apply<false>(c, s, M, ld, n, nflag, 0, 3);
}

// Slices t = t0, t0 + dt, ... , t1 of an L x L lattice on the shared matrix M:
// M <- B_t^rf M (rf != 0), then M <- M B_t^cf (cf != 0).  One function per L for
// the whole of it: a call costs its registers' round trip through local
// memory, which on small lattices was as much as a sweep.
template <int L>
static __device__ __noinline__ void kin_square(const ChainDesc &c, const Smem &s, double *M, int ld, int t0, int t1,
                                        int dt, int rf, int cf) {
  M = as_shared(M);
  double2 *cs = as_shared(s.cs);
  const short *gid = as_shared(s.gid);
  const signed char *sigma = c.sigma;
  constexpr int N = L * L;
  const double fr = (double)rf, fc = (double)cf;
  for (int t = t0;; t += dt) {
    build_table_on(sigma + (size_t)(t - 1) * (2 * N), 2 * N, cs, gid);
    if (rf) {
      kin_sweep_on<true, false, L>(cs, M, ld, N, L, L, fr, true, false);
      kin_sweep_on<true, true, L>(cs, M, ld, N, L, L, fr, true, true);
      kin_sweep_on<true, false, L>(cs, M, ld, N, L, L, fr, false, true);
    }
    if (cf) {
      kin_sweep_on<false, false, L>(cs, M, ld, N, L, L, fc, true, false);
      kin_sweep_on<false, true, L>(cs, M, ld, N, L, L, fc, true, true);
      kin_sweep_on<false, false, L>(cs, M, ld, N, L, L, fc, false, true);
    }
    if (t == t1) break;
  }
}

// The same for any lattice and matrix (N x N).
__device__ __forceinline__ void kin_slices(const ChainDesc &c, const Smem &s, double *M, int ld, int t0, int t1,
                                           int dt, int rf, int cf) {
  if (c.kin_lines && c.Lx == c.Ly && (ld & 1) == 0 && ((size_t)M & 15) == 0 && __isShared(M)) {
    switch (c.Lx) {
      case 4: kin_square<4>(c, s, M, ld, t0, t1, dt, rf, cf); return;
      case 6: kin_square<6>(c, s, M, ld, t0, t1, dt, rf, cf); return;
      case 8: kin_square<8>(c, s, M, ld, t0, t1, dt, rf, cf); return;
      case 10:
        if constexpr (Z2_NMAX > 64) { kin_square<10>(c, s, M, ld, t0, t1, dt, rf, cf); return; }
        break;
      case 12:
        if constexpr (Z2_NMAX > 64) { kin_square<12>(c, s, M, ld, t0, t1, dt, rf, cf); return; }
        break;
      default: break;
    }
  }
  for (int t = t0;; t += dt) {
    build_table(c, s, t);
    if (rf) kin_rows(c, s, M, ld, c.N, rf);
    if (cf) kin_cols(c, s, M, ld, c.N, cf);
    if (t == t1) break;
  }
}

// M <- B_nt^row_flag M, then M <- M B_nt^col_flag (0: not) of a global N x N matrix,
// staged through the arena when it fits (the arena must be free).
static __device__ __noinline__ void kin_global(const ChainDesc &c, const Smem &s, int nt, double *M,
                                               int row_flag, int col_flag) {
  const int N = c.N;
  if (c.g_in_smem) {
    double *A = s.arena;
    blk_copy(A, c.ldg, M, N, N, N);
    kin_slices(c, s, A, c.ldg, nt, nt, 1, row_flag, col_flag);
    blk_copy(M, N, A, c.ldg, N, N);
  } else {
    kin_slices(c, s, M, N, nt, nt, 1, row_flag, col_flag);
  }
}
