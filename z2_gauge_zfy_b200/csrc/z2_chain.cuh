// z2_chain.cuh -- per-chain DQMC drivers run by one CTA.
//
// Restates the reference's hot path (src/local_sweep.f90, src/localK.f90,
// src/multiply.f90, src/operator_kin.f90, src/stabilization.f90,
// src/dynamics.f90, src/obser_equal.f90, src/obser_tau.f90) for one spin
// sector in real FP64.  Orders of operations follow the reference; the
// implementation is B200-first: G stays in shared memory across a slice,
// accepted flips are queued as rank-2 factors and flushed as one rank-2k
// update, and the U factors of the UDV chains are propagated lazily (all
// Nwrap slices at once, right before the stabilization that needs them).
#pragma once
#include "z2_propose.cuh"
#include "z2_stab.cuh"

// Checkerboard group order of one B (src/operator_kin.f90:74-85).
__device__ __constant__ int c_gorder[8] = {0, 1, 2, 3, 3, 2, 1, 0};

// ---------------------------------------------------------------------------
// Shared-memory layout
// ---------------------------------------------------------------------------
__device__ __forceinline__ size_t align16(size_t x) { return (x + 15) & ~size_t(15); }

__device__ Smem make_smem(const ChainDesc &c, unsigned char *base, size_t smem_bytes) {
  Smem s;
  const int N = c.N;
  size_t off = 0;
  s.red = (double *)(base + off); off += sizeof(double) * Z2_NRED;
  s.vec = (double *)(base + off); off += sizeof(double) * 8 * N;
  s.tc = (double *)(base + off); off += sizeof(double) * 2 * N;
  s.ts = (double *)(base + off); off += sizeof(double) * 2 * N;
  s.ivec = (int *)(base + off); off += align16(sizeof(int) * 2 * N);
  s.tp = (int *)(base + off); off += align16(sizeof(int) * 4 * N);
  s.bond = (int *)(base + off); off += align16(sizeof(int) * 4 * N);
  s.flag = (int *)(base + off); off += sizeof(int) * 16;
  s.sig = (signed char *)(base + off); off += align16(6 * N);   // slices nt, nt-1, nt+1
  off = align16(off);
  s.arena = (double *)(base + off);
  const size_t arena_doubles = (smem_bytes - off) / sizeof(double);
  const size_t nn = (size_t)N * c.ldg;
  if (c.g_in_smem) {
    s.G = s.arena; s.ldg = c.ldg;
    s.ldx = z2_ldx(N); s.X = s.arena + nn; s.Yt = s.X + (size_t)s.ldx * c.k2;
    s.Wq = s.arena; s.ldq = c.ldg;
    s.tile = s.arena + nn;
    s.tile_doubles = (int)(arena_doubles - nn);
  } else {
    s.G = c.G; s.ldg = N;
    s.ldx = z2_ldx(N); s.X = s.arena; s.Yt = s.X + (size_t)s.ldx * c.k2;
    s.Wq = c.W4;
    s.ldq = N;
    s.tile = s.arena;
    s.tile_doubles = (int)arena_doubles;
  }
  return s;
}

// ---------------------------------------------------------------------------
// Checkerboard kinetic propagator (src/operator_kin.f90:61-179)
// ---------------------------------------------------------------------------
// Slice table in group order: position q = g*half + k holds bond groups[q].
__device__ __noinline__ void build_table(const ChainDesc &c, const Smem &s, int nt) {
  const signed char *sg = c.sigma + (size_t)(nt - 1) * c.nb;
  for (int q = threadIdx.x; q < c.nb; q += Z2_NT) {
    int b = c.groups[q];
    s.tp[2 * q] = c.bonds[2 * b];
    s.tp[2 * q + 1] = c.bonds[2 * b + 1];
    s.tc[q] = c.chsh[2 * b];
    s.ts[q] = (double)sg[b] * c.chsh[2 * b + 1];   // sinh(alpha*sigma) = sigma*sinh(alpha)
  }
  __syncthreads();
}

// One bond of a checkerboard group (process_group): [a, b] <- [[C, S], [S, C]]
// [a, b], with the rounding sequence fixed (one product, one FMA per output)
// so that every kinetic kernel below gives the same bits.
__device__ __forceinline__ void kin_rot(double &a, double &b, double C, double S) {
  const double na = __fma_rn(C, a, __dmul_rn(S, b));
  const double nb = __fma_rn(S, a, __dmul_rn(C, b));
  a = na;
  b = nb;
}

// M <- B^nflag M : rows P1, P2 rotated by [[C,S],[S,C]] (process_group).
// Row rotations never mix columns, so one thread carries its column through
// all eight group passes: no barrier between passes.
// Bonds of one group are disjoint, so a batch of 8 rotations is loaded,
// rotated and stored as a whole (no store-to-load ordering inside a batch).
template <bool ROWS>
__device__ __forceinline__ void kin_group_vec(const Smem &s, double *base, size_t stride, int g0,
                                              int half, double fl) {
  // table pointers in registers (the Smem struct would otherwise be re-read
  // after every store, which may alias it)
  const int2 *__restrict__ tp2 = reinterpret_cast<const int2 *>(s.tp);
  const double *__restrict__ tc = s.tc;
  const double *__restrict__ ts = s.ts;
  int kq = 0;
  for (; kq + 7 < half; kq += 8) {
    int2 pp[8];
    double C[8], S[8], a[8], b[8];
#pragma unroll
    for (int q = 0; q < 8; ++q) {
      pp[q] = tp2[g0 + kq + q];
      C[q] = tc[g0 + kq + q];
      S[q] = fl * ts[g0 + kq + q];
    }
#pragma unroll
    for (int q = 0; q < 8; ++q) { a[q] = base[pp[q].x * stride]; b[q] = base[pp[q].y * stride]; }
#pragma unroll
    for (int q = 0; q < 8; ++q) {
      kin_rot(a[q], b[q], C[q], S[q]);
      base[pp[q].x * stride] = a[q];
      base[pp[q].y * stride] = b[q];
    }
  }
  for (; kq < half; ++kq) {
    const int2 pp = tp2[g0 + kq];
    const double C = tc[g0 + kq], S = fl * ts[g0 + kq];
    double a = base[pp.x * stride], b = base[pp.y * stride];
    kin_rot(a, b, C, S);
    base[pp.x * stride] = a;
    base[pp.y * stride] = b;
  }
}

// Fused passes on an L x L lattice with periodic boundaries (sites
// y L + x).  The four groups are the x bonds from odd x (group 0) and from
// even x (group 1), and the y bonds from odd y (group 2) and from even y
// (group 3), each listed row by row (HostLattice, src/lattice.f90:72-102):
//   group 0: bond (y L + x, y L + x+1 mod L), x = 2m+1, table slot y L/2 + m
//   group 1: x = 2m, same slots;  group 2: (y L + x, (y+1 mod L) L + x),
//   y = 2m+1, slot m L + x;  group 3: y = 2m, same slots.
// Groups 0 and 1 only mix the sites of one lattice row and groups 2 and 3
// only those of one lattice column, so the pass sequence 0 1 | 2 3 3 2 | 1 0
// runs as three sweeps over lines: a thread loads one line of one matrix
// column (or row) into registers, applies its passes and stores it, instead
// of streaming the whole matrix through shared memory once per pass.  The
// rotations and their order within each bond are those of the pass-by-pass
// kernel, so the results are bitwise equal.
template <int L>
__device__ __forceinline__ void kin_line_odd(double (&v)[L], const double *__restrict__ tc,
                                             const double *__restrict__ ts, double fl, int q0,
                                             int qs) {
#pragma unroll
  for (int m = 0; m < L / 2; ++m) {
    const int q = q0 + m * qs;
    kin_rot(v[2 * m + 1], v[(2 * m + 2) % L], tc[q], fl * ts[q]);
  }
}
template <int L>
__device__ __forceinline__ void kin_line_even(double (&v)[L], const double *__restrict__ tc,
                                              const double *__restrict__ ts, double fl, int q0,
                                              int qs) {
#pragma unroll
  for (int m = 0; m < L / 2; ++m) {
    const int q = q0 + m * qs;
    kin_rot(v[2 * m], v[2 * m + 1], tc[q], fl * ts[q]);
  }
}

// The three sweeps for n independent vectors: vector i's site k sits at
// M[i * vs + k * ks] (kin_rows: vs = ld, ks = 1; kin_cols: vs = 1, ks = ld).
// Threads take (vector, line) pairs, vector fastest, so a warp touches one
// line of 32 consecutive vectors.
template <int L>
__device__ __noinline__ void kin_fused(const Smem &s, double *M, size_t vs, size_t ks, int n,
                                       int nflag) {
  constexpr int H = L * L / 2, HL = L / 2;
  const double fl = (double)nflag;
  const double *__restrict__ tc = s.tc;
  const double *__restrict__ ts = s.ts;
  const int tasks = n * L;
  // a lattice row of one matrix column is contiguous when ks == 1: with an
  // even column stride and an aligned matrix it moves as 16-byte pairs
  const bool pairs = ks == 1 && (vs & 1) == 0 && (reinterpret_cast<size_t>(M) & 15) == 0;
  // groups 0, 1 on lattice rows
  for (int t = threadIdx.x; t < tasks; t += Z2_NT) {
    const int i = t % n, y = t / n;
    double *p = M + (size_t)i * vs + (size_t)(y * L) * ks;
    double v[L];
    if (pairs) {
#pragma unroll
      for (int x = 0; x < L; x += 2) {
        const double2 w = reinterpret_cast<const double2 *>(p)[x >> 1];
        v[x] = w.x; v[x + 1] = w.y;
      }
    } else {
#pragma unroll
      for (int x = 0; x < L; ++x) v[x] = p[(size_t)x * ks];
    }
    kin_line_odd<L>(v, tc, ts, fl, y * HL, 1);
    kin_line_even<L>(v, tc, ts, fl, H + y * HL, 1);
    if (pairs) {
#pragma unroll
      for (int x = 0; x < L; x += 2) reinterpret_cast<double2 *>(p)[x >> 1] = make_double2(v[x], v[x + 1]);
    } else {
#pragma unroll
      for (int x = 0; x < L; ++x) p[(size_t)x * ks] = v[x];
    }
  }
  __syncthreads();
  // groups 2, 3, 3, 2 on lattice columns
  for (int t = threadIdx.x; t < tasks; t += Z2_NT) {
    const int i = t % n, x = t / n;
    double *p = M + (size_t)i * vs + (size_t)x * ks;
    double v[L];
#pragma unroll
    for (int y = 0; y < L; ++y) v[y] = p[(size_t)(y * L) * ks];
    kin_line_odd<L>(v, tc, ts, fl, 2 * H + x, L);
    kin_line_even<L>(v, tc, ts, fl, 3 * H + x, L);
    kin_line_even<L>(v, tc, ts, fl, 3 * H + x, L);
    kin_line_odd<L>(v, tc, ts, fl, 2 * H + x, L);
#pragma unroll
    for (int y = 0; y < L; ++y) p[(size_t)(y * L) * ks] = v[y];
  }
  __syncthreads();
  // groups 1, 0 on lattice rows
  for (int t = threadIdx.x; t < tasks; t += Z2_NT) {
    const int i = t % n, y = t / n;
    double *p = M + (size_t)i * vs + (size_t)(y * L) * ks;
    double v[L];
    if (pairs) {
#pragma unroll
      for (int x = 0; x < L; x += 2) {
        const double2 w = reinterpret_cast<const double2 *>(p)[x >> 1];
        v[x] = w.x; v[x + 1] = w.y;
      }
    } else {
#pragma unroll
      for (int x = 0; x < L; ++x) v[x] = p[(size_t)x * ks];
    }
    kin_line_even<L>(v, tc, ts, fl, H + y * HL, 1);
    kin_line_odd<L>(v, tc, ts, fl, y * HL, 1);
    if (pairs) {
#pragma unroll
      for (int x = 0; x < L; x += 2) reinterpret_cast<double2 *>(p)[x >> 1] = make_double2(v[x], v[x + 1]);
    } else {
#pragma unroll
      for (int x = 0; x < L; ++x) p[(size_t)x * ks] = v[x];
    }
  }
  __syncthreads();
}

// kin_fused for M <- M B (vectors are the rows of M, sites stride ld) when ld
// is even: a thread takes two adjacent rows, so every site moves as one
// 16-byte pair; the rotations and their order are kin_fused's.
template <int L>
__device__ __forceinline__ void kin_pair_odd(double (&v)[L], double (&w)[L], const double *__restrict__ tc,
                                             const double *__restrict__ ts, double fl, int q0, int qs) {
#pragma unroll
  for (int m = 0; m < L / 2; ++m) {
    const int q = q0 + m * qs;
    const double C = tc[q], S = fl * ts[q];
    kin_rot(v[2 * m + 1], v[(2 * m + 2) % L], C, S);
    kin_rot(w[2 * m + 1], w[(2 * m + 2) % L], C, S);
  }
}
template <int L>
__device__ __forceinline__ void kin_pair_even(double (&v)[L], double (&w)[L], const double *__restrict__ tc,
                                              const double *__restrict__ ts, double fl, int q0, int qs) {
#pragma unroll
  for (int m = 0; m < L / 2; ++m) {
    const int q = q0 + m * qs;
    const double C = tc[q], S = fl * ts[q];
    kin_rot(v[2 * m], v[2 * m + 1], C, S);
    kin_rot(w[2 * m], w[2 * m + 1], C, S);
  }
}
template <int L>
__device__ __noinline__ void kin_fused_rowpairs(const Smem &s, double *M, size_t ld, int n, int nflag) {
  constexpr int H = L * L / 2, HL = L / 2;
  const double fl = (double)nflag;
  const double *__restrict__ tc = s.tc;
  const double *__restrict__ ts = s.ts;
  const int n2 = n >> 1, tasks = n2 * L;
  for (int sweep = 0; sweep < 3; ++sweep) {
    for (int t = threadIdx.x; t < tasks; t += Z2_NT) {
      const int i = 2 * (t % n2), line = t / n2;
      double v[L], w[L];
      // sweep 0 and 2: lattice row `line` (sites line L + x); sweep 1:
      // lattice column `line` (sites y L + line)
      const size_t base = (sweep == 1) ? (size_t)line * ld : (size_t)(line * L) * ld;
      const size_t step = (sweep == 1) ? (size_t)L * ld : ld;
      double2 *p = reinterpret_cast<double2 *>(M + i + base);
      const size_t st2 = step >> 1;
#pragma unroll
      for (int x = 0; x < L; ++x) {
        const double2 u = p[(size_t)x * st2];
        v[x] = u.x; w[x] = u.y;
      }
      if (sweep == 0) {
        kin_pair_odd<L>(v, w, tc, ts, fl, line * HL, 1);
        kin_pair_even<L>(v, w, tc, ts, fl, H + line * HL, 1);
      } else if (sweep == 1) {
        kin_pair_odd<L>(v, w, tc, ts, fl, 2 * H + line, L);
        kin_pair_even<L>(v, w, tc, ts, fl, 3 * H + line, L);
        kin_pair_even<L>(v, w, tc, ts, fl, 3 * H + line, L);
        kin_pair_odd<L>(v, w, tc, ts, fl, 2 * H + line, L);
      } else {
        kin_pair_even<L>(v, w, tc, ts, fl, H + line * HL, 1);
        kin_pair_odd<L>(v, w, tc, ts, fl, line * HL, 1);
      }
#pragma unroll
      for (int x = 0; x < L; ++x) p[(size_t)x * st2] = make_double2(v[x], w[x]);
    }
    __syncthreads();
  }
}

// kin_fused for the lattice sizes it is instantiated for; false otherwise.
__device__ __forceinline__ bool kin_fused_any(int L, const Smem &s, double *M, size_t vs, size_t ks,
                                              int n, int nflag) {
  switch (L) {
    case 4: kin_fused<4>(s, M, vs, ks, n, nflag); return true;
    case 6: kin_fused<6>(s, M, vs, ks, n, nflag); return true;
    case 8: kin_fused<8>(s, M, vs, ks, n, nflag); return true;
    case 10: kin_fused<10>(s, M, vs, ks, n, nflag); return true;
    case 12: kin_fused<12>(s, M, vs, ks, n, nflag); return true;
    case 14: kin_fused<14>(s, M, vs, ks, n, nflag); return true;
    case 16: kin_fused<16>(s, M, vs, ks, n, nflag); return true;
    default: return false;
  }
}

__device__ __noinline__ void kin_rows(const ChainDesc &c, const Smem &s, double *M, int ld, int ncols,
                         int nflag) {
  if (kin_fused_any(c.kin_fused, s, M, (size_t)ld, 1, ncols, nflag)) return;
  const int half = c.half;
  const double fl = (double)nflag;
  for (int col = threadIdx.x; col < ncols; col += Z2_NT) {
    double *mc = M + (size_t)col * ld;
    for (int p = 0; p < 8; ++p) kin_group_vec<true>(s, mc, 1, c_gorder[p] * half, half, fl);
  }
  __syncthreads();
}

// M <- M B^nflag : columns P1, P2 rotated (process_group_L); one thread per
// row through all eight passes.
__device__ __noinline__ void kin_cols(const ChainDesc &c, const Smem &s, double *M, int ld, int nrows,
                         int nflag) {
  if ((ld & 1) == 0 && (nrows & 1) == 0 && (reinterpret_cast<size_t>(M) & 15) == 0) {
    switch (c.kin_fused) {
      case 4: kin_fused_rowpairs<4>(s, M, (size_t)ld, nrows, nflag); return;
      case 6: kin_fused_rowpairs<6>(s, M, (size_t)ld, nrows, nflag); return;
      case 8: kin_fused_rowpairs<8>(s, M, (size_t)ld, nrows, nflag); return;
      case 10: kin_fused_rowpairs<10>(s, M, (size_t)ld, nrows, nflag); return;
      case 12: kin_fused_rowpairs<12>(s, M, (size_t)ld, nrows, nflag); return;
      case 14: kin_fused_rowpairs<14>(s, M, (size_t)ld, nrows, nflag); return;
      case 16: kin_fused_rowpairs<16>(s, M, (size_t)ld, nrows, nflag); return;
      default: break;
    }
  }
  if (kin_fused_any(c.kin_fused, s, M, 1, (size_t)ld, nrows, nflag)) return;
  const int half = c.half;
  const double fl = (double)nflag;
  for (int row = threadIdx.x; row < nrows; row += Z2_NT) {
    double *mr = M + row;
    for (int p = 0; p < 8; ++p) kin_group_vec<false>(s, mr, (size_t)ld, c_gorder[p] * half, half, fl);
  }
  __syncthreads();
}

// One group (one factor E_g) of B applied to rows / columns.
__device__ __noinline__ void kin_group_rows(const ChainDesc &c, const Smem &s, double *M, int ld, int ncols,
                               int g, int nflag) {
  const int half = c.half, g0 = g * half;
  const double fl = (double)nflag;
  for (int col = threadIdx.x; col < ncols; col += Z2_NT)
    kin_group_vec<true>(s, M + (size_t)col * ld, 1, g0, half, fl);
  __syncthreads();
}
__device__ __noinline__ void kin_group_cols(const ChainDesc &c, const Smem &s, double *M, int ld, int nrows,
                               int g, int nflag) {
  const int half = c.half, g0 = g * half;
  const double fl = (double)nflag;
  for (int row = threadIdx.x; row < nrows; row += Z2_NT)
    kin_group_vec<false>(s, M + row, (size_t)ld, g0, half, fl);
  __syncthreads();
}

// Apply B-multiplications to a global N x N matrix, staging it through the
// arena when it fits (the arena must be free).
__device__ __noinline__ void kin_global(const ChainDesc &c, const Smem &s, double *M, int row_flag,
                           int col_flag) {
  const int N = c.N;
  if (c.g_in_smem) {
    double *A = s.arena;
    blk_copy(A, c.ldg, M, N, N, N);
    if (row_flag) kin_rows(c, s, A, c.ldg, N, row_flag);
    if (col_flag) kin_cols(c, s, A, c.ldg, N, col_flag);
    blk_copy(M, N, A, c.ldg, N, N);
  } else {
    if (row_flag) kin_rows(c, s, M, N, N, row_flag);
    if (col_flag) kin_cols(c, s, M, N, N, col_flag);
  }
}

// Lazily propagated U factors.  R chain: for nt' = lo..hi, U <- B_nt' U then
// U *= e^{dtau mu} (LocalK_prop_R + propT_R, src/localK.f90:395-396,
// src/multiply.f90:106).  L chain (ULT = UL^T, B symmetric): for nt' = hi
// down to lo, ULT *= e^{dtau mu} then ULT <- B_nt' ULT (propT_L + prop_L,
// src/multiply.f90:91, src/localK.f90:370).
__device__ __noinline__ void apply_pending_R(const ChainDesc &c, const Smem &s, double *A, int lda, int lo,
                                int hi, bool kin) {
  for (int t = lo; t <= hi; ++t) {
    if (kin) {
      build_table(c, s, t);
      kin_rows(c, s, A, lda, c.N, 1);
    }
    if (c.eP != 1.0) blk_scale(A, lda, c.N, c.N, c.eP);
  }
}
__device__ __noinline__ void apply_pending_L(const ChainDesc &c, const Smem &s, double *A, int lda, int lo,
                                int hi) {
  for (int t = hi; t >= lo; --t) {
    if (c.eP != 1.0) blk_scale(A, lda, c.N, c.N, c.eP);
    build_table(c, s, t);
    kin_rows(c, s, A, lda, c.N, 1);
  }
}

// ---------------------------------------------------------------------------
// Stabilization (src/stabilization.f90:42-264)
// ---------------------------------------------------------------------------
// stab_green_big (src/stabilization.f90:202-264): G(0,0), G(0,tau), G(tau,0),
// G(tau,tau) from the UDV factors of the two products.  The reference inverts a
// 2N x 2N matrix (its QR, the inverses of VR VL, VR, VL and bigV); the four
// blocks all contain the inverse of the same N x N middle matrix as stab_green:
// with B_tau..B_1 = UR DR VR, B_L..B_tau+1 = VL DL UL and
//   M' = DRb^-1 (UR^T UL^T) DLb^-1 + DRs (VR VL) DLs   (z2_stab.cuh)
//   G(tau,tau) = UL^T DLb^-1 M'^-1 DRb^-1 UR^T,   G(tau,0) = UL^T DLb^-1 M'^-1 DRs VR,
//   G(0,tau) = -VL DLs M'^-1 DRb^-1 UR^T,         G(0,0) = 1 - VL DLs M'^-1 DRs VR,
// every factor of order one, scales only divided out: one inverse and eight
// N x N x N products (at N = 100, 0.5 M cycles against 9 M for the 2N x 2N QR).
// M (ldm): work matrix (shared arena when it fits); W0..W3 N x N global
// workspaces; outputs N x N (ld N).
__device__ __noinline__ void dev_stab_green_big(const Smem &s, int N, const double *UR, const double *DR,
                                   const double *VR, const double *ULT, const double *DL,
                                   const double *VL, double *M, int ldm, double *W0, double *W1,
                                   double *W2, double *W3, double *G00, double *G0t, double *Gt0,
                                   double *Gtt) {
  double *rRb = s.vec + N, *rLb = s.vec + 2 * N, *neg = s.vec + 5 * N;
  int *piv = s.ivec, *inv = s.ivec + N;
  middle_inverse(s, N, UR, DR, VR, ULT, DL, VL, M, ldm, rRb, rLb, s.vec + 3 * N, s.vec + 4 * N, piv, W0,
                 W1);
  for (int m = threadIdx.x; m < N; m += Z2_NT) {
    inv[piv[m]] = m;
    neg[m] = -1.0;
  }
  __syncthreads();
  // DLb^-1 M'^-1 DRb^-1 UR^T -> W1; the columns of M times DR (DRs = DRb^-1 DR):
  // DLb^-1 M'^-1 DRs VR -> W2
  permute_cols(M, ldm, N, inv, rRb, W0);
  gemm_nnn(N, MatRef{M, 1, ldm}, piv, false, MatRef{UR, N, 1}, false, GemmOut{W1, N, rLb});
  blk_scale_cols(M, ldm, N, N, DR);
  gemm_nnn(N, MatRef{M, 1, ldm}, piv, false, MatRef{VR, 1, N}, false, GemmOut{W2, N, rLb});
  gemm_nnn(N, MatRef{ULT, 1, N}, nullptr, false, MatRef{W1, 1, N}, false, GemmOut{Gtt, N});
  gemm_nnn(N, MatRef{ULT, 1, N}, nullptr, false, MatRef{W2, 1, N}, false, GemmOut{Gt0, N});
  // DLs = DLb^-1 DL
  blk_walk<4, double2>(
      N, N, [&](int i, int j) { return make_double2(W1[i + (size_t)j * N], W2[i + (size_t)j * N]); },
      [&](double2 v, int i, int j) {
        W0[i + (size_t)j * N] = v.x * DL[i];
        W3[i + (size_t)j * N] = v.y * DL[i];
      });
  __syncthreads();
  gemm_nnn(N, MatRef{VL, 1, N}, nullptr, false, MatRef{W0, 1, N}, false, GemmOut{G0t, N, neg});
  gemm_nnn(N, MatRef{VL, 1, N}, nullptr, false, MatRef{W3, 1, N}, false, GemmOut{G00, N, neg});
  for (int i = threadIdx.x; i < N; i += Z2_NT) G00[i + (size_t)i * N] += 1.0;
  __syncthreads();
}

// ---------------------------------------------------------------------------
// Equal-time observables (Obs_equal_calc, src/obser_equal.f90:73-149)
// ---------------------------------------------------------------------------
__device__ __noinline__ void obs_equal(const ChainDesc &c, const Smem &s, int nt) {
  const int N = c.N;
  const double *G = s.G; const int ldg = s.ldg;
  const signed char *sg = c.sigma + (size_t)(nt - 1) * c.nb;
  double v[5] = {0, 0, 0, 0, 0};   // flux, pair, cdw, cdw_shift, density
  for (int i = threadIdx.x; i < N; i += Z2_NT) {
    const int *pl = c.plaq + 4 * i;
    v[0] += (double)sg[pl[0]] * (double)sg[pl[1]] * (double)sg[pl[2]] * (double)sg[pl[3]];
    double n = 1.0 - G[i + (size_t)i * ldg];
    v[4] += n + n;
  }
  const int W = 2 * c.Lx - 1;
  // task = (row i, one third of the columns j): the row's density, phase
  // and coordinates stay in registers, the warp's lanes take consecutive
  // rows (G(i, j) contiguous, G(j, i) at the stride ldg, column values
  // broadcast), and no element needs an index division
  const int J3 = (N + 2) / 3;
  for (int t = threadIdx.x; t < 3 * N; t += Z2_NT) {
    const int i = t % N, j0 = (t / N) * J3;
    const int j1 = (j0 + J3 < N) ? j0 + J3 : N;
    const double ni = 1.0 - G[i + (size_t)i * ldg];
    const double sti = c.stag[i];
    const int xi = c.xy[2 * i] + c.Lx - 1, yi = c.xy[2 * i + 1] + c.Ly - 1;
    const double *gi = G + i, *gj = G + (size_t)i * ldg;
#pragma unroll 4
    for (int j = j0; j < j1; ++j) {
      const double gij = gi[(size_t)j * ldg], gji = gj[j];
      const double nj = 1.0 - G[j + (size_t)j * ldg];
      const double dl = (i == j) ? 1.0 : 0.0;
      const double pq = dl - gij;
      v[1] += pq * pq;
      const double a = ni * nj;
      const double ex = (dl - gji) * gij;
      double dc = a - ex;
      dc = (dc + a) - ex;
      dc = (dc + a) + a;
      const double ph = sti * c.stag[j];
      const int dx = xi - c.xy[2 * j], dy = yi - c.xy[2 * j + 1];
      const double ps = c.pshift[dx + dy * W];
      v[2] += ph * dc;
      v[3] += ps * dc;
    }
  }
  blk_sum_n<5>(v, s.red);
  if (threadIdx.x == 0) {
    const double flux = v[0] / (double)N;
    acc_add(c, A_FLUX_SUM, flux);
    acc_add(c, A_FLUX_SQ, flux * flux);
    acc_add(c, A_PAIR, v[1]);
    acc_add(c, A_CDW, v[2]);
    acc_add(c, A_CDWS, v[3]);
    acc_add(c, A_DENS, v[4] / (double)N);
    acc_add(c, A_NOBS, 1.0);
  }
  __syncthreads();
}

// ---------------------------------------------------------------------------
// Time-displaced observables (Obs_tau_calc, src/obser_tau.f90:56-133), real
// parts, both identical spin sectors summed; binned by imj deterministically
// (one thread per displacement).
// ---------------------------------------------------------------------------
__device__ __noinline__ void obs_tau(const ChainDesc &c, const Smem &s, int nt) {
  const int N = c.N, Lx = c.Lx, Ly = c.Ly;
  const double *G00 = c.G00, *Gtt = c.Gtt, *Gt0 = c.Gt0, *G0t = c.G0t;
  const signed char *sgt = c.sigma + (size_t)(nt - 1) * c.nb;
  const signed char *sg1 = c.sigma;
  const double rt2 = c.rt_scalar * c.rt_scalar;
  for (int r = threadIdx.x; r < N; r += Z2_NT) {
    const int rx = c.xy[2 * r], ry = c.xy[2 * r + 1];
    double o[7] = {0, 0, 0, 0, 0, 0, 0};
    for (int ii = 0; ii < N; ++ii) {
      const int ix = c.xy[2 * ii], iy = c.xy[2 * ii + 1];
      int jx = ix - rx; if (jx < 1) jx += Lx;
      int jy = iy - ry; if (jy < 1) jy += Ly;
      const int jj = (jy - 1) * Lx + (jx - 1);
      const int ip = c.nbx[ii], jp = c.nbx[jj];
      // spin: sigma(ii, ntau) * sigma(jj, 1)
      o[0] += (double)sgt[ii] * (double)sg1[jj];
      const double g0t_ji = G0t[jj + (size_t)ii * N];
      const double gt0_ij = Gt0[ii + (size_t)jj * N];
      // single: term = Grt0u + Grt0d ; += term + conj(term)
      const double term = gt0_ij + gt0_ij;
      o[1] += term + term;
      // pair_d / pair_s: (diag1 + diag2) * 4
      const double d1 = g0t_ji * g0t_ji;
      const double pr = (d1 + d1) * 4.0;
      o[2] += pr;
      o[3] += pr;
      // charge: -Gr0t(jj,ii) Grt0(ii,jj) - conj(...) for both spins
      const double y = g0t_ji * gt0_ij;
      const double tt = 2.0 * (1.0 - Gtt[ii + (size_t)ii * N]);
      const double t0 = 2.0 * (1.0 - G00[jj + (size_t)jj * N]);
      const double chc = ((-y - y) - y) - y;
      o[4] += chc + (tt - tt) * (t0 - t0);
      o[5] += chc + (tt + tt) * (t0 + t0);
      // curxx with NB_field = 0
      const double tc = -G0t[jj + (size_t)ip * N] * Gt0[ii + (size_t)jp * N]
                        - G0t[jp + (size_t)ii * N] * Gt0[ip + (size_t)jj * N]
                        + G0t[jj + (size_t)ii * N] * Gt0[ip + (size_t)jp * N]
                        + G0t[jp + (size_t)ip * N] * Gt0[ii + (size_t)jj * N];
      const double cu = -rt2 * tc - rt2 * tc;
      o[6] += cu + cu;
    }
    double *ot = c.obs_tau + (size_t)(nt - 1) * N + r;
#pragma unroll
    for (int q = 0; q < 7; ++q) ot[(size_t)q * c.Ltrot * N] += o[q];
  }
  __syncthreads();
}

// ---------------------------------------------------------------------------
// Wraps (src/stabilization.f90:374-514)
// ---------------------------------------------------------------------------
struct Pend { int lo, hi; };   // lazily propagated slices, lo > hi = none

// Phase timer: accumulates SM cycles of a phase into the chain's counters.
struct PhTimer {
  const ChainDesc &c;
  int ph;
  long long t0;
  __device__ PhTimer(const ChainDesc &cc, int p) : c(cc), ph(p), t0(ph_now()) {}
  __device__ ~PhTimer() {
    if (threadIdx.x == 0) acc_add(c, A_PH0 + ph, (double)(ph_now() - t0));
  }
};

__device__ __forceinline__ double *qr_matrix(const ChainDesc &c, const Smem &s, int &ld) {
  ld = s.ldq;
  return s.Wq;
}

__device__ __noinline__ void spill_G(const ChainDesc &c, const Smem &s) {
  if (c.g_in_smem) blk_copy(c.G, c.N, s.G, s.ldg, c.N, c.N);
}
__device__ __noinline__ void load_G(const ChainDesc &c, const Smem &s) {
  if (c.g_in_smem) blk_copy(s.G, s.ldg, c.G, c.N, c.N, c.N);
}

// The stabilized Green's function Gn replaces the propagated one in one pass
// over both: returns the drift max |Gn - G| (compare_mat,
// src/stabilization.f90:365-372) and leaves G = Gn in global memory and, for
// a chain whose G lives in shared memory, there too.
__device__ __noinline__ double take_green(const ChainDesc &c, const Smem &s, const double *Gn) {
  const int N = c.N, ldg = s.ldg;
  double *Gg = c.G, *Gs = s.G;
  const bool sm = c.g_in_smem != 0;
  double m = 0.0;
  blk_walk<8, double2>(
      N, N, [&](int i, int j) { return make_double2(Gn[i + (size_t)j * N], Gg[i + (size_t)j * N]); },
      [&](double2 v, int i, int j) {
        const double d = fabs(v.x - v.y);
        m = (d > m || d != d) ? d : m;   // keep NaN visible
        Gg[i + (size_t)j * N] = v.x;
        if (sm) Gs[i + (size_t)j * ldg] = v.x;
      });
  const double r = blk_max(m, s.red);
  __syncthreads();
  return r;
}

__device__ __noinline__ void copy_vec(double *dst, const double *src, int n) {
  for (int i = threadIdx.x; i < n; i += Z2_NT) dst[i] = src[i];
  __syncthreads();
}

__device__ __noinline__ void record_drift(const ChainDesc &c, double dif, bool stats) {
  if (threadIdx.x == 0) {
    if (dif > c.acc[A_XMAX] || dif != dif) c.acc[A_XMAX] = dif;
    if (stats) c.acc[A_XMEAN] += dif;
    if (!(dif == dif) || isinf(dif)) atomicOr(c.status, ST_NONFINITE);
  }
}

// The chain's stabilization: the reference's pivoted QR, or the pre-pivoted
// blocked QR (dev_stab_U_fast / dev_stab_green_fast).
__device__ __forceinline__ void chain_stab_U(const ChainDesc &c, const Smem &s, double *A, int lda,
                                             double *U, double *D, double *V, bool left) {
  if (c.stab_exact) dev_stab_U(s, c.N, A, lda, U, D, V, c.W0, left);
  else dev_stab_U_fast(s, c.N, A, lda, U, D, V, c.W0, left);
}
__device__ __forceinline__ void chain_stab_green(const ChainDesc &c, const Smem &s, int nt, double *A,
                                                 int lda, double *Gout) {
  if (c.stab_exact)
    dev_stab_green(s, c.N, nt, c.Ltrot, c.UR, c.DR, c.VR, c.ULT, c.DL, c.VL, A, lda, c.W1, c.W2,
                   c.W0, Gout);
  else
    dev_stab_green_fast(s, c.N, nt, c.Ltrot, c.UR, c.DR, c.VR, c.ULT, c.DL, c.VL, A, lda, c.W1,
                        c.W2, c.W0, Gout);
}

// Wrap_pre (src/stabilization.f90:374-398)
__device__ __noinline__ void wrap_pre(const ChainDesc &c, const Smem &s, int nt, Pend &pd) {
  const int N = c.N, NN = N * N;
  int lda; double *A = qr_matrix(c, s, lda);
  const int st = nt / c.Nwrap;
  if (nt != 0) {
    blk_copy(A, lda, c.UR, N, N, N);
    { PhTimer t(c, PH_PEND); apply_pending_R(c, s, A, lda, pd.lo, pd.hi, c.use_kin != 0); }
    chain_stab_U(c, s, A, lda, c.UR, c.DR, c.VR, false);
  }
  pd.lo = 1; pd.hi = 0;
  { PhTimer t(c, PH_STACK);
    blk_copy(c.URs + (size_t)st * NN, N, c.UR, N, N, N);
    blk_copy(c.VRs + (size_t)st * NN, N, c.VR, N, N, N);
    copy_vec(c.DRs + (size_t)st * N, c.DR, N); }
  if (nt == c.Ltrot) {
    chain_stab_green(c, s, nt, A, lda, c.G);
  }
}

// Wrap_L (src/stabilization.f90:400-437)
__device__ __noinline__ void wrap_L(const ChainDesc &c, const Smem &s, int nt, Pend &pd, bool stats) {
  const int N = c.N, NN = N * N;
  spill_G(c, s);
  int lda; double *A = qr_matrix(c, s, lda);
  const int st = nt / c.Nwrap;
  { PhTimer t(c, PH_STACK);
    blk_copy(c.UR, N, c.URs + (size_t)st * NN, N, N, N);
    blk_copy(c.VR, N, c.VRs + (size_t)st * NN, N, N, N);
    copy_vec(c.DR, c.DRs + (size_t)st * N, N); }
  if (pd.lo <= pd.hi) {
    blk_copy(A, lda, c.ULT, N, N, N);
    { PhTimer t(c, PH_PEND); apply_pending_L(c, s, A, lda, pd.lo, pd.hi); }
    if (nt == c.Ltrot) blk_copy(c.ULT, N, A, lda, N, N);
  } else if (nt != c.Ltrot) {
    blk_copy(A, lda, c.ULT, N, N, N);
  }
  pd.lo = 1; pd.hi = 0;
  if (nt != c.Ltrot) {
    { PhTimer t(c, PH_STABU); chain_stab_U(c, s, A, lda, c.ULT, c.DL, c.VL, true); }
    { PhTimer t(c, PH_STABG); chain_stab_green(c, s, nt, A, lda, c.W3); }
    record_drift(c, take_green(c, s, c.W3), stats);
  }
  { PhTimer t(c, PH_STACK);
    blk_copy(c.ULTs + (size_t)st * NN, N, c.ULT, N, N, N);
    blk_copy(c.VLs + (size_t)st * NN, N, c.VL, N, N, N);
    copy_vec(c.DLs + (size_t)st * N, c.DL, N); }
  if (nt == c.Ltrot) load_G(c, s);   // otherwise take_green reloaded it
}

// Wrap_R (src/stabilization.f90:439-476)
__device__ __noinline__ void wrap_R(const ChainDesc &c, const Smem &s, int nt, Pend &pd, bool stats) {
  const int N = c.N, NN = N * N;
  spill_G(c, s);
  int lda; double *A = qr_matrix(c, s, lda);
  const int st = nt / c.Nwrap;
  { PhTimer t(c, PH_STACK);
    blk_copy(c.ULT, N, c.ULTs + (size_t)st * NN, N, N, N);
    blk_copy(c.VL, N, c.VLs + (size_t)st * NN, N, N, N);
    copy_vec(c.DL, c.DLs + (size_t)st * N, N); }
  if (pd.lo <= pd.hi) {
    blk_copy(A, lda, c.UR, N, N, N);
    { PhTimer t(c, PH_PEND); apply_pending_R(c, s, A, lda, pd.lo, pd.hi, true); }
    if (nt == 0) blk_copy(c.UR, N, A, lda, N, N);
  } else if (nt != 0) {
    blk_copy(A, lda, c.UR, N, N, N);
  }
  pd.lo = 1; pd.hi = 0;
  if (nt != 0) {
    { PhTimer t(c, PH_STABU); chain_stab_U(c, s, A, lda, c.UR, c.DR, c.VR, false); }
    { PhTimer t(c, PH_STABG); chain_stab_green(c, s, nt, A, lda, c.W3); }
    record_drift(c, take_green(c, s, c.W3), stats);
  }
  { PhTimer t(c, PH_STACK);
    blk_copy(c.URs + (size_t)st * NN, N, c.UR, N, N, N);
    blk_copy(c.VRs + (size_t)st * NN, N, c.VR, N, N, N);
    copy_vec(c.DRs + (size_t)st * N, c.DR, N); }
  if (nt == 0) load_G(c, s);   // otherwise take_green reloaded it
}

