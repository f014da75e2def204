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
#include "z2_kin.cuh"
#include "z2_propose.cuh"
#include "z2_stab.cuh"

// ---------------------------------------------------------------------------
// Shared-memory layout
// ---------------------------------------------------------------------------
__device__ __forceinline__ size_t align16(size_t x) { return (x + 15) & ~size_t(15); }

static __device__ Smem make_smem(const ChainDesc &c, unsigned char *base, size_t smem_bytes) {
  Smem s;
  const int N = c.N;
  size_t off = 0;
  s.red = (double *)(base + off); off += sizeof(double) * Z2_NRED;
  s.vec = (double *)(base + off); off += sizeof(double) * 8 * N;
  s.cs = (double2 *)(base + off); off += sizeof(double2) * 2 * N;
  s.ivec = (int *)(base + off); off += align16(sizeof(int) * 2 * N);
  s.tp = (int *)(base + off); off += align16(sizeof(int) * 4 * N);
  s.bond = (int *)(base + off); off += align16(sizeof(int) * 4 * N);
  s.gid = (short *)(base + off); off += align16(sizeof(short) * 2 * N);
  s.flag = (int *)(base + off); off += sizeof(int) * 16;
  s.sig = (signed char *)(base + off); off += align16(2 * N);
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

// Lazily propagated U factors.  R chain: for nt' = lo..hi, U <- B_nt' U then
// U *= e^{dtau mu} (LocalK_prop_R + propT_R, src/localK.f90:395-396,
// src/multiply.f90:106).  L chain (ULT = UL^T, B symmetric): for nt' = hi
// down to lo, ULT *= e^{dtau mu} then ULT <- B_nt' ULT (propT_L + prop_L,
// src/multiply.f90:91, src/localK.f90:370).
static __device__ __noinline__ void pending_mu(const ChainDesc &c, double *A, int lda, int n) {
  if (c.eP == 1.0) return;
  double x = 1.0;
  for (int i = 0; i < n; ++i) x *= c.eP;       // one pass for the n slices' factors
  blk_scale(A, lda, c.N, c.N, x);
}
__device__ __forceinline__ void apply_pending_R(const ChainDesc &c, const Smem &s, double *A, int lda, int lo,
                                int hi, bool kin) {
  if (lo > hi) return;
  if (kin) kin_slices(c, s, A, lda, lo, hi, 1, 1, 0);
  pending_mu(c, A, lda, hi - lo + 1);
}
__device__ __forceinline__ void apply_pending_L(const ChainDesc &c, const Smem &s, double *A, int lda, int lo,
                                int hi) {
  if (lo > hi) return;
  pending_mu(c, A, lda, hi - lo + 1);
  kin_slices(c, s, A, lda, hi, lo, -1, 1, 0);
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
static __device__ __noinline__ void dev_stab_green_big(const Smem &s, int N, const double *UR, const double *DR,
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
//
// With n_i = 1 - G_ii, t_ij = G_ij G_ji and the phases st_i st_j and
// cos(qx dx + pi dy) = pc_i pc_j + ps_i ps_j (products of site factors), the
// double sums split into squares of single sums and sums over unordered pairs:
//   sum_ij ph_ij (4 n_i n_j - 2 (d_ij - G_ji) G_ij)
//     = 4 (sum_i st_i n_i)^2 + 4 sum_{i<j} ph_ij t_ij - 2 sum_i (1 - G_ii) G_ii.
// Pairs are taken along the diagonals (i, i + d mod N), d = 1..N/2 (d = N/2
// meets each pair twice): lanes over i read G_ij and G_ji at the odd stride
// ldg + 1, free of bank conflicts, and each warp has its share of the d.  (One
// pass over all (i, j) with a gather of the phase took 20 K cycles per slice at
// N = 144.)
template <bool GS>
static __device__ __noinline__ void obs_equal_on(const ChainDesc &c, const Smem &s, int nt) {
  const int N = c.N, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const double *G = GS ? as_shared(s.G) : s.G;
  const int ldg = s.ldg;
  const signed char *sg = c.sigma + (size_t)(nt - 1) * c.nb;
  double *st = as_shared(s.vec), *pc = st + N, *ps = pc + N;
  // flux, density, pairs, sums of st n, pc n, ps n, and the two pair sums
  double v[8] = {0, 0, 0, 0, 0, 0, 0, 0};
  for (int i = tid; i < N; i += Z2_NT) {
    const int4 pl = reinterpret_cast<const int4 *>(c.plaq)[i];
    const double a = c.stag[i], x = c.phase[2 * i], y = c.phase[2 * i + 1];
    v[0] += (double)((int)sg[pl.x] * (int)sg[pl.y] * (int)sg[pl.z] * (int)sg[pl.w]);
    const double g = G[i + (size_t)i * ldg], n = 1.0 - g;
    st[i] = a;
    pc[i] = x;
    ps[i] = y;
    v[1] += n + n;
    v[2] += n * n;
    v[3] += a * n;
    v[4] += x * n;
    v[5] += y * n;
    v[6] -= 2.0 * n * g;
    v[7] -= 2.0 * n * g;
  }
  __syncthreads();
  const int H = N >> 1, per = (H + Z2_WARPS - 1) / Z2_WARPS;
  const int d0 = 1 + warp * per, d1 = min(H, d0 + per - 1);
  for (int i = lane; i < N; i += 32) {
    double s1 = 0.0, s2 = 0.0, s3 = 0.0, s4 = 0.0;
    int j = i + d0;
    if (j >= N) j -= N;
#pragma unroll 4
    for (int d = d0; d <= d1; ++d) {
      const double w = d == H ? 0.5 : 1.0;
      const double a = G[i + (size_t)j * ldg], b = G[j + (size_t)i * ldg];
      const double t = w * a * b;
      s1 = fma(w * a, a, fma(w * b, b, s1));
      s2 = fma(st[j], t, s2);
      s3 = fma(pc[j], t, s3);
      s4 = fma(ps[j], t, s4);
      if (++j == N) j = 0;
    }
    v[2] += s1;
    v[6] = fma(4.0 * st[i], s2, v[6]);
    v[7] = fma(4.0 * pc[i], s3, fma(4.0 * ps[i], s4, v[7]));
  }
  blk_sum_n<8>(v, s.red);
  if (tid == 0) {
    const double flux = v[0] / (double)N;
    acc_add(c, A_FLUX_SUM, flux);
    acc_add(c, A_FLUX_SQ, flux * flux);
    acc_add(c, A_PAIR, v[2]);
    acc_add(c, A_CDW, fma(4.0 * v[3], v[3], v[6]));
    acc_add(c, A_CDWS, fma(4.0 * v[4], v[4], fma(4.0 * v[5], v[5], v[7])));
    acc_add(c, A_DENS, v[1] / (double)N);
    acc_add(c, A_NOBS, 1.0);
  }
  __syncthreads();
}
__device__ __forceinline__ void obs_equal(const ChainDesc &c, const Smem &s, int nt) {
  if (c.g_in_smem) obs_equal_on<true>(c, s, nt);
  else obs_equal_on<false>(c, s, nt);
}

// ---------------------------------------------------------------------------
// Time-displaced observables (Obs_tau_calc, src/obser_tau.f90:56-133), real
// parts, both identical spin sectors summed; binned by imj deterministically
// (one thread per displacement).
// ---------------------------------------------------------------------------
static __device__ __noinline__ void obs_tau(const ChainDesc &c, const Smem &s, int nt) {
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

static __device__ __noinline__ void spill_G(const ChainDesc &c, const Smem &s) {
  if (c.g_in_smem) blk_copy(c.G, c.N, s.G, s.ldg, c.N, c.N);
}
static __device__ __noinline__ void load_G(const ChainDesc &c, const Smem &s) {
  if (c.g_in_smem) blk_copy(s.G, s.ldg, c.G, c.N, c.N, c.N);
}

// The stabilized Green's function Gn replaces the propagated one in one pass
// over both: returns the drift max |Gn - G| (compare_mat,
// src/stabilization.f90:365-372) and leaves G = Gn in global memory and, for
// a chain whose G lives in shared memory, there too.
static __device__ __noinline__ double take_green(const ChainDesc &c, const Smem &s, const double *Gn) {
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

static __device__ __noinline__ void copy_vec(double *dst, const double *src, int n) {
  for (int i = threadIdx.x; i < n; i += Z2_NT) dst[i] = src[i];
  __syncthreads();
}

static __device__ __noinline__ void record_drift(const ChainDesc &c, double dif, bool stats) {
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
static __device__ __noinline__ void wrap_pre(const ChainDesc &c, const Smem &s, int nt, Pend &pd) {
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
static __device__ __noinline__ void wrap_L(const ChainDesc &c, const Smem &s, int nt, Pend &pd, bool stats) {
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
static __device__ __noinline__ void wrap_R(const ChainDesc &c, const Smem &s, int nt, Pend &pd, bool stats) {
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

