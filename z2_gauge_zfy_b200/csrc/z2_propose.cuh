// z2_propose.cuh -- the 2N proposals of one slice: every outstanding proposal
// evaluated at once, accepted flips queued as rank-2 factors and flushed as
// one rank-2k DMMA update.
#pragma once
#include "z2_blocked.cuh"
#include "z2_flush.cuh"
#include "z2_window.h"

// 48828125^n mod 2^31 (the ranf multiplier power of the n-th draw): the low 32
// bits of the products are enough, 2^31 divides 2^32.
__device__ __forceinline__ unsigned int ranf_pow(int n) {
  unsigned int m = 1u, p = 48828125u;
  for (; n; n >>= 1) {
    if (n & 1) m *= p;
    p *= p;
  }
  return m & 0x7fffffffu;
}

// LocalK_prop_L / LocalK_prop_R's proposals (src/localK.f90:45-173): bonds
// 2N..1 (descending) or 1..2N, one ranf draw each (src/localK.f90:123),
// advanced in closed form.  Thread t owns proposal base + t of a window of
// Z2_NT: it keeps the four entries of G its bond needs, its uniform number
// and the sites of its plaquettes, so a round evaluates every outstanding
// proposal at once.  Everything before the first accepted one is a rejection
// (G and sigma unchanged); the later ones are evaluated again after the
// accept.  A round is
//   evaluate; each warp posts its first candidate; barrier;
//   the first candidate by a warp minimum; its columns u = G(:, P) and rows
//   z = Prod^-1 Delta (I - G)(P, :) of the current G = G0 - X Yt^T join X and
//   Yt; barrier;
//   each thread updates its own bond's four entries, G -= u z.
// After k accepts (or at the end of the slice) G0 -= X Yt^T.  A round without an
// accept ends the window with no second barrier, so the windows post in two
// sets of words in turn (z2_window.h).
//
// Bound: the latency of the round (the ratio, two barriers, the loop over the
// queued columns), not the arithmetic.  Evaluating from X and Yt for 32
// proposals at a time in one warp, as this did before, cost a loop over the
// queued columns per batch and a batch per 32 rejections: 3.8 K cycles per accept
// at L = 8 and, in two measurements, 5.7 and 6.6 K at L = 12; now 1957 (L = 4), 1738
// (8), 2728 (10), 2891 (12), one chain alone on its SM.  Keeping G in the
// register file instead (an update per accept, no queue) lost the gain to
// picking the accepted rows and columns out of the registers.
// GS: G is in shared memory.
template <bool GS>
static __device__ __noinline__ void propose_window(const ChainDesc &c, const Smem &s, int nt,
                                            bool descending, int dir) {
  const int N = c.N, nb = c.nb, k2 = c.k2, Lt = c.Ltrot;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const bool rec = c.dec != nullptr;
  double *G = GS ? as_shared(s.G) : s.G;
  const int ldg = s.ldg, ldx = s.ldx;
  // column pairs of X and Yt as 16-byte words: pair q of row i at q ldx + i
  double2 *X2 = reinterpret_cast<double2 *>(as_shared(s.X));
  double2 *Y2 = reinterpret_cast<double2 *>(as_shared(s.Yt));
  double2 *slot = reinterpret_cast<double2 *>(as_shared(s.red));   // [8][2] K of the posted candidates
  const int *bond = as_shared(s.bond);
  signed char *sg = c.sigma + (size_t)(nt - 1) * nb;
  const signed char *gprev = c.sigma + (size_t)((nt - 2 + Lt) % Lt) * nb;
  const signed char *gnext = c.sigma + (size_t)(nt % Lt) * nb;
  signed char *sig = as_shared(s.sig);
  for (int i = tid; i < nb; i += Z2_NT) sig[i] = sg[i];
  unsigned int st = *c.rng;
  long long rpos = c.replay ? *c.replay_pos : 0;
  const unsigned int ipl = ranf_pow(tid + 1);
  const int nw = (N + 31) & ~31;   // the rows' threads start at a warp of their own
  int np = 0, num = 0;          // queued pairs, accepts
  long long t_eval = 0, t_cols = 0, t_flush = 0;
  __syncthreads();              // sig staged
  for (int base = 0; base < nb; base += Z2_NT) {
    const int cnt = (nb - base) < Z2_NT ? (nb - base) : Z2_NT;
    const bool valid = tid < cnt;
    // ---- this thread's proposal ----
    const int b = valid ? (descending ? nb - 1 - (base + tid) : base + tid) : 0;
    const int i1 = bond[2 * b], i2 = bond[2 * b + 1];
    const int sold = sig[b];
    const double d11 = c.dlt[2 * b], d12 = -(double)sold * c.dlt[2 * b + 1];
    // temporal part of the boson ratio: the neighbours in tau do not change
    const int it = 1 - ((sold * ((int)gprev[b] + (int)gnext[b])) >> 1);
    const double rb0 = c.rb[it], rb1 = c.rb[3 + it], rb2 = c.rb[6 + it];
    const int *bb = c.bbonds + 6 * b;
    const int b0 = bb[0], b1 = bb[1], b2 = bb[2], b3 = bb[3], b4 = bb[4], b5 = bb[5];
    double rnd = (double)((st * ipl) & 0x7fffffffu) * (1.0 / 2147483648.0);
    if (c.replay && rpos + tid < c.nreplay) rnd = c.replay[rpos + tid];
    double g11 = G[i1 + (size_t)i1 * ldg], g12 = G[i1 + (size_t)i2 * ldg];
    double g21 = G[i2 + (size_t)i1 * ldg], g22 = G[i2 + (size_t)i2 * ldg];
    for (int q = 0; q < np; ++q) {
      const double2 xa = X2[q * ldx + i1], xb = X2[q * ldx + i2];
      const double2 ya = Y2[q * ldx + i1], yb = Y2[q * ldx + i2];
      g11 = fma(-xa.y, ya.y, fma(-xa.x, ya.x, g11));
      g12 = fma(-xa.y, yb.y, fma(-xa.x, yb.x, g12));
      g21 = fma(-xb.y, ya.y, fma(-xb.x, ya.x, g21));
      g22 = fma(-xb.y, yb.y, fma(-xb.x, yb.x, g22));
    }
    int done = 0;
    // the warps' candidates, proposal << 20 | p1 << 10 | p2
    int *flag = as_shared(s.flag) + z2_window_post<Z2_NT>(base);
    for (;;) {
      const long long t0 = ph_now();
      // ---- evaluate ----
      double ratio = 0.0;
      if (warp * 32 < cnt) {                        // warp-uniform
        // (I - G)_PP, Prod = I + Delta (I - G)_PP, determinant (no FMA
        // contraction: same rounding sequence as the reference)
        const double l11 = __dsub_rn(1.0, g11), l12 = -g12, l21 = -g21, l22 = __dsub_rn(1.0, g22);
        const double m11 = __dadd_rn(__dmul_rn(d11, l11), __dmul_rn(d12, l21));
        const double p12 = __dadd_rn(__dmul_rn(d11, l12), __dmul_rn(d12, l22));
        const double p21 = __dadd_rn(__dmul_rn(d12, l11), __dmul_rn(d11, l21));
        const double m22 = __dadd_rn(__dmul_rn(d12, l12), __dmul_rn(d11, l22));
        const double p11 = __dadd_rn(1.0, m11), p22 = __dadd_rn(1.0, m22);
        const double det = __dsub_rn(__dmul_rn(p11, p22), __dmul_rn(p12, p21));
        const double idet = rcp_newton(det);        // beside the ratio and the ballot
        // boson ratio (src/fields.f90:40-119) from the host table: the signs
        // of the two plaquette products pick the entry
        const int x = (int)sig[b0] ^ (int)sig[b1] ^ (int)sig[b2] ^ sold;
        const int y = (int)sig[b3] ^ (int)sig[b4] ^ (int)sig[b5] ^ sold;
        const double rb = (x ^ y) < 0 ? rb1 : (x < 0 ? rb2 : rb0);
        ratio = __dmul_rn(__dmul_rn(det, det), rb);
        const bool acc = valid && tid >= done && fabs(ratio) > rnd;
        const unsigned ball = __ballot_sync(Z2_FULL, acc);
        if (ball == 0) {
          if (lane == 0) flag[warp] = 0x7fffffff;
        } else if (lane == __ffs(ball) - 1) {
          flag[warp] = (tid << 20) | (i1 << 10) | i2;
          // K = Prod^-1 Delta
          const double q00 = p22 * idet, q01 = -p12 * idet, q10 = -p21 * idet, q11 = p11 * idet;
          double2 *sl = slot + 2 * warp;
          sl[0] = make_double2(fma(q00, d11, q01 * d12), fma(q00, d12, q01 * d11));
          sl[1] = make_double2(fma(q10, d11, q11 * d12), fma(q10, d12, q11 * d11));
        }
      } else if (lane == 0) {
        flag[warp] = 0x7fffffff;
      }
      __syncthreads();
      const long long t1 = ph_now();
      t_eval += t1 - t0;
      // ---- first accepted proposal (a warp minimum: a uniform result) ----
      const unsigned first =
          __reduce_min_sync(Z2_FULL, lane < Z2_WARPS ? (unsigned)flag[lane] : 0x7fffffffu);
      const int kf = (int)(first >> 20);            // 0x7ff: none
      if (rec && valid && tid >= done && tid <= kf) {
        const size_t li = ((size_t)dir * Lt + (nt - 1)) * nb + b;
        c.dec[li] = (tid == kf) ? 1 : 0;
        if (c.ratios) c.ratios[li] = ratio;
      }
      if (first == 0x7fffffffu) break;
      done = kf + 1;
      ++num;
      const int p1 = (int)((first >> 10) & 0x3ffu), p2 = (int)(first & 0x3ffu);
      // ---- columns p1, p2 and rows p1, p2 of the current G ----
      double2 *Xn = X2 + np * ldx, *Yn = Y2 + np * ldx;
      // the queued pairs are loaded one ahead of their use
      const auto u_side = [&](int i) {
        double u0 = G[i + (size_t)p1 * ldg], u1 = G[i + (size_t)p2 * ldg];
        double w0 = 0.0, w1 = 0.0;                  // second chain per output
        const double2 *xi = X2 + i, *ya = Y2 + p1, *yb = Y2 + p2;
        if (np > 0) {
          double2 xr = *xi, y1 = *ya, y2 = *yb;
#pragma unroll 2
          for (int q = 1; q < np; ++q) {
            xi += ldx; ya += ldx; yb += ldx;
            const double2 xn = *xi, y1n = *ya, y2n = *yb;
            u0 = fma(-xr.x, y1.x, u0); u1 = fma(-xr.x, y2.x, u1);
            w0 = fma(xr.y, y1.y, w0); w1 = fma(xr.y, y2.y, w1);
            xr = xn; y1 = y1n; y2 = y2n;
          }
          u0 = fma(-xr.x, y1.x, u0); u1 = fma(-xr.x, y2.x, u1);
          w0 = fma(xr.y, y1.y, w0); w1 = fma(xr.y, y2.y, w1);
        }
        Xn[i] = make_double2(u0 - w0, u1 - w1);
      };
      const auto v_side = [&](int j) {
        double v0 = ((j == p1) ? 1.0 : 0.0) - G[p1 + (size_t)j * ldg];
        double v1 = ((j == p2) ? 1.0 : 0.0) - G[p2 + (size_t)j * ldg];
        const double2 ka = slot[2 * (kf >> 5)], kb = slot[2 * (kf >> 5) + 1];
        double w0 = 0.0, w1 = 0.0;
        const double2 *yj = Y2 + j, *xa = X2 + p1, *xb = X2 + p2;
        if (np > 0) {
          double2 yr = *yj, x1 = *xa, x2 = *xb;
#pragma unroll 2
          for (int q = 1; q < np; ++q) {
            yj += ldx; xa += ldx; xb += ldx;
            const double2 yn = *yj, x1n = *xa, x2n = *xb;
            v0 = fma(x1.x, yr.x, v0); v1 = fma(x2.x, yr.x, v1);
            w0 = fma(x1.y, yr.y, w0); w1 = fma(x2.y, yr.y, w1);
            yr = yn; x1 = x1n; x2 = x2n;
          }
          v0 = fma(x1.x, yr.x, v0); v1 = fma(x2.x, yr.x, v1);
          w0 = fma(x1.y, yr.y, w0); w1 = fma(x2.y, yr.y, w1);
        }
        v0 += w0; v1 += w1;
        Yn[j] = make_double2(fma(ka.x, v0, ka.y * v1), fma(kb.x, v0, kb.y * v1));
      };
      if (nw + N <= Z2_NT) {                        // a thread per output pair
        if (tid < N) u_side(tid);
        else if (tid >= nw && tid < nw + N) v_side(tid - nw);
      } else {
        for (int i = tid; i < N; i += Z2_NT) { u_side(i); v_side(i); }
      }
      if (tid == kf) {
        sig[b] = (signed char)(-sold);
        sg[b] = (signed char)(-sold);
      }
      __syncthreads();
      ++np;
      // ---- this thread's bond ----
      if (warp * 32 < cnt) {
        const double2 xa = Xn[i1], xb = Xn[i2], ya = Yn[i1], yb = Yn[i2];
        g11 = fma(-xa.y, ya.y, fma(-xa.x, ya.x, g11));
        g12 = fma(-xa.y, yb.y, fma(-xa.x, yb.x, g12));
        g21 = fma(-xb.y, ya.y, fma(-xb.x, ya.x, g21));
        g22 = fma(-xb.y, yb.y, fma(-xb.x, yb.x, g22));
      }
      const long long t2 = ph_now();
      t_cols += t2 - t1;
      if (2 * np >= k2) {
        rank_update<GS>(s.G, ldg, s.X, s.Yt, N, ldx, 2 * np, c.flush_shape);
        np = 0;
        t_flush += ph_now() - t2;
      }
    }
    st = (st * ranf_pow(cnt)) & 0x7fffffffu;
    rpos += cnt;
  }
  if (np > 0) {
    const long long tf = ph_now();
    rank_update<GS>(s.G, ldg, s.X, s.Yt, N, ldx, 2 * np, c.flush_shape);
    t_flush += ph_now() - tf;
  }
  if (tid == 0) {
    *c.rng = st;
    if (c.replay) *c.replay_pos = rpos;
    acc_add(c, A_ACC_DEN, (double)nb);
    acc_add(c, A_DRAWS, (double)nb);
    acc_add(c, A_ACC_NUM, (double)num);
    acc_add(c, A_PH0 + PH_EVAL, (double)t_eval);
    acc_add(c, A_PH0 + PH_COLS, (double)t_cols);
    acc_add(c, A_PH0 + PH_FLUSH, (double)t_flush);
  }
  __syncthreads();
}

__device__ __forceinline__ void propose_slice(const ChainDesc &c, const Smem &s, int nt,
                                              bool descending, int dir) {
  if (c.g_in_smem) propose_window<true>(c, s, nt, descending, dir);
  else propose_window<false>(c, s, nt, descending, dir);
}
