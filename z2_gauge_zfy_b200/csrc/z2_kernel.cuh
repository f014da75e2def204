// z2_kernel.cuh -- the chain kernel and the operations it runs.  Included
// inside a namespace by each translation unit that compiles it, after the CUDA
// and C headers: with Z2_NT 256 (z2_api.cu) and 128 (z2_small.cu) threads.
#pragma once
#include "z2_drivers.cuh"

enum { OP_PRE = 1, OP_SWEEP = 2, OP_LOGDET = 3, OP_GLOBAL = 4, OP_THERM = 5, OP_UNIT = 6, OP_STATE = 7 };
enum { U_MMULT_R = 1, U_MMULT_L, U_STAB_UR, U_STAB_UL, U_STAB_GREEN, U_STAB_GREEN_BIG };

struct UnitArgs {
  double *M;                      // mmult: in/out
  double *U, *D, *V;              // stab_U: in/out (U = UR or UL^T)
  const double *UR, *DR, *VR, *ULT, *DL, *VL;
  double *G, *G0t, *Gt0, *Gtt;    // outputs
  int nt, nflag;
};

// Module procedures on a chain's resident state (OP_STATE).
enum {
  SO_PROPK_PRE = 1, SO_PROPT_PRE, SO_PROPK_L, SO_PROPK_R, SO_PROPT_L, SO_PROPT_R,
  SO_PROPGRK_R, SO_PROPGRT_R, SO_WRAP_PRE, SO_WRAP_L, SO_WRAP_R, SO_WRAP_TAU,
  SO_DYN_RESET, SO_SWEEP_RESET, SO_OBS_EQ_CALC, SO_OBS_EQ_AVE, SO_OBS_TAU_CALC,
  SO_OBS_TAU_AVE, SO_SLICE_L, SO_SLICE_R
};

// Arguments of the module procedures.
struct ModArgs {
  UnitArgs u;
  int nt, flag;
  double x;
};

// ---------------------------------------------------------------------------
// Kernels
// ---------------------------------------------------------------------------
__device__ __forceinline__ void load_desc(ChainDesc &sc, const ChainDesc *g) {
  const long long *src = (const long long *)g;
  long long *dst = (long long *)&sc;
  for (int i = threadIdx.x; i < (int)(sizeof(ChainDesc) / 8); i += Z2_NT) dst[i] = src[i];
  __syncthreads();
}

#if Z2_NT == 256
// A module procedure on single matrices, one CTA.
static __device__ __noinline__ void unit_op(const ChainDesc &sc, const Smem &s, int op, const UnitArgs &a) {
  const int N = sc.N;
  if (op == U_MMULT_R || op == U_MMULT_L) {
    kin_init(sc, s);
    if (op == U_MMULT_R) kin_global(sc, s, a.nt, a.M, a.nflag, 0);
    else kin_global(sc, s, a.nt, a.M, 0, a.nflag);
  } else if (op == U_STAB_UR || op == U_STAB_UL) {
    int lda; double *A = qr_matrix(sc, s, lda);
    blk_copy(A, lda, a.U, N, N, N);
    dev_stab_U(s, N, A, lda, a.U, a.D, a.V, sc.W0, op == U_STAB_UL);
  } else if (op == U_STAB_GREEN) {
    int lda; double *A = qr_matrix(sc, s, lda);
    dev_stab_green(s, N, a.nt, sc.Ltrot, a.UR, a.DR, a.VR, a.ULT, a.DL, a.VL, A, lda, sc.W1,
                   sc.W2, sc.W0, a.G);
  } else if (op == U_STAB_GREEN_BIG) {
    int lda; double *A = qr_matrix(sc, s, lda);
    dev_stab_green_big(s, N, a.UR, a.DR, a.VR, a.ULT, a.DL, a.VL, A, lda, sc.W0, sc.W1, sc.W2, sc.W3,
                       a.G, a.G0t, a.Gt0, a.Gtt);
  }
}

// A procedure of the reference's modules on a chain's resident state, one CTA.
static __device__ __noinline__ void state_op(const ChainDesc &c, const Smem &s, int op, int nt, int flag, double x) {
  const int N = c.N;
  Pend pd{1, 0};
  switch (op) {      // the slice table is set up for the procedures that use it
    case SO_PROPK_PRE: case SO_PROPK_L: case SO_PROPK_R: case SO_PROPGRK_R: case SO_SLICE_L: case SO_SLICE_R:
      kin_init(c, s);
      break;
    default:
      break;
  }
  switch (op) {
    case SO_PROPK_PRE:      // propK_pre (src/multiply.f90:8-15) as Local_sweep_pre calls it
      if (c.use_kin) kin_global(c, s, nt, c.UR, 1, 0);
      break;
    case SO_PROPT_PRE:      // propT_pre (src/multiply.f90:65-77)
      blk_scale(c.UR, N, N, N, c.eP);
      break;
    case SO_PROPK_L:        // propK_L (src/multiply.f90:17-28): G B, B^-1 G, UL B
      load_G(c, s);
      kin_slices(c, s, s.G, s.ldg, nt, nt, 1, -1, 1);   // B^-1 G B
      spill_G(c, s);
      kin_global(c, s, nt, c.ULT, 1, 0);      // UL^T <- B UL^T (B symmetric)
      break;
    case SO_PROPK_R:        // propK_R (src/multiply.f90:30-41): B G, G B^-1, B UR
      load_G(c, s);
      kin_slices(c, s, s.G, s.ldg, nt, nt, 1, 1, -1);   // B G B^-1
      spill_G(c, s);
      kin_global(c, s, nt, c.UR, 1, 0);
      break;
    case SO_PROPT_L:        // propT_L (src/multiply.f90:79-93)
      blk_scale(c.G, N, N, N, c.eP);
      blk_scale(c.G, N, N, N, c.eM);
      blk_scale(c.ULT, N, N, N, c.eP);
      break;
    case SO_PROPT_R:        // propT_R (src/multiply.f90:95-108)
      blk_scale(c.G, N, N, N, c.eP);
      blk_scale(c.G, N, N, N, c.eM);
      blk_scale(c.UR, N, N, N, c.eP);
      break;
    case SO_PROPGRK_R:      // propgrK_R (src/multiply.f90:43-63) on the Dyn copy
      if (c.use_kin) {
        propgr_R(c, s, nt, true, false);
        kin_global(c, s, nt, c.URd, 1, 0);
      }
      break;
    case SO_PROPGRT_R:      // propgrT_R (src/multiply.f90:110-130)
      propgr_R(c, s, nt, false, true);
      blk_scale(c.URd, N, N, N, c.eP);
      break;
    case SO_WRAP_PRE:       // Wrap_pre (src/stabilization.f90:374-398)
      wrap_pre(c, s, nt, pd);
      break;
    case SO_WRAP_L:         // Wrap_L (src/stabilization.f90:400-437)
      load_G(c, s);
      wrap_L(c, s, nt, pd, flag != 0);
      spill_G(c, s);
      break;
    case SO_WRAP_R:         // Wrap_R (src/stabilization.f90:439-476)
      load_G(c, s);
      wrap_R(c, s, nt, pd, flag != 0);
      spill_G(c, s);
      break;
    case SO_WRAP_TAU:       // Wrap_tau (src/stabilization.f90:478-514)
      wrap_tau(c, s, nt, pd);
      break;
    case SO_DYN_RESET:      // Dyn_reset (src/dynamics.f90:41-48)
      dyn_reset(c, s);
      break;
    case SO_SWEEP_RESET:    // Local_sweep_reset (src/local_sweep.f90:56-71)
      sweep_reset(c, flag != 0, c.hzero != 0);
      break;
    case SO_OBS_EQ_CALC:    // Obs_equal%calc (src/obser_equal.f90:73-149)
      load_G(c, s);
      obs_equal(c, s, nt);
      break;
    case SO_OBS_EQ_AVE:     // Obs_equal%ave (src/obser_equal.f90:50-71)
      obs_equal_ave(c, x);
      break;
    case SO_OBS_TAU_CALC:   // Obs_tau%calc (src/obser_tau.f90:56-133)
      obs_tau(c, s, nt);
      break;
    case SO_OBS_TAU_AVE:    // Obs_tau%ave (src/obser_tau.f90:37-47)
      obs_tau_ave(c, x);
      break;
    case SO_SLICE_L:        // LocalK_prop_L (src/localK.f90:347-373)
    case SO_SLICE_R:        // LocalK_prop_R (src/localK.f90:375-398)
      load_G(c, s);
      if (op == SO_SLICE_L) {
        propose_slice(c, s, nt, true, 0);            // bonds 2N..1
        kin_slices(c, s, s.G, s.ldg, nt, nt, 1, -1, 1);   // B^-1 G B
        spill_G(c, s);
        kin_global(c, s, nt, c.ULT, 1, 0);
      } else {
        kin_slices(c, s, s.G, s.ldg, nt, nt, 1, 1, -1);   // B G B^-1
        propose_slice(c, s, nt, false, 1);           // bonds 1..2N
        spill_G(c, s);
        kin_global(c, s, nt, c.UR, 1, 0);            // B_nt with the flipped links
      }
      break;
    default:
      break;
  }
}

#endif

// Persistent launch: every CTA pulls chains from a work queue (ordered by
// decreasing cost) and runs the whole operation of that chain.  The module
// procedures run in the same kernel (one CTA, queue null): one copy of the
// device code instead of three.
__global__ void __launch_bounds__(Z2_NT)
z2_chain_kernel(const ChainDesc *descs, const int *order, int nchains, int *queue, int op,
                int nsweep, int toggle, unsigned smem_bytes, const __grid_constant__ ModArgs m) {
  __shared__ ChainDesc sc;
  __shared__ Smem s;     // pointer table in shared memory, not on the local stack
  __shared__ int s_idx;
  for (;;) {
    if (queue != nullptr) {
      if (threadIdx.x == 0) s_idx = atomicAdd(queue, 1);
      __syncthreads();
      const int idx = s_idx;
      if (idx >= nchains) break;
      load_desc(sc, descs + order[idx]);
    } else {
      load_desc(sc, descs);
    }
    if (threadIdx.x == 0) s = make_smem(sc, z2_smem, smem_bytes);
    __syncthreads();
    if (op != OP_THERM && op != OP_UNIT && op != OP_STATE) kin_init(sc, s);
    if (op == OP_PRE) {
      chain_pre(sc, s);
    } else if (op == OP_SWEEP) {
      chain_sweep(sc, s, nsweep, toggle != 0, sc.hzero ? 1.0 : 0.0);
    } else if (op == OP_GLOBAL) {
      chain_global(sc, s, nsweep);
    } else if (op == OP_THERM) {
      chain_therm(sc, s, nsweep);
#if Z2_NT == 256
    } else if (op == OP_LOGDET) {
      chain_logdet_grad(sc, s);
    } else if (op == OP_UNIT) {
      unit_op(sc, s, nsweep, m.u);
    } else if (op == OP_STATE) {
      state_op(sc, s, nsweep, m.nt, m.flag, m.x);
#endif
    }
    if (queue == nullptr) break;
    __syncthreads();
  }
}
