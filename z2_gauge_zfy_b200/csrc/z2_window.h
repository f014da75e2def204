// z2_window.h -- where the warps of a chain's block post their candidates
// (propose_window, z2_propose.cuh).  No CUDA types: the host test of the
// hand-over compiles it as it is.
#pragma once
#ifdef __CUDACC__
#define Z2_HD __host__ __device__ __forceinline__
#else
#define Z2_HD inline
#endif

// First word of the posts of the window of NT proposals that begins at proposal
// `base`: one word per warp, in two sets that the windows of a slice use in turn.
// A warp leaves a window after the one barrier of its last round and posts for
// the next one while a slower warp may still read that round's posts; with one
// set it would overwrite them.  Two sets are enough: before a set is used again
// every warp has passed the barrier of the window between, and so has read it.
template <int NT>
Z2_HD int z2_window_post(int base) {
  return (base / NT & 1) * (NT / 32);
}
