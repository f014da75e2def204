// z2_small.cu -- the chain kernel with 128 threads per block and at most 128
// registers per thread (compiled with -maxrregcount=128): four blocks share an
// SM's register file where the 256-thread build fills it with one.  For
// launches of more chains than SMs on lattices of up to 64 sites, whose chains
// are bound by latency and leave most of an SM idle (the rule is in z2_schedule.h).
#include <cuda_runtime.h>
#include <stdint.h>

#define Z2_NT 128
namespace z2w4 {
#include "z2_kernel.cuh"
}
#include "z2_small.h"

cudaError_t z2_small_setup(int limit, unsigned smem, int *blocks) {
  cudaError_t e = cudaFuncSetAttribute(z2w4::z2_chain_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, limit);
  if (e != cudaSuccess) return e;
  return cudaOccupancyMaxActiveBlocksPerMultiprocessor(blocks, z2w4::z2_chain_kernel, Z2_NT, smem);
}

cudaError_t z2_small_launch(int grid, unsigned smem, cudaStream_t stream, const void *descs, const int *order,
                            int nchains, int *queue, int op, int nsweep, int toggle) {
  z2w4::z2_chain_kernel<<<grid, Z2_NT, smem, stream>>>((const z2w4::ChainDesc *)descs, order, nchains, queue, op,
                                                       nsweep, toggle, smem, z2w4::ModArgs{});
  return cudaGetLastError();
}
