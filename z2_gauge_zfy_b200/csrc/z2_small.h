// z2_small.h -- launches of the chain kernel built with 128 threads per block
// (z2_small.cu).  The descriptors are the same plain structs in both builds.
#pragma once
#include <cuda_runtime.h>

// Allows launches of up to limit bytes of dynamic shared memory; *blocks: resident
// blocks per SM at smem bytes.
cudaError_t z2_small_setup(int limit, unsigned smem, int *blocks);
// One launch; descs is a device array of ChainDesc, op one of OP_PRE, OP_SWEEP,
// OP_GLOBAL, OP_THERM.
cudaError_t z2_small_launch(int grid, unsigned smem, cudaStream_t stream, const void *descs, const int *order,
                            int nchains, int *queue, int op, int nsweep, int toggle);
