// Operator kernels on float-float vectors (spmv.cuh).
#include "spmv.cuh"

namespace edgpu {

template void launch_lz_mv<ffloat>(const LzBatch<ffloat> &, int, bool, MvShape, cudaStream_t);
}  // namespace edgpu
