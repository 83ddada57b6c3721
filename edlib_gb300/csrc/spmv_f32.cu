// Operator kernels on FP32 vectors (spmv.cuh).
#include "spmv.cuh"

namespace edgpu {

template void launch_mv<float>(const MvTask<float> *, const int *, int, MvShape, cudaStream_t);
template void launch_mv_vectors<float>(const Sector_mv<float> &, MvShape, cudaStream_t);
template void launch_lz_mv<float>(const LzBatch<float> &, int, bool, MvShape, cudaStream_t);
template void prepare_eig_mv<float>(MvShape);
template void launch_eig_mv<float>(const EigTask<float> *, const int *, int, MvShape, cudaStream_t, float *);
template OpTuning tune_eig_mv<float>(const EigTask<float> *, const int *, int, MvShape, float *, cudaStream_t);
}  // namespace edgpu
