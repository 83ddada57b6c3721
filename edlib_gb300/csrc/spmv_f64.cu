// Operator kernels on FP64 vectors (spmv.cuh).
#include "spmv.cuh"

namespace edgpu {

template void launch_mv<double>(const MvTask<double> *, const int *, int, MvShape, cudaStream_t);
template void launch_mv_vectors<double>(const Sector_mv<double> &, MvShape, cudaStream_t);
template void launch_lz_mv<double>(const LzBatch<double> &, int, bool, MvShape, cudaStream_t);
template void prepare_eig_mv<double>(MvShape);
template void launch_eig_mv<double>(const EigTask<double> *, const int *, int, MvShape, cudaStream_t, double *);
template OpTuning tune_eig_mv<double>(const EigTask<double> *, const int *, int, MvShape, double *, cudaStream_t);
}  // namespace edgpu
