// instances.cu -- explicit instantiation of the kernels for one number of GLL points per
// direction, FRSDG_N (set by the build, 2..10), in two parts (FRSDG_PART) that keep the build
// parallel: 0 the FP64 residuals, 1 the complex and FP32 ones, the 1D kernels and the
// Jacobian blocks.
#include "jac2d.cuh"
#include "residual1d.cuh"
#include "residual2d.cuh"

#if !defined(FRSDG_N) || !defined(FRSDG_PART)
#error "FRSDG_N and FRSDG_PART must be defined"
#endif

namespace frsdg
{
#if FRSDG_PART == 0
template cudaError_t launch_fr2d<double, FRSDG_N>(int, int, int, const Fr2dArgs&, cudaStream_t);
template cudaError_t launch_fr2d_batch<double, FRSDG_N>(int, int, int, const Fr2dBatchArgs&, int, cudaStream_t, int*);
#else
template cudaError_t launch_fr2d<cplx, FRSDG_N>(int, int, int, const Fr2dArgs&, cudaStream_t);
template cudaError_t launch_fr2d<float, FRSDG_N>(int, int, int, const Fr2dArgs&, cudaStream_t);
template cudaError_t launch_fr2d<dual, FRSDG_N>(int, int, int, const Fr2dArgs&, cudaStream_t);
template cudaError_t launch_jac2d<cplx, FRSDG_N>(int, int, const Fr2dArgs&, const JacOut&, cudaStream_t);
template cudaError_t launch_jac2d<dual, FRSDG_N>(int, int, const Fr2dArgs&, const JacOut&, cudaStream_t);
template cudaError_t launch_fr1d<double, FRSDG_N>(int, int, const Fr1dArgs&, cudaStream_t);
template cudaError_t launch_fr1d<cplx, FRSDG_N>(int, int, const Fr1dArgs&, cudaStream_t);
template cudaError_t launch_fr2d_batch<float, FRSDG_N>(int, int, int, const Fr2dBatchArgs&, int, cudaStream_t, int*);
#endif
} // namespace frsdg
