// jacobi.hpp -- launchers of the element-block preconditioners: their blocks (jac2d.cuh) and
// their application (jacobi.cu).
#pragma once
#include <cstddef>
#include <cstdint>
#include <cuda_runtime.h>

namespace frsdg
{
// Largest element block the preconditioner inverts (p <= 5 in 2D: 4 (p+1)^2 <= 144);
// the block sits in one CTA's registers, 9 x 9 FP64 entries a thread at p = 5.
constexpr int kMaxBlockDofs = 144;

// What one launch over the elements' Jacobian blocks leaves (jac2d.cuh): the blocks
// themselves (blocks, `slots` = 1 or 5 per element), or the FP32 inverses of the diagonal
// ones and (off not null) the FP32 nonzeros of the neighbours'; blocks with a zero pivot
// are counted in *singular and their inverse is left unwritten.
struct JacOut
{
    double* blocks;
    int     slots;
    float*  inv;
    float*  off;
    unsigned long long* singular;
};
struct Fr2dArgs;
template <class C, int N> cudaError_t launch_jac2d(int gas, int riem, const Fr2dArgs& a, const JacOut& o, cudaStream_t s);
// FP32 values of `off` per element: four neighbours, ND rows, four columns each
inline int64_t offdiag_floats(int nd) { return int64_t(16) * nd; }
// z = M^-1 r on an Nx x Ny element grid with n points per direction: the element blocks'
// inverses alone (off null), or one symmetric red-black block Gauss-Seidel sweep (no
// periodic wrap; jacobi.cu).
cudaError_t launch_pc_apply(const float* inv, const float* off, const double* r, double* z, int n, int Nx, int Ny,
                            cudaStream_t s);
} // namespace frsdg
