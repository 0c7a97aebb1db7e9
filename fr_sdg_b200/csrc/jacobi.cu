// jacobi.cu -- application of the element-block preconditioners of the implicit path.
//
// The reference preconditions its matrix-free Newton-Krylov solve with a
// finite-difference Jacobian assembled by DMDA colouring (MatFDColoringApply,
// include/petsc_solver_impl.hpp:72-95 and 223-248).  Here the preconditioner is built
// from the element blocks of the same Jacobian (jac2d.cuh): the inverses of the diagonal
// ones in FP32, and for the Gauss-Seidel form the neighbours' entries, nonzeros only.
//   block Jacobi       z_e = inv(J_ee) r_e, one launch;
//   block Gauss-Seidel one symmetric red-black sweep, three launches:
//     red    z_e = inv_e r_e
//     black  z_e = inv_e (r_e - sum_s J_es z_s)
//     red    z_e = z_e - inv_e (sum_s J_es z_s)
// Both are bound by reading the inverses (4 ND^2 bytes per element and pass).
#include "jacobi.hpp"

#include "frsdg_internal.hpp"

namespace frsdg
{

namespace
{

constexpr int kSweepThreads = 256;
enum Sweep : int
{
    SWEEP_ALL = 0,   // every element: z = inv r
    SWEEP_RED = 1,   // red elements: z = inv r
    SWEEP_BLACK = 2, // black elements: z = inv (r - J z)
    SWEEP_BACK = 3   // red elements: z -= inv (J z)
};

// One pass over the elements of a colour (the k-th element of a colour sits in row
// k / ceil(Nx/2)) or over all.  One thread per node: its four rows of the column-major
// FP32 inverse are 16 bytes of each column, so an element's threads read whole columns,
// kUnroll columns in flight.  A neighbour couples to the node's rows through the four
// variables of one of its face nodes (jac2d.cuh), 64 bytes of `off` per neighbour and
// node, where the dense blocks took 4 ND^2 per neighbour: 256 x 64 elements, n = 64, a
// sweep reads 0.5 GB instead of 1.5 GB and takes 97 instead of 299 us.
template <int N, int PHASE>
__global__ void __launch_bounds__(kSweepThreads) block_sweep_kernel(const float* __restrict__ inv,
                                                                    const float4* __restrict__ off, const double* r,
                                                                    double* z, int Nx, int Ny)
{
    constexpr int NN = N * N, ND = 4 * NN, EPC = kSweepThreads / NN;
    constexpr int kUnroll = ND % 8 == 0 ? 8 : ND % 10 == 0 ? 10 : 6;
    static_assert(ND % kUnroll == 0, "whole groups of columns");
    __shared__ __align__(16) double st[EPC][ND];
    const int slot = threadIdx.x / NN, node = threadIdx.x - slot * NN;
    const int64_t k = int64_t(blockIdx.x) * EPC + slot;
    int gi, gj;
    if constexpr (PHASE == SWEEP_ALL)
    {
        gj = int(k / Nx);
        gi = int(k - int64_t(gj) * Nx);
    }
    else
    {
        const int half = (Nx + 1) / 2;
        gj = int(k / half);
        gi = 2 * int(k - int64_t(gj) * half) + ((gj + (PHASE == SWEEP_BLACK ? 1 : 0)) & 1);
    }
    const bool active = slot < EPC && gj < Ny && gi < Nx;
    const int64_t e = int64_t(gj) * Nx + gi;
    const int64_t row = e * ND + node * 4;
    if (active)
    {
        double acc[4] = {0.0, 0.0, 0.0, 0.0};
        if constexpr (PHASE == SWEEP_BLACK || PHASE == SWEEP_BACK)
        {
            const int kk = node % N, l = node / N;
            // right, top, bottom, left neighbour and the face node the row couples to
            const int64_t nb[4] = {gi + 1 < Nx ? e + 1 : -1, gj + 1 < Ny ? e + Nx : -1, gj > 0 ? e - Nx : -1,
                                   gi > 0 ? e - 1 : -1};
            const int fn[4] = {l * N, kk, (N - 1) * N + kk, l * N + N - 1};
#pragma unroll
            for (int s = 0; s < 4; ++s)
            {
                if (nb[s] < 0) continue;
                const double* zn = z + nb[s] * ND + fn[s] * 4;
                const double v[4] = {zn[0], zn[1], zn[2], zn[3]};
#pragma unroll
                for (int eq = 0; eq < 4; ++eq)
                {
                    const float4 b = __ldg(off + ((e * 4 + s) * 4 + eq) * NN + node);
                    acc[eq] = fma(static_cast<double>(b.x), v[0], acc[eq]);
                    acc[eq] = fma(static_cast<double>(b.y), v[1], acc[eq]);
                    acc[eq] = fma(static_cast<double>(b.z), v[2], acc[eq]);
                    acc[eq] = fma(static_cast<double>(b.w), v[3], acc[eq]);
                }
            }
        }
#pragma unroll
        for (int eq = 0; eq < 4; ++eq)
            st[slot][node * 4 + eq] = PHASE == SWEEP_BACK ? acc[eq] : PHASE == SWEEP_BLACK ? r[row + eq] - acc[eq] : r[row + eq];
    }
    __syncthreads();
    if (!active) return;
    const float4* Bi = reinterpret_cast<const float4*>(inv + e * (int64_t(ND) * ND)) + node;
    const double* t = st[slot];
    double o[4] = {0.0, 0.0, 0.0, 0.0};
#pragma unroll 1
    for (int j = 0; j < ND; j += kUnroll)
    {
        float4 b[kUnroll];
#pragma unroll
        for (int q = 0; q < kUnroll; ++q) b[q] = __ldg(Bi + (j + q) * NN);
#pragma unroll
        for (int q = 0; q < kUnroll; ++q)
        {
            const double tj = t[j + q];
            o[0] = fma(static_cast<double>(b[q].x), tj, o[0]);
            o[1] = fma(static_cast<double>(b[q].y), tj, o[1]);
            o[2] = fma(static_cast<double>(b[q].z), tj, o[2]);
            o[3] = fma(static_cast<double>(b[q].w), tj, o[3]);
        }
    }
#pragma unroll
    for (int eq = 0; eq < 4; ++eq) z[row + eq] = PHASE == SWEEP_BACK ? z[row + eq] - o[eq] : o[eq];
}

template <int N, int PHASE>
cudaError_t sweep(const float* inv, const float* off, const double* r, double* z, int Nx, int Ny, cudaStream_t s)
{
    constexpr int EPC = kSweepThreads / (N * N);
    const int64_t slots = int64_t(PHASE == SWEEP_ALL ? Nx : (Nx + 1) / 2) * Ny;  // element slots of the pass
    block_sweep_kernel<N, PHASE><<<unsigned((slots + EPC - 1) / EPC), kSweepThreads, 0, s>>>(
        inv, reinterpret_cast<const float4*>(off), r, z, Nx, Ny);
    return cudaGetLastError();
}

template <int N>
cudaError_t apply_n(const float* inv, const float* off, const double* r, double* z, int Nx, int Ny, cudaStream_t s)
{
    if (!off) return sweep<N, SWEEP_ALL>(inv, off, r, z, Nx, Ny, s);
    cudaError_t e;
    if ((e = sweep<N, SWEEP_RED>(inv, off, r, z, Nx, Ny, s)) != cudaSuccess) return e;
    if ((e = sweep<N, SWEEP_BLACK>(inv, off, r, z, Nx, Ny, s)) != cudaSuccess) return e;
    return sweep<N, SWEEP_BACK>(inv, off, r, z, Nx, Ny, s);
}

} // namespace

cudaError_t launch_pc_apply(const float* inv, const float* off, const double* r, double* z, int n, int Nx, int Ny,
                            cudaStream_t s)
{
    switch (n)
    {
        case 2: return apply_n<2>(inv, off, r, z, Nx, Ny, s);
        case 3: return apply_n<3>(inv, off, r, z, Nx, Ny, s);
        case 4: return apply_n<4>(inv, off, r, z, Nx, Ny, s);
        case 5: return apply_n<5>(inv, off, r, z, Nx, Ny, s);
        case 6: return apply_n<6>(inv, off, r, z, Nx, Ny, s);
        default: return cudaErrorInvalidValue;
    }
}

} // namespace frsdg
