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

// z_e = inv_e r_e for every element.  Four threads per node: thread (part, node) takes the
// columns j = part mod 4 of the node's four rows (16 bytes of each column, an element's
// threads whole columns), and the four sums meet in shared memory.  One thread per node read
// the large meshes as fast, but on meshes that live in L2 its chain of ND columns set the
// time: 16 x 16 elements, p = 3, 4, 5 10.4, 14.0, 18.6 -> 4.3, 4.9, 6.4 us; 64 x 64 elements
// (67 to 340 MB of inverses from memory) 31.7, 51.3, 79.8 -> 22.4, 40.9, 71.7 us.
template <int N> struct Apply
{
    static constexpr int NN = N * N, ND = 4 * NN, TPE = 4 * NN;          // threads per element
    static constexpr int EPC = TPE <= 64 ? 128 / TPE : 1;                 // elements per CTA
    static constexpr int THREADS = (EPC * TPE + 31) / 32 * 32;
};
template <int N>
__global__ void __launch_bounds__(Apply<N>::THREADS) block_apply_kernel(const float* __restrict__ inv, const double* __restrict__ r,
                                                                        double* __restrict__ z, int64_t nelem)
{
    using P = Apply<N>;
    constexpr int NN = P::NN, ND = P::ND;
    __shared__ __align__(16) double st[P::EPC][ND];
    __shared__ __align__(16) double sp[P::EPC][3][ND];
    const int slot = threadIdx.x / P::TPE, t = threadIdx.x - slot * P::TPE, part = t / NN, node = t - part * NN;
    const int64_t e = int64_t(blockIdx.x) * P::EPC + slot;
    const bool active = slot < P::EPC && e < nelem;
    if (active) st[slot][t] = r[e * ND + t];
    const float4* B = reinterpret_cast<const float4*>(inv + e * (int64_t(ND) * ND)) + node + part * NN;
    __syncthreads();
    double o[4] = {0.0, 0.0, 0.0, 0.0};
    if (active)
    {
        constexpr int U = NN % 9 == 0 ? 9 : NN % 5 == 0 ? 5 : NN < 8 ? NN : 8;  // columns in flight
        static_assert(NN % U == 0, "whole groups of columns");
#pragma unroll
        for (int j = 0; j < NN; j += U)
        {
            float4 b[U];
#pragma unroll
            for (int q = 0; q < U; ++q) b[q] = __ldg(B + (j + q) * 4 * NN);
#pragma unroll
            for (int q = 0; q < U; ++q)
            {
                const double v = st[slot][(j + q) * 4 + part];
                o[0] = fma(static_cast<double>(b[q].x), v, o[0]);
                o[1] = fma(static_cast<double>(b[q].y), v, o[1]);
                o[2] = fma(static_cast<double>(b[q].z), v, o[2]);
                o[3] = fma(static_cast<double>(b[q].w), v, o[3]);
            }
        }
        if (part > 0)
        {
            double2* s = reinterpret_cast<double2*>(&sp[slot][part - 1][node * 4]);
            s[0] = make_double2(o[0], o[1]);
            s[1] = make_double2(o[2], o[3]);
        }
    }
    __syncthreads();
    if (!active || part > 0) return;
#pragma unroll
    for (int q = 0; q < 4; ++q)
        z[e * ND + node * 4 + q] = (o[q] + sp[slot][0][node * 4 + q]) + (sp[slot][1][node * 4 + q] + sp[slot][2][node * 4 + q]);
}

constexpr int kSweepThreads = 256;
enum Sweep : int
{
    SWEEP_RED = 1,   // red elements: z = inv r
    SWEEP_BLACK = 2, // black elements: z = inv (r - J z)
    SWEEP_BACK = 3   // red elements: z -= inv (J z)
};

// One pass over the elements of a colour (the k-th element of a colour sits in row
// k / ceil(Nx/2)).  One thread per node: its four rows of the column-major
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
    const int half = (Nx + 1) / 2;
    const int gj = int(k / half);
    const int gi = 2 * int(k - int64_t(gj) * half) + ((gj + (PHASE == SWEEP_BLACK ? 1 : 0)) & 1);
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
    const int64_t slots = int64_t((Nx + 1) / 2) * Ny;  // element slots of the pass
    block_sweep_kernel<N, PHASE><<<unsigned((slots + EPC - 1) / EPC), kSweepThreads, 0, s>>>(
        inv, reinterpret_cast<const float4*>(off), r, z, Nx, Ny);
    return cudaGetLastError();
}

template <int N>
cudaError_t apply_n(const float* inv, const float* off, const double* r, double* z, int Nx, int Ny, cudaStream_t s)
{
    if (!off)
    {
        using P = Apply<N>;
        const int64_t nelem = int64_t(Nx) * Ny;
        block_apply_kernel<N><<<unsigned((nelem + P::EPC - 1) / P::EPC), P::THREADS, 0, s>>>(inv, r, z, nelem);
        return cudaGetLastError();
    }
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
