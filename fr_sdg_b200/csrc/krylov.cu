// krylov.cu -- the Arnoldi step of restarted GMRES on the device.
//
// The implicit path solves every Newton system with right-preconditioned GMRES(m)
// (Saad, "Iterative Methods for Sparse Linear Systems", 2nd ed., algorithm 6.9 with
// Givens rotations, section 6.5.3); the reference hands this to PETSc's KSPGMRES
// (petsc_solver_impl.hpp:549-612).  One Arnoldi step here is, with no host round trip:
//   orthogonalisation  h = V_j^T w, w <- w - V_j h by classical Gram-Schmidt, repeated
//                      once when the first pass shrinks ||w|| below 1/sqrt(2) of its
//                      value (the criterion of Daniel, Gragg, Kaufman and Stewart,
//                      Math. Comp. 30, 1976); hn = ||w||;
//   Givens update      the new Hessenberg column takes the previous rotations, a new
//                      rotation zeroes its subdiagonal, and the residual vector g of the
//                      least-squares problem turns with it; 1/hn (0 at breakdown) scales
//                      the next basis vector;
//   back substitution  y = R^-1 g at the end of a cycle (R the rotated Hessenberg).
// One step is six launches and reads the basis three times: the update of the first pass
// takes the second pass's dot products along (1,048,576 unknowns, j = 5, 15, 30: 60, 171, 308 -> 33, 109,
// 209 us against eleven launches and four reads).
// Reductions are two-stage (per-block partial sums in a fixed order, then one block per
// sum), so repeated solves give identical bits.  Every kernel reads its sizes from the
// arguments; scratch is the caller's `work` array (frsdg_gmres_work_doubles).
#include <cstdint>
#include <cuda_runtime.h>

#include "../../include/frsdg.h"

namespace frsdg
{
int report(int code, const char* msg);
int report_cuda(cudaError_t e, const char* what);

constexpr int kKryThreads = 256;
constexpr int kKryPerThread = 8;                            // vector entries per thread
constexpr int kKryChunk = kKryThreads * kKryPerThread;      // entries per block
constexpr int kKryMaxBasis = 256;                           // Arnoldi vectors per cycle

static int64_t kry_blocks(int64_t n) { return (n + kKryChunk - 1) / kKryChunk; }

// work layout (doubles): part[(kKryMaxBasis + 1) * B] | h1[kKryMaxBasis] | h2[kKryMaxBasis] |
// scalars[4] (0: ||w||^2 before, 1: ||w||^2 after the first pass; 2 and 3 spare, as the size of
// `work` is part of the interface)
struct KryWork
{
    double* part;
    double* h1;
    double* h2;
    double* sc;
};

static KryWork kry_work(double* work, int64_t B)
{
    KryWork k;
    k.part = work;
    k.h1 = work + (kKryMaxBasis + 1) * B;
    k.h2 = k.h1 + kKryMaxBasis;
    k.sc = k.h2 + kKryMaxBasis;
    return k;
}

__device__ __forceinline__ double block_sum(double v, double* red)
{
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    __syncthreads();  // red is reused by consecutive calls
    if (lane == 0) red[wid] = v;
    __syncthreads();
    double s = 0.0;
    if (threadIdx.x == 0)
        for (int q = 0; q < kKryThreads / 32; ++q) s += red[q];
    return s;  // valid on thread 0
}

__device__ __forceinline__ double warp_sum(double v)
{
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
    return v;  // valid on lane 0
}

constexpr int kKryWarps = kKryThreads / 32;

// The block's sums red[i * warps + warp], i in [0, nv), to part[i * B + block].
__device__ __forceinline__ void store_partials(const double* red, int nv, double* part)
{
    __syncthreads();
    for (int i = threadIdx.x; i < nv; i += kKryThreads)
    {
        double s = 0.0;
#pragma unroll
        for (int q = 0; q < kKryWarps; ++q) s += red[i * kKryWarps + q];
        part[int64_t(i) * gridDim.x + blockIdx.x] = s;
    }
}

// Per-block partial dot products of w with V[0..nv) and of w with itself, into
// part[i * B + block] (w at i = nv).  Each warp leaves its sums in its own slots, so the
// block meets once.
__global__ void __launch_bounds__(kKryThreads) kry_dot_kernel(const double* V, int64_t ldv, int nv, const double* w,
                                                               int64_t n, double* part)
{
    __shared__ double red[(kKryMaxBasis + 1) * kKryWarps];
    const int64_t base = int64_t(blockIdx.x) * kKryChunk + threadIdx.x;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    double wv[kKryPerThread], s = 0.0;
#pragma unroll
    for (int k = 0; k < kKryPerThread; ++k)
    {
        const int64_t e = base + int64_t(k) * kKryThreads;
        wv[k] = e < n ? w[e] : 0.0;
        s = fma(wv[k], wv[k], s);
    }
    s = warp_sum(s);
    if (lane == 0) red[nv * kKryWarps + warp] = s;
#pragma unroll 2
    for (int i = 0; i < nv; ++i)
    {
        const double* v = V + int64_t(i) * ldv;
        double d = 0.0;
#pragma unroll
        for (int k = 0; k < kKryPerThread; ++k)
        {
            const int64_t e = base + int64_t(k) * kKryThreads;
            if (e < n) d = fma(__ldg(v + e), wv[k], d);
        }
        d = warp_sum(d);
        if (lane == 0) red[i * kKryWarps + warp] = d;
    }
    store_partials(red, nv + 1, part);
}

// w <- w - sum_i h[i] V[i], then the next pass's partial dot products of the new w with V and
// its partial ||w||^2 (row nv of part): the block works through its chunk in pieces of 512
// entries, whose columns of V the dot products find in cache, so the two passes read V from
// memory once.
__global__ void __launch_bounds__(kKryThreads) kry_update_dot_kernel(const double* V, int64_t ldv, int nv, double* w,
                                                                      int64_t n, const double* h, double* part)
{
    __shared__ double red[(kKryMaxBasis + 1) * kKryWarps];
    __shared__ double sh[kKryMaxBasis];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    for (int i = threadIdx.x; i < nv; i += kKryThreads) sh[i] = h[i];
    for (int i = lane; i < nv; i += 32) red[i * kKryWarps + warp] = 0.0;
    __syncthreads();
    double s = 0.0;
#pragma unroll 1
    for (int q = 0; q < kKryPerThread; q += 2)
    {
        const int64_t e0 = int64_t(blockIdx.x) * kKryChunk + q * kKryThreads + threadIdx.x, e1 = e0 + kKryThreads;
        const bool in0 = e0 < n, in1 = e1 < n;
        double a0 = in0 ? w[e0] : 0.0, a1 = in1 ? w[e1] : 0.0;
#pragma unroll 4
        for (int i = 0; i < nv; ++i)
        {
            const double* v = V + int64_t(i) * ldv;
            a0 = fma(-sh[i], in0 ? __ldg(v + e0) : 0.0, a0);
            a1 = fma(-sh[i], in1 ? __ldg(v + e1) : 0.0, a1);
        }
        if (in0) w[e0] = a0;
        if (in1) w[e1] = a1;
        s = fma(a0, a0, fma(a1, a1, s));
#pragma unroll 4
        for (int i = 0; i < nv; ++i)
        {
            const double* v = V + int64_t(i) * ldv;
            double d = in0 ? __ldg(v + e0) * a0 : 0.0;
            if (in1) d = fma(__ldg(v + e1), a1, d);
            d = warp_sum(d);
            if (lane == 0) red[i * kKryWarps + warp] += d;
        }
    }
    s = warp_sum(s);
    if (lane == 0) red[nv * kKryWarps + warp] = s;
    store_partials(red, nv + 1, part);
}

// Whether the second pass acts: ||w||^2 fell below half its value in the first.
__device__ __forceinline__ bool kry_again(const double* sc) { return sc[1] < 0.5 * sc[0]; }

// The second pass: w <- w - sum_i h[i] V[i] and the partial ||w||^2 into row nv of part.
__global__ void __launch_bounds__(kKryThreads) kry_update_kernel(const double* V, int64_t ldv, int nv, double* w,
                                                                  int64_t n, const double* h, double* part,
                                                                  const double* sc)
{
    if (!kry_again(sc)) return;
    __shared__ double red[kKryWarps];
    __shared__ double sh[kKryMaxBasis];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    for (int i = threadIdx.x; i < nv; i += kKryThreads) sh[i] = h[i];
    __syncthreads();
    double s = 0.0;
#pragma unroll 1
    for (int q = 0; q < kKryPerThread; q += 4)
    {
        const int64_t e0 = int64_t(blockIdx.x) * kKryChunk + q * kKryThreads + threadIdx.x;
        double a[4];
#pragma unroll
        for (int k = 0; k < 4; ++k) a[k] = e0 + k * kKryThreads < n ? w[e0 + k * kKryThreads] : 0.0;
#pragma unroll 2
        for (int i = 0; i < nv; ++i)
        {
            const double* v = V + int64_t(i) * ldv + e0;
#pragma unroll
            for (int k = 0; k < 4; ++k)
                if (e0 + k * kKryThreads < n) a[k] = fma(-sh[i], __ldg(v + k * kKryThreads), a[k]);
        }
#pragma unroll
        for (int k = 0; k < 4; ++k)
            if (e0 + k * kKryThreads < n)
            {
                w[e0 + k * kKryThreads] = a[k];
                s = fma(a[k], a[k], s);
            }
    }
    s = warp_sum(s);
    if (lane == 0) red[warp] = s;
    store_partials(red, 1, part + int64_t(nv) * gridDim.x);
}

// One block per sum: the sum of part[i * B ...] over its B entries to out[i] for i < nv and to
// *last for i = nv, in a fixed order.
__global__ void __launch_bounds__(kKryThreads) kry_reduce_kernel(const double* part, int64_t B, int nv, double* out,
                                                                  double* last)
{
    __shared__ double red[kKryThreads / 32];
    const double* p = part + int64_t(blockIdx.x) * B;
    double s = 0.0;
    for (int64_t b = threadIdx.x; b < B; b += kKryThreads) s += p[b];
    s = block_sum(s, red);
    if (threadIdx.x == 0) (int(blockIdx.x) < nv ? out + blockIdx.x : last)[0] = s;
}

// The new Hessenberg column j: H[0..j][j] = h1 + h2 (h2 only after a second pass),
// H[j+1][j] = ||w|| (after a second pass from its B partial sums `norm`); the previous
// rotations, the new one, the residual vector g, and 1/||w|| (0 when w vanished) for the next
// basis vector.  H is row-major with leading dimension ldh.  One block: the sum and the
// column's entries in parallel, the rotations on one thread from shared memory.
__global__ void __launch_bounds__(kKryThreads) kry_givens_kernel(double* H, int ldh, double* cs, double* sn, double* g,
                                                                  const double* h1, const double* h2, const double* sc,
                                                                  const double* norm, int64_t B, int j, double* inv_hn)
{
    __shared__ double red[kKryThreads / 32];
    __shared__ double col[kKryMaxBasis + 1], c_[kKryMaxBasis], s_[kKryMaxBasis];
    const bool second = kry_again(sc);
    for (int i = threadIdx.x; i <= j; i += kKryThreads) col[i] = second ? h1[i] + h2[i] : h1[i];
    for (int i = threadIdx.x; i < j; i += kKryThreads)
    {
        c_[i] = cs[i];
        s_[i] = sn[i];
    }
    double v = 0.0;
    if (second)
        for (int64_t b = threadIdx.x; b < B; b += kKryThreads) v += norm[b];
    v = block_sum(v, red);  // its barriers also order the shared column
    if (threadIdx.x == 0)
    {
        const double nrm2 = second ? v : sc[1];
        const double hn = sqrt(nrm2 > 0.0 ? nrm2 : 0.0);
        double a = col[0];
        for (int i = 0; i < j; ++i)
        {
            const double b = col[i + 1];
            col[i] = c_[i] * a + s_[i] * b;
            a = -s_[i] * a + c_[i] * b;
        }
        const double b = hn;
        const double den = hypot(a, b);
        const double c = den == 0.0 ? 1.0 : a / den, s = den == 0.0 ? 0.0 : b / den;
        cs[j] = c;
        sn[j] = s;
        col[j] = c * a + s * b;
        g[j + 1] = -s * g[j];
        g[j] = c * g[j];
        *inv_hn = hn > 0.0 ? 1.0 / hn : 0.0;
    }
    __syncthreads();
    for (int i = threadIdx.x; i <= j + 1; i += kKryThreads) H[int64_t(i) * ldh + j] = i <= j ? col[i] : 0.0;
}

// y = R^-1 g over the first k columns; a zero diagonal (columns after a breakdown)
// leaves y at zero there.
__global__ void kry_solve_kernel(const double* H, int ldh, const double* g, int k, double* y)
{
    for (int i = k - 1; i >= 0; --i)
    {
        double s = g[i];
        for (int l = i + 1; l < k; ++l) s -= H[int64_t(i) * ldh + l] * y[l];
        const double d = H[int64_t(i) * ldh + i];
        y[i] = d != 0.0 ? s / d : 0.0;
    }
}

} // namespace frsdg

using namespace frsdg;

extern "C" {

int64_t frsdg_gmres_work_doubles(int64_t n)
{
    if (n <= 0) return 0;
    return (kKryMaxBasis + 1) * kry_blocks(n) + 2 * kKryMaxBasis + 4;
}

int frsdg_gmres_arnoldi(const double* V, int64_t ldv, int32_t j, double* w, int64_t n, double* H, int32_t ldh,
                        double* cs, double* sn, double* g, double* inv_hn, double* work, void* stream)
{
    if (!V || !w || !H || !cs || !sn || !g || !inv_hn || !work || n <= 0 || j < 0 || j + 1 > kKryMaxBasis ||
        ldv < n || ldh < j + 1)
        return report(FRSDG_ERR_ARG, "frsdg_gmres_arnoldi: bad argument (at most 256 basis vectors)");
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    const int64_t B = kry_blocks(n);
    const KryWork k = kry_work(work, B);
    const int nv = j + 1;
    const unsigned grid = unsigned(B);
    const double* norm = k.part + int64_t(nv) * B;
    // first pass: h1 = V^T w and ||w||^2 (sc[0]); w -= V h1, its ||w||^2 (sc[1]) and h2 = V^T w
    kry_dot_kernel<<<grid, kKryThreads, 0, s>>>(V, ldv, nv, w, n, k.part);
    kry_reduce_kernel<<<unsigned(nv) + 1, kKryThreads, 0, s>>>(k.part, B, nv, k.h1, k.sc);
    kry_update_dot_kernel<<<grid, kKryThreads, 0, s>>>(V, ldv, nv, w, n, k.h1, k.part);
    kry_reduce_kernel<<<unsigned(nv) + 1, kKryThreads, 0, s>>>(k.part, B, nv, k.h2, k.sc + 1);
    // second pass when the first shrank w (kry_again): w -= V h2 and its ||w||^2
    kry_update_kernel<<<grid, kKryThreads, 0, s>>>(V, ldv, nv, w, n, k.h2, k.part, k.sc);
    kry_givens_kernel<<<1, kKryThreads, 0, s>>>(H, ldh, cs, sn, g, k.h1, k.h2, k.sc, norm, B, j, inv_hn);
    const cudaError_t e = cudaGetLastError();
    return e == cudaSuccess ? FRSDG_OK : report_cuda(e, "frsdg_gmres_arnoldi launch");
}

int frsdg_gmres_solve(const double* H, int32_t ldh, const double* g, int32_t k, double* y, void* stream)
{
    if (!H || !g || !y || k < 0 || ldh < k) return report(FRSDG_ERR_ARG, "frsdg_gmres_solve: bad argument");
    if (k == 0) return FRSDG_OK;
    kry_solve_kernel<<<1, 1, 0, static_cast<cudaStream_t>(stream)>>>(H, ldh, g, k, y);
    const cudaError_t e = cudaGetLastError();
    return e == cudaSuccess ? FRSDG_OK : report_cuda(e, "frsdg_gmres_solve launch");
}

} // extern "C"
