// jac2d.cuh -- element blocks of the 2D Jacobian J = sigma dM/dU + dR(M(U))/dU by
// complex step, assembled from the derivatives of the node fluxes and of the face fluxes
// (the preconditioner's part of ComplexStepJacobianStrategy::pre_jv_eval,
// petsc_solver_impl.hpp:72-95 and 223-248, which the reference fills by coloured finite
// differences).
//
// The residual is linear in the node fluxes F, G and in the face fluxes F*; each of them
// depends on the state of one node, or of the two traces of a face point.  A column of the
// Jacobian therefore needs no residual of its own: per node the 4 x 4 derivatives of F and
// G, per face point those of F* with respect to either trace (one seeded variable per
// complex evaluation, the same functions on the same seeded states as a JVP of that
// column), and the entries follow from the differentiation matrix, the metrics and the
// lifts -- in an element block, row node (k, l) and column node (k', l') couple only when
// k = k' or l = l', and a neighbour's block has entries only in the columns of the shared
// face's nodes with l = l' (x-faces) or k = k' (y-faces).
//
// One CTA per element.  Two forms:
//   blocks   every entry of 1 or 5 blocks per element written out (frsdg_jac_blocks,
//            frsdg_jac_blocks5): 256 x 64 elements, p = 3, five blocks (2.7 GB) 13.95 ms
//            with one residual per column and colour, 1.71 ms assembled (one
//            CTA per SM, complex), 0.77 ms with three and first-order scalars;
//   inverse  the diagonal block assembled into registers, inverted there in FP64 and kept
//            in FP32, and the neighbours' entries kept in FP32, nonzeros only
//            (frsdg_pc_setup, frsdg_pc_setup_gs): bound by the elimination's FP64 work and
//            its serial chain of pivots.
#pragma once
#include "device_math.cuh"
#include "frsdg_internal.hpp"
#include "jacobi.hpp"
#include "physics.cuh"

namespace frsdg
{

constexpr int kJacThreads = 256;

template <int N> struct Jac2D
{
    static constexpr int NN = N * N, ND = 4 * NN;
    // shared memory, doubles: flux Jacobians per node [node][var][F eq 0-3, G eq 0-3], dM/dU
    // per node [node][var][eq], face-flux derivatives [side][pos][own / other][var][eq]
    // (side 0 left, 1 right, 2 bottom, 3 top; the own part less that of F.n), D, dL, dR
    static constexpr int oA = 0, oM = oA + NN * 32, oFace = oM + NN * 16, oD = oFace + 4 * N * 32, oL = oD + NN,
                         oR = oL + N, nD = (oR + N + 1) / 2 * 2;  // even: what follows is 16-byte aligned
    static constexpr size_t bytes = sizeof(double) * nD;
    // register tile of the inversion: 16 x 16 threads, R x R entries each (cyclic)
    static constexpr int R = (ND + 15) / 16;
    // inversion: pivot column and row, the FP32 block on its way out, the pivot order
    static constexpr size_t inv_bytes = bytes + sizeof(double) * 2 * ND + sizeof(float) * ND * ND + sizeof(int) * 2 * ND;
};

// The seeded complex state of one node: U + i h e_var (var < 0: no seed), through M for
// the change of variables (NodeLoader<cplx> of the JVP on the same seed).
template <class C> __device__ __forceinline__ void jac_load(const Fr2dArgs& a, int64_t off, int var, C s[4])
{
    const double2 x0 = __ldg(reinterpret_cast<const double2*>(a.U + off));
    const double2 x1 = __ldg(reinterpret_cast<const double2*>(a.U + off + 2));
    s[0] = C(x0.x, var == 0 ? a.h : 0.0);
    s[1] = C(x0.y, var == 1 ? a.h : 0.0);
    s[2] = C(x1.x, var == 2 ? a.h : 0.0);
    s[3] = C(x1.y, var == 3 ? a.h : 0.0);
    if (a.cond_sys)
    {
        const C rho  = s_exp(s[0]);
        const C ssq  = (C(0.0) + s[1] * s[1]) + s[2] * s[2];
        const C rhoE = rho * (s_exp(s[3]) + 0.5 * ssq);
        const C u = s[1], v = s[2];
        s[0] = rho; s[1] = rho * u; s[2] = rho * v; s[3] = rhoE;
    }
}

template <int GAS, class C> __device__ __forceinline__ void jac_record(const GasParams& g, const C s[4], C rec[RF_N])
{
    const NodePrim<C> pr = node_prim<GAS>(g, s[0], s[1], s[2], s[3]);
    rec[RF_RHO] = s[0];
    rec[RF_E] = s[3];
    rec[RF_U] = pr.u;
    rec[RF_V] = pr.v;
    rec[RF_P] = pr.p;
    rec[RF_C] = node_sound_speed<GAS>(g, pr);
}

// The derivatives of element (gi, gj) into shared memory (Jac2D layout).
template <class C, int N, int GAS, int RIEM>
__device__ __forceinline__ void jac_derivatives(const Fr2dArgs& a, int gi, int gj, double* sm)
{
    using J = Jac2D<N>;
    constexpr int NN = J::NN, ND = J::ND;
    const int tid = threadIdx.x;
    const GasParams g = a.gas;
    const bool curved = a.metrics != nullptr;
    const int64_t base = (int64_t(gj) * a.Nx + gi) * ND;
    const int64_t mbase = (int64_t(gj + a.row_base) * a.Nx + gi) * NN;
    for (int q = tid; q < NN; q += kJacThreads) sm[J::oD + q] = a.ops.D[q];
    for (int q = tid; q < N; q += kJacThreads)
    {
        sm[J::oL + q] = a.ops.dL[q];
        sm[J::oR + q] = a.ops.dR[q];
    }
    // node fluxes, one thread per (node, variable)
    for (int q = tid; q < NN * 4; q += kJacThreads)
    {
        const int node = q >> 2, var = q & 3;
        C s[4];
        jac_load(a, base + node * 4, var, s);
        if (var == 0 && !density_ok(s[0].re) && a.bad) atomicAdd(a.bad, 1ull);
        const NodePrim<C> pr = node_prim<GAS>(g, s[0], s[1], s[2], s[3]);
        const C rEp = s[3] + pr.p, ruv = s[1] * pr.v;
        double* A = sm + J::oA + (node * 4 + var) * 8;
        A[0] = s[1].im * a.inv_h;
        A[1] = (s[1] * pr.u + pr.p).im * a.inv_h;
        A[2] = ruv.im * a.inv_h;
        A[3] = (pr.u * rEp).im * a.inv_h;
        A[4] = s[2].im * a.inv_h;
        A[5] = ruv.im * a.inv_h;
        A[6] = (s[2] * pr.v + pr.p).im * a.inv_h;
        A[7] = (pr.v * rEp).im * a.inv_h;
        double* M = sm + J::oM + (node * 4 + var) * 4;
#pragma unroll
        for (int eq = 0; eq < 4; ++eq) M[eq] = s[eq].im * a.inv_h;
    }
    // face fluxes, one thread per (side, position, seeded trace and variable)
#pragma unroll 1
    for (int q = tid; q < 4 * N * 8; q += kJacThreads)
    {
        const int seed = q & 7, pos = (q >> 3) % N, side = (q >> 3) / N;
        const bool xf = side < 2, hi = (side & 1) != 0;
        const int own = xf ? pos * N + (hi ? N - 1 : 0) : (hi ? N - 1 : 0) * N + pos;
        const int oth = xf ? pos * N + (hi ? 0 : N - 1) : (hi ? 0 : N - 1) * N + pos;
        int ni = gi + (xf ? (hi ? 1 : -1) : 0), nj = gj + (xf ? 0 : (hi ? 1 : -1));
        bool wall = false;
        if (ni < 0 || ni >= a.Nx)
        {
            wall = !a.per_x;
            ni = ni < 0 ? a.Nx - 1 : 0;
        }
        if (nj < 0 || nj >= a.Ny)
        {
            wall = !a.per_y;
            nj = nj < 0 ? a.Ny - 1 : 0;
        }
        const bool mine = seed < 4;
        const int var = seed & 3;
        double nx = xf ? 1.0 : 0.0, ny = xf ? 0.0 : 1.0, sc;
        if (curved)
        {
            const int face = (xf ? gi : gj + a.row_base) + (hi ? 1 : 0);
            const double2 nn = xf ? __ldg(reinterpret_cast<const double2*>(a.xnorm) + (int64_t(gj + a.row_base) * (a.Nx + 1) + face) * N + pos)
                                  : __ldg(reinterpret_cast<const double2*>(a.ynorm) + (int64_t(face) * a.Nx + gi) * N + pos);
            nx = nn.x;
            ny = nn.y;
            const double2 m = __ldg(reinterpret_cast<const double2*>(a.metrics + (mbase + own) * 4 + (xf ? 0 : 2)));
            sc = sqrt(m.x * m.x + m.y * m.y);
        }
        else
            sc = xf ? a.scale_x : a.scale_y;
        C s[4], ro[RF_N], rn[RF_N], Fs[4];
        jac_load(a, base + own * 4, mine ? var : -1, s);
        jac_record<GAS>(g, s, ro);
        if (wall)
        {
            const int dir = xf ? (hi ? FRSDG_RIGHT : FRSDG_LEFT) : (hi ? FRSDG_TOP : FRSDG_BOTTOM);
            const int bi = xf ? (gj + a.row_base) * N + pos : gi * N + pos;
            const double2 xy = __ldg(reinterpret_cast<const double2*>(a.bxy[dir]) + bi);
            C gh[4];
            bc_ghost2<GAS>(a.bc[dir], dir, g, a.t, xy.x, xy.y, nx, ny, a.Lx, a.Ly, s, gh, a.exact_bc != 0);
#pragma unroll
            for (int eq = 0; eq < 4; ++eq) s[eq] = gh[eq];
        }
        else
            jac_load(a, (int64_t(nj) * a.Nx + ni) * ND + oth * 4, mine ? -1 : var, s);
        jac_record<GAS>(g, s, rn);
        // the low side of the face is the left argument
        C L[RF_N], Rr[RF_N];
#pragma unroll
        for (int f = 0; f < RF_N; ++f)
        {
            L[f] = hi ? ro[f] : rn[f];
            Rr[f] = hi ? rn[f] : ro[f];
        }
        riemann_rec<RIEM>(L, Rr, nx, ny, Fs);
        C fn[4] = {C(0.0), C(0.0), C(0.0), C(0.0)};
        if (mine)
        {
            // F.n of the own trace
            const C rEp = ro[RF_E] + ro[RF_P];
            const C ru = ro[RF_RHO] * ro[RF_U], rv = ro[RF_RHO] * ro[RF_V], ruv = ru * ro[RF_V];
            fn[0] = ru * nx + rv * ny;
            fn[1] = (ru * ro[RF_U] + ro[RF_P]) * nx + ruv * ny;
            fn[2] = ruv * nx + (rv * ro[RF_V] + ro[RF_P]) * ny;
            fn[3] = (ro[RF_U] * rEp) * nx + (ro[RF_V] * rEp) * ny;
        }
        double* out = sm + J::oFace + ((side * N + pos) * 8 + seed) * 4;
#pragma unroll
        for (int eq = 0; eq < 4; ++eq) out[eq] = wall && !mine ? 0.0 : sc * (Fs[eq].im - fn[eq].im) * a.inv_h;
    }
    __syncthreads();
}

// Entry (row node and eq, column node and variable) of the diagonal block.
template <int N>
__device__ __forceinline__ double jac_self(const Fr2dArgs& a, const double* sm, int64_t mbase, int rn, int eq, int cn,
                                           int var)
{
    using J = Jac2D<N>;
    const int k = rn % N, l = rn / N, kc = cn % N, lc = cn / N;
    double v = 0.0;
    const double* A = sm + J::oA + (cn * 4 + var) * 8 + eq;
    const double* face = sm + J::oFace + var * 4 + eq;
    const double* m = a.metrics ? a.metrics + (mbase + rn) * 4 : nullptr;
    if (l == lc)
    {
        const double d = sm[J::oD + k * N + kc];
        v = m ? __ldg(m) * (d * A[0]) + __ldg(m + 1) * (d * A[4]) : a.xi_x * (d * A[0]);
    }
    if (k == kc)
    {
        const double d = sm[J::oD + l * N + lc];
        v += m ? __ldg(m + 2) * (d * A[0]) + __ldg(m + 3) * (d * A[4]) : a.eta_y * (d * A[4]);
    }
    if (l == lc)
    {
        if (kc == 0) v += face[(0 * N + l) * 32] * sm[J::oL + k];
        if (kc == N - 1) v += face[(1 * N + l) * 32] * sm[J::oR + k];
    }
    if (k == kc)
    {
        if (lc == 0) v += face[(2 * N + k) * 32] * sm[J::oL + l];
        if (lc == N - 1) v += face[(3 * N + k) * 32] * sm[J::oR + l];
    }
    if (rn == cn) v += a.sigma * sm[J::oM + (cn * 4 + var) * 4 + eq];
    return v;
}
// out of line: one copy for the inversion's R x R entries per thread
template <int N>
__device__ __noinline__ double jac_self_entry(const Fr2dArgs& a, const double* sm, int64_t mbase, int i, int j)
{
    return jac_self<N>(a, sm, mbase, i >> 2, i & 3, j >> 2, j & 3);
}

// Side of an element's face towards the neighbour of slot 1 right, 2 top, 3 bottom, 4 left
__device__ __forceinline__ int jac_side(int slot) { return slot == 1 ? 1 : slot == 2 ? 3 : slot == 3 ? 2 : 0; }

// Rows (row node, eq 0-3) of a neighbour's block in the column of variable var at the
// face node the row couples to.
template <int N>
__device__ __forceinline__ void jac_other(const double* sm, int slot, int rn, int var, double v[4])
{
    using J = Jac2D<N>;
    const int k = rn % N, l = rn / N, side = jac_side(slot);
    const bool xf = side < 2;
    const double* f = sm + J::oFace + ((side * N + (xf ? l : k)) * 8 + 4 + var) * 4;
    const double lift = sm[((side & 1) ? J::oR : J::oL) + (xf ? k : l)];
#pragma unroll
    for (int eq = 0; eq < 4; ++eq) v[eq] = f[eq] * lift;
}

// All entries of `slots` blocks per element, blocks[((e * slots + s) * ND + col) * ND + row].
template <class C, int N, int GAS, int RIEM>
__global__ void __launch_bounds__(kJacThreads, 3) jac2d_blocks_kernel(const __grid_constant__ Fr2dArgs a, double* blocks,
                                                                   int slots)
{
    using J = Jac2D<N>;
    constexpr int NN = J::NN, ND = J::ND;
    extern __shared__ __align__(16) double sm[];
    const int gi = int(blockIdx.x) % a.Nx, gj = a.row_begin + int(blockIdx.x) / a.Nx;
    jac_derivatives<C, N, GAS, RIEM>(a, gi, gj, sm);
    const int64_t mbase = (int64_t(gj + a.row_base) * a.Nx + gi) * NN;
    double* out = blocks + (int64_t(gj) * a.Nx + gi) * slots * (int64_t(ND) * ND);
    for (int q = threadIdx.x; q < slots * ND * NN; q += kJacThreads)
    {
        const int rn = q % NN, c = (q / NN) % ND, s = q / (NN * ND), cn = c >> 2, var = c & 3;
        double v[4];
        if (s == 0)
        {
            const bool on = rn % N == cn % N || rn / N == cn / N;
#pragma unroll
            for (int eq = 0; eq < 4; ++eq) v[eq] = on ? jac_self<N>(a, sm, mbase, rn, eq, cn, var) : 0.0;
        }
        else
        {
            const int side = jac_side(s);
            // the neighbour's face node this row couples to
            const int cf = side == 1 ? (rn / N) * N : side == 0 ? (rn / N) * N + N - 1 : side == 3 ? rn % N : (N - 1) * N + rn % N;
            v[0] = v[1] = v[2] = v[3] = 0.0;
            if (cn == cf) jac_other<N>(sm, s, rn, var, v);
        }
        double2* o = reinterpret_cast<double2*>(out + (int64_t(s) * ND + c) * ND + rn * 4);
        o[0] = make_double2(v[0], v[1]);
        o[1] = make_double2(v[2], v[3]);
    }
}

// The inverse of each element's diagonal block in FP32, column-major inv[(e ND + col) ND +
// row], and (off not null) the neighbours' entries in FP32, nonzeros only:
// off[((e * 4 + slot - 1) * 4 + eq) * NN + row node] holds the four columns (variables of
// the face node the row couples to) of row (node, eq).
// The block lives in registers, R x R cyclic entries per thread of a 16 x 16 grid.
// In-place Gauss-Jordan elimination with row pivoting: step k exchanges variable k with
// equation r_k, the unused row with the largest entry of column k, without moving rows; the
// inverse is B[r_k][j] at (k, r_j).  Two barriers per step (the column, from which every
// warp finds the pivot by itself, and the pivot row) instead of six in shared memory.
// 256 x 64 elements, p = 3 (n = 64), the whole Gauss-Seidel set-up: 21.9 -> 2.0 ms against
// the coloured launch with the shared-memory elimination; p = 5 (n = 144) 286 -> 19 ms (3.3 and
// 31 ms with run-time column selects and ten shuffles per pivot).
template <class C, int N, int GAS, int RIEM>
__global__ void __launch_bounds__(kJacThreads, Jac2D<N>::R <= 4 ? 3 : 1) jac2d_inverse_kernel(const __grid_constant__ Fr2dArgs a, float* inv,
                                                                    float4* off, unsigned long long* singular)
{
    using J = Jac2D<N>;
    constexpr int NN = J::NN, ND = J::ND, R = J::R;
    extern __shared__ __align__(16) double sm[];
    double* scol = sm + J::nD;
    double* srow = scol + ND;
    float* sout = reinterpret_cast<float*>(srow + ND);
    int* perm = reinterpret_cast<int*>(sout + ND * ND);  // r_k
    int* pinv = perm + ND;                               // k of row r_k
    const int tid = threadIdx.x, tx = tid & 15, ty = tid >> 4, lane = tid & 31;
    const int gi = int(blockIdx.x) % a.Nx, gj = a.row_begin + int(blockIdx.x) / a.Nx;
    const int64_t e = int64_t(gj + a.row_base) * a.Nx + gi;  // by global row: any window's rows fit the mesh's storage
    const int64_t mbase = e * NN;
    jac_derivatives<C, N, GAS, RIEM>(a, gi, gj, sm);
    if (off)
        for (int q = tid; q < 4 * NN; q += kJacThreads)
        {
            const int rn = q % NN, s = 1 + q / NN;
            double v[4][4];
#pragma unroll
            for (int var = 0; var < 4; ++var) jac_other<N>(sm, s, rn, var, v[var]);
#pragma unroll
            for (int eq = 0; eq < 4; ++eq)
                off[((e * 4 + s - 1) * 4 + eq) * NN + rn] =
                    make_float4(float(v[0][eq]), float(v[1][eq]), float(v[2][eq]), float(v[3][eq]));
        }
    // entry (i, j) of thread (ty, tx): rows i = ty + 16 p, columns j = tx + 16 q; rows and
    // columns past ND are zero and never chosen
    double B[R][R];
#pragma unroll
    for (int p = 0; p < R; ++p)
#pragma unroll
        for (int q = 0; q < R; ++q)
        {
            const int i = ty + 16 * p, j = tx + 16 * q;
            B[p][q] = 0.0;
            if (i < ND && j < ND && ((i >> 2) % N == (j >> 2) % N || (i >> 2) / N == (j >> 2) / N))
                B[p][q] = jac_self_entry<N>(a, sm, mbase, i, j);
        }
    unsigned used = 0;  // bit t: row lane + 32 t is exchanged already
    bool bad = false;
    // steps k = 16 kq + kk: the column's place among the thread's R is known at compile time
    auto steps = [&](auto kq_tag) {
        constexpr int kq = decltype(kq_tag)::value;
        constexpr int kend = ND - kq * 16 < 16 ? ND - kq * 16 : 16;
        if (bad) return;
#pragma unroll 1
        for (int kk = 0; kk < kend; ++kk)
        {
            const int k = kq * 16 + kk;
            if (tx == kk)
            {
                // hand the column out; its entries restart from the exchange's 0
#pragma unroll
                for (int p = 0; p < R; ++p)
                {
                    if (ty + 16 * p < ND) scol[ty + 16 * p] = B[p][kq];
                    B[p][kq] = 0.0;
                }
            }
            __syncthreads();
            // pivot: the unused row with the largest |column entry|, compared by the leading 32
            // bits (the lowest row among equals), two warp reductions in every warp
            unsigned best = 0;
            int br = ND;
#pragma unroll
            for (int t = 0; t < (ND + 31) / 32; ++t)
            {
                const int i = lane + 32 * t;
                if (i < ND && !((used >> t) & 1u))
                {
                    // NaN entries are never chosen; a subnormal one counts as zero
                    const unsigned v = static_cast<unsigned>(__double2hiint(scol[i])) & 0x7fffffffu;
                    if (v > best && v <= 0x7ff00000u) { best = v; br = i; }
                }
            }
            const unsigned top = __reduce_max_sync(0xffffffffu, best);
            br = __reduce_min_sync(0xffffffffu, best == top ? br : ND);
            if (top < 0x00100000u)
            {
                bad = true;  // uniform over the CTA: every warp reads the same column
                break;
            }
            if ((br & 31) == lane) used |= 1u << (br >> 5);
            if (tid == 0)
            {
                perm[k] = br;
                pinv[br] = k;
            }
            double f[R];
#pragma unroll
            for (int p = 0; p < R; ++p) f[p] = ty + 16 * p < ND ? scol[ty + 16 * p] : 0.0;
            if (ty == (br & 15))
            {
                // the pivot row, scaled (selects: branches on p would index B at run time)
                const double rp = s_rcp(scol[br]);
                const int rq = br >> 4;
                double fac[R];
#pragma unroll
                for (int p = 0; p < R; ++p)
                {
                    fac[p] = p == rq ? rp : 1.0;
                    f[p] = p == rq ? 0.0 : f[p];
                    B[p][kq] = tx == kk && p == rq ? 1.0 : B[p][kq];
                }
#pragma unroll
                for (int q = 0; q < R; ++q)
                {
                    double v = 0.0;
#pragma unroll
                    for (int p = 0; p < R; ++p)
                    {
                        B[p][q] *= fac[p];
                        v = p == rq ? B[p][q] : v;
                    }
                    if (tx + 16 * q < ND) srow[tx + 16 * q] = v;
                }
            }
            __syncthreads();
#pragma unroll
            for (int q = 0; q < R; ++q)
            {
                const double rj = tx + 16 * q < ND ? srow[tx + 16 * q] : 0.0;
#pragma unroll
                for (int p = 0; p < R; ++p) B[p][q] = fma(-f[p], rj, B[p][q]);
            }
        }
    };
    static_assert(R <= 9, "register tile");
    steps(std::integral_constant<int, 0>{});
    if constexpr (R > 1) steps(std::integral_constant<int, 1>{});
    if constexpr (R > 2) steps(std::integral_constant<int, 2>{});
    if constexpr (R > 3) steps(std::integral_constant<int, 3>{});
    if constexpr (R > 4) steps(std::integral_constant<int, 4>{});
    if constexpr (R > 5) steps(std::integral_constant<int, 5>{});
    if constexpr (R > 6) steps(std::integral_constant<int, 6>{});
    if constexpr (R > 7) steps(std::integral_constant<int, 7>{});
    if constexpr (R > 8) steps(std::integral_constant<int, 8>{});
    if (bad)
    {
        // zero pivot: the inverse is left unwritten; the caller reports the failure
        if (tid == 0 && singular) atomicAdd(singular, 1ull);
        return;
    }
    __syncthreads();
#pragma unroll
    for (int p = 0; p < R; ++p)
#pragma unroll
        for (int q = 0; q < R; ++q)
        {
            const int i = ty + 16 * p, j = tx + 16 * q;
            if (i < ND && j < ND) sout[perm[j] * ND + pinv[i]] = static_cast<float>(B[p][q]);
        }
    __syncthreads();
    float4* dst = reinterpret_cast<float4*>(inv + e * (int64_t(ND) * ND));
    for (int q = tid; q < ND * ND / 4; q += kJacThreads) dst[q] = reinterpret_cast<const float4*>(sout)[q];
}

template <class C, int N, int GAS, int RIEM> cudaError_t launch_jac2d_kernel(const Fr2dArgs& a, const JacOut& o, cudaStream_t st)
{
    using J = Jac2D<N>;
    const unsigned grid = unsigned(int64_t(a.Nx) * (a.row_end - a.row_begin));
    if (o.blocks)
    {
        cudaError_t e = cudaFuncSetAttribute(jac2d_blocks_kernel<C, N, GAS, RIEM>,
                                             cudaFuncAttributeMaxDynamicSharedMemorySize, int(J::bytes));
        if (e != cudaSuccess) return e;
        jac2d_blocks_kernel<C, N, GAS, RIEM><<<grid, kJacThreads, J::bytes, st>>>(a, o.blocks, o.slots);
        return cudaGetLastError();
    }
    if constexpr (J::ND <= kMaxBlockDofs)
    {
        cudaError_t e = cudaFuncSetAttribute(jac2d_inverse_kernel<C, N, GAS, RIEM>,
                                             cudaFuncAttributeMaxDynamicSharedMemorySize, int(J::inv_bytes));
        if (e != cudaSuccess) return e;
        jac2d_inverse_kernel<C, N, GAS, RIEM>
            <<<grid, kJacThreads, J::inv_bytes, st>>>(a, o.inv, reinterpret_cast<float4*>(o.off), o.singular);
        return cudaGetLastError();
    }
    return cudaErrorInvalidValue;
}

template <class C, int N> cudaError_t launch_jac2d(int gas, int riem, const Fr2dArgs& a, const JacOut& o, cudaStream_t s)
{
    switch (gas * 2 + riem)
    {
        case 0: return launch_jac2d_kernel<C, N, 0, 0>(a, o, s);
        case 1: return launch_jac2d_kernel<C, N, 0, 1>(a, o, s);
        case 2: return launch_jac2d_kernel<C, N, 1, 0>(a, o, s);
        case 3: return launch_jac2d_kernel<C, N, 1, 1>(a, o, s);
        default: return cudaErrorInvalidValue;
    }
}

} // namespace frsdg
