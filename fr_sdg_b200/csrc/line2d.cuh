// line2d.cuh -- the real FR residual of the 2D Euler equations with one thread per line of
// nodes (PhysicsEvaluator<Traits,2>::residual_kernel and compute_volume_term,
// include/physics_impl_2D.hpp:268-357 and 646-902).
//
// One CTA owns TX x TY elements and N threads per element, which work on the element's
// columns and rows in turn:
//   column pass  thread (e, k): loads the N nodes of its column (32-byte nodes, N of them
//                contiguous across the element's threads), primitives and both fluxes; F
//                goes to shared memory, G stays in registers, where its eta-derivative is
//                taken; boundary nodes and the tile's halo traces leave face records;
//   face pass    one thread per face point: Riemann flux and the jumps scale (F* - F.n) of
//                both sides, F.n from the records;
//   row pass     thread (e, l): the xi-derivatives of its row of F and the lifts of the
//                left and right faces, back in place;
//   output pass  thread (e, k): the row part, its own eta part, the lifts of the bottom and
//                top faces, the requested output form.
// Each sum is taken by one thread from one inlined copy of the code, whichever tile an
// element falls into, so results do not depend on where a row window cuts the mesh.
//
// Why a thread per line: one per node (or per face point) spent 790 warp instructions per
// element at n = 6, 240 of them FP64, on index arithmetic and on moving values between its
// phases; a line keeps its indices and one of its two derivatives in registers: 375, of
// which 180 FP64.  1024^2 elements, p = 5 (2.42 GB): 1.23 -> 0.73 ms, 3.3 TB/s, FP64 pipe 43 %,
// load/store pipe 60 % busy, issue 46 % with three warps per scheduler: bound by the latency
// of dependent FP64 and shared-memory operations.
#pragma once
#include "device_math.cuh"
#include "frsdg_internal.hpp"
#include "physics.cuh"
#include "pplimit.cuh"

namespace frsdg
{

// Face points of a tile: the records of both sides and whether they are the tile's own
// lines (else halo or ghost), packed: low side | high side << 12 | flags.
enum : unsigned
{
    FP_LOW = 1u << 24,
    FP_HIGH = 1u << 25,
    FP_ANY = 1u << 26
};

constexpr int kSMs = 148;  // B200: residencies and prefetch distances are counted in its SMs

// The FP32 residual (S = float) keeps the four equations of a node in one 16-byte plane and a
// record in a float4 and a float2.
template <int N, int GEO, int VAR = 0, class S = double> struct Line2D
{
    static constexpr bool F32 = sizeof(S) == 4;
    static constexpr int NN = N * N, ND = 4 * NN;
    // VAR 0: the tuned tile; 1: half its rows (a candidate of the batch autotuner); 2: a
    // 4 x 4 tile with a warp per 32 face points, one round of the face pass instead of
    // several: the shorter chain of small meshes (launch_line)
    static constexpr bool CURVED = GEO == GEO_CURVED;
    static constexpr int TX = VAR == 2 ? 4 : line_tile_x(N, CURVED), TY0 = line_tile_y(N, CURVED);
    static constexpr int TY = VAR == 2 ? 4 : VAR == 0 || TY0 == 1 ? TY0 : TY0 / 2;
    static constexpr int TE = TX * TY;
    static constexpr int NT = TE * N;                      // line threads
    // face points: x-faces [row][face][pos], then y-faces [face][column][pos], each in chunks of 32
    static constexpr int NXF = (TX + 1) * TY * N, NYF = TX * (TY + 1) * N;
    static constexpr int CX = (NXF + 31) / 32, CY = (NYF + 31) / 32;
    static constexpr int BT = VAR == 2 && CX + CY > (NT + 31) / 32 ? (CX + CY) * 32 : (NT + 31) / 32 * 32;
    static constexpr int NW = BT / 32;
    static constexpr int NHALO = 2 * TY * N + 2 * TX * N;
    // Shared memory in units of 16 bytes, strides chosen so that eight consecutive lanes hit
    // distinct banks both along columns and along rows (N = 3, 5 and 10: nearly).
    // Flux planes (two equations of a node each): [e ES + l RS + k].
    static constexpr int RS = N == 2 ? 3 : N == 3 || N == 4 ? 5 : N == 5 ? 7 : N <= 9 ? 9 : 11;
    static constexpr int ES = N == 2 ? 6 : N == 3 ? 15 : N == 4 ? 20 : N == 5 ? 37 : N <= 9 ? N * RS : 114;
    static constexpr int ROT = N == 5 ? 2 : 0;             // row of thread m of element e: (m + ROT e) mod N
    static constexpr int PLANE = TE * ES;
    static constexpr int NP = F32 ? 1 : 2;                 // planes of a flux
    static constexpr int NPLANE = GEO == GEO_CURVED ? 2 * NP : NP;
    // Face records, three planes (rho, rho E | u, v | p, c): the four face lines of each
    // element (corner nodes twice), then the halo traces.  A record is read by the one face
    // point of its line and then holds the jump of that side in its first two planes.
    // Lines at 0 (left), oB, oR, oT; oR keeps the left and right lines' stores apart.
    static constexpr int oB = N, oR = N == 2 ? 5 : N == 3 ? 9 : N == 4 ? 10 : N == 8 ? 17 : 2 * N, oT = oR + N;
    static constexpr int DS = N == 8 ? 33 : oT + N + ((N - oT - N) % 8 + 8) % 8;
    static constexpr int HXL = TE * DS, HXR = HXL + TY * N, HYB = HXR + TY * N, HYT = HYB + TX * N;
    static constexpr int RPL = TE * DS + NHALO;
    static constexpr size_t oRec = size_t(NPLANE) * PLANE * 16;
    static constexpr size_t bytes = oRec + size_t(RPL) * (F32 ? 24 : 48);
    static_assert(RPL < 4096, "records fit the packed face points");
    __host__ __device__ static constexpr unsigned face_point(bool xf, int t, int txe, int tye)
    {
        const int pos = t % N, r = t / N;
        const int row = xf ? r / (TX + 1) : r % TX, fc = xf ? r % (TX + 1) : r / TX;
        const int lim = xf ? txe : tye;
        if (t >= (xf ? NXF : NYF) || row >= (xf ? tye : txe) || fc > lim) return 0u;
        const int eM = xf ? row * TX + fc - 1 : (fc - 1) * TX + row, eP = xf ? eM + 1 : eM + TX;
        const int rM = fc > 0 ? eM * DS + (xf ? oR : oT) + pos : (xf ? HXL : HYB) + row * N + pos;
        const int rP = fc < lim ? eP * DS + (xf ? 0 : oB) + pos : (xf ? HXR : HYT) + row * N + pos;
        return unsigned(rM) | unsigned(rP) << 12 | (fc > 0 ? FP_LOW : 0u) | (fc < lim ? FP_HIGH : 0u) | FP_ANY;
    }
    // Co-resident CTAs: what shared memory admits, at most 16 warps at n <= 4 and in the small
    // variant (128 registers), 15 at n = 5, 12 above (168 registers: at n = 6, 15 warps with
    // narrower strides spill, 0.80 against 0.73 ms on the 1024^2 blast; nine warps are as fast; n >= 7
    // not swept, and the affine tuned tile spills 0.2 KB at n = 8 and 0.7 KB at n = 10);
    // FP32 16 (512^2 blast, p = 3, 4, 5: 0.134, 0.201, 0.217 ms with the face tiles, 0.059,
    // 0.094, 0.117 here; 12 to 24 warps within 8 %)
    static constexpr int CTAS_SM = int((227 * 1024) / (bytes + 1024));
    static constexpr int WARPS = F32 || VAR == 2 || N <= 4 ? 16 : N == 5 ? 15 : 12;
    static constexpr int CTAS_W = WARPS / NW > 0 ? WARPS / NW : 1;
    static constexpr int CTAS = CTAS_SM < CTAS_W ? (CTAS_SM > 0 ? CTAS_SM : 1) : CTAS_W;
};

// The packed face points of a whole tile (a partial one computes its own).
template <class T> struct FaceTable
{
    unsigned v[(T::CX + T::CY) * 32];
    constexpr FaceTable() : v{}
    {
        for (int c = 0; c < T::CX + T::CY; ++c)
            for (int i = 0; i < 32; ++i)
                v[c * 32 + i] = T::face_point(c < T::CX, (c < T::CX ? c : c - T::CX) * 32 + i, T::TX, T::TY);
    }
};
template <class T> __device__ const FaceTable<T> kFaceTable{};

struct Node4
{
    double v[4];
};
__device__ __forceinline__ void load_node(const Fr2dArgs& a, int64_t off, double s[4])
{
    const double2 x0 = __ldg(reinterpret_cast<const double2*>(a.U + off));
    const double2 x1 = __ldg(reinterpret_cast<const double2*>(a.U + off + 2));
    s[0] = x0.x; s[1] = x0.y; s[2] = x1.x; s[3] = x1.y;
}
__device__ __forceinline__ void load_node(const Fr2dArgs& a, int64_t off, float s[4])
{
    const float4 x = __ldg(reinterpret_cast<const float4*>(reinterpret_cast<const float*>(a.U) + off));
    s[0] = x.x; s[1] = x.y; s[2] = x.z; s[3] = x.w;
}
// 32-byte accesses of a node (p 32-byte aligned)
__device__ __forceinline__ void load_node32(const double* p, double s[4])
{
    asm("ld.global.nc.v4.f64 {%0, %1, %2, %3}, [%4];" : "=d"(s[0]), "=d"(s[1]), "=d"(s[2]), "=d"(s[3]) : "l"(p));
}
__device__ __forceinline__ void store_node32(double* p, double v0, double v1, double v2, double v3)
{
    asm volatile("st.global.v4.f64 [%0], {%1, %2, %3, %4};" ::"l"(p), "d"(v0), "d"(v1), "d"(v2), "d"(v3) : "memory");
}
// M of the change of variables (prim_to_cons_elem, problem_def.hpp:36-51), out of line:
// its branch must not come between the loads of a column
static __device__ __noinline__ Node4 prim_to_cons_node(double q0, double q1, double q2, double q3)
{
    Node4 s;
    const double rho = exp(q0);
    const double ssq = (0.0 + q1 * q1) + q2 * q2;
    s.v[0] = rho;
    s.v[1] = rho * q1;
    s.v[2] = rho * q2;
    s.v[3] = rho * (exp(q3) + 0.5 * ssq);
    return s;
}
__device__ __forceinline__ void to_conservative(const Fr2dArgs& a, double s[4])
{
    if (!a.cond_sys) return;
    const Node4 c = prim_to_cons_node(s[0], s[1], s[2], s[3]);
    s[0] = c.v[0]; s[1] = c.v[1]; s[2] = c.v[2]; s[3] = c.v[3];
}

// Stage epilogue (Fr2dArgs::post): V holds the stage outputs of the thread's column.  The
// spectral filter of the post-step (SpectralFilter::apply_filter, filter.hpp:425-445: half
// the sum of the filter along the element's rows and along its columns) takes the rows
// through the flux planes and the columns in registers; the tile is stored, and elements
// with a node whose density or pressure may lie below the limiter's floor go through the
// positivity limiter in place, one warp each (pp_element2d, which screens them again).
template <class T, int N, int GAS>
__device__ __forceinline__ void line_epilogue(const Fr2dArgs& a, const Ops& ops, bool own, int e, int m, int i0, int j0,
                                              int txe, int tye, double (&V)[4][N], double* out, double2* sF)
{
    constexpr int TX = T::TX, TE = T::TE, BT = T::BT, ND = T::ND;
    const int tid = threadIdx.x;
    const PostArgs& P = *a.pa;
    const bool limit = (a.post & POST_PP) != 0, want_amax = (a.post & POST_AMAX) != 0;
    __shared__ int s_flag[TE];
    __shared__ unsigned long long s_amax;
    for (int q = tid; q < TE; q += BT) s_flag[q] = 0;
    if (tid == 0) s_amax = 0ull;
    if (a.post & POST_FILTER)
    {
        // the thread's own column of the planes: read by no other thread since the row pass
        if (own)
        {
#pragma unroll
            for (int l = 0; l < N; ++l)
            {
                const int at = e * T::ES + l * T::RS + m;
                sF[at] = make_double2(V[0][l], V[1][l]);
                sF[T::PLANE + at] = make_double2(V[2][l], V[3][l]);
            }
        }
        __syncthreads();
        if (own)
        {
#pragma unroll
            for (int pl = 0; pl < 2; ++pl)
            {
                double2* f = sF + pl * T::PLANE + e * T::ES + (T::ROT ? (m + T::ROT * e) % N : m) * T::RS;
                double2 x[N];
#pragma unroll
                for (int q = 0; q < N; ++q) x[q] = f[q];
#pragma unroll
                for (int r = 0; r < N; ++r)
                {
                    double s0 = 0.0, s1 = 0.0;
#pragma unroll
                    for (int c = 0; c < N; ++c)
                    {
                        s0 += ops.F[r * N + c] * x[c].x;
                        s1 += ops.F[r * N + c] * x[c].y;
                    }
                    f[r] = make_double2(s0, s1);
                }
            }
        }
        __syncthreads();
        if (own)
        {
#pragma unroll
            for (int pl = 0; pl < 2; ++pl)
            {
                double y0[N], y1[N];
#pragma unroll
                for (int r = 0; r < N; ++r)
                {
                    y0[r] = y1[r] = 0.0;
#pragma unroll
                    for (int c = 0; c < N; ++c)
                    {
                        y0[r] += ops.F[r * N + c] * V[2 * pl][c];
                        y1[r] += ops.F[r * N + c] * V[2 * pl + 1][c];
                    }
                }
#pragma unroll
                for (int r = 0; r < N; ++r)
                {
                    const double2 x = sF[pl * T::PLANE + e * T::ES + r * T::RS + m];
                    V[2 * pl][r] = 0.5 * (x.x + y0[r]);
                    V[2 * pl + 1][r] = 0.5 * (x.y + y1[r]);
                }
            }
        }
    }
    else
        __syncthreads();  // s_flag
    const PPView v{GAS == 0 ? FRSDG_GAS_IDEAL : FRSDG_GAS_VDW, a.gas, P.pp_eps, P.w, P.detJ};
    const double thr = v.eps0 * (1.0 + 1e-10);
    bool clear = true;
    if (own)
    {
        unsigned bad = 0;
#pragma unroll
        for (int l = 0; l < N; ++l)
        {
            double2* o = reinterpret_cast<double2*>(out + l * N * 4);
            o[0] = make_double2(V[0][l], V[1][l]);
            o[1] = make_double2(V[2][l], V[3][l]);
            if (limit)
            {
                const double u[4] = {V[0][l], V[1][l], V[2][l], V[3][l]};
                clear = clear && u[0] > thr && pp_pressure_fast(v, u, MathDeferred{bad}) > thr;
            }
        }
        clear = clear && !bad;
        if (!clear) s_flag[e] = 1;
    }
    if (!limit && !want_amax) return;
    if (want_amax)
    {
        // every node above the floor as it leaves the stage, in marked elements too (as the tiles
        // of mixed stages: both forms of a batch then take the same steps); the limiter adds
        // the marked elements' speeds after limiting
        double w = 0.0;
        if (own)
        {
#pragma unroll 1
            for (int l = 0; l < N; ++l)
            {
                const double2* o = reinterpret_cast<const double2*>(out + l * N * 4);  // this thread's own stores
                const double2 x = o[0], y = o[1];
                const double u[4] = {x.x, x.y, y.x, y.y};
                if (clear || (u[0] > thr && pp_pressure_fast(v, u) > thr)) w = fmax(w, node_wave_speed_fast(v, u));
            }
        }
        w = -pp_warp_min(-w);
        if ((tid & 31) == 0 && w > 0.0 && w < 1e300)
            atomicMax(&s_amax, static_cast<unsigned long long>(__double_as_longlong(w)));
    }
    __syncthreads();  // flags and stores
    if (limit)
    {
        double* base = static_cast<double*>(a.out);
        for (int q = tid / 32; q < TE; q += BT / 32)
        {
            const int tx = q % TX, ty = q / TX;
            if (tx >= txe || ty >= tye || !s_flag[q]) continue;  // uniform across the warp
            const int64_t e_glob = int64_t(j0 + ty + a.row_base) * a.Nx + (i0 + tx);
            pp_element2d<N>(v, base + (int64_t(j0 + ty) * a.Nx + (i0 + tx)) * ND, nullptr, e_glob, true, false,
                            want_amax ? &s_amax : nullptr);
        }
    }
    __syncthreads();  // s_flag and s_amax are reused by the CTA's next tile
    if (want_amax && tid == 0 && s_amax) atomicMax(P.amax, s_amax);
}

// The requested output form of an FP64 column (Mode), E its residual.
template <class T, int N, int GAS, bool POST>
__device__ __forceinline__ void line_output(const Fr2dArgs& a, const Ops& ops, bool own, int e, int m, int64_t ebase,
                                            int i0, int j0, int txe, int tye, double (&E)[4][N], double2* sF)
{
    double* out = static_cast<double*>(a.out) + ebase + m * 4;
    auto put = [&](int l, double v0, double v1, double v2, double v3) {
        double2* o = reinterpret_cast<double2*>(out + l * N * 4);
        o[0] = make_double2(v0, v1);
        o[1] = make_double2(v2, v3);
    };
    if (a.mode == MODE_STAGE)
    {
        if (own)
        {
            const int64_t o0 = ebase + m * 4;
            auto get = [&](const double* p, int l, double v[4]) {
                const double2 x = __ldg(reinterpret_cast<const double2*>(p + o0 + l * N * 4));
                const double2 y = __ldg(reinterpret_cast<const double2*>(p + o0 + l * N * 4 + 2));
                v[0] = x.x; v[1] = x.y; v[2] = y.x; v[3] = y.y;
            };
#pragma unroll
            for (int l = 0; l < N; ++l)
            {
                double o[4] = {0.0, 0.0, 0.0, 0.0}, q[4];
                if (a.st.A)
                {
                    get(a.st.A, l, q);
#pragma unroll
                    for (int eq = 0; eq < 4; ++eq) o[eq] = a.st.alpha * q[eq];
                }
                if (a.st.B)
                {
                    get(a.st.B, l, q);
#pragma unroll
                    for (int eq = 0; eq < 4; ++eq) o[eq] = o[eq] + a.st.beta * q[eq];
                }
                if (a.st.acc)
                {
                    double2* p = reinterpret_cast<double2*>(a.st.acc + o0 + l * N * 4);
                    const double2 x = p[0], y = p[1];
                    p[0] = make_double2(x.x - a.st.delta * E[0][l], x.y - a.st.delta * E[1][l]);
                    p[1] = make_double2(y.x - a.st.delta * E[2][l], y.y - a.st.delta * E[3][l]);
                }
#pragma unroll
                for (int eq = 0; eq < 4; ++eq) E[eq][l] = o[eq] - a.st.gamma * E[eq][l];
                if constexpr (!POST) put(l, E[0][l], E[1][l], E[2][l], E[3][l]);
            }
        }
        if constexpr (POST) line_epilogue<T, N, GAS>(a, ops, own, e, m, i0, j0, txe, tye, E, out, sF);
    }
    else if (own)
    {
        if (a.mode == MODE_IFUNC)
        {
            const double* w = a.W + ebase + m * 4;
#pragma unroll
            for (int l = 0; l < N; ++l)
            {
                const double2 x = __ldg(reinterpret_cast<const double2*>(w + l * N * 4));
                const double2 y = __ldg(reinterpret_cast<const double2*>(w + l * N * 4 + 2));
                put(l, x.x + E[0][l], x.y + E[1][l], y.x + E[2][l], y.y + E[3][l]);
            }
        }
        else
        {
            const double sg = a.mode == MODE_RHS ? -1.0 : 1.0;
            if ((reinterpret_cast<uintptr_t>(a.out) & 31) == 0)
            {
#pragma unroll
                for (int l = 0; l < N; ++l) store_node32(out + l * N * 4, sg * E[0][l], sg * E[1][l], sg * E[2][l], sg * E[3][l]);
            }
            else
            {
#pragma unroll
                for (int l = 0; l < N; ++l) put(l, sg * E[0][l], sg * E[1][l], sg * E[2][l], sg * E[3][l]);
            }
        }
    }
}

// A tile's inputs of one thread: its column and its halo node (record -1: none).
template <class S, int N> struct LineIn
{
    S   u[N][4];
    S   hs[4];
    int    hrec;
};

// Halo node q of tile (bx, by): its offset in U and its record, or -1.
template <class T, int N>
__device__ __forceinline__ int line_halo(const Fr2dArgs& a, int bx, int by, int q, int64_t& off)
{
    constexpr int TX = T::TX, TY = T::TY, ND = T::ND;
    const int Nx = a.Nx, Ny = a.Ny;
    const int i0 = bx * TX, j0 = by * TY + a.row_begin;
    const int txe = min(TX, Nx - i0), tye = min(TY, a.row_end - j0);
    int ge_i, ge_j, node, r;
    bool ok;
    if (q < 2 * TY * N)
    {
        const int side = q / (TY * N), y = (q % (TY * N)) / N, p = q % N;
        ok = y < tye;
        ge_j = j0 + y;
        ge_i = side == 0 ? i0 - 1 : i0 + txe;
        if (ge_i < 0 || ge_i >= Nx)
        {
            ok = ok && a.per_x;
            ge_i = ge_i < 0 ? ge_i + Nx : ge_i - Nx;
        }
        node = p * N + (side == 0 ? N - 1 : 0);
        r = T::HXL + q;
    }
    else
    {
        const int qq = q - 2 * TY * N;
        const int side = qq / (TX * N), x = (qq % (TX * N)) / N, p = qq % N;
        ok = x < txe;
        ge_i = i0 + x;
        ge_j = side == 0 ? j0 - 1 : j0 + tye;
        if (ge_j < 0 || ge_j >= Ny)
        {
            ok = ok && a.per_y;
            ge_j = ge_j < 0 ? ge_j + Ny : ge_j - Ny;
        }
        node = side == 0 ? (N - 1) * N + p : p;
        r = T::HYB + qq;
    }
    off = (int64_t(ge_j) * Nx + ge_i) * ND + node * 4;
    return ok ? r : -1;
}

// The loads of a tile's inputs, all in flight at once (as stored; cond_sys maps them later).
template <class T, class S, int N>
__device__ __forceinline__ void line_load(const Fr2dArgs& a, int bx, int by, LineIn<S, N>& in)
{
    constexpr int TX = T::TX, TY = T::TY, ND = T::ND;
    const int tid = threadIdx.x;
    const int m = tid % N, e = tid / N, i = bx * TX + e % TX, j = by * TY + a.row_begin + e / TX;
    int64_t hoff = 0;
    in.hrec = tid < T::NHALO ? line_halo<T, N>(a, bx, by, tid, hoff) : -1;
    const bool mine = tid < T::NT && i < a.Nx && j < a.row_end;
    const int64_t base = (int64_t(j) * a.Nx + i) * ND + m * 4;
    if constexpr (!T::F32)
    {
        if ((reinterpret_cast<uintptr_t>(a.U) & 31) == 0)
        {
            if (in.hrec >= 0) load_node32(a.U + hoff, in.hs);
            if (!mine) return;
#pragma unroll
            for (int l = 0; l < N; ++l) load_node32(a.U + base + l * N * 4, in.u[l]);
            return;
        }
    }
    {
        if (in.hrec >= 0) load_node(a, hoff, in.hs);
        if (!mine) return;
#pragma unroll
        for (int l = 0; l < N; ++l) load_node(a, base + l * N * 4, in.u[l]);
    }
}

// One tile (bx, by); smem: T::bytes, 16-byte aligned.  Consecutive tiles of a CTA need no
// barrier in between: what the output pass reads of shared memory, the same thread
// overwrites next.  S = float: MODE_RESIDUAL on an FP32 state, FP32 output.
template <class S, int N, int GAS, int RIEM, int GEO, int VAR, bool POST>
__device__ __forceinline__ void fr2d_line_tile(const Fr2dArgs& a, const Ops& ops, int bx, int by, unsigned char* smem)
{
    using T = Line2D<N, GEO, VAR, S>;
    using V = typename std::conditional<T::F32, float4, double2>::type;  // 16 bytes of a flux plane or a record
    constexpr int TX = T::TX, TY = T::TY, NN = T::NN, ND = T::ND, BT = T::BT;
    constexpr bool F32 = T::F32;
    V* sF = reinterpret_cast<V*>(smem);                    // [plane][e ES + l RS + k]
    V* sG = sF + T::NP * T::PLANE;                         // curved only
    V* sR = reinterpret_cast<V*>(smem + T::oRec);          // records [plane][e DS + line + pos], halo
    float2* sR2 = reinterpret_cast<float2*>(sR + T::RPL);  // FP32: (p, c)
    LineIn<S, N> in;
    line_load<T>(a, bx, by, in);
    const int tid = threadIdx.x;
    const int Nx = a.Nx, Ny = a.Ny;
    const int i0 = bx * TX, j0 = by * TY + a.row_begin;
    const int txe = min(TX, Nx - i0), tye = min(TY, a.row_end - j0);
    const GasParams g = a.gas;
    const bool line = tid < T::NT;
    const int m = tid % N, e = line ? tid / N : 0, tx = e % TX, ty = e / TX;  // line m of element e
    const bool own = line && tx < txe && ty < tye;
    const int64_t ebase = (int64_t(j0 + ty) * Nx + (i0 + tx)) * ND;
    const int64_t mbase = (int64_t(j0 + ty + a.row_base) * Nx + (i0 + tx)) * NN;

    // operands of the output pass: their lines into L2 first (hints)
    if (a.mode == MODE_STAGE || a.mode == MODE_IFUNC)
    {
        constexpr int LROW = (TX * ND * int(sizeof(double)) + 127) / 128;
        const int lrow = (txe * ND * int(sizeof(double)) + 127) / 128;
        const double* b0 = a.mode == MODE_STAGE ? a.st.A : a.W;
        const double* b1 = a.mode == MODE_STAGE ? a.st.B : nullptr;
        for (int q = tid; q < 2 * TY * LROW; q += BT)
        {
            const int which = q / (TY * LROW), r = q % (TY * LROW), y = r / LROW, ln = r % LROW;
            const double* base = which ? b1 : b0;
            if (base && base != a.U && y < tye && ln < lrow)
                asm volatile("prefetch.global.L2 [%0];" ::"l"(base + (int64_t(j0 + y) * Nx + i0) * ND + ln * 16));
        }
    }

    // A face record.  Affine meshes keep the velocities in the face's frame (normal,
    // tangential: (u, v) on x-faces, (v, -u) on y-faces), so that one copy of the face
    // pass serves both directions; jumps are left in that frame too.
    constexpr bool AFF = GEO == GEO_AFFINE;
    // face point of this lane in chunk c, loaded a round ahead
    const bool full = txe == TX && tye == TY;
    auto face_word = [&](int c) -> unsigned {
        if (c >= T::CX + T::CY) return 0u;
        return full ? __ldg(&kFaceTable<T>.v[c * 32 + (tid & 31)])
                    : T::face_point(c < T::CX, (c < T::CX ? c : c - T::CX) * 32 + (tid & 31), txe, tye);
    };
    unsigned next_fp = face_word(tid / 32);
    // a node's four values into the planes of a flux
    auto put_flux = [&](V* p, int at, const S v[4]) {
        if constexpr (F32) p[at] = make_float4(v[0], v[1], v[2], v[3]);
        else
        {
            p[at] = make_double2(v[0], v[1]);
            p[T::PLANE + at] = make_double2(v[2], v[3]);
        }
    };
    auto get_flux = [&](const V* p, int at, S v[4]) {
        if constexpr (F32)
        {
            const float4 x = p[at];
            v[0] = x.x; v[1] = x.y; v[2] = x.z; v[3] = x.w;
        }
        else
        {
            const double2 x = p[at], y = p[T::PLANE + at];
            v[0] = x.x; v[1] = x.y; v[2] = y.x; v[3] = y.y;
        }
    };
    // the jump of a side, in the record's place
    auto get_jump = [&](int q, S v[4]) {
        if constexpr (F32)
        {
            const float4 x = sR[q];
            v[0] = x.x; v[1] = x.y; v[2] = x.z; v[3] = x.w;
        }
        else
        {
            const double2 x = sR[q], y = sR[T::RPL + q];
            v[0] = x.x; v[1] = x.y; v[2] = y.x; v[3] = y.y;
        }
    };
    auto put_record = [&](int r, bool yface, const S s[4], const NodePrim<S>& pr, S c) {
        const S un = AFF && yface ? pr.v : pr.u, ut = AFF && yface ? -pr.u : pr.v;
        if constexpr (F32)
        {
            sR[r] = make_float4(s[0], s[3], un, ut);
            sR2[r] = make_float2(pr.p, c);
        }
        else
        {
            sR[r] = make_double2(s[0], s[3]);
            sR[T::RPL + r] = make_double2(un, ut);
            sR[2 * T::RPL + r] = make_double2(pr.p, c);
        }
    };
    auto halo_node = [&](int r, const S s[4], const auto& mth) {
        const NodePrim<S> pr = node_prim<GAS>(g, s[0], s[1], s[2], s[3], mth);
        put_record(r, r >= T::HYB, s, pr, node_sound_speed<GAS>(g, pr, mth));
    };
    // one node of the column: fluxes to shared memory (F; curved also G) and g4, records
    auto column_node = [&](int l, const S s[4], S g4[4], const auto& mth) {
        const NodePrim<S> pr = node_prim<GAS>(g, s[0], s[1], s[2], s[3], mth);
        // (every node's sound speed: a branch on boundary nodes diverges in every warp)
        const S c = node_sound_speed<GAS>(g, pr, mth);
        const S rEp = s[3] + pr.p, ruv = s[1] * pr.v;
        const S f4[4] = {s[1], s[1] * pr.u + pr.p, ruv, pr.u * rEp};
        g4[0] = s[2];
        g4[1] = ruv;
        g4[2] = s[2] * pr.v + pr.p;
        g4[3] = pr.v * rEp;
        const int at = e * T::ES + l * T::RS + m;
        put_flux(sF, at, f4);
        if constexpr (!AFF) put_flux(sG, at, g4);
        if (m == 0 || m == N - 1) put_record(e * T::DS + (m == 0 ? 0 : T::oR) + l, false, s, pr, c);
        if (l == 0 || l == N - 1) put_record(e * T::DS + (l == 0 ? T::oB : T::oT) + m, true, s, pr, c);
    };

    // ---- column pass
    S E[4][N];  // eta part of the column's residual
    {
        S G[4][AFF ? N : 1];  // curved: both fluxes come back from shared memory
        if (own)
        {
            unsigned bad = 0;
            if constexpr (!F32)
            {
                if (a.cond_sys)
                {
#pragma unroll
                    for (int l = 0; l < N; ++l) to_conservative(a, in.u[l]);
                }
            }
#pragma unroll
            for (int l = 0; l < N; ++l)
            {
                S g4[4];
                column_node(l, in.u[l], g4, MathDeferred{bad});
#pragma unroll
                for (int eq = 0; eq < 4; ++eq)
                    if constexpr (AFF) G[eq][l] = g4[eq];
            }
            if (bad)
            {
                // a reciprocal or square root met an input outside the fast range: the whole
                // column again with the checked functions, the densities counted (a node
                // without such an input has a positive finite density)
#pragma unroll 1
                for (int l = 0; l < N; ++l)
                {
                    S s[4], g4[4];
                    load_node(a, ebase + (l * N + m) * 4, s);
                    if constexpr (!F32) to_conservative(a, s);
                    if (!density_ok(s[0]) && a.bad) atomicAdd(a.bad, 1ull);
                    column_node(l, s, g4, MathChecked{});
                    if constexpr (AFF)
                    {
#pragma unroll
                        for (int q = 0; q < N; ++q)
                            if (q == l)
                            {
#pragma unroll
                                for (int eq = 0; eq < 4; ++eq) G[eq][q] = g4[eq];
                            }
                    }
                }
            }
        }
        for (int q = tid; q < T::NHALO; q += BT)
        {
            if (q != tid)
            {
                int64_t hoff;
                in.hrec = line_halo<T, N>(a, bx, by, q, hoff);
                if (in.hrec >= 0) load_node(a, hoff, in.hs);
            }
            if (in.hrec < 0) continue;
            if constexpr (!F32) to_conservative(a, in.hs);
            unsigned bad = 0;
            halo_node(in.hrec, in.hs, MathDeferred{bad});
            if (bad) halo_node(in.hrec, in.hs, MathChecked{});
        }
        if (own)
        {
            // eta-derivative of the column (curved: of F too, with the node's metrics; affine:
            // unscaled)
            if constexpr (!AFF)
            {
                const double* mt = a.metrics + (mbase + m) * 4 + 2;
                const int at = e * T::ES + m;
#pragma unroll
                for (int pl = 0; pl < T::NP; ++pl)
                {
                    constexpr int W = F32 ? 4 : 2;  // equations per plane
                    S f[W][N], h[W][N];
#pragma unroll
                    for (int q = 0; q < N; ++q)
                    {
                        const V x = sF[pl * T::PLANE + at + q * T::RS], y = sG[pl * T::PLANE + at + q * T::RS];
                        f[0][q] = x.x; f[1][q] = x.y;
                        h[0][q] = y.x; h[1][q] = y.y;
                        if constexpr (F32)
                        {
                            f[2][q] = x.z; f[3][q] = x.w;
                            h[2][q] = y.z; h[3][q] = y.w;
                        }
                    }
#pragma unroll
                    for (int w = 0; w < W; ++w)
                    {
                        center_line<S, N>(f[w]);
                        center_line<S, N>(h[w]);
                    }
#pragma unroll
                    for (int l = 0; l < N; ++l)
                    {
                        const double2 me = __ldg(reinterpret_cast<const double2*>(mt + l * N * 4));
#pragma unroll
                        for (int w = 0; w < W; ++w)
                        {
                            S df = S(0.0), dh = S(0.0);
#pragma unroll
                            for (int q = 0; q < N; ++q)
                            {
                                df = df + opD<S>(ops, l * N + q) * f[w][q];
                                dh = dh + opD<S>(ops, l * N + q) * h[w][q];
                            }
                            E[W * pl + w][l] = S(me.x) * df + S(me.y) * dh;
                        }
                    }
                }
            }
            else
            {
#pragma unroll
                for (int eq = 0; eq < 4; ++eq)
                {
                    center_line<S, N>(G[eq]);
#pragma unroll
                    for (int l = 0; l < N; ++l)
                    {
                        S dG = S(0.0);
#pragma unroll
                        for (int q = 0; q < N; ++q) dG = dG + opD<S>(ops, l * N + q) * G[eq][q];
                        E[eq][l] = dG;
                    }
                }
            }
        }
    }
    __syncthreads();

    // ---- face pass: x-faces on the first chunks of 32 points, y-faces on the others
    {
        const bool lowx = !a.per_x && i0 == 0, highx = !a.per_x && i0 + txe == Nx;
        const bool lowy = !a.per_y && j0 == 0, highy = !a.per_y && j0 + tye == Ny;
#pragma unroll 1
        for (int c = tid / 32; c < T::CX + T::CY; c += T::NW)
        {
            const bool XF = c < T::CX;  // uniform across the warp
            const unsigned fp = next_fp;
            next_fp = face_word(c + T::NW);
            if (!(fp & FP_ANY)) continue;
            const int rM = fp & 0xfffu, rP = (fp >> 12) & 0xfffu;
            const bool inM = fp & FP_LOW, inP = fp & FP_HIGH;
            S L[RF_N], R[RF_N];
            auto get = [&](int q, S v[RF_N]) {
                if constexpr (F32)
                {
                    const float4 x = sR[q];
                    const float2 z = sR2[q];
                    v[RF_RHO] = x.x; v[RF_E] = x.y; v[RF_U] = x.z; v[RF_V] = x.w; v[RF_P] = z.x; v[RF_C] = z.y;
                }
                else
                {
                    const double2 x = sR[q], y = sR[T::RPL + q], z = sR[2 * T::RPL + q];
                    v[RF_RHO] = x.x; v[RF_E] = x.y; v[RF_U] = y.x; v[RF_V] = y.y; v[RF_P] = z.x; v[RF_C] = z.y;
                }
            };
            get(rM, L);
            get(rP, R);
            // element and position of an own side, the low one if there is
            const int sideM = XF ? T::oR : T::oT, sideP = XF ? 0 : T::oB;
            auto pos_of = [&](int& ei) {
                ei = (inM ? rM : rP) / T::DS;
                return (inM ? rM - sideM : rP - sideP) - ei * T::DS;
            };
            double nx = XF ? 1.0 : 0.0, ny = XF ? 0.0 : 1.0;
            if constexpr (GEO == GEO_CURVED)
            {
                int ei;
                const int pos = pos_of(ei), up = inM ? 1 : 0;
                const int gI = i0 + ei % TX + (XF ? up : 0), gJ = j0 + ei / TX + (XF ? 0 : up);
                const double2 nn = XF ? __ldg(reinterpret_cast<const double2*>(a.xnorm) + (int64_t(gJ + a.row_base) * (Nx + 1) + gI) * N + pos)
                                      : __ldg(reinterpret_cast<const double2*>(a.ynorm) + (int64_t(gJ + a.row_base) * Nx + gI) * N + pos);
                nx = nn.x;
                ny = nn.y;
            }
            // physical boundary (rare): the ghost of the interior trace
            if ((!inM && (XF ? lowx : lowy)) || (!inP && (XF ? highx : highy)))
            {
                int ei;
                const int pos = pos_of(ei);
                const int gI = i0 + ei % TX, gJ = j0 + ei / TX;
                const int dir = XF ? (inM ? FRSDG_RIGHT : FRSDG_LEFT) : (inM ? FRSDG_TOP : FRSDG_BOTTOM);
                const int bi = XF ? (gJ + a.row_base) * N + pos : gI * N + pos;
                const double2 xy = __ldg(reinterpret_cast<const double2*>(a.bxy[dir]) + bi);
                const int node = XF ? pos * N + (inM ? N - 1 : 0) : (inM ? N - 1 : 0) * N + pos;
                const int64_t ioff = (int64_t(gJ) * Nx + gI) * ND + node * 4;
                const Rec<S> gh = ghost_record<GAS, S>(a, dir, ioff, xy.x, xy.y, nx, ny);
#pragma unroll
                for (int f = 0; f < RF_N; ++f)
                {
                    const S q = !AFF || XF || (f != RF_U && f != RF_V) ? gh.v[f] : f == RF_U ? gh.v[RF_V] : -gh.v[RF_U];
                    if (inM) R[f] = q;
                    else L[f] = q;
                }
            }
            constexpr int AXIS = AFF ? 0 : 2;
            S Fs[4], FL[4], FR[4];
            unsigned bad = 0;
            riemann_sides<RIEM, AXIS, S>(L, R, S(nx), S(ny), Fs, FL, FR, MathDeferred{bad});
            if (bad) riemann_sides<RIEM, AXIS, S>(L, R, S(nx), S(ny), Fs, FL, FR, MathChecked{});
            // affine: unscaled, the scale joins the metric factor of the element
            auto jump = [&](int q, int side, bool hi, const S Fn[4]) {
                S d[4];
#pragma unroll
                for (int eq = 0; eq < 4; ++eq) d[eq] = Fs[eq] - Fn[eq];
                if constexpr (!AFF)
                {
                    const int fe = q / T::DS, pos = q - fe * T::DS - side;
                    const int node = XF ? pos * N + (hi ? N - 1 : 0) : (hi ? N - 1 : 0) * N + pos;
                    const double* mt = a.metrics + ((int64_t(j0 + fe / TX + a.row_base) * Nx + (i0 + fe % TX)) * NN + node) * 4 + (XF ? 0 : 2);
                    const double2 mm = __ldg(reinterpret_cast<const double2*>(mt));
                    const S sc = S(sqrt(mm.x * mm.x + mm.y * mm.y));
#pragma unroll
                    for (int eq = 0; eq < 4; ++eq) d[eq] = sc * d[eq];
                }
                if constexpr (F32) sR[q] = make_float4(d[0], d[1], d[2], d[3]);
                else
                {
                    sR[q] = make_double2(d[0], d[1]);
                    sR[T::RPL + q] = make_double2(d[2], d[3]);
                }
            };
            if (inM) jump(rM, sideM, true, FL);
            if (inP) jump(rP, sideP, false, FR);
        }
    }
    __syncthreads();

    // ---- row pass: one row of element e, in place
    if (own)
    {
        const int mr = T::ROT ? (m + T::ROT * e) % N : m;
        const int at = e * T::ES + mr * T::RS;
        S dl[4], dr[4];
        get_jump(e * T::DS + mr, dl);
        get_jump(e * T::DS + T::oR + mr, dr);
#pragma unroll
        for (int pl = 0; pl < T::NP; ++pl)
        {
            constexpr int W = F32 ? 4 : 2;
            V* f = sF + pl * T::PLANE + at;
            S x[W][N], y[AFF ? 1 : W][N];
#pragma unroll
            for (int q = 0; q < N; ++q)
            {
                const V t = f[q];
                x[0][q] = t.x; x[1][q] = t.y;
                if constexpr (F32) { x[2][q] = t.z; x[3][q] = t.w; }
                if constexpr (!AFF)
                {
                    const V u = sG[pl * T::PLANE + at + q];
                    y[0][q] = u.x; y[1][q] = u.y;
                    if constexpr (F32) { y[2][q] = u.z; y[3][q] = u.w; }
                }
            }
#pragma unroll
            for (int w = 0; w < W; ++w)
            {
                center_line<S, N>(x[w]);
                if constexpr (!AFF) center_line<S, N>(y[w]);
            }
#pragma unroll
            for (int k = 0; k < N; ++k)
            {
                S r[W];
                double2 mx = make_double2(0.0, 0.0);
                if constexpr (!AFF) mx = __ldg(reinterpret_cast<const double2*>(a.metrics + (mbase + mr * N + k) * 4));
#pragma unroll
                for (int w = 0; w < W; ++w)
                {
                    const int eq = W * pl + w;
                    S d = S(0.0);
#pragma unroll
                    for (int q = 0; q < N; ++q) d = d + opD<S>(ops, k * N + q) * x[w][q];
                    if constexpr (!AFF)
                    {
                        S h = S(0.0);
#pragma unroll
                        for (int q = 0; q < N; ++q) h = h + opD<S>(ops, k * N + q) * y[w][q];
                        r[w] = ((S(mx.x) * d + S(mx.y) * h) + dl[eq] * opL<S>(ops, k)) + dr[eq] * opR<S>(ops, k);
                    }
                    else  // xi_x is also the scale of the jumps
                        r[w] = S(a.xi_x) * ((d + dl[eq] * opL<S>(ops, k)) + dr[eq] * opR<S>(ops, k));
                }
                if constexpr (F32) f[k] = make_float4(r[0], r[1], r[2], r[3]);
                else f[k] = make_double2(r[0], r[1]);
            }
        }
    }
    __syncthreads();

    // ---- output pass: column m of element e
    if (own)
    {
        S b[4], t[4];
        get_jump(e * T::DS + T::oB + m, b);
        get_jump(e * T::DS + T::oT + m, t);
        if constexpr (AFF)
        {
            // from the y-faces' frame: (d0, dn, dt, d3) to (d0, -dt, dn, d3)
            const S bn = b[1], tn = t[1];
            b[1] = -b[2];
            b[2] = bn;
            t[1] = -t[2];
            t[2] = tn;
        }
#pragma unroll
        for (int l = 0; l < N; ++l)
        {
            S x[4];
            get_flux(sF, e * T::ES + l * T::RS + m, x);
            const S dLl = opL<S>(ops, l), dRl = opR<S>(ops, l);
#pragma unroll
            for (int eq = 0; eq < 4; ++eq)
                // affine: eta_y is also the scale of the jumps
                E[eq][l] = AFF ? x[eq] + S(a.eta_y) * ((E[eq][l] + b[eq] * dLl) + t[eq] * dRl)
                               : ((x[eq] + E[eq][l]) + b[eq] * dLl) + t[eq] * dRl;
        }
    }
    if constexpr (F32)
    {
        if (own)
        {
            float4* o = reinterpret_cast<float4*>(static_cast<float*>(a.out) + ebase + m * 4);
#pragma unroll
            for (int l = 0; l < N; ++l) o[l * N] = make_float4(E[0][l], E[1][l], E[2][l], E[3][l]);
        }
    }
    else
        line_output<T, N, GAS, POST>(a, ops, own, e, m, ebase, i0, j0, txe, tye, E, sF);
}

template <class S, int N, int GAS, int RIEM, int GEO, int VAR, bool POST>
__global__ void __launch_bounds__((Line2D<N, GEO, VAR, S>::BT), (Line2D<N, GEO, VAR, S>::CTAS))
    fr2d_line_kernel(const __grid_constant__ Fr2dArgs a)
{
    extern __shared__ __align__(128) unsigned char smem_raw[];
    if constexpr (VAR != 2)
    {
        // the state of the tile one residency ahead into L2 (hints): its CTA starts on this
        // one's shared memory and registers, and finds its loads near
        using T = Line2D<N, GEO, VAR, S>;
        const int nb = int(blockIdx.y * gridDim.x + blockIdx.x) + T::CTAS * kSMs;
        const int by = nb / int(gridDim.x), bx = nb - by * int(gridDim.x);
        constexpr int LROW = (T::TX * T::ND * int(sizeof(S)) + 127) / 128, LV = 128 / int(sizeof(S));
        for (int q = threadIdx.x; q < T::TY * LROW; q += T::BT)
        {
            const int y = q / LROW, ln = q % LROW, j = by * T::TY + a.row_begin + y;
            if (j < a.row_end && bx * T::TX * T::ND + ln * LV < a.Nx * T::ND)
                asm volatile("prefetch.global.L2 [%0];" ::"l"(reinterpret_cast<const S*>(a.U) + (int64_t(j) * a.Nx + bx * T::TX) * T::ND + ln * LV));
        }
    }
    fr2d_line_tile<S, N, GAS, RIEM, GEO, VAR, POST>(a, a.ops, blockIdx.x, blockIdx.y, smem_raw);
}

// Kernel attributes are per device: set once on each device that launches.
template <class K> cudaError_t set_smem_once(K kern, size_t bytes, bool (&done)[64])
{
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    if (dev >= 0 && dev < 64 && done[dev]) return cudaSuccess;
    e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, int(bytes));
    if (e != cudaSuccess) return e;
    e = cudaFuncSetAttribute(kern, cudaFuncAttributePreferredSharedMemoryCarveout, 100);
    if (e != cudaSuccess) return e;
    if (dev >= 0 && dev < 64) done[dev] = true;
    return cudaSuccess;
}

template <class S, int N, int GAS, int RIEM, int GEO, int VAR, bool POST>
cudaError_t launch_line_v(const Fr2dArgs& a, cudaStream_t st)
{
    using T = Line2D<N, GEO, VAR, S>;
    auto kern = fr2d_line_kernel<S, N, GAS, RIEM, GEO, VAR, POST>;
    static bool done[64] = {};
    const cudaError_t e = set_smem_once(kern, T::bytes, done);
    if (e != cudaSuccess) return e;
    dim3 grid((a.Nx + T::TX - 1) / T::TX, (a.row_end - a.row_begin + T::TY - 1) / T::TY);
    kern<<<grid, T::BT, T::bytes, st>>>(a);
    return cudaGetLastError();
}

// The small variant as long as all of its CTAs are resident at once: then the launch lasts
// one tile's chain, which its face warps shorten (64^2 elements, affine / curved: p = 3 6.5 /
// 7.4 -> 4.7 / 5.2 us, p = 4 8.1 / 8.6 -> 6.1 / 7.2, p = 5 8.4 / 10.0 -> 7.4 / 8.6); beyond one
// residency the tuned tile does less halo work per element (96^2: p = 3 8.1 -> 7.4, p = 5
// 12.9 -> 10.5 us).  Curved meshes, small / tuned at 48^2, 96^2, 200^2: p = 3 0.74, 0.77, 1.16; p = 4
// 0.79, 1.00, 1.13; p = 6 0.84, 1.33, 1.42; p = 7 0.90, 1.28, 1.40; p = 8 1.06, 1.43, 1.46; p = 9 1.22,
// 1.35, 1.49 (one residency ends at 69^2 up to n = 6, at 49^2 above, where p = 9 is on the wrong side
// of it).  Curved p = 5, whose tuned tile fills few warps, takes the small variant at any size:
// 0.81, 0.85, 0.85, and 0.87 at 256^2.
template <class S, int N, int GAS, int RIEM, int GEO> cudaError_t launch_line(const Fr2dArgs& a, cudaStream_t st)
{
    using L = Line2D<N, GEO, 2, S>;
    const bool post = !L::F32 && a.mode == MODE_STAGE && a.post;
    auto launch = [&](auto var) -> cudaError_t {
        constexpr int VAR = decltype(var)::value;
        if constexpr (!L::F32)
            if (post) return launch_line_v<S, N, GAS, RIEM, GEO, VAR, true>(a, st);
        return launch_line_v<S, N, GAS, RIEM, GEO, VAR, false>(a, st);
    };
    if constexpr (GEO == GEO_CURVED && N == 6 && !L::F32) return launch(std::integral_constant<int, 2>{});
    else
    {
        const int64_t tiles = int64_t((a.Nx + L::TX - 1) / L::TX) * ((a.row_end - a.row_begin + L::TY - 1) / L::TY);
        if (tiles <= L::CTAS * kSMs) return launch(std::integral_constant<int, 2>{});
        return launch(std::integral_constant<int, 0>{});
    }
}

} // namespace frsdg
