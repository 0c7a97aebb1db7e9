// device_math.cuh -- scalar types of the residual kernels.
//
// The residual is templated on its scalar S:
//   double  the FP64 residual (rhs_func / fun_implicit),
//   cplx    complex FP64 for the complex-step JVP (matmult of the reference),
//   dual    complex FP64 to first order in the imaginary part, which takes the place of cplx
//           when h^2 is below rounding (csd_eps <= 1e-20);
//   float   the FP32 residual of the mixed-precision form.
// cplx follows std::complex<double> semantics for finite values: principal-branch
// sqrt, Smith's division (R. L. Smith, "Algorithm 116: Complex division",
// CACM 5(8), 1962) and the textbook product.
#pragma once
#include <cstdint>
#include <cuda_runtime.h>

namespace frsdg
{

struct __align__(16) cplx
{
    double re, im;
    __host__ __device__ constexpr cplx() : re(0.0), im(0.0) {}
    __host__ __device__ constexpr cplx(double r) : re(r), im(0.0) {}
    __host__ __device__ constexpr cplx(double r, double i) : re(r), im(i) {}
};

__device__ __forceinline__ cplx operator+(cplx a, cplx b) { return {a.re + b.re, a.im + b.im}; }
__device__ __forceinline__ cplx operator-(cplx a, cplx b) { return {a.re - b.re, a.im - b.im}; }
__device__ __forceinline__ cplx operator-(cplx a) { return {-a.re, -a.im}; }
__device__ __forceinline__ cplx operator*(cplx a, cplx b)
{
    return {a.re * b.re - a.im * b.im, a.re * b.im + a.im * b.re};
}
__device__ __forceinline__ cplx operator*(double s, cplx a) { return {s * a.re, s * a.im}; }
__device__ __forceinline__ cplx operator*(cplx a, double s) { return {a.re * s, a.im * s}; }
__device__ __forceinline__ cplx operator+(cplx a, double s) { return {a.re + s, a.im}; }
__device__ __forceinline__ cplx operator+(double s, cplx a) { return {s + a.re, a.im}; }
__device__ __forceinline__ cplx operator-(cplx a, double s) { return {a.re - s, a.im}; }
__device__ __forceinline__ cplx operator-(double s, cplx a) { return {s - a.re, -a.im}; }
__device__ __forceinline__ cplx operator/(cplx a, cplx b)
{
    // Smith's algorithm.
    if (fabs(b.re) >= fabs(b.im))
    {
        const double r   = b.im / b.re;
        const double den = b.re + b.im * r;
        return {(a.re + a.im * r) / den, (a.im - a.re * r) / den};
    }
    const double r   = b.re / b.im;
    const double den = b.re * r + b.im;
    return {(a.re * r + a.im) / den, (a.im * r - a.re) / den};
}
__device__ __forceinline__ cplx operator/(cplx a, double s) { return {a.re / s, a.im / s}; }
__device__ __forceinline__ cplx operator/(double s, cplx b) { return cplx(s) / b; }
__device__ __forceinline__ cplx& operator+=(cplx& a, cplx b) { a = a + b; return a; }
__device__ __forceinline__ cplx& operator-=(cplx& a, cplx b) { a = a - b; return a; }

// A complex number with an imaginary part of order h, |h| <= 1e-20 (the step is in im, as in
// cplx): the products' second-order terms, h^2 smaller than the first-order ones, are left
// out, and a quotient needs one reciprocal.  As in cplx the imaginary part decides where the
// real one is zero, and the root of a negative value stands in the imaginary part.  The real
// parts round as cplx's do (a product of two by itself, not fused with a sum beside it): where
// two wave speeds are equal but for rounding, smooth_abs divides that by its 1e-7, and other
// roundings give other derivatives (bump channel: a product's distance to a complex FP64
// restatement 1e-15 fused, 4e-16 so, in the same time).
struct __align__(16) dual
{
    double re, im;
    __host__ __device__ constexpr dual() : re(0.0), im(0.0) {}
    __host__ __device__ constexpr dual(double r) : re(r), im(0.0) {}
    __host__ __device__ constexpr dual(double r, double i) : re(r), im(i) {}
};
__device__ __forceinline__ dual operator+(dual a, dual b) { return {a.re + b.re, a.im + b.im}; }
__device__ __forceinline__ dual operator-(dual a, dual b) { return {a.re - b.re, a.im - b.im}; }
__device__ __forceinline__ dual operator-(dual a) { return {-a.re, -a.im}; }
__device__ __forceinline__ dual operator*(dual a, dual b) { return {__dmul_rn(a.re, b.re), fma(a.re, b.im, a.im * b.re)}; }
__device__ __forceinline__ dual operator*(double s, dual a) { return {s * a.re, s * a.im}; }
__device__ __forceinline__ dual operator*(dual a, double s) { return {a.re * s, a.im * s}; }
__device__ __forceinline__ dual operator+(dual a, double s) { return {a.re + s, a.im}; }
__device__ __forceinline__ dual operator+(double s, dual a) { return {s + a.re, a.im}; }
__device__ __forceinline__ dual operator-(dual a, double s) { return {a.re - s, a.im}; }
__device__ __forceinline__ dual operator-(double s, dual a) { return {s - a.re, -a.im}; }

// ---- generic scalar functions -------------------------------------------
// Exponent tests of the fast paths: |x| (or x, positive) in [2^-122, 2^123), well
// inside the range of normal floats, by the biased exponent with integer operations
// (zero, subnormals, inf and NaN fail them; so do negatives in the signed test).
__device__ __forceinline__ bool in_float_range(double x)
{
    const unsigned e = (static_cast<unsigned>(__double2hiint(x)) >> 20) & 0x7ffu;
    return e - (1023u - 122u) < 245u;
}
__device__ __forceinline__ bool positive_in_float_range(double x)
{
    return (static_cast<unsigned>(__double2hiint(x)) >> 20) - (1023u - 122u) < 245u;
}
// The IEEE operations for inputs outside that range, out of line so that the fast
// path does not carry them (measured on the 1024^2 p = 5 residual: 1.400 ms with the
// IEEE operations inline behind the branch, 1.366 ms out of line; selects instead of
// the branch, with exact power-of-two scaling of the outside inputs, 1.385 ms).
static __device__ __noinline__ double ieee_sqrt(double x) { return sqrt(x); }
static __device__ __noinline__ double ieee_rcp(double x) { return 1.0 / x; }

// sqrt in FP64 from the hardware's approximate FP64 reciprocal square root y
// (rsqrt.approx.f64 of the PTX ISA, the leading 32 bits): with g = x y ~ sqrt(x) and
// h = y / 2, one coupled Newton step r = 1/2 - g h, g <- g + g r, h <- h + h r, then a Heron
// correction g + (x - g^2) h (Markstein, IBM J. Res. Dev. 34(1), 1990): the seed's error is
// squared twice.  Inputs outside [2^-122, 2^123) (zero, negatives, subnormals, inf, NaN)
// take the IEEE square root.
__device__ __forceinline__ double sqrt_fast(double x)
{
    double y;
    asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(x));
    double g = x * y, h = 0.5 * y;
    const double r = fma(-g, h, 0.5);
    g = fma(g, r, g);
    h = fma(h, r, h);
    return fma(fma(-g, g, x), h, g);
}
// the same with h = 1 / (2 sqrt(x)) to full precision
__device__ __forceinline__ double sqrt_fast(double x, double& h_out)
{
    double y;
    asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(x));
    double g = x * y, h = 0.5 * y;
    const double r = fma(-g, h, 0.5);
    g = fma(g, r, g);
    h = fma(h, r, h);
    g = fma(fma(-g, g, x), h, g);
    h_out = fma(h, fma(-g, h, 0.5) * 2.0, h);
    return g;
}
__device__ __forceinline__ double s_sqrt(double x)
{
    if (!positive_in_float_range(x)) return ieee_sqrt(x);
    return sqrt_fast(x);
}
__device__ __forceinline__ float s_sqrt(float x) { return sqrtf(x); }
__device__ __forceinline__ cplx s_sqrt(cplx z)
{
    // principal branch, as C99 csqrt
    if (z.re == 0.0 && z.im == 0.0) return {0.0, z.im};
    const double t = sqrt(0.5 * (fabs(z.re) + hypot(z.re, z.im)));
    if (z.re >= 0.0) return {t, z.im / (2.0 * t)};
    return {fabs(z.im) / (2.0 * t), copysign(t, z.im)};
}
// Outside the fast range: the complex root, principal branch, to first order in the smaller part.
__device__ __forceinline__ dual s_sqrt(dual z)
{
    if (positive_in_float_range(z.re))
    {
        double h;
        const double g = sqrt_fast(z.re, h);
        return {g, z.im * h};
    }
    const double t = ieee_sqrt(z.re == 0.0 ? 0.5 * fabs(z.im) : fabs(z.re));
    if (t == 0.0) return {0.0, z.im};
    const double q = z.im / (2.0 * t);
    return z.re < 0.0 ? dual(fabs(q), copysign(t, z.im)) : dual(t, q);
}
__device__ __forceinline__ double s_log(double x) { return log(x); }
__device__ __forceinline__ cplx s_log(cplx z) { return {log(hypot(z.re, z.im)), atan2(z.im, z.re)}; }
__device__ __forceinline__ double s_exp(double x) { return exp(x); }
__device__ __forceinline__ dual s_exp(dual z)
{
    const double m = exp(z.re);
    return {m, m * z.im};
}
__device__ __forceinline__ float s_exp(float x) { return expf(x); }
__device__ __forceinline__ cplx s_exp(cplx z)
{
    const double m = exp(z.re);
    double       s, c;
    sincos(z.im, &s, &c);
    return {m * c, m * s};
}

// reciprocal: 1/x.  In FP64 the hardware's approximate FP64 reciprocal r (rcp.approx.f64 of
// the PTX ISA, the leading 32 bits) and one third-order step r + r (e + e^2), e = 1 - x r
// (the seed's error cubed; Markstein, IBM J. Res. Dev. 34(1), 1990).  Inputs outside
// [2^-122, 2^123) in magnitude take the IEEE division.
__device__ __forceinline__ double rcp_fast(double x)
{
    double r;
    asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(r) : "d"(x));
    const double e = fma(-x, r, 1.0);
    return fma(r, fma(e, e, e), r);
}
__device__ __forceinline__ double s_rcp(double x)
{
    if (!in_float_range(x)) return ieee_rcp(x);
    return rcp_fast(x);
}
__device__ __forceinline__ float s_rcp(float x) { return 1.0f / x; }
__device__ __forceinline__ cplx s_rcp(cplx z) { return cplx(1.0) / z; }
__device__ __forceinline__ dual s_rcp(dual z)
{
    if (in_float_range(z.re))
    {
        const double r = rcp_fast(z.re);
        return {r, -(z.im * r) * r};
    }
    const double r = ieee_rcp(z.re == 0.0 ? z.im : z.re);
    return z.re == 0.0 ? dual(0.0, -r) : dual(r, -(z.im * r) * r);
}

// wrap_positive (macro_and_libc.hpp:117-138): max(DBL_MIN, rho); for complex, the
// real part decides and a clamped value loses its imaginary part.
__device__ __forceinline__ double s_wrap_positive(double r)
{
    const double floor = 2.2250738585072014e-308; // DBL_MIN
    return fmax(floor, r);
}
__device__ __forceinline__ float s_wrap_positive(float r)
{
    const float floor = 1.17549435e-38f; // FLT_MIN
    return fmaxf(floor, r);
}
__device__ __forceinline__ cplx s_wrap_positive(cplx r)
{
    const double floor = 2.2250738585072014e-308;
    return (r.re < floor) ? cplx(floor, 0.0) : r;
}
__device__ __forceinline__ dual s_wrap_positive(dual r)
{
    const double floor = 2.2250738585072014e-308;
    return (r.re < floor) ? dual(floor, 0.0) : r;
}

// Math policies of the physics helpers.  MathChecked: s_rcp and s_sqrt.  MathDeferred:
// in FP64 the fast paths alone, each recording in `bad` whether its input lay outside
// their range; a computation that ends with bad == 0 equals its MathChecked twin bit for
// bit, and one that does not is redone with MathChecked.  A node or face computation
// then carries one branch instead of one per reciprocal and square root (measured on the
// 1024^2 p = 5 residual: the per-operation branches cost 8 %).  Other scalars take the
// checked functions (bad stays 0).
struct MathChecked
{
    template <class S> __device__ __forceinline__ S rcp(S x) const { return s_rcp(x); }
    template <class S> __device__ __forceinline__ S sqrt(S x) const { return s_sqrt(x); }
    template <class S> __device__ __forceinline__ S wrap(S x) const { return s_wrap_positive(x); }
};
struct MathDeferred
{
    unsigned& bad;
    // wrap_positive leaves normal positive finite values as they are; others are recorded
    __device__ __forceinline__ double wrap(double x) const
    {
        if (static_cast<unsigned>(__double2hiint(x)) - 0x00100000u >= 0x7fe00000u) bad = 1u;
        return x;
    }
    __device__ __forceinline__ float wrap(float x) const { return s_wrap_positive(x); }
    __device__ __forceinline__ cplx wrap(cplx x) const { return s_wrap_positive(x); }
    __device__ __forceinline__ dual wrap(dual x) const { return {wrap(x.re), x.im}; }
    __device__ __forceinline__ dual rcp(dual x) const
    {
        const double r = rcp(x.re);
        return {r, -(x.im * r) * r};
    }
    __device__ __forceinline__ dual sqrt(dual x) const
    {
        if (!positive_in_float_range(x.re)) bad = 1u;
        double h;
        const double t = sqrt_fast(x.re, h);
        return {t, x.im * h};
    }
    __device__ __forceinline__ double rcp(double x) const
    {
        if (!in_float_range(x)) bad = 1u;
        return rcp_fast(x);
    }
    __device__ __forceinline__ double sqrt(double x) const
    {
        if (!positive_in_float_range(x)) bad = 1u;
        return sqrt_fast(x);
    }
    // FP32: the hardware approximations with one Newton step for normal inputs whose results
    // stay normal (equal to the IEEE results on every mantissa, so a redo of nodes that need
    // none leaves their bits); zero, subnormals, huge values, inf and NaN (exponent tests as
    // above) take the redo with the IEEE operations
    __device__ __forceinline__ float rcp(float x) const
    {
        const unsigned e = (__float_as_uint(x) >> 23) & 0xffu;
        bad |= e - 2u < 250u ? 0u : 1u;  // 2^-125 <= |x| < 2^125
        float r;
        asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
        return fmaf(r, fmaf(-x, r, 1.0f), r);
    }
    __device__ __forceinline__ float sqrt(float x) const
    {
        // positive, 2^-100 <= x < 2^125 (below, the correction's x - s^2 is subnormal)
        bad |= (__float_as_uint(x) >> 23) - 27u < 225u ? 0u : 1u;
        float y;
        asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
        const float s = x * y;
        return fmaf(fmaf(-s, s, x), 0.5f * y, s);
    }
    __device__ __forceinline__ cplx rcp(cplx x) const { return s_rcp(x); }
    __device__ __forceinline__ cplx sqrt(cplx x) const { return s_sqrt(x); }
};

// real part, and the value the HLLC branch tests (riemann_solver.hpp:149-155:
// Re + Im for complex, the value itself for real scalars).
__device__ __forceinline__ double s_re(double x) { return x; }
__device__ __forceinline__ double s_re(float x) { return x; }
__device__ __forceinline__ double s_re(cplx z) { return z.re; }
__device__ __forceinline__ double s_im(cplx z) { return z.im; }
__device__ __forceinline__ double s_re(dual z) { return z.re; }
__device__ __forceinline__ double s_im(dual z) { return z.im; }
__device__ __forceinline__ double s_branch(dual z) { return z.re + z.im; }
__device__ __forceinline__ double s_branch(double x) { return x; }
__device__ __forceinline__ double s_branch(float x) { return x; }
__device__ __forceinline__ double s_branch(cplx z) { return z.re + z.im; }

template <class S> __device__ __forceinline__ S s_select(bool c, S a, S b) { return c ? a : b; }

// The health word's test of a density: positive and finite.  Positive finite doubles
// (subnormals included) are exactly the bit patterns 1 .. 0x7fefffffffffffff.
__device__ __forceinline__ bool density_ok(double rho)
{
    return static_cast<unsigned long long>(__double_as_longlong(rho)) - 1ull < 0x7fefffffffffffffull;
}

template <class S> struct scalar_traits;
template <> struct scalar_traits<double>
{
    using real = double;
    static constexpr int words = 1;
};
template <> struct scalar_traits<float>
{
    using real = float;
    static constexpr int words = 1;
};
template <> struct scalar_traits<dual>
{
    using real = double;
    static constexpr int words = 2;
};
template <> struct scalar_traits<cplx>
{
    using real = double;
    static constexpr int words = 2;
};

} // namespace frsdg
