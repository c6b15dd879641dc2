// mpcf_math.cuh -- device math of one cell face: WENO5 reconstruction with
// clipping, Einfeldt / Batten wave speeds and the HLLC fluxes of the
// 7-component stiffened-gas system, written for sm_100a.
//
// The arithmetic follows the reference device functions
//   WENO5-JS             source/GPU/GPUonly.cuh:99-194
//   Einfeldt, s*         source/GPU/GPUonly.cuh:802-866
//   HLLC fluxes          source/GPU/GPUonly.cuh:869-1026
//   extra-term velocity  source/GPU/GPUonly.cuh:1029-1042
// in the same evaluation order.  A precision policy selects the rounding:
//
//   PolRef32   float storage and arithmetic, the reference's double-promoted
//              sub-expressions kept in double, IEEE division and sqrt.  Its
//              translation unit is compiled with --fmad=false, so every
//              operation rounds exactly like the literal C semantics of the
//              reference source: results are bit-identical to the CPU
//              restatement built with -ffp-contract=off.
//   PolFast32  float everywhere; WENO smoothness indicators in factored
//              (cancellation-free, shared-curvature) form, weights from
//              single-precision reciprocals, fused multiply-adds allowed.
//   PolMixed   PolFast32 plus the stiffened-gas pressure recovery in
//              compensated FP32 (two-sum) and FP64 conservation sums.
//   PolFP64    double storage and arithmetic (the all-FP64 GPU oracle run).
//   PolFast64  double storage and arithmetic with the fast forms' algebra
//              (factored indicators and fluxes, refined double reciprocals):
//              the tuned FP64 yardstick of the mixed form.
//   PolRef32W3, PolFP64W3  the two reference-rounding forms with the
//              reference's compile-time WENO3 reconstruction.
//
// Primitive index convention used throughout the device code:
//   0 rho, 1 u, 2 v, 3 w, 4 p, 5 G = 1/(gamma-1), 6 P = gamma*pc/(gamma-1)
// Face outputs: 0..6 fluxes of (rho, rho u, rho v, rho w, E, G, P),
//   7 u* (extra-term velocity).
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

namespace mpcf {

#ifndef MPCF_WENOEPS
#define MPCF_WENOEPS 1e-6   // Makefile.config:15 (weps ?= 1e-6)
#endif

struct PolRef32  { typedef float  T; static constexpr bool kFastWeno = false; static constexpr bool kCompP = false; static constexpr bool kRefRounding = true;  static constexpr bool kWeno3 = false; static constexpr int id = 0; };
struct PolFast32 { typedef float  T; static constexpr bool kFastWeno = true;  static constexpr bool kCompP = false; static constexpr bool kRefRounding = false; static constexpr bool kWeno3 = false; static constexpr int id = 1; };
struct PolMixed  { typedef float  T; static constexpr bool kFastWeno = true;  static constexpr bool kCompP = true;  static constexpr bool kRefRounding = false; static constexpr bool kWeno3 = false; static constexpr int id = 2; };
struct PolFP64   { typedef double T; static constexpr bool kFastWeno = false; static constexpr bool kCompP = false; static constexpr bool kRefRounding = true;  static constexpr bool kWeno3 = false; static constexpr int id = 3; };
struct PolFast64 { typedef double T; static constexpr bool kFastWeno = true;  static constexpr bool kCompP = false; static constexpr bool kRefRounding = false; static constexpr bool kWeno3 = false; static constexpr int id = 4; };
// The reference's compile-time WENO3 build (-D_WENO3_, GPUonly.cuh:102,141)
// of the two reference-rounding forms.
struct PolRef32W3 { typedef float  T; static constexpr bool kFastWeno = false; static constexpr bool kCompP = false; static constexpr bool kRefRounding = true; static constexpr bool kWeno3 = true; static constexpr int id = 0; };
struct PolFP64W3  { typedef double T; static constexpr bool kFastWeno = false; static constexpr bool kCompP = false; static constexpr bool kRefRounding = true; static constexpr bool kWeno3 = true; static constexpr int id = 3; };

__device__ __forceinline__ float  dmin(float a, float b)   { return fminf(a, b); }
__device__ __forceinline__ float  dmax(float a, float b)   { return fmaxf(a, b); }
__device__ __forceinline__ double dmin(double a, double b) { return fmin(a, b); }
__device__ __forceinline__ double dmax(double a, double b) { return fmax(a, b); }
__device__ __forceinline__ float  dsqrt(float a)  { return sqrtf(a); }
__device__ __forceinline__ double dsqrt(double a) { return sqrt(a); }

// Approximate reciprocal of the special-function unit (relative error below
// 2^-22); only the fast policies use it.
__device__ __forceinline__ float rcp_approx(float x)
{
    float r;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
    return r;
}
// Reciprocal in double precision without a division: the special-function
// unit's approximate reciprocal refined by two Newton-Raphson steps
// y <- y + y (1 - x y) (each step doubles the number of correct bits).
__device__ __forceinline__ double rcp_f64(const double x)
{
    double y;
    asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(x));
    double e = fma(-x, y, 1.0);
    y = fma(y, e, y);
    e = fma(-x, y, 1.0);
    return fma(y, e, y);
}
// the fast FP64 form's reciprocal
__device__ __forceinline__ double rcp_approx(double x) { return rcp_f64(x); }

// Approximate square root of the special-function unit (fast policies).
__device__ __forceinline__ float sqrt_approx(float x)
{
    float r;
    asm("sqrt.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
    return r;
}

// ---------------------------------------------------------------------------
// WENO5 smoothness indicators.  For a window of three consecutive cells
// (x, y, z) left to right, the reference uses three polynomial forms:
//   beta_f(x,y,z) = x(4/3 x - 19/3 y + 11/3 z) + y(25/3 y - 31/3 z) + 10/3 z^2
//   beta_h(x,y,z) = x(4/3 x - 13/3 y +  5/3 z) + y(13/3 y - 13/3 z) +  4/3 z^2
//   beta_g(x,y,z) = x(10/3 x - 31/3 y + 11/3 z) + y(25/3 y - 19/3 z) + 4/3 z^2
// minus side (a..e): is0 = f(a,b,c), is1 = h(b,c,d), is2 = g(c,d,e)
// plus side  (b..f): is0 = g(d,e,f), is1 = h(c,d,e), is2 = f(b,c,d)
// (GPUonly.cuh:102-104 and :141-143, same operation order).
// ---------------------------------------------------------------------------
template <class T> __device__ __forceinline__ T beta_f(const T x, const T y, const T z)
{
    return x*(x*(T)(4./3.)  - y*(T)(19./3.) + z*(T)(11./3.)) + y*(y*(T)(25./3.) - z*(T)(31./3.)) + z*z*(T)(10./3.);
}
template <class T> __device__ __forceinline__ T beta_h(const T x, const T y, const T z)
{
    return x*(x*(T)(4./3.)  - y*(T)(13./3.) + z*(T)(5./3.))  + y*(y*(T)(13./3.) - z*(T)(13./3.)) + z*z*(T)(4./3.);
}
template <class T> __device__ __forceinline__ T beta_g(const T x, const T y, const T z)
{
    return x*(x*(T)(10./3.) - y*(T)(31./3.) + z*(T)(11./3.)) + y*(y*(T)(25./3.) - z*(T)(19./3.)) + z*z*(T)(4./3.);
}

// Correctly rounded reciprocal without a branch, for arguments whose
// reciprocal is far from under- and overflow: Newton-Raphson from the
// special-function unit's approximation, the last step on the exact residual
// 1 - x y of an approximation y within one unit in the last place, which
// rounds correctly unless x's mantissa is all ones (Markstein, "Computation
// of elementary functions on the IBM RISC System/6000 processor", 1990; there
// it is at most one unit off, and equal to division on 1.3e7 indicators, sums
// of weights and edges of the mantissa).  Other
// arguments (0, subnormal, huge, infinite, NaN) give a NaN or a wrong value:
// the caller checks.
__device__ __forceinline__ double rcp_rn(const double x)
{
    double y;
    asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(x));
    const double e = __fma_rn(-x, y, 1.0);
    y = __fma_rn(y, __fma_rn(e, e, e), y);      // y (1 + e + e^2): 3 times the correct bits
    return __fma_rn(y, __fma_rn(-x, y, 1.0), y);
}

// Whether a positive x (or a NaN, which is not) lies in [lo, hi), powers of
// two: an integer comparison of the exponents, off the FP64 pipe.
__device__ __forceinline__ bool in_range(const double x, const double lo, const double hi)
{
    return (unsigned)(__double2hiint(x) - __double2hiint(lo)) < (unsigned)(__double2hiint(hi) - __double2hiint(lo));
}

// Both edge values of one cell in the reference-rounding policies, from the
// cells y0..y4 = l-2..l+2 (GPUonly.cuh:99-194):
//   R, the minus side of face l+1/2: indicators (is0, is1, is2) =
//     (beta_f(y0,y1,y2), beta_h(y1,y2,y3), beta_g(y2,y3,y4)), candidates
//     from y0..y4, clipped to [min, max] of y1, y2, y3;
//   L, the plus side of face l-1/2: indicators (beta_g(y2,y3,y4),
//     beta_h(y1,y2,y3), beta_f(y0,y1,y2)), the mirrored candidates, the same
//     clip;
//   weights alpha_j = c_j * (1/(10.0*(is_j+eps)^2)) with c = (1, 6, 3) (the
//   10.0 literal promotes the reciprocal to double, GPUonly.cuh:111-113),
//   w0 = alpha0/sum, w1 = alpha1/sum, w2 = 1 - w0 - w1.
// The reference evaluates each face's two sides separately; the three
// indicator calls, their double reciprocals and the clip bounds of the two
// edges of a cell are the same operations on the same values, so they are
// evaluated once here.  Every other operation is the reference's in its
// order, so R and L are bit-identical to its per-face results.
//
// kBranchFree: the reciprocals through rcp_rn; returns whether both sums of
// weights lie where those are exact (false also when a sum is NaN, which a
// zero or infinite pf, ph or pg leads to).  The compiler's own division
// carries a branch to its slow path for each of the five reciprocals, which
// cuts the code of a cell's 7 quantities into pieces too short to overlap.
template <class Pol, bool kBranchFree>
__device__ __forceinline__ bool weno_cell_ref(const typename Pol::T y0, const typename Pol::T y1,
        const typename Pol::T y2, const typename Pol::T y3, const typename Pol::T y4,
        typename Pol::T& R, typename Pol::T& L)
{
    typedef typename Pol::T T;
    static_assert(!Pol::kFastWeno, "reference-rounding policies only");
    const T pf = beta_f<T>(y0, y1, y2) + (T)MPCF_WENOEPS;
    const T ph = beta_h<T>(y1, y2, y3) + (T)MPCF_WENOEPS;
    const T pg = beta_g<T>(y2, y3, y4) + (T)MPCF_WENOEPS;
    // the 10.0 literal promotes these to double (GPUonly.cuh:111-113)
    const double xf = 10.0*pf*pf, xh = 10.0*ph*ph, xg = 10.0*pg*pg;
    const double qf = kBranchFree ? rcp_rn(xf) : ((T)1)/xf;
    const double qh = kBranchFree ? rcp_rn(xh) : ((T)1)/xh;
    const double qg = kBranchFree ? rcp_rn(xg) : ((T)1)/xg;
    const T a1 = (T)((T)(6)*qh);
    const T lo = dmin(dmin(y1, y2), y3);
    const T hi = dmax(dmax(y1, y2), y3);
    bool exact = true;
    static_assert(!kBranchFree || sizeof(T) == 8, "branch-free: FP64 only");
    const double kLo = 0x1p-900, kHi = 0x1p900;
    {
        // minus side: indicators (f, h, g)
        const T a0 = (T)((T)(1)*qf), a2 = (T)((T)(3)*qg);
        const T sum = a0 + a1 + a2;
        T inv;
        if constexpr (kBranchFree) { exact = sum >= kLo && sum <= kHi; inv = rcp_rn(sum); }
        else                       inv = ((T)1)/sum;
        const T w0 = a0 * inv, w1 = a1 * inv, w2 = 1 - w0 - w1;
        const T r = w0*((T)(1.0/3.)*y0-(T)(7./6.)*y1+(T)(11./6.)*y2) + w1*(-(T)(1./6.)*y1+(T)(5./6.)*y2+(T)(1./3.)*y3) + w2*((T)(1./3.)*y2+(T)(5./6.)*y3-(T)(1./6.)*y4);
        R = dmin(dmax(r, lo), hi);
    }
    {
        // plus side: indicators (g, h, f)
        const T a0 = (T)((T)(1)*qg), a2 = (T)((T)(3)*qf);
        const T sum = a0 + a1 + a2;
        T inv;
        if constexpr (kBranchFree) { exact = exact && sum >= kLo && sum <= kHi; inv = rcp_rn(sum); }
        else                       inv = ((T)1)/sum;
        const T w0 = a0 * inv, w1 = a1 * inv, w2 = 1 - w0 - w1;
        const T r = w0*((T)(1./3.)*y4-(T)(7./6.)*y3+(T)(11./6.)*y2) + w1*(-(T)(1./6.)*y3+(T)(5./6.)*y2+(T)(1./3.)*y1) + w2*((T)(1./3.)*y2+(T)(5./6.)*y1-(T)(1./6.)*y0);
        L = dmin(dmax(r, lo), hi);
    }
    return exact;
}

// ---------------------------------------------------------------------------
// Explicitly rounded operations on one value (float, double) or on a pair of
// floats.  sm_100 executes fma / add / mul on two FP32 lanes in one
// instruction, each lane rounded like the scalar instruction; the face
// pipeline is bound by instruction issue, so the fast FP32 forms reconstruct
// two quantities at a time.  No operation here may be contracted with
// another, and no sum below takes a product that a code generator could fuse:
// an edge value is the same bits whether a pair, a single value, an interior
// cell or a ghost cell produced it.
// ---------------------------------------------------------------------------
__device__ __forceinline__ float  add_(const float a, const float b)   { return __fadd_rn(a, b); }
__device__ __forceinline__ float  sub_(const float a, const float b)   { return __fsub_rn(a, b); }
__device__ __forceinline__ float  mul_(const float a, const float b)   { return __fmul_rn(a, b); }
__device__ __forceinline__ float  fma_(const float a, const float b, const float c)    { return __fmaf_rn(a, b, c); }
__device__ __forceinline__ double add_(const double a, const double b) { return __dadd_rn(a, b); }
__device__ __forceinline__ double sub_(const double a, const double b) { return __dsub_rn(a, b); }
__device__ __forceinline__ double mul_(const double a, const double b) { return __dmul_rn(a, b); }
__device__ __forceinline__ double fma_(const double a, const double b, const double c) { return __fma_rn(a, b, c); }
__device__ __forceinline__ float2 add_(const float2 a, const float2 b) { return __fadd2_rn(a, b); }
__device__ __forceinline__ float2 mul_(const float2 a, const float2 b) { return __fmul2_rn(a, b); }
__device__ __forceinline__ float2 fma_(const float2 a, const float2 b, const float2 c) { return __ffma2_rn(a, b, c); }
// a - b as one packed instruction (b * -1 is exact)
__device__ __forceinline__ float2 sub_(const float2 a, const float2 b) { return __ffma2_rn(b, make_float2(-1.0f, -1.0f), a); }
__device__ __forceinline__ float2 rcp_approx(const float2 a) { return make_float2(rcp_approx(a.x), rcp_approx(a.y)); }
// a * b as one instruction per lane
__device__ __forceinline__ float  mul1_(const float a, const float b)   { return __fmul_rn(a, b); }
__device__ __forceinline__ double mul1_(const double a, const double b) { return __dmul_rn(a, b); }
__device__ __forceinline__ float2 mul1_(const float2 a, const float2 b) { return make_float2(__fmul_rn(a.x, b.x), __fmul_rn(a.y, b.y)); }
__device__ __forceinline__ float2 dsqrt(const float2 a) { return make_float2(dsqrt(a.x), dsqrt(a.y)); }
__device__ __forceinline__ float2 dmin(const float2 a, const float2 b) { return make_float2(dmin(a.x, b.x), dmin(a.y, b.y)); }
__device__ __forceinline__ float2 dmax(const float2 a, const float2 b) { return make_float2(dmax(a.x, b.x), dmax(a.y, b.y)); }
// conditions of one value or of both lanes, and selection by them
struct Bool2 { bool x, y; };
template <class T> __device__ __forceinline__ bool not_negative(const T a) { return !(a < (T)0); }
template <class T> __device__ __forceinline__ bool is_zero(const T a) { return a == (T)0; }
template <class T> __device__ __forceinline__ T pick(const bool c, const T a, const T b) { return c ? a : b; }
__device__ __forceinline__ Bool2 not_negative(const float2 a) { return Bool2{!(a.x < 0.0f), !(a.y < 0.0f)}; }
__device__ __forceinline__ Bool2 is_zero(const float2 a) { return Bool2{a.x == 0.0f, a.y == 0.0f}; }
__device__ __forceinline__ float2 pick(const Bool2 c, const float2 a, const float2 b) { return make_float2(c.x ? a.x : b.x, c.y ? a.y : b.y); }
// the constant c in every lane
template <class V> __device__ __forceinline__ V splat(const double c);
template <> __device__ __forceinline__ float  splat<float>(const double c)  { return (float)c; }
template <> __device__ __forceinline__ double splat<double>(const double c) { return c; }
template <> __device__ __forceinline__ float2 splat<float2>(const double c) { return make_float2((float)c, (float)c); }

// Minimum / maximum of three values in one operation (sm_100).
__device__ __forceinline__ float min3f(const float a, const float b, const float c)
{
    float r;
    asm("min.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(a), "f"(b), "f"(c));
    return r;
}
__device__ __forceinline__ float max3f(const float a, const float b, const float c)
{
    float r;
    asm("max.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(a), "f"(b), "f"(c));
    return r;
}
__device__ __forceinline__ double min3f(const double a, const double b, const double c) { return fmin(fmin(a, b), c); }
__device__ __forceinline__ double max3f(const double a, const double b, const double c) { return fmax(fmax(a, b), c); }

// v clipped to [min, max] of three neighbours
template <class T> __device__ __forceinline__ T clip3(const T v, const T a, const T b, const T c)
{
    return dmin(dmax(v, min3f(a, b, c)), max3f(a, b, c));
}
__device__ __forceinline__ float2 clip3(const float2 v, const float2 a, const float2 b, const float2 c)
{
    return make_float2(clip3(v.x, a.x, b.x, c.x), clip3(v.y, a.y, b.y, c.y));
}

// Edge values of one cell (fast policies), from the cell and its two
// neighbours on either side, y0..y4 = cells l-2..l+2:
//   R = value at the right edge l+1/2 (minus side of that face),
//   L = value at the left edge l-1/2 (plus side of that face; kBoth only).
// The Jiang-Shu smoothness indicators of the three sub-stencils
// (l-2..l, l-1..l+1, l..l+2) integrate over cell l, so they are the same for
// both edges (GPUonly.cuh:99-194 evaluates them again for every face): with
// the differences d_i = y_{i+1} - y_i,
//   k_j = d_{j+1} - d_j,  a_0 = k0 + 2 d1,  a_1 = d1 + d2,  a_2 = k2 - 2 d2,
//   J_j = 13/3 k_j^2 + a_j^2 + 4 eps,  g_j = 1/J_j^2
// (the indicators times 12/3, a common factor that cancels), the two edges
// weigh them with mirrored linear weights d = (1, 6, 3):
//   R = y2 + d2/2 - k1/6 + (g0 (k0-k1)/3 + g2 (k1-k2)/2) / (g0 + 6 g1 + 3 g2)
//   L = y2 - d1/2 - k1/6 - (g2 (k1-k2)/3 + g0 (k0-k1)/2) / (3 g0 + 6 g1 + g2)
// and both are clipped to [min, max] of y1, y2, y3.  Reversing y0..y4 turns R
// into L bit for bit (every operation has its mirror image), so a ghost cell
// whose left edge is wanted is reconstructed as the right edge of its
// mirrored stencil.  In double (kShared) the weights are multiplied through
// by J0^2 J1^2 J2^2 and the two sums share one reciprocal: one reciprocal
// with its four Newton operations instead of five.  That holds up to
// differences of about 1e18; beyond (the product of the sums out of range)
// the result is false and the caller takes the form with five.
template <bool kBoth, bool kShared, class V>
__device__ __forceinline__ bool weno_edges(const V y0, const V y1, const V y2, const V y3, const V y4, V& R, V& L)
{
    const V d0 = sub_(y1, y0), d1 = sub_(y2, y1), d2 = sub_(y3, y2), d3 = sub_(y4, y3);
    const V k0 = sub_(d1, d0), k1 = sub_(d2, d1), k2 = sub_(d3, d2);
    const V a0 = fma_(d1, splat<V>(2), k0), a1 = add_(d1, d2), a2 = fma_(d2, splat<V>(-2), k2);
    const V c13 = splat<V>(13. / 3.), e4 = splat<V>(4. * MPCF_WENOEPS);
    const V J0 = fma_(mul_(k0, c13), k0, fma_(a0, a0, e4));
    const V J1 = fma_(mul_(k1, c13), k1, fma_(a1, a1, e4));
    const V J2 = fma_(mul_(k2, c13), k2, fma_(a2, a2, e4));
    V g0, g1, g2;
    if constexpr (kShared)
    {
        const V p12 = mul_(J1, J2), p02 = mul_(J0, J2), p01 = mul_(J0, J1);
        g0 = mul_(p12, p12); g1 = mul_(p02, p02); g2 = mul_(p01, p01);
    }
    else
    {
        g0 = rcp_approx(mul_(J0, J0)); g1 = rcp_approx(mul_(J1, J1)); g2 = rcp_approx(mul_(J2, J2));
    }
    const V E0 = mul_(g0, sub_(k0, k1)), E2 = mul_(g2, sub_(k1, k2));
    const V denR = fma_(g2, splat<V>(3), fma_(g1, splat<V>(6), g0));
    const V numR = fma_(E0, splat<V>(1. / 3.), mul_(E2, splat<V>(0.5)));
    const V b = fma_(k1, splat<V>(-1. / 6.), y2);
    const V pR = fma_(d2, splat<V>(0.5), b);
    if constexpr (kShared)
    {
        const V denL = fma_(g0, splat<V>(3), fma_(g1, splat<V>(6), g2));
        const V den = mul_(denR, denL), inv = rcp_approx(den);
        R = clip3(fma_(mul_(numR, denL), inv, pR), y1, y2, y3);
        if constexpr (kBoth)
        {
            const V numL = fma_(E2, splat<V>(-1. / 3.), mul_(E0, splat<V>(-0.5)));
            L = clip3(fma_(mul_(numL, denR), inv, fma_(d1, splat<V>(-0.5), b)), y1, y2, y3);
        }
        return in_range(den, 0x1p-960, 0x1p960);
    }
    else
    {
        R = clip3(fma_(numR, rcp_approx(denR), pR), y1, y2, y3);
        if constexpr (kBoth)
        {
            const V denL = fma_(g0, splat<V>(3), fma_(g1, splat<V>(6), g2));
            const V numL = fma_(E2, splat<V>(-1. / 3.), mul_(E0, splat<V>(-0.5)));
            L = clip3(fma_(numL, rcp_approx(denL), fma_(d1, splat<V>(-0.5), b)), y1, y2, y3);
        }
        return true;
    }
}

// ---------------------------------------------------------------------------
// HLLC pieces.  sign_star in {-1,0,1}; the two weights (1+s)/2 and (1-s)/2.
// ---------------------------------------------------------------------------
__device__ __forceinline__ int sign_star_of(const float ss)  { return ss == 0 ? 0 : (ss < 0 ? -1 : 1); }
__device__ __forceinline__ int sign_star_of(const double ss) { return ss == 0 ? 0 : (ss < 0 ? -1 : 1); }

// (0.5f*(1+s))*L + (0.5*(1-s))*R.  In the FP32 reference the second weight
// of _hllc_rho is a double literal (GPUonly.cuh:900), which promotes that
// sum to double; kept exactly under the reference rounding policy.
template <class Pol, bool kDoubleSecondWeight>
__device__ __forceinline__ typename Pol::T hllc_blend(const int s, const typename Pol::T L, const typename Pol::T R)
{
    typedef typename Pol::T T;
    if (kDoubleSecondWeight && Pol::kRefRounding)
        return (T)((double)((0.5f*(1 + s)) * L) + (0.5*(1 - s)) * (double)R);
    else
        return (T)(0.5f*(1 + s)) * L + (T)(0.5f*(1 - s)) * R;
}

// What one face gives its two cells: the fluxes of rho, rho u, rho v, rho w,
// E, G, P and, last, the extra-term velocity.
constexpr int kFaceOut = 8;

// The face state after reconstruction: m = left (minus), p = right (plus).
// n = normal velocity, t1/t2 = the transverse velocities in the order the
// reference passes them to _hllc_e (x: v,w; y: u,w; z: u,v).
template <class T>
struct FaceState
{
    T rm, rp, nm, np, t1m, t1p, t2m, t2p, pm, pp, Gm, Gp, Pm, Pp;
};

// Wave speeds + HLLC fluxes of one face (GPUkernels.cu:255-289 for x,
// :636-668 for y, :932-963 for z; GPUonly.cuh:802-1042).  `dir` is a runtime
// value: the normal / transverse momenta are scattered with selects, so one
// instance of this code serves all three directions (the face pipeline is
// ~1000 instructions; one copy keeps it resident in the instruction cache).
template <class Pol>
__device__ __forceinline__ void hllc_face(const FaceState<typename Pol::T>& S, const int dir, typename Pol::T o[kFaceOut])
{
    typedef typename Pol::T T;
    const T rm = S.rm, rp = S.rp, um = S.nm, up = S.np;
    const T pm = S.pm, pp = S.pp, Gm = S.Gm, Gp = S.Gp, Pm = S.Pm, Pp = S.Pp;

    // Einfeldt bounds (GPUonly.cuh:802-847)
    const T Rr   = dsqrt(rp / rm);
    const T Rinv = (T)1.0f / ((T)1.0f + Rr);
    const T cm2 = ((pm + Pm)/Gm + pm) / rm;
    const T cp2 = ((pp + Pp)/Gp + pp) / rp;
    const T cm  = dsqrt(cm2);
    const T cp  = dsqrt(cp2);
    const T eta_2 = (T)0.5f*Rr*Rinv*Rinv;
    const T d2    = (cm2 + Rr*cp2)*Rinv + eta_2*(up - um)*(up - um);
    const T d     = dsqrt(d2);
    const T uu    = (um + Rr*up)*Rinv;
    const T sm = dmin(uu - d, um - cm);
    const T sp = dmax(uu + d, up + cp);

    // Batten star speed (GPUonly.cuh:857-866)
    const T facm = rm * (sm - um);
    const T facp = rp * (sp - up);
    const T ss = (pp - pm + um*facm - up*facp) / (facm - facp);

    const int s = sign_star_of(ss);
    // The blend (1+s)/2 L + (1-s)/2 R of a flux's two sides is 1*L + 0*R or
    // 0*L + 1*R unless s* is exactly 0, so only the upwind side is evaluated
    // (one pass, weight 1: the same value); at s = 0 a second pass evaluates
    // the other side and both are blended as the reference does.  The other
    // side's transverse velocities still enter as 0*t: a NaN or an infinity
    // there reaches the fluxes as it does in the reference's sum (any other
    // non-finite quantity makes s*, and with it everything, NaN).
    // The signs of zeros follow: for s* > 0 the other side's flux has the sign
    // of its quantity and is +0 where that is a zero of either sign, so a -0
    // of this side stays -0 only beside a negative transverse velocity
    // (z, +0 for t = -0) and becomes +0 in the others (the + z0 below, in the
    // exactly rounding FP32 forms); for s* < 0 this side's zeros are +0.
    const T z0 = (T)0;
    const T o1 = s < 0 ? S.t1m : S.t1p, o2 = s < 0 ? S.t2m : S.t2p;
    const T z1 = (T)0 * (sizeof(T) == 4 ? o1 + z0 : o1), z2 = (T)0 * (sizeof(T) == 4 ? o2 + z0 : o2);
#pragma unroll 1
    for (int side = s < 0 ? 1 : 0; ; side = 1)
    {
        const bool left = side == 0;
        const T r = left ? rm : rp, u = left ? um : up, p = left ? pm : pp;
        const T G = left ? Gm : Gp, P = left ? Pm : Pp;
        const T t1 = left ? S.t1m : S.t1p, t2 = left ? S.t2m : S.t2p;
        const T sk = left ? sm : sp;
        const T sc = left ? dmin((T)0.0f, sm) : dmax((T)0.0f, sp);
        const T du = sk - u;
        // every flux of this face divides by the same denominator with the
        // same normal velocity, so chi* is shared (identical operations)
        const T chi = du / (sk - ss);
        T f[kFaceOut];
        // rho, G, P (passive): _hllc_rho (GPUonly.cuh:869-903)
        const T q0 = r*u;
        f[0] = q0 + sc*(r*chi - r);
        f[5] = G*u + sc*(G*chi - G);
        f[6] = P*u + sc*(P*chi - P);
        // normal momentum: _hllc_pvel (GPUonly.cuh:947-984)
        const T fn = (q0*u + p) + sc*(r*ss*chi - q0);
        // transverse momenta: _hllc_vel (GPUonly.cuh:906-944)
        const T q1 = r*t1, q2 = r*t2;
        const T ft1 = q1*u + sc*(q1*chi - q1);
        const T ft2 = q2*u + sc*(q2*chi - q2);
        // energy: _hllc_e (GPUonly.cuh:987-1026)
        {
            const T q = G*p + P + (T)0.5f*r*(u*u + t1*t1 + t2*t2);
            f[4] = u*(q + p) + sc*(chi*(q + (ss - u)*(r*ss + p/du)) - q);
        }
        // extra-term velocity: _extraterm_hllc_vel (GPUonly.cuh:1029-1042)
        f[7] = u + sc*(chi - (T)1.0f);
        // normal / transverse momenta back to (rho u, rho v, rho w):
        // x: (n, t1, t2), y: (t1, n, t2), z: (t1, t2, n)
        f[1] = dir == 0 ? fn : ft1;
        f[2] = dir == 1 ? fn : (dir == 0 ? ft1 : ft2);
        f[3] = dir == 2 ? fn : ft2;
        if (s != 0)
        {
#pragma unroll
            for (int m = 0; m < kFaceOut; ++m) o[m] = f[m];
            if constexpr (sizeof(T) == 4)
            {
                o[0] = o[0] + z0; o[5] = o[5] + z0; o[6] = o[6] + z0; o[7] = o[7] + z0;
            }
            o[1] = o[1] + (dir == 0 ? (T)0 : z1);
            o[2] = o[2] + (dir == 1 ? (T)0 : (dir == 0 ? z1 : z2));
            o[3] = o[3] + (dir == 2 ? (T)0 : z2);
            o[4] = o[4] + (z1 + z2);
            return;
        }
        if (side)
        {
#pragma unroll
            for (int m = 0; m < kFaceOut; ++m)
                o[m] = (m == 0 || m == 5 || m == 6) ? hllc_blend<Pol, true>(0, o[m], f[m]) : hllc_blend<Pol, false>(0, o[m], f[m]);
            return;
        }
#pragma unroll
        for (int m = 0; m < kFaceOut; ++m) o[m] = f[m];
    }
}

// The same face in the fast policies.  The wave speeds follow hllc_face above
// term by term with approximate reciprocals.  The flux is then evaluated for
// the upwind side alone (the sign of s* picks the side; at s* = 0 the two
// sides' star fluxes agree), in the star state's own form: with
// chi = (S - u)/(S - s*), S_ = min(0, S_left) or max(0, S_right) and
//   w = s* chi  (S_ != 0: inside the fan)  or  u  (S_ = 0: supersonic)
// the reference's F + S_ (U* - U) is
//   X w for the advected quantities X, w itself for the extra-term velocity,
//   rho (w u + (s* - u) S_ chi) + p          for the normal momentum,
//   w (E + p + rho (s* - u) S_)              for the energy.
// It needs half the operations of the two-sided blend, no division by S - u,
// and is exactly 0 for the advected quantities when s* = 0.
// V is one face, or a pair of faces (the y and x faces of a cell, each in its
// own normal / transverse components).  Products that a sum follows directly
// are formed lane by lane (mul1_): a packed product before a packed sum may
// be contracted, and every face must come out the same from either form.
template <class V> struct FaceFlux { V r, n, t1, t2, e, G, P, w; };

template <class V>
__device__ __forceinline__ void hllc_face_upwind(const FaceState<V>& S, FaceFlux<V>& o)
{
    const V um = S.nm, up = S.np;
    // Einfeldt bounds
    const V irm = rcp_approx(S.rm), irp = rcp_approx(S.rp);
    const V cm2 = mul_(fma_(add_(S.pm, S.Pm), rcp_approx(S.Gm), S.pm), irm);
    const V cp2 = mul_(fma_(add_(S.pp, S.Pp), rcp_approx(S.Gp), S.pp), irp);
    const V cm = dsqrt(cm2), cp = dsqrt(cp2);
    const V Rr   = dsqrt(mul_(S.rp, irm));
    const V Rinv = rcp_approx(add_(splat<V>(1), Rr));
    const V eta  = mul_(mul_(mul_(splat<V>(0.5), Rr), Rinv), Rinv);
    const V du   = sub_(up, um);
    const V d    = dsqrt(fma_(mul_(eta, du), du, mul_(fma_(Rr, cp2, cm2), Rinv)));
    const V uu   = mul1_(fma_(Rr, up, um), Rinv);
    const V sm = dmin(sub_(uu, d), sub_(um, cm));
    const V sp = dmax(add_(uu, d), add_(up, cp));

    // Batten star speed (numerator and denominator with their signs changed)
    const V um_s = sub_(um, sm), sp_u = sub_(sp, up);
    const V fm = mul_(S.rm, um_s);
    const V num = fma_(up, mul_(S.rp, sp_u), fma_(um, fm, sub_(S.pm, S.pp)));
    const V ss = mul1_(num, rcp_approx(fma_(S.rp, sp_u, fm)));

    // the upwind side (left for s* >= 0, and for NaN, which then propagates)
    const auto left = not_negative(ss);
    const V r = pick(left, S.rm, S.rp), u = pick(left, um, up), p = pick(left, S.pm, S.pp);
    const V t1 = pick(left, S.t1m, S.t1p), t2 = pick(left, S.t2m, S.t2p);
    const V G = pick(left, S.Gm, S.Gp), P = pick(left, S.Pm, S.Pp);
    const V s  = pick(left, sm, sp);
    const V sc = pick(left, dmin(splat<V>(0), sm), dmax(splat<V>(0), sp));

    const V chi = mul_(sub_(s, u), rcp_approx(sub_(s, ss)));
    const V X   = mul_(sub_(ss, u), sc);
    // (X = 0: S_ = 0, or s* = u and so chi = 1; a NaN s* is in X and in w)
    const V w   = pick(is_zero(X), u, mul_(ss, chi));
    const V ke  = fma_(t2, t2, fma_(t1, t1, mul_(u, u)));
    const V E   = fma_(mul_(splat<V>(0.5), r), ke, fma_(G, p, P));
    o.r  = mul_(r, w);
    o.n  = fma_(mul_(r, X), chi, fma_(o.r, u, p));
    o.t1 = mul_(t1, o.r);
    o.t2 = mul_(t2, o.r);
    o.e  = mul_(w, fma_(r, X, add_(E, p)));
    o.G  = mul_(G, w);
    o.P  = mul_(P, w);
    o.w  = w;
}

// Both edge values of one cell with the reference's WENO3 reconstruction
// (the -D_WENO3_ build, GPUonly.cuh:124-137 for the plus side, 163-176 for
// the minus side), from the cells y1, y2, y3 = l-1, l, l+1:
//   R, the minus side of face l+1/2 (_weno_minus with b, c, d = y1, y2, y3):
//     is0 = (c-b)^2, is1 = (d-c)^2, alpha0 = 1./(3.(is0+eps)^2),
//     alpha1 = 2./(3.(is1+eps)^2), w0 = alpha0/(alpha0+alpha1), w1 = 1.-w0,
//     R = w0 (1.5c - .5b) + w1 (.5c + .5d);
//   L, the plus side of face l-1/2 (_weno_pluss with c, d, e = y1, y2, y3):
//     is0 = (d-e)^2, is1 = (d-c)^2, alpha0 = (1./3.)/(is0+eps)^2,
//     alpha1 = (2./3.)/(is1+eps)^2, w0 = alpha0/(alpha0+alpha1), w1 = 1.-w0,
//     L = w0 (1.5d - .5e) + w1 (.5d + .5c);
// both clipped to [min, max] of y1, y2, y3.  The double literals promote the
// weights' arithmetic and the final combination to double, as in the
// reference.  The squared differences are shared: (y2-y3)^2 is (y3-y2)^2
// bit for bit (rounding to nearest is symmetric under negation).
template <class Pol>
__device__ __forceinline__ void weno3_cell_ref(const typename Pol::T y1, const typename Pol::T y2,
        const typename Pol::T y3, typename Pol::T& R, typename Pol::T& L)
{
    typedef typename Pol::T T;
    const T dl = y2 - y1, dr = y3 - y2;
    const T sl = dl*dl, sr = dr*dr;
    const double el = sl + MPCF_WENOEPS, er = sr + MPCF_WENOEPS;
    const T am0 = (T)(1./(3.*el*el)), am1 = (T)(2./(3.*er*er));
    const T wm0 = am0/(am0 + am1);
    const T wm1 = (T)(1. - wm0);
    const T rm = (T)(wm0*(1.5*y2 - .5*y1) + wm1*(.5*y2 + .5*y3));
    const T ap0 = (T)((1./3.)/(er*er)), ap1 = (T)((2./3.)/(el*el));
    const T wp0 = ap0/(ap0 + ap1);
    const T wp1 = (T)(1. - wp0);
    const T rp = (T)(wp0*(1.5*y2 - .5*y3) + wp1*(.5*y2 + .5*y1));
    const T lo = dmin(dmin(y1, y2), y3);
    const T hi = dmax(dmax(y1, y2), y3);
    R = dmin(dmax(rm, lo), hi);
    L = dmin(dmax(rp, lo), hi);
}

// Both edge values of one cell in the policy's arithmetic.
template <class Pol>
__device__ __forceinline__ void weno_cell(const typename Pol::T y0, const typename Pol::T y1,
        const typename Pol::T y2, const typename Pol::T y3, const typename Pol::T y4,
        typename Pol::T& R, typename Pol::T& L)
{
    if constexpr (Pol::kWeno3)         weno3_cell_ref<Pol>(y1, y2, y3, R, L);
    else if constexpr (Pol::kFastWeno) weno_edges<true, false>(y0, y1, y2, y3, y4, R, L);
    else                               weno_cell_ref<Pol, false>(y0, y1, y2, y3, y4, R, L);
}

// The same as a call, for the rare cells whose weights the forms without
// branches (weno_cell_ref's, weno_edges' kShared) cannot take.
template <class T> struct Edges { T R, L; };
template <class Pol>
__device__ __noinline__ Edges<typename Pol::T> weno_cell_call(const typename Pol::T y0, const typename Pol::T y1,
        const typename Pol::T y2, const typename Pol::T y3, const typename Pol::T y4)
{
    Edges<typename Pol::T> e;
    if constexpr (Pol::kFastWeno)
    {
        if (weno_edges<true, true>(y0, y1, y2, y3, y4, e.R, e.L)) return e;
    }
    weno_cell<Pol>(y0, y1, y2, y3, y4, e.R, e.L);
    return e;
}

// The edge values m (minus side) and p (plus side) of a face, 7 primitives
// each, in the face's components (x: normal u, transverse v, w; y: normal v,
// transverse u, w; z: normal w, transverse u, v).
template <class T>
__device__ __forceinline__ void face_state(const T m[8], const T p[8], const int dir, FaceState<T>& S)
{
    S.rm = m[0]; S.rp = p[0];
    S.nm  = dir == 0 ? m[1] : (dir == 1 ? m[2] : m[3]);  S.np  = dir == 0 ? p[1] : (dir == 1 ? p[2] : p[3]);
    S.t1m = dir == 0 ? m[2] : m[1];                      S.t1p = dir == 0 ? p[2] : p[1];
    S.t2m = dir == 2 ? m[2] : m[3];                      S.t2p = dir == 2 ? p[2] : p[3];
    S.pm = m[4]; S.pp = p[4]; S.Gm = m[5]; S.Gp = p[5]; S.Pm = m[6]; S.Pp = p[6];
}

// Wave speeds and fluxes of the face between m and p in the policy's
// arithmetic.
template <class Pol>
__device__ __forceinline__ void face_hllc(const typename Pol::T m[8], const typename Pol::T p[8], const int dir,
                                          typename Pol::T o[kFaceOut])
{
    typedef typename Pol::T T;
    FaceState<T> S;
    face_state<T>(m, p, dir, S);
    if constexpr (Pol::kFastWeno)
    {
        FaceFlux<T> f;
        hllc_face_upwind<T>(S, f);
        o[0] = f.r;
        o[1] = dir == 0 ? f.n : f.t1;
        o[2] = dir == 1 ? f.n : (dir == 0 ? f.t1 : f.t2);
        o[3] = dir == 2 ? f.n : f.t2;
        o[4] = f.e; o[5] = f.G; o[6] = f.P; o[7] = f.w;
    }
    else hllc_face<Pol>(S, dir, o);
}

// A y face and an x face at once, as the two lanes of a pair (the fast FP32
// forms).
__device__ __forceinline__ void face_hllc_yx(const float my[8], const float py[8], const float mx[8], const float px[8],
                                             float oy[kFaceOut], float ox[kFaceOut])
{
    FaceState<float2> S;
    S.rm  = make_float2(my[0], mx[0]); S.rp  = make_float2(py[0], px[0]);
    S.nm  = make_float2(my[2], mx[1]); S.np  = make_float2(py[2], px[1]);
    S.t1m = make_float2(my[1], mx[2]); S.t1p = make_float2(py[1], px[2]);
    S.t2m = make_float2(my[3], mx[3]); S.t2p = make_float2(py[3], px[3]);
    S.pm  = make_float2(my[4], mx[4]); S.pp  = make_float2(py[4], px[4]);
    S.Gm  = make_float2(my[5], mx[5]); S.Gp  = make_float2(py[5], px[5]);
    S.Pm  = make_float2(my[6], mx[6]); S.Pp  = make_float2(py[6], px[6]);
    FaceFlux<float2> f;
    hllc_face_upwind<float2>(S, f);
    oy[0] = f.r.x; oy[1] = f.t1.x; oy[2] = f.n.x;  oy[3] = f.t2.x; oy[4] = f.e.x; oy[5] = f.G.x; oy[6] = f.P.x; oy[7] = f.w.x;
    ox[0] = f.r.y; ox[1] = f.n.y;  ox[2] = f.t1.y; ox[3] = f.t2.y; ox[4] = f.e.y; ox[5] = f.G.y; ox[6] = f.P.y; ox[7] = f.w.y;
}

// Conserved (rho, rho u, rho v, rho w, E, G, P) -> primitives (rho, u, v, w,
// p, G, P).  Reference form (GPUkernels.cu:209-244):
//   u = (rho u)/rho, ...;  p = (E - 0.5f*rho*(u*u + v*v + w*w) - P) / G
// in the reference-rounding and FP64 policies.  The fast policies multiply
// by reciprocals.  In the liquid E and P are ~50x the internal energy G p,
// so E - ke - P cancels catastrophically in FP32; the mixed policy recovers
// the pressure in compensated FP32 (comp_pressure below).
// Compensated FP32 pressure recovery p = ((E - P) - ke) / G.  E - P is
// formed as the unevaluated sum s + e of the two-sum algorithm (Knuth; s the
// rounded difference, e its exact rounding error), so the cancellation of E
// against P loses nothing; ke (small against E) is subtracted from s and e
// added back; the quotient is a product with the approximate reciprocal of
// G, corrected once by its residual (num - G q) / G.  Every operation is an
// explicit round-to-nearest instruction, so the result does not depend on
// the translation unit's contraction flags.
__device__ __forceinline__ float comp_pressure(const float E, const float P, const float G, const float ke)
{
    const float s = __fsub_rn(E, P);
    const float z = __fsub_rn(s, E);
    const float e = __fadd_rn(__fsub_rn(E, __fsub_rn(s, z)), __fsub_rn(-P, z));
    const float num = __fadd_rn(__fsub_rn(s, ke), e);
    const float iG = rcp_approx(G);
    const float q = __fmul_rn(num, iG);
    return __fmaf_rn(__fmaf_rn(-G, q, num), iG, q);
}

template <class Pol>
__device__ __forceinline__ void to_primitive(const typename Pol::T c[7], typename Pol::T q[7])
{
    typedef typename Pol::T T;
    q[0] = c[0];
    if constexpr (Pol::kFastWeno)
    {
        const T ir = rcp_approx(c[0]);
        q[1] = c[1] * ir;
        q[2] = c[2] * ir;
        q[3] = c[3] * ir;
        if constexpr (Pol::kCompP)
            q[4] = comp_pressure(c[4], c[6], c[5],
                                 __fmul_rn(__fmaf_rn(c[3], q[3], __fmaf_rn(c[2], q[2], __fmul_rn(c[1], q[1]))), 0.5f));
        else
            q[4] = (c[4] - (T)0.5*c[0]*(q[1]*q[1] + q[2]*q[2] + q[3]*q[3]) - c[6]) * rcp_approx(c[5]);
    }
    else
    {
        q[1] = c[1] / c[0];
        q[2] = c[2] / c[0];
        q[3] = c[3] / c[0];
        q[4] = (c[4] - (T)0.5f*c[0]*(q[1]*q[1] + q[2]*q[2] + q[3]*q[3]) - c[6]) / c[5];
    }
    q[5] = c[5];
    q[6] = c[6];
}

// Maximum of non-negative values through the order of their bit patterns
// (a NaN's pattern orders above every finite value, so it surfaces).
__device__ __forceinline__ void atomic_max_bits(void* p, float v)
{
    atomicMax((unsigned*)p, __float_as_uint(v));
}
__device__ __forceinline__ void atomic_max_bits(void* p, double v)
{
    atomicMax((unsigned long long*)p, (unsigned long long)__double_as_longlong(v));
}
__device__ __forceinline__ float  shfl_max(float v)  { for (int o = 16; o > 0; o >>= 1) v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, o)); return v; }
__device__ __forceinline__ double shfl_max(double v) { for (int o = 16; o > 0; o >>= 1) v = fmax(v, __shfl_xor_sync(0xffffffffu, v, o)); return v; }

// Maximum characteristic speed of one cell, |u|max + c with
//   p = (E - (ru^2+rv^2+rw^2)*(0.5/rho) - P)/G,  c = sqrt(((p+P)/G + p)/rho)
// (GPUkernels.cu:1182-1222; the mixed policy recovers p in compensated FP32).  Every
// operation is an explicit instruction -- round-to-nearest intrinsics, and
// in the fast policies the approximate reciprocal and square root -- so the
// result is the same whatever the translation unit's contraction and
// division flags: the stand-alone reduction and the one fused into the stage
// kernel agree bit for bit.
template <class Pol>
__device__ __forceinline__ typename Pol::T cell_sos_rn(const typename Pol::T r, const typename Pol::T u,
        const typename Pol::T v, const typename Pol::T w, const typename Pol::T e,
        const typename Pol::T G, const typename Pol::T P)
{
    typedef typename Pol::T T;
    if constexpr (sizeof(T) == 8)
    {
        const double sq = __dadd_rn(__dadd_rn(__dmul_rn(u, u), __dmul_rn(v, v)), __dmul_rn(w, w));
        const double p = __ddiv_rn(__dsub_rn(__dsub_rn(e, __dmul_rn(sq, __ddiv_rn(0.5, r))), P), G);
        const double c = __dsqrt_rn(__ddiv_rn(__dadd_rn(__ddiv_rn(__dadd_rn(p, P), G), p), r));
        return __dadd_rn(c, __ddiv_rn(fmax(fmax(fabs(u), fabs(v)), fabs(w)), r));
    }
    else if constexpr (Pol::kFastWeno)
    {
        // the fast policies: reciprocals and square root of the special-
        // function unit, the compensated pressure in the mixed policy,
        // every operation an explicit instruction (so the two reductions
        // still agree bit for bit)
        const float ir = rcp_approx(r), iG = rcp_approx(G);
        const float sq = __fmaf_rn(w, w, __fmaf_rn(v, v, __fmul_rn(u, u)));
        const float ke = __fmul_rn(sq, __fmul_rn(0.5f, ir));
        float p;
        if constexpr (Pol::kCompP)
            p = comp_pressure(e, P, G, ke);
        else
            p = __fmul_rn(__fsub_rn(__fsub_rn(e, ke), P), iG);
        const float c = sqrt_approx(__fmul_rn(__fmaf_rn(__fadd_rn(p, P), iG, p), ir));
        return __fmaf_rn(fmaxf(fmaxf(fabsf(u), fabsf(v)), fabsf(w)), ir, c);
    }
    else
    {
        // the reference-rounding policy: IEEE division and square root
        static_assert(!Pol::kCompP, "compensated pressure: fast policies only");
        const float sq = __fadd_rn(__fadd_rn(__fmul_rn(u, u), __fmul_rn(v, v)), __fmul_rn(w, w));
        const float p = __fdiv_rn(__fsub_rn(__fsub_rn(e, __fmul_rn(sq, __fdiv_rn(0.5f, r))), P), G);
        const float c = __fsqrt_rn(__fdiv_rn(__fadd_rn(__fdiv_rn(__fadd_rn(p, P), G), p), r));
        return __fadd_rn(c, __fdiv_rn(fmaxf(fmaxf(fabsf(u), fabsf(v)), fabsf(w)), r));
    }
}

} // namespace mpcf
