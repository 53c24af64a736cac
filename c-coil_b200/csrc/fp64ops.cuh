// Reciprocal square root, square root and division in FP64.  First the forms for
// FP64 work that needs FP64 accuracy but not the reference's operation sequence
// (the refinement pass of FP32_REFINED plans and the FP64 nodes of the FP32
// arrangement kernels), each from the FP64 estimate of the special-function
// unit:
//
//   rsqrt64u(x): 1/sqrt(x) from rsqrt.approx.ftz.f64 and one third-order step
//                (Householder's), y <- y + (e y)(1/2 + 3/8 e), e = 1 - (x y) y;
//   sqrt64u(x):  sqrt(x) by the same step applied to s = x y;
//   div64u(n, d): n / d from rcp.approx.ftz.f64, one step y <- y + y (1 - d y)
//                and the residual correction q + (n - q d) y with n - q d exact
//                in a fused multiply-add (Markstein's final step), which squares
//                the remaining relative error;
//   sqrt64(x), rsqrt64(x): the IEEE path outside [kLo64, kHi64].
//
// The unchecked forms take arguments in [kLo64, kHi64] (positive, normal, far
// from both ends of the exponent range, so no intermediate overflows or
// flushes).  Loops that can bound their arguments beforehand take them through
// the CHECKED template argument: the range check and the IEEE paths are
// branches, and a branch per root keeps the compiler from interleaving
// independent roots.  ccoil_eval_fp64_op exposes the unchecked forms (and
// logRatio64) for accuracy checks against the host.
#ifndef CCOIL_FP64OPS_CUH
#define CCOIL_FP64OPS_CUH

constexpr double kLo64 = 1e-36, kHi64 = 1e36;

__device__ __forceinline__ double rsqrt64u(double x)
{
    double y;
    asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(x));
    const double e = fma(-(x * y), y, 1.0);
    return fma(e * y, fma(0.375, e, 0.5), y);
}

__device__ __forceinline__ double sqrt64u(double x)
{
    double y;
    asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(x));
    const double s = x * y;
    const double e = fma(-s, y, 1.0);
    return fma(e * s, fma(0.375, e, 0.5), s);
}

__device__ __forceinline__ double rsqrt64(double x)
{
    if (!(x > kLo64 && x < kHi64))
        return 1.0 / sqrt(x);
    return rsqrt64u(x);
}

__device__ __forceinline__ double sqrt64(double x)
{
    if (!(x > kLo64 && x < kHi64))
        return sqrt(x);
    return sqrt64u(x);
}

__device__ __forceinline__ double div64u(double n, double d)
{
    double y;
    asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(d));
    y = fma(y, fma(-d, y, 1.0), y);
    const double q = n * y;
    return fma(fma(-q, d, n), y, q);
}

// Square root, reciprocal of the rounded root, and quotients that round as the
// IEEE operations do, for the integrands that keep the reference's operation
// sequence (arguments in [kLo64, kHi64]).  Each takes the special-function
// unit's estimate (relative error below 2^-20), an iteration step, and
// Markstein's correction by the residual, exact in a fused multiply-add.
//   root64   third-order step, so that the estimate is good to an ulp before the
//            correction: none of 7.3e9 random arguments differed from the IEEE
//            root, nor did the reciprocals and quotients formed from it;
//   root64n  Newton step (relative error below 2^-38): the corrected root is
//            within 0.5 ulp + 2^-24 ulp, so about one in 10^8 rounds the other
//            way, for two FP64 operations less.  For every integrand but the
//            gradient, whose RZ bracket magnifies a single rounding 10^8 times;
//   div64u   (above) likewise 0.5 ulp + 2^-26 ulp: 2 of 7.3e9 differed.
// FP64-pipe operations: root64 8, root64n 6, a reciprocal 2, a quotient 3, div64u
// 5, where the compiler's IEEE root takes 13 and its division 8.
// ccoil_eval_integrand_op exposes them (tests/test_log64_gpu.py).
struct Root64
{
    double y;  // 1 / sqrt(x), to about one ulp (root64) or 2^-38 (root64n)
    double s;  // sqrt(x), rounded
};

__device__ __forceinline__ double half64(double x)  // x / 2 on the integer pipe
{
    return __hiloint2double(__double2hiint(x) - 0x100000, __double2loint(x));
}

__device__ __forceinline__ Root64 root64(double x)
{
    Root64 r;
    r.y = rsqrt64u(x);
    const double s = x * r.y;
    r.s = fma(fma(-s, s, x), half64(r.y), s);
    return r;
}

__device__ __forceinline__ Root64 root64n(double x)
{
    double y;
    asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(x));
    Root64 r;
    r.y = fma(fma(-(x * y), y, 1.0), half64(y), y);
    const double s = x * r.y;
    r.s = fma(fma(-s, s, x), half64(r.y), s);
    return r;
}

// n / d given y, the reciprocal of d to a few ulp
__device__ __forceinline__ double quotient64(double n, double d, double y)
{
    const double q = n * y;
    return fma(fma(-q, d, n), y, q);
}

// 1 / d likewise
__device__ __forceinline__ double reciprocal64(double d, double y) { return fma(y, fma(-d, y, 1.0), y); }

// 1 / d to about one ulp
__device__ __forceinline__ double rcp64u(double d)
{
    double y;
    asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(d));
    const double e = fma(-d, y, 1.0);
    return fma(y, fma(e, e, e), y);
}

template <bool CHECKED> __device__ __forceinline__ double rsqrt64t(double x)
{
    return CHECKED ? rsqrt64(x) : rsqrt64u(x);
}

template <bool CHECKED> __device__ __forceinline__ double sqrt64t(double x)
{
    return CHECKED ? sqrt64(x) : sqrt64u(x);
}

template <bool CHECKED> __device__ __forceinline__ double div64t(double n, double d)
{
    return CHECKED ? n / d : div64u(n, d);
}

// Every argument of an angular loop lies in [lo, hi] when the loop forms it as
// base + k c or base - k c with k >= 0 and |c| <= 1 and the bounds are the
// computed base - k and base + k (rounding is monotone).
__device__ __forceinline__ bool inRange64(double lo, double hi) { return lo > kLo64 && hi < kHi64; }

#endif
