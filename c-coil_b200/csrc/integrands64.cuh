// FP64 integrands of the reference's CPU quadrature, node for node, shared by
// the field kernels (fields.cu) and the coil-pair kernels (pairs.cu).  Included
// inside an anonymous namespace.
//
//   A fast  src/Coil/Fields/CalculateFieldsFast.cxx:13-83
//   B fast  src/Coil/Fields/CalculateFieldsFast.cxx:85-160
//   G fast  src/Coil/Fields/CalculateFieldsFast.cxx:162-266
//   A/B/G slow  src/Coil/Fields/CalculateFieldsSlow.cxx:13-265
//   Cartesian wrappers  src/Coil/Fields/CalculateFieldsMethods.cxx:6-84

#include "fp64ops.cuh"
#include "log64.cuh"

// angular nodes in flight per thread in the FP64 loops: a node is one serial
// chain of roots, and 4 keep the FP64 pipe busier than 3, 2 or 1 (A of 128 coils
// at 2^17 points: 36.8, 37.4, 43.4 and 48.0 ms; before the root forms of
// fp64ops.cuh were cut further, the last two)
constexpr int kUnroll64 = 4;

// body(node) for nodes lane, lane + LANES, ... of n, kUnroll64 = 4 in flight and the
// rest two and one at a time: a left-over node on its own is one serial chain (A and B
// of 128 coils at 2^17 points 0.5 % faster than with the compiler's remainder loop, M
// and F/T of 2^15 arrangements 1.5 and 1 %)
template <int LANES, typename Body>
__device__ __forceinline__ void forNodes64(const double2 *pt, int n, int lane, Body body)
{
    int k = lane;
#pragma unroll 1
    for (; k + 3 * LANES < n; k += 4 * LANES)
    {
        const double2 a = pt[k], b = pt[k + LANES], c = pt[k + 2 * LANES], d = pt[k + 3 * LANES];
        body(a);
        body(b);
        body(c);
        body(d);
    }
    if (k + LANES < n)
    {
        const double2 a = pt[k], b = pt[k + LANES];
        body(a);
        body(b);
        k += 2 * LANES;
    }
    if (k < n)
        body(pt[k]);
}

// The gradient: the same (GROUPED, in the batched kernel: B + G of 48 systems 24.8
// against 26.0 ms) or the compiler's unrolled loop (in the field kernels: G of 128 coils
// 50.9 against 51.3 ms)
template <int LANES, bool GROUPED, typename Body>
__device__ __forceinline__ void loopNodes64(const double2 *pt, int n, int lane, Body body)
{
    if constexpr (GROUPED)
        forNodes64<LANES>(pt, n, lane, body);
    else
    {
#pragma unroll kUnroll64
        for (int k = lane; k < n; k += LANES)
        {
            const double2 q = pt[k];
            body(q);
        }
    }
}

// part i of n of a segment's thickness nodes (the field kernels split few points
// this way); the default is all of them
struct Slice
{
    int i = 0, n = 1;
    __device__ __forceinline__ int begin(int nodes) const { return nodes * i / n; }
    __device__ __forceinline__ int end(int nodes) const { return nodes * (i + 1) / n; }
};

struct Frame
{
    double z, r, cphi, sphi;
};

// point -> coil frame cylindrical coordinates: inverse transform of (p - centre)
// as vec3::Matrix3 * vec3::Vector3 evaluates it (Matrix3.cxx:50-55, left to right,
// no fused multiply-add), then (z, sqrt(x^2 + y^2), atan2(y, x)) as
// Vector3::getAsCylindricalCoords (Vector3.cxx:99-102); cos and sin of the
// azimuth are taken as x/r and y/r
// (T is double, or volatile double for a pose kept in shared memory)
template <typename T>
__device__ __forceinline__ Frame toCoilFrameAt(const T *pos, const T *M, double px, double py, double pz)
{
    double dx = __dsub_rn(px, pos[0]), dy = __dsub_rn(py, pos[1]), dz = __dsub_rn(pz, pos[2]);
    double x = __dadd_rn(__dadd_rn(__dmul_rn(M[0], dx), __dmul_rn(M[1], dy)), __dmul_rn(M[2], dz));
    double y = __dadd_rn(__dadd_rn(__dmul_rn(M[3], dx), __dmul_rn(M[4], dy)), __dmul_rn(M[5], dz));
    Frame f;
    f.z = __dadd_rn(__dadd_rn(__dmul_rn(M[6], dx), __dmul_rn(M[7], dy)), __dmul_rn(M[8], dz));
    f.r = __dsqrt_rn(__dadd_rn(__dmul_rn(x, x), __dmul_rn(y, y)));
    if (f.r > 0.0)
    {
        f.cphi = x / f.r;
        f.sphi = y / f.r;
    }
    else
    {
        f.cphi = 1.0;  // atan2(0, 0) = 0
        f.sphi = 0.0;
    }
    return f;
}

__device__ __forceinline__ Frame toCoilFrame(const SegmentHeader &h, double px, double py, double pz)
{
    return toCoilFrameAt(h.position, h.inv_transform, px, py, pz);
}

// ---------------------------------------------------------------------------
// FP64 segment integrals (cylindrical partial sums for one segment)
//
// Several integrands cancel catastrophically inside a node (e + d for d << 0 in
// A, G2 - G1 in B, the RZ bracket of G), and what is in front of such a
// cancellation would show any other rounding amplified far above 1e-12.  There
// the reference's order of operations is kept, each rounded by itself:
// multiplications, additions and subtractions without contraction (mul, add,
// sub), roots and reciprocals as IEEE operations round, in G always (root64), in
// A, B and the slow sums but for about one in 10^8 (root64n).  What only scales a
// node's term need not be: A's logarithm is that of a ratio without its rounded
// quotient (logRatio64, a few ulp), B's fast quotient is within 0.5 ulp + 2^-26
// ulp (div64u), G's 1 / M^2 comes from a reciprocal within an ulp (rcp64u),
// constant factors are taken out of the loops, and the weighting and the
// accumulation are reassociated and fused.
// ---------------------------------------------------------------------------
__device__ __forceinline__ double mul(double a, double b) { return __dmul_rn(a, b); }
__device__ __forceinline__ double add(double a, double b) { return __dadd_rn(a, b); }
__device__ __forceinline__ double sub(double a, double b) { return __dsub_rn(a, b); }
__device__ __forceinline__ double dvd(double a, double b) { return __ddiv_rn(a, b); }
__device__ __forceinline__ double sqr(double a) { return __dsqrt_rn(a); }

// The angular loops take roots, reciprocals and quotients from fp64ops.cuh, at
// about half the FP64-pipe cost of the compiler's IEEE operations, for arguments
// in [kLo64, kHi64]; that pipe bounds every kernel built on these
// integrands.  Whether a thickness node's arguments stay inside is decided
// once per node from bounds of them (base - k and base + k for base - k c,
// |c| <= 1: rounding is monotone).  The nodes that do not (a point on a winding
// node, infinities, NaN) run the same loop with the IEEE operations, out of
// line so that the loops' register budget does not carry it.
__device__ __noinline__ double phiA64Ieee(const double2 *pt, int n, int lane, int lanes, double cA, double cB,
                                          double top, double bot)
{
    double part = 0.0;
    for (int k = lane; k < n; k += lanes)
    {
        const double2 q = pt[k];
        const double g = dvd(1.0, sqr(sub(cB, mul(cA, q.x))));
        const double d1 = mul(top, g), d2 = mul(bot, g);
        const double e1 = sqr(add(mul(d1, d1), 1.0)), e2 = sqr(add(mul(d2, d2), 1.0));
        part += mul(mul(q.y, q.x), log64(dvd(add(e1, d1), add(e2, d2))));
    }
    return part;
}

__device__ __noinline__ double phiSlowA64Ieee(const double2 *pt, int n, int lane, int lanes, double p, double cA,
                                              double cB)
{
    double part = 0.0;
    for (int k = lane; k < n; k += lanes)
    {
        const double2 q = pt[k];
        part += mul(q.y, dvd(mul(p, q.x), sqr(sub(cB, mul(cA, q.x)))));
    }
    return part;
}

template <int LANES>
__device__ __forceinline__ double segmentA64(const SegmentHeader &h, const double2 *tt, const double2 *lt,
                                             const double2 *pt, const Frame &f, int lane,
                                             Slice th = Slice())
{
    double sum = 0.0;
    const int n = h.n_phi;
    if (h.fast)
    {
        // CalculateFieldsFast.cxx:27-78
        const double top = add(f.z, h.half_length), bot = sub(f.z, h.half_length);
        const double far2 = fmax(top * top, bot * bot);
        for (int j = th.begin(h.n_t), jEnd = th.end(h.n_t); j < jEnd; ++j)
        {
            const double2 t = tt[j];
            const double cA = mul(mul(2.0, t.x), f.r);
            const double cB = add(mul(t.x, t.x), mul(f.r, f.r));
            const double lo = cB - fabs(cA);
            double part = 0.0;
            // (top / rho)^2 below 1e13 keeps e + d well above zero
            if (lo > kLo64 && cB + fabs(cA) < kHi64 && far2 < 1e13 * lo)
                forNodes64<LANES>(pt, n, lane, [&](const double2 q) {
                    const Root64 rho = root64n(sub(cB, mul(cA, q.x)));
                    const double g = reciprocal64(rho.s, rho.y);
                    const double d1 = mul(top, g), d2 = mul(bot, g);
                    const double e1 = root64n(add(mul(d1, d1), 1.0)).s, e2 = root64n(add(mul(d2, d2), 1.0)).s;
                    part = fma(q.y * q.x, logRatio64(add(e1, d1), add(e2, d2)), part);
                });
            else
                part = phiA64Ieee(pt, n, lane, LANES, cA, cB, top, bot);
            sum += mul(mul(t.y, t.x), part);
        }
    }
    else
    {
        // CalculateFieldsSlow.cxx:55-78
        for (int i = 0; i < h.n_l; ++i)
        {
            const double2 l = lt[i];
            const double zl = add(l.x, f.z);
            for (int j = th.begin(h.n_t), jEnd = th.end(h.n_t); j < jEnd; ++j)
            {
                const double2 t = tt[j];
                const double cA = mul(mul(2.0, t.x), f.r);
                const double cB = add(add(mul(t.x, t.x), mul(f.r, f.r)), mul(zl, zl));
                double part = 0.0;
                if (inRange64(cB - fabs(cA), cB + fabs(cA)))
                    forNodes64<LANES>(pt, n, lane, [&](const double2 q) {
                        const Root64 d = root64n(sub(cB, mul(cA, q.x)));
                        part = fma(q.y, quotient64(mul(t.x, q.x), d.s, d.y), part);
                    });
                else
                    part = phiSlowA64Ieee(pt, n, lane, LANES, t.x, cA, cB);
                sum += mul(mul(l.y, t.y), part);
            }
        }
    }
    return sum;
}

__device__ __noinline__ double2 phiB64Ieee(const double2 *pt, int n, int lane, int lanes, double cA, double cB,
                                           double cC, double d1, double d2, double top, double bot)
{
    double h0 = 0.0, z0 = 0.0;
    for (int k = lane; k < n; k += lanes)
    {
        const double2 q = pt[k];
        const double F = mul(mul(2.0, cB), q.x);
        const double g1 = dvd(1.0, sqr(sub(d1, F))), g2 = dvd(1.0, sqr(sub(d2, F)));
        h0 += mul(mul(q.y, q.x), sub(g2, g1));
        z0 += mul(mul(q.y, dvd(sub(cA, mul(0.5, F)), sub(cC, F))), sub(mul(top, g1), mul(bot, g2)));
    }
    return make_double2(h0, z0);
}

__device__ __noinline__ double2 phiSlowB64Ieee(const double2 *pt, int n, int lane, int lanes, double cA, double cB,
                                               double cC, double cD)
{
    double h0 = 0.0, z0 = 0.0;
    for (int k = lane; k < n; k += lanes)
    {
        const double2 q = pt[k];
        const double F = mul(mul(2.0, cC), q.x);
        const double den = sub(cD, F);
        const double g = dvd(q.y, mul(den, sqr(den)));
        z0 += mul(g, sub(cA, mul(cC, q.x)));
        h0 += mul(g, mul(cB, q.x));
    }
    return make_double2(h0, z0);
}

template <int LANES>
__device__ __forceinline__ void segmentB64(const SegmentHeader &h, const double2 *tt, const double2 *lt,
                                           const double2 *pt, const Frame &f, int lane, double &H, double &Z,
                                           Slice th = Slice())
{
    H = 0.0;
    Z = 0.0;
    const int n = h.n_phi;
    if (h.fast)
    {
        // CalculateFieldsFast.cxx:100-155
        const double top = add(f.z, h.half_length), bot = sub(f.z, h.half_length);
        for (int j = th.begin(h.n_t), jEnd = th.end(h.n_t); j < jEnd; ++j)
        {
            const double2 t = tt[j];
            const double cA = mul(t.x, t.x), cB = mul(t.x, f.r);
            const double cC = add(cA, mul(f.r, f.r));
            const double d1 = add(mul(top, top), cC), d2 = add(mul(bot, bot), cC);
            const double cF = 2.0 * cB;
            double h0 = 0.0, z0 = 0.0;
            if (inRange64(cC - fabs(cF), fmax(d1, d2) + fabs(cF)))
                forNodes64<LANES>(pt, n, lane, [&](const double2 q) {
                    const double F = mul(cF, q.x);
                    const Root64 r1 = root64n(sub(d1, F)), r2 = root64n(sub(d2, F));
                    const double g1 = reciprocal64(r1.s, r1.y), g2 = reciprocal64(r2.s, r2.y);
                    h0 = fma(q.y * q.x, sub(g2, g1), h0);
                    // cA - F / 2 rounds once either way
                    z0 = fma(q.y * div64u(fma(-0.5, F, cA), sub(cC, F)), sub(mul(top, g1), mul(bot, g2)), z0);
                });
            else
            {
                const double2 hz = phiB64Ieee(pt, n, lane, LANES, cA, cB, cC, d1, d2, top, bot);
                h0 = hz.x;
                z0 = hz.y;
            }
            H += mul(mul(t.y, t.x), h0);
            Z += mul(t.y, z0);
        }
    }
    else
    {
        // CalculateFieldsSlow.cxx:129-158
        for (int i = 0; i < h.n_l; ++i)
        {
            const double2 l = lt[i];
            const double zl = add(l.x, f.z);
            for (int j = th.begin(h.n_t), jEnd = th.end(h.n_t); j < jEnd; ++j)
            {
                const double2 t = tt[j];
                const double cA = mul(t.x, t.x), cB = mul(t.x, zl), cC = mul(t.x, f.r);
                const double cD = add(add(cA, mul(f.r, f.r)), mul(zl, zl));
                const double cF = 2.0 * cC;
                double h0 = 0.0, z0 = 0.0;
                if (inRange64(cD - fabs(cF), cD + fabs(cF)))
                {
                    forNodes64<LANES>(pt, n, lane, [&](const double2 q) {
                        const double F = mul(cF, q.x);
                        const double den = sub(cD, F);
                        const Root64 d = root64n(den);
                        const double g = quotient64(q.y, mul(den, d.s), d.y * d.y * d.y);
                        z0 = fma(g, fma(-0.5, F, cA), z0);
                        h0 = fma(g, q.x, h0);
                    });
                    h0 *= cB;
                }
                else
                {
                    const double2 hz = phiSlowB64Ieee(pt, n, lane, LANES, cA, cB, cC, cD);
                    h0 = hz.x;
                    z0 = hz.y;
                }
                const double w = mul(l.y, t.y);
                H += mul(w, h0);
                Z += mul(w, z0);
            }
        }
    }
}

__device__ __noinline__ double4 phiG64Ieee(const double2 *pt, int n, int lane, int lanes, double p, double r,
                                           double top, double bot)
{
    const double A = mul(p, p), B = mul(r, r), C = mul(p, r);
    const double D = add(A, B), E = add(mul(A, A), mul(B, B)), F = mul(C, C);
    const double G1 = add(D, mul(top, top)), G2 = add(D, mul(bot, bot));
    double s0 = 0.0, s1 = 0.0, s2 = 0.0, s3 = 0.0;
    for (int k = lane; k < n; k += lanes)
    {
        const double2 q = pt[k];
        const double c = q.x, c2 = mul(c, c);
        const double pe = mul(mul(2.0, C), c);
        const double J1 = sub(G1, pe), J2 = sub(G2, pe);
        const double K1 = sqr(J1), K2 = sqr(J2);
        const double L1 = dvd(1.0, mul(J1, K1)), L2 = dvd(1.0, mul(J2, K2));
        const double M = sub(D, pe);
        const double N = add(sub(mul(mul(mul(2.0, F), c), add(c2, 2.0)),
                                 mul(mul(C, add(mul(3.0, c2), 1.0)), D)),
                             mul(c, E));
        const double O = sub(mul(c, D), mul(2.0, C));
        const double w = q.y;
        s0 += mul(mul(w, dvd(mul(p, c), r)), sub(dvd(1.0, K2), dvd(1.0, K1)));
        s1 += mul(mul(mul(w, sub(C, mul(A, c))), c), sub(L1, L2));
        s3 += mul(mul(w, sub(A, mul(C, c))), sub(L1, L2));
        s2 += mul(dvd(mul(w, p), mul(M, M)), sub(mul(mul(top, L1), add(mul(O, J1), N)),
                                                mul(mul(bot, L2), add(mul(O, J2), N))));
    }
    return make_double4(s0, s1, s2, s3);
}

__device__ __noinline__ double4 phiSlowG64Ieee(const double2 *pt, int n, int lane, int lanes, double p, double r,
                                               double zl)
{
    const double A = mul(p, p), B = mul(r, r), C = mul(zl, zl);
    const double D = mul(r, p), E = mul(p, zl), F = dvd(1.0, r);
    const double G = sub(add(mul(2.0, A), mul(2.0, B)), C), Hh = add(add(A, B), C);
    double s0 = 0.0, s1 = 0.0, s2 = 0.0, s3 = 0.0;
    for (int k = lane; k < n; k += lanes)
    {
        const double2 q = pt[k];
        const double c = q.x;
        const double J = sub(Hh, mul(mul(2.0, D), c));
        const double sJ = sqr(J);
        const double X = dvd(q.y, mul(J, sJ));
        const double Y = dvd(q.y, mul(mul(J, J), sJ));
        s0 += mul(X, mul(mul(F, E), c));
        s1 += mul(mul(Y, mul(-3.0, mul(E, sub(r, mul(p, c))))), c);
        s3 += mul(Y, mul(-3.0, mul(E, sub(p, mul(r, c)))));
        s2 += mul(Y, sub(mul(mul(p, sub(G, mul(D, c))), c), mul(mul(3.0, A), r)));
    }
    return make_double4(s0, s1, s2, s3);
}

// {RPhi, RR, RZ, ZZ}
template <int LANES, bool GROUPED = false>
__device__ __forceinline__ void segmentG64(const SegmentHeader &h, const double2 *tt, const double2 *lt,
                                           const double2 *pt, const Frame &f, int lane, double *g,
                                           Slice th = Slice())
{
    double rphi = 0.0, rr = 0.0, rz = 0.0, zz = 0.0;
    const double r = f.r;
    const int n = h.n_phi;
    if (h.fast)
    {
        // CalculateFieldsFast.cxx:179-254.  The RZ bracket (N, O, L, J) keeps the
        // reference's roundings: near the winding's radius it cancels so far that
        // they are all that is left of it.  What only scales a node's term
        // (p c / r, w p / M^2) is rounded on its own
        const double top = add(f.z, h.half_length), bot = sub(f.z, h.half_length);
        for (int j = th.begin(h.n_t), jEnd = th.end(h.n_t); j < jEnd; ++j)
        {
            const double2 t = tt[j];
            const double A = mul(t.x, t.x), B = mul(r, r), C = mul(t.x, r);
            const double D = add(A, B), E = add(mul(A, A), mul(B, B)), F2 = 2.0 * mul(C, C);
            const double G1 = add(D, mul(top, top)), G2 = add(D, mul(bot, bot));
            const double C2 = 2.0 * C;
            double s0 = 0.0, s1 = 0.0, s2 = 0.0, s3 = 0.0;
            if (inRange64(D - fabs(C2), fmax(G1, G2) + fabs(C2)))
            {
                loopNodes64<LANES, GROUPED>(pt, n, lane, [&](const double2 &q) {
                    const double c = q.x, c2 = mul(c, c);
                    const double pe = mul(C2, c);
                    const double J1 = sub(G1, pe), J2 = sub(G2, pe);
                    const Root64 K1 = root64(J1), K2 = root64(J2);
                    const double i1 = reciprocal64(K1.s, K1.y), i2 = reciprocal64(K2.s, K2.y);
                    const double L1 = reciprocal64(mul(J1, K1.s), i1 * i1 * i1);
                    const double L2 = reciprocal64(mul(J2, K2.s), i2 * i2 * i2);
                    const double iM = rcp64u(sub(D, pe));
                    const double N = add(sub(mul(mul(F2, c), add(c2, 2.0)), mul(mul(C, add(mul(3.0, c2), 1.0)), D)),
                                         mul(c, E));
                    const double O = sub(mul(c, D), C2);
                    const double w = q.y, wdL = w * sub(L1, L2);
                    s0 = fma(w * c, sub(i2, i1), s0);
                    s1 = fma(wdL * c, sub(C, mul(A, c)), s1);
                    s3 = fma(wdL, fma(-0.5, pe, A), s3);
                    s2 = fma(w * (iM * iM), sub(mul(mul(top, L1), add(mul(O, J1), N)),
                                                mul(mul(bot, L2), add(mul(O, J2), N))), s2);
                });
                s0 *= t.x / r;
                s2 *= t.x;
            }
            else
            {
                const double4 s = phiG64Ieee(pt, n, lane, LANES, t.x, r, top, bot);
                s0 = s.x;
                s1 = s.y;
                s2 = s.z;
                s3 = s.w;
            }
            rphi += mul(t.y, s0);
            rr += mul(t.y, s1);
            rz += mul(t.y, s2);
            zz += mul(t.y, s3);
        }
    }
    else
    {
        // CalculateFieldsSlow.cxx:212-251
        for (int i = 0; i < h.n_l; ++i)
        {
            const double2 l = lt[i];
            const double zl = add(l.x, f.z);
            for (int j = th.begin(h.n_t), jEnd = th.end(h.n_t); j < jEnd; ++j)
            {
                const double2 t = tt[j];
                const double A = mul(t.x, t.x), B = mul(r, r), C = mul(zl, zl);
                const double D = mul(r, t.x), D2 = 2.0 * D, A3r = mul(mul(3.0, A), r);
                const double G = sub(add(2.0 * A, 2.0 * B), C), Hh = add(add(A, B), C);
                double s0 = 0.0, s1 = 0.0, s2 = 0.0, s3 = 0.0;
                if (inRange64(Hh - fabs(D2), Hh + fabs(D2)))
                {
                    const double E = mul(t.x, zl);
                    loopNodes64<LANES, GROUPED>(pt, n, lane, [&](const double2 &q) {
                        const double c = q.x;
                        const double J = sub(Hh, mul(D2, c));
                        const Root64 K = root64(J);
                        const double y2 = K.y * K.y, y3 = y2 * K.y;
                        const double X = quotient64(q.y, mul(J, K.s), y3);
                        const double Y = quotient64(q.y, mul(mul(J, J), K.s), y3 * y2);
                        s0 = fma(X, c, s0);
                        s1 = fma(Y * c, sub(r, mul(t.x, c)), s1);
                        s3 = fma(Y, sub(t.x, mul(r, c)), s3);
                        s2 = fma(Y, sub(mul(mul(t.x, sub(G, mul(D, c))), c), A3r), s2);
                    });
                    s0 *= E / r;
                    s1 *= -3.0 * E;
                    s3 *= -3.0 * E;
                }
                else
                {
                    const double4 s = phiSlowG64Ieee(pt, n, lane, LANES, t.x, r, zl);
                    s0 = s.x;
                    s1 = s.y;
                    s2 = s.z;
                    s3 = s.w;
                }
                const double w = mul(l.y, t.y);
                rphi += mul(w, s0);
                rr += mul(w, s1);
                rz += mul(w, s2);
                zz += mul(w, s3);
            }
        }
    }
    g[0] = rphi;
    g[1] = rr;
    g[2] = rz;
    g[3] = zz;
}
// ---------------------------------------------------------------------------
// Epilogues: cylindrical partials -> Cartesian, rotated by the coil transform,
// added to the point's accumulators (linear in the partials, so per-lane
// partials can be rotated before the cross-lane reduction).
// ---------------------------------------------------------------------------
__device__ __forceinline__ void addRotated(const SegmentHeader &h, double vx, double vy, double vz, double *acc)
{
    acc[0] += h.transform[0] * vx + h.transform[1] * vy + h.transform[2] * vz;
    acc[1] += h.transform[3] * vx + h.transform[4] * vy + h.transform[5] * vz;
    acc[2] += h.transform[6] * vx + h.transform[7] * vy + h.transform[8] * vz;
}

// CalculateFieldsMethods.cxx:39-84, including the on-axis branch and the T*G
// product of the reference.
__device__ __forceinline__ void addGradient(const SegmentHeader &h, const Frame &f, const double *g, double *acc)
{
    double G[9];
    double rphi = g[0], rr = g[1], rz = g[2], zz = g[3];
    if (f.r / h.inner_radius < 1e-12)
    {
        G[0] = rr; G[1] = 0.0; G[2] = 0.0;
        G[3] = 0.0; G[4] = rr; G[5] = 0.0;
        G[6] = 0.0; G[7] = 0.0; G[8] = zz;
    }
    else
    {
        double c = f.cphi, s = f.sphi;
        double xx = rr * c * c + rphi * s * s;
        double yy = rr * s * s + rphi * c * c;
        double xy = s * c * (rr - rphi);
        double xz = rz * c, yz = rz * s;
        G[0] = xx; G[1] = xy; G[2] = xz;
        G[3] = xy; G[4] = yy; G[5] = yz;
        G[6] = xz; G[7] = yz; G[8] = zz;
    }
    const double *T = h.transform;
#pragma unroll
    for (int i = 0; i < 3; ++i)
#pragma unroll
        for (int j = 0; j < 3; ++j)
            acc[3 * i + j] += T[3 * i] * G[j] + T[3 * i + 1] * G[3 + j] + T[3 * i + 2] * G[6 + j];
}

template <int FIELD, int LANES, bool GROUPED = false>
__device__ __forceinline__ void integrateSegment64(const unsigned char *seg, double px, double py, double pz, int lane,
                                                   double *acc, Slice th = Slice())
{
    const SegmentHeader &h = *reinterpret_cast<const SegmentHeader *>(seg);
    const double2 *tt = reinterpret_cast<const double2 *>(seg) + h.off_t;
    const double2 *lt = reinterpret_cast<const double2 *>(seg) + h.off_l;
    const double2 *pt = reinterpret_cast<const double2 *>(seg) + h.off_phi;
    if (th.begin(h.n_t) == th.end(h.n_t))
        return;  // fewer thickness nodes than parts
    Frame f = toCoilFrame(h, px, py, pz);
    if (FIELD == CCOIL_FIELD_B)
    {
        double H, Z;
        segmentB64<LANES>(h, tt, lt, pt, f, lane, H, Z, th);
        addRotated(h, H * f.cphi, H * f.sphi, Z, acc);
    }
    else if (FIELD == CCOIL_FIELD_G)
    {
        double g[4];
        segmentG64<LANES, GROUPED>(h, tt, lt, pt, f, lane, g, th);
        addGradient(h, f, g, acc);
    }
    else
    {
        double a = segmentA64<LANES>(h, tt, lt, pt, f, lane, th) * h.field_factor;
        addRotated(h, -a * f.sphi, a * f.cphi, 0.0, acc);
    }
}

