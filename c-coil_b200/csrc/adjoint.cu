// Adjoint of the coil-group B field with respect to every coil's parameters
// {R, a, b, N*I, x, y, z, yAxisAngle, zAxisAngle}, for every coil type: the fast
// method (RECTANGULAR and THIN, analytic length integral,
// src/Coil/Fields/CalculateFieldsFast.cxx:85-160) and the slow method (FLAT and
// FILAMENT, length nodes, src/Coil/Fields/CalculateFieldsSlow.cxx:86-165).
//
// Given points p and the upstream gradient v(p) = dL/dB(p), it accumulates
// dL/dtheta_c = sum_p v(p) . dB_c(p)/dtheta_c.  Nothing from the forward pass
// is stored: every node is recomputed here (the quadrature is cheap to redo and
// would cost n x nodes x 12 words to keep).
//
// Fast method, per node (weight w, node radius r', azimuth cos c; point at
// radius r, height z; top/bot = z +- b/2; rho^2 = r'^2 + r^2 - 2 r' r c;
// g1,2 = (rho^2 + top^2, bot^2)^-1/2):
//   H node  r' c (g2 - g1)                     (radial field, the reference's H term)
//   Z node  (r'^2 - r' r c) / rho^2 (top g1 - bot g2)
//   d/dr'   H: c (g2 - g1) + r' c (r' - r c)(g1^3 - g2^3)
//           Z: [(2r' - r c) E + N dE/dr'] / rho^2 - 2 N E (r' - r c) / rho^4,
//              E = top g1 - bot g2, N = r'^2 - r' r c, dE/dr' = -(r' - r c)(top g1^3 - bot g2^3)
//   d/dtop  H: r' c top g1^3       Z: N g1^3
//   d/dbot  H: -r' c bot g2^3      Z: -N g2^3
//   local Jacobian (RPhi, RR, RZ, ZZ) = (H/r, dH/dr, dH/dz, dZ/dz) in the stable
//   forms r' c (g2 - g1) / r, r' c (r - r' c)(g1^3 - g2^3), r' c (top g1^3 - bot g2^3),
//   (r'^2 - r' r c)(g1^3 - g2^3).
// With r' = R + a u (u the node's fraction of the thickness), B = K sum w h and
// K = 1e-7 (N I / (a b)) (a / tB) (pi / aB) / 2 (the reference's constant):
//   dB/dR = K sum w dh/dr',  dB/da = K sum w u dh/dr',
//   dB/db = -B/b + K sum w (dh/dtop - dh/dbot) / 2,  dB/d(NI) = B / (NI).
// Slow method, per node at height zl = z + l (l = b v the length node, v in
// [-1/2, 1/2]; G = (r'^2 + r^2 + zl^2 - 2 r' r c)^-1/2):
//   H node  r' c zl G^3,  Z node N G^3,
//   d/dr'   H: c zl G^3 - 3 r' c zl (r' - r c) G^5,  Z: (2 r' - r c) G^3 - 3 N (r' - r c) G^5
//   d/dzl   H: r' c G^3 - 3 r' c zl^2 G^5 (= the RZ node),  Z: -3 N zl G^5 (= the ZZ node)
//   RR node -3 r' c zl (r - r' c) G^5
// and K = 1e-7 N I (pi / aB) / (4 lB tB) does not depend on a or b:
//   dB/da = K sum w u dh/dr',  dB/db = K sum w v dh/dzl.
// Thin dimensions are 1e-25 R as in the reference (src/Coil/Coil.cxx:27-28); the
// derivative with respect to such a dimension is the one at that value.
// Globally B = T Bloc(T^T (p - pos)): dB/dpos = -T Gloc T^T,
// dB/dangle = T' Bloc + T Gloc T'^T (p - pos).
#include "ccoil_internal.h"

#include <cuda_runtime.h>

#include <algorithm>

#include <cmath>
#include <cstring>
#include <vector>

namespace ccoil
{
int cudaFail(cudaError_t e, const char *what);

namespace
{
constexpr double kPi = 3.14159265358979323846;
constexpr int kAdjLanes = 4;
constexpr int kAdjThreads = 128;
constexpr int kAdjPoints = kAdjThreads / kAdjLanes;

struct alignas(16) AdjCoil
{
    double R, a, b, K1, half_b, NI;  // K1 = K / (N I): the constant per unit N I
    double pos[3];
    double T[9], Ta[9], Tb[9];  // transform and its derivatives by yAxisAngle, zAxisAngle
    int nt, nphi, off_t, off_phi;  // tables in 16-byte units from the record start
    int nl, off_l, fast, pad2;     // slow method: length nodes
};

// thickness node {r', w, u}; length node {l, w, v}
struct alignas(16) AdjT
{
    double rp, w, u, pad;
};

__device__ __forceinline__ void matvec(const double *M, const double *v, double *o)
{
    o[0] = M[0] * v[0] + M[1] * v[1] + M[2] * v[2];
    o[1] = M[3] * v[0] + M[4] * v[1] + M[5] * v[2];
    o[2] = M[6] * v[0] + M[7] * v[1] + M[8] * v[2];
}

__device__ __forceinline__ void matTvec(const double *M, const double *v, double *o)
{
    o[0] = M[0] * v[0] + M[3] * v[1] + M[6] * v[2];
    o[1] = M[1] * v[0] + M[4] * v[1] + M[7] * v[2];
    o[2] = M[2] * v[0] + M[5] * v[1] + M[8] * v[2];
}

#include "fp64ops.cuh"

// The sums of one angular loop.  Fast method, each weighted by w (and the ones
// marked c by w c): with D3 = g1^3 - g2^3, T3 = top g1^3 - bot g2^3,
// Y = (top g1 - bot g2) / rho^2 and m = r' - r c (so N = r' m),
//   a0 c (g2 - g1)     a1 m Y          a2 c D3 m       a3 Y
//   a4 m (m / rho^2) (T3 + 2 Y)        a5 c (top g1^3 + bot g2^3)
//   a6 m (g1^3 + g2^3) a7 c D3 (r - r' c)              a8 c T3    a9 m D3
// from which dZ/dr' = r' a3 + a1 - r' a4 (the node's form above, with
// 2 r' - r c = r' + m), and the other terms by factors of r' alone.
// Slow method (G3 = G^3, G5 = G^5):
//   a0 c G3  a1 m G3  a2 c m G5  a3 G3  a4 m m G5  a5 c G5  a6 m G5  a7 c G5 (r - r' c)
struct AdjSums
{
    double a[10];
};

// One fast node costs 49 FP64-pipe operations this way; with the terms formed one
// by one, CUDA's reciprocal roots and IEEE divisions it took 133.  The FP64 pipe
// bounds the kernel: 64 RECTANGULAR coils at 4,096 points 3.54 -> 1.61 ms, 128
// mixed coils at 200,000 points 129 -> 61.6 ms (81 % of that pipe's measured rate;
// two nodes in flight per thread, and register caps of 168, 128 and 96 measured
// slower than the compiler's own choice).  Arguments outside [kLo64, kHi64] take
// the IEEE operations (CHECKED).
template <bool CHECKED>
__device__ __forceinline__ void adjFastLoop(const double2 *pt, int n, int lane, double rp, double r, double top,
                                            double bot, AdjSums &S)
{
    const double cF = 2.0 * rp * r, cC = rp * rp + r * r, T2 = top * top, B2 = bot * bot;
#pragma unroll 2
    for (int k = lane; k < n; k += kAdjLanes)
    {
        const double2 q = pt[k];
        const double c = q.x, w = q.y, wc = w * c;
        const double rho2 = fma(-cF, c, cC);
        const double g1 = rsqrt64t<CHECKED>(rho2 + T2), g2 = rsqrt64t<CHECKED>(rho2 + B2);
        const double i = CHECKED ? 1.0 / rho2 : rcp64u(rho2);
        const double g13 = g1 * (g1 * g1), g23 = g2 * (g2 * g2);
        const double D3 = g13 - g23, t1 = top * g13, t2 = bot * g23, T3 = t1 - t2;
        const double Y = fma(top, g1, -bot * g2) * i;
        const double m = fma(-r, c, rp), wm = w * m, wcD = wc * D3;
        S.a[0] = fma(wc, g2 - g1, S.a[0]);
        S.a[1] = fma(wm, Y, S.a[1]);
        S.a[2] = fma(wcD, m, S.a[2]);
        S.a[3] = fma(w, Y, S.a[3]);
        S.a[4] = fma(wm * (m * i), fma(2.0, Y, T3), S.a[4]);
        S.a[5] = fma(wc, t1 + t2, S.a[5]);
        S.a[6] = fma(wm, g13 + g23, S.a[6]);
        S.a[7] = fma(wcD, fma(-rp, c, r), S.a[7]);
        S.a[8] = fma(wc, T3, S.a[8]);
        S.a[9] = fma(wm, D3, S.a[9]);
    }
}

template <bool CHECKED>
__device__ __forceinline__ void adjSlowLoop(const double2 *pt, int n, int lane, double rp, double r, double zl2,
                                            AdjSums &S)
{
    const double cF = 2.0 * rp * r, cD = rp * rp + r * r + zl2;
#pragma unroll 2
    for (int k = lane; k < n; k += kAdjLanes)
    {
        const double2 q = pt[k];
        const double c = q.x, w = q.y, wc = w * c;
        const double G = rsqrt64t<CHECKED>(fma(-cF, c, cD));
        const double G2 = G * G, G3 = G2 * G, G5 = G3 * G2;
        const double m = fma(-r, c, rp), wm = w * m, wcG5 = wc * G5, wmG5 = wm * G5;
        S.a[0] = fma(wc, G3, S.a[0]);
        S.a[1] = fma(wm, G3, S.a[1]);
        S.a[2] = fma(wcG5, m, S.a[2]);
        S.a[3] = fma(w, G3, S.a[3]);
        S.a[4] = fma(wmG5, m, S.a[4]);
        S.a[5] += wcG5;
        S.a[6] += wmG5;
        S.a[7] = fma(wcG5, fma(-rp, c, r), S.a[7]);
    }
}

__device__ __noinline__ AdjSums adjFastIeee(const double2 *pt, int n, int lane, double rp, double r, double top,
                                            double bot)
{
    AdjSums S = {};
    adjFastLoop<true>(pt, n, lane, rp, r, top, bot, S);
    return S;
}

__device__ __noinline__ AdjSums adjSlowIeee(const double2 *pt, int n, int lane, double rp, double r, double zl2)
{
    AdjSums S = {};
    adjSlowLoop<true>(pt, n, lane, rp, r, zl2, S);
    return S;
}

__global__ void __launch_bounds__(kAdjThreads) adjointKernel(const unsigned char *__restrict__ blob,
                                                             const long long *__restrict__ offsets, int ncoils,
                                                             const double *__restrict__ points,
                                                             const double *__restrict__ gradB, long long npts,
                                                             double *__restrict__ partial)
{
    __shared__ double red[kAdjThreads / 32][9];
    const int lane = threadIdx.x % kAdjLanes;
    const long long p = (long long)blockIdx.x * kAdjPoints + threadIdx.x / kAdjLanes;
    const bool active = p < npts;
    double P[3] = {0, 0, 0}, v[3] = {0, 0, 0};
    if (active)
        for (int i = 0; i < 3; ++i)
        {
            P[i] = points[3 * p + i];
            v[i] = gradB[3 * p + i];
        }
    // blockIdx.x: a tile of kAdjPoints points; blockIdx.y (grid-strided): the coil
    for (int c = blockIdx.y; c < ncoils; c += gridDim.y)
    {
        const unsigned char *base = blob + offsets[c];
        const AdjCoil &C = *reinterpret_cast<const AdjCoil *>(base);
        const AdjT *tt = reinterpret_cast<const AdjT *>(reinterpret_cast<const double2 *>(base) + C.off_t);
        const double2 *pt = reinterpret_cast<const double2 *>(base) + C.off_phi;
        double d[3] = {P[0] - C.pos[0], P[1] - C.pos[1], P[2] - C.pos[2]};
        double xl[3];
        matTvec(C.T, d, xl);
        const double r = sqrt(xl[0] * xl[0] + xl[1] * xl[1]), z = xl[2];
        const double cph = r > 0.0 ? xl[0] / r : 1.0, sph = r > 0.0 ? xl[1] / r : 0.0;
        const double top = z + C.half_b, bot = z - C.half_b;
        // H, Z, dH/dR, dZ/dR, dH/da, dZ/da, dH/db', dZ/db', RPhi*r, RR, RZ, ZZ
        double s[12];
        for (int i = 0; i < 12; ++i)
            s[i] = 0.0;
        if (C.fast)
            for (int j = 0; j < C.nt; ++j)
            {
                const AdjT t = tt[j];
                const double rp = t.rp, k = 2.0 * rp * r, cC = rp * rp + r * r;
                AdjSums S = {};
                if (inRange64(cC - k, fmax(top * top, bot * bot) + (cC + k)))
                    adjFastLoop<false>(pt, C.nphi, lane, rp, r, top, bot, S);
                else
                    S = adjFastIeee(pt, C.nphi, lane, rp, r, top, bot);
                const double *a = S.a;
                const double H = t.w * rp * a[0];
                const double dH = t.w * fma(rp, a[2], a[0]), dZ = t.w * (fma(rp, a[3] - a[4], a[1]));
                const double wp = t.w * rp;
                s[0] += H;
                s[1] += wp * a[1];
                s[2] += dH;
                s[3] += dZ;
                s[4] += t.u * dH;
                s[5] += t.u * dZ;
                s[6] += 0.5 * wp * a[5];
                s[7] += 0.5 * wp * a[6];
                s[8] += H;  // RPhi * r
                s[9] += wp * a[7];
                s[10] += wp * a[8];
                s[11] += wp * a[9];
            }
        else
        {
            const AdjT *lt = reinterpret_cast<const AdjT *>(reinterpret_cast<const double2 *>(base) + C.off_l);
            for (int l = 0; l < C.nl; ++l)
            {
                const AdjT L = lt[l];
                const double zl = z + L.rp;
                for (int j = 0; j < C.nt; ++j)
                {
                    const AdjT t = tt[j];
                    const double rp = t.rp, k = 2.0 * rp * r, cD = rp * rp + r * r + zl * zl;
                    AdjSums S = {};
                    if (inRange64(cD - k, cD + k))
                        adjSlowLoop<false>(pt, C.nphi, lane, rp, r, zl * zl, S);
                    else
                        S = adjSlowIeee(pt, C.nphi, lane, rp, r, zl * zl);
                    const double *a = S.a;
                    const double lw = L.w * t.w, wp = lw * rp;
                    const double H = wp * zl * a[0];
                    const double dH = lw * zl * fma(-3.0 * rp, a[2], a[0]);
                    const double dZ = lw * (fma(rp, a[3], a[1]) - 3.0 * rp * a[4]);
                    const double RZ = wp * fma(-3.0 * zl * zl, a[5], a[0]);  // dH/dzl
                    const double ZZ = -3.0 * wp * zl * a[6];                 // dZ/dzl
                    s[0] += H;
                    s[1] += wp * a[1];
                    s[2] += dH;
                    s[3] += dZ;
                    s[4] += t.u * dH;
                    s[5] += t.u * dZ;
                    s[6] += L.u * RZ;
                    s[7] += L.u * ZZ;
                    s[8] += H;  // RPhi * r
                    s[9] -= 3.0 * wp * zl * a[7];
                    s[10] += RZ;
                    s[11] += ZZ;
                }
            }
        }
        for (int off = kAdjLanes / 2; off > 0; off /= 2)
            for (int i = 0; i < 12; ++i)
                s[i] += __shfl_xor_sync(0xffffffffu, s[i], off);
        double g[9] = {0, 0, 0, 0, 0, 0, 0, 0, 0};
        if (active && lane == 0)
        {
            const double K = C.K1 * C.NI;
            const double H = K * s[0], Z = K * s[1];
            const double Bl[3] = {H * cph, H * sph, Z};
            const double Bu[3] = {C.K1 * s[0] * cph, C.K1 * s[0] * sph, C.K1 * s[1]};  // per unit N I
            double B[3];
            matvec(C.T, Bu, B);
            double Tv[3];
            matTvec(C.T, v, Tv);  // local components of v
            // dB/dR, dB/da, dB/db (local components, rotated by T: v.T x = (T^T v).x)
            const double dR[3] = {K * s[2] * cph, K * s[2] * sph, K * s[3]};
            const double da[3] = {K * s[4] * cph, K * s[4] * sph, K * s[5]};
            // the fast method's constant holds 1 / b (its length integral is analytic)
            const double ib = C.fast ? 1.0 / C.b : 0.0;
            const double db[3] = {-Bl[0] * ib + K * s[6] * cph, -Bl[1] * ib + K * s[6] * sph, -Bl[2] * ib + K * s[7]};
            g[0] = Tv[0] * dR[0] + Tv[1] * dR[1] + Tv[2] * dR[2];
            g[1] = Tv[0] * da[0] + Tv[1] * da[1] + Tv[2] * da[2];
            g[2] = Tv[0] * db[0] + Tv[1] * db[1] + Tv[2] * db[2];
            g[3] = v[0] * B[0] + v[1] * B[1] + v[2] * B[2];
            // local Jacobian
            double G[9];
            const double rphi = K * s[8], rr = K * s[9], rz = K * s[10], zz = K * s[11];
            if (r / C.R < 1e-12)
            {
                G[0] = rr; G[1] = 0; G[2] = 0; G[3] = 0; G[4] = rr; G[5] = 0; G[6] = 0; G[7] = 0; G[8] = zz;
            }
            else
            {
                const double rp_ = rphi / r;
                G[0] = rr * cph * cph + rp_ * sph * sph;
                G[4] = rr * sph * sph + rp_ * cph * cph;
                G[1] = G[3] = sph * cph * (rr - rp_);
                G[2] = G[6] = rz * cph;
                G[5] = G[7] = rz * sph;
                G[8] = zz;
            }
            // position: -(T G T^T)^T v = -T G (T^T v)   (G symmetric)
            double GTv[3], pg[3];
            matvec(G, Tv, GTv);
            matvec(C.T, GTv, pg);
            g[4] = -pg[0];
            g[5] = -pg[1];
            g[6] = -pg[2];
            // angles: v . (T' Bl + T G T'^T d)
            for (int m = 0; m < 2; ++m)
            {
                const double *Tp = m == 0 ? C.Ta : C.Tb;
                double t1[3], u1[3], u2[3];
                matvec(Tp, Bl, t1);
                matTvec(Tp, d, u1);
                matvec(G, u1, u2);
                double t2[3];
                matvec(C.T, u2, t2);
                g[7 + m] = v[0] * (t1[0] + t2[0]) + v[1] * (t1[1] + t2[1]) + v[2] * (t1[2] + t2[2]);
            }
        }
        // CTA sum over its points: lanes of a warp (offsets kAdjLanes..16), then warps
        for (int off = kAdjLanes; off < 32; off *= 2)
            for (int i = 0; i < 9; ++i)
                g[i] += __shfl_xor_sync(0xffffffffu, g[i], off);
        if (threadIdx.x % 32 == 0)
            for (int i = 0; i < 9; ++i)
                red[threadIdx.x / 32][i] = g[i];
        __syncthreads();
        if (threadIdx.x < 9)
        {
            double sum = 0.0;
            for (int w = 0; w < kAdjThreads / 32; ++w)
                sum += red[w][threadIdx.x];
            partial[((long long)blockIdx.x * ncoils + c) * 9 + threadIdx.x] = sum;
        }
        __syncthreads();
    }
}

// Sum of the CTA partials in a fixed order: a block takes 32 values, its 32 rows of
// threads every 32nd CTA's each
__global__ void __launch_bounds__(1024) adjointReduce(const double *__restrict__ partial, int blocks, int ncoils,
                                                      double *__restrict__ out)
{
    __shared__ double rows[32][32];
    const int x = threadIdx.x % 32, y = threadIdx.x / 32, n = ncoils * 9;
    const int i = blockIdx.x * 32 + x;
    double s = 0.0;
    if (i < n)
    {
#pragma unroll 4
        for (int b = y; b < blocks; b += 32)
            s += partial[(long long)b * n + i];
    }
    rows[y][x] = s;
    __syncthreads();
    if (y == 0 && i < n)
    {
        for (int r = 1; r < 32; ++r)
            s += rows[r][x];
        out[i] = s;
    }
}

void putBytes(std::vector<unsigned char> &blob, const void *p, size_t n)
{
    const unsigned char *c = static_cast<const unsigned char *>(p);
    blob.insert(blob.end(), c, c + n);
}

struct DBuf  // stream-ordered temporary from the library's memory pool
{
    void *p = nullptr;
    cudaStream_t st = nullptr;
    cudaError_t alloc(size_t bytes, cudaStream_t s)
    {
        st = s;
        return scratchAlloc(&p, bytes, s);
    }
    ~DBuf()
    {
        if (p)
            cudaFreeAsync(p, st);
    }
};
} // namespace
} // namespace ccoil

using namespace ccoil;

extern "C" int ccoil_b_field_adjoint(const double *params, const ccoil_precision_args_t *precisions, int coil_count,
                                     const double *points, long long point_count, const double *grad_b,
                                     double *grad_params, void *stream)
{
    if (coil_count < 0 || (coil_count > 0 && (!params || !precisions)))
        return failMessage(CCOIL_ERR_INVALID_ARGUMENT, "null params/precisions or coil_count < 0");
    if (point_count < 0 || (point_count > 0 && (!points || !grad_b)) || (coil_count > 0 && !grad_params))
        return failMessage(CCOIL_ERR_INVALID_ARGUMENT, "null device buffers or point_count < 0");
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    if (coil_count == 0)
        return CCOIL_OK;
    std::vector<unsigned char> blob;
    std::vector<long long> offsets;
    for (int c = 0; c < coil_count; ++c)
    {
        const double *q = params + 9 * c;
        const PrecisionArgs &pa = precisions[c];
        if (!validArgs(pa))
            return failMessage(CCOIL_ERR_INVALID_ARGUMENT, "precision arguments out of range");
        const double R = q[0], NI = q[3];
        if (!(R > 0.0) || !(q[1] >= 0.0) || !(q[2] >= 0.0) || !std::isfinite(NI))
            return failMessage(CCOIL_ERR_INVALID_ARGUMENT, "coil parameters need R > 0, a >= 0, b >= 0, finite N*I");
        // thin dimensions as the reference's Coil replaces them; b / R >= 1e-7 selects the fast method
        const double thin = 1e-7;
        const double a = q[1] / R < thin ? 1e-18 * R * thin : q[1];
        const double b = q[2] / R < thin ? 1e-18 * R * thin : q[2];
        const bool fast = q[2] / R >= thin;
        AdjCoil C;
        std::memset(&C, 0, sizeof(C));
        C.R = R;
        C.a = a;
        C.b = b;
        C.NI = NI;
        C.fast = fast ? 1 : 0;
        if (fast)
            C.K1 = 1e-7 * (1.0 / b) * (1.0 / pa.thickness_blocks) * (kPi / pa.angular_blocks) * 0.5;
        else
            C.K1 = 1e-7 * (kPi / pa.angular_blocks) * 0.25 / (pa.length_blocks * pa.thickness_blocks);
        C.half_b = 0.5 * b;
        C.pos[0] = q[4];
        C.pos[1] = q[5];
        C.pos[2] = q[6];
        const double cY = std::cos(q[7]), sY = std::sin(q[7]), cZ = std::cos(q[8]), sZ = std::sin(q[8]);
        const double T[9] = {cZ * cZ * cY - sZ * sZ, -sZ * cZ * cY - sZ * cZ, cZ * sY,
                             sZ * cZ * cY + sZ * cZ, cZ * cZ - sZ * sZ * cY, sZ * sY,
                             -sY * cZ, sY * sZ, cY};
        const double Ta[9] = {-cZ * cZ * sY, sZ * cZ * sY, cZ * cY,
                              -sZ * cZ * sY, sZ * sZ * sY, sZ * cY,
                              -cY * cZ, cY * sZ, -sY};
        const double k1 = cY + 1.0, dc = cZ * cZ - sZ * sZ;
        const double Tb[9] = {-2.0 * sZ * cZ * k1, -dc * k1, -sZ * sY,
                              dc * k1, -2.0 * sZ * cZ * k1, cZ * sY,
                              sY * sZ, sY * cZ, 0.0};
        std::memcpy(C.T, T, sizeof(T));
        std::memcpy(C.Ta, Ta, sizeof(Ta));
        std::memcpy(C.Tb, Tb, sizeof(Tb));
        C.nt = pa.thickness_blocks * pa.thickness_increments;
        C.nphi = pa.angular_blocks * pa.angular_increments;
        C.nl = fast ? 0 : pa.length_blocks * pa.length_increments;
        C.off_t = (int)(sizeof(AdjCoil) / 16);
        C.off_phi = C.off_t + 2 * C.nt;
        C.off_l = C.off_phi + C.nphi;
        offsets.push_back((long long)blob.size());
        putBytes(blob, &C, sizeof(C));
        const double tb = a / pa.thickness_blocks, ab = kPi / pa.angular_blocks;
        const double *tx = legendreNodes(pa.thickness_increments), *tw = legendreWeights(pa.thickness_increments);
        for (int bt = 0; bt < pa.thickness_blocks; ++bt)
            for (int i = 0; i < pa.thickness_increments; ++i)
            {
                const double u = (bt + 0.5 + 0.5 * tx[i]) / pa.thickness_blocks;
                AdjT e{R + tb * (bt + 0.5) + (tb * 0.5) * tx[i], tw[i], u, 0.0};
                putBytes(blob, &e, sizeof(e));
            }
        const double *ax = legendreNodes(pa.angular_increments), *aw = legendreWeights(pa.angular_increments);
        for (int bp = 0; bp < pa.angular_blocks; ++bp)
            for (int i = 0; i < pa.angular_increments; ++i)
            {
                double e[2] = {std::cos(ab * (bp + 0.5) + (ab * 0.5) * ax[i]), aw[i]};
                putBytes(blob, e, sizeof(e));
            }
        if (!fast)
        {
            // length nodes l = b v, v in [-1/2, 1/2] (CalculateFieldsSlow.cxx's length layer)
            const double lb = b / pa.length_blocks;
            const double *lx = legendreNodes(pa.length_increments), *lw = legendreWeights(pa.length_increments);
            for (int bl = 0; bl < pa.length_blocks; ++bl)
                for (int i = 0; i < pa.length_increments; ++i)
                {
                    const double l = -0.5 * b + lb * (bl + 0.5) + (lb * 0.5) * lx[i];
                    AdjT e{l, lw[i], -0.5 + (bl + 0.5 + 0.5 * lx[i]) / pa.length_blocks, 0.0};
                    putBytes(blob, &e, sizeof(e));
                }
        }
    }
    const long long blocks = point_count > 0 ? (point_count + kAdjPoints - 1) / kAdjPoints : 1;
    if (blocks > (1LL << 24))
        return failMessage(CCOIL_ERR_INVALID_ARGUMENT, "point_count too large for the adjoint's partial sums");
    // one block of device memory: the tables and their offsets, in one copy, and the
    // partial sums
    const size_t offAt = (blob.size() + 15) / 16 * 16, partialAt = (offAt + sizeof(long long) * offsets.size() + 255) / 256 * 256;
    blob.resize(offAt);
    putBytes(blob, offsets.data(), sizeof(long long) * offsets.size());
    DBuf arena;
    cudaError_t e = arena.alloc(partialAt + sizeof(double) * 9 * coil_count * blocks, st);
    if (e == cudaSuccess)
        e = cudaMemcpyAsync(arena.p, blob.data(), blob.size(), cudaMemcpyHostToDevice, st);
    if (e != cudaSuccess)
        return cudaFail(e, "adjoint set-up");
    const unsigned char *base = static_cast<const unsigned char *>(arena.p);
    double *partial = reinterpret_cast<double *>(static_cast<unsigned char *>(arena.p) + partialAt);
    if (point_count == 0)
        e = cudaMemsetAsync(partial, 0, sizeof(double) * 9 * coil_count, st);
    else
        adjointKernel<<<dim3((unsigned)blocks, (unsigned)std::min(coil_count, 65535)), kAdjThreads, 0, st>>>(
            base, reinterpret_cast<const long long *>(base + offAt), coil_count, points, grad_b, point_count, partial);
    if (e == cudaSuccess)
        e = cudaGetLastError();
    if (e == cudaSuccess)
        adjointReduce<<<(coil_count * 9 + 31) / 32, 1024, 0, st>>>(partial, (int)blocks, coil_count, grad_params);
    if (e == cudaSuccess)
        e = cudaGetLastError();
    if (e == cudaSuccess)
        e = cudaStreamSynchronize(st);  // results in grad_params when the call returns
    return e == cudaSuccess ? CCOIL_OK : cudaFail(e, "adjoint");
}
