// Coil-pair kernels: mutual inductance and force/torque over many arrangements
// (the reference's CPU general case, evaluated for every arrangement at once).
//
// Reference algorithm per arrangement and primary (CPU path):
//   Coil::calculateMutualInductanceGeneral  src/Coil/MInductance/CalculateMInductanceGeneral.cxx:8-117
//   Coil::calculateForceTorqueGeneral       src/Coil/ForceAndTorque/CalculateForceGeneral.cxx:9-131
//   ring nodes  Coil::calculateRingIncrementPosition  src/Coil/Utils/SupportFunctions.cxx:72-122
//   coplanar axes  Coil::improvedPrecisionCase       src/Coil/Utils/SupportFunctions.cxx:124-161
//   group sums  CoilGroup::computeMutualInductance / computeForceTorque
//               src/CoilGroup/MInductance/ComputeMInductance.cxx:4-20,
//               src/CoilGroup/ForceAndTorque/ComputeForce.cxx:4-28
// The secondary is a cloud of nodes (length x thickness x azimuth); at each
// node the primary's A (for M) or B (for F/T) is the full field quadrature:
// FP64 (integrands64.cuh), or FP32-compensated (integrands32.cuh) with FP64
// for secondary nodes in the primary's near-field box.
//
// Mapping.  One warp per work unit (grid-stride): an arrangement, or, of few
// arrangements, a group of its primaries and a range of its secondary's nodes
// (PairSplit), which a second kernel adds up.  The 32 lanes split the unit's
// secondary nodes, each lane, or below a wave of units each 8 neighbouring lanes,
// evaluating the primary's whole quadrature at its node; FP32_REFINED gives few
// arrangements a CTA of 4 or 12 warps each instead.  One primary's node tables
// are staged in shared memory where they fit, others are read from global memory
// (all lanes read the same primary node: L1 broadcast).  Every sum has a fixed
// order: results repeat exactly.
#include "ccoil_internal.h"

#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstring>
#include <memory>
#include <new>
#include <vector>

namespace ccoil
{
namespace
{
#include "integrands64.cuh"
#include "integrands32.cuh"
#include "integrands64f.cuh"

constexpr double kPi = 3.14159265358979323846;
constexpr double kMuReduced = 1e-7;

// One primary of a pair, followed in the blob by its tables.
struct alignas(16) PairHeader
{
    SegmentHeader prim;  // primary geometry (its own pose, used when primaries do not move) and node counts
    double m_factor;     // 2 pi N2 / (I1 lB tB aB): mutual inductance scale
    double f_factor;     // 2 pi I2 N2 / (lB tB aB): force/torque scale
    double prim_y_angle; // the primary's own orientation (used when primaries do not move)
    double prim_z_angle;
    int s_nl, s_nt, s_na, s_ablocks;  // secondary node counts and angular blocks
    int off_sl, off_st, off_sa;       // secondary tables (16-byte units from the header)
    int full_ring;                    // 1: always integrate the whole secondary ring (the reference's GPU
                                      // kernels), 0: half ring for coplanar axes (its CPU path)
    // parameter-gradient tables (16-byte units; 0 when absent): d(node position)/d(dimension)
    // of the primary's thickness and length nodes and of the secondary's length and
    // thickness nodes, i.e. the nodes' positions on [0, 1] (thickness) or [-1/2, 1/2] (length)
    int off_tu, off_lu, off_slu, off_stu;
};
static_assert(sizeof(PairHeader) % 16 == 0, "pair header alignment");

struct alignas(16) SecAngular
{
    double bpos;  // angular block index + 0.5
    double x;     // Gauss-Legendre node in [-1, 1]
    double w;     // its weight
    double pad;
};

struct Pose
{
    double pos[3];
    double T[9];
    double Ti[9];
};

// Coil::calculateTransformationMatrices (src/Coil/Utils/CalculateAttributes.cxx:65-78)
__device__ __forceinline__ void poseFromAngles(const double *p, Pose &o)
{
    o.pos[0] = p[0];
    o.pos[1] = p[1];
    o.pos[2] = p[2];
    double sY, cY, sZ, cZ;
    sincos(p[3], &sY, &cY);
    sincos(p[4], &sZ, &cZ);
    o.T[0] = cZ * cZ * cY - sZ * sZ;  o.T[1] = -sZ * cZ * cY - sZ * cZ;  o.T[2] = cZ * sY;
    o.T[3] = sZ * cZ * cY + sZ * cZ;  o.T[4] = cZ * cZ - sZ * sZ * cY;   o.T[5] = sZ * sY;
    o.T[6] = -sY * cZ;                o.T[7] = sY * sZ;                  o.T[8] = cY;
    o.Ti[0] = cZ * cZ * cY - sZ * sZ; o.Ti[1] = sZ * cZ * cY + sZ * cZ;  o.Ti[2] = -cZ * sY;
    o.Ti[3] = -sZ * cZ * cY - sZ * cZ; o.Ti[4] = cZ * cZ - sZ * sZ * cY; o.Ti[5] = sZ * sY;
    o.Ti[6] = sY * cZ;                o.Ti[7] = sY * sZ;                 o.Ti[8] = cY;
}

__device__ __forceinline__ void cross3(const double *a, const double *b, double *o)
{
    o[0] = a[1] * b[2] - a[2] * b[1];
    o[1] = a[2] * b[0] - a[0] * b[2];
    o[2] = a[0] * b[1] - a[1] * b[0];
}

// improvedPrecisionCase: when the two axes and the centre offset are coplanar
// the reference integrates half of the secondary ring starting at `offset`
__device__ __forceinline__ bool improvedCase(const double *pp, const double *sp, double &offset)
{
    const double pn[3] = {sin(pp[3]) * cos(pp[4]), sin(pp[3]) * sin(pp[4]), cos(pp[3])};
    const double sn[3] = {sin(sp[3]) * cos(sp[4]), sin(sp[3]) * sin(sp[4]), cos(sp[3])};
    const double d[3] = {pp[0] - sp[0], pp[1] - sp[1], pp[2] - sp[2]};
    double pl[3];
    cross3(pn, d, pl);
    const double dot = pl[0] * sn[0] + pl[1] * sn[1] + pl[2] * sn[2];
    offset = 0.0;
    if (!(fabs(dot) <= 1e-14))
        return false;
    if (pl[0] == 0.0 && pl[1] == 0.0 && pl[2] == 0.0)
        cross3(sn, d, pl);
    if (pl[0] == 0.0 && pl[1] == 0.0 && pl[2] == 0.0)
        cross3(sn, pn, pl);
    offset = atan2(cos(sp[3]) * (pl[0] * cos(sp[4]) + pl[1] * sin(sp[4])) - pl[2] * sin(sp[3]),
                   pl[0] * sin(sp[4]) - pl[1] * cos(sp[4]));
    return true;
}

// Coil::isZAxisCase (src/Coil/Utils/SupportFunctions.cxx:55-70)
__device__ __forceinline__ bool zAxisCase(const double *pp, const double *sp, double primR)
{
    return fabs(pp[0] / primR) < 1e-12 && fabs(pp[1] / primR) < 1e-12 && fabs(sp[0] / primR) < 1e-12 &&
           fabs(sp[1] / primR) < 1e-12 && fabs(pp[3] / (2 * kPi)) < 1e-12 && fabs(sp[3] / (2 * kPi)) < 1e-12;
}

// sum over the LANES neighbouring lanes that share a secondary node
template <int LANES> __device__ __forceinline__ double laneSum(double v)
{
#pragma unroll
    for (int off = LANES / 2; off > 0; off /= 2)
        v += __shfl_xor_sync(0xffffffffu, v, off);
    return v;
}

// Sums of one angular loop of segmentAD64: weighted by w c, the node's value
// (analytic length integral V, or g) and its derivatives' parts
struct ADSums
{
    double v = 0.0, z = 0.0, r = 0.0, p = 0.0, b = 0.0;
};

// Fast method: nodes phi and pi - phi together, since a mirror pair takes one
// logarithm (as phiLoopA64, integrands64f.cuh, whose num / den form of
// V = asinh(top / rho) - asinh(bot / rho) this is)
template <bool PARAMS, bool CHECKED, int LANES>
__device__ __forceinline__ ADSums phiLoopAD64(const double2 *pt, int n, int lane, double p, double r, double top,
                                              double bot)
{
    const double cF = 2.0 * p * r, cC = p * p + r * r, T2 = top * top, B2 = bot * bot;
    const double aT = fabs(top), aB = fabs(bot);
    const bool above = bot >= 0.0, below = top < 0.0;
    ADSums S;
    auto node = [&](const double2 q, double &num, double &den) {
        const double c = q.x, wc = q.y * c;
        const double rho2 = fma(-cF, c, cC);
        const double x1 = rho2 + T2, x2 = rho2 + B2;
        const double g1 = rsqrt64t<CHECKED>(x1), g2 = rsqrt64t<CHECKED>(x2);
        const double a1 = fma(x1, g1, aT), a2 = fma(x2, g2, aB);
        num = above ? a1 : (below ? a2 : a1 * a2);
        den = above ? a2 : (below ? a1 : rho2);
        const double tg = fma(top, g1, -bot * g2);
        const double wy = wc * (CHECKED ? tg / rho2 : tg * rcp64u(rho2));
        S.z = fma(wc, g1 - g2, S.z);
        S.r = fma(wy, fma(-p, c, r), S.r);
        if (PARAMS)
        {
            S.p = fma(wy, fma(-r, c, p), S.p);
            S.b = fma(wc, g1 + g2, S.b);
        }
    };
#pragma unroll 1
    for (int m = lane; m < n / 2; m += LANES)
    {
        const double2 q = pt[m], qm = pt[n - 1 - m];
        double n1, e1, n2, e2;
        node(q, n1, e1);
        node(qm, n2, e2);
        // (outside the range the products of four lengths would leave that of FP64)
        const double lg = CHECKED ? logRatio64t<CHECKED>(n1, e1) - logRatio64t<CHECKED>(n2, e2)
                                  : logRatio64t<CHECKED>(n1 * e2, e1 * n2);
        S.v = fma(0.5 * (q.y * q.x - qm.y * qm.x), lg, S.v);
    }
    if ((n & 1) && lane == 0)
    {
        const double2 q = pt[n / 2];
        double n1, e1;
        node(q, n1, e1);
        S.v = fma(q.y * q.x, logRatio64t<CHECKED>(n1, e1), S.v);
    }
    return S;
}

template <bool PARAMS, bool CHECKED, int LANES>
__device__ __forceinline__ ADSums phiLoopSlowAD64(const double2 *pt, int n, int lane, double p, double r, double zl2)
{
    const double cF = 2.0 * p * r, cD = p * p + r * r + zl2;
    ADSums S;
#pragma unroll 2
    for (int k = lane; k < n; k += LANES)
    {
        const double2 q = pt[k];
        const double c = q.x, wc = q.y * c;
        const double g = rsqrt64t<CHECKED>(fma(-cF, c, cD));
        const double wg = wc * g, wg3 = wg * (g * g);
        S.v += wg;
        S.z += wg3;
        S.r = fma(wg3, fma(-p, c, r), S.r);
        if (PARAMS)
            S.p = fma(wg3, fma(-r, c, p), S.p);
    }
    return S;
}

// A_phi of the primary at one point (coil frame) and its derivatives: in r and z
// (for the Jacobian), and with PARAMS by the primary's inner radius R, thickness a
// and length b.  With the current density N I / (a b) folded into the node weights,
// the thickness integral (a / 2) sum w_i f(r'_i) makes the weights independent of
// a, so d/dR = sum w_i df/dr', d/da = sum w_i u_i df/dr' (u_i = dr'_i/da), and
// for the fast method d/db = -a/b + the derivative of the length limits
// (top, bot = z +- b/2); for the slow method d/db moves the length nodes.
//   fast node  f = r' c V,  V = asinh(top/rho) - asinh(bot/rho)
//              df/dz = r' c (g1 - g2),  df/dr = -r' c (r - r' c) y,
//              df/dr' = c V - r' c (r' - r c) y,  dV/db = (g1 + g2) / 2,
//              y = (top g1 - bot g2) / rho^2
//   slow node  f = r' c g,  g = D^-1/2
//              df/dz = df/dzl = -r' c zl g^3,  df/dr = -r' c (r - r' c) g^3,
//              df/dr' = c g - r' c (r' - r c) g^3
// One loop yields all of them: the roots and the reciprocal are shared, 47
// FP64-pipe operations per fast node where a loop for the value, in the
// reference's sequence, and one with two asinh and CUDA's rsqrt for the
// derivatives took about 250.  LANES neighbouring lanes split the angular nodes
// and every one of them returns their sums.
// out: {A, dA/dr, dA/dz, dA/dR, dA/da, dA/db} (the first three without PARAMS)
template <bool PARAMS, int LANES>
__device__ __noinline__ void segmentAD64(const SegmentHeader &h, const double2 *tt, const double2 *lt,
                                         const double2 *pt, const double2 *tu, const double2 *lu, double z, double r,
                                         int lane, double *out)
{
    double A = 0.0, Ar = 0.0, Az = 0.0, dR = 0.0, dA = 0.0, dB = 0.0;
    const int n = h.n_phi;
    if (h.fast)
    {
        const double top = z + h.half_length, bot = z - h.half_length;
        for (int j = 0; j < h.n_t; ++j)
        {
            const double2 t = tt[j];
            const double p = t.x, k = 2.0 * p * r, cC = p * p + r * r;
            // every root's argument lies in [cC - k, max(top^2, bot^2) + cC + k]
            const ADSums S = inRange64(cC - k, fmax(top * top, bot * bot) + (cC + k))
                                 ? phiLoopAD64<PARAMS, false, LANES>(pt, n, lane, p, r, top, bot)
                                 : phiLoopAD64<PARAMS, true, LANES>(pt, n, lane, p, r, top, bot);
            A += t.y * p * S.v;
            Ar -= t.y * p * S.r;
            Az += t.y * p * S.z;
            if (PARAMS)
            {
                const double sp = t.y * (S.v - p * S.p);
                dR += sp;
                dA += tu[j].x * sp;
                dB += t.y * p * 0.5 * S.b;
            }
        }
        if (PARAMS)
            dB -= A / (2.0 * h.half_length);
    }
    else
    {
        for (int i = 0; i < h.n_l; ++i)
        {
            const double2 l = lt[i];
            const double zl = l.x + z, zl2 = zl * zl;
            for (int j = 0; j < h.n_t; ++j)
            {
                const double2 t = tt[j];
                const double p = t.x, k = 2.0 * p * r, cD = p * p + r * r + zl2;
                const ADSums S = inRange64(cD - k, cD + k)
                                     ? phiLoopSlowAD64<PARAMS, false, LANES>(pt, n, lane, p, r, zl2)
                                     : phiLoopSlowAD64<PARAMS, true, LANES>(pt, n, lane, p, r, zl2);
                const double w = l.y * t.y;
                A += w * p * S.v;
                Ar -= w * p * S.r;
                Az -= w * p * zl * S.z;
                if (PARAMS)
                {
                    const double sp = w * (S.v - p * S.p);
                    dR += sp;
                    dA += tu[j].x * sp;
                    dB -= w * lu[i].x * p * zl * S.z;
                }
            }
        }
    }
    out[0] = laneSum<LANES>(A);
    out[1] = laneSum<LANES>(Ar);
    out[2] = laneSum<LANES>(Az);
    if (PARAMS)
    {
        out[3] = laneSum<LANES>(dR);
        out[4] = laneSum<LANES>(dA);
        out[5] = laneSum<LANES>(dB);
    }
}

// The five derivatives of segmentAD64 with the primary's quadrature in FP32 (mirror
// pairs, two per packed step, differences by subtraction as in the FP32
// arrangement integrands; the FP64 sum over the secondary's nodes follows).
// Per node h(c) multiplies c, so a pair adds w c (h(c) - h(-c)):
//   fast  h_z = g1 - g2 = -dD g1^2 g2^2 / (g1 + g2),  h_r = -(r - p c) y,
//         h_p = V - p (p - r c) y,  h_b = (g1 + g2) / 2,
//         y = (top g1 - bot g2) / rho^2 (its cancellation-free form outside the slab),
//         V = asinh(u) in the single-asinh form of segmentA32Direct
//   slow  h_z = -zl g^3,  h_r = -(r - p c) g^3,  h_p = g - p (p - r c) g^3
__device__ __noinline__ void segmentAParams32(const SegmentHeader &h, const double2 *tt, const double2 *lt,
                                              const PhiPair2 *pn, const double2 *tu, const double2 *lu,
                                              const Frame &f, double a, double *out)
{
    const double r = f.r;
    const int ne = packedEntries(h.n_phi);
    double Ar = 0.0, Az = 0.0, dR = 0.0, dA = 0.0, dB = 0.0;
    const V2 RF = v2((float)r);
    if (h.fast)
    {
        const double top = f.z + h.half_length, bot = f.z - h.half_length;
        const bool outside = top * bot > 0.0;
        const float topf = (float)top, botf = (float)bot;
        const float dDf = (float)(2.0 * f.z * (2.0 * h.half_length));
        const V2 TOP = v2(topf), BOT = v2(botf), NBOT = v2(-botf), DDF = v2(dDf), NDDF = v2(-dDf);
        for (int j = 0; j < h.n_t; ++j)
        {
            const double2 t = tt[j];
            const double p = t.x, q = (p - r) * (p - r), b2d = 2.0 * p * r;
            const float qf = (float)q, d1 = (float)(top * top + q), d2 = (float)(bot * bot + q);
            float u0;
            {
                const float e1 = d1 * rsqrtNR(d1), e2 = d2 * rsqrtNR(d2);
                u0 = outside ? fabsf(dDf * rcpApprox(fmaf(topf, e2, botf * e1)))
                             : fabsf(fmaf(topf, e2, -botf * e1) * rcpApprox(qf));
            }
            const unsigned mask = __activemask();
            const int tier = __all_sync(mask, u0 < 0.25f) ? 0 : (__all_sync(mask, u0 <= 1.0f) ? 1 : 2);
            const V2 B2 = v2((float)b2d), Q = v2(qf), D1 = v2(d1), D2 = v2(d2), PF = v2((float)p);
            const V2 RMP = v2((float)(r - p)), PMR = v2((float)(p - r));
            Acc4 a0, a1;
            forEntries<1>(ne, 0, a0, a1, [&](int k, Acc4 &acc) {
                const PhiPair2 nd = pn[k];
                auto node = [&](V2 om, V2 &hz, V2 &hr, V2 &hp, V2 &hb) {
                    const V2 den1 = fma2(B2, om, D1), den2 = fma2(B2, om, D2), rho2 = fma2(B2, om, Q);
                    const V2 g1 = rsq2(den1), g2 = rsq2(den2);
                    const V2 s = g1 + g2, gg = g1 * g2, gg2 = gg * gg;
                    const V2 t1 = TOP * g1, t2 = BOT * g2;
                    const V2 X = sel(outside, t1 + t2, rho2);
                    const V2 R = rcp2(s * X);
                    const V2 y = sel(outside, DDF * gg2, t1 - t2) * (s * R);
                    const V2 s1 = den1 * g1, s2 = den2 * g2;
                    const V2 u = sel(outside, DDF, fma2(TOP, s2, NBOT * s1)) *
                                 rcp2(sel(outside, fma2(TOP, s2, BOT * s1), rho2));
                    const V2 V = asinhTier2(u, tier);
                    hz = NDDF * gg2 * (X * R);
                    hr = v2(0.0f) - fma2(PF, om, RMP) * y;
                    hp = V - PF * fma2(RF, om, PMR) * y;
                    hb = v2(0.5f) * s;
                };
                V2 hz, hr, hp, hb, hzm, hrm, hpm, hbm;
                node(nd.omc, hz, hr, hp, hb);
                node(nd.omcm, hzm, hrm, hpm, hbm);
                const V2 wc = nd.wc;
                acc.a = fma2(wc, hz - hzm, acc.a);
                acc.b = fma2(wc, hr - hrm, acc.b);
                acc.c = fma2(wc, hp - hpm, acc.c);
                acc.d = fma2(wc, hb - hbm, acc.d);
            });
            const double sz = hsum(a0.a) + hsum(a1.a), sr = hsum(a0.b) + hsum(a1.b);
            const double sp = hsum(a0.c) + hsum(a1.c), sb = hsum(a0.d) + hsum(a1.d);
            Ar += t.y * p * sr;
            Az += t.y * p * sz;
            dR += t.y * sp;
            dA += t.y * tu[j].x * sp;
            dB += t.y * p * sb;
        }
        dB -= a / (2.0 * h.half_length);
    }
    else
    {
        for (int i = 0; i < h.n_l; ++i)
        {
            const double2 l = lt[i];
            const double zl = l.x + f.z;
            const V2 NZL = v2(-(float)zl);
            for (int j = 0; j < h.n_t; ++j)
            {
                const double2 t = tt[j];
                const double p = t.x, q = (p - r) * (p - r) + zl * zl, b2d = 2.0 * p * r;
                const V2 B2 = v2((float)b2d), Q = v2((float)q), PF = v2((float)p);
                const V2 RMP = v2((float)(r - p)), PMR = v2((float)(p - r));
                Acc4 a0, a1;
                forEntries<1>(ne, 0, a0, a1, [&](int k, Acc4 &acc) {
                    const PhiPair2 nd = pn[k];
                    auto node = [&](V2 om, V2 &hz, V2 &hr, V2 &hp) {
                        const V2 g = rsq2(fma2(B2, om, Q)), g3 = g * g * g;
                        hz = NZL * g3;
                        hr = v2(0.0f) - fma2(PF, om, RMP) * g3;
                        hp = g - PF * fma2(RF, om, PMR) * g3;
                    };
                    V2 hz, hr, hp, hzm, hrm, hpm;
                    node(nd.omc, hz, hr, hp);
                    node(nd.omcm, hzm, hrm, hpm);
                    const V2 wc = nd.wc;
                    acc.a = fma2(wc, hz - hzm, acc.a);
                    acc.b = fma2(wc, hr - hrm, acc.b);
                    acc.c = fma2(wc, hp - hpm, acc.c);
                });
                const double sz = hsum(a0.a) + hsum(a1.a), sr = hsum(a0.b) + hsum(a1.b);
                const double sp = hsum(a0.c) + hsum(a1.c);
                const double w = l.y * t.y;
                Ar += w * p * sr;
                Az += w * p * sz;
                dR += w * sp;
                dA += w * tu[j].x * sp;
                dB += w * lu[i].x * p * sz;
            }
        }
    }
    out[0] = Ar;
    out[1] = Az;
    out[2] = dR;
    out[3] = dA;
    out[4] = dB;
}

// d T / d(y axis angle) and d T / d(z axis angle) of poseFromAngles' transform
__device__ __forceinline__ void transformDerivatives(double yA, double zA, double *dTy, double *dTz)
{
    double sY, cY, sZ, cZ;
    sincos(yA, &sY, &cY);
    sincos(zA, &sZ, &cZ);
    dTy[0] = -cZ * cZ * sY; dTy[1] = sZ * cZ * sY;  dTy[2] = cZ * cY;
    dTy[3] = -sZ * cZ * sY; dTy[4] = sZ * sZ * sY;  dTy[5] = sZ * cY;
    dTy[6] = -cY * cZ;      dTy[7] = cY * sZ;       dTy[8] = -sY;
    const double c2 = cZ * cZ - sZ * sZ, s2 = 2.0 * sZ * cZ;
    dTz[0] = -s2 * (cY + 1.0); dTz[1] = -c2 * (cY + 1.0); dTz[2] = -sZ * sY;
    dTz[3] = c2 * (cY + 1.0);  dTz[4] = -s2 * (1.0 + cY); dTz[5] = cZ * sY;
    dTz[6] = sY * sZ;          dTz[7] = sY * cZ;          dTz[8] = 0.0;
}

// CTAs per SM the register allocation targets, FP64 kernels: as the field
// kernels', four nodes in flight per thread without spills (M 128 registers, F/T
// 168).  2^15 arrangements of the 408 x 374-node pair: M 19.3 ms at 4 (19.8 at 5,
// 19.2 at 3), F/T 12.9 ms at 3 (13.1 at 4, 13.6 at 2); with the compiler's IEEE
// root and division 35.0 and 21.3 ms
#ifndef CCOIL_PAIR_MIN_BLOCKS
#define CCOIL_PAIR_MIN_BLOCKS 4
#endif
#ifndef CCOIL_PAIR_MIN_BLOCKS_FT
#define CCOIL_PAIR_MIN_BLOCKS_FT 3
#endif
// the same for the FP32 variants (M and F/T, packed integrands with the
// subtracted mirror differences): 9 measured best against 6 (M 69.6 and
// 75.2 ms at 2^18 arrangements; F/T 48.0 and 48.5 ms); their lanes wait on
// fixed-latency chains, which more resident warps hide
#ifndef CCOIL_PAIR32_MIN_BLOCKS
#define CCOIL_PAIR32_MIN_BLOCKS 9
#endif
// the FP32_REFINED variants, whose refined nodes run the FP64 forms: 9 measured
// as fast as 8, 7 and 6 (80 registers) at the fractions that reach 1e-7 (M
// 124.4 against 124.7-126.5 ms at 2^18 arrangements; F/T 104.1 against
// 103.0-104.1 ms), and faster at the default fraction (M 72.1 against 73.9-76.0)
#ifndef CCOIL_PAIR32R_MIN_BLOCKS
#define CCOIL_PAIR32R_MIN_BLOCKS 9
#endif
constexpr int pairThreads(int team) { return team > 4 ? 32 * team : 128; }
constexpr int pairMinBlocks(int qty, bool fp32, bool refine)
{
    return refine ? CCOIL_PAIR32R_MIN_BLOCKS
           : fp32 ? CCOIL_PAIR32_MIN_BLOCKS
           : qty == 1 ? CCOIL_PAIR_MIN_BLOCKS_FT
                      : CCOIL_PAIR_MIN_BLOCKS;
}
// FP32_REFINED arrangements: the largest scratch of node contributions (the
// grid shrinks to fit it)
constexpr size_t kPairRefineScratchBytes = size_t(1) << 30;
// largest single-primary blob staged in shared memory (0 turns staging off)
#ifndef CCOIL_PAIR_STAGE_MAX_BYTES
#define CCOIL_PAIR_STAGE_MAX_BYTES (48 * 1024)
#endif

// units per arrangement: groups of primaries x ranges of secondary nodes
struct PairSplit
{
    int groups = 1, parts = 1;
};

// What a warp needs of its current arrangement and primary, written by lane 0
// into shared memory and read back by all lanes inside the secondary-node loop
// (volatile: kept out of registers, which the primary quadrature needs)
struct WarpPose
{
    double pos[3], T[9], Ti[9];  // primary pose
    double sp[3];                // secondary centre
    double sA, cA, sB, cB;       // sin / cos of the secondary's y and z axis angles
    double offset, ablk;         // secondary azimuth offset and angular block size
    double dTy[9], dTz[9];       // d(primary transform)/d(y, z axis angle) (parameter gradient only)
    int skip;                    // coaxial pair left to the z-axis pass
};

// pairKernel64's own shared memory for W sums and a team of that many warps, at
// most; the staged tables come on top
constexpr size_t pairStaticBytes(int W, int team)
{
    const size_t warps = pairThreads(team) / 32;
    return warps * (sizeof(WarpPose) + 64 * sizeof(int)) + sizeof(double) * (size_t)W * (32 * warps + 2 * warps) + 64;
}

// FP64 primary quadrature at one secondary node, out of line for the FP32
// kernel (which takes it only for near-field nodes) so that its register
// budget does not carry the FP64 integrands.  The point's frame coordinates
// pass by value (the quadrature reads z and r only), so nothing of the
// caller's has to sit in memory for the call.
__device__ __forceinline__ Frame frameZR(double z, double r)
{
    Frame f;
    f.z = z;
    f.r = r;
    f.cphi = 1.0;
    f.sphi = 0.0;
    return f;
}

// The FP32 kernels' FP64 nodes (near-field and refined): FP64 accuracy without
// the reference's operation sequence, in the cheaper forms of
// integrands64f.cuh (the table is in the reference's order)
__device__ __noinline__ double pairA64Fast(const SegmentHeader &h, const double2 *tt, const double2 *lt,
                                           const double2 *pt, double z, double r)
{
    return segmentA64Fast<false>(h, tt, lt, pt, frameZR(z, r));
}

__device__ __noinline__ double2 pairB64Fast(const SegmentHeader &h, const double2 *tt, const double2 *lt,
                                            const double2 *pt, double z, double r)
{
    double H, Z;
    segmentB64Fast(h, tt, lt, pt, frameZR(z, r), 0, H, Z);
    return make_double2(H, Z);
}

// The FP32 primary quadrature, out of line as well: the loop over the
// primary's nodes gets the whole register budget.  Its pair sums are plain
// FP32: the FP64 sum over the secondary's nodes averages their rounding
// (measured: the same error statistics against FP64 as with compensated sums,
// at 7-18 % less time)
__device__ __noinline__ double pairA32(const SegmentHeader &h, const double2 *tt, const double2 *lt,
                                       const PhiPair2 *pn, double z, double r)
{
    return segmentA32Direct<1, PlainSum>(h, tt, lt, pn, frameZR(z, r), 0);
}

__device__ __noinline__ double2 pairB32(const SegmentHeader &h, const double2 *tt, const double2 *lt,
                                        const PhiPair2 *pn, double z, double r)
{
    double H, Z;
    segmentB32Direct<1, PlainSum>(h, tt, lt, pn, frameZR(z, r), 0, H, Z);
    return make_double2(H, Z);
}

// stagedBytes > 0: there is one primary and its whole pair blob (stagedBytes,
// a multiple of 16) is copied into shared memory once per CTA, so the inner
// quadrature reads its tables from shared memory instead of through L1.
//
// FP32 (mutual inductance and force/torque only): the primary quadrature at a
// secondary node runs in the FP32-compensated integrands, except for nodes in
// the primary's near-field box: the warp defers those to a list in shared
// memory and evaluates them with the FP64 integrands 32 at a time, so the FP64
// work runs on full warps instead of dragging whole mixed iterations along;
// the secondary-node sums and the cross-lane reduction stay FP64.
//
// REFINE (FP32_REFINED, M and F/T): each secondary node's FP32 contribution is
// also written to the warp's region of nodeScratch (node-major, W doubles per
// node; deferred near-field nodes as zeros).  Once the warp has the primary's
// total, every node whose contribution exceeds `fraction` of it (for F/T: of
// the force or of the torque) is taken out of the sums and evaluated again
// with the FP64 integrands, 32 at a time like the near-field nodes: the nodes
// that dominate an arrangement whose ring sum cancels, whose FP32 errors the
// cancellation magnifies.
//
// Few arrangements are cut into more work units than one per arrangement: groups
// of primaries and, within one primary, ranges of its secondary nodes
// (PairSplit).  Each unit's sums go to `partial` and pairReduceKernel adds an
// arrangement's units in a fixed order.  LANES > 1 (FP64 M, F/T and position gradient): that many
// lanes share a secondary node and split the primary's angular nodes.
//
// TEAM > 1 (REFINE): that many warps, a whole CTA, share each arrangement's nodes,
// since the selection needs the primary's total.
template <int QTY, bool FP32, bool REFINE = false, int LANES = 1, int TEAM = 1>
__global__ void __launch_bounds__(pairThreads(TEAM), pairMinBlocks(QTY, FP32, REFINE) * 4 / (pairThreads(TEAM) / 32))
    pairKernel64(const unsigned char *__restrict__ blob, const long long *__restrict__ primOffsets, int nprim,
                 const double *__restrict__ primPoses, const double *__restrict__ secPoses, long long count,
                 double *__restrict__ out, unsigned long long *__restrict__ zAxisCount, int stagedBytes,
                 const long long *__restrict__ zOffsets, long long *__restrict__ zList,
                 unsigned long long *__restrict__ zListCount, double *__restrict__ nodeScratch, int scratchNodes,
                 double fraction, PairSplit split, double *__restrict__ partial)
{
    extern __shared__ __align__(16) unsigned char stagedPair[];
    constexpr int THREADS = pairThreads(TEAM), WARPS = THREADS / 32;
    __shared__ WarpPose warpPoses[WARPS];
    __shared__ int nearLists[WARPS][64];  // FP32: each warp's deferred near-field secondary nodes
    constexpr int W = QTY == 0 ? 1 : QTY == 1 ? 6 : QTY == 2 ? 3 : 14;
    // Running sums in shared memory: each thread's sums over its secondary nodes
    // (one column per thread, so a warp's accesses hit 32 consecutive doubles)
    // and each warp's sums over the primaries (lane 0).  Held in registers they
    // stayed live across the out-of-line quadrature call and spilled to local
    // memory at the register budget of 9 CTAs per SM.
    __shared__ double laneSums[W][THREADS];
    __shared__ double warpSums[WARPS][W];
    __shared__ double teamSums[TEAM > 1 ? WARPS : 1][W];  // each warp's sums of the current primary
    if (stagedBytes > 0)
    {
        const int4 *src = reinterpret_cast<const int4 *>(blob + primOffsets[0]);
        int4 *dst = reinterpret_cast<int4 *>(stagedPair);
        for (int i = threadIdx.x; i < stagedBytes / 16; i += blockDim.x)
            dst[i] = src[i];
        __syncthreads();
    }
    const int lane = threadIdx.x % 32;
    volatile WarpPose &S = warpPoses[threadIdx.x / 32];
    const long long warp = ((long long)blockIdx.x * blockDim.x + threadIdx.x) / 32;
    const long long warps = (long long)gridDim.x * blockDim.x / 32;
    double *part = &laneSums[0][threadIdx.x];  // part[THREADS i]: this thread's sum i
    double *total = warpSums[threadIdx.x / 32];
    const int perArr = split.groups * split.parts;
    const long long units = count * perArr;
    // a team takes whole arrangements, each warp its part of the nodes
    const int parts = TEAM > 1 ? TEAM : split.parts;
    for (long long u = TEAM > 1 ? (long long)blockIdx.x : warp; u < units; u += TEAM > 1 ? (long long)gridDim.x : warps)
    {
        const long long a = u / perArr;
        const int piece = (int)(u - a * perArr), group = piece / split.parts;
        const int part_i = TEAM > 1 ? threadIdx.x / 32 : piece - group * split.parts;
        const int j0 = (int)((long long)nprim * group / split.groups);
        const int j1 = (int)((long long)nprim * (group + 1) / split.groups);
        if (lane == 0)
            for (int i = 0; i < W; ++i)
                total[i] = 0.0;
        bool hasZ = false;  // lane 0: some primary of this arrangement is left to the z-axis pass
        for (int j = j0; j < j1; ++j)
        {
            const unsigned char *base = stagedBytes > 0 ? stagedPair : blob + primOffsets[j];
            const PairHeader &ph = *reinterpret_cast<const PairHeader *>(base);
            const SegmentHeader &h = ph.prim;
            const double2 *tt = reinterpret_cast<const double2 *>(base) + h.off_t;
            const double2 *lt = reinterpret_cast<const double2 *>(base) + h.off_l;
            const double2 *pt = reinterpret_cast<const double2 *>(base) + h.off_phi;
            const double2 *sl = reinterpret_cast<const double2 *>(base) + ph.off_sl;
            const double2 *st = reinterpret_cast<const double2 *>(base) + ph.off_st;
            const SecAngular *sa = reinterpret_cast<const SecAngular *>(reinterpret_cast<const double2 *>(base) +
                                                                        ph.off_sa);
            const PhiPair2 *pn = reinterpret_cast<const PhiPair2 *>(reinterpret_cast<const double2 *>(base) +
                                                                    h.off_f32);
            __syncwarp();  // every lane is done with the previous pose
            if (lane == 0)
            {
                const double *sp = secPoses + 5 * a;
                Pose P;
                double ppose[5], spose[5];
                for (int i = 0; i < 5; ++i)
                    spose[i] = sp[i];
                if (primPoses)
                {
                    for (int i = 0; i < 5; ++i)
                        ppose[i] = primPoses[5 * a + i];
                    poseFromAngles(ppose, P);
                }
                else
                {
                    for (int i = 0; i < 3; ++i)
                        P.pos[i] = ppose[i] = h.position[i];
                    for (int i = 0; i < 9; ++i)
                    {
                        P.T[i] = h.transform[i];
                        P.Ti[i] = h.inv_transform[i];
                    }
                    ppose[3] = ph.prim_y_angle;
                    ppose[4] = ph.prim_z_angle;
                }
                const bool isZ = zAxisCase(ppose, spose, h.inner_radius);
                if (zAxisCount && isZ && part_i == 0)
                    atomicAdd(zAxisCount, 1ull);
                const bool skip = isZ && zOffsets && zOffsets[j] >= 0;
                S.skip = skip ? 1 : 0;
                hasZ = hasZ || skip;
                double offset = 0.0;
                const bool improved = QTY != 1 && !ph.full_ring ? improvedCase(ppose, spose, offset) : false;
                for (int i = 0; i < 3; ++i)
                {
                    S.pos[i] = P.pos[i];
                    S.sp[i] = spose[i];
                }
                for (int i = 0; i < 9; ++i)
                {
                    S.T[i] = P.T[i];
                    S.Ti[i] = P.Ti[i];
                }
                double sA, cA, sB, cB;
                sincos(spose[3], &sA, &cA);
                sincos(spose[4], &sB, &cB);
                S.sA = sA;
                S.cA = cA;
                S.sB = sB;
                S.cB = cB;
                S.offset = offset;
                S.ablk = (improved ? kPi : 2 * kPi) / ph.s_ablocks;
                if (QTY == 3)
                {
                    double dTy[9], dTz[9];
                    transformDerivatives(ppose[3], ppose[4], dTy, dTz);
                    for (int i = 0; i < 9; ++i)
                    {
                        S.dTy[i] = dTy[i];
                        S.dTz[i] = dTz[i];
                    }
                }
            }
            __syncwarp();
            if (S.skip)
                continue;  // warp-uniform: the z-axis pass adds this primary
            // this unit's secondary nodes: whole warp iterations of 32 / LANES nodes
            constexpr int STEP = 32 / LANES;
            const int nodes = ph.s_nl * ph.s_nt * ph.s_na, iters = (nodes + STEP - 1) / STEP;
            const int nBegin = (int)((long long)iters * part_i / parts) * STEP;
            const int nsec = min(nodes, (int)((long long)iters * (part_i + 1) / parts) * STEP);
            const int sub = lane % LANES, slot = lane / LANES;
            for (int i = 0; i < W; ++i)
                part[THREADS * i] = 0.0;
            // every lane runs the same number of iterations (warp-uniform choices
            // below); a lane past the end evaluates the last node and drops it
            // One secondary node per lane.  mode 0: the FP64 kernel; mode 1: the FP32
            // pass, which defers near-field nodes to the warp's list; mode 2: a batch
            // of deferred nodes, in FP64, one per lane
            int nNear = 0;
            int *list = nearLists[threadIdx.x / 32];
            // REFINE: this warp's node contributions
            double *scr = REFINE ? nodeScratch + (size_t)(TEAM > 1 ? (long long)blockIdx.x : warp) *
                                                   (size_t)scratchNodes * W
                                 : nullptr;
            auto node = [&](int n, bool valid, int mode) {
                const int k = n % ph.s_na, lt_i = n / ph.s_na;
                const int t = lt_i % ph.s_nt, l = lt_i / ph.s_nt;
                const double2 L = sl[l], R = st[t];
                const SecAngular A = sa[k];
                const double ablk = S.ablk;
                const double phi = (S.offset + ablk * A.bpos) + (ablk * 0.5) * A.x;
                double sP, cP;
                sincos(phi, &sP, &cP);
                const double sA = S.sA, cA = S.cA, sB = S.sB, cB = S.cB;
                const double ringP[3] = {cB * cA * cP - sB * sP, sB * cA * cP + cB * sP, -sA * cP};
                const double tan[3] = {-cB * cA * sP - sB * cP, -sB * cA * sP + cB * cP, sA * sP};
                const double q[3] = {S.sp[0] + L.x * sA * cB + R.x * ringP[0],
                                     S.sp[1] + L.x * sA * sB + R.x * ringP[1], S.sp[2] + L.x * cA + R.x * ringP[2]};
                const double w = 0.125 * R.x * L.y * R.y * A.w;
                const Frame f = toCoilFrameAt(S.pos, S.Ti, q[0], q[1], q[2]);
                const bool far = mode == 1;
                if (mode == 1)
                {
                    const bool near = valid && nearWinding(h, f);
                    const unsigned bal = __ballot_sync(0xffffffffu, near);
                    if (bal)
                    {
                        if (near)
                            list[nNear + __popc(bal & ((1u << lane) - 1u))] = n;
                        nNear += __popc(bal);
                        valid = valid && !near;
                    }
                    if (REFINE && near)
                        for (int i = 0; i < W; ++i)
                            scr[(size_t)n * W + i] = 0.0;
                }
                if (QTY == 0)
                {
                    double av;
                    if (!FP32)
                        av = laneSum<LANES>(segmentA64<LANES>(h, tt, lt, pt, f, sub));
                    else if (far)
                        av = pairA32(h, tt, lt, pn, f.z, f.r);
                    else
                        av = pairA64Fast(h, tt, lt, pt, f.z, f.r);
                    const double vx = -av * f.sphi, vy = av * f.cphi;
                    const double Ax = S.T[0] * vx + S.T[1] * vy, Ay = S.T[3] * vx + S.T[4] * vy,
                                 Az = S.T[6] * vx + S.T[7] * vy;
                    const double c = (Ax * tan[0] + Ay * tan[1] + Az * tan[2]) * w;
                    if (valid)
                    {
                        part[0] += c;
                        if (REFINE && far)
                            scr[n] = c;
                    }
                }
                else if (QTY == 3)
                {
                    // parameter gradient: per secondary node, the derivative of
                    // w (A(q) . t) with respect to every coil parameter
                    const double2 *tu = reinterpret_cast<const double2 *>(base) + ph.off_tu;
                    const double2 *lu = reinterpret_cast<const double2 *>(base) + ph.off_lu;
                    const double ul = (reinterpret_cast<const double2 *>(base) + ph.off_slu)[l].x;
                    const double ut = (reinterpret_cast<const double2 *>(base) + ph.off_stu)[t].x;
                    double ad[6], *d = ad + 1;
                    if (FP32 && far)
                    {
                        ad[0] = pairA32(h, tt, lt, pn, f.z, f.r);
                        segmentAParams32(h, tt, lt, pn, tu, lu, f, ad[0], d);
                    }
                    else
                        segmentAD64<true, LANES>(h, tt, lt, pt, tu, lu, f.z, f.r, sub, ad);
                    const double av = ad[0], ar = d[0], az = d[1];
                    const double c = f.cphi, s_ = f.sphi;
                    const double ao = f.r > 0.0 ? av / f.r : ar;
                    const double J[9] = {s_ * c * (ao - ar), -s_ * s_ * ar - c * c * ao, -s_ * az,
                                         c * c * ar + s_ * s_ * ao, s_ * c * (ar - ao), c * az,
                                         0.0, 0.0, 0.0};
                    double e[3], u[3], v[3], gp[3];
                    for (int i = 0; i < 3; ++i)
                        e[i] = -S.T[3 * i] * s_ + S.T[3 * i + 1] * c;                      // T (-sin, cos, 0)
                    for (int i = 0; i < 3; ++i)
                        u[i] = S.T[i] * tan[0] + S.T[3 + i] * tan[1] + S.T[6 + i] * tan[2];  // T^T t
                    for (int i = 0; i < 3; ++i)
                        v[i] = J[i] * u[0] + J[3 + i] * u[1] + J[6 + i] * u[2];           // J^T u
                    for (int i = 0; i < 3; ++i)
                        gp[i] = S.T[3 * i] * v[0] + S.T[3 * i + 1] * v[1] + S.T[3 * i + 2] * v[2];
                    const double et = e[0] * tan[0] + e[1] * tan[1] + e[2] * tan[2];
                    double g[14];
                    g[0] = av * et;
                    g[1] = d[2] * et;
                    g[2] = d[3] * et;
                    g[3] = d[4] * et;
                    // primary orientation: (dT A_loc) . t + (J_loc dT^T (q - c)) . (T^T t)
                    const double aloc[2] = {-s_ * av, c * av};
                    const double dv[3] = {q[0] - S.pos[0], q[1] - S.pos[1], q[2] - S.pos[2]};
                    for (int k = 0; k < 2; ++k)
                    {
                        double dT[9];
                        for (int i = 0; i < 9; ++i)
                            dT[i] = k == 0 ? S.dTy[i] : S.dTz[i];
                        double y[3], gk = 0.0;
                        for (int j = 0; j < 3; ++j)
                            y[j] = dT[j] * dv[0] + dT[3 + j] * dv[1] + dT[6 + j] * dv[2];
                        for (int i = 0; i < 3; ++i)
                        {
                            gk += (dT[3 * i] * aloc[0] + dT[3 * i + 1] * aloc[1]) * tan[i];
                            gk += (J[3 * i] * y[0] + J[3 * i + 1] * y[1] + J[3 * i + 2] * y[2]) * u[i];
                        }
                        g[4 + k] = gk;
                    }
                    // secondary inner radius, thickness, length (node positions; the
                    // weight is proportional to the ring radius)
                    const double axis[3] = {sA * cB, sA * sB, cA};
                    g[6] = av * et / R.x + ringP[0] * gp[0] + ringP[1] * gp[1] + ringP[2] * gp[2];
                    g[7] = ut * g[6];
                    g[8] = ul * (axis[0] * gp[0] + axis[1] * gp[1] + axis[2] * gp[2]);
                    g[9] = gp[0];
                    g[10] = gp[1];
                    g[11] = gp[2];
                    // secondary orientation: node position and tangent move
                    const double A_[3] = {av * e[0], av * e[1], av * e[2]};
                    const double dE1A[3] = {-cB * sA, -sB * sA, -cA}, dAxA[3] = {cA * cB, cA * sB, -sA};
                    const double dE1B[3] = {-sB * cA, cB * cA, 0.0}, dE2B[3] = {-cB, -sB, 0.0},
                                 dAxB[3] = {-sA * sB, sA * cB, 0.0};
                    double gA = 0.0, gB = 0.0;
                    for (int i = 0; i < 3; ++i)
                    {
                        const double dqA = L.x * dAxA[i] + R.x * cP * dE1A[i], dtA = -sP * dE1A[i];
                        const double dqB = L.x * dAxB[i] + R.x * (cP * dE1B[i] + sP * dE2B[i]),
                                     dtB = -sP * dE1B[i] + cP * dE2B[i];
                        gA += dqA * gp[i] + A_[i] * dtA;
                        gB += dqB * gp[i] + A_[i] * dtB;
                    }
                    g[12] = gA;
                    g[13] = gB;
                    if (valid)
                        for (int i = 0; i < 14; ++i)
                            part[THREADS * i] += g[i] * w;
                }
                else if (QTY == 2)
                {
                    // dM/d(secondary position) = factor sum_n w_n J_A(q_n)^T t_n,
                    // J_A = T J_loc T^T; J_loc of A_loc = a(r, z) (-sin, cos, 0)
                    double ad[3];
                    segmentAD64<false, LANES>(h, tt, lt, pt, nullptr, nullptr, f.z, f.r, sub, ad);
                    const double av = ad[0], ar = ad[1], az = ad[2];
                    const double c = f.cphi, s_ = f.sphi;
                    const double ao = f.r > 0.0 ? av / f.r : ar;
                    const double J[9] = {s_ * c * (ao - ar), -s_ * s_ * ar - c * c * ao, -s_ * az,
                                         c * c * ar + s_ * s_ * ao, s_ * c * (ar - ao), c * az,
                                         0.0, 0.0, 0.0};
                    // T J^T T^T t
                    double u[3], v[3], o[3];
                    for (int i = 0; i < 3; ++i)
                        u[i] = S.T[i] * tan[0] + S.T[3 + i] * tan[1] + S.T[6 + i] * tan[2];  // T^T t
                    for (int i = 0; i < 3; ++i)
                        v[i] = J[i] * u[0] + J[3 + i] * u[1] + J[6 + i] * u[2];           // J^T u
                    for (int i = 0; i < 3; ++i)
                        o[i] = S.T[3 * i] * v[0] + S.T[3 * i + 1] * v[1] + S.T[3 * i + 2] * v[2];
                    if (valid)
                        for (int i = 0; i < 3; ++i)
                            part[THREADS * i] += o[i] * w;
                }
                else
                {
                    double H, Z;
                    if (!FP32)
                    {
                        segmentB64<LANES>(h, tt, lt, pt, f, sub, H, Z);
                        H = laneSum<LANES>(H);
                        Z = laneSum<LANES>(Z);
                    }
                    else
                    {
                        const double2 hz = far ? pairB32(h, tt, lt, pn, f.z, f.r)
                                               : pairB64Fast(h, tt, lt, pt, f.z, f.r);
                        H = hz.x;
                        Z = hz.y;
                    }
                    const double vx = H * f.cphi, vy = H * f.sphi;
                    const double B[3] = {S.T[0] * vx + S.T[1] * vy + S.T[2] * Z, S.T[3] * vx + S.T[4] * vy + S.T[5] * Z,
                                         S.T[6] * vx + S.T[7] * vy + S.T[8] * Z};
                    double dF[3], dT[3];
                    cross3(tan, B, dF);
                    for (int i = 0; i < 3; ++i)
                        dF[i] *= w;
                    const double rel[3] = {q[0] - S.sp[0], q[1] - S.sp[1], q[2] - S.sp[2]};
                    cross3(rel, dF, dT);
                    if (valid)
                        for (int i = 0; i < 3; ++i)
                        {
                            part[THREADS * i] += dF[i];
                            part[THREADS * (3 + i)] += dT[i];
                            if (REFINE && far)
                            {
                                scr[(size_t)n * W + i] = dF[i];
                                scr[(size_t)n * W + 3 + i] = dT[i];
                            }
                        }
                }
            };
            // 32 listed nodes (or the last few) in FP64
            auto fp64Batch = [&]() {
                __syncwarp();
                const bool v = lane < nNear;
                node(list[v ? lane : 0], v, 2);
                const int rest = nNear > 32 ? nNear - 32 : 0;
                const int moved = lane < rest ? list[32 + lane] : 0;
                __syncwarp();
                if (lane < rest)
                    list[lane] = moved;
                __syncwarp();
                nNear = rest;
            };
            // REFINE at fraction 0 refines every node: each node in the FP64 forms
            // directly, without the FP32 pass
            const bool allFp64 = REFINE && !(fraction > 0.0);
            if (!FP32)
                for (int n0 = nBegin; n0 < nsec; n0 += STEP)
                    node(n0 + slot < nsec ? n0 + slot : nsec - 1, sub == 0 && n0 + slot < nsec, 0);
            else if (allFp64)
                for (int n0 = nBegin; n0 < nsec; n0 += 32)
                    node(n0 + lane < nsec ? n0 + lane : nsec - 1, n0 + lane < nsec, 2);
            else
                for (int n0 = nBegin; n0 < nsec || nNear > 0;)
                {
                    if (nNear >= 32 || n0 >= nsec)
                        fp64Batch();  // deferred near-field nodes
                    else
                    {
                        node(n0 + lane < nsec ? n0 + lane : nsec - 1, n0 + lane < nsec, 1);
                        n0 += 32;
                    }
                }
            if (REFINE && !allFp64)
            {
                // the primary's totals (every lane), then the dominating nodes in FP64;
                // node n was evaluated, and its contribution stored, by lane n % 32
                if (TEAM > 1)
                {
                    for (int i = 0; i < W; ++i)
                    {
                        const double v = laneSum<32>(part[THREADS * i]);
                        if (lane == 0)
                            teamSums[TEAM > 1 ? threadIdx.x / 32 : 0][i] = v;
                    }
                    __syncthreads();
                }
                double lim[2] = {0.0, 0.0};
                for (int g = 0; g < (QTY == 0 ? 1 : 2); ++g)
                {
                    double n2 = 0.0;
                    for (int i = 0; i < (QTY == 0 ? 1 : 3); ++i)
                    {
                        double v = 0.0;
                        if (TEAM > 1)
                            for (int t = 0; t < TEAM; ++t)
                                v += teamSums[TEAM > 1 ? t : 0][3 * g + i];
                        else
                            v = laneSum<32>(part[THREADS * (3 * g + i)]);
                        n2 += v * v;
                    }
                    lim[g] = fraction * fraction * n2;  // not finite: nothing is picked
                }
                if (TEAM > 1)
                    __syncthreads();  // every warp has read the totals
                for (int b0 = nBegin; b0 < nsec; b0 += 32)
                {
                    const int n = b0 + lane;
                    bool pick = false;
                    if (n < nsec)
                    {
                        double c[W];
                        for (int i = 0; i < W; ++i)
                            c[i] = scr[(size_t)n * W + i];
                        if (QTY == 0)
                            pick = c[0] * c[0] > lim[0];
                        else
                            pick = c[0] * c[0] + c[1] * c[1] + c[2] * c[2] > lim[0] ||
                                   c[3] * c[3] + c[4] * c[4] + c[5] * c[5] > lim[1];
                        if (pick)
                            for (int i = 0; i < W; ++i)
                                part[THREADS * i] -= c[i];
                    }
                    const unsigned bal = __ballot_sync(0xffffffffu, pick);
                    if (pick)
                        list[nNear + __popc(bal & ((1u << lane) - 1u))] = n;
                    nNear += __popc(bal);
                    if (nNear >= 32)
                        fp64Batch();
                }
                while (nNear > 0)
                    fp64Batch();
            }
            const double scale = QTY == 1 ? ph.f_factor : ph.m_factor;
#pragma unroll
            for (int i = 0; i < W; ++i)
            {
                double v = part[THREADS * i];
#pragma unroll
                for (int off = 16; off > 0; off /= 2)
                    v += __shfl_xor_sync(0xffffffffu, v, off);
                if (lane == 0)
                    total[i] += v * scale;
            }
        }
        if (TEAM > 1)
        {
            // warp 0 adds the warps' sums, in order
            __syncthreads();
            if (threadIdx.x == 0)
                for (int t = 1; t < TEAM; ++t)
                    for (int i = 0; i < W; ++i)
                        total[i] += warpSums[TEAM > 1 ? t : 0][i];
            __syncthreads();
        }
        if (lane == 0 && (TEAM == 1 || threadIdx.x == 0))
        {
            double *dst = partial ? partial + W * u : out + W * a;
#pragma unroll
            for (int i = 0; i < W; ++i)
                dst[i] = total[i];
            if (hasZ && !partial)
                zList[atomicAdd(zListCount, 1ull)] = a;
        }
    }
}

// Adds the units of each arrangement, one warp per arrangement, and lists the
// arrangements with a primary left to the z-axis pass.
template <int W>
__global__ void __launch_bounds__(128) pairReduceKernel(const double *__restrict__ partial, int perArr,
                                                        const unsigned char *__restrict__ blob,
                                                        const long long *__restrict__ primOffsets, int nprim,
                                                        const double *__restrict__ primPoses,
                                                        const double *__restrict__ secPoses, long long count,
                                                        double *__restrict__ out,
                                                        const long long *__restrict__ zOffsets,
                                                        long long *__restrict__ zList,
                                                        unsigned long long *__restrict__ zListCount)
{
    const int lane = threadIdx.x % 32;
    const long long warps = (long long)gridDim.x * blockDim.x / 32;
    for (long long a = ((long long)blockIdx.x * blockDim.x + threadIdx.x) / 32; a < count; a += warps)
    {
        double v[W];
#pragma unroll
        for (int i = 0; i < W; ++i)
            v[i] = 0.0;
        for (int k = lane; k < perArr; k += 32)
#pragma unroll
            for (int i = 0; i < W; ++i)
                v[i] += partial[(a * perArr + k) * W + i];
#pragma unroll
        for (int off = 16; off > 0; off /= 2)
#pragma unroll
            for (int i = 0; i < W; ++i)
                v[i] += __shfl_xor_sync(0xffffffffu, v[i], off);
        if (lane == 0)
#pragma unroll
            for (int i = 0; i < W; ++i)
                out[W * a + i] = v[i];
        if (!zOffsets)
            continue;
        bool z = false;
        for (int j = lane; j < nprim; j += 32)
        {
            const PairHeader &ph = *reinterpret_cast<const PairHeader *>(blob + primOffsets[j]);
            double own[5] = {ph.prim.position[0], ph.prim.position[1], ph.prim.position[2], ph.prim_y_angle,
                             ph.prim_z_angle};
            z = z || (zOffsets[j] >= 0 &&
                      zAxisCase(primPoses ? primPoses + 5 * a : own, secPoses + 5 * a, ph.prim.inner_radius));
        }
        if (__any_sync(0xffffffffu, z) && lane == 0)
            zList[atomicAdd(zListCount, 1ull)] = a;
    }
}

// How `count` arrangements are cut into units for warps of which `resident` run
// at once.  `nodes`: the largest secondary cloud; `step`: secondary nodes per
// warp iteration.  One unit per arrangement leaves the last wave nearly empty
// unless there are several waves of them, and the machine idle below one, so
// units are made until there are kPairWaves waves: first groups of primaries,
// then node ranges of equal length (whole iterations) down to one iteration.
// A unit repeats the arrangement's pose set-up (~2 us of one warp, against
// 60 us or more for an iteration of M at PrecisionFactor 5).  Whole calls, before
// and after: one M 745 -> 113 us (with 8 lanes per secondary node; its host work
// takes ~90 us of both), 1,000 parameter gradients 7.5 -> 4.2 ms, 4,099 M (1.7
// waves of whole arrangements) 2.72 -> 2.68 ms.
constexpr long long kPairWaves = 8;
PairSplit pairSplit(long long count, int nprim, int nodes, int step, long long resident)
{
    PairSplit s;
    const long long want = (kPairWaves * resident + count - 1) / count;  // units per arrangement
    if (want <= 1)
        return s;
    s.groups = (int)std::min<long long>(nprim, want);
    const int iters = (nodes + step - 1) / step;
    if (s.groups == nprim && want > nprim)
    {
        const long long parts = std::min<long long>((want + nprim - 1) / nprim, iters);
        const long long each = iters / parts;  // iterations per part, at least
        s.parts = (int)((iters + each - 1) / each);
    }
    return s;
}

void put(std::vector<unsigned char> &blob, const void *p, size_t n)
{
    const unsigned char *c = static_cast<const unsigned char *>(p);
    blob.insert(blob.end(), c, c + n);
}

// The primary's field tables: thickness nodes {r', constant w} with the
// integrator's constant folded in, length nodes {z, w} (slow method) and
// angular nodes {cos, w}, as the reference's field integrators lay them out
// (CalculateFieldsFast.cxx:17-55, CalculateFieldsSlow.cxx:17-66).
void primaryTables(const Coil &prim, const PrecisionArgs &pp, std::vector<double> &pt_, std::vector<double> &pl_,
                   std::vector<double> &pa_)
{
    const bool fast = prim.use_fast_method != 0;
    const double tBlock = prim.thickness / pp.thickness_blocks, aBlock = kPi / pp.angular_blocks;
    const double constant = fast ? kMuReduced * prim.current_density * tBlock * aBlock * 2 * 0.25
                                 : kMuReduced * prim.current_density * (prim.length / pp.length_blocks) * tBlock *
                                       aBlock * 2 * 0.125;
    const double *tx = legendreNodes(pp.thickness_increments), *tw = legendreWeights(pp.thickness_increments);
    for (int b = 0; b < pp.thickness_blocks; ++b)
        for (int i = 0; i < pp.thickness_increments; ++i)
        {
            pt_.push_back(prim.inner_radius + tBlock * (b + 0.5) + (tBlock * 0.5) * tx[i]);
            pt_.push_back(constant * tw[i]);
        }
    if (!fast)
    {
        const double lBlock = prim.length / pp.length_blocks;
        const double *lx = legendreNodes(pp.length_increments), *lw = legendreWeights(pp.length_increments);
        for (int b = 0; b < pp.length_blocks; ++b)
            for (int i = 0; i < pp.length_increments; ++i)
            {
                pl_.push_back(-prim.length * 0.5 + lBlock * (b + 0.5) + (lBlock * 0.5) * lx[i]);
                pl_.push_back(lw[i]);
            }
    }
    const double *ax = legendreNodes(pp.angular_increments), *aw = legendreWeights(pp.angular_increments);
    for (int b = 0; b < pp.angular_blocks; ++b)
        for (int i = 0; i < pp.angular_increments; ++i)
        {
            pa_.push_back(std::cos(aBlock * (b + 0.5) + (aBlock * 0.5) * ax[i]));
            pa_.push_back(aw[i]);
        }
}

// Primary tables as the reference's field integrators lay them out
// (CalculateFieldsFast.cxx:17-55, CalculateFieldsSlow.cxx:17-66), secondary
// cloud as CalculateMInductanceGeneral.cxx:41-103 builds it.
bool buildPair(const Coil &prim, const Coil &sec, const PrecisionArgs &pp, const PrecisionArgs &spa, bool fp32,
               bool units, const PairOptions &opt, std::vector<unsigned char> &blob, std::string &err)
{
    if (!validArgs(pp) || !validArgs(spa))
    {
        err = "pair precision arguments out of range (increments 1..100, blocks >= 1)";
        return false;
    }
    if (!(prim.inner_radius > 0.0) || !(prim.thickness > 0.0) || !(prim.length > 0.0) || !(sec.inner_radius > 0.0) ||
        !(sec.thickness > 0.0) || !(sec.length > 0.0) || prim.current == 0.0)
    {
        err = "coil dimensions must be positive and the primary current non-zero";
        return false;
    }
    const size_t start = blob.size();
    const bool fast = prim.use_fast_method != 0;
    std::vector<double> pt_, pl_, pa_;
    primaryTables(prim, pp, pt_, pl_, pa_);
    // secondary cloud tables
    std::vector<double> sl_, st_;
    std::vector<SecAngular> sa_;
    const double lbs = sec.length / spa.length_blocks, tbs = sec.thickness / spa.thickness_blocks;
    const double *slx = legendreNodes(spa.length_increments), *slw = legendreWeights(spa.length_increments);
    for (int b = 0; b < spa.length_blocks; ++b)
        for (int i = 0; i < spa.length_increments; ++i)
        {
            sl_.push_back(-sec.length * 0.5 + lbs * (b + 0.5) + (lbs * 0.5) * slx[i]);
            sl_.push_back(slw[i]);
        }
    const double *stx = legendreNodes(spa.thickness_increments), *stw = legendreWeights(spa.thickness_increments);
    for (int b = 0; b < spa.thickness_blocks; ++b)
        for (int i = 0; i < spa.thickness_increments; ++i)
        {
            st_.push_back(sec.inner_radius + tbs * (b + 0.5) + (tbs * 0.5) * stx[i]);
            st_.push_back(stw[i]);
        }
    const double *sax = legendreNodes(spa.angular_increments), *saw = legendreWeights(spa.angular_increments);
    for (int b = 0; b < spa.angular_blocks; ++b)
        for (int i = 0; i < spa.angular_increments; ++i)
            sa_.push_back({b + 0.5, sax[i], saw[i], 0.0});

    PairHeader ph;
    std::memset(&ph, 0, sizeof(ph));
    SegmentHeader &h = ph.prim;
    for (int i = 0; i < 3; ++i)
        h.position[i] = prim.position[i];
    std::memcpy(h.transform, prim.transform, sizeof(h.transform));
    std::memcpy(h.inv_transform, prim.inverse_transform, sizeof(h.inv_transform));
    h.half_length = prim.length * 0.5;
    h.field_factor = 1.0;
    h.inner_radius = prim.inner_radius;
    h.n_t = (int)pt_.size() / 2;
    h.n_l = (int)pl_.size() / 2;
    h.n_phi = (int)pa_.size() / 2;
    h.fast = fast ? 1 : 0;
    const int hdr16 = (int)sizeof(PairHeader) / 16;
    h.off_t = hdr16;
    h.off_l = h.off_t + h.n_t;
    h.off_phi = h.off_l + h.n_l;
    ph.s_nl = (int)sl_.size() / 2;
    ph.s_nt = (int)st_.size() / 2;
    ph.s_na = (int)sa_.size();
    ph.s_ablocks = spa.angular_blocks;
    ph.off_sl = h.off_phi + h.n_phi;
    ph.off_st = ph.off_sl + ph.s_nl;
    ph.off_sa = ph.off_st + ph.s_nt;
    std::vector<PhiPair2> p32;
    if (fp32)
    {
        // FP32 angular mirror-pair table (entries of two pairs) after the secondary tables
        std::vector<PhiNode32> single;
        buildPhiPairs32(pp, single);
        packPhiPairs2(single.data(), (int)single.size(), p32);
        h.off_f32 = ph.off_sa + 2 * ph.s_na;
        setNearBox(prim, h);
    }
    // parameter-gradient tables: each node's position per unit of its layer's
    // dimension, {u, 0} (thickness on [0, 1], length on [-1/2, 1/2])
    std::vector<double> tu_, lu_, slu_, stu_;
    if (units)
    {
        auto thicknessUnits = [](const PrecisionArgs &a, std::vector<double> &o) {
            const double *x = legendreNodes(a.thickness_increments);
            for (int b = 0; b < a.thickness_blocks; ++b)
                for (int i = 0; i < a.thickness_increments; ++i)
                    o.insert(o.end(), {((b + 0.5) + 0.5 * x[i]) / a.thickness_blocks, 0.0});
        };
        auto lengthUnits = [](const PrecisionArgs &a, std::vector<double> &o) {
            const double *x = legendreNodes(a.length_increments);
            for (int b = 0; b < a.length_blocks; ++b)
                for (int i = 0; i < a.length_increments; ++i)
                    o.insert(o.end(), {-0.5 + ((b + 0.5) + 0.5 * x[i]) / a.length_blocks, 0.0});
        };
        thicknessUnits(pp, tu_);
        if (!fast)
            lengthUnits(pp, lu_);
        lengthUnits(spa, slu_);
        thicknessUnits(spa, stu_);
        const int base16 = ph.off_sa + 2 * ph.s_na + (int)(sizeof(PhiPair2) / 16 * p32.size());
        ph.off_tu = base16;
        ph.off_lu = ph.off_tu + (int)tu_.size() / 2;
        ph.off_slu = ph.off_lu + (int)lu_.size() / 2;
        ph.off_stu = ph.off_slu + (int)slu_.size() / 2;
    }
    const double blocks = double(spa.length_blocks) * spa.thickness_blocks * spa.angular_blocks;
    ph.m_factor = 2 * kPi * sec.num_turns / prim.current / blocks * opt.scale;
    ph.f_factor = 2 * kPi * (sec.current * sec.num_turns) / blocks * opt.scale;
    ph.full_ring = opt.full_ring ? 1 : 0;
    ph.prim_y_angle = prim.y_axis_angle;
    ph.prim_z_angle = prim.z_axis_angle;
    put(blob, &ph, sizeof(ph));
    put(blob, pt_.data(), sizeof(double) * pt_.size());
    put(blob, pl_.data(), sizeof(double) * pl_.size());
    put(blob, pa_.data(), sizeof(double) * pa_.size());
    put(blob, sl_.data(), sizeof(double) * sl_.size());
    put(blob, st_.data(), sizeof(double) * st_.size());
    put(blob, sa_.data(), sizeof(SecAngular) * sa_.size());
    put(blob, p32.data(), sizeof(PhiPair2) * p32.size());
    put(blob, tu_.data(), sizeof(double) * tu_.size());
    put(blob, lu_.data(), sizeof(double) * lu_.size());
    put(blob, slu_.data(), sizeof(double) * slu_.size());
    put(blob, stu_.data(), sizeof(double) * stu_.size());
    (void)start;
    return true;
}

#include "zaxis.cuh"

// Stream-ordered temporary from the library's memory pool: no device-wide
// synchronisation and no driver mapping work per call
struct DevBuf
{
    void *p = nullptr;
    cudaStream_t st = nullptr;
    cudaError_t alloc(size_t bytes, cudaStream_t s)
    {
        st = s;
        return scratchAlloc(&p, bytes, s);
    }
    ~DevBuf()
    {
        if (p)
            cudaFreeAsync(p, st);
    }
};

// poses and results up to this size share a copy with a call's tables and counters
constexpr size_t kPackedBytes = size_t(1) << 16;

void packHostPoses(const PoseSource &s, long long n, double *dst)
{
    if (s.packed)
    {
        std::memcpy(dst, s.packed, sizeof(ccoil_pose_t) * (size_t)n);
        return;
    }
    for (long long i = 0; i < n; ++i)
    {
        for (int k = 0; k < 3; ++k)
            dst[5 * i + k] = s.position[3 * i + k];
        dst[5 * i + 3] = s.yAngle[i];
        dst[5 * i + 4] = s.zAngle[i];
    }
}
} // namespace

int cudaFail(cudaError_t e, const char *what);
} // namespace ccoil

using namespace ccoil;

int ccoil::pairArrangements(const ccoil_coil_t *primaries, int primary_count, const ccoil_coil_t *secondary,
                            const ccoil_precision_args_t *secondary_precisions,
                            const ccoil_precision_args_t *zaxis_precisions, const PoseSource &prim,
                            const PoseSource &sec, long long count, int quantity, int precision, double *out,
                            long long *z_axis_count, int memory, void *stream, const PairOptions &opt)
{
    const bool havePrim = prim.given(), split_poses = sec.position != nullptr || prim.position != nullptr;
    if (primary_count < 0 || (primary_count > 0 && (!primaries || !secondary_precisions)) || !secondary)
        return failMessage(CCOIL_ERR_INVALID_ARGUMENT, "null coils or negative primary_count");
    if (count < 0 || (count > 0 && (!sec.given() || !out)))
        return failMessage(CCOIL_ERR_INVALID_ARGUMENT, "count < 0 or null poses/out");
    if (havePrim && primary_count != 1)
        return failMessage(CCOIL_ERR_INVALID_ARGUMENT, "per-arrangement primary poses need exactly one primary");
    if (quantity != CCOIL_PAIR_MUTUAL_INDUCTANCE && quantity != CCOIL_PAIR_FORCE_TORQUE &&
        quantity != CCOIL_PAIR_MUTUAL_INDUCTANCE_GRADIENT && quantity != CCOIL_PAIR_MUTUAL_INDUCTANCE_PARAMETER_GRADIENT)
        return failMessage(CCOIL_ERR_INVALID_ARGUMENT, "unknown pair quantity");
    if (quantity == CCOIL_PAIR_MUTUAL_INDUCTANCE_PARAMETER_GRADIENT && count > 0 && (primary_count != 1 || !havePrim))
        return failMessage(CCOIL_ERR_INVALID_ARGUMENT,
                           "the parameter gradient needs exactly one primary with per-arrangement poses");
    if (precision != CCOIL_PRECISION_FP64 && precision != CCOIL_PRECISION_FP32_COMPENSATED &&
        precision != CCOIL_PRECISION_FP32_REFINED)
        return failMessage(CCOIL_ERR_INVALID_ARGUMENT, "unknown precision mode");
    if (precision == CCOIL_PRECISION_FP32_COMPENSATED && quantity == CCOIL_PAIR_MUTUAL_INDUCTANCE_GRADIENT)
        return failMessage(CCOIL_ERR_NOT_SUPPORTED,
                           "the position gradient is evaluated in FP64 only (the parameter gradient has an FP32 form)");
    if (precision == CCOIL_PRECISION_FP32_REFINED && quantity != CCOIL_PAIR_MUTUAL_INDUCTANCE &&
        quantity != CCOIL_PAIR_FORCE_TORQUE)
        return failMessage(CCOIL_ERR_NOT_SUPPORTED, "FP32_REFINED covers mutual inductance and force/torque");
    const bool fp32 = precision != CCOIL_PRECISION_FP64;
    const bool refine = precision == CCOIL_PRECISION_FP32_REFINED;
    if (memory != CCOIL_MEMORY_HOST && memory != CCOIL_MEMORY_DEVICE)
        return failMessage(CCOIL_ERR_INVALID_ARGUMENT, "memory must be HOST or DEVICE");
    if (z_axis_count)
        *z_axis_count = 0;
    const int width = quantity == CCOIL_PAIR_MUTUAL_INDUCTANCE            ? 1
                      : quantity == CCOIL_PAIR_FORCE_TORQUE               ? 6
                      : quantity == CCOIL_PAIR_MUTUAL_INDUCTANCE_GRADIENT ? 3
                                                                          : 14;
    if (count == 0)
        return CCOIL_OK;
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    if (primary_count == 0)
    {
        cudaError_t e = memory == CCOIL_MEMORY_HOST ? cudaSuccess : cudaMemsetAsync(out, 0, sizeof(double) * width * count, st);
        if (memory == CCOIL_MEMORY_HOST)
            std::memset(out, 0, sizeof(double) * width * count);
        return e == cudaSuccess ? CCOIL_OK : cudaFail(e, "memset");
    }

    std::vector<unsigned char> blob;
    std::vector<long long> offsets;
    std::string err;
    for (int j = 0; j < primary_count; ++j)
    {
        offsets.push_back((long long)blob.size());
        if (!buildPair(primaries[j], *secondary, primaries[j].precision, secondary_precisions[j], fp32,
                       quantity == CCOIL_PAIR_MUTUAL_INDUCTANCE_PARAMETER_GRADIENT, opt, blob, err))
            return fail(CCOIL_ERR_INVALID_ARGUMENT, "primary " + std::to_string(j) + ": " + err);
    }
    const size_t generalBytes = blob.size();
    // coaxial pairs: the z-axis tables of every primary (M and F/T only)
    const bool zPass = zaxis_precisions && (quantity == CCOIL_PAIR_MUTUAL_INDUCTANCE ||
                                            quantity == CCOIL_PAIR_FORCE_TORQUE);
    std::vector<long long> zOffsets(primary_count, -1);
    if (zPass)
        for (int j = 0; j < primary_count; ++j)
        {
            zOffsets[j] = (long long)blob.size();
            if (!buildZAxis(primaries[j], *secondary, zaxis_precisions[2 * j], zaxis_precisions[2 * j + 1], blob, err))
                return fail(CCOIL_ERR_INVALID_ARGUMENT, "primary " + std::to_string(j) + ": " + err);
        }
    // One block of device memory for the call.  First what is uploaded, in one copy:
    // tables, offsets, the two z-axis counters (zero) and the poses, unless they are a
    // large array that can be copied as it is; after them the results, so that few results come back in one copy with
    // the counters; then what stays on the device.
    const bool host = memory == CCOIL_MEMORY_HOST;
    const size_t poseBytes = sizeof(ccoil_pose_t) * (size_t)count, outBytes = sizeof(double) * width * (size_t)count;
    const bool packPoses = host && (split_poses || poseBytes <= kPackedBytes), packOut = host && outBytes <= kPackedBytes;
    size_t arenaBytes = 0;
    auto region = [&](size_t bytes) {
        const size_t at = arenaBytes;
        arenaBytes += (bytes + 255) / 256 * 256;
        return at;
    };
    const size_t atBlob = region(blob.size()), atOff = region(sizeof(long long) * offsets.size()),
                 atZOff = region(sizeof(long long) * zOffsets.size());
    const size_t atSec = packPoses ? region(poseBytes) : 0, atPrim = packPoses && havePrim ? region(poseBytes) : 0;
    const size_t atCount = region(2 * sizeof(unsigned long long)), uploadBytes = arenaBytes;
    const size_t atOut = region(host ? outBytes : 0), atZList = region(zPass ? sizeof(long long) * count : 0);
    const size_t atBigSec = region(host && !packPoses ? poseBytes : 0);
    const size_t atBigPrim = region(host && !packPoses && havePrim ? poseBytes : 0);
    int secNodes = 0;
    for (long long off : offsets)
    {
        const PairHeader *ph = reinterpret_cast<const PairHeader *>(blob.data() + off);
        secNodes = std::max(secNodes, ph->s_nl * ph->s_nt * ph->s_na);
    }
    // work units (the refining kernel needs a primary's whole total in one warp or CTA)
    const long long resident = 148LL * 4 * pairMinBlocks(quantity, fp32, refine);
    PairSplit split;
    int lanes = 1;
    if (!refine)
    {
        // fewer warp iterations in all than resident warps: 8 lanes share a secondary
        // node (not for the parameter gradient, some of whose columns vanish by
        // symmetry: a node evaluated by one lane leaves the same rounding in them
        // however the arrangement is cut)
        if (!fp32 && quantity != CCOIL_PAIR_MUTUAL_INDUCTANCE_PARAMETER_GRADIENT && count * primary_count * ((secNodes + 31) / 32) < resident)
            lanes = 8;
        split = pairSplit(count, primary_count, secNodes, 32 / lanes, resident);
    }
    // the refining kernel shares few arrangements among the warps of a CTA: 12 while
    // every arrangement then has a resident CTA, else 4 up to three waves of whole
    // arrangements (each warp's last FP64 batch of 32 nodes is partly empty).  Whole
    // calls with 1, 4 and 12 warps: M of 445 arrangements 1.36, 0.53 and 0.38 ms, 2,000
    // 1.62, 0.98 and 0.96, 15,984 5.28, 5.22 and 6.04, 20,000 6.35, 6.54 and 7.58; F/T of
    // 1,000 0.94, 0.46 and 0.40 ms, 2,000 1.14, 0.70 and 0.67, 20,000 4.79, 4.47 and 5.14
    const int team = !refine ? 1 : count <= 148LL * 3 ? 12 : count <= resident * 3 ? 4 : 1;
    const long long perArr = (long long)split.groups * split.parts;
    const size_t atPartial = region(perArr > 1 ? sizeof(double) * (size_t)width * (size_t)(count * perArr) : 0);
    long long blocks = team > 1 ? count : (count * perArr + 3) / 4;
    if (blocks > 148LL * 64)
        blocks = 148LL * 64;
    // FP32_REFINED: every warp's region of node contributions (the grid strides over
    // the arrangements, so the scratch is sized by the grid, not by the count)
    const int scratchNodes = refine ? secNodes : 0;
    size_t scratchBytes = 0;
    if (refine)
    {
        // at most kPairRefineScratchBytes: a secondary with many nodes runs on fewer
        // warps (each keeps 1 or 6 doubles per node), never fewer than one CTA per SM
        const size_t perBlock = sizeof(double) * (size_t)width * (size_t)scratchNodes * (team > 1 ? 1 : 4);
        const long long fit = (long long)(kPairRefineScratchBytes / perBlock);
        blocks = std::max(1LL, std::min(blocks, std::max(fit, 148LL)));
        scratchBytes = perBlock * (size_t)blocks;
    }
    const size_t atScratch = region(scratchBytes);
    DevBuf arena;
    cudaError_t e = arena.alloc(arenaBytes, st);
    if (e != cudaSuccess)
        return cudaFail(e, "device memory of the call");
    unsigned char *base = static_cast<unsigned char *>(arena.p);
    const size_t backBytes = packOut ? atOut - atCount + outBytes : 0;  // counters and results
    std::unique_ptr<unsigned char[]> image(new (std::nothrow) unsigned char[std::max(uploadBytes, backBytes)]);
    if (!image)
        return failMessage(CCOIL_ERR_OUT_OF_MEMORY, "host allocation failed");
    std::memcpy(image.get() + atBlob, blob.data(), blob.size());
    std::memcpy(image.get() + atOff, offsets.data(), sizeof(long long) * offsets.size());
    std::memcpy(image.get() + atZOff, zOffsets.data(), sizeof(long long) * zOffsets.size());
    std::memset(image.get() + atCount, 0, 2 * sizeof(unsigned long long));
    if (packPoses)
    {
        packHostPoses(sec, count, reinterpret_cast<double *>(image.get() + atSec));
        if (havePrim)
            packHostPoses(prim, count, reinterpret_cast<double *>(image.get() + atPrim));
    }
    e = cudaMemcpyAsync(base, image.get(), uploadBytes, cudaMemcpyHostToDevice, st);
    const double *secP = sec.packed, *primP = prim.packed;
    if (host)
    {
        secP = reinterpret_cast<const double *>(base + (packPoses ? atSec : atBigSec));
        primP = havePrim ? reinterpret_cast<const double *>(base + (packPoses ? atPrim : atBigPrim)) : nullptr;
        if (e == cudaSuccess && !packPoses)
            e = cudaMemcpyAsync(base + atBigSec, sec.packed, poseBytes, cudaMemcpyHostToDevice, st);
        if (e == cudaSuccess && !packPoses && havePrim)
            e = cudaMemcpyAsync(base + atBigPrim, prim.packed, poseBytes, cudaMemcpyHostToDevice, st);
    }
    if (e != cudaSuccess)
        return cudaFail(e, "host->device copy");
    double *o = host ? reinterpret_cast<double *>(base + atOut) : out;
    // one primary whose tables fit: stage them in shared memory
    const int stagedBytes = (primary_count == 1 && generalBytes <= CCOIL_PAIR_STAGE_MAX_BYTES &&
                             generalBytes % 16 == 0)
                                ? (int)generalBytes
                                : 0;
    const double fraction = refineFraction();
    auto *scratch = reinterpret_cast<double *>(base + atScratch);
    auto *partial = perArr > 1 ? reinterpret_cast<double *>(base + atPartial) : nullptr;
    auto *zc = reinterpret_cast<unsigned long long *>(base + atCount), *zN = zc + 1;
    const unsigned char *dB = base + atBlob;
    const auto *dO = reinterpret_cast<const long long *>(base + atOff);
    const size_t smem = (size_t)stagedBytes;
    const auto *zO = zPass ? reinterpret_cast<const long long *>(base + atZOff) : nullptr;
    auto *zL = reinterpret_cast<long long *>(base + atZList);
    // beyond 48 KiB together with the kernel's own shared memory, the staged tables
    // have to be asked for
    const bool beyondDefault = smem + pairStaticBytes(width, team) > size_t(48) * 1024;
#define CCOIL_PAIR_LAUNCH(Q, F, ...)                                                                                   \
    do                                                                                                                 \
    {                                                                                                                  \
        if (beyondDefault)                                                                                             \
            cudaFuncSetAttribute(pairKernel64<Q, F, ##__VA_ARGS__>, cudaFuncAttributeMaxDynamicSharedMemorySize,      \
                                 CCOIL_PAIR_STAGE_MAX_BYTES);                                                          \
        pairKernel64<Q, F, ##__VA_ARGS__><<<(unsigned)blocks, pairThreads(team), smem, st>>>(                          \
            dB, dO, primary_count, primP, secP, count, o, zc, stagedBytes, zO, zL, zN, scratch, scratchNodes, fraction, \
            split, partial);                                                                                           \
    } while (0)
    if (quantity == CCOIL_PAIR_MUTUAL_INDUCTANCE && !fp32 && lanes == 8)
        CCOIL_PAIR_LAUNCH(0, false, false, 8);
    else if (quantity == CCOIL_PAIR_FORCE_TORQUE && !fp32 && lanes == 8)
        CCOIL_PAIR_LAUNCH(1, false, false, 8);
    else if (quantity == CCOIL_PAIR_MUTUAL_INDUCTANCE_GRADIENT && lanes == 8)
        CCOIL_PAIR_LAUNCH(2, false, false, 8);
    else if (quantity == CCOIL_PAIR_MUTUAL_INDUCTANCE && !fp32)
        CCOIL_PAIR_LAUNCH(0, false);
    else if (quantity == CCOIL_PAIR_MUTUAL_INDUCTANCE && refine && team == 12)
        CCOIL_PAIR_LAUNCH(0, true, true, 1, 12);
    else if (quantity == CCOIL_PAIR_MUTUAL_INDUCTANCE && refine && team == 4)
        CCOIL_PAIR_LAUNCH(0, true, true, 1, 4);
    else if (quantity == CCOIL_PAIR_FORCE_TORQUE && refine && team == 12)
        CCOIL_PAIR_LAUNCH(1, true, true, 1, 12);
    else if (quantity == CCOIL_PAIR_FORCE_TORQUE && refine && team == 4)
        CCOIL_PAIR_LAUNCH(1, true, true, 1, 4);
    else if (quantity == CCOIL_PAIR_MUTUAL_INDUCTANCE && refine)
        CCOIL_PAIR_LAUNCH(0, true, true);
    else if (quantity == CCOIL_PAIR_MUTUAL_INDUCTANCE)
        CCOIL_PAIR_LAUNCH(0, true);
    else if (quantity == CCOIL_PAIR_FORCE_TORQUE && !fp32)
        CCOIL_PAIR_LAUNCH(1, false);
    else if (quantity == CCOIL_PAIR_FORCE_TORQUE && refine)
        CCOIL_PAIR_LAUNCH(1, true, true);
    else if (quantity == CCOIL_PAIR_FORCE_TORQUE)
        CCOIL_PAIR_LAUNCH(1, true);
    else if (quantity == CCOIL_PAIR_MUTUAL_INDUCTANCE_GRADIENT)
        CCOIL_PAIR_LAUNCH(2, false);
    else if (!fp32)
        CCOIL_PAIR_LAUNCH(3, false);
    else
        CCOIL_PAIR_LAUNCH(3, true);
#undef CCOIL_PAIR_LAUNCH
    e = cudaGetLastError();
    if (e == cudaSuccess && partial)
    {
        const unsigned grid = (unsigned)std::min<long long>((count + 3) / 4, 148LL * 16);
#define CCOIL_PAIR_REDUCE(W)                                                                                        \
    pairReduceKernel<W><<<grid, 128, 0, st>>>(partial, (int)perArr, dB, dO, primary_count, primP, secP, count, o,   \
                                              zPass ? zO : nullptr, zL, zN)
        if (width == 1)
            CCOIL_PAIR_REDUCE(1);
        else if (width == 3)
            CCOIL_PAIR_REDUCE(3);
        else if (width == 6)
            CCOIL_PAIR_REDUCE(6);
        else
            CCOIL_PAIR_REDUCE(14);
#undef CCOIL_PAIR_REDUCE
        e = cudaGetLastError();
    }
    if (e == cudaSuccess && zPass)
    {
        // the z-axis pass: one warp per recorded arrangement
        if (quantity == CCOIL_PAIR_MUTUAL_INDUCTANCE)
            zAxisKernel<0><<<148 * 8, 128, 0, st>>>(dB, dO, zO, primary_count, primP, secP, zL, zN, o);
        else
            zAxisKernel<1><<<148 * 8, 128, 0, st>>>(dB, dO, zO, primary_count, primP, secP, zL, zN, o);
        e = cudaGetLastError();
    }
    if (e != cudaSuccess)
        return cudaFail(e, "pair kernel launch");
    // the call is synchronous, as the reference's: host outputs and the z-axis count
    unsigned long long zcount = 0;
    if (packOut)
    {
        e = cudaMemcpyAsync(image.get(), base + atCount, backBytes, cudaMemcpyDeviceToHost, st);
    }
    else
    {
        if (host)
            e = cudaMemcpyAsync(out, o, outBytes, cudaMemcpyDeviceToHost, st);
        if (e == cudaSuccess)
            e = cudaMemcpyAsync(&zcount, zc, sizeof(zcount), cudaMemcpyDeviceToHost, st);
    }
    if (e == cudaSuccess)
        e = cudaStreamSynchronize(st);
    if (e != cudaSuccess)
        return cudaFail(e, "pair arrangements");
    if (packOut)
    {
        std::memcpy(&zcount, image.get(), sizeof(zcount));
        std::memcpy(out, image.get() + (atOut - atCount), outBytes);
    }
    if (z_axis_count)
        *z_axis_count = (long long)zcount;
    return CCOIL_OK;
}

extern "C" int ccoil_pair_arrangements_zaxis(const ccoil_coil_t *primaries, int primary_count,
                                             const ccoil_coil_t *secondary,
                                             const ccoil_precision_args_t *secondary_precisions,
                                             const ccoil_precision_args_t *zaxis_precisions,
                                             const ccoil_pose_t *primary_poses, const ccoil_pose_t *secondary_poses,
                                             long long count, int quantity, int precision, double *out,
                                             long long *z_axis_count, int memory, void *stream)
{
    PoseSource prim, sec;
    prim.packed = reinterpret_cast<const double *>(primary_poses);
    sec.packed = reinterpret_cast<const double *>(secondary_poses);
    return pairArrangements(primaries, primary_count, secondary, secondary_precisions, zaxis_precisions, prim, sec,
                            count, quantity, precision, out, z_axis_count, memory, stream, PairOptions{});
}

extern "C" int ccoil_pair_arrangements_arrays(const ccoil_coil_t *primaries, int primary_count,
                                              const ccoil_coil_t *secondary,
                                              const ccoil_precision_args_t *secondary_precisions,
                                              const ccoil_precision_args_t *zaxis_precisions,
                                              const ccoil_pose_arrays_t *primary_poses,
                                              const ccoil_pose_arrays_t *secondary_poses, long long count,
                                              int quantity, int precision, double *out, long long *z_axis_count,
                                              void *stream)
{
    auto source = [](const ccoil_pose_arrays_t *a) {
        PoseSource s;
        if (a && a->position && a->y_angle && a->z_angle)
        {
            s.position = a->position;
            s.yAngle = a->y_angle;
            s.zAngle = a->z_angle;
        }
        return s;
    };
    const PoseSource prim = source(primary_poses), sec = source(secondary_poses);
    if (primary_poses && count > 0 && !prim.given())
        return failMessage(CCOIL_ERR_INVALID_ARGUMENT, "null primary pose arrays");
    return pairArrangements(primaries, primary_count, secondary, secondary_precisions, zaxis_precisions, prim, sec,
                            count, quantity, precision, out, z_axis_count, CCOIL_MEMORY_HOST, stream, PairOptions{});
}

extern "C" int ccoil_pair_arrangements(const ccoil_coil_t *primaries, int primary_count, const ccoil_coil_t *secondary,
                                       const ccoil_precision_args_t *secondary_precisions,
                                       const ccoil_pose_t *primary_poses, const ccoil_pose_t *secondary_poses,
                                       long long count, int quantity, int precision, double *out,
                                       long long *z_axis_count, int memory, void *stream)
{
    return ccoil_pair_arrangements_zaxis(primaries, primary_count, secondary, secondary_precisions, nullptr,
                                         primary_poses, secondary_poses, count, quantity, precision, out,
                                         z_axis_count, memory, stream);
}
