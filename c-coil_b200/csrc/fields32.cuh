// FP32-compensated field kernels (included by fields.cu inside its anonymous
// namespace, so they share the staging pipeline and the FP64 integrands);
// the integrands themselves are in integrands32.cuh.
//
// Near field.  A point inside a coil's winding box (inflated by a margin) is
// left out by the FP32 loop.  A second kernel lists such (point, segment) pairs,
// a point's pairs next to each other and in segment order, and a third evaluates
// them with the FP64 integrands, so warps never diverge between the two paths.
// A warp evaluates a pair, and a point's pairs are added in order: results repeat
// exactly however the FP32 pass is cut into pieces, and a point that lies in many
// windings' boxes does not wait for one warp.  If the list is too short for all pairs,
// the third kernel finds them itself, a warp per point.
//
// FP32_REFINED.  The FP32 kernel also stores every (point, segment)
// contribution; once the point's total is known, a selection kernel removes
// each contribution whose norm exceeds a set fraction of the total's norm
// (the contributions that dominate a point where the coils' fields cancel,
// whose FP32 errors the cancellation magnifies) and lists the pair, and the
// near-field kernel adds those pairs back evaluated with the FP64 integrands.

#include "integrands32.cuh"
#include "integrands64f.cuh"

// Integrates one segment for one lane and adds the lane's contribution to acc.
template <int FIELD, int LANES>
__device__ __forceinline__ void integrateSegment32(const unsigned char *seg, const Frame &f, int lane, double *acc,
                                                   Slice th = Slice())
{
    const SegmentHeader &h = *reinterpret_cast<const SegmentHeader *>(seg);
    const double2 *tt = reinterpret_cast<const double2 *>(seg) + h.off_t;
    const double2 *lt = reinterpret_cast<const double2 *>(seg) + h.off_l;
    const PhiPair2 *pn = reinterpret_cast<const PhiPair2 *>(reinterpret_cast<const double2 *>(seg) + h.off_f32);
    if (FIELD == CCOIL_FIELD_B)
    {
        double H, Z;
        segmentB32<LANES>(h, tt, lt, pn, f, lane, H, Z, th);
        addRotated(h, H * f.cphi, H * f.sphi, Z, acc);
    }
    else if (FIELD == CCOIL_FIELD_G)
    {
        double g[4];
        segmentG32<LANES>(h, tt, lt, pn, f, lane, g, th);
        addGradient(h, f, g, acc);
    }
    else
    {
        double a = segmentA32<LANES>(h, tt, lt, pn, f, lane, th) * h.field_factor;
        addRotated(h, -a * f.sphi, a * f.cphi, 0.0, acc);
    }
}

// Near-field work list entry: (point, segment)
struct NearPair
{
    int point;
    int segment;
};
// Its run, where the third kernel adds up the runs itself: the entries of one point, and,
// with the run's first entry, how many of them have been evaluated
struct NearRun
{
    int first, count, done;
};

// CTAs per SM the register allocation targets (128 threads each): the packed
// FP32 integrands hold two mirror pairs per value, and these are the highest
// occupancies at which they compile without spills -- 5 for the vector
// potential (96 registers), 4 for the field and the gradient (128 registers)
#ifndef CCOIL_FP32_MIN_BLOCKS_A
#define CCOIL_FP32_MIN_BLOCKS_A 5
#endif
#ifndef CCOIL_FP32_MIN_BLOCKS_B
#define CCOIL_FP32_MIN_BLOCKS_B 4
#endif
#ifndef CCOIL_FP32_MIN_BLOCKS_G
#define CCOIL_FP32_MIN_BLOCKS_G 4
#endif
constexpr int fp32MinBlocks(int field)
{
    return field == CCOIL_FIELD_B ? CCOIL_FP32_MIN_BLOCKS_B
                                  : (field == CCOIL_FIELD_G ? CCOIL_FP32_MIN_BLOCKS_G : CCOIL_FP32_MIN_BLOCKS_A);
}
// 1: segments are staged into shared memory by bulk copies (double-buffered,
// one CTA barrier per segment); 0 (default, 1.9x faster on B200): each warp
// reads the segment tables from global memory through L1 -- the same table
// bytes are read by every warp of the SM, so they stay L1/L2-resident -- and
// warps never wait for each other
#ifndef CCOIL_FP32_STAGE
#define CCOIL_FP32_STAGE 0
#endif

// Whether the field kernel clears the near-field list's counter, which saves a launch (2
// of 24 us for 2 coils at 37 points).  Not the refined gradient's: the compiler then gives
// its loops other registers (128 coils at 65,536 points 9.89 -> 10.05 ms).
constexpr bool clearsNearCount(int field, bool refine) { return !(refine && field == CCOIL_FIELD_G); }

// REFINE (FP32_REFINED): every (point, segment) contribution is also written
// to contrib, segment-major ([segment][point][W], so a warp's stores for one
// segment are contiguous), near-field pairs as zeros (they are FP64 already)
template <int FIELD, int LANES, bool REFINE>
__global__ void __launch_bounds__(128, fp32MinBlocks(FIELD)) fieldsKernel32(const unsigned char *__restrict__ blob,
                                                      const SegmentDesc *__restrict__ segs, int nseg,
                                                      const double *__restrict__ points, long long npts,
                                                      double *__restrict__ out, double *__restrict__ contrib,
                                                      FieldSplit split,
                                                      double *__restrict__ partial,
                                                      unsigned long long *__restrict__ workCount)
{
    constexpr int W = FIELD == CCOIL_FIELD_G ? 9 : 3;
    extern __shared__ __align__(128) unsigned char smem[];
    __shared__ __align__(8) unsigned long long bars[kSegmentStages];
    __shared__ int timedOut;
    if (clearsNearCount(FIELD, REFINE) && blockIdx.x == 0 && blockIdx.y == 0 && threadIdx.x == 0)
        *workCount = 0;

    const int lane = threadIdx.x % LANES;
    const long long p = (long long)blockIdx.x * (blockDim.x / LANES) + threadIdx.x / LANES;
    const bool active = p < npts;

#if CCOIL_FP32_STAGE
    if (threadIdx.x == 0)
    {
        timedOut = 0;
        for (int s = 0; s < kSegmentStages; ++s)
            mbarInit(&bars[s], 1);
        fenceBarrierInit();
        for (int s = 0; s < kSegmentStages && s < nseg; ++s)
            stageSegment(smem + s * kSegmentBytes, blob + segs[s].offset, (unsigned)segs[s].bytes, &bars[s]);
    }
    __syncthreads();
#endif

    double px = 0.0, py = 0.0, pz = 0.0;
    if (active)
    {
        px = points[3 * p];
        py = points[3 * p + 1];
        pz = points[3 * p + 2];
    }
    // the sums of the gradient, and of the field where it is not refined, live in
    // shared memory, one column per thread: in registers they crowd the loops at 128
    // (128 coils: G at 2^17 points 17.1 ms against 19.0, B at 200,003 points 21.9
    // against 22.35; the vector potential measured 0.5 % slower this way)
    constexpr bool kShared = FIELD == CCOIL_FIELD_G || (FIELD == CCOIL_FIELD_B && !REFINE);
    __shared__ double sums[kShared ? W : 1][kShared ? 128 : 1];
    double acc[W];
#pragma unroll
    for (int i = 0; i < W; ++i)
    {
        acc[i] = 0.0;
        if (kShared)
            sums[kShared ? i : 0][kShared ? threadIdx.x : 0] = 0.0;
    }
    // this block's piece of the work (FieldSplit)
    const int piece = blockIdx.y, group = piece / split.parts;
    const Slice th = {piece - group * split.parts, split.parts};
    const int sBegin = (int)((long long)nseg * group / split.groups);
    const int sEnd = (int)((long long)nseg * (group + 1) / split.groups);
    // the lanes of one point
    auto groupMask = [] {
        return LANES == 32 ? 0xffffffffu : (((1u << LANES) - 1u) << ((threadIdx.x % 32) / LANES * LANES));
    };

    for (int s = sBegin; s < sEnd; ++s)
    {
#if CCOIL_FP32_STAGE
        const int stage = s % kSegmentStages;
        const unsigned parity = (unsigned)((s / kSegmentStages) & 1);
        const bool ok = mbarWait(&bars[stage], parity);
        if (!ok)
            timedOut = 1;
        const unsigned char *seg = smem + stage * kSegmentBytes;
#else
        const bool ok = true;
        const unsigned char *seg = blob + segs[s].offset;
#endif
        if (active && ok)
        {
            const SegmentHeader &h = *reinterpret_cast<const SegmentHeader *>(seg);
            const Frame f = toCoilFrame(h, px, py, pz);
            const bool nearPair = nearWinding(h, f);
            if (!nearPair && kShared && !REFINE)
            {
                double c[W];
#pragma unroll
                for (int i = 0; i < W; ++i)
                    c[i] = 0.0;
                integrateSegment32<FIELD, LANES>(seg, f, lane, c, th);
#pragma unroll
                for (int i = 0; i < W; ++i)
                    sums[kShared ? i : 0][kShared ? threadIdx.x : 0] += c[i];
            }
            else if (!nearPair && !REFINE)
                integrateSegment32<FIELD, LANES>(seg, f, lane, acc, th);
            else if (!nearPair)
            {
                // the segment's contribution on its own: combined over the point's
                // lanes (all of them take this branch), added to the total by lane 0
                // and stored for the selection
                double c[W];
#pragma unroll
                for (int i = 0; i < W; ++i)
                    c[i] = 0.0;
                integrateSegment32<FIELD, LANES>(seg, f, lane, c);
#pragma unroll
                for (int off = LANES / 2; off > 0; off /= 2)
#pragma unroll
                    for (int i = 0; i < W; ++i)
                        c[i] += __shfl_xor_sync(groupMask(), c[i], off);
                if (lane == 0)
                {
                    double *dst = contrib + ((size_t)s * (size_t)npts + (size_t)p) * W;
#pragma unroll
                    for (int i = 0; i < W; ++i)
                    {
                        if (kShared)
                            sums[kShared ? i : 0][kShared ? threadIdx.x : 0] += c[i];
                        else
                            acc[i] += c[i];
                        dst[i] = c[i];
                    }
                }
            }
            else if (REFINE && lane == 0)
            {
                double *dst = contrib + ((size_t)s * (size_t)npts + (size_t)p) * W;
#pragma unroll
                for (int i = 0; i < W; ++i)
                    dst[i] = 0.0;
            }
        }
#if CCOIL_FP32_STAGE
        __syncthreads();
        if (timedOut)
        {
            // a stage never arrived: drain what is in flight (bounded) and leave
            if (threadIdx.x == 0)
            {
                atomicAdd(&g_timeouts, 1ull);
                int last = min(s + kSegmentStages - 1, nseg - 1);
                for (int t = 0; t < kSegmentStages; ++t)
                {
                    int j = last - ((last - t) % kSegmentStages + kSegmentStages) % kSegmentStages;
                    if (j >= s)
                        mbarWait(&bars[t], (unsigned)((j / kSegmentStages) & 1));
                }
            }
            return;
        }
        if (threadIdx.x == 0 && s + kSegmentStages < nseg)
            stageSegment(smem + stage * kSegmentBytes, blob + segs[s + kSegmentStages].offset,
                         (unsigned)segs[s + kSegmentStages].bytes, &bars[stage]);
#endif
    }

    if (kShared)
#pragma unroll
        for (int i = 0; i < W; ++i)
            acc[i] = sums[kShared ? i : 0][kShared ? threadIdx.x : 0];
#pragma unroll
    for (int off = LANES / 2; off > 0; off /= 2)
#pragma unroll
        for (int i = 0; i < W; ++i)
            acc[i] += __shfl_xor_sync(0xffffffffu, acc[i], off);
    if (active && lane == 0)
    {
        double *dst = partial ? partial + ((size_t)piece * (size_t)npts + (size_t)p) * W : out + W * p;
#pragma unroll
        for (int i = 0; i < W; ++i)
            dst[i] = acc[i];
    }
}

// Whether a point lies in a segment's near box: nearWinding on toCoilFrame, operation
// for operation, but the radius (a square root) only where the height is in range
__device__ __forceinline__ bool isNearPair(const unsigned char *blob, const SegmentDesc *segs, int s, double px,
                                           double py, double pz)
{
    const SegmentHeader &h = *reinterpret_cast<const SegmentHeader *>(blob + segs[s].offset);
    const double *M = h.inv_transform;
    const double dx = sub(px, h.position[0]), dy = sub(py, h.position[1]), dz = sub(pz, h.position[2]);
    const double z = add(add(mul(M[6], dx), mul(M[7], dy)), mul(M[8], dz));
    if (!(z > h.near_lo[1] && z < h.near_hi[1]))
        return false;
    const double x = add(add(mul(M[0], dx), mul(M[1], dy)), mul(M[2], dz));
    const double y = add(add(mul(M[3], dx), mul(M[4], dy)), mul(M[5], dz));
    const double r = sqr(add(mul(x, x), mul(y, y)));
    return r > h.near_lo[0] && r < h.near_hi[0];
}

// A warp's walk over a point's near-field segments of [next, end), in order: the
// lanes test 32 of them at once
struct NearScan
{
    int next, end, first = 0;
    unsigned found = 0;
    __device__ __forceinline__ int take(const unsigned char *blob, const SegmentDesc *segs, double px, double py,
                                        double pz, int lane)
    {
        while (found == 0)
        {
            if (next >= end)
                return -1;
            first = next;
            next += 32;
            found = __ballot_sync(0xffffffffu, first + lane < end && isNearPair(blob, segs, first + lane, px, py, pz));
        }
        const int s = first + __ffs(found) - 1;
        found &= found - 1;
        return s;
    }
};

// How many of the segments [begin, end) have the point in their near box, and the first
// one; LANES (1 or 32) threads share them
template <int LANES>
__device__ __forceinline__ int countNear(const unsigned char *blob, const SegmentDesc *segs, int begin, int end,
                                         double px, double py, double pz, int lane, int &first)
{
    int count = 0;
    first = end;
#pragma unroll 2
    for (int s = begin + lane; s < end; s += LANES)
        if (isNearPair(blob, segs, s, px, py, pz))
        {
            first = min(first, s);
            ++count;
        }
    if (LANES > 1)
    {
        count = (int)__reduce_add_sync(0xffffffffu, (unsigned)count);
        first = (int)__reduce_min_sync(0xffffffffu, (unsigned)first);
    }
    return count;
}

// Their entries, in segment order from slot on, with `tag` in the segment's top bits, and
// beside every entry its run (runs != null)
template <int LANES>
__device__ __forceinline__ void listNear(const unsigned char *blob, const SegmentDesc *segs, int first, int end,
                                         double px, double py, double pz, long long p, int lane, int tag,
                                         unsigned long long slot, int count, NearPair *work, NearRun *runs,
                                         unsigned long long workCapacity)
{
    const NearRun run = {(int)slot, count, 0};  // not read if the list is too short
    for (int s0 = first; s0 < end && slot < workCapacity; s0 += LANES)
    {
        const bool near = s0 + lane < end && isNearPair(blob, segs, s0 + lane, px, py, pz);
        const unsigned before = LANES > 1 ? __ballot_sync(0xffffffffu, near) : (near ? 1u : 0u);
        const unsigned long long at = slot + __popc(before & ((1u << lane) - 1u));
        if (near && at < workCapacity)
        {
            work[at].point = (int)p;
            work[at].segment = (s0 + lane) | tag;
            if (runs)
                runs[at] = run;
        }
        slot += __popc(before);
    }
}

// Lists the near-field pairs: the pairs of a point in one run of entries, in segment
// order.  It takes every frame transform once more.  LANES (1 or 32) threads per point
// share its segments.
template <int LANES>
__global__ void __launch_bounds__(256, 4) nearListKernel(const unsigned char *__restrict__ blob,
                                                         const SegmentDesc *__restrict__ segs, int nseg,
                                                         const double *__restrict__ points, long long npts,
                                                         NearPair *__restrict__ work, NearRun *__restrict__ runs,
                                                         unsigned long long workCapacity,
                                                         unsigned long long *__restrict__ workCount)
{
    const int lane = threadIdx.x % LANES;
    const long long p = (long long)blockIdx.x * (blockDim.x / LANES) + threadIdx.x / LANES;
    if (p >= npts)
        return;
    const double px = points[3 * p], py = points[3 * p + 1], pz = points[3 * p + 2];
    int first;
    const int count = countNear<LANES>(blob, segs, 0, nseg, px, py, pz, lane, first);
    if (count == 0)
        return;
    unsigned long long slot = lane == 0 ? atomicAdd(workCount, (unsigned long long)count) : 0ull;
    if (LANES > 1)
        slot = __shfl_sync(0xffffffffu, slot, 0);
    listNear<LANES>(blob, segs, first, nseg, px, py, pz, p, lane, 0, slot, count, work, runs, workCapacity);
}

// One value of one point: the sum of its contributions, entries first, first + 1, ... of
// the list while in(entry) holds, eight loaded at a time (a run of 64 is a chain of 8
// loads) and added in order.
template <typename In>
__device__ __forceinline__ double nearRunSum(const double *contrib, int stride, unsigned long long first, In in)
{
    double sum = 0.0;
    for (bool more = true; more; first += 8)
    {
        double v[8];
        bool is[8];
#pragma unroll
        for (int j = 0; j < 8; ++j)
        {
            is[j] = in(first + j);
            v[j] = is[j] ? __ldcg(contrib + (size_t)stride * (first + j)) : 0.0;
        }
#pragma unroll
        for (int j = 0; j < 8; ++j)
        {
            more = more && is[j];
            if (more)
                sum += v[j];
        }
    }
    return sum;
}

// A warp's sums of listed pair i (every lane has them) on their way to out: the warp
// that brings the last pair of a run adds the run, whichever warp that is.
template <int W>
__device__ __forceinline__ void addListedPair(const double *acc, unsigned long long i, NearRun *runs, double *contrib,
                                              double *out, int lane)
{
    const int first = runs[i].first, count = runs[i].count;
    if (count == 1)
    {
        if (lane == 0)
#pragma unroll
            for (int k = 0; k < W; ++k)
                out[k] += acc[k];
        return;
    }
    int before = 0;
    if (lane == 0)
    {
#pragma unroll
        for (int k = 0; k < W; ++k)
            __stcg(&contrib[(size_t)W * i + k], acc[k]);
        __threadfence();
        before = atomicAdd(&runs[first].done, 1);
    }
    if (__shfl_sync(0xffffffffu, before, 0) != count - 1)
        return;
    __syncwarp();
    __threadfence();
    if (lane < W)
        out[lane] += nearRunSum(contrib + lane, W, first, [&](unsigned long long e) { return e < first + count; });
}

// Evaluates the near-field pairs, the FP64 integrands read from the segment blob in
// global memory, the lanes of a warp splitting the angular nodes: a warp per entry of
// the list, its sums to contrib[entry], or, with more pairs than it holds, a warp per
// point of all points.  runs != null: this kernel adds the runs; else nearSumKernel does.
template <int FIELD>
__global__ void __launch_bounds__(256) nearFieldKernel(const unsigned char *__restrict__ blob,
                                                       const SegmentDesc *__restrict__ segs, int nseg,
                                                       const double *__restrict__ points, long long npts,
                                                       double *__restrict__ out, const NearPair *__restrict__ work,
                                                       NearRun *runs, double *contrib,
                                                       unsigned long long workCapacity,
                                                       const unsigned long long *__restrict__ workCount)
{
    constexpr int W = FIELD == CCOIL_FIELD_G ? 9 : 3;
    const unsigned long long n = *workCount;
    const bool listed = n <= workCapacity;
    const int lane = threadIdx.x % 32;
    const unsigned long long warp = ((unsigned long long)blockIdx.x * blockDim.x + threadIdx.x) / 32;
    const unsigned long long warps = (unsigned long long)gridDim.x * blockDim.x / 32;
    const unsigned long long end = listed ? n : (unsigned long long)npts;
    for (unsigned long long i = warp; i < end; i += warps)
    {
        const long long p = listed ? work[i].point : (long long)i;
        const double px = points[3 * p], py = points[3 * p + 1], pz = points[3 * p + 2];
        double sum = 0.0;  // lane k of a warp per point: value k
        NearScan scan = {0, nseg};
        for (int s = listed ? work[i].segment : scan.take(blob, segs, px, py, pz, lane); s >= 0;
             s = listed ? -1 : scan.take(blob, segs, px, py, pz, lane))
        {
            double acc[W];
#pragma unroll
            for (int k = 0; k < W; ++k)
                acc[k] = 0.0;
            integrateSegment64<FIELD, 32>(blob + segs[s].offset, px, py, pz, lane, acc);
            // pair by pair, so that a point's sum is the same either way
#pragma unroll
            for (int off = 16; off > 0; off /= 2)
#pragma unroll
                for (int k = 0; k < W; ++k)
                    acc[k] += __shfl_xor_sync(0xffffffffu, acc[k], off);
            if (listed && runs)
                addListedPair<W>(acc, i, runs, contrib, out + W * p, lane);
            else
#pragma unroll
                for (int k = 0; k < W; ++k)
                    sum += lane == k ? acc[k] : 0.0;
        }
        if (listed && !runs && lane < W)
            contrib[W * i + lane] = sum;
        else if (!listed && lane < W && sum != 0.0)
            out[W * p + lane] += sum;
    }
}

// Adds the listed pairs' contributions to the output: a thread per entry and value,
// those of a run's first entry take the run.
template <int W>
__global__ void __launch_bounds__(256) nearSumKernel(const NearPair *__restrict__ work,
                                                     unsigned long long workCapacity,
                                                     const unsigned long long *__restrict__ workCount,
                                                     const double *__restrict__ contrib, double *__restrict__ out)
{
    const unsigned long long n = *workCount;
    if (n > workCapacity)
        return;
    const unsigned long long threads = (unsigned long long)gridDim.x * blockDim.x;
    for (unsigned long long t = (unsigned long long)blockIdx.x * blockDim.x + threadIdx.x; t < n * W; t += threads)
    {
        const unsigned long long i = t / W;
        const int k = (int)(t - i * W), p = work[i].point;
        if (i > 0 && work[i - 1].point == p)
            continue;
        out[(size_t)W * p + k] +=
            nearRunSum(contrib + k, W, i, [&](unsigned long long e) { return e < n && work[e].point == p; });
    }
}

// One segment at one point for the refinement pass: the vector potential (and
// E) and the field with the forms above, the gradient with the FP64 field
// integrands; LANES neighbouring lanes split the angular nodes
template <int FIELD, int LANES>
__device__ __forceinline__ void integrateSegmentRefine(const unsigned char *seg, double px, double py, double pz,
                                                       int lane, double *acc)
{
    if (FIELD == CCOIL_FIELD_G)
    {
        integrateSegment64<FIELD, LANES>(seg, px, py, pz, lane, acc);
        return;
    }
    const SegmentHeader &h = *reinterpret_cast<const SegmentHeader *>(seg);
    const double2 *tt = reinterpret_cast<const double2 *>(seg) + h.off_t;
    const double2 *lt = reinterpret_cast<const double2 *>(seg) + h.off_l;
    const double2 *pt = reinterpret_cast<const double2 *>(seg) + h.off_phi;
    const Frame f = toCoilFrame(h, px, py, pz);
    if (FIELD == CCOIL_FIELD_B)
    {
        double H, Z;
        segmentB64Fast<LANES>(h, tt, lt, pt, f, lane, H, Z);
        addRotated(h, H * f.cphi, H * f.sphi, Z, acc);
    }
    else
    {
        const double a = segmentA64Fast<true, LANES>(h, tt, lt, pt, f, lane) * h.field_factor;
        addRotated(h, -a * f.sphi, a * f.cphi, 0.0, acc);
    }
}

// FP32_REFINED's FP64 pass: LANES threads per listed (point, segment) pair, the
// result added to the point's output (FP64 atomics).  One thread per pair while
// there are enough of them (each thickness node's set-up serves all its angular
// nodes, as in the FP64 field kernel, where one warp per pair measured 1.2x the
// time): the selection lists the pairs segment-major, so the lanes of a warp read
// one segment's tables and run loops of the same length.  With fewer pairs than
// threads, 4, 16 or 32 of them share a pair.  The kernel picks by the device-side
// count (this pass for A of 15 coils at 389 points, 1,500 pairs: 263 us with one
// thread per pair, 59 us with 32).
// CTAs per SM of the FP64 pair pass: several nodes in flight per thread without
// spills (vector potential and field 120 registers, gradient 152) measured 1 %
// faster for the whole call than the most CTAs that fit without (6, 5 and 4)
constexpr int refineMinBlocks(int field) { return field == CCOIL_FIELD_G ? 3 : 4; }
template <int FIELD, int LANES>
__device__ __forceinline__ void refinePairs(const unsigned char *__restrict__ blob,
                                            const SegmentDesc *__restrict__ segs, const double *__restrict__ points,
                                            double *__restrict__ out, const NearPair *__restrict__ work,
                                            unsigned long long n)
{
    constexpr int W = FIELD == CCOIL_FIELD_G ? 9 : 3;
    const int lane = threadIdx.x % LANES;
    const unsigned long long stride = (unsigned long long)gridDim.x * blockDim.x / LANES;
    const unsigned long long rounds = (n + stride - 1) / stride;  // the same for all lanes of a warp
    unsigned long long i = ((unsigned long long)blockIdx.x * blockDim.x + threadIdx.x) / LANES;
    for (unsigned long long r = 0; LANES == 1 ? i < n : r < rounds; ++r, i += stride)
    {
        const bool valid = LANES == 1 || i < n;
        double acc[W];
#pragma unroll
        for (int k = 0; k < W; ++k)
            acc[k] = 0.0;
        long long p = 0;
        if (valid)
        {
            const NearPair e = work[i];
            p = e.point;
            integrateSegmentRefine<FIELD, LANES>(blob + segs[e.segment].offset, points[3 * p], points[3 * p + 1],
                                                 points[3 * p + 2], lane, acc);
        }
#pragma unroll
        for (int off = LANES / 2; off > 0; off /= 2)
#pragma unroll
            for (int k = 0; k < W; ++k)
                acc[k] += __shfl_xor_sync(0xffffffffu, acc[k], off);
        if (valid && lane == 0)
#pragma unroll
            for (int k = 0; k < W; ++k)
                atomicAdd(&out[W * p + k], acc[k]);
    }
}

template <int FIELD>
__global__ void __launch_bounds__(128, refineMinBlocks(FIELD)) refinePairsKernel64(
    const unsigned char *__restrict__ blob, const SegmentDesc *__restrict__ segs, const double *__restrict__ points,
    double *__restrict__ out, const NearPair *__restrict__ work, unsigned long long workCapacity,
    const unsigned long long *__restrict__ workCount)
{
    const unsigned long long n = min(*workCount, workCapacity);
    const unsigned long long threads = (unsigned long long)gridDim.x * blockDim.x;
    if (n >= threads)
        refinePairs<FIELD, 1>(blob, segs, points, out, work, n);
    else if (4 * n >= threads)
        refinePairs<FIELD, 4>(blob, segs, points, out, work, n);
    else if (16 * n >= threads)
        refinePairs<FIELD, 16>(blob, segs, points, out, work, n);
    else
        refinePairs<FIELD, 32>(blob, segs, points, out, work, n);
}

// FP32_REFINED selection.  A pair is picked when its stored contribution's
// norm exceeds `fraction` times the norm of the point's total (near-field FP64
// pairs included); a non-finite total picks nothing.  Both passes below make
// the same decision from the same data.
template <int W>
__device__ __forceinline__ bool refinePick(const double *total, const double *c, double fraction)
{
    double n2 = 0.0, c2 = 0.0;
#pragma unroll
    for (int i = 0; i < W; ++i)
    {
        n2 += total[i] * total[i];
        c2 += c[i] * c[i];
    }
    return c2 > fraction * fraction * n2;
}

// Pass 1, one thread per point: picks per segment (segCount, zeroed before).
// Whole warps iterate (base is the warp's first point), so each warp adds once
// per segment.
template <int W>
__global__ void __launch_bounds__(256) refineCountKernel(const double *__restrict__ out,
                                                         const double *__restrict__ contrib, long long npts, int nseg,
                                                         double fraction, unsigned long long *__restrict__ segCount)
{
    const int lane = threadIdx.x % 32;
    const long long stride = (long long)gridDim.x * blockDim.x;
    for (long long base = (long long)blockIdx.x * blockDim.x + (threadIdx.x - lane); base < npts; base += stride)
    {
        const long long p = base + lane;
        const bool active = p < npts;
        double total[W];
#pragma unroll
        for (int i = 0; i < W; ++i)
            total[i] = active ? out[W * p + i] : 0.0;
        for (int s = 0; s < nseg; ++s)
        {
            double c[W];
#pragma unroll
            for (int i = 0; i < W; ++i)
                c[i] = active ? contrib[((size_t)s * (size_t)npts + (size_t)p) * W + i] : 0.0;
            const unsigned mask = __ballot_sync(0xffffffffu, active && refinePick<W>(total, c, fraction));
            if (mask != 0u && lane == 0)
                atomicAdd(&segCount[s], (unsigned long long)__popc(mask));
        }
    }
}

// Pass 2, one block: segCount becomes each segment's first list slot (exclusive
// prefix sum in segment order), *count the number of picks (the list length,
// read by the FP64 pass), *refined grows by the picks that fit the list.
__global__ void __launch_bounds__(1024) refineScanKernel(unsigned long long *__restrict__ segCount, int nseg,
                                                         unsigned long long capacity,
                                                         unsigned long long *__restrict__ count,
                                                         unsigned long long *__restrict__ refined)
{
    __shared__ unsigned long long part[1024];
    __shared__ unsigned long long carry;
    if (threadIdx.x == 0)
        carry = 0;
    __syncthreads();
    for (int base = 0; base < nseg; base += 1024)
    {
        const int s = base + threadIdx.x;
        const unsigned long long v = s < nseg ? segCount[s] : 0ull;
        part[threadIdx.x] = v;
        __syncthreads();
        // Hillis-Steele inclusive scan of the block's slice
        for (int off = 1; off < 1024; off *= 2)
        {
            const unsigned long long add = threadIdx.x >= off ? part[threadIdx.x - off] : 0ull;
            __syncthreads();
            part[threadIdx.x] += add;
            __syncthreads();
        }
        if (s < nseg)
            segCount[s] = carry + part[threadIdx.x] - v;
        __syncthreads();
        if (threadIdx.x == 1023)
            carry += part[1023];
        __syncthreads();
    }
    if (threadIdx.x == 0)
    {
        *count = carry;
        *refined += carry < capacity ? carry : capacity;
    }
}

// Pass 3, one thread per point: every picked pair takes the next slot of its
// segment's range (one atomic per warp and segment), is listed if the slot
// fits the list, and then leaves the point's total; the list comes out
// segment-major, so the FP64 pass's warps read one segment's tables.
template <int W>
__global__ void __launch_bounds__(256) refineSelectKernel(double *__restrict__ out,
                                                          const double *__restrict__ contrib, long long npts, int nseg,
                                                          double fraction, unsigned long long *__restrict__ segNext,
                                                          NearPair *__restrict__ work, unsigned long long capacity)
{
    const int lane = threadIdx.x % 32;
    const long long stride = (long long)gridDim.x * blockDim.x;
    for (long long base = (long long)blockIdx.x * blockDim.x + (threadIdx.x - lane); base < npts; base += stride)
    {
        const long long p = base + lane;
        const bool active = p < npts;
        double total[W], picked[W];
#pragma unroll
        for (int i = 0; i < W; ++i)
        {
            total[i] = active ? out[W * p + i] : 0.0;
            picked[i] = 0.0;
        }
        for (int s = 0; s < nseg; ++s)
        {
            double c[W];
#pragma unroll
            for (int i = 0; i < W; ++i)
                c[i] = active ? contrib[((size_t)s * (size_t)npts + (size_t)p) * W + i] : 0.0;
            const bool pick = active && refinePick<W>(total, c, fraction);
            const unsigned mask = __ballot_sync(0xffffffffu, pick);
            if (mask == 0u)
                continue;
            unsigned long long first = 0;
            if (lane == 0)
                first = atomicAdd(&segNext[s], (unsigned long long)__popc(mask));
            first = __shfl_sync(0xffffffffu, first, 0);
            const unsigned long long slot = first + (unsigned long long)__popc(mask & ((1u << lane) - 1u));
            if (pick && slot < capacity)
            {
                work[slot].point = (int)p;
                work[slot].segment = s;
#pragma unroll
                for (int i = 0; i < W; ++i)
                    picked[i] += c[i];
            }
        }
        if (active)
        {
#pragma unroll
            for (int i = 0; i < W; ++i)
                out[W * p + i] = total[i] - picked[i];
        }
    }
}
