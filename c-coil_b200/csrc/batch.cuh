// Batched persistent field kernel (included by fields.cu inside its anonymous
// namespace, after fields32.cuh).
//
// Many independent coil systems of uneven size in one launch.  The host cuts
// every (system, field) into work items -- a tile of up to 128/L points of one
// system, L lanes per point -- and sorts them longest first.  A grid sized to
// the machine (CTAs per SM x 148) pulls items from an atomic counter until the
// list is exhausted, so long items start first and short ones fill the tail.
// An item reads its system's segment tables straight from global memory
// (through L1, as the single-system kernels do), so warps synchronise only to
// take the next item.  In FP32_COMPENSATED mode the items leave near-field pairs
// out; a second kernel lists them, a point's next to each other with the field in
// the top bits of the segment index, and a third evaluates them (as the
// single-system kernels, fields32.cuh).

struct BatchItem
{
    int seg_begin;    // the system's segments [seg_begin, seg_end)
    int seg_end;
    int point_begin;  // first point of the item (global index)
    int point_count;  // points in the item (<= 128 / lanes)
    int lanes;        // 1, 4 or 32 threads per point
    int field;        // CCOIL_FIELD_A, _B, _E or _G
    int pad0, pad1;
};

constexpr int kFieldShift = 28;  // NearPair.segment = segment | field << 28

template <int PREC, int FIELD, int LANES>
__device__ __forceinline__ void batchItem(const BatchItem &I, const unsigned char *__restrict__ blob,
                                          const SegmentDesc *__restrict__ segs, const double *__restrict__ points,
                                          double *__restrict__ out, double (*sums)[128])
{
    constexpr int W = FIELD == CCOIL_FIELD_G ? 9 : 3;
    // the FP32 gradient's sums in shared memory, as fieldsKernel32's
    constexpr bool kShared = FIELD == CCOIL_FIELD_G && PREC != CCOIL_PRECISION_FP64;
    const int lane = threadIdx.x % LANES;
    const int local = threadIdx.x / LANES;
    const bool active = local < I.point_count;
    const long long p = (long long)I.point_begin + local;
    const int nseg = I.seg_end - I.seg_begin;

    double px = 0.0, py = 0.0, pz = 0.0;
    if (active)
    {
        px = points[3 * p];
        py = points[3 * p + 1];
        pz = points[3 * p + 2];
    }
    double acc[W];
#pragma unroll
    for (int i = 0; i < W; ++i)
    {
        acc[i] = 0.0;
        if (kShared)
            sums[kShared ? i : 0][threadIdx.x] = 0.0;
    }

    for (int s = 0; s < nseg && active; ++s)
    {
        const unsigned char *seg = blob + segs[I.seg_begin + s].offset;
        if (PREC == CCOIL_PRECISION_FP64)
            integrateSegment64<FIELD, LANES, true>(seg, px, py, pz, lane, acc);
        else
        {
            const SegmentHeader &h = *reinterpret_cast<const SegmentHeader *>(seg);
            const Frame f = toCoilFrame(h, px, py, pz);
            if (nearWinding(h, f))
                continue;
            if (kShared)
            {
                double c[W];
#pragma unroll
                for (int i = 0; i < W; ++i)
                    c[i] = 0.0;
                integrateSegment32<FIELD, LANES>(seg, f, lane, c);
#pragma unroll
                for (int i = 0; i < W; ++i)
                    sums[kShared ? i : 0][threadIdx.x] += c[i];
            }
            else
                integrateSegment32<FIELD, LANES>(seg, f, lane, acc);
        }
    }
    if (kShared)
#pragma unroll
        for (int i = 0; i < W; ++i)
            acc[i] = sums[kShared ? i : 0][threadIdx.x];
#pragma unroll
    for (int off = LANES / 2; off > 0; off /= 2)
#pragma unroll
        for (int i = 0; i < W; ++i)
            acc[i] += __shfl_xor_sync(0xffffffffu, acc[i], off);
    if (active && lane == 0)
    {
#pragma unroll
        for (int i = 0; i < W; ++i)
            out[W * p + i] = acc[i];
    }
}

template <int PREC, int FIELD>
__device__ __forceinline__ void batchItemLanes(const BatchItem &I, const unsigned char *blob, const SegmentDesc *segs,
                                               const double *points, double *out, double (*sums)[128])
{
    switch (I.lanes)
    {
        case 1: batchItem<PREC, FIELD, 1>(I, blob, segs, points, out, sums); break;
        case 4: batchItem<PREC, FIELD, 4>(I, blob, segs, points, out, sums); break;
        default: batchItem<PREC, FIELD, 32>(I, blob, segs, points, out, sums); break;
    }
}

// CTAs per SM the register allocation targets, per precision.  FP64: 3
// (168 registers, no spills; 18.7 ms for B + G over 40 systems of up to 64 coils
// and 16,384 points, against 20.6 ms at 4 and 23.0 ms at 5).  FP32: 4 (128
// registers, no spills): B + G over 2,048 systems 2.28 s per step, 2.39 s at 5 and
// 2.43 s at 6; 3, at 2.22 s, was found since
#ifndef CCOIL_BATCH_MIN_BLOCKS
#define CCOIL_BATCH_MIN_BLOCKS 3
#endif
#ifndef CCOIL_BATCH32_MIN_BLOCKS
#define CCOIL_BATCH32_MIN_BLOCKS 4
#endif

constexpr int batchMinBlocks(int prec)
{
    return prec == CCOIL_PRECISION_FP64 ? CCOIL_BATCH_MIN_BLOCKS : CCOIL_BATCH32_MIN_BLOCKS;
}

template <int PREC>
__global__ void __launch_bounds__(128, batchMinBlocks(PREC)) batchKernel(const unsigned char *__restrict__ blob,
                                                      const SegmentDesc *__restrict__ segs,
                                                      const BatchItem *__restrict__ items, int nitems,
                                                      unsigned *__restrict__ next, const double *__restrict__ points,
                                                      double *__restrict__ outA, double *__restrict__ outB,
                                                      double *__restrict__ outG,
                                                      unsigned long long *__restrict__ workCount)
{
    if (PREC != CCOIL_PRECISION_FP64 && blockIdx.x == 0 && threadIdx.x == 0)
        *workCount = 0;  // the near-field list's counter, for the kernels that follow
    __shared__ int itemIndex;
    __shared__ double sums[PREC == CCOIL_PRECISION_FP64 ? 1 : 9][128];
    for (;;)
    {
        if (threadIdx.x == 0)
            itemIndex = (int)atomicAdd(next, 1u);
        __syncthreads();
        const int it = itemIndex;
        __syncthreads();  // every thread has read the index before it is replaced
        if (it >= nitems)
            break;
        const BatchItem I = items[it];
        if (I.field == CCOIL_FIELD_B)
            batchItemLanes<PREC, CCOIL_FIELD_B>(I, blob, segs, points, outB, sums);
        else if (I.field == CCOIL_FIELD_G)
            batchItemLanes<PREC, CCOIL_FIELD_G>(I, blob, segs, points, outG, sums);
        else
            batchItemLanes<PREC, CCOIL_FIELD_A>(I, blob, segs, points, outA, sums);
    }
}

// The pairs of one point: its entries are consecutive, field by field.  LANES (1 or 32)
// threads share its segments.
template <int LANES>
__device__ __forceinline__ void batchListPoint(const BatchItem &I, const unsigned char *blob, const SegmentDesc *segs,
                                               int fieldsMask, const double *points, int local, int lane,
                                               NearPair *work, unsigned long long workCapacity,
                                               unsigned long long *workCount)
{
    const long long p = (long long)I.point_begin + local;
    const double px = points[3 * p], py = points[3 * p + 1], pz = points[3 * p + 2];
    int first;
    const int count = countNear<LANES>(blob, segs, I.seg_begin, I.seg_end, px, py, pz, lane, first);
    if (count == 0)
        return;
    unsigned long long slot =
        lane == 0 ? atomicAdd(workCount, (unsigned long long)count * __popc(fieldsMask)) : 0ull;
    if (LANES > 1)
        slot = __shfl_sync(0xffffffffu, slot, 0);
    for (int f = CCOIL_FIELD_A; f <= CCOIL_FIELD_G; ++f)
        if (fieldsMask & (1 << f))
        {
            listNear<LANES>(blob, segs, first, I.seg_end, px, py, pz, p, lane, f << kFieldShift, slot, count, work,
                            nullptr, workCapacity);
            slot += count;
        }
}

// Lists the near-field pairs: a block per item of the lowest field, a thread per point,
// or, for many segments at few points in all (warps), a warp.  The whole call with
// threads and with warps: one system of 64 coils at 64 points 247 and 178 us, 20 of 32
// coils at 64 points 244 and 220 us, at 3,000 points 797 and 793 us; 2,048 systems with
// 24.7 million points 2,276 and 2,284 ms.
__global__ void __launch_bounds__(128) batchNearListKernel(const unsigned char *__restrict__ blob,
                                                           const SegmentDesc *__restrict__ segs,
                                                           const BatchItem *__restrict__ items, int nitems,
                                                           int fieldsMask, bool warps,
                                                           const double *__restrict__ points,
                                                           NearPair *__restrict__ work,
                                                           unsigned long long workCapacity,
                                                           unsigned long long *__restrict__ workCount)
{
    const int lowest = __ffs(fieldsMask) - 1;
    for (int it = blockIdx.x; it < nitems; it += gridDim.x)
    {
        const BatchItem I = items[it];
        if (I.field != lowest)
            continue;
        if (warps && I.seg_end - I.seg_begin >= 16)
            for (int local = threadIdx.x / 32; local < I.point_count; local += 4)
                batchListPoint<32>(I, blob, segs, fieldsMask, points, local, threadIdx.x % 32, work, workCapacity,
                                   workCount);
        else if ((int)threadIdx.x < I.point_count)
            batchListPoint<1>(I, blob, segs, fieldsMask, points, threadIdx.x, 0, work, workCapacity, workCount);
    }
}

// One warp: near-field pairs of one point and field, FP64, the lanes splitting the
// angular nodes: a listed pair, whose sums go to contrib, or those of [segBegin,
// segEnd), in order, which go to out (segment < 0).
template <int FIELD>
__device__ __forceinline__ void batchNearPairs(const unsigned char *blob, const SegmentDesc *segs,
                                               const double *points, long long p, int segment, int segBegin,
                                               int segEnd, int lane, double *contrib, double *out)
{
    constexpr int W = FIELD == CCOIL_FIELD_G ? 9 : 3;
    const double px = points[3 * p], py = points[3 * p + 1], pz = points[3 * p + 2];
    const bool listed = segment >= 0;
    double sum = 0.0;
    NearScan scan = {segBegin, segEnd};
    for (int s = listed ? segment : scan.take(blob, segs, px, py, pz, lane); s >= 0;
         s = listed ? -1 : scan.take(blob, segs, px, py, pz, lane))
    {
        double acc[W];
#pragma unroll
        for (int k = 0; k < W; ++k)
            acc[k] = 0.0;
        integrateSegment64<FIELD, 32>(blob + segs[s].offset, px, py, pz, lane, acc);
#pragma unroll
        for (int off = 16; off > 0; off /= 2)
#pragma unroll
            for (int k = 0; k < W; ++k)
                acc[k] += __shfl_xor_sync(0xffffffffu, acc[k], off);
#pragma unroll
        for (int k = 0; k < W; ++k)
            sum += lane == k ? acc[k] : 0.0;
    }
    if (listed && lane < W)
        contrib[lane] = sum;
    else if (!listed && lane < W && sum != 0.0)
        out[W * p + lane] += sum;
}

// Near-field pass of the batched kernel: a warp per entry (batchNearSumKernel adds them
// up), or, with more pairs than the list holds, a warp per point of each item.
__global__ void __launch_bounds__(256) batchNearKernel(const unsigned char *__restrict__ blob,
                                                       const SegmentDesc *__restrict__ segs,
                                                       const BatchItem *__restrict__ items, int nitems,
                                                       const double *__restrict__ points, double *__restrict__ outA,
                                                       double *__restrict__ outB, double *__restrict__ outG,
                                                       const NearPair *__restrict__ work,
                                                       double *__restrict__ contrib, int width,
                                                       unsigned long long workCapacity,
                                                       const unsigned long long *__restrict__ workCount)
{
    const unsigned long long n = *workCount;
    const bool listed = n <= workCapacity;
    const int lane = threadIdx.x % 32;
    const unsigned long long warp = ((unsigned long long)blockIdx.x * blockDim.x + threadIdx.x) / 32;
    const unsigned long long warps = (unsigned long long)gridDim.x * blockDim.x / 32;
    // list entry, or point threadIdx of 128 of an item
    const unsigned long long end = listed ? n : (unsigned long long)nitems * 128;
    for (unsigned long long i = warp; i < end; i += warps)
    {
        long long p;
        int field, segment = -1, segBegin = 0, segEnd = 0;
        if (listed)
        {
            const NearPair e = work[i];
            field = e.segment >> kFieldShift;
            segment = e.segment & ((1 << kFieldShift) - 1);
            p = e.point;
        }
        else
        {
            const BatchItem I = items[i / 128];
            if ((int)(i % 128) >= I.point_count)
                continue;
            field = I.field;
            p = (long long)I.point_begin + (int)(i % 128);
            segBegin = I.seg_begin;
            segEnd = I.seg_end;
        }
        double *entry = contrib + (size_t)width * i;  // listed only
        if (field == CCOIL_FIELD_G)
            batchNearPairs<CCOIL_FIELD_G>(blob, segs, points, p, segment, segBegin, segEnd, lane, entry, outG);
        else if (field == CCOIL_FIELD_B)
            batchNearPairs<CCOIL_FIELD_B>(blob, segs, points, p, segment, segBegin, segEnd, lane, entry, outB);
        else
            batchNearPairs<CCOIL_FIELD_A>(blob, segs, points, p, segment, segBegin, segEnd, lane, entry, outA);
    }
}

// Adds the listed pairs' contributions to the outputs, as nearSumKernel
__global__ void __launch_bounds__(256) batchNearSumKernel(const NearPair *__restrict__ work,
                                                          unsigned long long workCapacity,
                                                          const unsigned long long *__restrict__ workCount,
                                                          const double *__restrict__ contrib, int width,
                                                          double *__restrict__ outA, double *__restrict__ outB,
                                                          double *__restrict__ outG)
{
    const unsigned long long n = *workCount;
    if (n > workCapacity)
        return;
    const unsigned long long threads = (unsigned long long)gridDim.x * blockDim.x;
    for (unsigned long long t = (unsigned long long)blockIdx.x * blockDim.x + threadIdx.x; t < n * width; t += threads)
    {
        const unsigned long long i = t / width;
        const int k = (int)(t - i * width);
        const NearPair e = work[i];
        const int field = e.segment >> kFieldShift, W = field == CCOIL_FIELD_G ? 9 : 3;
        auto same = [&](unsigned long long j) {
            return j < n && work[j].point == e.point && work[j].segment >> kFieldShift == field;
        };
        if (k >= W || (i > 0 && same(i - 1)))
            continue;
        double *out = field == CCOIL_FIELD_G ? outG : field == CCOIL_FIELD_B ? outB : outA;
        out[(size_t)W * e.point + k] += nearRunSum(contrib + k, width, i, same);
    }
}

// Launch of one batched execution: counters reset, persistent kernel, near pass.
int launchBatchImpl(const BatchLaunch &B, cudaStream_t st)
{
    cudaError_t e = cudaMemsetAsync(B.d_next, 0, sizeof(unsigned), st);
    if (e != cudaSuccess)
        return failMessage(CCOIL_ERR_CUDA, cudaGetErrorString(e));
    if (B.nitems == 0)
        return CCOIL_OK;
    NearPair *work = reinterpret_cast<NearPair *>(B.d_work);
    const BatchItem *items = static_cast<const BatchItem *>(B.d_items);
    if (B.precision == CCOIL_PRECISION_FP64)
        batchKernel<CCOIL_PRECISION_FP64><<<B.grid, 128, 0, st>>>(B.d_blob, B.d_segs, items, B.nitems, B.d_next,
                                                                     B.d_points, B.d_outA, B.d_outB, B.d_outG,
                                                                     nullptr);
    else
        batchKernel<CCOIL_PRECISION_FP32_COMPENSATED><<<B.grid, 128, 0, st>>>(
            B.d_blob, B.d_segs, items, B.nitems, B.d_next, B.d_points, B.d_outA, B.d_outB, B.d_outG,
            B.d_work_count);
    e = cudaGetLastError();
    if (e == cudaSuccess && B.precision == CCOIL_PRECISION_FP32_COMPENSATED)
    {
        batchNearListKernel<<<(unsigned)std::min(B.nitems, 148 * 64), 128, 0, st>>>(
            B.d_blob, B.d_segs, items, B.nitems, B.fields_mask, B.points <= (1 << 15), B.d_points, work,
            B.near.capacity, B.d_work_count);
        batchNearKernel<<<148 * 8, 256, 0, st>>>(B.d_blob, B.d_segs, items, B.nitems, B.d_points, B.d_outA, B.d_outB,
                                                 B.d_outG, work, B.near.contrib, B.near_width, B.near.capacity,
                                                 B.d_work_count);
        batchNearSumKernel<<<148 * 8, 256, 0, st>>>(work, B.near.capacity, B.d_work_count, B.near.contrib,
                                                    B.near_width, B.d_outA, B.d_outB, B.d_outG);
        e = cudaGetLastError();
    }
    return e == cudaSuccess ? CCOIL_OK : failMessage(CCOIL_ERR_CUDA, cudaGetErrorString(e));
}
