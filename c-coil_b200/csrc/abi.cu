// The C-ABI entry points (include/ccoil_gpu.h): argument checks, device
// buffers, host<->device staging and kernel dispatch.  Nothing here exits the
// process: every failure becomes a status code plus a thread-local message.
#include "ccoil_internal.h"

#include <cuda_runtime.h>

#include <algorithm>
#include <atomic>
#include <cmath>
#include <cstdio>
#include <cstring>
#include <mutex>
#include <new>

namespace ccoil
{
namespace
{
// last error message of the calling thread (fixed storage: reporting an error
// never allocates)
thread_local char t_error[512] = "";

// Grow-only device buffer owned by a plan.  A plan that a user keeps serves any
// stream (calls that use its buffers one after the other), so these are allocated
// and replaced with the device idle; the plan
// of a one-shot call (scoped) has its buffers in the order of the call's stream.
struct BufferOwner
{
    bool scoped = false;
    cudaStream_t stream = nullptr;
};
struct DeviceBuffer
{
    void *ptr = nullptr;
    size_t bytes = 0;
    int reserve(size_t n, const BufferOwner &o);
    // the device is idle, or the owner is scoped
    void release(const BufferOwner &o)
    {
        if (ptr)
            cudaFreeAsync(ptr, o.scoped ? o.stream : nullptr);
        ptr = nullptr;
        bytes = 0;
    }
};
} // namespace

void setError(const std::string &msg) { failMessage(CCOIL_OK, msg.c_str()); }

int fail(int status, const std::string &msg) { return failMessage(status, msg.c_str()); }

int failMessage(int status, const char *msg)
{
    std::snprintf(t_error, sizeof(t_error), "%s", msg ? msg : "");
    return status;
}

int cudaFail(cudaError_t e, const char *what)
{
    if (e == cudaErrorMemoryAllocation)
        return fail(CCOIL_ERR_OUT_OF_MEMORY, std::string(what) + ": " + cudaGetErrorString(e));
    if (e == cudaErrorNoDevice || e == cudaErrorInsufficientDriver)
        return fail(CCOIL_ERR_NO_DEVICE, std::string(what) + ": " + cudaGetErrorString(e));
    return fail(CCOIL_ERR_CUDA, std::string(what) + ": " + cudaGetErrorString(e));
}

namespace
{
std::mutex g_poolMutex;
constexpr int kMaxDevices = 64;
cudaMemPool_t g_pools[kMaxDevices] = {};
// allocations still to fail on purpose (ccoil_inject_allocation_failures)
std::atomic<int> g_failAllocations{0};
// FP32_REFINED: re-evaluate in FP64 every (point, segment) pair whose FP32
// contribution's norm exceeds this fraction of the norm of the point's total
std::atomic<double> g_refineFraction{kDefaultRefineFraction};
// device-side wait timeouts already reported to a caller
std::atomic<long long> g_timeoutsReported{0};
// FP32 plans sort their points along a Morton curve (ccoil_set_point_ordering)
std::atomic<int> g_pointOrdering{1};
} // namespace

cudaError_t scratchAlloc(void **p, size_t bytes, cudaStream_t st)
{
    for (int n = g_failAllocations.load(); n > 0;)
        if (g_failAllocations.compare_exchange_weak(n, n - 1))
            return cudaErrorMemoryAllocation;
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess)
        return e;
    if (dev < 0 || dev >= kMaxDevices)
        return cudaErrorInvalidDevice;
    cudaMemPool_t pool;
    {
        std::lock_guard<std::mutex> lock(g_poolMutex);
        if (!g_pools[dev])
        {
            cudaMemPoolProps props;
            std::memset(&props, 0, sizeof(props));
            props.allocType = cudaMemAllocationTypePinned;
            props.location.type = cudaMemLocationTypeDevice;
            props.location.id = dev;
            e = cudaMemPoolCreate(&g_pools[dev], &props);
            if (e != cudaSuccess)
            {
                g_pools[dev] = nullptr;
                return e;
            }
            // freed blocks up to 16 GiB stay mapped for the next allocation: a
            // one-shot FP32_REFINED call frees and takes again ~5 GB of scratch
            // (with 4 GiB kept, the remapping made those calls 1.5x slower)
            unsigned long long keep = 1ULL << 34;
            e = cudaMemPoolSetAttribute(g_pools[dev], cudaMemPoolAttrReleaseThreshold, &keep);
            if (e != cudaSuccess)
                return e;
        }
        pool = g_pools[dev];
    }
    return cudaMallocFromPoolAsync(p, bytes, pool, st);
}

namespace
{
int DeviceBuffer::reserve(size_t n, const BufferOwner &o)
{
    if (n <= bytes)
        return CCOIL_OK;
    // no kernel on any stream may still read a buffer that is replaced
    if (ptr && !o.scoped)
        cudaDeviceSynchronize();
    release(o);
    cudaError_t e = scratchAlloc(&ptr, n, o.scoped ? o.stream : nullptr);
    if (e == cudaSuccess && !o.scoped)
        e = cudaStreamSynchronize(nullptr);
    if (e != cudaSuccess)
    {
        ptr = nullptr;
        return cudaFail(e, "device buffer");
    }
    bytes = n;
    return CCOIL_OK;
}

// FP32 modes: enough threads to fill the 148 SMs several times over; below that,
// split the angular nodes of each point across lanes (a lane count is part of an
// FP32 sum's order, so this rule stands however the work is cut into pieces)
int autoLanes32(long long npts)
{
    const long long target = 148LL * 1024;
    int lanes = 1;
    while (lanes < 8 && npts * lanes < target)
        lanes *= 2;
    return lanes;
}

// FP64 in one piece (a captured call, or one without memory for the pieces' sums):
// only lanes fill the machine.  The rule of the FP32 modes, and 16 or 32 lanes while
// they take no more than two CTAs per SM.  B captured, 24 coils at 1,001 points: 1, 8
// and 32 lanes 1,180, 267 and 174 us; at 4,096 points 8, 16 and 32 lanes 313, 326 and
// 376 us; at 20,000 points 1, 8 and 16 lanes 1,691, 1,117 and 1,269 us.
int autoLanesOnePiece64(long long npts)
{
    int lanes = autoLanes32(npts);
    while (lanes >= 8 && lanes < 32 && npts * lanes * 2 <= 148LL * 128 * 2)
        lanes *= 2;
    return lanes;
}

// FP64 in pieces: points and pieces (segments x thickness nodes) fill the machine first,
// because lanes that share a point repeat every thickness node's set-up (8 lanes
// and 59 angular nodes: a fifth of the work); lanes come in where those are too
// few for two waves, and to give the warps of a few points something to do
int autoLanes64(long long npts, long long pieces, int blocksPerSM)
{
    const long long target = 2 * 148LL * 128 * blocksPerSM;
    int lanes = 1;
    while (lanes < 32 && npts * lanes * pieces < target)
        lanes *= 2;
    return lanes;
}

// Pieces per tile of points (FieldSplit): the tiles alone leave the last wave
// nearly empty unless there are several waves of them, and the machine idle below
// one, so segments are dealt out, and then every segment's thickness nodes, until
// there are kFieldWaves waves of blocks.  A piece repeats its points' frame
// transform, so beyond one wave it keeps kPieceNodes nodes per thread.  FP64 kernel
// times before and after: A of 24 coils at 1,001 points 310 -> 93 us, B of 64 coils
// at 4,096 points 1.73 -> 1.07 ms, B of one coil at 37 points 24 -> 8 us; FP32_REFINED
// A of 128 coils at 200,003 points (2.1 waves whole) 20.4 -> 18.5 ms.  24 waves instead
// of 8 take 1 to 3 % off calls of 128 coils at 65,536 to 400,000 points (B at 262,144
// FP32 28.5 -> 28.1, FP64 55.2 -> 54.5 ms), 48 and 96 nothing more.
constexpr long long kFieldWaves = 24, kPieceNodes = 128;
FieldSplit fieldSplit(long long npts, int lanes, int nseg, int thickness, long long nodes, int blocksPerSM,
                      bool wholeSegments)
{
    FieldSplit s;
    const long long wave = 148LL * blocksPerSM;
    const long long tiles = (npts + 128 / lanes - 1) / (128 / lanes);
    const long long one = (wave + tiles - 1) / tiles, full = (kFieldWaves * wave + tiles - 1) / tiles;
    const long long want = std::min(full, std::max(one, nodes / (lanes * kPieceNodes)));
    s.groups = (int)std::max(1LL, std::min<long long>(want, nseg));
    if (s.groups == nseg && !wholeSegments)
        s.parts = (int)std::max(1LL, std::min<long long>((want + nseg - 1) / nseg, thickness));
    return s;
}

// host arrays up to this size are packed into one copy with a call's tables: a
// copy costs ~4 us whatever its size below that
constexpr size_t kPackedCopyBytes = size_t(1) << 16;

bool validLanes(int l) { return l == 1 || l == 2 || l == 4 || l == 8 || l == 16 || l == 32; }
} // namespace
} // namespace ccoil

using namespace ccoil;

struct ccoil_field_plan
{
    int field = 0;
    int precision = 0;
    int coil_count = 0;
    int thickness = 1;    // most thickness nodes of a segment
    long long nodes = 0;  // quadrature nodes of all segments
    SegmentSet set;       // set.blob holds the blobs and, after them, the descriptors
    size_t segsOffset = 0;
    BufferOwner owner;
    DeviceBuffer tables, points, out, work, workCount;
    DeviceBuffer contrib, refineSegs, refinedTotal;  // FP32_REFINED
    DeviceBuffer orderScratch, order, sortedPoints, sortedOut;  // point ordering
};

namespace
{
// Argument checks and the host side of a plan: segment blobs and descriptors in
// one block, one upload.
int buildTables(ccoil_field_plan &p, const ccoil_coil_t *coils, int coil_count, int field, int precision)
{
    if (coil_count < 0 || (coil_count > 0 && !coils))
        return fail(CCOIL_ERR_INVALID_ARGUMENT, "coil_count < 0 or coils null");
    if (field < CCOIL_FIELD_A || field > CCOIL_FIELD_G)
        return fail(CCOIL_ERR_INVALID_ARGUMENT, "field must be A, B, E or G");
    if (precision != CCOIL_PRECISION_FP64 && precision != CCOIL_PRECISION_FP32_COMPENSATED &&
        precision != CCOIL_PRECISION_FP32_REFINED)
        return fail(CCOIL_ERR_INVALID_ARGUMENT, "precision must be FP64, FP32_COMPENSATED or FP32_REFINED");
    p.field = field;
    p.precision = precision;
    p.coil_count = coil_count;
    std::string err;
    const int tables = precision == CCOIL_PRECISION_FP64 ? CCOIL_PRECISION_FP64 : CCOIL_PRECISION_FP32_COMPENSATED;
    if (!buildFieldSegments(coils, coil_count, field, tables, p.set, err))
        return fail(CCOIL_ERR_INVALID_ARGUMENT, err);
    for (const SegmentDesc &d : p.set.segs)
    {
        const SegmentHeader &h = *reinterpret_cast<const SegmentHeader *>(p.set.blob.data() + d.offset);
        p.thickness = std::max(p.thickness, h.n_t);
        p.nodes += (long long)h.n_t * h.n_phi * std::max(h.n_l, 1);
    }
    p.segsOffset = p.set.blob.size();  // a multiple of 16
    const auto *d = reinterpret_cast<const unsigned char *>(p.set.segs.data());
    p.set.blob.insert(p.set.blob.end(), d, d + sizeof(SegmentDesc) * p.set.segs.size());
    return CCOIL_OK;
}

int checkExecute(const double *points, long long point_count, const double *out, int memory)
{
    if (point_count < 0 || (point_count > 0 && (!points || !out)))
        return fail(CCOIL_ERR_INVALID_ARGUMENT, "point_count < 0 or null points/out");
    if (memory != CCOIL_MEMORY_HOST && memory != CCOIL_MEMORY_DEVICE)
        return fail(CCOIL_ERR_INVALID_ARGUMENT, "memory must be HOST or DEVICE");
    return CCOIL_OK;
}

// host results: the copy back, and the wait for it
int finishHost(double *out, const double *dOut, size_t outBytes, cudaStream_t st)
{
    cudaError_t e = cudaMemcpyAsync(out, dOut, outBytes, cudaMemcpyDeviceToHost, st);
    if (e == cudaSuccess)
        e = cudaStreamSynchronize(st);
    if (e != cudaSuccess)
        return cudaFail(e, "field evaluation");
    if (!fieldKernelsWait())
        return CCOIL_OK;
    long long timeouts = 0;
    const int rc = readTimeouts(timeouts);
    if (rc != CCOIL_OK)
        return rc;
    if (timeouts > g_timeoutsReported.load())
    {
        g_timeoutsReported.store(timeouts);
        return fail(CCOIL_ERR_TIMEOUT, "a staging wait in the field kernel timed out");
    }
    return CCOIL_OK;
}

// The kernels of one execution, asynchronous on the stream: dPoints and dOut are
// device memory.
int runFields(ccoil_field_plan *plan, const double *dPoints, long long point_count, double *dOut, int lanes_per_point,
              void *stream)
{
    const int width = plan->field == CCOIL_FIELD_G ? 9 : 3;
    const size_t inBytes = sizeof(double) * 3 * (size_t)point_count;
    const size_t outBytes = sizeof(double) * width * (size_t)point_count;
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    FieldLaunch L;
    L.d_blob = static_cast<const unsigned char *>(plan->tables.ptr);
    L.d_segs = reinterpret_cast<const SegmentDesc *>(L.d_blob + plan->segsOffset);
    L.nseg = (int)plan->set.segs.size();
    L.d_points = dPoints;
    L.npts = point_count;
    L.d_out = dOut;
    L.field = plan->field;
    L.precision = plan->precision;
    const int perSM = fieldBlocksPerSM(plan->field, plan->precision);
    // a captured call runs in one piece: it must not hold an allocation that each
    // replay would make again
    cudaStreamCaptureStatus capture = cudaStreamCaptureStatusNone;
    const cudaError_t captureQuery = cudaStreamIsCapturing(st, &capture);
    if (captureQuery != cudaSuccess)
        cudaGetLastError();  // the launches report what is wrong with the stream
    const bool pieced = L.nseg > 0 && perSM > 0 && captureQuery == cudaSuccess && capture == cudaStreamCaptureStatusNone;
    const bool autoFp64 = lanes_per_point == 0 && plan->precision == CCOIL_PRECISION_FP64;
    L.lanes = lanes_per_point ? lanes_per_point
              : !autoFp64     ? autoLanes32(point_count)
              : pieced        ? autoLanes64(point_count, (long long)L.nseg * plan->thickness, perSM)
                              : autoLanesOnePiece64(point_count);
    // FP32_REFINED runs in chunks of points whose stored contributions fit
    // kRefineContribBytes and whose pairs fit a list of kRefineListPairs
    const bool refined = plan->precision == CCOIL_PRECISION_FP32_REFINED && L.nseg > 0;
    long long chunk = point_count;
    if (refined)
    {
        const size_t perPoint = (size_t)L.nseg * (size_t)width * sizeof(double);
        long long maxChunk = (long long)(kRefineContribBytes / perPoint);
        const long long byList = (long long)(kRefineListPairs / (unsigned long long)L.nseg);
        maxChunk = std::max(1LL, std::min(maxChunk, byList));
        const long long chunks = (point_count + maxChunk - 1) / maxChunk;
        chunk = (point_count + chunks - 1) / chunks;
        if (L.lanes > 8)
            L.lanes = 8;  // the refining kernel is compiled for 1 to 8 lanes per point
    }
    if (plan->precision == CCOIL_PRECISION_FP32_COMPENSATED || plan->precision == CCOIL_PRECISION_FP32_REFINED)
    {
        // near-field work list: room for every (point, segment) pair up to
        // kNearListPairs, for few points kNearListPairsFewPoints (with more near-field pairs the near-field pass finds them
        // itself; FP32_REFINED's selection: every pair of a chunk, up to
        // kRefineListPairs), and after it what else the near-field pass needs
        const unsigned long long want = std::max(1ULL, (unsigned long long)chunk * (unsigned long long)L.nseg);
        unsigned long long near =
            std::min(want, chunk <= kNearFewPoints ? kNearListPairsFewPoints : kNearListPairs);
        auto bytes = [&] {
            return (refined ? std::min(want, kRefineListPairs) : near) * kNearPairBytes + NearScratch::bytes(near, width);
        };
        // a captured call allocates nothing: it takes the buffer of an earlier call of at
        // least as many points, which may have had the short list
        if (capture != cudaStreamCaptureStatusNone && bytes() > plan->work.bytes)
            near = std::min(want, kNearListPairs);
        const unsigned long long cap = refined ? std::min(want, kRefineListPairs) : near;
        int rc0 = plan->work.reserve(bytes(), plan->owner);
        if (rc0 == CCOIL_OK)
            rc0 = plan->workCount.reserve(sizeof(unsigned long long), plan->owner);
        if (rc0 != CCOIL_OK)
            return rc0;
        L.d_work = plan->work.ptr;
        L.work_capacity = cap;
        L.near.carve(static_cast<unsigned char *>(plan->work.ptr) + cap * kNearPairBytes, near, width);
        L.d_work_count = static_cast<unsigned long long *>(plan->workCount.ptr);
        L.near_blocks = 148 * 8;
    }
    if (refined)
    {
        int rc0 = plan->contrib.reserve((size_t)chunk * (size_t)L.nseg * (size_t)width * sizeof(double), plan->owner);
        if (rc0 == CCOIL_OK)
            rc0 = plan->refineSegs.reserve(sizeof(unsigned long long) * (size_t)L.nseg, plan->owner);
        if (rc0 == CCOIL_OK)
            rc0 = plan->refinedTotal.reserve(sizeof(unsigned long long), plan->owner);
        if (rc0 != CCOIL_OK)
            return rc0;
        cudaError_t e = cudaMemsetAsync(plan->refinedTotal.ptr, 0, sizeof(unsigned long long), st);
        if (e != cudaSuccess)
            return cudaFail(e, "refinement count");
        L.refine_fraction = g_refineFraction.load();
        L.d_contrib = static_cast<double *>(plan->contrib.ptr);
        L.d_refine_segs = static_cast<unsigned long long *>(plan->refineSegs.ptr);
        L.d_refined_total = static_cast<unsigned long long *>(plan->refinedTotal.ptr);
    }
    // FP32 modes: evaluate the points in Morton order (ordering.cu)
    const bool ordered = g_pointOrdering.load() != 0 && plan->precision != CCOIL_PRECISION_FP64 &&
                         point_count >= kPointOrderMinPoints && point_count <= kPointOrderMaxPoints;
    if (ordered)
    {
        const size_t scratch = pointOrderScratchBytes(point_count);
        int rc0 = plan->orderScratch.reserve(scratch, plan->owner);
        if (rc0 == CCOIL_OK)
            rc0 = plan->order.reserve(sizeof(int) * (size_t)point_count, plan->owner);
        if (rc0 == CCOIL_OK)
            rc0 = plan->sortedPoints.reserve(inBytes, plan->owner);
        if (rc0 == CCOIL_OK)
            rc0 = plan->sortedOut.reserve(outBytes, plan->owner);
        if (rc0 == CCOIL_OK)
            rc0 = orderPoints(dPoints, point_count, plan->orderScratch.ptr, plan->orderScratch.bytes,
                              static_cast<int *>(plan->order.ptr), static_cast<double *>(plan->sortedPoints.ptr),
                              stream);
        if (rc0 != CCOIL_OK)
            return rc0;
        L.d_points = static_cast<const double *>(plan->sortedPoints.ptr);
        L.d_out = static_cast<double *>(plan->sortedOut.ptr);
    }
    // the pieces' sums: memory of this call alone (FP64 calls of one plan may overlap
    // on several streams), in the order of the stream.  Without it the points are
    // evaluated in one piece
    void *partial = nullptr;
    if (pieced)
    {
        const FieldSplit split = fieldSplit(chunk, L.lanes, L.nseg, plan->thickness, plan->nodes, perSM,
                                            refined);
        const size_t pieces = (size_t)split.groups * (size_t)split.parts;
        if (pieces > 1 && scratchAlloc(&partial, pieces * (size_t)chunk * width * sizeof(double), st) == cudaSuccess)
        {
            L.split = split;
            L.d_partial = static_cast<double *>(partial);
        }
        else if (pieces > 1)
        {
            partial = nullptr;
            cudaGetLastError();  // an allocation that failed is not this call's error
            if (autoFp64)
                L.lanes = autoLanesOnePiece64(point_count);
        }
    }
    int rc = CCOIL_OK;
    for (long long off = 0; off < point_count && rc == CCOIL_OK; off += chunk)
    {
        FieldLaunch C = L;
        C.d_points = L.d_points + 3 * off;
        C.d_out = L.d_out + (long long)width * off;
        C.npts = std::min(chunk, point_count - off);
        rc = launchFields(C, stream);
    }
    if (partial)
        cudaFreeAsync(partial, st);
    if (rc == CCOIL_OK && ordered)
        rc = scatterResults(static_cast<const double *>(plan->sortedOut.ptr), static_cast<const int *>(plan->order.ptr),
                            point_count, width, dOut, stream);
    return rc;
}
} // namespace

extern "C" {

int ccoil_abi_version(void) { return CCOIL_ABI_VERSION; }

const char *ccoil_last_error_message(void) { return t_error; }

int ccoil_coil_init(double inner_radius, double thickness, double length, int num_turns, double current,
                    double sine_frequency, const double position[3], double y_axis_angle, double z_axis_angle,
                    double precision_factor, int gpu_increments, ccoil_coil_t *out)
{
    if (!out)
        return fail(CCOIL_ERR_INVALID_ARGUMENT, "out is null");
    if (!(inner_radius > 0.0) || thickness < 0.0 || length < 0.0 || num_turns < 1 || gpu_increments < 0 ||
        gpu_increments > kMaxOrder)
        return fail(CCOIL_ERR_INVALID_ARGUMENT,
                    "coil needs inner_radius > 0, thickness >= 0, length >= 0, num_turns >= 1, "
                    "gpu_increments in [0, 100]");
    initCoil(inner_radius, thickness, length, num_turns, current, sine_frequency, position, y_axis_angle,
             z_axis_angle, *out);
    out->precision = coilPrecision(*out, precision_factor, gpu_increments);
    return CCOIL_OK;
}

int ccoil_coils_from_params(const double *params, const ccoil_precision_args_t *precisions, int coil_count,
                            ccoil_coil_t *coils)
{
    if (coil_count < 0 || (coil_count > 0 && (!params || !precisions || !coils)))
        return fail(CCOIL_ERR_INVALID_ARGUMENT, "null params, precisions or coils, or coil_count < 0");
    for (int c = 0; c < coil_count; ++c)
    {
        const double *q = params + 9 * c;
        const int rc = ccoil_coil_init(q[0], q[1], q[2], 1, q[3], 0.0, q + 4, q[7], q[8], 5.0, 0, coils + c);
        if (rc != CCOIL_OK)
            return rc;
        coils[c].precision = precisions[c];
    }
    return CCOIL_OK;
}

int ccoil_precision_arguments(const ccoil_coil_t *coil, double precision_factor, int gpu_increments,
                              ccoil_precision_args_t *out)
{
    if (!coil || !out)
        return fail(CCOIL_ERR_INVALID_ARGUMENT, "null argument");
    if (gpu_increments < 0 || gpu_increments > kMaxOrder)
        return fail(CCOIL_ERR_INVALID_ARGUMENT, "gpu_increments must be in [0, 100]");
    *out = coilPrecision(*coil, precision_factor, gpu_increments);
    return CCOIL_OK;
}

int ccoil_pair_arguments(const ccoil_coil_t *primary, const ccoil_coil_t *secondary, double precision_factor,
                         int gpu_increments, int z_axis_case, int pure_gpu, ccoil_precision_args_t *primary_out,
                         ccoil_precision_args_t *secondary_out)
{
    if (!primary || !secondary || !primary_out || !secondary_out)
        return fail(CCOIL_ERR_INVALID_ARGUMENT, "null argument");
    if (gpu_increments < 0 || gpu_increments > kMaxOrder)
        return fail(CCOIL_ERR_INVALID_ARGUMENT, "gpu_increments must be in [0, 100]");
    pairPrecision(*primary, *secondary, precision_factor, gpu_increments, z_axis_case != 0, pure_gpu != 0,
                  *primary_out, *secondary_out);
    return CCOIL_OK;
}

int ccoil_legendre(int order, double *nodes, double *weights)
{
    if (order < 1 || order > kMaxOrder || !nodes || !weights)
        return fail(CCOIL_ERR_INVALID_ARGUMENT, "order must be in [1, 100] and buffers non-null");
    std::memcpy(nodes, legendreNodes(order), sizeof(double) * order);
    std::memcpy(weights, legendreWeights(order), sizeof(double) * order);
    return CCOIL_OK;
}

int ccoil_field_plan_create(const ccoil_coil_t *coils, int coil_count, int field, int precision,
                            ccoil_field_plan_t **plan)
{
    if (!plan)
        return fail(CCOIL_ERR_INVALID_ARGUMENT, "plan is null");
    *plan = nullptr;
    ccoil_field_plan *p = new (std::nothrow) ccoil_field_plan();
    if (!p)
        return fail(CCOIL_ERR_OUT_OF_MEMORY, "host allocation failed");
    int rc = buildTables(*p, coils, coil_count, field, precision);
    if (rc == CCOIL_OK && !p->set.blob.empty())
    {
        rc = p->tables.reserve(p->set.blob.size(), p->owner);
        if (rc == CCOIL_OK)
        {
            const cudaError_t e =
                cudaMemcpy(p->tables.ptr, p->set.blob.data(), p->set.blob.size(), cudaMemcpyHostToDevice);
            if (e != cudaSuccess)
                rc = cudaFail(e, "cudaMemcpy");
        }
    }
    if (rc != CCOIL_OK)
    {
        ccoil_field_plan_destroy(p);
        return rc;
    }
    *plan = p;
    return CCOIL_OK;
}

int ccoil_field_plan_execute(ccoil_field_plan_t *plan, const double *points, long long point_count, double *out,
                             int memory, int lanes_per_point, void *stream)
{
    if (!plan)
        return fail(CCOIL_ERR_INVALID_ARGUMENT, "plan is null");
    int rc = checkExecute(points, point_count, out, memory);
    if (rc != CCOIL_OK)
        return rc;
    if (lanes_per_point != 0 && !validLanes(lanes_per_point))
        return fail(CCOIL_ERR_INVALID_ARGUMENT, "lanes_per_point must be 0, 1, 2, 4, 8, 16 or 32");
    if (point_count == 0)
        return CCOIL_OK;
    // grid.x limit: 2^31-1 CTAs of 128/lanes points
    if (point_count > (1LL << 36))
        return fail(CCOIL_ERR_INVALID_ARGUMENT, "point_count above 2^36");
    if (memory == CCOIL_MEMORY_DEVICE)
        return runFields(plan, points, point_count, out, lanes_per_point, stream);

    const size_t inBytes = sizeof(double) * 3 * (size_t)point_count;
    const size_t outBytes = sizeof(double) * (plan->field == CCOIL_FIELD_G ? 9 : 3) * (size_t)point_count;
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    rc = plan->points.reserve(inBytes, plan->owner);
    if (rc == CCOIL_OK)
        rc = plan->out.reserve(outBytes, plan->owner);
    if (rc != CCOIL_OK)
        return rc;
    cudaError_t e = cudaMemcpyAsync(plan->points.ptr, points, inBytes, cudaMemcpyHostToDevice, st);
    if (e != cudaSuccess)
        return cudaFail(e, "host->device copy of points");
    rc = runFields(plan, static_cast<const double *>(plan->points.ptr), point_count,
                   static_cast<double *>(plan->out.ptr), lanes_per_point, stream);
    return rc == CCOIL_OK ? finishHost(out, static_cast<const double *>(plan->out.ptr), outBytes, st) : rc;
}

int ccoil_field_plan_segment_count(const ccoil_field_plan_t *plan, int *count)
{
    if (!plan || !count)
        return fail(CCOIL_ERR_INVALID_ARGUMENT, "null plan or count");
    *count = (int)plan->set.segs.size();
    return CCOIL_OK;
}

int ccoil_field_plan_destroy(ccoil_field_plan_t *plan)
{
    if (!plan)
        return CCOIL_OK;
    // no kernel on any stream may still use the buffers
    if (!plan->owner.scoped)
        cudaDeviceSynchronize();
    for (DeviceBuffer *b : {&plan->tables, &plan->points, &plan->out, &plan->work, &plan->workCount, &plan->contrib,
                            &plan->refineSegs, &plan->refinedTotal, &plan->orderScratch, &plan->order,
                            &plan->sortedPoints, &plan->sortedOut})
        b->release(plan->owner);
    delete plan;
    return CCOIL_OK;
}

int ccoil_compute_fields(const ccoil_coil_t *coils, int coil_count, const double *points, long long point_count,
                         int field, int precision, double *out, int memory, void *stream)
{
    // the execute step's own checks, before any device work
    int rc = checkExecute(points, point_count, out, memory);
    if (rc != CCOIL_OK)
        return rc;
    if (point_count > (1LL << 36))
        return fail(CCOIL_ERR_INVALID_ARGUMENT, "point_count above 2^36");
    ccoil_field_plan *p = new (std::nothrow) ccoil_field_plan();
    if (!p)
        return fail(CCOIL_ERR_OUT_OF_MEMORY, "host allocation failed");
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    p->owner.scoped = true;
    p->owner.stream = st;
    rc = buildTables(*p, coils, coil_count, field, precision);
    if (rc == CCOIL_OK && point_count > 0)
    {
        // one block of device memory for the call: tables, and with host arrays the
        // points and the results; few points travel with the tables in one copy
        const size_t inBytes = sizeof(double) * 3 * (size_t)point_count;
        const size_t outBytes = sizeof(double) * (field == CCOIL_FIELD_G ? 9 : 3) * (size_t)point_count;
        const bool host = memory == CCOIL_MEMORY_HOST, together = host && inBytes <= kPackedCopyBytes;
        std::vector<unsigned char> &image = p->set.blob;
        const size_t pointsAt = (image.size() + 255) / 256 * 256, outAt = (pointsAt + inBytes + 255) / 256 * 256;
        const size_t tableBytes = image.size();
        rc = p->tables.reserve(host ? outAt + outBytes : std::max<size_t>(tableBytes, 16), p->owner);
        if (rc == CCOIL_OK)
        {
            unsigned char *base = static_cast<unsigned char *>(p->tables.ptr);
            if (together)
            {
                image.resize(pointsAt + inBytes);
                std::memcpy(image.data() + pointsAt, points, inBytes);
            }
            cudaError_t e = image.empty() ? cudaSuccess
                                          : cudaMemcpyAsync(base, image.data(), image.size(), cudaMemcpyHostToDevice, st);
            if (e == cudaSuccess && host && !together)
                e = cudaMemcpyAsync(base + pointsAt, points, inBytes, cudaMemcpyHostToDevice, st);
            if (e != cudaSuccess)
                rc = cudaFail(e, "host->device copy");
            double *dOut = host ? reinterpret_cast<double *>(base + outAt) : out;
            if (rc == CCOIL_OK)
                rc = runFields(p, host ? reinterpret_cast<const double *>(base + pointsAt) : points, point_count, dOut,
                               0, stream);
            if (rc == CCOIL_OK && host)
                rc = finishHost(out, dOut, outBytes, st);
            else if (rc == CCOIL_OK && (e = cudaStreamSynchronize(st)) != cudaSuccess)
                rc = cudaFail(e, "field evaluation");
        }
    }
    ccoil_field_plan_destroy(p);
    return rc;
}

int ccoil_check_bounded_wait(long long limit_cycles, void *stream)
{
    if (limit_cycles < 0 || limit_cycles > 4000000000LL)
        return failMessage(CCOIL_ERR_INVALID_ARGUMENT, "limit_cycles must lie in [0, 4e9]");
    const int rc = checkBoundedWait(limit_cycles, stream);
    // this call reports its own timeout; field calls report only theirs
    long long count = 0;
    if (readTimeouts(count) == CCOIL_OK)
        g_timeoutsReported.store(count);
    return rc;
}

int ccoil_set_point_ordering(int enabled)
{
    g_pointOrdering.store(enabled ? 1 : 0);
    return CCOIL_OK;
}

int ccoil_point_ordering(void) { return g_pointOrdering.load(); }

}  // extern "C"

double ccoil::refineFraction() { return g_refineFraction.load(); }

extern "C" {

int ccoil_set_refine_fraction(double fraction)
{
    if (!(fraction >= 0.0) || !std::isfinite(fraction))
        return failMessage(CCOIL_ERR_INVALID_ARGUMENT, "the refinement fraction must be finite and >= 0");
    g_refineFraction.store(fraction);
    return CCOIL_OK;
}

double ccoil_refine_fraction(void) { return g_refineFraction.load(); }

int ccoil_field_plan_refined_pairs(ccoil_field_plan_t *plan, long long *count)
{
    if (!plan || !count)
        return failMessage(CCOIL_ERR_INVALID_ARGUMENT, "null plan or count");
    *count = 0;
    if (plan->precision != CCOIL_PRECISION_FP32_REFINED || !plan->refinedTotal.ptr)
        return CCOIL_OK;
    unsigned long long v = 0;
    cudaError_t e = cudaMemcpy(&v, plan->refinedTotal.ptr, sizeof(v), cudaMemcpyDeviceToHost);
    if (e != cudaSuccess)
        return cudaFail(e, "refinement count");
    *count = (long long)v;
    return CCOIL_OK;
}

int ccoil_inject_allocation_failures(int count)
{
    if (count < 0)
        return failMessage(CCOIL_ERR_INVALID_ARGUMENT, "count < 0");
    g_failAllocations.store(count);
    return CCOIL_OK;
}

long long ccoil_timeout_count(void)
{
    long long v = 0;
    if (readTimeouts(v) != CCOIL_OK)
        return -1;
    return v;
}

} // extern "C"
