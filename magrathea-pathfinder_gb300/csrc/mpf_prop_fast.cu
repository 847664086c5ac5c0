// Throughput mode: FP32 gather arithmetic through the per-cell stencil
// records, FP64 RK4 state (with FMA).
#include "mpf_fast.cuh"
#include "mpf_internal.h"
#include "mpf_tune.h"

#include <algorithm>
#include <cstdio>
#include <cstdlib>
#include <map>
#include <mutex>
#include <thread>
#include <tuple>
#include <utility>

namespace mpf {
cudaError_t launch_gather_exact(const DevTree& T, int kind, const double* d_xyz, long long n, void* d_out, cudaStream_t stream);

// The kernel instantiation a launch uses: per interpolation order and mode
// (surfaces / sources / wide surfaces, per-ray surfaces, direction launches,
// trajectories; Born rays; a velocity-field octree, plain surfaces only).
static int fast_mode(const DevTree& T, const PropParams& P, const PropOut& O)
{
    if (P.homogeneous == 2) return P.ray_stop ? 0 : 1;
    if (P.ray_stop) return (P.order == 1) ? 2 : 3;
    if (P.wide || P.ray_planes || P.direct || O.traj) return (P.order == 1) ? 4 : 5;
    if (T.vel) return (P.order == 1) ? 8 : 9;
    return (P.order == 1) ? 6 : 7;
}

// A velocity-field octree runs the FP32-gather kernel in the plain mode only
// (surface records: propagation and maps); its other modes (Born, source,
// bundle and trajectory rays) run the float64 kernel.
static bool fast_mode_supported(const DevTree& T, const PropParams& P, const PropOut& O)
{
    const int m = fast_mode(T, P, O);
    return !T.vel || m == 8 || m == 9;
}

// Launches rays [lo, n) of the batch as grid blocks of tpb threads, each warp
// claiming rays x depth rays at a time and tracing them with per_ray lanes
// each, in the order of perm (or as given).
static void launch_fast_kernel(long long grid, int tpb, int rays, int per_ray, int depth, long long lo, const DevTree& T, const DevCosmo& C,
                               const PropParams& P, const double* d_launch, long long n, const PropOut& O,
                               unsigned long long* queue, const int* perm, cudaStream_t stream)
{
    const unsigned g = (unsigned)grid;
    const size_t smem = (size_t)tpb * (per_ray > 1 ? kSharedRaySlotBytes : kSlotBytes);
    switch (fast_mode(T, P, O)) {
    // Born rays: the field is homogeneous, so the interpolation order does
    // not enter (the Jacobian gathers are TSC)
    case 0: k_propagate_fast<2, true, false, true><<<g, tpb, smem, stream>>>(T, C, P, d_launch, n, O, queue, rays, per_ray, depth, lo, perm); break;
    case 1: k_propagate_fast<2, false, true, true><<<g, tpb, smem, stream>>>(T, C, P, d_launch, n, O, queue, rays, per_ray, depth, lo, perm); break;
    case 2: k_propagate_fast<1, true, false><<<g, tpb, smem, stream>>>(T, C, P, d_launch, n, O, queue, rays, per_ray, depth, lo, perm); break;
    case 3: k_propagate_fast<2, true, false><<<g, tpb, smem, stream>>>(T, C, P, d_launch, n, O, queue, rays, per_ray, depth, lo, perm); break;
    case 4: k_propagate_fast<1, false, true><<<g, tpb, smem, stream>>>(T, C, P, d_launch, n, O, queue, rays, per_ray, depth, lo, perm); break;
    case 5: k_propagate_fast<2, false, true><<<g, tpb, smem, stream>>>(T, C, P, d_launch, n, O, queue, rays, per_ray, depth, lo, perm); break;
    case 6: k_propagate_fast<1, false, false><<<g, tpb, smem, stream>>>(T, C, P, d_launch, n, O, queue, rays, per_ray, depth, lo, perm); break;
    case 8: k_propagate_fast<1, false, false, false, true><<<g, tpb, smem, stream>>>(T, C, P, d_launch, n, O, queue, rays, per_ray, depth, lo, perm); break;
    case 9: k_propagate_fast<2, false, false, false, true><<<g, tpb, smem, stream>>>(T, C, P, d_launch, n, O, queue, rays, per_ray, depth, lo, perm); break;
    default: k_propagate_fast<2, false, false><<<g, tpb, smem, stream>>>(T, C, P, d_launch, n, O, queue, rays, per_ray, depth, lo, perm); break;
    }
}

// Launch shape of the persistent kernel.  A ray's steps are one serial chain,
// and what a warp spends on a step grows with the rays in it (other cells,
// levels, table intervals and step counts: 32.6 ms for one ray a warp, 46 for
// 16, 60 to 72 for 32 on a refined cone with the Jacobian) and with the warps
// that share its SM sub-partition.  So a batch of fewer rays than one full
// warp per sub-partition is spread over one-warp blocks, one per
// sub-partition (4 an SM; two a sub-partition measured 48 -> 79 ms at 4096
// rays, half a warp each 48 -> 55), with the rays' Jacobian gathers shared out
// to the lanes left over.  Above that, blocks of one warp while they do not
// fill the warp slots, then blocks of kFastThreads, as many as are resident.
struct FastShape {
    long long grid;
    int tpb;
    int rays, per_ray;   // rays of a warp, lanes of a ray
    bool full;           // blocks of kFastThreads: the autotuner's case
};
static FastShape fast_launch_shape(long long n, int blocks_per_sm, int sms, bool jacobian)
{
    const long long slots = (long long)blocks_per_sm * sms * (kFastThreads / 32);
    const int rays = (int)std::min<long long>(32, (n + 4 * sms - 1) / (4 * sms));
    const int per_ray = jacobian ? rays_to_lanes(rays) : 1;
    const long long warps = (n + rays - 1) / rays;
    if (warps < slots) return FastShape{warps, 32, rays, per_ray, false};
    return FastShape{std::min<long long>((n + kFastThreads - 1) / kFastThreads, (long long)blocks_per_sm * sms), kFastThreads, 32, 1, true};
}

// ---------------------------------------------------------------------------
// Order of a batch's rays on a refined octree: by the Morton index of their
// direction on a 128 x 128 grid over the directions' own bounding box.  The
// rays of a warp then read the same stencils, and the warps at work at one time
// the same cells, whatever the caller's order: 160 000 rays to z = 2 on a
// refined cone 432 -> 393 ms from rows of a pixel grid and 709 -> 394 ms from a
// shuffled list, 60 000 204 -> 188 and 290 -> 188, 20 011 103 -> 97 and 124 ->
// 98; the maps of 60 000 pixels to z = 1 138 -> 118.  Rays in one square of the grid come
// in any order; a ray's result does not depend on it.  Below kOrderMinRays the
// five launches (25 us) cost more than they give; on an octree of one level,
// where the rays of a warp hardly diverge, rows measured 6 % faster than the
// squares (160 000 rays 17.3 against 18.4 ms); bundle, source and Born rays
// come pixel by pixel or sorted.  A call under stream capture keeps the
// caller's order: a graph would hold the order's memory.
// ---------------------------------------------------------------------------
constexpr long long kOrderMinRays = 1ll << 14, kOrderMaxRays = 1ll << 22;
constexpr int kOrderBits = 7;   // per axis
constexpr int kOrderBins = 1 << (2 * kOrderBits);

// the direction on the octahedral map about +x (the axis of narrow cones)
static __device__ __forceinline__ void direction_uv(const double* L, float& u, float& v)
{
    const float x = (float)(L[3] - L[0]), y = (float)(L[4] - L[1]), z = (float)(L[5] - L[2]);
    const float s = 1.f / (fabsf(x) + fabsf(y) + fabsf(z));
    u = y * s;
    v = z * s;
    if (x < 0.f) {
        const float fu = (1.f - fabsf(v)) * (u < 0.f ? -1.f : 1.f), fv = (1.f - fabsf(u)) * (v < 0.f ? -1.f : 1.f);
        u = fu;
        v = fv;
    }
}

// unsigned integers in the order of the floats
static __device__ __forceinline__ unsigned ordered(float f)
{
    const unsigned b = __float_as_uint(f);
    return (b & 0x80000000u) ? ~b : (b | 0x80000000u);
}
static __device__ __forceinline__ float unordered(unsigned o) { return __uint_as_float((o & 0x80000000u) ? (o & 0x7fffffffu) : ~o); }

// w: the bins' counts, then the bounds (u and v smallest, u and v largest)
static __global__ void k_order_reset(unsigned* w)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < kOrderBins) w[i] = 0u;
    else if (i < kOrderBins + 4) w[i] = (i < kOrderBins + 2) ? 0xffffffffu : 0u;
}

static __global__ void __launch_bounds__(256) k_order_bounds(const double* __restrict__ launch, long long n, unsigned* w)
{
    __shared__ unsigned part[4];
    if (threadIdx.x < 4) part[threadIdx.x] = (threadIdx.x < 2) ? 0xffffffffu : 0u;
    __syncthreads();
    unsigned b[4] = {0xffffffffu, 0xffffffffu, 0u, 0u};
    for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x) {
        float u, v;
        direction_uv(launch + 6 * i, u, v);
        if (u == u && v == v) {
            b[0] = min(b[0], ordered(u)); b[2] = max(b[2], ordered(u));
            b[1] = min(b[1], ordered(v)); b[3] = max(b[3], ordered(v));
        }
    }
    for (int q = 0; q < 4; ++q) {
        const unsigned r = (q < 2) ? __reduce_min_sync(0xffffffffu, b[q]) : __reduce_max_sync(0xffffffffu, b[q]);
        if ((threadIdx.x & 31) == 0) {
            if (q < 2) atomicMin(part + q, r);
            else atomicMax(part + q, r);
        }
    }
    __syncthreads();
    if (threadIdx.x < 2) atomicMin(w + kOrderBins + threadIdx.x, part[threadIdx.x]);
    else if (threadIdx.x < 4) atomicMax(w + kOrderBins + threadIdx.x, part[threadIdx.x]);
}

static __device__ __forceinline__ unsigned order_bin(const double* L, const unsigned* bounds)
{
    float u, v;
    direction_uv(L, u, v);
    const float u0 = unordered(bounds[0]), v0 = unordered(bounds[1]);
    // one scale for both axes: the squares of the grid are squares of directions
    const float side = fmaxf(unordered(bounds[2]) - u0, unordered(bounds[3]) - v0);
    const float sc = (float)(1 << kOrderBits) / fmaxf(side, 1e-30f);
    const int last = (1 << kOrderBits) - 1;
    const unsigned a = (unsigned)min(max((int)((u - u0) * sc), 0), last), b = (unsigned)min(max((int)((v - v0) * sc), 0), last);
    unsigned k = 0;
#pragma unroll
    for (int q = 0; q < kOrderBits; ++q) k |= ((a >> q) & 1u) << (2 * q) | ((b >> q) & 1u) << (2 * q + 1);
    return k;
}

static __global__ void k_order_count(const double* __restrict__ launch, long long n, unsigned* w)
{
    const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) atomicAdd(w + order_bin(launch + 6 * i, w + kOrderBins), 1u);
}

// counts to first positions: one block
static __global__ void __launch_bounds__(1024) k_order_scan(unsigned* w)
{
    __shared__ unsigned part[1024];
    constexpr int per = kOrderBins / 1024;
    uint4* const mine = reinterpret_cast<uint4*>(w + threadIdx.x * per);
    uint4 c[per / 4];
    unsigned s = 0;
#pragma unroll
    for (int q = 0; q < per / 4; ++q) { c[q] = mine[q]; s += c[q].x + c[q].y + c[q].z + c[q].w; }
    part[threadIdx.x] = s;
    __syncthreads();
    for (int off = 1; off < 1024; off <<= 1) {
        const unsigned v = (threadIdx.x >= off) ? part[threadIdx.x - off] : 0u;
        __syncthreads();
        part[threadIdx.x] += v;
        __syncthreads();
    }
    unsigned at = part[threadIdx.x] - s;
#pragma unroll
    for (int q = 0; q < per / 4; ++q) {
        const uint4 o = make_uint4(at, at + c[q].x, at + c[q].x + c[q].y, at + c[q].x + c[q].y + c[q].z);
        at = o.w + c[q].w;
        mine[q] = o;
    }
}

static __global__ void k_order_scatter(const double* __restrict__ launch, long long n, unsigned* w, int* __restrict__ perm)
{
    const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) perm[atomicAdd(w + order_bin(launch + 6 * i, w + kOrderBins), 1u)] = (int)i;
}

// Memory of the orders: at most kOrderBuffers buffers per device and octree,
// each of the largest batch's size (16 MiB, so that none is ever replaced or
// outgrown), made when a call finds none free and freed with the octree.  A
// call claims one until its last kernel is queued and records the buffer's
// event behind that.  A buffer is free again once its event has passed, or for
// the stream whose work it still serves; whoever takes it waits for the event
// on its own stream, so that a stream handle or thread that comes again cannot
// read or write it early.  With none free (more calls in flight on different
// streams than buffers) a call traces in the caller's order.
constexpr int kOrderBuffers = 8;
struct OrderBuffer {
    unsigned* p = nullptr;
    cudaEvent_t done = nullptr;
    cudaStream_t stream = nullptr;   // of the last call (and its thread, where a handle stands for a stream of each)
    std::thread::id who;
    bool claimed = false;
};
struct OrderPool {
    OrderBuffer buffer[kOrderBuffers];
};
static std::mutex g_order_mu;
static std::map<std::pair<int, const void*>, OrderPool> g_orders;

// A capture of another thread must not see this thread's allocation or event
// queries as its own.
struct OutsideCapture {
    cudaStreamCaptureMode mode = cudaStreamCaptureModeRelaxed;
    OutsideCapture() { cudaThreadExchangeStreamCaptureMode(&mode); }
    ~OutsideCapture() { cudaThreadExchangeStreamCaptureMode(&mode); }
};

static void free_orders(const void* keys)
{
    std::lock_guard<std::mutex> lock(g_order_mu);
    for (auto it = g_orders.begin(); it != g_orders.end();) {
        if (it->first.second != keys) {
            ++it;
            continue;
        }
        for (OrderBuffer& b : it->second.buffer) {
            if (b.p) cudaFree(b.p);
            if (b.done) cudaEventDestroy(b.done);
        }
        it = g_orders.erase(it);
    }
}

// A call's hold on a buffer, given back behind the work queued on its stream.
struct OrderClaim {
    OrderBuffer* b = nullptr;
    cudaStream_t stream = nullptr;
    std::thread::id who;
    OrderClaim() = default;
    OrderClaim(const OrderClaim&) = delete;
    OrderClaim& operator=(const OrderClaim&) = delete;
    ~OrderClaim()
    {
        if (!b) return;
        const bool queued = !b->p || cudaEventRecord(b->done, stream) == cudaSuccess;
        std::lock_guard<std::mutex> lock(g_order_mu);
        b->stream = stream;
        b->who = who;
        b->claimed = !queued;   // without its event nobody may take it again
    }
    // a buffer for work on s; false: none is free, or there is no memory
    bool take(int dev, const void* keys, cudaStream_t s)
    {
        const OutsideCapture outside;
        const std::thread::id id = (s == cudaStreamPerThread) ? std::this_thread::get_id() : std::thread::id();
        OrderBuffer* got = nullptr;
        {
            std::lock_guard<std::mutex> lock(g_order_mu);
            OrderBuffer *own = nullptr, *idle = nullptr, *fresh = nullptr;
            for (OrderBuffer& q : g_orders[std::make_pair(dev, keys)].buffer) {
                if (q.claimed) continue;
                if (!q.p) {
                    if (!fresh) fresh = &q;
                } else if (q.stream == s && q.who == id) {
                    own = &q;
                } else if (!idle) {
                    if (cudaEventQuery(q.done) == cudaSuccess) idle = &q;
                    else (void)cudaGetLastError();   // not ready
                }
            }
            got = own ? own : idle ? idle : fresh;
            if (!got) return false;
            got->claimed = true;
        }
        b = got;
        stream = s;
        who = id;
        if (b->p) return cudaStreamWaitEvent(s, b->done, 0) == cudaSuccess;
        if (cudaEventCreateWithFlags(&b->done, cudaEventDisableTiming) != cudaSuccess) {
            (void)cudaGetLastError();
            b->done = nullptr;
            return false;
        }
        if (cudaMalloc(&b->p, (size_t)(kOrderBins + 4 + kOrderMaxRays) * sizeof(int)) != cudaSuccess) {
            (void)cudaGetLastError();   // no room
            b->p = nullptr;
            cudaEventDestroy(b->done);
            b->done = nullptr;
            return false;
        }
        return true;
    }
};

// The order of a batch's rays on the device, in the buffer of `claim` (to be
// held until the last kernel that reads it is queued), or null where the
// caller's stays.
static cudaError_t order_rays(const DevTree& T, const double* d_launch, long long n, int sms, cudaStream_t s, OrderClaim& claim,
                              const int** perm)
{
    *perm = nullptr;
    if (n < kOrderMinRays || n > kOrderMaxRays || T.Lmax <= T.Lt) return cudaSuccess;
    cudaStreamCaptureStatus cap = cudaStreamCaptureStatusNone;
    if (cudaStreamIsCapturing(s, &cap) != cudaSuccess) {
        (void)cudaGetLastError();
        return cudaSuccess;
    }
    if (cap != cudaStreamCaptureStatusNone) return cudaSuccess;
    int dev = 0;
    const cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    if (!claim.take(dev, T.keys, s)) return cudaSuccess;
    unsigned* const w = claim.b->p;
    int* const order = reinterpret_cast<int*>(w + kOrderBins + 4);
    const unsigned blocks = (unsigned)((n + 255) / 256);
    k_order_reset<<<(kOrderBins + 4 + 255) / 256, 256, 0, s>>>(w);
    k_order_bounds<<<std::min(blocks, (unsigned)sms), 256, 0, s>>>(d_launch, n, w);
    k_order_count<<<blocks, 256, 0, s>>>(d_launch, n, w);
    k_order_scan<<<1, 1024, 0, s>>>(w);
    k_order_scatter<<<blocks, 256, 0, s>>>(d_launch, n, w, order);
    *perm = order;
    return cudaGetLastError();
}

// Work-queue counter and occupancy of the persistent kernel, per (device,
// stream): calls on one stream are ordered and may share a counter; calls on
// different streams (or devices) may run at the same time and must not.  One
// 8-byte counter per stream handle seen, kept for the process's lifetime.
// cudaStreamPerThread is one handle value for as many streams as there are
// host threads, so it is keyed per calling thread as well.  The counter is
// zeroed by an asynchronous memset before each launch, so a stream must not
// be shared by host threads that call at the same time (their memsets and
// launches could interleave): each concurrent caller passes its own stream.
struct FastLaunchState {
    unsigned long long* queue = nullptr;
    int blocks_per_sm = 0, sms = 0;
};
static cudaError_t fast_launch_state(cudaStream_t stream, FastLaunchState* out)
{
    static std::mutex mu;
    static std::map<std::tuple<int, cudaStream_t, std::thread::id>, FastLaunchState> states;
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    const std::thread::id who = (stream == cudaStreamPerThread) ? std::this_thread::get_id() : std::thread::id();
    std::lock_guard<std::mutex> lock(mu);
    FastLaunchState& s = states[std::make_tuple(dev, stream, who)];
    if (!s.queue) {
        e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&s.blocks_per_sm, k_propagate_fast<2, false, false>, kFastThreads, kFastThreads * kSlotBytes);
        if (e == cudaSuccess) e = cudaDeviceGetAttribute(&s.sms, cudaDevAttrMultiProcessorCount, dev);
        if (e == cudaSuccess) e = cudaMalloc(&s.queue, sizeof(unsigned long long));
        if (e != cudaSuccess) {
            s = FastLaunchState{};
            return e;
        }
        if (s.blocks_per_sm < 1) s.blocks_per_sm = 1;
    }
    *out = s;
    return cudaSuccess;
}

// ---------------------------------------------------------------------------
// Autotuner of the persistent launch shape: threads per block and the depth
// of a warp's claim on the work queue (32 x depth rays).  The first batch of
// at least kTuneMinRays rays for a (device, octree, kernel mode) is split into
// one slice per candidate shape (mpf_tune.h; contiguous parts of the caller's
// list where the rays are not reordered); each slice is traced with its shape and
// timed with CUDA events, and its photon-steps are summed on the device.  The
// shape with the most photon-steps per second is kept for that key and used
// by every later launch.  Every ray is traced exactly once and its results do
// not depend on the shape, so tuning changes no output; the tuning call
// waits for its slices.  MPF_AUTOTUNE=0 keeps the default shape.
struct TuneShape {
    int tpb, depth;
};
static const TuneShape kTuneCandidates[] = {{kFastThreads, 1}, {64, 1}, {32, 1}, {kFastThreads, 2}};
constexpr int kTuneN = kTuneSlices;
constexpr long long kTuneMinRays = 1ll << 17;

struct TuneResult {
    int done = 0;
    TuneShape best{kFastThreads, 1};
    double rate[kTuneN] = {0, 0, 0, 0};   // photon-steps/s of each candidate
};
static std::mutex g_tune_mu;
static std::map<std::tuple<int, const void*, int>, TuneResult> g_tune;

static __global__ void k_sum_steps(const long long* __restrict__ steps, const int* __restrict__ perm, long long lo, long long hi,
                                   unsigned long long* __restrict__ out)
{
    unsigned long long s = 0;
    for (long long i = lo + (long long)blockIdx.x * blockDim.x + threadIdx.x; i < hi; i += (long long)gridDim.x * blockDim.x)
    {
        const long long t = steps[perm ? perm[i] : i];
        s += (unsigned long long)(t > 0 ? t - 1 : 0);
    }
    for (int o = 16; o > 0; o >>= 1) s += __shfl_down_sync(0xffffffffu, s, o);
    if ((threadIdx.x & 31) == 0) atomicAdd(out, s);
}

static __global__ void k_deal(const int* __restrict__ perm, long long n, int* __restrict__ dealt)
{
    const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) dealt[i] = perm[tune_dealt(i, n)];
}

// resident blocks per SM of the kernel at tpb threads (at least 1)
static int blocks_per_sm_at(int tpb)
{
    int b = 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&b, k_propagate_fast<2, false, false>, tpb, (size_t)tpb * kSlotBytes) != cudaSuccess) b = 1;
    return std::max(1, b);
}

// the grid of a shape for `rays` rays: every SM's resident blocks, fewer when
// the rays do not fill them
static long long shape_grid(const TuneShape& sh, long long rays, int sms)
{
    const long long need = (rays + (long long)sh.tpb * sh.depth - 1) / ((long long)sh.tpb * sh.depth);
    return std::max<long long>(1, std::min<long long>(need, (long long)blocks_per_sm_at(sh.tpb) * sms));
}

// Tunes the shape on this batch (tracing all of it); fills *res.
static cudaError_t tune_and_launch(const DevTree& T, const DevCosmo& C, const PropParams& P, const double* d_launch,
                                   long long n, const PropOut& O, unsigned long long* queue, const int* perm, int sms, cudaStream_t stream,
                                   TuneResult* res)
{
    unsigned long long* dsum = nullptr;
    int* dealt = nullptr;
    cudaEvent_t ev[kTuneN + 1] = {};
    cudaError_t e = cudaMalloc(&dsum, kTuneN * sizeof(unsigned long long));
    if (e == cudaSuccess && perm) e = cudaMalloc(&dealt, (size_t)n * sizeof(int));
    if (e == cudaSuccess && perm) {
        k_deal<<<(unsigned)((n + 255) / 256), 256, 0, stream>>>(perm, n, dealt);
        perm = dealt;
        e = cudaGetLastError();
    }
    if (e == cudaSuccess) e = cudaMemsetAsync(dsum, 0, kTuneN * sizeof(unsigned long long), stream);
    for (int k = 0; k <= kTuneN && e == cudaSuccess; ++k) e = cudaEventCreate(&ev[k]);
    if (e == cudaSuccess) e = cudaEventRecord(ev[0], stream);
    const long long slice = perm ? tune_slice(n) : n / kTuneN;
    for (int k = 0; k < kTuneN && e == cudaSuccess; ++k) {
        const long long lo = k * slice, hi = (k == kTuneN - 1) ? n : lo + slice;
        const TuneShape& sh = kTuneCandidates[k];
        e = cudaMemsetAsync(queue, 0, sizeof(unsigned long long), stream);
        if (e != cudaSuccess) break;
        launch_fast_kernel(shape_grid(sh, hi - lo, sms), sh.tpb, 32, 1, sh.depth, lo, T, C, P, d_launch, hi, O, queue, perm, stream);
        if ((e = cudaGetLastError()) != cudaSuccess) break;
        e = cudaEventRecord(ev[k + 1], stream);
        if (e == cudaSuccess) k_sum_steps<<<64, 256, 0, stream>>>(O.steps, perm, lo, hi, dsum + k);
        if (e == cudaSuccess) e = cudaGetLastError();
    }
    unsigned long long ps[kTuneN] = {0, 0, 0, 0};
    if (e == cudaSuccess) e = cudaMemcpyAsync(ps, dsum, sizeof(ps), cudaMemcpyDeviceToHost, stream);
    if (e == cudaSuccess) e = cudaStreamSynchronize(stream);
    if (e == cudaSuccess) {
        double best = -1.0;
        for (int k = 0; k < kTuneN; ++k) {
            float ms = 0.f;
            cudaEventElapsedTime(&ms, ev[k], ev[k + 1]);
            res->rate[k] = (ms > 0.f) ? (double)ps[k] / (ms * 1e-3) : 0.0;
            if (res->rate[k] > best) {
                best = res->rate[k];
                res->best = kTuneCandidates[k];
            }
        }
        res->done = 1;
    }
    for (int k = 0; k <= kTuneN; ++k)
        if (ev[k]) cudaEventDestroy(ev[k]);
    if (dealt) cudaFree(dealt);   // the slices are done: waited for above, or by this call
    if (dsum) cudaFree(dsum);
    return e;
}

// the tuned shape of (device, octree, kernel mode), or false
bool tuned_shape(int dev, const DevTree& T, int mode, int* tpb, int* depth, double* rates)
{
    std::lock_guard<std::mutex> lock(g_tune_mu);
    auto it = g_tune.find(std::make_tuple(dev, (const void*)T.keys, mode));
    if (it == g_tune.end() || !it->second.done) return false;
    *tpb = it->second.best.tpb;
    *depth = it->second.best.depth;
    if (rates)
        for (int k = 0; k < kTuneN; ++k) rates[k] = it->second.rate[k];
    return true;
}

// drops the tuned shapes and ray orders of an octree whose device arrays are
// freed (a later octree may reuse the addresses)
void forget_tuned_shape(const void* keys)
{
    free_orders(keys);
    std::lock_guard<std::mutex> lock(g_tune_mu);
    for (auto it = g_tune.begin(); it != g_tune.end();) {
        if (std::get<1>(it->first) == keys) it = g_tune.erase(it);
        else ++it;
    }
}

// the kernel mode of the plain (surface-record) instantiation for `order`
// (8 / 9 on a velocity-field octree)
int plain_fast_mode(int order, bool velocity) { return velocity ? ((order == 1) ? 8 : 9) : ((order == 1) ? 6 : 7); }

template <>
cudaError_t launch_propagate<false>(const DevTree& T, const DevCosmo& C, const PropParams& P, const double* d_launch, long long n,
                                    const PropOut& O, cudaStream_t stream)
{
    if (n <= 0) return cudaSuccess;
    // NGP (ORDER = 0) has no interpolation arithmetic to lighten: the float64 kernel
    if (P.order == 0 || !fast_mode_supported(T, P, O)) return launch_propagate<true>(T, C, P, d_launch, n, O, stream);
    FastLaunchState st;
    cudaError_t e = fast_launch_state(stream, &st);
    if (e != cudaSuccess) return e;
    unsigned long long* const queue = st.queue;
    e = cudaMemsetAsync(queue, 0, sizeof(unsigned long long), stream);
    if (e != cudaSuccess) return e;
    FastShape shape = fast_launch_shape(n, st.blocks_per_sm, st.sms, P.jacobian != 0);
    const int* perm = nullptr;
    OrderClaim claim;
    if (fast_mode(T, P, O) >= 6 && (e = order_rays(T, d_launch, n, st.sms, stream, claim, &perm)) != cudaSuccess) return e;
    int depth = 1;
#if MPF_DIAG
    // MPF_STATS=1: print the counts of the rare paths (diagnostics; serialises the call)
    static const bool want_stats = getenv("MPF_STATS") != nullptr;
#endif
    static const bool want_tune = !(getenv("MPF_AUTOTUNE") && getenv("MPF_AUTOTUNE")[0] == '0');
    if (shape.full && want_tune) {
        // a batch that fills the GPU: the tuned shape of this octree and kernel mode
        int dev = 0;
        if ((e = cudaGetDevice(&dev)) != cudaSuccess) return e;
        const auto key = std::make_tuple(dev, (const void*)T.keys, fast_mode(T, P, O));
        TuneResult res;
        bool have = false;
        {
            std::lock_guard<std::mutex> lock(g_tune_mu);
            auto it = g_tune.find(key);
            if (it != g_tune.end() && it->second.done) {
                res = it->second;
                have = true;
            }
        }
        if (!have && n >= kTuneMinRays) {
            e = tune_and_launch(T, C, P, d_launch, n, O, queue, perm, st.sms, stream, &res);
            if (e == cudaSuccess) {
                std::lock_guard<std::mutex> lock(g_tune_mu);
                g_tune[key] = res;
            }
            return e;
        }
        if (have) {
            shape.tpb = res.best.tpb;
            depth = res.best.depth;
            shape.grid = shape_grid(res.best, n, st.sms);
        }
    }
    launch_fast_kernel(shape.grid, shape.tpb, shape.rays, shape.per_ray, depth, 0, T, C, P, d_launch, n, O, queue, perm, stream);
    e = cudaGetLastError();
#if MPF_DIAG
    if (want_stats) {
        unsigned long long dg[4] = {0, 0, 0, 0};
        cudaStreamSynchronize(stream);
        cudaMemcpyFromSymbol(dg, g_diag, sizeof(dg));
        fprintf(stderr, "mpf_diag restarts %llu full_walks %llu\n", dg[0], dg[1]);
    }
#endif
    return e;
}
cudaError_t launch_gather_fast(const DevTree& T, int kind, const double* d_xyz, long long n, void* d_out, cudaStream_t stream)
{
    if (n <= 0) return cudaSuccess;
    if (kind == 3) return launch_gather_exact(T, kind, d_xyz, n, d_out, stream);   // NGP: a copy of the cell's record
    k_gather_rec<<<(unsigned)((n + 127) / 128), 128, 0, stream>>>(T, kind, d_xyz, n, d_out);
    return cudaGetLastError();
}
}  // namespace mpf

namespace mpf {
// Same launch as launch_propagate<false>, with the work-queue counter supplied
// by the caller (no allocation here).  The counter must be zero on entry.
cudaError_t launch_propagate_fast_with_queue(const DevTree& T, const DevCosmo& C, const PropParams& P, const double* d_launch,
                                             long long n, const PropOut& O, unsigned long long* queue, cudaStream_t stream)
{
    if (n <= 0) return cudaSuccess;
    const int tpb = kFastThreads;
    int blocks_per_sm = 0, sms = 0, dev = 0;
    cudaError_t e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&blocks_per_sm, k_propagate_fast<2, false, false>, tpb, (size_t)tpb * kSlotBytes);
    if (e == cudaSuccess) e = cudaGetDevice(&dev);
    if (e == cudaSuccess) e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    if (e != cudaSuccess) return e;
    if (blocks_per_sm < 1) blocks_per_sm = 1;
    const FastShape shape = fast_launch_shape(n, blocks_per_sm, sms, P.jacobian != 0);
    launch_fast_kernel(shape.grid, shape.tpb, shape.rays, shape.per_ray, 1, 0, T, C, P, d_launch, n, O, queue, nullptr, stream);
    return cudaGetLastError();
}
}  // namespace mpf
