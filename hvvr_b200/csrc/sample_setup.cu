// sample_setup.cu - the sample hierarchy built on the device: SampleData::SampleData
// (libraries/hvvr/raycaster/camera.cpp:21-64) for the perspective mapping, with naiveXYCluster
// (sample_clustering.h:17-49), BeamBatch2D (sample_hierarchy.cpp:154-190), get3DFrustumFrom2D
// (sample_hierarchy.cpp:46-123), the beams of BeamBatch::generateFrom2D (sample_hierarchy.cpp:
// 129-152) and imageLocationToSampleIndex.
//
// naiveXYCluster is four rounds of std::sort with lexicographic comparators on the sample
// position. When no two samples share a position, every round has one sorted order whatever the
// algorithm, so stable device radix sorts of (y, x) and (x, y) keys reproduce the reference's
// order exactly; the builder reports duplicate or NaN positions to the caller, which then builds
// on the host (where std::sort decides the order among equal positions). The rectangle and
// frustum arithmetic keeps the host builder's operation order (every .cu file is compiled without
// FMA contraction and with IEEE division and square root, under FTZ like the host's MXCSR).
#include "dev_common.cuh"
#include "host_objects.h"
#include "sample_setup.h"

#include <cub/device/device_radix_sort.cuh>
#include <cub/block/block_radix_sort.cuh>

#include <math.h>

#include <vector>

namespace hvb {
namespace {

enum : uint32_t { kFlagNaN = 1, kFlagDuplicate = 2 };

// float -> uint32 with the float order (-0 and +0 equal, as the comparators treat them)
__device__ __forceinline__ uint32_t orderKey(float f) {
    uint32_t u = __float_as_uint(f);
    if (u == 0x80000000u) u = 0;
    return (u & 0x80000000u) ? ~u : (u | 0x80000000u);
}

// the samples' order keys along x and y, and what the first sort takes
__global__ void keysKernel(const hvvr_sample* __restrict__ samples, uint32_t count, uint32_t* __restrict__ kx,
                           uint32_t* __restrict__ ky, unsigned long long* __restrict__ keys, uint32_t* __restrict__ perm,
                           uint32_t* __restrict__ flags) {
    const uint32_t p = blockIdx.x * blockDim.x + threadIdx.x;
    if (p >= count) return;
    const float x = samples[p].position.x, y = samples[p].position.y;
    if (isnan(x) || isnan(y)) atomicOr(flags, kFlagNaN);
    const uint32_t ox = orderKey(x), oy = orderKey(y);
    kx[p] = ox;
    ky[p] = oy;
    keys[p] = (uint64_t(oy) << 32) | ox;
    perm[p] = p;
}

// a round over runs of `run` positions as one sort: the run in the upper half of the key
__global__ void runKeysKernel(const uint32_t* __restrict__ axis, const uint32_t* __restrict__ perm, uint32_t count, uint32_t run,
                              unsigned long long* __restrict__ keys) {
    const uint32_t p = blockIdx.x * blockDim.x + threadIdx.x;
    if (p < count) keys[p] = (uint64_t(p / run) << 32) | axis[perm[p]];
}

// a round over runs of THREADS * ITEMS positions, one CTA each (stable; positions past the end sort last)
template <int THREADS, int ITEMS>
__global__ void __launch_bounds__(THREADS) runSortKernel(const uint32_t* __restrict__ axis, const uint32_t* __restrict__ in,
                                                         uint32_t* __restrict__ out, uint32_t count) {
    using Sort = cub::BlockRadixSort<uint32_t, THREADS, ITEMS, uint32_t>;
    __shared__ typename Sort::TempStorage temp;
    const uint32_t first = blockIdx.x * (THREADS * ITEMS) + threadIdx.x * ITEMS;
    uint32_t key[ITEMS], val[ITEMS];
#pragma unroll
    for (int k = 0; k < ITEMS; k++) {
        val[k] = first + k < count ? in[first + k] : 0u;
        key[k] = first + k < count ? axis[val[k]] : ~0u;
    }
    Sort(temp).SortBlockedToStriped(key, val);
#pragma unroll
    for (int k = 0; k < ITEMS; k++) {
        const uint32_t p = blockIdx.x * (THREADS * ITEMS) + k * THREADS + threadIdx.x;
        if (p < count) out[p] = val[k];
    }
}

// equal neighbours in the (y, x)-sorted order: two samples at one position
__global__ void duplicateKernel(const unsigned long long* __restrict__ keys, uint32_t count, uint32_t* __restrict__ flags) {
    const uint32_t p = blockIdx.x * blockDim.x + threadIdx.x;
    if (p == 0 || p >= count) return;
    if (keys[p] == keys[p - 1]) atomicOr(flags, kFlagDuplicate);
}

struct M3 {
    F3 c0, c1, c2;
};
__device__ __forceinline__ F3 mul(const M3& m, F3 v) {
    return f3(m.c0.x * v.x + m.c1.x * v.y + m.c2.x * v.z, m.c0.y * v.x + m.c1.y * v.y + m.c2.y * v.z,
              m.c0.z * v.x + m.c1.z * v.y + m.c2.z * v.z);
}
__device__ __forceinline__ float fmin2(float a, float b) { return a < b ? a : b; }
__device__ __forceinline__ float fmax2(float a, float b) { return a > b ? a : b; }

// get3DFrustumFrom2D (perspective branch). f = {xMin, -xMax, yMin, -yMax}.
__device__ Rays4 frustumFrom2D(const float f[4], const M3& S, float lensRadius, float focalDistance) {
    const float farPlane = -100.0f;
    const float xMin = f[0], xMax = -f[1], yMin = f[2], yMax = -f[3];
    const F3 nearP[4] = {f3(-lensRadius, -lensRadius, 0), f3(+lensRadius, -lensRadius, 0),
                         f3(+lensRadius, +lensRadius, 0), f3(-lensRadius, +lensRadius, 0)};
    const F3 rd[4] = {mul(S, f3(xMin, yMax, 1)), mul(S, f3(xMax, yMax, 1)), mul(S, f3(xMax, yMin, 1)),
                      mul(S, f3(xMin, yMin, 1))};
    F3 focus[4];
    for (int i = 0; i < 4; i++) focus[i] = rd[i] * (focalDistance / -rd[i].z);
    float fxMax = -INFINITY, fxMin = INFINITY, fyMax = -INFINITY, fyMin = INFINITY;
    for (int i = 0; i < 4; ++i) {
        for (int j = 0; j < 4; ++j) {
            const F3 pos = nearP[i];
            const F3 dir = normalize3(focus[j] - pos);
            const F3 p = pos + dir * (farPlane / dir.z);
            fxMax = fmax2(fxMax, p.x);
            fxMin = fmin2(fxMin, p.x);
            fyMax = fmax2(fyMax, p.y);
            fyMin = fmin2(fyMin, p.y);
        }
    }
    const F3 farP[4] = {f3(fxMin, fyMin, farPlane), f3(fxMax, fyMin, farPlane), f3(fxMax, fyMax, farPlane),
                        f3(fxMin, fyMax, farPlane)};
    Rays4 r;
    for (int i = 0; i < 4; i++) {
        const F3 d = normalize3(farP[i] - nearP[i]);
        r.o[i][0] = nearP[i].x;
        r.o[i][1] = nearP[i].y;
        r.o[i][2] = nearP[i].z;
        r.d[i][0] = d.x;
        r.d[i][1] = d.y;
        r.d[i][2] = d.z;
    }
    return r;
}

// BeamBatch2D per tile: the rectangle of its 128 samples padded by the major axis, in sample
// order (positions past the last sample repeat it), then the tile's frustum. One warp per tile: a lane
// folds four samples in order and the lanes are folded in order too, which is the sequential fold (the
// later of two equal values stays) unless a value is NaN: then lane 0 folds all 128.
__global__ void tileKernel(const hvvr_sample* __restrict__ samples, const uint32_t* __restrict__ perm, uint32_t count,
                           uint32_t tiles, M3 S, float lensRadius, float focalDistance, float4* __restrict__ rects,
                           Rays4* __restrict__ tileRays) {
    const uint32_t t = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31u;
    if (t >= tiles) return;
    float tf[4];
    auto fold = [&](uint32_t k0, uint32_t n) {
        bool nan = false;
        for (int j = 0; j < 4; j++) tf[j] = INFINITY;
        for (uint32_t k = k0; k < k0 + n; k++) {
            const uint32_t p = min(t * kTileSize + k, count - 1);
            const hvvr_sample& s = samples[perm[p]];
            const float x = s.position.x, y = s.position.y, mj = s.major_axis_length;
            const float xs[2] = {x + mj, x - mj}, ys[2] = {y + mj, y - mj};
            for (int q = 0; q < 2; q++) {
                tf[0] = fmin2(tf[0], xs[q]);
                tf[1] = fmin2(tf[1], -xs[q]);
                tf[2] = fmin2(tf[2], ys[q]);
                tf[3] = fmin2(tf[3], -ys[q]);
                nan = nan || isnan(xs[q]) || isnan(ys[q]);
            }
        }
        return nan;
    };
    if (__any_sync(0xffffffffu, fold(lane * 4, 4))) {
        if (lane == 0) fold(0, kTileSize);
    } else {
#pragma unroll
        for (uint32_t o = 1; o < 32; o <<= 1)
            for (int j = 0; j < 4; j++) {
                const float later = __shfl_down_sync(0xffffffffu, tf[j], o);
                if ((lane & (2 * o - 1)) == 0) tf[j] = fmin2(tf[j], later);
            }
    }
    if (lane) return;
    for (int j = 0; j < 4; j++) tf[j] = fmax2(tf[j], -INFINITY);
    rects[t] = make_float4(tf[0], tf[1], tf[2], tf[3]);
    tileRays[t] = frustumFrom2D(tf, S, lensRadius, focalDistance);
}

// a block's rectangle is the union of its tiles' in tile order
__global__ void blockKernel(const float4* __restrict__ rects, uint32_t blocks, M3 S, float lensRadius,
                            float focalDistance, Rays4* __restrict__ blockRays) {
    const uint32_t b = blockIdx.x * blockDim.x + threadIdx.x;
    if (b >= blocks) return;
    float bf[4] = {INFINITY, INFINITY, INFINITY, INFINITY};
    for (uint32_t t = 0; t < kTilesPerBlock; t++) {
        const float4 r = rects[b * kTilesPerBlock + t];
        bf[0] = fmin2(bf[0], r.x);
        bf[1] = fmin2(bf[1], r.y);
        bf[2] = fmin2(bf[2], r.z);
        bf[3] = fmin2(bf[3], r.w);
    }
    blockRays[b] = frustumFrom2D(bf, S, lensRadius, focalDistance);
}

// unpackSample (libraries/hvvr/raycaster/samples.cpp:144-159) and the camera-space beam
// {S (c, 1), S (major, 0), S (minor, 0)}; padding positions are zero samples
__global__ void beamsKernel(const hvvr_sample* __restrict__ samples, const uint32_t* __restrict__ perm, uint32_t count,
                            uint32_t padded, M3 S, float4* __restrict__ beams) {
    const uint32_t p = blockIdx.x * blockDim.x + threadIdx.x;
    if (p >= padded) return;
    float cx = 0.0f, cy = 0.0f, mjx = 0.0f, mjy = 0.0f, mnx = 0.0f, mny = 0.0f;
    if (p < count) {
        const hvvr_sample& s = samples[perm[p]];
        const float ext = 0.70710678118f;
        mnx = s.minor_axis.x * ext;
        mny = s.minor_axis.y * ext;
        const float mlen = sqrtf(s.minor_axis.x * s.minor_axis.x + s.minor_axis.y * s.minor_axis.y);
        const float rescale = s.major_axis_length * ext / mlen;
        cx = s.position.x;
        cy = s.position.y;
        mjx = -mny * rescale;
        mjy = mnx * rescale;
    }
    const F3 c = mul(S, f3(cx, cy, 1.0f));
    const F3 du = mul(S, f3(mjx, mjy, 0.0f));
    const F3 dv = mul(S, f3(mnx, mny, 0.0f));
    beams[3 * size_t(p) + 0] = make_float4(c.x, c.y, c.z, du.x);
    beams[3 * size_t(p) + 1] = make_float4(du.y, du.z, dv.x, dv.y);
    beams[3 * size_t(p) + 2] = make_float4(dv.z, 0.0f, 0.0f, 0.0f);
}

// imageLocationToSampleIndex: the last sample (in cluster order) at a pixel location wins
__global__ void remapKernel(const hvvr_sample* __restrict__ samples, const uint32_t* __restrict__ perm, uint32_t count,
                            uint32_t split, uint32_t width, uint32_t height, int32_t* __restrict__ remap) {
    const uint32_t p = blockIdx.x * blockDim.x + threadIdx.x;
    if (p >= count) return;
    const uint32_t i = perm[p];
    const hvvr_sample& s = samples[i];
    if (s.pixel_x < width && s.pixel_y < height) {
        const size_t idx = (size_t(s.pixel_y) * width + s.pixel_x) * split + i % split;
        atomicMax(remap + idx, int32_t(p));
    }
}

inline uint32_t grid(size_t n, uint32_t block) { return uint32_t((n + block - 1) / block); }

} // namespace

int buildSampleSetupDevice(const hvvr_sample* samples, uint32_t count, uint32_t split, const hvvr_float_rect& vp,
                           const hvvr_thin_lens& lens, uint32_t width, uint32_t height, SetupScratch& scratch,
                           DeviceSampleSetup& out, cudaStream_t st, bool& needsHost) {
    needsHost = false;
    if (count == 0) return fail(HVVR_ERR_STATE, "camera has no samples");
    const uint32_t blocks = (count + kBlockSize - 1) / kBlockSize;
    const uint32_t tiles = blocks * kTilesPerBlock, padded = blocks * kBlockSize;
    // strata of naiveXYCluster, as the host computes them
    const size_t k = blocks;
    const size_t yStrata = (size_t)sqrt((double)k);
    const size_t xStrata = (k + yStrata - 1) / yStrata;
    const size_t blockYStrata = (size_t)sqrt((double)kTilesPerBlock);
    const size_t blockXStrata = (kTilesPerBlock + blockYStrata - 1) / blockYStrata;

    // The scratch of one build, carved from the raycaster's: a new sample set every frame (a gaze that
    // moves) would otherwise allocate and free fourteen buffers each time, each free a device-wide wait
    // (3.3 ms of 6.7 for 300,007 samples).
    std::lock_guard<std::mutex> lock(scratch.mutex);
    size_t sortBytes = 0;
    CUDA_TRY(cub::DeviceRadixSort::SortPairs(nullptr, sortBytes, (unsigned long long*)nullptr, (unsigned long long*)nullptr,
                                             (uint32_t*)nullptr, (uint32_t*)nullptr, int(count), 0, 64, st));
    size_t bytes = 0;
    auto carve = [&](size_t n) {
        const size_t at = bytes;
        bytes += (n + 255) / 256 * 256;
        return at;
    };
    const size_t atSamples = carve(size_t(count) * sizeof(hvvr_sample)), atKeys0 = carve(size_t(count) * 8),
                 atKeys1 = carve(size_t(count) * 8), atPerm0 = carve(size_t(count) * 4), atPerm1 = carve(size_t(count) * 4),
                 atX = carve(size_t(count) * 4), atY = carve(size_t(count) * 4), atRects = carve(size_t(tiles) * sizeof(float4)),
                 atFlags = carve(4), atSort = carve(sortBytes);
    TRY(scratch.buf.ensure(bytes));
    struct Release { // (a large one is given back)
        DevBuf<uint8_t>& b;
        ~Release() {
            if (b.n > kSetupScratchKept) b.release();
        }
    } release{scratch.buf};
    uint8_t* base = scratch.buf.p;
    hvvr_sample* dSamples = reinterpret_cast<hvvr_sample*>(base + atSamples);
    unsigned long long* keys[2] = {reinterpret_cast<unsigned long long*>(base + atKeys0), reinterpret_cast<unsigned long long*>(base + atKeys1)};
    uint32_t* perm[2] = {reinterpret_cast<uint32_t*>(base + atPerm0), reinterpret_cast<uint32_t*>(base + atPerm1)};
    uint32_t *kx = reinterpret_cast<uint32_t*>(base + atX), *ky = reinterpret_cast<uint32_t*>(base + atY),
             *flags = reinterpret_cast<uint32_t*>(base + atFlags);
    float4* rects = reinterpret_cast<float4*>(base + atRects);
    CUDA_TRY(cudaMemcpyAsync(dSamples, samples, size_t(count) * sizeof(hvvr_sample), cudaMemcpyHostToDevice, st));
    CUDA_TRY(cudaMemsetAsync(flags, 0, 4, st));
    // sort 1 of naiveXYCluster: the whole set by (y, x)
    keysKernel<<<grid(count, 256), 256, 0, st>>>(dSamples, count, kx, ky, keys[0], perm[0], flags);
    CUDA_TRY(cub::DeviceRadixSort::SortPairs(base + atSort, sortBytes, keys[0], keys[1], perm[0], perm[1], int(count), 0, 64, st));
    duplicateKernel<<<grid(count, 256), 256, 0, st>>>(keys[1], count, flags);
    // Sorts 2-4 order fixed-size runs of the current order. Each alternates the axes, so within a run the
    // current order already has the minor axis ascending, and a stable sort by the major axis alone is the
    // whole sort: rows of blocks by (x, y) as one radix sort with the run above the key, blocks of 8192 by
    // (y, x) and runs of eight tiles by (x, y) by a CTA each. 300,007 samples: 1,045 us as segmented sorts
    // of 64-bit keys, 120 us so (the whole build and frame 6.7 and 2.9 ms).
    static_assert(kBlockSize == 1024 * 8 && kTileSize * 8 == 256 * 4, "runs of the CTA sorts");
    const size_t rowRun = kBlockSize * xStrata, rows = (count + rowRun - 1) / rowRun;
    int rowBits = 0;
    while ((size_t(1) << rowBits) < rows) rowBits++;
    runKeysKernel<<<grid(count, 256), 256, 0, st>>>(kx, perm[1], count, uint32_t(rowRun), keys[0]);
    CUDA_TRY(cub::DeviceRadixSort::SortPairs(base + atSort, sortBytes, keys[0], keys[1], perm[1], perm[0], int(count), 0,
                                             32 + rowBits, st));
    runSortKernel<1024, 8><<<grid(count, kBlockSize), 1024, 0, st>>>(ky, perm[0], perm[1], count);
    if (blockXStrata != 8) return fail(HVVR_ERR_STATE, "tile runs of %zu", blockXStrata);
    runSortKernel<256, 4><<<grid(count, 1024), 256, 0, st>>>(kx, perm[1], perm[0], count);
    const uint32_t* order = perm[0];

    // Camera::getSampleToCamera (libraries/hvvr/raycaster/camera.cpp:167-171)
    const M3 S{F3{vp.upper.x - vp.lower.x, 0, 0}, F3{0, vp.lower.y - vp.upper.y, 0}, F3{vp.lower.x, vp.upper.y, -1}};
    TRY(out.tileRays->alloc(tiles));
    TRY(out.blockRays->alloc(blocks));
    TRY(out.beams->alloc(size_t(padded) * 3));
    TRY(out.remap->alloc(size_t(width) * height * split));
    tileKernel<<<grid(size_t(tiles) * 32, 128), 128, 0, st>>>(dSamples, order, count, tiles, S, lens.radius, lens.focal_distance,
                                                              rects, out.tileRays->p);
    blockKernel<<<grid(blocks, 64), 64, 0, st>>>(rects, blocks, S, lens.radius, lens.focal_distance,
                                                 out.blockRays->p);
    beamsKernel<<<grid(padded, 256), 256, 0, st>>>(dSamples, order, count, padded, S, out.beams->p);
    if (out.remap->n) {
        CUDA_TRY(cudaMemsetAsync(out.remap->p, 0xff, out.remap->n * sizeof(int32_t), st));
        remapKernel<<<grid(count, 256), 256, 0, st>>>(dSamples, order, count, split, width, height, out.remap->p);
    }
    CUDA_TRY(cudaGetLastError());
    // equal or NaN positions: what was written is an order of no meaning, and the caller builds on the host
    uint32_t flag = 0;
    CUDA_TRY(cudaMemcpyAsync(&flag, flags, 4, cudaMemcpyDeviceToHost, st));
    CUDA_TRY(cudaStreamSynchronize(st));
    if (flag) {
        needsHost = true;
        return HVVR_OK;
    }
    out.blocks = blocks;
    out.tiles = tiles;
    out.padded = padded;
    out.valid = count;
    return HVVR_OK;
}

} // namespace hvb
