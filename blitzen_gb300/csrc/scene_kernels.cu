// scene_kernels.cu — scene-side kernels around the cull: transform scatter (UpdateObjectTransform),
// dynamic-object rotation, and the occluder-box depth rasteriser that produces the per-view depth
// buffers the pyramid is built from.
#include "blz_device.cuh"
#include "kernels.h"

namespace blz {

// transforms[ids[i]] = in[i]: the device half of UpdateObjectTransform + UpdateBuffers
// (src/Renderer/BlitzenVulkan/vulkanDraw.cpp:46-60,816-820).
__global__ void transforms_scatter_kernel(BlzMeshTransform* table, uint32_t tableCount, const uint32_t* ids,
                                          const BlzMeshTransform* in, uint32_t n, unsigned int* status) {
    pdl_wait();
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const uint32_t id = ids[i];
    if (id >= tableCount) {
        atomicOr(status, BLZ_FLAG_BAD_INDEX);
        return;
    }
    const float4* src = reinterpret_cast<const float4*>(in + i);
    float4* dst = reinterpret_cast<float4*>(table + id);
    dst[0] = src[0];
    dst[1] = src[1];
}

// dst[i] = table[ids[i]] with orientation r (x) q, r = (s * axis_i, c); the rotation of
// src/Game/blitzenObject.cpp:30-46 applied incrementally on the device. s, c = sin/cos(angle/2)
// are computed once on the host.
__global__ void transforms_rotate_kernel(const BlzMeshTransform* table, uint32_t tableCount, const BlzMeshTransform* dynRows,
                                         uint32_t dynCount, const uint32_t* ids, const float* axes, float s, float c,
                                         uint32_t n, BlzMeshTransform* dst, unsigned int* status) {
    pdl_wait();
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const uint32_t id = ids[i];
    if (id >= tableCount) {
        atomicOr(status, BLZ_FLAG_BAD_INDEX);
        return;
    }
    const float4* src = reinterpret_cast<const float4*>((id < dynCount ? dynRows : table) + id);
    const float4 ps = src[0], q = src[1];
    const float rx = BLZ_FM(s, axes[3 * i + 0]), ry = BLZ_FM(s, axes[3 * i + 1]), rz = BLZ_FM(s, axes[3 * i + 2]);
    const float rw = c;
    float4 o;
    o.x = BLZ_FS(BLZ_FA(BLZ_FA(BLZ_FM(rw, q.x), BLZ_FM(rx, q.w)), BLZ_FM(ry, q.z)), BLZ_FM(rz, q.y));
    o.y = BLZ_FA(BLZ_FA(BLZ_FS(BLZ_FM(rw, q.y), BLZ_FM(rx, q.z)), BLZ_FM(ry, q.w)), BLZ_FM(rz, q.x));
    o.z = BLZ_FA(BLZ_FS(BLZ_FA(BLZ_FM(rw, q.z), BLZ_FM(rx, q.y)), BLZ_FM(ry, q.x)), BLZ_FM(rz, q.w));
    o.w = BLZ_FS(BLZ_FS(BLZ_FS(BLZ_FM(rw, q.w), BLZ_FM(rx, q.x)), BLZ_FM(ry, q.y)), BLZ_FM(rz, q.z));
    float4* d = reinterpret_cast<float4*>(dst + i);
    d[0] = ps;
    d[1] = o;
}

cudaError_t launch_transforms_scatter(BlzMeshTransform* table, uint32_t tableCount, const uint32_t* ids,
                                      const BlzMeshTransform* in, uint32_t n, unsigned int* status, cudaStream_t s) {
    if (n == 0) return cudaSuccess;
    return launch_pdl(transforms_scatter_kernel, (n + 255) / 256, 256, 0, s, table, tableCount, ids, in, n, status);
}

cudaError_t launch_transforms_rotate(const BlzMeshTransform* table, uint32_t tableCount, const BlzMeshTransform* dynRows,
                                     uint32_t dynCount, const uint32_t* ids, const float* axes, float angle, uint32_t n,
                                     BlzMeshTransform* dst, unsigned int* status, cudaStream_t s) {
    if (n == 0) return cudaSuccess;
    const float h = angle * 0.5f;
    const float sn = sinf(h), cs = cosf(h);  // host libm, the same values the host oracle uses
    return launch_pdl(transforms_rotate_kernel, (n + 255) / 256, 256, 0, s, table, tableCount, dynRows, dynCount, ids, axes, sn,
                      cs, n, dst, status);
}

cudaError_t load_transform_kernels() {
    cudaFuncAttributes a;
    return cudaFuncGetAttributes(&a, reinterpret_cast<const void*>(transforms_rotate_kernel));
}

// ------------------------------------------------------------------ occluder raster

struct BoxRect {
    int x0, y0, x1, y1;
    float depth;
};

// Screen position of a box corner (view space).
__device__ __forceinline__ void box_corner(const ViewConsts& v, Vec3 q, uint32_t width, uint32_t height, float& sx, float& sy) {
    sx = BLZ_FM(BLZ_FA(BLZ_FM(BLZ_FD(BLZ_FM(q.x, v.proj0), q.z), 0.5f), 0.5f), static_cast<float>(width));
    sy = BLZ_FM(BLZ_FS(0.5f, BLZ_FM(BLZ_FD(BLZ_FM(q.y, v.proj5), q.z), 0.5f)), static_cast<float>(height));
}

// The pixel rectangle of the corners' extent, clipped to the screen, and its depth.
__device__ __forceinline__ BoxRect box_extent(const ViewConsts& v, float minx, float miny, float maxx, float maxy, float zmax,
                                              uint32_t width, uint32_t height) {
    BoxRect r;
    r.depth = BLZ_FD(v.zNear, zmax);
    const float fw = static_cast<float>(width), fh = static_cast<float>(height);
    const float fx0 = floorf(minx), fy0 = floorf(miny), fx1 = ceilf(maxx), fy1 = ceilf(maxy);
    r.x0 = fx0 < 0.0f ? 0 : (fx0 > fw ? static_cast<int>(width) : static_cast<int>(fx0));
    r.y0 = fy0 < 0.0f ? 0 : (fy0 > fh ? static_cast<int>(height) : static_cast<int>(fy0));
    r.x1 = fx1 < 0.0f ? 0 : (fx1 > fw ? static_cast<int>(width) : static_cast<int>(fx1));
    r.y1 = fy1 < 0.0f ? 0 : (fy1 > fh ? static_cast<int>(height) : static_cast<int>(fy1));
    return r;
}

__device__ __forceinline__ BoxRect box_rect(const ViewConsts& v, const float* bx, uint32_t width, uint32_t height) {
    float minx = INFINITY, maxx = -INFINITY, miny = INFINITY, maxy = -INFINITY, zmax = -INFINITY;
    for (int k = 0; k < 8; ++k) {
        const Vec3 p{bx[(k & 1) ? 3 : 0], bx[(k & 2) ? 4 : 1], bx[(k & 4) ? 5 : 2]};
        const Vec3 q = view_transform(v.rows, p);
        if (!(q.z > v.zNear)) return BoxRect{0, 0, 0, 0, 0.0f};  // boxes reaching the near plane are skipped
        float sx, sy;
        box_corner(v, q, width, height, sx, sy);
        minx = fmin_nan(minx, sx);
        maxx = fmax_nan(maxx, sx);
        miny = fmin_nan(miny, sy);
        maxy = fmax_nan(maxy, sy);
        zmax = fmax_nan(zmax, q.z);
    }
    return box_extent(v, minx, miny, maxx, maxy, zmax, width, height);
}

__global__ void depth_clear_kernel(float4* depth, size_t n4, float* tail, uint32_t ntail) {
    pdl_wait();
    for (size_t i = blockIdx.x * static_cast<size_t>(blockDim.x) + threadIdx.x; i < n4; i += static_cast<size_t>(gridDim.x) * blockDim.x)
        depth[i] = make_float4(0.f, 0.f, 0.f, 0.f);
    if (blockIdx.x == 0 && threadIdx.x < ntail) tail[threadIdx.x] = 0.0f;
}

// One block per box: the block walks the box's screen rectangle and max-writes its depth.
// Depths are positive, so the float maximum is the integer maximum of the bit patterns, which
// makes the result independent of the order boxes land in.
__global__ void depth_raster_kernel(const BlzCameraViewData view, const float* boxes, uint32_t boxCount, float* depth,
                                    uint32_t width, uint32_t height) {
    __shared__ BoxRect s_r;
    pdl_wait();
    const ViewConsts v = load_view(view);
    for (uint32_t b = blockIdx.x; b < boxCount; b += gridDim.x) {
        if (threadIdx.x == 0) s_r = box_rect(v, boxes + 6 * static_cast<size_t>(b), width, height);
        __syncthreads();
        const BoxRect r = s_r;
        if (r.x1 > r.x0 && r.y1 > r.y0 && r.depth > 0.0f) {
            const int w = r.x1 - r.x0;
            const int n = w * (r.y1 - r.y0);
            const int bits = __float_as_int(r.depth);
            for (int idx = threadIdx.x; idx < n; idx += blockDim.x) {
                const int x = r.x0 + idx % w, y = r.y0 + idx / w;
                atomicMax(reinterpret_cast<int*>(depth) + static_cast<size_t>(y) * width + x, bits);
            }
        }
        __syncthreads();
    }
}

// The screen tiles of the other form: one block per kTileW x kTileH pixels, a warp per 32x16 of them, 16
// pixels a thread (four neighbours in each of four rows). The block keeps the boxes whose rectangle meets its tile (every box
// tested once per tile, up to kTileHits at a time), takes the largest depth over each pixel in registers and
// writes the pixel once, the cleared ones included: the image is written once and never read, where the
// block per box clears it and then sends one atomic a covered pixel.
// 2000 boxes of the stress scene's sizes at 3840x2160: 13 us a raster (2.8 rectangles, 12.0 tiles, in a
// stream) against 32; 8192 boxes of 1 to 4 units, the tile form's worst: 15 against 37, and 177 against 195 at
// 16384x16384, where most of either is the writing of the image.
constexpr uint32_t kTileW = 64, kTileH = 64;  // (128 x 64: 16.1 us a tile launch against 12.0: a warp meets more boxes it has no pixel of)
constexpr uint32_t kTileThreads = kTileW / 4u * kTileH / 4u;
constexpr uint32_t kTileHits = 1024;
constexpr uint32_t kTileScan = 4;  // rectangles a thread loads at a time
constexpr uint32_t kTilePart = kTileHits / kTileThreads;  // of which this many join the list before it is used
constexpr uint32_t kRasterTileExtent = 1u << 16;  // a side whose tiles fit a launch grid
static_assert(kTileHits % kTileThreads == 0 && kTileScan % kTilePart == 0, "whole parts");

// box_rect by eight lanes, one per corner (the same corners compared in the same order).
__global__ void __launch_bounds__(128) box_rects_kernel(const BlzCameraViewData view, const float* boxes, uint32_t boxCount,
                                                        uint32_t width, uint32_t height, int4* rects, int* depths) {
    pdl_wait();
    const uint32_t at = blockIdx.x * 16u + threadIdx.x / 8u, k = threadIdx.x % 8u;
    const uint32_t b = min(at, boxCount - 1u);
    const ViewConsts v = load_view(view);
    const float* bx = boxes + 6 * static_cast<size_t>(b);
    const Vec3 q = view_transform(v.rows, Vec3{bx[(k & 1u) ? 3 : 0], bx[(k & 2u) ? 4 : 1], bx[(k & 4u) ? 5 : 2]});
    float minx, miny, maxx, maxy, zmax = q.z;
    box_corner(v, q, width, height, minx, miny);
    maxx = minx;
    maxy = miny;
    const unsigned front = __ballot_sync(0xFFFFFFFFu, q.z > v.zNear);
#pragma unroll
    for (int d = 1; d < 8; d <<= 1) {  // the lower corner's value first, as in box_rect
        const bool low = (k & static_cast<uint32_t>(d)) == 0u;
        auto pair = [&](float x, auto op) {
            const float o = __shfl_xor_sync(0xFFFFFFFFu, x, d);
            return low ? op(x, o) : op(o, x);
        };
        minx = pair(minx, [](float l, float h) { return fmin_nan(l, h); });
        maxx = pair(maxx, [](float l, float h) { return fmax_nan(l, h); });
        miny = pair(miny, [](float l, float h) { return fmin_nan(l, h); });
        maxy = pair(maxy, [](float l, float h) { return fmax_nan(l, h); });
        zmax = pair(zmax, [](float l, float h) { return fmax_nan(l, h); });
    }
    if (k != 0u || at >= boxCount) return;
    const uint32_t lane = threadIdx.x & 31u;
    BoxRect r{0, 0, 0, 0, 0.0f};
    if (((front >> lane) & 0xFFu) == 0xFFu)  // boxes reaching the near plane are skipped
        r = box_extent(v, fmin_nan(INFINITY, minx), fmin_nan(INFINITY, miny), fmax_nan(-INFINITY, maxx), fmax_nan(-INFINITY, maxy),
                       fmax_nan(-INFINITY, zmax), width, height);
    const bool drawn = r.x1 > r.x0 && r.y1 > r.y0 && r.depth > 0.0f;
    rects[b] = drawn ? make_int4(r.x0, r.y0, r.x1, r.y1) : make_int4(0, 0, 0, 0);
    depths[b] = __float_as_int(r.depth);
}

// Bins of the screen, kRasterBinSide by kRasterBinSide at most, whole tiles each: a block per bin marks the boxes
// that meet it, a bit each, so that a tile tests the boxes of its bin and not all of them.
constexpr uint32_t kBinThreads = 1024;
constexpr uint32_t kBinWords = kRasterTileBoxes / 32u;
static_assert(kBinWords <= kTileThreads, "a word of the bin's boxes per thread of a tile");

__global__ void __launch_bounds__(kBinThreads) box_bins_kernel(const int4* rects, uint32_t boxCount, uint32_t binW, uint32_t binH,
                                                               uint32_t* masks) {
    pdl_wait();
    const int X0 = static_cast<int>(blockIdx.x * binW), Y0 = static_cast<int>(blockIdx.y * binH);
    const int X1 = X0 + static_cast<int>(binW), Y1 = Y0 + static_cast<int>(binH);
    uint32_t* const mask = masks + static_cast<size_t>(blockIdx.y * gridDim.x + blockIdx.x) * kBinWords;
    for (uint32_t first = 0; first < boxCount; first += kBinThreads) {
        const uint32_t b = first + threadIdx.x;
        const int4 r = b < boxCount ? rects[b] : make_int4(0, 0, 0, 0);  // (empty, as those of boxes not drawn)
        const uint32_t word = __ballot_sync(0xFFFFFFFFu, r.z > r.x && r.x < X1 && r.z > X0 && r.y < Y1 && r.w > Y0);
        if (threadIdx.x % 32u == 0u && b < boxCount) mask[b / 32u] = word;
    }
}

template <bool BINS>
__global__ void __launch_bounds__(kTileThreads) depth_tiles_kernel(const int4* rects, const int* depths, uint32_t boxCount,
                                                                   float* depth, uint32_t width, uint32_t height, uint32_t vec4,
                                                                   const uint32_t* masks, uint32_t binW, uint32_t binH, uint32_t binsX) {
    __shared__ int4 s_rect[kTileHits];
    __shared__ int s_depth[kTileHits];
    __shared__ uint32_t s_hits;
    pdl_wait();
    const int X0 = static_cast<int>(blockIdx.x * kTileW), Y0 = static_cast<int>(blockIdx.y * kTileH);
    const int lane = static_cast<int>(threadIdx.x & 31u), warp = static_cast<int>(threadIdx.x >> 5);
    const int wx = X0 + warp % static_cast<int>(kTileW / 32u) * 32, wy = Y0 + warp / static_cast<int>(kTileW / 32u) * 16;
    const int x = wx + lane % 8 * 4, y = wy + lane / 8;  // rows y, y + 4, y + 8, y + 12
    int v[4][4];  // depths are positive: the largest float has the largest bits
#pragma unroll
    for (int j = 0; j < 4; ++j)
#pragma unroll
        for (int i = 0; i < 4; ++i) v[j][i] = 0;
    auto meets = [&](const int4& q) {
        return q.x < X0 + static_cast<int>(kTileW) && q.z > X0 && q.y < Y0 + static_cast<int>(kTileH) && q.w > Y0;
    };
    auto keep = [&](const int4& q, uint32_t b) {
        const uint32_t at = atomicAdd(&s_hits, 1u);
        s_rect[at] = q;
        s_depth[at] = depths[b];
    };
    auto draw_list = [&] {
        const uint32_t n = s_hits;
        for (uint32_t h = 0; h < n; ++h) {
            const int4 q = s_rect[h];
            if (q.x >= wx + 32 || q.z <= wx || q.y >= wy + 16 || q.w <= wy) continue;  // (the whole warp)
            const int d = s_depth[h];
            int c[4];
#pragma unroll
            for (int i = 0; i < 4; ++i) c[i] = x + i >= q.x && x + i < q.z ? d : 0;
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const int row = y + 4 * j;
                if (row >= q.y && row < q.w) {
#pragma unroll
                    for (int i = 0; i < 4; ++i) v[j][i] = max(v[j][i], c[i]);
                }
            }
        }
    };
    bool all = true;  // whether every box is tested
    if constexpr (BINS) {
        // the boxes of the tile's bin, when the list holds them: at most kTileHits, tested in one go
        __shared__ uint16_t s_bin[kTileHits];
        __shared__ uint32_t s_marked;
        const uint32_t bin = static_cast<uint32_t>(Y0) / binH * binsX + static_cast<uint32_t>(X0) / binW;
        uint32_t word = threadIdx.x * 32u < boxCount ? masks[static_cast<size_t>(bin) * kBinWords + threadIdx.x] : 0u;
        if (threadIdx.x == 0) s_hits = s_marked = 0u;
        __syncthreads();
        if (word != 0u) {
            uint32_t at = atomicAdd(&s_marked, static_cast<uint32_t>(__popc(word)));
            for (; word != 0u && at < kTileHits; word &= word - 1u)
                s_bin[at++] = static_cast<uint16_t>(threadIdx.x * 32u + static_cast<uint32_t>(__ffs(static_cast<int>(word)) - 1));
        }
        __syncthreads();
        const uint32_t marked = s_marked;
        all = marked > kTileHits;
        if (!all) {
            for (uint32_t i = threadIdx.x; i < marked; i += kTileThreads) {
                const uint32_t b = s_bin[i];
                const int4 q = rects[b];
                if (meets(q)) keep(q, b);
            }
            __syncthreads();
            draw_list();
        }
    }
    for (uint32_t first = 0; all && first < boxCount; first += kTileThreads * kTileScan) {
        int4 r[kTileScan];
#pragma unroll
        for (uint32_t k = 0; k < kTileScan; ++k) {
            const uint32_t b = first + k * kTileThreads + threadIdx.x;
            r[k] = b < boxCount ? rects[b] : make_int4(0, 0, 0, 0);
        }
#pragma unroll
        for (uint32_t part = 0; part < kTileScan; part += kTilePart) {
            if (first + part * kTileThreads >= boxCount) break;  // (the whole block)
            __syncthreads();                                     // the list before this one is done with
            if (threadIdx.x == 0) s_hits = 0u;
            __syncthreads();
#pragma unroll
            for (uint32_t k = part; k < part + kTilePart; ++k) {
                if (meets(r[k])) keep(r[k], first + k * kTileThreads + threadIdx.x);
            }
            __syncthreads();
            draw_list();
        }
    }
#pragma unroll
    for (int j = 0; j < 4; ++j) {
        const int row = y + 4 * j;
        if (row >= static_cast<int>(height)) continue;
        float* out = depth + static_cast<size_t>(row) * width + x;
        if (vec4) {  // the width is a multiple of 4: the four are in the row or none is
            if (x < static_cast<int>(width)) *reinterpret_cast<int4*>(out) = make_int4(v[j][0], v[j][1], v[j][2], v[j][3]);
        } else {
#pragma unroll
            for (int i = 0; i < 4; ++i)
                if (x + i < static_cast<int>(width)) out[i] = __int_as_float(v[j][i]);
        }
    }
}

// Whether the boxes are sorted into bins first. A tile without bins loads 1,024 rectangles a round, so up to there is
// nothing to save (1,000 tiny boxes at 16384x16384: 144 us, 155 with bins; 2,000: 184 and 164), and the bins' launch
// costs 2 to 3 us. us a raster without and with them, boxes of 1 to 4 units and of 10 to 200:
//   2,000 boxes, 3840x2160    11.0  11.5   |  13.5  13.5
//   3,000 boxes, 3840x2160    13.2  12.4   |  17.4  15.7
//   8,192 boxes, 3840x2160    25.4  14.9   |  36.0  24.8
//   8,192 boxes, 8192x8192     140    56   |   185    88
//   8,192 boxes, 16384x16384   546   177   |   691   305
static bool raster_bins(uint32_t boxCount, uint64_t tiles) { return boxCount > 1536u && boxCount * tiles >= 5'000'000u; }

cudaError_t launch_depth_raster(const BlzCameraViewData& view, const float* boxes, uint32_t boxCount, float* depth,
                                uint32_t width, uint32_t height, void* rectScratch, cudaStream_t s, uint32_t* launches) {
    if (boxCount > 0 && boxCount <= kRasterTileBoxes && width <= kRasterTileExtent && height <= kRasterTileExtent) {
        int4* rects = static_cast<int4*>(rectScratch);
        int* depths = reinterpret_cast<int*>(rects + kRasterTileBoxes);
        cudaError_t e = launch_pdl(box_rects_kernel, (boxCount + 15) / 16, 128, 0, s, view, boxes, boxCount, width, height, rects, depths);
        if (e != cudaSuccess) return e;
        const dim3 grid((width + kTileW - 1) / kTileW, (height + kTileH - 1) / kTileH);
        const uint32_t vec4 = width % 4u == 0u && reinterpret_cast<uintptr_t>(depth) % 16 == 0 ? 1u : 0u;
        if (launches) *launches += 2;
        if (!raster_bins(boxCount, static_cast<uint64_t>(grid.x) * grid.y))
            return launch_pdl(depth_tiles_kernel<false>, grid, kTileThreads, 0, s, static_cast<const int4*>(rects), static_cast<const int*>(depths),
                              boxCount, depth, width, height, vec4, static_cast<const uint32_t*>(nullptr), 0u, 0u, 0u);
        if (launches) *launches += 1;
        uint32_t* masks = reinterpret_cast<uint32_t*>(depths + kRasterTileBoxes);
        const uint32_t binW = (grid.x + kRasterBinSide - 1) / kRasterBinSide * kTileW, binH = (grid.y + kRasterBinSide - 1) / kRasterBinSide * kTileH;
        const dim3 bins((width + binW - 1) / binW, (height + binH - 1) / binH);
        e = launch_pdl(box_bins_kernel, bins, kBinThreads, 0, s, static_cast<const int4*>(rects), boxCount, binW, binH, masks);
        if (e != cudaSuccess) return e;
        return launch_pdl(depth_tiles_kernel<true>, grid, kTileThreads, 0, s, static_cast<const int4*>(rects), static_cast<const int*>(depths),
                          boxCount, depth, width, height, vec4, static_cast<const uint32_t*>(masks), binW, binH, bins.x);
    }
    const size_t n = static_cast<size_t>(width) * height;
    const size_t n4 = (reinterpret_cast<uintptr_t>(depth) % 16 == 0) ? n / 4 : 0;
    const uint32_t ntail = static_cast<uint32_t>(n - n4 * 4);
    if (ntail > 1024) {
        cudaError_t e = cudaMemsetAsync(depth, 0, n * sizeof(float), s);
        if (e != cudaSuccess) return e;
    } else {
        cudaError_t e = launch_pdl(depth_clear_kernel, 1024, 256, 0, s, reinterpret_cast<float4*>(depth), n4, depth + n4 * 4, ntail);
        if (e != cudaSuccess) return e;
        if (launches) *launches += 1;
    }
    if (boxCount > 0) {
        const uint32_t grid = boxCount < 4096 ? boxCount : 4096;
        cudaError_t e = launch_pdl(depth_raster_kernel, grid, 256, 0, s, view, boxes, boxCount, depth, width, height);
        if (e != cudaSuccess) return e;
        if (launches) *launches += 1;
    }
    return cudaSuccess;
}

}  // namespace blz

namespace blz {

__global__ void take_status_kernel(unsigned int* status, unsigned int* out) { *out = atomicExch(status, 0u); }

__global__ void add_word_kernel(unsigned int* word, unsigned int n) { atomicAdd(word, n); }

cudaError_t launch_add_word(unsigned int* word, unsigned int n, cudaStream_t s) {
    add_word_kernel<<<1, 1, 0, s>>>(word, n);
    return cudaGetLastError();
}

cudaError_t launch_take_status(unsigned int* status, unsigned int* out, cudaStream_t s) {
    take_status_kernel<<<1, 1, 0, s>>>(status, out);
    return cudaGetLastError();
}

}  // namespace blz
