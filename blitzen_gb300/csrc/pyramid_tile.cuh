// pyramid_tile.cuh — the Hi-Z pyramid's block-level building steps, shared by the pyramid kernel
// (pyramid.cu) and the one-call frame kernel (cull_objects.cu), which builds the pyramid's tiles
// before its sweep.
//
// A block owns a 32x32 tile of mip 0. The texels of mip 0 and the levels above it are built in registers,
// through shuffles inside a warp, and only the tile's mip 3 (Vulkan: mip 2) goes through shared memory,
// from which one warp builds the rest up to mip 5. The block that finishes the build's last tile (a
// counter, taken with acquire-release semantics; no block waits) builds the few remaining small mips from
// mip 5.
//
// What bounds it: the depth buffer read once and mip 0 written (44 MB at 4K, 6.6 us of copy bandwidth),
// in the Vulkan form the L1 wavefronts of four loads a texel, and, at the end, the last block's chain of
// counter, mip 5 and top levels (about 3 us). With every level going through shared memory and a barrier
// between, and two divisions per texel of every level in the Vulkan form, it took 13.3 us at 3840x2160
// and 6.4 us at 1366x768 (D3D12) and 31 us at 2560x1440 (Vulkan); now 11.1, 5.6 and 12.9 us.
//
// Texel rules:
//   D3D12   depthPyramid.cs.hlsl:16-26 — min(r, min(g, min(b, a))) of the 2x2 Loads at
//           (2x, 2y) .. (2x+1, 2y+1) of the previous level (the depth buffer for mip 0); a Load
//           outside the previous level returns 0.
//   VULKAN  DepthPyramidGeneration.comp.glsl:15-19 — MIN-reduction bilinear footprint of the
//           previous level at ((x + 0.5) / w, (y + 0.5) / h), clamp to edge. Mip 0 is a power of
//           two, so from mip 1 on the footprint of texel x is {2x, 2x+1} (or {0} on a 1-wide level)
//           and stays inside the block's tile. (A descriptor whose mip 0 is not gets mip 0 from the
//           tiles and the rest, level by level, from the last block.)
#pragma once

#include "blz_device.cuh"
#include "kernels.h"

namespace blz {

constexpr uint32_t kPyrTile = 32;
constexpr uint32_t kPyrInTileLevels = 5;
constexpr uint32_t kPyrSmemA = kPyrTile * kPyrTile;      // floats: the tile's mip 3 and footprints, or a top level
constexpr uint32_t kPyrSmemB = kPyrTile * kPyrTile / 2;  // floats: a top level
constexpr uint32_t kPyrQuads = kPyrTile * kPyrTile / 4;  // 2x2 quads of a tile's mip 0, one per thread

// Footprint indices of texel x of a w-wide level sampling an sw-wide source (Vulkan sampler).
__device__ __forceinline__ void vk_footprint(uint32_t x, uint32_t w, uint32_t sw, uint32_t& i0, uint32_t& i1) {
    const float s = BLZ_FD(BLZ_FA(static_cast<float>(x), 0.5f), static_cast<float>(w));
    const float u = BLZ_FS(BLZ_FM(s, static_cast<float>(sw)), 0.5f);
    const float fu = floorf(u);
    const float au = BLZ_FS(u, fu);
    long long a = to_index(fu);
    long long b = (au > 0.0f) ? a + 1 : a;
    const long long hi = static_cast<long long>(sw) - 1;
    a = a < 0 ? 0 : (a > hi ? hi : a);
    b = b < 0 ? 0 : (b > hi ? hi : b);
    i0 = static_cast<uint32_t>(a);
    i1 = static_cast<uint32_t>(b);
}

// The minimum of a texel's four sources, in each form's order (r, g: upper row; b, a: lower row).
template <uint32_t MODE>
__device__ __forceinline__ float min4(float r, float g, float b, float a) {
    if (MODE == BLZ_HIZ_D3D12) return fmin_nan(r, fmin_nan(g, fmin_nan(b, a)));
    return fmin_nan(fmin_nan(fmin_nan(r, g), b), a);
}

// Texel (x, y) of a w x h level from the level below it, sw x sh texels at src (shared or global memory;
// G: global memory another block wrote, read from L2).
template <uint32_t MODE, bool G>
__device__ __forceinline__ float level_texel(const float* src, uint32_t sw, uint32_t sh, uint32_t x, uint32_t y, uint32_t w,
                                             uint32_t h) {
    auto at = [&](uint32_t i, uint32_t j) -> float {
        const float* t = src + static_cast<size_t>(j) * sw + i;
        return G ? __ldcg(t) : *t;
    };
    uint32_t i0 = 2u * x, i1 = i0 + 1u, j0 = 2u * y, j1 = j0 + 1u;
    if (MODE == BLZ_HIZ_D3D12) {
        const bool xi = i0 < sw, yi = j0 < sh, xn = i1 < sw, yn = j1 < sh;
        return min4<MODE>(xi && yi ? at(i0, j0) : 0.0f, xn && yi ? at(i1, j0) : 0.0f, xi && yn ? at(i0, j1) : 0.0f,
                          xn && yn ? at(i1, j1) : 0.0f);
    }
    if (sw != 2u * w || sh != 2u * h) {  // a level of odd extent, or one side already 1
        vk_footprint(x, w, sw, i0, i1);
        vk_footprint(y, h, sh, j0, j1);
    }
    return min4<MODE>(at(i0, j0), at(i1, j0), at(i0, j1), at(i1, j1));
}

// Whether mips 1..5 are built inside the tiles (always, but for a Vulkan descriptor whose mip 0 is not a
// power of two, where a footprint can cross tiles).
template <uint32_t MODE>
__device__ __forceinline__ bool tiles_hold_levels(const PyramidBuildParams& p) {
    return MODE == BLZ_HIZ_D3D12 || ((p.width & (p.width - 1u)) | (p.height & (p.height - 1u))) == 0u;
}

// The levels from k on, built by one block from level k - 1 in global memory: level by level through
// global memory until a level fits bufA (capA texels), from then on in shared memory (each level has at
// most half the texels of the one before, a quarter unless one side is already 1, so the levels
// alternate between bufA and bufB).
template <uint32_t MODE, int NT>
__device__ __forceinline__ void top_levels(const PyramidBuildParams& p, uint32_t k, float* bufA, uint32_t capA, float* bufB) {
    const uint32_t W0 = p.width, H0 = p.height;
    const float* prev = nullptr;  // the level below in shared memory, once it is there
    float* next = bufA;
    for (; k < p.mipCount; ++k) {
        const uint32_t Wp = mip_dim(W0, k - 1), Hp = mip_dim(H0, k - 1);
        const uint32_t Wk = mip_dim(W0, k), Hk = mip_dim(H0, k);
        const bool fits = prev != nullptr || static_cast<uint64_t>(Wk) * Hk <= capA;
        float* out = p.data + p.mipOffset[k];
        for (uint32_t idx = threadIdx.x; idx < Wk * Hk; idx += NT) {
            const uint32_t gx = idx % Wk, gy = idx / Wk;
            const float t = prev != nullptr ? level_texel<MODE, false>(prev, Wp, Hp, gx, gy, Wk, Hk)
                                            : level_texel<MODE, true>(p.data + p.mipOffset[k - 1], Wp, Hp, gx, gy, Wk, Hk);
            out[idx] = t;
            if (fits) next[idx] = t;
        }
        __syncthreads();  // this block's writes of level k are visible to its reads of level k + 1
        if (fits) {
            prev = next;
            next = next == bufA ? bufB : bufA;
        }
    }
}

// Quad (qx, qy) of a tile in patch `patch` (D3D12): the lanes of a warp take 8x4 quads in Morton order,
// the tile's 8 patches lie 2 across and 4 down.
__device__ __forceinline__ uint2 quad_place(uint32_t patch, uint32_t lane) {
    const uint32_t x = (lane & 1u) | ((lane >> 1) & 2u) | ((lane >> 2) & 4u);
    const uint32_t y = ((lane >> 1) & 1u) | ((lane >> 2) & 2u);
    return make_uint2((patch & 1u) * 8u + x, (patch >> 1) * 4u + y);
}

// The four texels of one level that a texel of the next is made of, where the right or lower ones can be
// past the level's edge (xn, yn: they are not): absent ones count as 0 (D3D12) or as the edge (Vulkan).
template <uint32_t MODE>
__device__ __forceinline__ float min4_edge(float r, float g, float b, float a, bool xn, bool yn) {
    if (MODE == BLZ_HIZ_D3D12) return min4<MODE>(r, xn ? g : 0.0f, yn ? b : 0.0f, xn && yn ? a : 0.0f);
    return min4<MODE>(r, xn ? g : r, yn ? b : r, yn ? (xn ? a : b) : (xn ? g : r));
}

// One level up inside a warp: v is the lane's texel (x, y) of level k - 1 (W x H texels), g, b and a come
// from the lanes `step`, 2 * step and 3 * step away; the lane that holds the upper left one of the four gets
// texel (x / 2, y / 2) of level k.
template <uint32_t MODE>
__device__ __forceinline__ float warp_level(float v, uint32_t step, uint32_t x, uint32_t y, uint32_t W, uint32_t H) {
    const float g = __shfl_xor_sync(0xFFFFFFFFu, v, static_cast<int>(step));
    const float b = __shfl_xor_sync(0xFFFFFFFFu, v, static_cast<int>(2u * step));
    const float a = __shfl_xor_sync(0xFFFFFFFFu, v, static_cast<int>(3u * step));
    return min4_edge<MODE>(v, g, b, a, x + 1u < W, y + 1u < H);
}

// Stores a texel of level k, if the level and the texel exist.
__device__ __forceinline__ void put_texel(const PyramidBuildParams& p, uint32_t k, uint32_t x, uint32_t y, bool mine, float v) {
    const uint32_t W = mip_dim(p.width, k), H = mip_dim(p.height, k);
    if (mine && k < p.mipCount && x < W && y < H) p.data[p.mipOffset[k] + static_cast<size_t>(y) * W + x] = v;
}

// D3D12: mips 0..3 of the tile, the 4x4 texels of mip 3 left in m3. Each warp takes PATCHES patches, the
// depth loads of all of them issued before any is used.
template <int NT>
__device__ __forceinline__ void tile_quads(const PyramidBuildParams& p, uint32_t X0, uint32_t Y0, float* m3) {
    constexpr uint32_t MODE = BLZ_HIZ_D3D12;
    constexpr uint32_t NW = NT / 32, PATCHES = NW < kPyrQuads / 32u ? kPyrQuads / 32u / NW : 1u;
    const uint32_t W0 = p.width, H0 = p.height;
    const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
    if (warp >= kPyrQuads / 32u) return;
    float d[PATCHES][4][4];  // depth rows 2gy .. 2gy + 3, columns 2gx .. 2gx + 3
#pragma unroll
    for (uint32_t i = 0; i < PATCHES; ++i) {
        const uint2 qd = quad_place(warp + i * NW, lane);
        const uint32_t gx = X0 + 2u * qd.x, gy = Y0 + 2u * qd.y;
        const bool in00 = gx < W0 && gy < H0, in10 = gx + 1u < W0 && gy < H0;
        const bool in01 = gx < W0 && gy + 1u < H0, in11 = gx + 1u < W0 && gy + 1u < H0;
        const uint32_t dw = p.depthWidth, dh = p.depthHeight;
        if (p.vec == 4u) {
            // every texel's four Loads are inside the depth buffer; an even width, so the quad has both its
            // columns or none
#pragma unroll
            for (uint32_t j = 0; j < 4u; ++j) {
                const float* row = p.depth + static_cast<size_t>(2u * gy + j) * dw + 2u * gx;
                const float4 q = (j < 2u ? in00 : in01) ? ldp(reinterpret_cast<const float4*>(row)) : make_float4(0.f, 0.f, 0.f, 0.f);
                d[i][j][0] = q.x, d[i][j][1] = q.y, d[i][j][2] = q.z, d[i][j][3] = q.w;
            }
        } else if (p.vec == 2u) {
#pragma unroll
            for (uint32_t j = 0; j < 4u; ++j) {
                const float* row = p.depth + static_cast<size_t>(2u * gy + j) * dw + 2u * gx;
                const float2 l = (j < 2u ? in00 : in01) ? ldp(reinterpret_cast<const float2*>(row)) : make_float2(0.f, 0.f);
                const float2 r = (j < 2u ? in10 : in11) ? ldp(reinterpret_cast<const float2*>(row) + 1) : make_float2(0.f, 0.f);
                d[i][j][0] = l.x, d[i][j][1] = l.y, d[i][j][2] = r.x, d[i][j][3] = r.y;
            }
        } else {
#pragma unroll
            for (uint32_t j = 0; j < 4u; ++j)
#pragma unroll
                for (uint32_t c = 0; c < 4u; ++c) {
                    const uint64_t x = 2ull * gx + c, y = 2ull * gy + j;
                    const bool in = j < 2u ? (c < 2u ? in00 : in10) : (c < 2u ? in01 : in11);
                    d[i][j][c] = in && x < dw && y < dh ? ldp(p.depth + y * dw + x) : 0.0f;
                }
        }
    }
#pragma unroll
    for (uint32_t i = 0; i < PATCHES; ++i) {
        const uint32_t patch = warp + i * NW;
        const uint2 qd = quad_place(patch, lane);
        const uint32_t gx = X0 + 2u * qd.x, gy = Y0 + 2u * qd.y;
        const bool xn = gx + 1u < W0, yn = gy + 1u < H0;
        const bool in00 = gx < W0 && gy < H0, in01 = gx < W0 && yn;
        const float t00 = min4<MODE>(d[i][0][0], d[i][0][1], d[i][1][0], d[i][1][1]);
        const float t10 = min4<MODE>(d[i][0][2], d[i][0][3], d[i][1][2], d[i][1][3]);
        const float t01 = min4<MODE>(d[i][2][0], d[i][2][1], d[i][3][0], d[i][3][1]);
        const float t11 = min4<MODE>(d[i][2][2], d[i][2][3], d[i][3][2], d[i][3][3]);
        float* out = p.data + p.mipOffset[0] + static_cast<size_t>(gy) * W0 + gx;
        if (p.pairs) {  // an even width, and pairs of texels are 8-byte aligned
            if (in00) *reinterpret_cast<float2*>(out) = make_float2(t00, t10);
            if (in01) *reinterpret_cast<float2*>(out + W0) = make_float2(t01, t11);
        } else {
            if (in00) out[0] = t00;
            if (in00 && xn) out[1] = t10;
            if (in01) out[W0] = t01;
            if (in01 && xn) out[W0 + 1u] = t11;
        }
        // mip 1: the lane's own quad; mips 2 and 3: quads of lanes
        const uint32_t x1 = gx >> 1, y1 = gy >> 1;
        const float v1 = min4_edge<MODE>(t00, t10, t01, t11, xn, yn);
        put_texel(p, 1u, x1, y1, true, v1);
        const float v2 = warp_level<MODE>(v1, 1u, x1, y1, mip_dim(W0, 1), mip_dim(H0, 1));
        put_texel(p, 2u, x1 >> 1, y1 >> 1, (lane & 3u) == 0u, v2);
        const float v3 = warp_level<MODE>(v2, 4u, x1 >> 1, y1 >> 1, mip_dim(W0, 2), mip_dim(H0, 2));
        put_texel(p, 3u, x1 >> 2, y1 >> 2, (lane & 15u) == 0u, v3);
        if ((lane & 15u) == 0u) m3[(patch >> 1) * 4u + (patch & 1u) * 2u + (lane >> 4)] = v3;
    }
}

// Vulkan: mip 0 of the tile and, when the levels stay inside the tiles, mips 1 and 2, the 8x8 texels of
// mip 2 left in m2. A warp takes four whole rows of mip 0 at a time, a column per lane: the four texels a
// lane loads for each of its texels then lie, over the lanes, in runs of 128 to 256 bytes, two or three
// L1 wavefronts a load instead of four to six for an 8x4 patch.
template <int NT>
__device__ __forceinline__ void tile_rows(const PyramidBuildParams& p, uint32_t X0, uint32_t Y0, const uint32_t* foot0,
                                          const uint32_t* foot1, bool levels, float* m2) {
    constexpr uint32_t MODE = BLZ_HIZ_VULKAN;
    constexpr uint32_t NW = NT / 32, ROWS = 4u, PATCHES = NW < kPyrTile / ROWS ? kPyrTile / ROWS / NW : 1u;
    const uint32_t W0 = p.width, H0 = p.height;
    const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
    if (warp >= kPyrTile / ROWS) return;
    const uint32_t gx = X0 + lane, c0 = foot0[lane], c1 = foot1[lane];
    float t[PATCHES][ROWS];
#pragma unroll
    for (uint32_t i = 0; i < PATCHES; ++i) {
        float s[ROWS][4];
#pragma unroll
        for (uint32_t j = 0; j < ROWS; ++j) {
            const uint32_t r = kPyrTile + (warp + i * NW) * ROWS + j;
            const float* up = p.depth + static_cast<size_t>(foot0[r]) * p.depthWidth;
            const float* lo = p.depth + static_cast<size_t>(foot1[r]) * p.depthWidth;
            s[j][0] = ldp(up + c0), s[j][1] = ldp(up + c1), s[j][2] = ldp(lo + c0), s[j][3] = ldp(lo + c1);
        }
#pragma unroll
        for (uint32_t j = 0; j < ROWS; ++j) t[i][j] = min4<MODE>(s[j][0], s[j][1], s[j][2], s[j][3]);
    }
#pragma unroll
    for (uint32_t i = 0; i < PATCHES; ++i) {
        const uint32_t patch = warp + i * NW, gy = Y0 + patch * ROWS;
#pragma unroll
        for (uint32_t j = 0; j < ROWS; ++j) put_texel(p, 0u, gx, gy + j, true, t[i][j]);
        if (!levels) continue;
        // mip 1: two texels on every even lane; mip 2: one on every fourth
        const bool xn = gx + 1u < W0;
        float v1[2];
#pragma unroll
        for (uint32_t j = 0; j < 2u; ++j) {
            const float g = __shfl_down_sync(0xFFFFFFFFu, t[i][2u * j], 1), a = __shfl_down_sync(0xFFFFFFFFu, t[i][2u * j + 1u], 1);
            v1[j] = min4_edge<MODE>(t[i][2u * j], g, t[i][2u * j + 1u], a, xn, gy + 2u * j + 1u < H0);
            put_texel(p, 1u, gx >> 1, (gy >> 1) + j, (lane & 1u) == 0u, v1[j]);
        }
        const float g = __shfl_down_sync(0xFFFFFFFFu, v1[0], 2), a = __shfl_down_sync(0xFFFFFFFFu, v1[1], 2);
        const float v2 = min4_edge<MODE>(v1[0], g, v1[1], a, (gx >> 1) + 1u < mip_dim(W0, 1), (gy >> 1) + 1u < mip_dim(H0, 1));
        put_texel(p, 2u, gx >> 2, gy >> 2, (lane & 3u) == 0u, v2);
        if ((lane & 3u) == 0u) m2[patch * 8u + (lane >> 2)] = v2;
    }
}

// One 32x32 tile of mip 0 at (X0, Y0), written and reduced through mips 1..5 by the block's NT
// threads; sA holds kPyrSmemA floats (any 4-byte alignment). It ends on a block barrier that every
// thread's writes precede.
template <uint32_t MODE, int NT>
__device__ __forceinline__ void pyramid_tile(const PyramidBuildParams& p, uint32_t X0, uint32_t Y0, float* sA) {
    static_assert(NT >= 64 && NT % 32 == 0, "a tile needs whole warps, two at least");
    const uint32_t W0 = p.width, H0 = p.height;
    const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
    const bool levels = tiles_hold_levels<MODE>(p);
    float* below = sA;  // D3D12: the tile's 4x4 texels of mip 3; Vulkan: its 8x8 texels of mip 2
    if (MODE == BLZ_HIZ_VULKAN) {
        // first and second footprint index of the tile's columns, then of its rows (absent ones repeat the edge's)
        uint32_t* foot0 = reinterpret_cast<uint32_t*>(sA + 64);
        uint32_t* foot1 = foot0 + 2u * kPyrTile;
        static_assert(64u + 4u * kPyrTile <= kPyrSmemA, "the footprints fit");
        for (uint32_t i = threadIdx.x; i < 2u * kPyrTile; i += NT) {
            uint32_t f0, f1;
            if (i < kPyrTile) vk_footprint(min(X0 + i, W0 - 1u), W0, p.depthWidth, f0, f1);
            else vk_footprint(min(Y0 + i - kPyrTile, H0 - 1u), H0, p.depthHeight, f0, f1);
            foot0[i] = f0;
            foot1[i] = f1;
        }
        __syncthreads();
        tile_rows<NT>(p, X0, Y0, foot0, foot1, levels, below);
    } else {
        tile_quads<NT>(p, X0, Y0, below);
    }
    __syncthreads();
    // the rest up to mip 5: one warp, lanes 0..15 in Morton order over the tile's 4x4 texels of mip 3
    if (levels && p.mipCount > 3u && warp == 0u) {
        const uint32_t lx = (lane & 1u) | ((lane >> 1) & 2u), ly = ((lane >> 1) & 1u) | ((lane >> 2) & 2u);
        const uint32_t x3 = (X0 >> 3) + lx, y3 = (Y0 >> 3) + ly;
        const bool has = lane < 16u;
        float v3 = 0.0f;
        if (MODE == BLZ_HIZ_VULKAN) {
            if (has) {
                const float* q = below + 16u * ly + 2u * lx;
                v3 = min4_edge<MODE>(q[0], q[1], q[8], q[9], 2u * x3 + 1u < mip_dim(W0, 2), 2u * y3 + 1u < mip_dim(H0, 2));
            }
            put_texel(p, 3u, x3, y3, has, v3);
        } else if (has) {
            v3 = below[ly * 4u + lx];
        }
        const float v4 = warp_level<MODE>(v3, 1u, x3, y3, mip_dim(W0, 3), mip_dim(H0, 3));
        put_texel(p, 4u, x3 >> 1, y3 >> 1, has && (lane & 3u) == 0u, v4);
        const float v5 = warp_level<MODE>(v4, 4u, x3 >> 1, y3 >> 1, mip_dim(W0, 4), mip_dim(H0, 4));
        put_texel(p, 5u, x3 >> 2, y3 >> 2, lane == 0u, v5);
    }
    __syncthreads();
}

// Whether any level is left for the last block.
template <uint32_t MODE>
__device__ __forceinline__ uint32_t first_top_level(const PyramidBuildParams& p) {
    return tiles_hold_levels<MODE>(p) ? kPyrInTileLevels + 1u : 1u;
}

// Counts the block's tile done in `done`, after the barrier that closes pyramid_tile. Thread 0's
// add has acquire-release semantics at GPU scope: it releases the tile the whole block wrote (the
// writes precede the barrier, the barrier precedes the add) and, in the block that finishes the
// build's last tile (tiles in all), acquires every other block's tile. That block builds the levels
// the tiles do not hold (above mip 5) and then, with `ready` given, publishes the finished pyramid (a
// barrier, then thread 0 stores 1 with release semantics); without `ready` it rewinds `done` for the
// next build. sA holds kPyrSmemA floats, sB kPyrSmemB.
template <uint32_t MODE, int NT>
__device__ __forceinline__ void pyramid_tile_finish(const PyramidBuildParams& p, uint32_t tiles, unsigned int* done,
                                                    unsigned int* ready, float* sA, float* sB) {
    __shared__ unsigned int s_last;
    if (threadIdx.x == 0) s_last = atom_add_acq_rel_gpu(done, 1u) == tiles - 1u ? 1u : 0u;
    __syncthreads();
    if (s_last) {
        if (p.mipCount > first_top_level<MODE>(p)) top_levels<MODE, NT>(p, first_top_level<MODE>(p), sA, kPyrSmemA, sB);
        if (ready != nullptr) {
            __syncthreads();
            if (threadIdx.x == 0) st_release_gpu(ready, 1u);
        } else if (threadIdx.x == 0) {
            *done = 0u;
        }
    }
}

}  // namespace blz
