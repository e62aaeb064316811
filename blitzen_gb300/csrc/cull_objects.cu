// cull_objects.cu — per-object cull kernels: frustum, occlusion pass 1 / pass 2, temporal
// occlusion, for one view or many views in one launch.
//
// Two or three kernels per call, no block ever waiting on another (lists of up to 4,096 objects: one kernel
// doing both steps, its blocks meeting at their cluster's barrier, cull_small_kernel):
//   decide   a streaming grid of warps, each deciding contiguous chunks of a view's render objects
//            (single views: one chunk per resident warp, assigned by warp index; batches: chunks
//            of 64 to 1024 objects of all views, taken from a work counter), staging the emitted ones compacted in
//            object order — (objectId, lodId), 8 bytes — in the chunk's slice of a scratch buffer,
//            with the chunk's count;
//   scatter  finds the chunks' output offsets from the counts, copies the staged records to their final
//            slots as full indirect records and writes the draw count (single views: one block per 32
//            chunks; batches: a scan launch, a block per view, then one warp per chunk).
// The scratch traffic is 16 bytes per emitted object, against 40-48 bytes read per object.
//
// Reference passes (paths inside the Blitzen project):
//   FRUSTUM   TransparentDrawCull.comp.glsl:13-65, drawCull.cs.hlsl:10-52
//   FIRST     InitialDrawCull.comp.glsl:12-59,     drawOccFirst.cs.hlsl:13-58
//   LATE      LateDrawCull.comp.glsl:13-72,        drawOccLate.cs.hlsl:13-67
//   TEMPORAL  drawOccTemporal.hlsl:13-64
#include <algorithm>

#include "blz_device.cuh"
#include "pyramid_tile.cuh"
#include "kernels.h"

namespace blz {

constexpr int kModeRuntime = -1;  // batch: the mode is read per view

// ------------------------------------------------------------------ per-view access

template <bool SINGLE>
__device__ __forceinline__ const BatchViewDev& view_of(const PipeParams& p, uint32_t vi) {
    if constexpr (SINGLE) {
        return p.single;
    } else {
        return p.views[vi];
    }
}

// Chunk c belongs to the view v with tileStart[v] <= c < tileStart[v + 1]; c is equal on every lane of the
// warp: a 32-ary search, one round
// of loads per factor of 32 views instead of one dependent load per halving.
__device__ __forceinline__ uint32_t find_view_warp(const uint32_t* tileStart, uint32_t nViews, uint32_t c) {
    const uint32_t lane = threadIdx.x & 31u;
    uint32_t lo = 0, n = nViews;  // the view is in [lo, lo + n), and tileStart[lo] <= c
    while (n > 1u) {
        const uint32_t step = (n + 31u) >> 5;
        const uint32_t cand = lo + lane * step;
        const bool le = cand < lo + n && ldp(tileStart + cand) <= c;
        const uint32_t k = 31u - static_cast<uint32_t>(__clz(static_cast<int>(__ballot_sync(0xFFFFFFFFu, le))));
        const uint32_t end = lo + n;
        lo += k * step;
        n = min(step, end - lo);
    }
    return lo;
}

// ------------------------------------------------------------------ decisions

constexpr uint32_t kChunk = 512;  // objects per chunk of batched views, unless the shape or a small batch wants others (single views size theirs)
// Chunks per group of the instanced counting sort. 16 and 8 took 46.0 and 48.7 us against 44.9 for the
// instanced pass of 4M objects and 256 LODs, 24.5 and 31.3 against 18.6 for 250k and 2000 (more rows to
// scan, fewer warps to place them).
constexpr uint32_t kInstGroup = 32;

// Where the reject test (surely_outside) comes before the exact frustum test, and the exact test runs in the
// dense stage, on the objects the bound cannot drop: the one-call frame and batches whose views all run one pass. The
// frame of 4M objects took 52.3 us without and 48.8 with it, a batch of 64 views 300 and 287. The other
// single-view passes test every object exactly where it is loaded: most of their lists are short or, in
// pass 1, mostly inside the frustum, and the second stage's latency cost 0.2 to 0.9 us of passes of 100k to
// 1M objects (at 4M the instanced pass gained 0.2 us). So does the frame in blocks of 128 threads with four objects
// each (5,000 to 200,000 objects: 8.6 to 11.3 us without, 9.8 to 12.5 with it). The kernel that reads each view's pass holds the
// code of all four, which the bound makes longer: with it 32 views of 500,000 objects, 8 of each pass, took 185 us at
// two objects a thread and 307 at four against 169 and 256 without; with one object a thread it is 160 against 221.
__host__ __device__ constexpr bool reject_mode(int mode, bool single, int threads, int opt) {
    return single ? (mode == 5 || mode == 6) && !(threads == 128 && opt == 4) : mode != kModeRuntime || opt == 1;
}
static_assert(kModeFrameFused == 5 && kModeFramePyr == 6, "reject_mode names the fused modes");

// A warp's queue of objects waiting for the dense stage, in shared memory.
constexpr uint32_t kRing = 64;  // slots: under 32 waiting plus one 32-object slice
template <bool REJECT>
struct Ring {
    // object index within the view and, in bits 30-31, min(visibility word, 2); then
    // REJECT: surface id, pos.xy | pos.z, scale, quat.xy | quat.zw; else: view-space centre | r, scale, LOD range
    uint4 a[kRing];
    uint4 b[kRing];
    uint2 c[REJECT ? kRing : 1u];
};
constexpr uint32_t kBadObject = 0xFFFFFFFFu;  // in place of the surface id: a transform or surface id was out of range

// A frustum survivor pass 1 of a kept frame hands to pass 2 (32 bytes, two 16-byte words).
struct Survivor {
    uint32_t obj;      // object index within the view (bit 31: visibility word was not 0, bit 30: it was 1)
    float cx, cy, cz;  // view-space sphere centre
    float r, scale;
    uint32_t lodOff, lodCnt;
};

// Both passes of a frame decided in one sweep, with the pyramid built before the launch or inside it.
__host__ __device__ constexpr bool fused_mode(int m) { return m == kModeFrameFused || m == kModeFramePyr; }

// A warp's wait for the pyramid its own launch builds (kModeFramePyr): the whole warp polls the
// ready flag with acquire semantics (one load serves every lane, so all see the same value), at
// most `limit` times; then it raises BLZ_FLAG_TIMEOUT and goes on with whatever the pyramid holds.
__device__ __forceinline__ void wait_pyramid(const unsigned int* ready, uint32_t limit, unsigned int& flags) {
    for (uint32_t polls = 0; ld_acquire_gpu(ready) == 0u;) {
        if (++polls >= limit) {
            flags |= BLZ_FLAG_TIMEOUT;
            break;
        }
        __nanosleep(128);
    }
    __syncwarp();
}

// The lanes of the warp whose record has the same LOD id as this lane's (ids below 2^bits): one
// ballot per bit of the id, each lane keeping the lanes that agree with it on every bit. Votes, not
// a match instruction, so the ranking stays off the shared-memory pipe. Lanes without a record
// (valid false) get a mask their callers do not use.
__device__ __forceinline__ unsigned same_lod_lanes(uint32_t b, uint32_t bits, bool valid) {
    unsigned m = __ballot_sync(0xFFFFFFFFu, valid);
    for (uint32_t k = 0; k < bits; ++k) {
        const bool bit = ((b >> k) & 1u) != 0u;
        const unsigned v = __ballot_sync(0xFFFFFFFFu, bit);
        m &= bit ? v : ~v;
    }
    return m;
}

// The surface table's fields the object stages read, copied into shared memory by each block when the
// table is small enough; null pointers: read the table in global memory.
struct SurfaceCache {
    const float2* bound;  // what the reject test reads: radius, centre norm (see surface_bound)
    const float4* sphere;
    const uint2* lod;     // lodOffset, lodCount
    const float* error;   // every LOD's error, when there are few enough; null: read the LOD table
};

__device__ __forceinline__ bool lod_range_ok(uint2 lod, uint32_t lodCount) {
    return lod.x < lodCount && lod.y <= lodCount - lod.x;
}

// Dense stage over n <= 32 queued objects starting at ring index head, one per lane, in object order:
// the exact frustum test, where it is not behind them (REJECT); for the objects inside, the sphere projection and Hi-Z test (LATE/TEMPORAL);
// LATE's visibility write; LOD selection of the emitted ones, and their staging as (objectId, lodId)
// after the `run` already staged for the chunk.
// kModeFrame1 emits the survivors visible last frame (its pass-1 records), tests no pyramid and appends
// every object inside the frustum to the chunk's kept survivors (keep[kept ...], 32 bytes each).
// The fused modes stage pass 2's records in `stage` and pass 1's in `stage1` (run1).
template <int MODE, bool REJECT>
__device__ __forceinline__ void dense_round(const SceneTables& sc, const BatchViewDev& bv, const ViewConsts& v,
                                            const SurfaceCache& surf, const Ring<REJECT>& ring, uint32_t head, uint32_t n,
                                            unsigned int& flags, uint2* stage, uint32_t& run, uint4* keep, uint32_t& kept,
                                            uint2* stage1, uint32_t* run1, uint32_t* hist, uint32_t lt) {
    constexpr bool FUSED = fused_mode(MODE);
    constexpr bool REWRITE = MODE == BLZ_MODE_LATE || FUSED;  // pass 2's visibility rewrite
    const uint32_t lane = threadIdx.x & 31u;
    const uint32_t at = (head + lane) & (kRing - 1u);
    const uint4 ra = ring.a[at], rb = ring.b[at];
    const bool mine = lane < n;
    const uint32_t obj = ra.x & 0x3FFFFFFFu, vis = ra.x >> 30;  // (vis: 2 for every word above 1)
    const bool wasNonZero = vis != 0u;
    Vec3 c;
    float r, scale;
    uint2 lod;
    bool inside = mine;
    if constexpr (REJECT) {
        const uint2 rc = ring.c[at];
        const bool known = mine && ra.y != kBadObject;
        const uint32_t sid = known ? ra.y : 0u;
        float4 sph;
        if (surf.sphere != nullptr) {
            sph = surf.sphere[sid];
            lod = surf.lod[sid];
        } else {
            const float4* sp = reinterpret_cast<const float4*>(sc.surfaces + sid);
            sph = ldp(sp);
            const uint4 s1 = ldp(reinterpret_cast<const uint4*>(sp + 1));  // materialId, lodOffset, lodCount, vertexOffset
            lod = make_uint2(s1.y, s1.z);
        }
        const bool good = known && lod_range_ok(lod, sc.lodCount);
        if (mine && !good) flags |= BLZ_FLAG_BAD_INDEX;
        const float4 ps = make_float4(__uint_as_float(ra.z), __uint_as_float(ra.w), __uint_as_float(rb.x), __uint_as_float(rb.y));
        const float4 q = make_float4(__uint_as_float(rb.z), __uint_as_float(rb.w), __uint_as_float(rc.x), __uint_as_float(rc.y));
        c = view_transform(v.rows, model_to_world(Vec3{sph.x, sph.y, sph.z}, ps, q));
        r = BLZ_FM(sph.w, ps.w);
        scale = ps.w;
        inside = good && frustum_check(c, r, v);
    } else {
        c = Vec3{__uint_as_float(ra.y), __uint_as_float(ra.z), __uint_as_float(ra.w)};
        r = __uint_as_float(rb.x);
        scale = __uint_as_float(rb.y);
        lod = make_uint2(rb.z, rb.w);
    }
    bool visible = inside;
    if (inside && (MODE == BLZ_MODE_LATE || MODE == BLZ_MODE_TEMPORAL || FUSED)) {
        float4 aabb;
        if (project_sphere(c, r, v.zNear, v.proj0, v.proj5, aabb))
            visible = occlusion<MODE == kModeFramePyr>(aabb, bv.pyr, v, c, r);
    }
    if (MODE == kModeFrame1) {
        const unsigned k = __ballot_sync(0xFFFFFFFFu, inside);
        if (inside) {
            uint4* e = keep + 2u * (kept + __popc(k & lt));
            const uint32_t tag = (vis != 0u ? 0x80000000u : 0u) | (vis == 1u ? 0x40000000u : 0u);
            e[0] = make_uint4(obj | tag, __float_as_uint(c.x), __float_as_uint(c.y), __float_as_uint(c.z));
            e[1] = make_uint4(__float_as_uint(r), __float_as_uint(scale), lod.x, lod.y);
        }
        kept += __popc(k);
    } else if (REWRITE && mine) {
        // drawOccLate.cs.hlsl:67, storing only a value that changes
        const uint32_t now = visible ? 1u : 0u;
        if (vis != now) bv.vis[obj] = now;
    }
    // drawOccLate.cs.hlsl:45; a kept frame's pass 1 emits what drawOccFirst.cs.hlsl:22-25 admits
    const bool emitted = visible && (REWRITE ? !wasNonZero : (MODE == kModeFrame1 ? wasNonZero : true));
    // the fused sweep's pass 1: every object inside the frustum that was visible last frame
    const bool emitted1 = FUSED && inside && wasNonZero;
    uint32_t lid = 0u;
    if (emitted || emitted1) {
        // cullBuffers.hlsl:42-55 — last LOD in [1, lodCount) with error < threshold
        const float threshold = lod_threshold(c, r, scale, v.lodTarget);
        uint32_t sel = 0;
        if (surf.error != nullptr) {
            for (uint32_t t = 1; t < lod.y; ++t)
                if (surf.error[lod.x + t] < threshold) sel = t;
        } else {
            for (uint32_t t = 1; t < lod.y; ++t)
                if (ldp(&sc.lods[lod.x + t].error) < threshold) sel = t;
        }
        lid = lod.x + sel;
    }
    const unsigned e = __ballot_sync(0xFFFFFFFFu, emitted);
    if (emitted) stage[run + __popc(e & lt)] = make_uint2(obj, lid);
    run += __popc(e);
    if constexpr (MODE == kModeInstanced) {
        // the group's histogram row (hist = row of this chunk's group): one add per distinct LOD
        const uint32_t idBits = sc.lodCount > 1u ? 32u - static_cast<uint32_t>(__clz(static_cast<int>(sc.lodCount - 1u))) : 0u;
        const unsigned peers = same_lod_lanes(lid, idBits, emitted);
        if (emitted && (peers & lt) == 0u) atomicAdd(hist + lid, static_cast<uint32_t>(__popc(peers)));
    }
    if constexpr (FUSED) {
        const unsigned e1 = __ballot_sync(0xFFFFFFFFu, emitted1);
        if (emitted1) stage1[*run1 + __popc(e1 & lt)] = make_uint2(obj, lid);
        *run1 += __popc(e1);
    }
}

// A view's constants as a batch's warp keeps them.
struct SharedView {
    ViewConsts v;
    RejectBounds rj;
    float pad;
};

// Pass 1's queue of the objects visible last frame (single views; empty in every other kernel), per warp.
template <uint32_t SLOTS>
struct Candidates {
    uint2 ro[SLOTS];
    uint32_t obj[SLOTS];
};
__host__ __device__ constexpr uint32_t candidate_slots(int mode, bool single, int opt) {
    return mode == BLZ_MODE_FIRST && single ? 2u * 32u * opt : 1u;
}

// One warp decides the objects [base, limit) of a view, 32 * OPT at a time (object
// sb + k * 32 + lane for k < OPT, so lanes ascend within each 32-object slice):
//   1  every lane loads its OPT render objects (fetched one step ahead) and their transforms, and runs
//      the frustum test (REJECT: drops the objects a bound proves outside, 34 operations against 75)
//      — without branches: an object that is out of range, not active in this pass or has a bad id reads
//      the tables' first rows and is masked out (REJECT: or queued). Pass 1 (single views) first packs
//      the objects visible last frame into a candidate ring, so this stage runs on full lanes there too;
//   2  what is left of each slice is appended, in object order, to the warp's ring in shared memory;
//      whenever 32 are waiting they go through the dense stage on full lanes, so the costly part
//      (REJECT: the exact frustum test; projection, Hi-Z, LOD) never runs on a lane without an object;
//   3  the dense stage stages the emitted ones in order; the rest drains at the end.
// Returns the number of records staged. No block barrier: warps never wait for one another.
template <int MODE, bool SINGLE, int OPT, bool REJECT>
__device__ __forceinline__ uint32_t decide_run_warp(const SceneTables& sc, const BatchViewDev& bv, uint32_t base,
                                                    uint32_t limit, uint2* stage, Ring<REJECT>& ring, Candidates<candidate_slots(MODE, SINGLE, OPT)>& cand,
                                                    const SurfaceCache& surf, SharedView* shared, unsigned int& flags, uint4* keep,
                                                    uint32_t& kept, uint2* stage1 = nullptr, uint32_t* run1 = nullptr,
                                                    const unsigned int* ready = nullptr, uint32_t spinLimit = 0u,
                                                    uint32_t* hist = nullptr) {
    constexpr uint32_t STEP = 32u * OPT;
    constexpr bool OWN = SINGLE || !REJECT;  // the view's constants in registers
    constexpr bool PACK = (MODE == BLZ_MODE_FIRST) && SINGLE;  // candidate ring of 2 * STEP entries
    // Single-view pass 2 walks its chunk from the last object down: pass 1 walked the same chunk
    // upwards just before (with only the pyramid build between), so the lines it touched last are
    // the ones still in L2. Records are then staged in descending order; the scatter writes each
    // chunk's records back to front. Slot i of the walk is object `walk(i)`; past the end it is
    // kNoObject, never active.
    constexpr bool DOWN = (MODE == BLZ_MODE_LATE) && SINGLE;
    constexpr uint32_t kNoObject = 0xFFFFFFFFu;
    auto walk = [&](uint32_t i) -> uint32_t { return i < limit ? (DOWN ? base + limit - 1u - i : i) : kNoObject; };
    const uint32_t lane = threadIdx.x & 31u, lt = (1u << lane) - 1u;
    if (sc.transformCount == 0u || sc.surfaceCount == 0u) {
        // nothing can be looked up: every object of the pass has a bad id and none is visible
        for (uint32_t i = base + lane; i < limit; i += 32u) {
            const bool act = MODE != BLZ_MODE_FIRST || ldp(bv.vis + i) != 0u;
            if (act) flags |= BLZ_FLAG_BAD_INDEX;
            if (MODE == BLZ_MODE_LATE || MODE == kModeFrame1 || fused_mode(MODE)) bv.vis[i] = 0u;
        }
        return 0u;
    }
    // The view's constants: a single view's come from the launch parameters, whose reads are operands of the
    // arithmetic; a batch's are kept in shared memory by the warp and read again by each step and each
    // dense round, since together with the loop's state they do not fit the registers.
    if constexpr (!OWN) {
        __syncwarp();  // the chunk before this one is done with them
        if (threadIdx.x % 32u == 0u) {
            shared->v = load_view(bv.view);
            shared->rj = reject_bounds(shared->v);
        }
        __syncwarp();
    }
    ViewConsts own;
    RejectBounds ownRj;
    if constexpr (OWN) {
        own = load_view(bv.view);
        ownRj = reject_bounds(own);
    }
    const ViewConsts& v = OWN ? own : shared->v;
    [[maybe_unused]] const RejectBounds& rj = OWN ? ownRj : shared->rj;
    // what the loop reads of the view, kept in registers (a batch's views lie in global memory, from where
    // every field would be read again after each store)
    const uint2* const objects = reinterpret_cast<const uint2*>(bv.objects);
    uint32_t* const visWords = bv.vis;
    const BlzMeshTransform* const dynT = SINGLE ? nullptr : bv.dynT;
    const uint32_t dynCount = SINGLE || dynT == nullptr ? 0u : bv.dynCount;
    uint32_t run = 0, head = 0, tail = 0;
    // kModeFramePyr: the pyramid is waited for once, before the warp's first dense round
    bool pyrSeen = MODE != kModeFramePyr;
    auto dense = [&](uint32_t n) {
        if (!pyrSeen) {
            wait_pyramid(ready, spinLimit, flags);
            pyrSeen = true;
        }
        dense_round<MODE, REJECT>(sc, bv, v, surf, ring, head, n, flags, stage, run, keep, kept, stage1, run1, hist, lt);
    };

    // frustum stage over OPT slices: obj[k] the object index, ro[k] its render object, vis[k] the
    // object's visibility word (LATE: as read; the object is active when in range) or, in the other
    // passes, non-zero when the object is active
    float4 ps[OPT], q[OPT];
    float2 bound[OPT];   // REJECT
    float4 sph[OPT];     // else
    uint2 lod[OPT];
    uint32_t sid[OPT];   // or kBadObject
    // LATE and kModeFrame1 test every object (vis[k] holds its visibility word), the others the
    // objects with vis[k] != 0
    constexpr bool ALL = MODE == BLZ_MODE_LATE || MODE == kModeFrame1 || fused_mode(MODE);
    auto active = [&](uint32_t obj, uint32_t vis) -> bool { return ALL ? obj < limit : vis != 0u; };
    auto gather = [&](const uint32_t (&obj)[OPT], const uint2 (&ro)[OPT], const uint32_t (&vis)[OPT]) {
#pragma unroll
        for (int k = 0; k < OPT; ++k) {
            const bool ok = active(obj[k], vis[k]) && ro[k].x < sc.transformCount && ro[k].y < sc.surfaceCount;
            const uint32_t tid = ok ? ro[k].x : 0u, s = ok ? ro[k].y : 0u;
            sid[k] = ok ? s : kBadObject;
            const BlzMeshTransform* rows = tid < sc.dynCount ? sc.dynRows : sc.transforms;
            if (!SINGLE && tid < dynCount) rows = dynT;  // the view's own rows first
            ldg_transform(rows + tid, ps[k], q[k]);
            const float4* sp = reinterpret_cast<const float4*>(sc.surfaces + s);
            if constexpr (REJECT) {
                if (surf.bound != nullptr) {
                    bound[k] = surf.bound[s];
                } else {
                    const uint4 s1 = ldp(reinterpret_cast<const uint4*>(sp + 1));
                    bound[k] = surface_bound(ldp(sp), lod_range_ok(make_uint2(s1.y, s1.z), sc.lodCount));
                }
            } else if (surf.sphere != nullptr) {
                sph[k] = surf.sphere[s];
                lod[k] = surf.lod[s];
            } else {
                sph[k] = ldp(sp);
                const uint4 s1 = ldp(reinterpret_cast<const uint4*>(sp + 1));  // materialId, lodOffset, lodCount, vertexOffset
                lod[k] = make_uint2(s1.y, s1.z);
            }
        }
    };
    auto test = [&](const uint32_t (&obj)[OPT], const uint32_t (&vis)[OPT]) {
#pragma unroll
        for (int k = 0; k < OPT; ++k) {
            const bool act = active(obj[k], vis[k]);
            bool queued;
            Vec3 c{0.f, 0.f, 0.f};
            float r = 0.f;
            if constexpr (REJECT) {
                queued = act && (sid[k] == kBadObject || !surely_outside(ps[k], q[k], bound[k], v, rj));
            } else {
                const bool good = sid[k] != kBadObject && lod_range_ok(lod[k], sc.lodCount);
                if (act && !good) flags |= BLZ_FLAG_BAD_INDEX;
                c = view_transform(v.rows, model_to_world(Vec3{sph[k].x, sph[k].y, sph[k].z}, ps[k], q[k]));
                r = BLZ_FM(sph[k].w, ps[k].w);
                queued = good && frustum_check(c, r, v);
            }
            // drawOccLate.cs.hlsl:67, storing only a value that changes
            if (ALL && act && !queued && vis[k] != 0u) visWords[obj[k]] = 0u;
            const unsigned m = __ballot_sync(0xFFFFFFFFu, queued);
            if (queued) {
                const uint32_t at = (tail + __popc(m & lt)) & (kRing - 1u);
                const uint32_t o = obj[k] | (ALL ? min(vis[k], 2u) << 30 : 0u);
                if constexpr (REJECT) {
                    ring.a[at] = make_uint4(o, sid[k], __float_as_uint(ps[k].x), __float_as_uint(ps[k].y));
                    ring.b[at] = make_uint4(__float_as_uint(ps[k].z), __float_as_uint(ps[k].w), __float_as_uint(q[k].x), __float_as_uint(q[k].y));
                    ring.c[at] = make_uint2(__float_as_uint(q[k].z), __float_as_uint(q[k].w));
                } else {
                    ring.a[at] = make_uint4(o, __float_as_uint(c.x), __float_as_uint(c.y), __float_as_uint(c.z));
                    ring.b[at] = make_uint4(__float_as_uint(r), __float_as_uint(ps[k].w), lod[k].x, lod[k].y);
                }
            }
            tail += __popc(m);
            if (tail - head >= 32u) {
                __syncwarp();
                dense(32u);
                head += 32u;
                __syncwarp();
            }
        }
    };

    uint2 nro[OPT];
    uint32_t nvis[OPT];
    auto prefetch = [&](uint32_t at) {
#pragma unroll
        for (int k = 0; k < OPT; ++k) {
            const uint32_t i = walk(at + k * 32u + lane);
            const bool in = i != kNoObject;
            nro[k] = in ? ldp(objects + i) : make_uint2(0u, 0u);
            nvis[k] = in ? 1u : 0u;
            if (MODE == BLZ_MODE_FIRST && in) nvis[k] = ldp(visWords + i);
            if (ALL) nvis[k] = in ? visWords[i] : 0u;
        }
    };
    // candidates packed by pass 1, taken STEP at a time (or the rest, at the end)
    uint32_t ahead = 0, atail = 0;
    auto take_candidates = [&](uint32_t n) {
        uint2 ro[OPT];
        uint32_t obj[OPT], vis[OPT];
        __syncwarp();
#pragma unroll
        for (int k = 0; k < OPT; ++k) {
            const uint32_t j = k * 32u + lane;
            const uint32_t at = (ahead + j) & (2u * STEP - 1u);
            const bool in = j < n;
            obj[k] = cand.obj[at];
            ro[k] = cand.ro[at];
            vis[k] = in ? 1u : 0u;
        }
        __syncwarp();
        ahead += n;
        gather(obj, ro, vis);
        test(obj, vis);
    };

    if (base < limit) prefetch(base);
    for (uint32_t sb = base; sb < limit; sb += STEP) {
        uint2 ro[OPT];
        uint32_t obj[OPT], vis[OPT];
#pragma unroll
        for (int k = 0; k < OPT; ++k) {
            ro[k] = nro[k];
            vis[k] = nvis[k];  // pass 1: active when visible last frame (drawOccFirst.cs.hlsl:22-25)
            obj[k] = DOWN ? walk(sb + k * 32u + lane) : sb + k * 32u + lane;
        }
        if constexpr (PACK) {
            if (sb + STEP < limit) prefetch(sb + STEP);
#pragma unroll
            for (int k = 0; k < OPT; ++k) {
                const bool act = vis[k] != 0u;
                const unsigned m = __ballot_sync(0xFFFFFFFFu, act);
                if (act) {
                    const uint32_t at = (atail + __popc(m & lt)) & (2u * STEP - 1u);
                    cand.obj[at] = obj[k];
                    cand.ro[at] = ro[k];
                }
                atail += __popc(m);
            }
            if (atail - ahead >= STEP) take_candidates(STEP);
        } else {
            gather(obj, ro, vis);
            if (sb + STEP < limit) prefetch(sb + STEP);
            test(obj, vis);
        }
    }
    if constexpr (PACK) {
        if (atail != ahead) take_candidates(atail - ahead);
    }
    if (tail != head) {
        __syncwarp();
        dense(tail - head);
        __syncwarp();
    }
    return run;
}

// Writes one record {objId, indexCount, 1, firstIndex, 0, 0}; pad words of 32-byte records are
// left untouched like the reference shaders leave them.
__device__ __forceinline__ void put_record(uint8_t* cmds, uint32_t stride, uint32_t slot, uint32_t objId,
                                           uint32_t indexCount, uint32_t firstIndex) {
    uint8_t* rec = cmds + static_cast<size_t>(slot) * stride;
    if (stride == BLZ_STRIDE_D3D12) {
        *reinterpret_cast<uint4*>(rec) = make_uint4(objId, indexCount, 1u, firstIndex);
        *reinterpret_cast<uint2*>(rec + 16) = make_uint2(0u, 0u);
    } else {
        uint2* w = reinterpret_cast<uint2*>(rec);
        w[0] = make_uint2(objId, indexCount);
        w[1] = make_uint2(1u, firstIndex);
        w[2] = make_uint2(0u, 0u);
    }
}

// ------------------------------------------------------------------ decide kernel

// Shared memory of the decide kernels: one ring per warp, pass 1's candidate rings, and the surface
// table in what static shared memory is left (48 KB per block).
template <int MODE, bool SINGLE, int THREADS, int OPT>
struct DecideSmem {
    static constexpr int NW = THREADS / 32;
    using Cand = Candidates<candidate_slots(MODE, SINGLE, OPT)>;
    using Queue = Ring<reject_mode(MODE, SINGLE, THREADS, OPT)>;
    static constexpr bool REJECT = reject_mode(MODE, SINGLE, THREADS, OPT);
    static constexpr uint32_t kViews = SINGLE || !REJECT ? 1u : NW;
    static constexpr size_t kUsed = (sizeof(Queue) + sizeof(Cand)) * NW + kViews * sizeof(SharedView);
    static constexpr uint32_t kLods = REJECT && kUsed + 2048 + 1024 <= 48 * 1024 ? 512u : 1u;  // LOD errors
    static constexpr size_t kLeft = kUsed + kLods * 4 + 1024 < 48 * 1024 ? 48 * 1024 - 1024 - kLods * 4 - kUsed : 0;
    static constexpr size_t kSurfBytes = (REJECT ? sizeof(float2) : 0) + sizeof(float4) + sizeof(uint2);
    static constexpr uint32_t kSurf = kLeft >= 512 * kSurfBytes ? 512u : (kLeft >= 256 * kSurfBytes ? 256u : (kLeft >= 64 * kSurfBytes ? 64u : 1u));
    Queue ring[NW];
    SharedView view[kViews];
    Cand cand[NW];
    float4 sphere[kSurf];
    float2 bound[REJECT ? kSurf : 1u];
    uint2 lod[kSurf];
    float error[kLods];
};

// The decide kernels' body: each warp decides chunks of a view (decide_run_warp) and records each
// chunk's count; the count of the warp's last chunk is returned (0 when it had none). kModeFramePyr
// passes the context's pyramid-ready flag and its wait limit. LOCAL: one chunk a warp at most, its
// records staged at warpStage and its count only returned.
template <int MODE, bool SINGLE, int THREADS, int OPT, bool LOCAL = false>
__device__ __forceinline__ uint32_t decide_body(const PipeParams& p, DecideSmem<MODE, SINGLE, THREADS, OPT>& sm,
                                                const unsigned int* ready = nullptr, uint32_t spinLimit = 0u,
                                                uint2* warpStage = nullptr) {
    using Smem = DecideSmem<MODE, SINGLE, THREADS, OPT>;
    constexpr int NW = Smem::NW;
    constexpr uint32_t kSurf = Smem::kSurf;
    SurfaceCache surf{nullptr, nullptr, nullptr, nullptr};
    if (Smem::kLods > 1u && p.sc.lodCount <= Smem::kLods) {
        for (uint32_t i = threadIdx.x; i < p.sc.lodCount; i += THREADS) sm.error[i] = ldp(&p.sc.lods[i].error);
        surf.error = sm.error;
    }
    if (kSurf > 1u && p.sc.surfaceCount <= kSurf) {
        for (uint32_t i = threadIdx.x; i < p.sc.surfaceCount; i += THREADS) {
            const float4* sp = reinterpret_cast<const float4*>(p.sc.surfaces + i);
            const float4 sph = ldp(sp);
            const uint4 s1 = ldp(reinterpret_cast<const uint4*>(sp + 1));  // materialId, lodOffset, lodCount, vertexOffset
            const uint2 lod = make_uint2(s1.y, s1.z);
            sm.sphere[i] = sph;
            if (Smem::REJECT) sm.bound[i] = surface_bound(sph, lod_range_ok(lod, p.sc.lodCount));
            sm.lod[i] = lod;
        }
        surf = SurfaceCache{sm.bound, sm.sphere, sm.lod, surf.error};
    }
    __syncthreads();
    const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
    const uint32_t warpsTotal = gridDim.x * NW;
    const uint32_t chunkSize = p.chunkSize;
    unsigned int flags = 0u;
    uint32_t last = 0u;
    // every warp starts on the chunk of its index; later chunks come from the work counter when
    // there is one (a warp that finishes early takes the next, so warps finish together), else by
    // a stride of the grid's warp count
    auto next_chunk = [&](uint32_t cur) -> uint32_t {
        if (p.workCounter == nullptr) return cur + warpsTotal;
        uint32_t c = 0;
        if (lane == 0) c = warpsTotal + atomicAdd(p.workCounter, 1u);
        return __shfl_sync(0xFFFFFFFFu, c, 0);
    };
    uint32_t item = blockIdx.x * NW + warp;
    while (item < p.totalTiles) {
        const uint32_t next = next_chunk(item);  // asked now, used after this chunk
        const uint32_t chunk = !SINGLE && p.order != nullptr ? __ldcg(p.order + item) : item;
        uint32_t vi = 0, first = 0;
        if constexpr (!SINGLE) {
            vi = find_view_warp(p.tileStart, p.viewCount, chunk);
            first = ldp(p.tileStart + vi);
        }
        const BatchViewDev& bv = view_of<SINGLE>(p, vi);
        const uint32_t base = (chunk - first) * chunkSize;
        const uint32_t limit = min(base + chunkSize, bv.count);
        uint2* stage = LOCAL ? warpStage : p.staged + static_cast<size_t>(chunk) * chunkSize;
        auto& ring = sm.ring[warp];
        auto& cand = sm.cand[warp];
        SharedView* shared = &sm.view[Smem::kViews == 1u ? 0u : warp];
        uint32_t total = 0, kept = 0, total1 = 0;
        uint4* keep = nullptr;
        if constexpr (MODE == kModeFrame1) keep = static_cast<uint4*>(p.keep) + 2u * static_cast<size_t>(chunk) * chunkSize;
        uint2* stage1 = nullptr;
        if constexpr (fused_mode(MODE)) stage1 = p.staged2 + static_cast<size_t>(chunk) * chunkSize;
        if constexpr (MODE == kModeRuntime) {
            switch (bv.mode) {
                case BLZ_MODE_FIRST: total = decide_run_warp<BLZ_MODE_FIRST, SINGLE, OPT, Smem::REJECT>(p.sc, bv, base, limit, stage, ring, cand, surf, shared, flags, keep, kept); break;
                case BLZ_MODE_LATE: total = decide_run_warp<BLZ_MODE_LATE, SINGLE, OPT, Smem::REJECT>(p.sc, bv, base, limit, stage, ring, cand, surf, shared, flags, keep, kept); break;
                case BLZ_MODE_TEMPORAL: total = decide_run_warp<BLZ_MODE_TEMPORAL, SINGLE, OPT, Smem::REJECT>(p.sc, bv, base, limit, stage, ring, cand, surf, shared, flags, keep, kept); break;
                default: total = decide_run_warp<BLZ_MODE_FRUSTUM, SINGLE, OPT, Smem::REJECT>(p.sc, bv, base, limit, stage, ring, cand, surf, shared, flags, keep, kept); break;
            }
        } else {
            uint32_t* hist = nullptr;
            if constexpr (MODE == kModeInstanced) hist = p.instHist + static_cast<size_t>(chunk / kInstGroup) * p.instLods;
            total = decide_run_warp<(MODE < 0 ? 0 : MODE), SINGLE, OPT, Smem::REJECT>(p.sc, bv, base, limit, stage, ring, cand, surf, shared, flags, keep, kept,
                                                                       stage1, &total1, ready, spinLimit, hist);
        }
        if (!LOCAL && lane == 0) {
            p.chunkCount[chunk] = total;
            if constexpr (MODE == kModeFrame1) p.keepCount[chunk] = kept;
            if constexpr (fused_mode(MODE)) p.chunkCount2[chunk] = total1;
        }
        last = total;
        item = next;
    }
    if (flags) atomicOr(&p.scratch->status, flags);
    return last;
}

template <int MODE, bool SINGLE, int THREADS, int OPT>
__global__ void __launch_bounds__(THREADS, SINGLE || MODE >= 0 ? 1024 / THREADS : 1) cull_decide_kernel(const PipeParams p) {
    __shared__ DecideSmem<MODE, SINGLE, THREADS, OPT> sm;
    pdl_wait();
    decide_body<MODE, SINGLE, THREADS, OPT>(p, sm);
}

// The one-call frame with its pyramid (blz_cull_frame given a depth buffer) in one launch. Each
// block first takes pyramid tiles by ticket until none is left, building each with the pyramid
// kernel's block steps in the shared memory its survivor rings use later; the block that finishes
// the last tile builds the top levels and publishes the pyramid (the context's ready flag). Then the
// block's warps run the fused sweep, each waiting for the flag before its first Hi-Z test. Tiles go
// to running blocks only, and a block waits for nothing while it builds, so every tile a warp waits
// for belongs to a block that is running; the waits are bounded all the same. The frame's scatter
// rewinds the ticket, the tile count and the flag.
template <uint32_t HIZ, int THREADS, int OPT>
__global__ void __launch_bounds__(THREADS, 1024 / THREADS) cull_frame_kernel(const PipeParams p,
                                                                           const __grid_constant__ PyramidBuildParams bp) {
    using Smem = DecideSmem<kModeFramePyr, true, THREADS, OPT>;
    __shared__ Smem sm;
    static_assert(sizeof(sm.ring) >= sizeof(float) * (kPyrSmemA + kPyrSmemB), "the tile buffers live in the rings");
    float* sA = reinterpret_cast<float*>(&sm.ring[0]);
    float* sB = sA + kPyrSmemA;
    __shared__ uint32_t s_tile;
    pdl_wait();
    Scratch* scr = p.scratch;
    const uint32_t tilesX = (bp.width + kPyrTile - 1) / kPyrTile;
    const uint32_t tiles = tilesX * ((bp.height + kPyrTile - 1) / kPyrTile);
    for (;;) {
        if (threadIdx.x == 0) s_tile = atomicAdd(&scr->frameTicket, 1u);
        __syncthreads();
        const uint32_t t = s_tile;
        if (t >= tiles) break;
        pyramid_tile<HIZ, THREADS>(bp, (t % tilesX) * kPyrTile, (t / tilesX) * kPyrTile, sA);
        pyramid_tile_finish<HIZ, THREADS>(bp, tiles, &scr->frameTilesDone, &scr->frameReady, sA, sB);
        __syncthreads();  // s_tile and the tile buffers are free again
    }
    decide_body<kModeFramePyr, true, THREADS, OPT>(p, sm, &scr->frameReady, bp.spinLimit);
}

// ------------------------------------------------------------------ scatter kernel

// Single views. Each block owns 32 consecutive chunks, one per warp, and finds where their records go
// without any grid-wide step: it sums the counts that precede its first chunk (a strided read of the counts,
// from L2), and warp 0 scans the 32 chunks' counts. The block's warps then copy the chunks' staged records
// to their slots as full records, and the lane holding the last chunk writes the draw count.
constexpr int kScatterWarps = 32;  // one warp per chunk
constexpr uint32_t kScatterChunks = 32;
constexpr uint32_t kScatterPre = 3;  // 32-record slices of its chunk a warp loads before the offsets are known

__device__ __forceinline__ void scatter_block(const PipeParams& p, const uint32_t block) {
    __shared__ uint32_t s_part[kScatterWarps];
    __shared__ uint32_t s_base[kScatterChunks], s_n[kScatterChunks];
    const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
    const uint32_t chunkSize = p.chunkSize;
    const uint32_t c0 = block * kScatterChunks;
    if (c0 >= p.totalTiles) return;
    // 0. each warp fetches its chunk's count (handed to warp 0 through shared memory) and, once it
    //    is known, its first kScatterPre * 32 staged records, which arrive while the block scans;
    //    their LODs are fetched after the barrier
    const uint32_t myChunk = c0 + warp;
    const uint32_t myN = myChunk < p.totalTiles ? __ldcg(p.chunkCount + myChunk) : 0u;
    const uint2* myStage = p.staged + static_cast<size_t>(myChunk) * chunkSize;
    // 1. records before c0, loaded while the count is on its way
    uint32_t part = 0;
    for (uint32_t c = threadIdx.x; c < c0; c += 8u * kScatterWarps * 32u) {
        uint32_t x[8];  // eight loads in flight per thread
#pragma unroll
        for (uint32_t k = 0; k < 8u; ++k) {
            const uint32_t ck = c + k * kScatterWarps * 32u;
            x[k] = ck < c0 ? __ldcg(p.chunkCount + ck) : 0u;
        }
#pragma unroll
        for (uint32_t k = 0; k < 8u; ++k) part += x[k];
    }
    uint2 pre[kScatterPre], preLod[kScatterPre];
#pragma unroll
    for (uint32_t u = 0; u < kScatterPre; ++u) {
        const uint32_t i = lane + 32u * u;
        pre[u] = i < myN ? __ldcg(myStage + i) : make_uint2(0u, 0u);
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) part += __shfl_xor_sync(0xFFFFFFFFu, part, o);
    if (lane == 0) {
        s_part[warp] = part;
        s_n[warp] = myN;
    }
    __syncthreads();
#pragma unroll
    for (uint32_t u = 0; u < kScatterPre; ++u) {
        const uint32_t i = lane + 32u * u;
        preLod[u] = i < myN ? ldp(reinterpret_cast<const uint2*>(p.sc.lods + pre[u].y)) : make_uint2(0u, 0u);
    }
    // 2. warp 0: exclusive offsets of the block's chunks
    if (warp == 0) {
        uint32_t carry = 0;
#pragma unroll
        for (int w = 0; w < kScatterWarps; ++w) carry += s_part[w];
        const uint32_t n = s_n[lane];  // 0 past the last chunk
        uint32_t sum = n;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t ps = __shfl_up_sync(0xFFFFFFFFu, sum, o);
            if (lane >= static_cast<uint32_t>(o)) sum += ps;
        }
        const uint32_t excl = carry + sum - n;
        s_base[lane] = excl;
        if (c0 + lane + 1u == p.totalTiles) {
            *p.single.drawCount = excl + n;
            if (excl + n > p.single.capacity) atomicOr(&p.scratch->status, BLZ_FLAG_COMMAND_OVERFLOW);
        }
    }
    __syncthreads();
    // 3. scatter: each warp its own chunk (kScatterWarps == kScatterChunks)
    static_assert(kScatterWarps == static_cast<int>(kScatterChunks), "one warp per chunk");
    if (myChunk >= p.totalTiles) return;
    const uint32_t base = s_base[warp];
    const BatchViewDev& bv = p.single;
    // staged record i goes to slot base + i, or base + n - 1 - i for a chunk staged last object first
    const bool down = p.descending != 0u;
#pragma unroll
    for (uint32_t u = 0; u < kScatterPre; ++u) {
        const uint32_t i = lane + 32u * u;
        const uint32_t slot = base + (down ? myN - 1u - i : i);
        if (i < myN && slot < bv.capacity) put_record(bv.cmds, bv.stride, slot, pre[u].x, preLod[u].x, preLod[u].y);
    }
    for (uint32_t i = lane + 32u * kScatterPre; i < myN; i += 32) {
        const uint32_t slot = base + (down ? myN - 1u - i : i);
        if (slot >= bv.capacity) {
            if (down) continue;
            break;
        }
        const uint2 rec = __ldcg(myStage + i);
        const uint2 lod = ldp(reinterpret_cast<const uint2*>(p.sc.lods + rec.y));  // indexCount, firstIndex
        put_record(bv.cmds, bv.stride, slot, rec.x, lod.x, lod.y);
    }
}

__global__ void __launch_bounds__(kScatterWarps * 32, 2) cull_scatter_kernel(const PipeParams p) {
    pdl_wait();
    scatter_block(p, blockIdx.x);
}

// A short list in one launch: up to kSmallChunks chunks, one per warp of one cluster. The decide body stages
// the chunk's records in shared memory; the warp hands its count to every block of the cluster (distributed
// shared memory) and, behind the cluster's barrier, knows where its records go and writes them, the draw
// count with them. While the barrier completes it fetches its records' LODs. Bound by that chain of latencies:
// of two launches the second costs a dependent start, a reload of the counts and two block barriers. Replayed
// back to back, 1,000 to 4,096 objects take 3.7 to 4.4 us a call by the pass; two launches took 4.75 to 5.4 (4,097
// objects take that still). Lists of more than a step per warp stay with two launches: a further step costs
// about what the second launch does.
constexpr uint32_t kSmallBlocks = 8;  // the portable cluster size
constexpr uint32_t kSmallChunks = kSmallBlocks * (kObjThreads / 32);
constexpr uint32_t kSmallChunkSize = 32 * kObjOpt;

template <int MODE>
__global__ void __launch_bounds__(kObjThreads) cull_small_kernel(const PipeParams p) {
    constexpr uint32_t NW = kObjThreads / 32;
    __shared__ DecideSmem<MODE, true, kObjThreads, kObjOpt> sm;
    __shared__ uint32_t s_count[kSmallChunks];
    __shared__ uint2 s_stage[NW][kSmallChunkSize];
    // Every block of the cluster is running before the first write to its shared memory (awaited below). The
    // barriers are not of the .aligned form: the second arrive follows a branch that some lanes do not take,
    // and that form wants the warp's lanes together, which nothing here promises.
    asm volatile("barrier.cluster.arrive.relaxed;" ::: "memory");
    pdl_wait();
    const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5, chunk = blockIdx.x * NW + warp;
    const uint32_t n = decide_body<MODE, true, kObjThreads, kObjOpt, true>(p, sm, nullptr, 0u, s_stage[warp]);
    __syncwarp();
    asm volatile("barrier.cluster.wait;" ::: "memory");
    if (lane < gridDim.x) {  // one cluster is the whole grid: lane k writes block k's copy
        const uint32_t mine = static_cast<uint32_t>(__cvta_generic_to_shared(&s_count[chunk]));
        uint32_t theirs;
        asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(theirs) : "r"(mine), "r"(lane));
        asm volatile("st.shared::cluster.u32 [%0], %1;" ::"r"(theirs), "r"(n) : "memory");
    }
    asm volatile("barrier.cluster.arrive.release;" ::: "memory");
    uint2 rec[kObjOpt], lod[kObjOpt];
#pragma unroll
    for (uint32_t u = 0; u < kObjOpt; ++u) {
        const uint32_t i = lane + 32u * u;
        rec[u] = i < n ? s_stage[warp][i] : make_uint2(0u, 0u);
    }
#pragma unroll
    for (uint32_t u = 0; u < kObjOpt; ++u)
        lod[u] = lane + 32u * u < n ? ldp(reinterpret_cast<const uint2*>(p.sc.lods + rec[u].y)) : make_uint2(0u, 0u);
    asm volatile("barrier.cluster.wait.acquire;" ::: "memory");
    uint32_t base = 0, total = 0;
    for (uint32_t c = lane; c < gridDim.x * NW; c += 32u) {
        const uint32_t x = s_count[c];
        total += x;
        if (c < chunk) base += x;
    }
    base = __reduce_add_sync(0xFFFFFFFFu, base);
    const BatchViewDev& bv = p.single;
    // staged record i goes to slot base + i, or base + n - 1 - i for a chunk staged last object first
#pragma unroll
    for (uint32_t u = 0; u < kObjOpt; ++u) {
        const uint32_t i = lane + 32u * u, slot = base + (MODE == BLZ_MODE_LATE ? n - 1u - i : i);
        if (i < n && slot < bv.capacity) put_record(bv.cmds, bv.stride, slot, rec[u].x, lod[u].x, lod[u].y);
    }
    if (chunk == 0u) {
        total = __reduce_add_sync(0xFFFFFFFFu, total);
        if (lane == 0u) {
            *bv.drawCount = total;
            if (total > bv.capacity) atomicOr(&p.scratch->status, BLZ_FLAG_COMMAND_OVERFLOW);
        }
    }
}

// Batched views: two launches. The scan has a block or a warp per view (batch_scan_by_warps): it scans the counts of
// the view's chunks into {offset in the view's records, view} per chunk and writes the view's draw count (block 0
// also rewinds the decide kernel's work counter). The scatter then is one warp per chunk with nothing to wait for. (One launch
// of 1024-thread blocks, each finding its chunks' views and offsets behind two barriers, took 23 to 30 us for
// the 33,000 chunks of the 64-view batch, 3.4 waves of them; the two take 3.6 and 14.)
constexpr uint32_t kBatchScanThreads = 512, kBatchScanEach = 8;
constexpr uint32_t kBatchScatterThreads = 256, kBatchScatterChunks = 4;

__global__ void __launch_bounds__(kBatchScanThreads) batch_scan_kernel(const PipeParams p) {
    constexpr uint32_t NW = kBatchScanThreads / 32u;
    static_assert(NW <= 32u, "a lane per warp");
    __shared__ uint32_t s_warp[kBatchScanEach][NW];
    pdl_wait();
    const uint32_t vi = blockIdx.x, lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
    const uint32_t first = ldp(p.tileStart + vi), end = ldp(p.tileStart + vi + 1u);
    if (vi == 0u && threadIdx.x == 0u && p.workCounter != nullptr) *p.workCounter = 0u;
    uint32_t carry = 0;
    for (uint32_t c0 = first; c0 < end; c0 += kBatchScanThreads * kBatchScanEach) {
        // thread t takes chunks c0 + t, c0 + t + T, ...: their counts loaded together, T of them scanned at a time
        uint32_t n[kBatchScanEach], sum[kBatchScanEach];
#pragma unroll
        for (uint32_t k = 0; k < kBatchScanEach; ++k) {
            const uint32_t c = c0 + k * kBatchScanThreads + threadIdx.x;
            n[k] = c < end ? __ldcg(p.chunkCount + c) : 0u;
        }
#pragma unroll
        for (uint32_t k = 0; k < kBatchScanEach; ++k) {
            sum[k] = n[k];
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const uint32_t x = __shfl_up_sync(0xFFFFFFFFu, sum[k], o);
                if (lane >= static_cast<uint32_t>(o)) sum[k] += x;
            }
            if (lane == 31u) s_warp[k][warp] = sum[k];
        }
        __syncthreads();
        // a warp's total before it, over the parts and warps in order
#pragma unroll
        for (uint32_t k = 0; k < kBatchScanEach; ++k) {
            const uint32_t x = lane < NW ? s_warp[k][lane] : 0u;
            const uint32_t before = __reduce_add_sync(0xFFFFFFFFu, lane < warp ? x : 0u);
            const uint32_t c = c0 + k * kBatchScanThreads + threadIdx.x;
            if (c < end) p.chunkBase[c] = make_uint2(carry + before + sum[k] - n[k], vi);
            carry += __reduce_add_sync(0xFFFFFFFFu, x);
        }
        __syncthreads();
    }
    if (threadIdx.x == 0u) {
        const BatchViewDev& bv = p.views[vi];
        *bv.drawCount = carry;
        if (carry > bv.capacity) atomicOr(&p.scratch->status, BLZ_FLAG_COMMAND_OVERFLOW);
    }
}

constexpr uint32_t kBatchScanWarpThreads = 256, kBatchScanWarpEach = 8;

// The same with a warp per view, 256 chunks a round, for many views or short ones: a chain of three round trips
// and no block barrier.
__global__ void __launch_bounds__(kBatchScanWarpThreads) batch_scan_warp_kernel(const PipeParams p) {
    constexpr uint32_t EACH = kBatchScanWarpEach;
    pdl_wait();
    const uint32_t vi = (blockIdx.x * kBatchScanWarpThreads + threadIdx.x) / 32u, lane = threadIdx.x & 31u;
    if (blockIdx.x == 0u && threadIdx.x == 0u && p.workCounter != nullptr) *p.workCounter = 0u;
    if (vi >= p.viewCount) return;
    const uint32_t first = ldp(p.tileStart + vi), end = ldp(p.tileStart + vi + 1u);
    const BatchViewDev& bv = p.views[vi];
    uint32_t* const drawCount = bv.drawCount;
    const uint32_t capacity = bv.capacity;
    uint32_t carry = 0;
    for (uint32_t c0 = first; c0 < end; c0 += 32u * EACH) {
        uint32_t n[EACH];
#pragma unroll
        for (uint32_t k = 0; k < EACH; ++k) {
            const uint32_t c = c0 + 32u * k + lane;
            n[k] = c < end ? __ldcg(p.chunkCount + c) : 0u;
        }
#pragma unroll
        for (uint32_t k = 0; k < EACH; ++k) {
            const uint32_t c = c0 + 32u * k + lane;
            if (c0 + 32u * k >= end) break;  // (the whole warp)
            uint32_t sum = n[k];
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const uint32_t x = __shfl_up_sync(0xFFFFFFFFu, sum, o);
                if (lane >= static_cast<uint32_t>(o)) sum += x;
            }
            if (c < end) p.chunkBase[c] = make_uint2(carry + sum - n[k], vi);
            carry += __shfl_sync(0xFFFFFFFFu, sum, 31);
        }
    }
    if (lane == 0u) {
        *drawCount = carry;
        if (carry > capacity) atomicOr(&p.scratch->status, BLZ_FLAG_COMMAND_OVERFLOW);
    }
}

__global__ void __launch_bounds__(kBatchScatterThreads) batch_scatter_kernel(const PipeParams p) {
    constexpr uint32_t CH = kBatchScatterChunks;
    pdl_wait();
    const uint32_t lane = threadIdx.x & 31u, c0 = (blockIdx.x * (kBatchScatterThreads / 32u) + (threadIdx.x >> 5)) * CH;
    // lane k < CH holds chunk c0 + k: its count, its records' first slot, its view
    const bool has = lane < CH && c0 + lane < p.totalTiles;
    const uint32_t n = has ? __ldcg(p.chunkCount + c0 + lane) : 0u;
    const uint2 at = has ? __ldcg(p.chunkBase + c0 + lane) : make_uint2(0u, 0u);
    uint32_t start[CH + 1u];  // the warp's records run through its chunks in order
    start[0] = 0u;
#pragma unroll
    for (uint32_t k = 0; k < CH; ++k) start[k + 1u] = start[k] + __shfl_sync(0xFFFFFFFFu, n, static_cast<int>(k));
    const uint32_t total = start[CH];
    for (uint32_t j0 = 0; j0 < total; j0 += 64u) {  // two records a lane, their loads together
        uint2 rec[2], lod[2];
        uint32_t slot[2], vi[2];
#pragma unroll
        for (uint32_t u = 0; u < 2u; ++u) {
            const uint32_t j = j0 + 32u * u + lane;
            uint32_t k = 0, from = 0;
#pragma unroll
            for (uint32_t t = 1; t < CH; ++t)
                if (j >= start[t]) k = t, from = start[t];
            slot[u] = __shfl_sync(0xFFFFFFFFu, at.x, static_cast<int>(k)) + (j - from);
            vi[u] = __shfl_sync(0xFFFFFFFFu, at.y, static_cast<int>(k));
            rec[u] = j < total ? __ldcg(p.staged + static_cast<size_t>(c0 + k) * p.chunkSize + (j - from)) : make_uint2(0u, 0u);
        }
#pragma unroll
        for (uint32_t u = 0; u < 2u; ++u)
            lod[u] = j0 + 32u * u + lane < total ? ldp(reinterpret_cast<const uint2*>(p.sc.lods + rec[u].y)) : make_uint2(0u, 0u);
#pragma unroll
        for (uint32_t u = 0; u < 2u; ++u) {
            if (j0 + 32u * u + lane >= total) continue;
            const BatchViewDev& bv = p.views[vi[u]];
            if (slot[u] < bv.capacity) put_record(bv.cmds, bv.stride, slot[u], rec[u].x, lod[u].x, lod[u].y);
        }
    }
}

constexpr uint32_t kBatchOrderThreads = 64;

// The order in which a batch's chunks are decided: by their place in their view, order[k] = the chunk that
// comes k-th when the middle of chunk r of a view of R chunks counts as (2r + 1) / 2R, and equal ones go by
// view. A render list that follows the scene's order then reads the same transform rows at the same time as
// every other, so the table comes from memory once and not once per view. Exact integers: chunk (v, r) comes
// after the chunks r' of view u with (2r' + 1) R_v < (2r + 1) R_u, or equal and u < v.
__global__ void __launch_bounds__(kBatchOrderThreads) batch_order_kernel(const uint32_t* tileStart, uint32_t viewCount, uint32_t total,
                                                                         uint32_t small, uint32_t* order) {
    __shared__ uint32_t s_start[kBatchOrderViews + 1u];
    pdl_wait();
    for (uint32_t i = threadIdx.x; i <= viewCount; i += kBatchOrderThreads) s_start[i] = ldp(tileStart + i);
    __syncthreads();
    const uint32_t c = blockIdx.x * kBatchOrderThreads + threadIdx.x;
    if (c >= total) return;
    uint32_t v = 0, hi = viewCount;
    while (hi - v > 1u) {
        const uint32_t mid = (v + hi) >> 1;
        if (s_start[mid] <= c) v = mid;
        else hi = mid;
    }
    const uint32_t Rv = s_start[v + 1u] - s_start[v], odd = 2u * (c - s_start[v]) + 1u;
    uint32_t rank = 0;
    if (small) {
        // fewer than 2^15 chunks a view: (2r + 1) R_u stays below 2^31 and its quotient by R_v below 2^16, so the
        // quotient from a float reciprocal is at most one off
        const float inv = 1.0f / static_cast<float>(Rv);
#pragma unroll 4
        for (uint32_t u = 0; u < viewCount; ++u) {
            const uint32_t a = odd * (s_start[u + 1u] - s_start[u]) - (u < v ? 0u : 1u);
            uint32_t m = static_cast<uint32_t>(static_cast<float>(a) * inv);
            const int rest = static_cast<int>(a - m * Rv);
            m = rest < 0 ? m - 1u : (rest >= static_cast<int>(Rv) ? m + 1u : m);
            rank += (m + 1u) >> 1;
        }
    } else {
        for (uint32_t u = 0; u < viewCount; ++u) {
            const uint64_t a = static_cast<uint64_t>(odd) * (s_start[u + 1u] - s_start[u]) - (u < v ? 0u : 1u);
            rank += (static_cast<uint32_t>(a / Rv) + 1u) >> 1;
        }
    }
    order[rank] = c;
}

// Both record lists of a one-call frame in one launch: blocks [0, blocks1) scatter list 1, the rest
// list 2. Block 0 also rewinds the frame kernel's pyramid ticket, tile count and ready flag (the
// frame kernel has finished: this launch follows it on the stream).
__global__ void __launch_bounds__(kScatterWarps * 32, 2) cull_scatter2_kernel(const PipeParams p1, const PipeParams p2,
                                                                           const uint32_t blocks1) {
    pdl_wait();
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        p1.scratch->frameTicket = 0u;
        p1.scratch->frameTilesDone = 0u;
        p1.scratch->frameReady = 0u;
    }
    if (blockIdx.x < blocks1) scatter_block(p1, blockIdx.x);
    else scatter_block(p2, blockIdx.x - blocks1);
}

// ------------------------------------------------------------------ kept frame, pass 2

// Pass 2 of a kept frame (blz_frame_late): one warp per chunk runs the dense stage of pass 2 over
// the survivors pass 1 kept for that chunk, in object order: projectSphere and the Hi-Z test
// (drawOccLate.cs.hlsl:48-58), the visibility rewrite (:67) and the emission of objects not visible
// last frame (:45), staged as (objectId, lodId) for the scatter. Every object pass 1 did not keep was
// outside the frustum and got its visibility in pass 1. A lane takes kLateRounds survivors at once
// (j, j + 32, ...): their loads, tests and LOD selections are independent, so their latencies
// overlap; they are staged in order afterwards.
constexpr uint32_t kLateRounds = 4;

template <int THREADS>
__global__ void __launch_bounds__(THREADS) frame_late_kernel(const PipeParams p) {
    pdl_wait();
    constexpr int NW = THREADS / 32;
    constexpr uint32_t R = kLateRounds;
    const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
    const uint32_t warpsTotal = gridDim.x * NW;
    const BatchViewDev& bv = p.single;
    const ViewConsts v = load_view(bv.view);
    const uint32_t lt = lanemask_lt();
    for (uint32_t chunk = blockIdx.x * NW + warp; chunk < p.totalTiles; chunk += warpsTotal) {
        const uint32_t n = __ldcg(p.keepCount + chunk);
        const uint4* keep = static_cast<const uint4*>(p.keep) + 2u * static_cast<size_t>(chunk) * p.chunkSize;
        uint2* stage = p.staged + static_cast<size_t>(chunk) * p.chunkSize;
        uint32_t run = 0;
        for (uint32_t j0 = 0; j0 < n; j0 += 32u * R) {
            uint4 a[R], b[R];
#pragma unroll
            for (uint32_t r = 0; r < R; ++r) {
                const uint32_t j = j0 + r * 32u + lane;
                a[r] = make_uint4(0u, 0u, 0u, 0u);
                b[r] = a[r];
                if (j < n) {
                    a[r] = __ldcg(keep + 2u * j);
                    b[r] = __ldcg(keep + 2u * j + 1u);
                }
            }
            bool emit[R];
            uint32_t lid[R];
#pragma unroll
            for (uint32_t r = 0; r < R; ++r) {
                const bool mine = j0 + r * 32u + lane < n;
                const uint32_t obj = a[r].x & 0x3FFFFFFFu;
                const Vec3 c{__uint_as_float(a[r].y), __uint_as_float(a[r].z), __uint_as_float(a[r].w)};
                const float rad = __uint_as_float(b[r].x);
                bool visible = mine;
                if (mine) {
                    float4 aabb;
                    if (project_sphere(c, rad, v.zNear, v.proj0, v.proj5, aabb)) visible = occlusion(aabb, bv.pyr, v, c, rad);
                    // drawOccLate.cs.hlsl:67, storing only a value that changes
                    const bool wasNonZero = (a[r].x >> 31) != 0u, wasOne = ((a[r].x >> 30) & 1u) != 0u;
                    if (visible ? !wasOne : wasNonZero) bv.vis[obj] = visible ? 1u : 0u;
                }
                emit[r] = visible && (a[r].x >> 31) == 0u;  // drawOccLate.cs.hlsl:45
                lid[r] = 0u;
                if (emit[r]) {
                    // cullBuffers.hlsl:42-55 — last LOD in [1, lodCount) with error < threshold
                    const float threshold = lod_threshold(c, rad, __uint_as_float(b[r].y), v.lodTarget);
                    uint32_t sel = 0;
                    for (uint32_t t = 1; t < b[r].w; ++t)
                        if (ldp(&p.sc.lods[b[r].z + t].error) < threshold) sel = t;
                    lid[r] = b[r].z + sel;
                }
            }
#pragma unroll
            for (uint32_t r = 0; r < R; ++r) {
                const unsigned e = __ballot_sync(0xFFFFFFFFu, emit[r]);
                if (emit[r]) stage[run + __popc(e & lt)] = make_uint2(a[r].x & 0x3FFFFFFFu, lid[r]);
                run += __popc(e);
            }
        }
        if (lane == 0) p.chunkCount[chunk] = run;
    }
}

// ------------------------------------------------------------------ launchers

// Resident blocks per SM of one instantiation (a property of the kernel, asked once).
template <int MODE, bool SINGLE, int THREADS, int OPT>
static uint32_t occupancy_t() {
    static const uint32_t occ = [] {
        int o = 0;
        if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&o, cull_decide_kernel<MODE, SINGLE, THREADS, OPT>, THREADS, 0) !=
            cudaSuccess) {
            (void)cudaGetLastError();
            o = 1;
        }
        return static_cast<uint32_t>(o < 1 ? 1 : o);
    }();
    return occ;
}

template <int MODE, bool SINGLE, int THREADS, int OPT>
static cudaError_t launch_decide_t(const PipeParams& p, uint32_t blocksPerSm, int smCount, cudaStream_t s) {
    auto kern = cull_decide_kernel<MODE, SINGLE, THREADS, OPT>;
    const uint32_t occ = occupancy_t<MODE, SINGLE, THREADS, OPT>();
    const uint32_t per = blocksPerSm ? (blocksPerSm < occ ? blocksPerSm : occ) : occ;
    uint32_t grid = per * static_cast<uint32_t>(smCount);
    const uint32_t needed = (p.totalTiles + THREADS / 32 - 1) / (THREADS / 32);  // one warp per chunk at most
    if (grid > needed) grid = needed;
    if (grid == 0) grid = 1;
    return launch_pdl(kern, grid, THREADS, 0, s, p);
}

// One scatter block per kScatterChunks chunks.
static uint32_t scatter_blocks(const PipeParams& p) {
    const uint32_t n = (p.totalTiles + kScatterChunks - 1) / kScatterChunks;
    return n ? n : 1u;
}

// Whether a batch's chunks are scanned by a warp per view. Views of one round (256 chunks) always are: 2.0 us against
// 2.9 to 3.9 for up to 256 views, 2.1 against 8.8 for 1,024, 3.3 against 62 for 10,000, since the blocks of the
// other form take 0.9 us for each view an SM gets. With longer views a round costs 1.2 us: 4,096 views of which one has
// 16 rounds take 19.8 us against 27.2, 1,024 such 19.7 against 8.9, 2 views of 16 rounds 20.6 against 3.4.
static bool batch_scan_by_warps(const PipeParams& p, int smCount) {
    const uint64_t rounds = (p.largest + 32u * kBatchScanWarpEach - 1u) / (32u * kBatchScanWarpEach);
    return rounds <= 1u || 4u * rounds * static_cast<uint64_t>(smCount > 0 ? smCount : 1) <= 3u * static_cast<uint64_t>(p.viewCount);
}

template <int MODE, bool SINGLE, int THREADS, int OPT>
static cudaError_t launch_t(const PipeParams& p, uint32_t blocksPerSm, int smCount, cudaStream_t s) {
    cudaError_t e = launch_decide_t<MODE, SINGLE, THREADS, OPT>(p, blocksPerSm, smCount, s);
    if (e != cudaSuccess) return e;
    if constexpr (SINGLE) {
        return launch_pdl(cull_scatter_kernel, scatter_blocks(p), kScatterWarps * 32, 0, s, p);
    } else {
        if (batch_scan_by_warps(p, smCount)) {
            constexpr uint32_t views = kBatchScanWarpThreads / 32u;
            e = launch_pdl(batch_scan_warp_kernel, (p.viewCount + views - 1u) / views, kBatchScanWarpThreads, 0, s, p);
        } else {
            e = launch_pdl(batch_scan_kernel, p.viewCount, kBatchScanThreads, 0, s, p);
        }
        if (e != cudaSuccess) return e;
        constexpr uint32_t per = kBatchScatterThreads / 32u * kBatchScatterChunks;
        return launch_pdl(batch_scatter_kernel, (p.totalTiles + per - 1u) / per, kBatchScatterThreads, 0, s, p);
    }
}

uint32_t object_tile_size() { return kChunk; }

cudaError_t launch_batch_order(const PipeParams& p, uint32_t* order, cudaStream_t s) {
    return launch_pdl(batch_order_kernel, (p.totalTiles + kBatchOrderThreads - 1u) / kBatchOrderThreads, kBatchOrderThreads, 0, s, p.tileStart, p.viewCount, p.totalTiles,
                      p.largest < (1u << 15) ? 1u : 0u, order);
}

template <int THREADS, int OPT>
static cudaError_t launch_frame_first_t(const PipeParams& p, int smCount, cudaStream_t s, bool scatter) {
    cudaError_t e = launch_decide_t<kModeFrame1, true, THREADS, OPT>(p, 0, smCount, s);
    if (e != cudaSuccess || !scatter) return e;
    return launch_pdl(cull_scatter_kernel, scatter_blocks(p), kScatterWarps * 32, 0, s, p);
}

cudaError_t launch_frame_first(const PipeParams& p, uint32_t threads, uint32_t opt, int smCount, cudaStream_t s,
                               bool scatter) {
    PipeParams q = p;
    q.descending = 0u;
    if (threads == 256 && opt == 1) return launch_frame_first_t<256, 1>(q, smCount, s, scatter);
    if (threads == 256 && opt == 4) return launch_frame_first_t<256, 4>(q, smCount, s, scatter);
    if (threads == 128 && opt == 2) return launch_frame_first_t<128, 2>(q, smCount, s, scatter);
    if (threads == 128 && opt == 4) return launch_frame_first_t<128, 4>(q, smCount, s, scatter);
    if (threads == 512 && opt == 1) return launch_frame_first_t<512, 1>(q, smCount, s, scatter);
    return launch_frame_first_t<kObjThreads, kObjOpt>(q, smCount, s, scatter);
}

cudaError_t launch_frame_fused(const PipeParams& p, uint32_t threads, uint32_t opt, int smCount, cudaStream_t s) {
    PipeParams q = p;
    q.descending = 0u;
    if (threads == 256 && opt == 1) return launch_decide_t<kModeFrameFused, true, 256, 1>(q, 0, smCount, s);
    if (threads == 256 && opt == 4) return launch_decide_t<kModeFrameFused, true, 256, 4>(q, 0, smCount, s);
    if (threads == 128 && opt == 2) return launch_decide_t<kModeFrameFused, true, 128, 2>(q, 0, smCount, s);
    if (threads == 128 && opt == 4) return launch_decide_t<kModeFrameFused, true, 128, 4>(q, 0, smCount, s);
    if (threads == 512 && opt == 1) return launch_decide_t<kModeFrameFused, true, 512, 1>(q, 0, smCount, s);
    return launch_decide_t<kModeFrameFused, true, kObjThreads, kObjOpt>(q, 0, smCount, s);
}

template <uint32_t HIZ, int THREADS, int OPT>
static cudaError_t launch_frame_pyr_t(const PipeParams& p, const PyramidBuildParams& bp, int smCount, cudaStream_t s) {
    auto kern = cull_frame_kernel<HIZ, THREADS, OPT>;
    static const uint32_t occ = [&] {
        int o = 0;
        if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&o, kern, THREADS, 0) != cudaSuccess) {
            (void)cudaGetLastError();
            o = 1;
        }
        return static_cast<uint32_t>(o < 1 ? 1 : o);
    }();
    // one warp per chunk at most, but enough blocks (up to one wave) to build the pyramid's tiles
    const uint32_t wave = occ * static_cast<uint32_t>(smCount > 0 ? smCount : 1);
    const uint32_t tiles = ((bp.width + kPyrTile - 1) / kPyrTile) * ((bp.height + kPyrTile - 1) / kPyrTile);
    uint32_t grid = (p.totalTiles + THREADS / 32 - 1) / (THREADS / 32);
    if (grid < tiles) grid = tiles;
    if (grid > wave) grid = wave;
    if (grid == 0) grid = 1;
    return launch_pdl(kern, grid, THREADS, 0, s, p, bp);
}

template <uint32_t HIZ>
static cudaError_t launch_frame_pyr_hiz(const PipeParams& q, const PyramidBuildParams& bp, uint32_t threads, uint32_t opt,
                                        int smCount, cudaStream_t s) {
    if (threads == 256 && opt == 1) return launch_frame_pyr_t<HIZ, 256, 1>(q, bp, smCount, s);
    if (threads == 256 && opt == 4) return launch_frame_pyr_t<HIZ, 256, 4>(q, bp, smCount, s);
    if (threads == 128 && opt == 2) return launch_frame_pyr_t<HIZ, 128, 2>(q, bp, smCount, s);
    if (threads == 128 && opt == 4) return launch_frame_pyr_t<HIZ, 128, 4>(q, bp, smCount, s);
    if (threads == 512 && opt == 1) return launch_frame_pyr_t<HIZ, 512, 1>(q, bp, smCount, s);
    return launch_frame_pyr_t<HIZ, kObjThreads, kObjOpt>(q, bp, smCount, s);
}

cudaError_t launch_frame_pyr(const PipeParams& p, const PyramidBuildParams& bp, uint32_t threads, uint32_t opt, int smCount,
                             cudaStream_t s) {
    PipeParams q = p;
    q.descending = 0u;
    if (bp.mode == BLZ_HIZ_VULKAN) return launch_frame_pyr_hiz<BLZ_HIZ_VULKAN>(q, bp, threads, opt, smCount, s);
    return launch_frame_pyr_hiz<BLZ_HIZ_D3D12>(q, bp, threads, opt, smCount, s);
}

constexpr int kFrameLateThreads = 256;

cudaError_t launch_frame_late(const PipeParams& p, int smCount, cudaStream_t s, bool scatter) {
    static const uint32_t occ = [] {
        int o = 0;
        if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&o, frame_late_kernel<kFrameLateThreads>, kFrameLateThreads, 0) !=
            cudaSuccess) {
            (void)cudaGetLastError();
            o = 1;
        }
        return static_cast<uint32_t>(o < 1 ? 1 : o);
    }();
    constexpr uint32_t NW = kFrameLateThreads / 32;
    uint32_t grid = occ * static_cast<uint32_t>(smCount > 0 ? smCount : 1);
    const uint32_t needed = (p.totalTiles + NW - 1) / NW;
    if (grid > needed) grid = needed;
    if (grid == 0) grid = 1;
    PipeParams q = p;
    q.descending = 0u;
    cudaError_t e = launch_pdl(frame_late_kernel<kFrameLateThreads>, grid, kFrameLateThreads, 0, s, q);
    if (e != cudaSuccess || !scatter) return e;
    return launch_pdl(cull_scatter_kernel, scatter_blocks(q), kScatterWarps * 32, 0, s, q);
}

cudaError_t launch_frame_scatter2(const PipeParams& p1, const PipeParams& p2, cudaStream_t s) {
    const uint32_t g1 = scatter_blocks(p1), g2 = scatter_blocks(p2);
    PipeParams q1 = p1, q2 = p2;
    q1.descending = q2.descending = 0u;
    return launch_pdl(cull_scatter2_kernel, g1 + g2, kScatterWarps * 32, 0, s, q1, q2, g1);
}

template <int MODE>
static uint32_t single_blocks_per_sm(uint32_t threads, uint32_t opt) {
    if (threads == 256 && opt == 1) return occupancy_t<MODE, true, 256, 1>();
    if (threads == 256 && opt == 4) return occupancy_t<MODE, true, 256, 4>();
    if (threads == 128 && opt == 2) return occupancy_t<MODE, true, 128, 2>();
    if (threads == 128 && opt == 4) return occupancy_t<MODE, true, 128, 4>();
    if (threads == 512 && opt == 1) return occupancy_t<MODE, true, 512, 1>();
    return occupancy_t<MODE, true, kObjThreads, kObjOpt>();
}

uint32_t single_chunk_size(uint32_t mode, uint32_t threads, uint32_t opt, uint32_t count, int smCount) {
    if (!single_shape_supported(threads, opt)) {
        threads = kObjThreads;
        opt = kObjOpt;
    }
    uint32_t per = 1;
    switch (mode) {
        case kModeFrame1: per = single_blocks_per_sm<kModeFrame1>(threads, opt); break;
        case kModeFrameFused: per = single_blocks_per_sm<kModeFrameFused>(threads, opt); break;
        case BLZ_MODE_FIRST: per = single_blocks_per_sm<BLZ_MODE_FIRST>(threads, opt); break;
        case BLZ_MODE_LATE: per = single_blocks_per_sm<BLZ_MODE_LATE>(threads, opt); break;
        case BLZ_MODE_TEMPORAL: per = single_blocks_per_sm<BLZ_MODE_TEMPORAL>(threads, opt); break;
        case kModeInstanced: per = single_blocks_per_sm<kModeInstanced>(threads, opt); break;
        default: per = single_blocks_per_sm<BLZ_MODE_FRUSTUM>(threads, opt); break;
    }
    const uint64_t warps = static_cast<uint64_t>(per) * static_cast<uint64_t>(smCount > 0 ? smCount : 1) * (threads / 32u);
    const uint32_t step = 32u * opt;
    uint64_t size = (count + warps - 1) / warps;
    size = (size + step - 1) / step * step;
    return static_cast<uint32_t>(size < step ? step : size);
}

bool single_shape_supported(uint32_t threads, uint32_t opt) {
    return (threads == 256 && (opt == 1 || opt == 2 || opt == 4)) || (threads == 128 && (opt == 2 || opt == 4)) ||
           (threads == 512 && opt == 1);
}

// One launch for the default shape's short lists, where every warp has one step of one chunk and all warps
// fit one cluster: up to 4,096 objects (measured on both sides of the line: cull_small_kernel).
static bool small_list(const PipeParams& p, uint32_t threads, uint32_t opt) {
    return (threads == kObjThreads && opt == kObjOpt) && p.totalTiles <= kSmallChunks && p.chunkSize == kSmallChunkSize;
}

template <int MODE>
static cudaError_t launch_small_t(const PipeParams& p, cudaStream_t s) {
    constexpr uint32_t NW = kObjThreads / 32;
    uint32_t blocks = 1;
    while (blocks * NW < p.totalTiles) blocks *= 2u;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = blocks;
    cfg.blockDim = kObjThreads;
    cfg.stream = s;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    attr[1].id = cudaLaunchAttributeClusterDimension;
    attr[1].val.clusterDim = {blocks, 1, 1};
    cfg.attrs = attr;
    cfg.numAttrs = 2;
    return cudaLaunchKernelEx(&cfg, cull_small_kernel<MODE>, p);
}

template <int MODE>
static cudaError_t launch_single_mode(const PipeParams& p, uint32_t threads, uint32_t opt, int smCount, cudaStream_t s) {
    if (small_list(p, threads, opt)) return launch_small_t<MODE>(p, s);
    if (threads == 256 && opt == 1) return launch_t<MODE, true, 256, 1>(p, 0, smCount, s);
    if (threads == 256 && opt == 4) return launch_t<MODE, true, 256, 4>(p, 0, smCount, s);
    if (threads == 128 && opt == 2) return launch_t<MODE, true, 128, 2>(p, 0, smCount, s);
    if (threads == 128 && opt == 4) return launch_t<MODE, true, 128, 4>(p, 0, smCount, s);
    if (threads == 512 && opt == 1) return launch_t<MODE, true, 512, 1>(p, 0, smCount, s);
    return launch_t<MODE, true, kObjThreads, kObjOpt>(p, 0, smCount, s);
}

cudaError_t launch_object_cull(uint32_t mode, const PipeParams& p, uint32_t threads, uint32_t opt, int smCount,
                               cudaStream_t s, uint32_t* launches) {
    *launches = small_list(p, threads, opt) ? 1u : 2u;  // decide + scatter
    PipeParams q = p;
    q.descending = mode == BLZ_MODE_LATE ? 1u : 0u;  // the single-view pass-2 decide walks its chunks downwards
    switch (mode) {
        case BLZ_MODE_FRUSTUM: return launch_single_mode<BLZ_MODE_FRUSTUM>(q, threads, opt, smCount, s);
        case BLZ_MODE_FIRST: return launch_single_mode<BLZ_MODE_FIRST>(q, threads, opt, smCount, s);
        case BLZ_MODE_LATE: return launch_single_mode<BLZ_MODE_LATE>(q, threads, opt, smCount, s);
        case BLZ_MODE_TEMPORAL: return launch_single_mode<BLZ_MODE_TEMPORAL>(q, threads, opt, smCount, s);
        default: return cudaErrorInvalidValue;
    }
}

// ------------------------------------------------------------------ instanced cull from the staged records
//
// The instanced cull (drawInstCountReset + drawInstCull + drawInstCmd) decides exactly what the
// frustum + LOD pass decides: every visible object and its LOD. So it runs that decide kernel
// (kModeInstanced), whose staged (objectId, lodId) records are in object order per chunk and which
// also counts each group's records per LOD (hist[group][lod], groups of kInstGroup chunks, zeroed
// before the launch), and then two launches:
//   scan   every LOD's counts scanned over the groups, in place: hist[group][lod] becomes the group's
//          offset in the LOD's list; totals[lod] the list's length;
//   place  a block per group: each warp counts its chunks' records per LOD (a row of counts in shared
//          memory), the block scans the rows per LOD, and each warp places its records in order (ranks
//          inside 32-record slices from one ballot per bit of the LOD id). The last group's block writes
//          the counters and, in ascending LOD order, one command per non-empty LOD.
// A row of counts takes 4 bytes a LOD, so scenes of more LODs get fewer warps a block, each with more
// of the group's chunks (inst_warps). All three launches are latency chains of a few block phases; 4M
// objects and 256 LODs: decide 33, scan 3.1, place 9.6 us (11.4 when each place block summed the earlier
// groups' counts itself); 250k objects and 2000 LODs: 6.2, 2.9 and 10.0 us, against 37 us for the one
// launch whose tiles look back over one another's counts of every LOD (cull_instanced.cu).

constexpr uint32_t kInstBatch = 5;  // 32-record slices whose loads are issued together (the first batch's ranks are kept)
constexpr uint32_t kInstMaxPerWarp = 4;  // chunks of a group one warp takes at most
constexpr uint32_t kScanLods = 32, kScanParts = 32, kScanKeep = 8;

__global__ void __launch_bounds__(kScanLods* kScanParts) inst_scan_kernel(uint32_t* hist, uint32_t* totals, uint32_t groups, uint32_t nL) {
    __shared__ uint32_t s_part[kScanParts][kScanLods];
    pdl_wait();
    const uint32_t l = threadIdx.x % kScanLods, part = threadIdx.x / kScanLods, lod = blockIdx.x * kScanLods + l;
    const uint32_t per = (groups + kScanParts - 1u) / kScanParts;
    const uint32_t g0 = min(groups, part * per), g1 = min(groups, g0 + per);
    const bool in = lod < nL;
    // the part's first kScanKeep counts stay in registers, loaded together
    uint32_t keep[kScanKeep], sum = 0;
#pragma unroll
    for (uint32_t k = 0; k < kScanKeep; ++k) {
        keep[k] = in && g0 + k < g1 ? __ldcg(hist + static_cast<size_t>(g0 + k) * nL + lod) : 0u;
    }
#pragma unroll
    for (uint32_t k = 0; k < kScanKeep; ++k) sum += keep[k];
    for (uint32_t g = g0 + kScanKeep; in && g < g1; ++g) sum += __ldcg(hist + static_cast<size_t>(g) * nL + lod);
    s_part[part][l] = sum;
    __syncthreads();
    if (!in) return;
    uint32_t run = 0;
    for (uint32_t q = 0; q < part; ++q) run += s_part[q][l];
    if (part == kScanParts - 1u) totals[lod] = run + sum;
#pragma unroll
    for (uint32_t k = 0; k < kScanKeep; ++k) {
        if (g0 + k < g1) hist[static_cast<size_t>(g0 + k) * nL + lod] = run;
        run += keep[k];
    }
    for (uint32_t g = g0 + kScanKeep; g < g1; ++g) {
        uint32_t* h = hist + static_cast<size_t>(g) * nL + lod;
        const uint32_t c = __ldcg(h);
        *h = run;
        run += c;
    }
}

// Words of a row of per-LOD counts: a multiple of 4, so that the rows are scanned four LODs at a time.
__host__ __device__ __forceinline__ uint32_t inst_stride(uint32_t nL) { return (nL + 3u) & ~3u; }

// Parts the rows are scanned in by T threads, each thread four LODs of one part (0: one, no partial sums).
__host__ __device__ __forceinline__ uint32_t inst_parts(uint32_t nL, uint32_t T) {
    const uint32_t r = T / (inst_stride(nL) / 4u);
    return r >= 8u ? 8u : (r >= 4u ? 4u : (r >= 2u ? 2u : 0u));
}

constexpr uint32_t kInstSmem = 220u * 1024u;

// Warps of a place block for nL LODs: what 220 KB of shared memory hold rows for, a power of two.
static uint32_t inst_warps(uint32_t nL) {
    const uint32_t rows = kInstSmem / 4u / inst_stride(nL);  // W + 2 rows, and the scan's parts
    uint32_t w = kInstGroup;
    while (w > kInstGroup / kInstMaxPerWarp && w + 2u + inst_parts(nL, w * 32u) > rows) w /= 2u;
    return w;
}

__global__ void __launch_bounds__(kInstGroup * 32) inst_place_kernel(const InstStagedParams q) {
    // rows of nS words: [W] per-warp counts, then offsets; the group's offset in each LOD's list; each
    // LOD's instanceOffset; [R] partial sums
    extern __shared__ __align__(16) uint32_t s_rows[];
    __shared__ unsigned int s_flags;
    __shared__ uint32_t s_warpSums[32];
    pdl_wait();
    const uint32_t T = blockDim.x, W = T / 32u, per = kInstGroup / W;
    const uint32_t nL = q.nL, nS = inst_stride(nL), G = q.groups, g = blockIdx.x;
    const uint32_t warp = threadIdx.x >> 5, lane = threadIdx.x & 31u;
    uint32_t* s_goff = s_rows + W * nS;
    uint32_t* s_ioff = s_goff + nS;
    uint32_t* s_part = s_ioff + nS;
    if (threadIdx.x == 0) s_flags = 0u;
    for (uint32_t j = threadIdx.x; j < W * nS / 4u; j += T) reinterpret_cast<uint4*>(s_rows)[j] = make_uint4(0u, 0u, 0u, 0u);
    __syncthreads();
    unsigned int flags = 0u;
    // the warp's records: those of its `per` chunks, one after another
    const uint32_t c0 = g * kInstGroup + warp * per;
    uint32_t first[kInstMaxPerWarp], n = 0;  // record index each chunk starts at
#pragma unroll
    for (uint32_t k = 0; k < kInstMaxPerWarp; ++k) {
        first[k] = n;
        if (k < per && c0 + k < q.totalTiles) n += __ldcg(q.chunkCount + c0 + k);
    }
    auto record = [&](uint32_t j) -> uint2 {
        uint32_t k = 0, from = 0;
#pragma unroll
        for (uint32_t t = 1; t < kInstMaxPerWarp; ++t)
            if (t < per && j >= first[t]) k = t, from = first[t];
        return __ldcg(q.staged + static_cast<size_t>(c0 + k) * q.chunkSize + (j - from));
    };
    auto load_batch = [&](uint32_t j0, uint2 (&r)[kInstBatch]) {
#pragma unroll
        for (uint32_t k = 0; k < kInstBatch; ++k) {
            const uint32_t j = j0 + k * 32u + lane;
            r[k] = j < n ? record(j) : make_uint2(0u, 0xFFFFFFFFu);
        }
    };
    uint2 head[kInstBatch];  // the warp's first kInstBatch * 32 records, loaded once for both walks
    load_batch(0, head);
    const uint32_t idBits = nL > 1u ? 32u - static_cast<uint32_t>(__clz(static_cast<int>(nL - 1u))) : 0u;
    for (uint32_t b = threadIdx.x; b < nL; b += T) {
        s_goff[b] = __ldcg(q.hist + static_cast<size_t>(g) * nL + b);
        s_ioff[b] = __ldcg(&q.counters[b].instanceOffset);
    }
    uint32_t* row = s_rows + warp * nS;
    const uint32_t lt = lanemask_lt();
    // 1. the warp's records per LOD (only this warp touches its row); each of the first batch's
    //    records also keeps its rank among the warp's records of its LOD (the count before its
    //    32-record slice, from the slice's lowest lane of that LOD, plus the lanes below it)
    uint32_t rank[kInstBatch];
    for (uint32_t j0 = 0; j0 < n; j0 += 32u * kInstBatch) {
        uint2 r[kInstBatch];
        if (j0 == 0) {
#pragma unroll
            for (uint32_t k = 0; k < kInstBatch; ++k) r[k] = head[k];
        } else {
            load_batch(j0, r);
        }
#pragma unroll
        for (uint32_t k = 0; k < kInstBatch; ++k) {
            if (j0 + k * 32u >= n) break;  // (the whole warp)
            const uint32_t b = r[k].y;
            const unsigned peers = same_lod_lanes(b, idBits, b != 0xFFFFFFFFu);
            uint32_t before = 0;
            if (b != 0xFFFFFFFFu && (peers & lt) == 0u) {
                before = row[b];
                row[b] = before + __popc(peers);
            }
            if (j0 == 0) {  // warp-uniform
                before = __shfl_sync(0xFFFFFFFFu, before, (__ffs(peers) - 1) & 31);
                rank[k] = before + __popc(peers & lt);
            }
            __syncwarp();
        }
    }
    __syncthreads();
    // 2. per LOD, exclusive offsets of the warps' records: the group's offset and the counts of the warps
    //    before, four LODs a thread; R parts of the rows at a time when there are threads for them, each
    //    starting from the sums of the parts before it
    {
        const uint32_t Q = nS / 4u, R = inst_parts(nL, T);
        auto add = [](uint4& x, const uint4 y) { x.x += y.x, x.y += y.y, x.z += y.z, x.w += y.w; };
        auto at = [&](uint32_t* rows, uint32_t i, uint32_t b) -> uint4& { return reinterpret_cast<uint4*>(rows + i * nS)[b]; };
        auto scan = [&](uint4 run, uint32_t w0, uint32_t w1, uint32_t b) {
            for (uint32_t w = w0; w < w1; w += 4u) {
                uint4 c[4];
#pragma unroll
                for (uint32_t k = 0; k < 4u; ++k) c[k] = w + k < w1 ? at(s_rows, w + k, b) : make_uint4(0u, 0u, 0u, 0u);
#pragma unroll
                for (uint32_t k = 0; k < 4u; ++k) {
                    if (w + k < w1) at(s_rows, w + k, b) = run;
                    add(run, c[k]);
                }
            }
        };
        if (R == 0u) {
            for (uint32_t b = threadIdx.x; b < Q; b += T) scan(at(s_goff, 0, b), 0u, W, b);
        } else {
            const uint32_t b = threadIdx.x % Q, part = threadIdx.x / Q, span = W / R;  // W and R are powers of two, R <= W
            if (part < R) {
                uint4 sum = make_uint4(0u, 0u, 0u, 0u);
                for (uint32_t w = part * span; w < part * span + span; ++w) add(sum, at(s_rows, w, b));
                at(s_part, part, b) = sum;
            }
            __syncthreads();
            if (part < R) {
                uint4 run = at(s_goff, 0, b);
                for (uint32_t k = 0; k < part; ++k) add(run, at(s_part, k, b));
                scan(run, part * span, part * span + span, b);
            }
        }
    }
    __syncthreads();
    // 3. place the records in object order: a warp whose records the first batch holds places each at its
    //    LOD's offset for the warp + its rank; a longer one ranks its records again, slice by slice
    const uint32_t slots = q.slotsPerLod ? q.slotsPerLod : 0xFFFFFFFFu;
    auto put = [&](uint32_t obj, uint32_t b, uint32_t pos) {
        const uint64_t at = static_cast<uint64_t>(s_ioff[b]) + pos;
        if (pos < slots && at < q.instanceCapacity) q.instances[at] = obj;
        else flags |= BLZ_FLAG_INSTANCE_OVERFLOW;
    };
    if (n <= 32u * kInstBatch) {
#pragma unroll
        for (uint32_t k = 0; k < kInstBatch; ++k) {
            const uint32_t b = head[k].y;
            if (b != 0xFFFFFFFFu) put(head[k].x, b, row[b] + rank[k]);
        }
    }
    for (uint32_t j0 = 0; n > 32u * kInstBatch && j0 < n; j0 += 32u * kInstBatch) {
        uint2 r[kInstBatch];
        if (j0 == 0) {
#pragma unroll
            for (uint32_t k = 0; k < kInstBatch; ++k) r[k] = head[k];
        } else {
            load_batch(j0, r);
        }
#pragma unroll
        for (uint32_t k = 0; k < kInstBatch; ++k) {
            if (j0 + k * 32u >= n) break;  // (the whole warp)
            const uint32_t b = r[k].y;
            const unsigned peers = same_lod_lanes(b, idBits, b != 0xFFFFFFFFu);
            uint32_t before = 0;
            if (b != 0xFFFFFFFFu) before = row[b];
            __syncwarp();
            if (b != 0xFFFFFFFFu) {
                if ((peers & lt) == 0u) row[b] = before + __popc(peers);
                put(r[k].x, b, before + __popc(peers & lt));
            }
            __syncwarp();
        }
    }
    // 4. the last group's block: the counters and, in ascending LOD order, one command per non-empty LOD
    //    (drawInstCmd.cs.hlsl:9-38)
    if (g == G - 1u) {
        const uint32_t perT = (nL + T - 1u) / T;
        const uint32_t b0 = min(nL, threadIdx.x * perT), b1 = min(nL, b0 + perT);
        uint32_t mine = 0;
        for (uint32_t l = b0; l < b1; ++l) mine += __ldcg(q.totals + l) ? 1u : 0u;
        uint32_t incl = mine;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t x = __shfl_up_sync(0xFFFFFFFFu, incl, o);
            if (lane >= static_cast<uint32_t>(o)) incl += x;
        }
        if (lane == 31) s_warpSums[warp] = incl;
        __syncthreads();
        uint32_t warpOff = 0, all = 0;
        for (uint32_t w = 0; w < W; ++w) {
            if (w < warp) warpOff += s_warpSums[w];
            all += s_warpSums[w];
        }
        uint32_t out = warpOff + incl - mine;
        for (uint32_t l = b0; l < b1; ++l) {
            const uint32_t total = __ldcg(q.totals + l);
            q.counters[l].instanceCount = total;
            const uint32_t offset = s_ioff[l];
            if (total > slots || static_cast<uint64_t>(offset) + min(total, slots) > q.instanceCapacity)
                flags |= BLZ_FLAG_INSTANCE_OVERFLOW;
            if (total == 0u) continue;
            if (out < q.capacity) {
                uint32_t* w = reinterpret_cast<uint32_t*>(q.cmds + static_cast<size_t>(out) * q.stride);
                const uint2 lod = ldp(reinterpret_cast<const uint2*>(q.lods + l));  // indexCount, firstIndex
                w[0] = offset;
                w[1] = lod.x;
                w[2] = min(total, slots);
                w[3] = lod.y;
                w[4] = 0u;
                w[5] = 0u;
            }
            ++out;
        }
        if (all > q.capacity) flags |= BLZ_FLAG_COMMAND_OVERFLOW;
        if (threadIdx.x == 0) *q.drawCount = all;
    }
    if (flags) atomicOr(&s_flags, flags);
    __syncthreads();
    if (threadIdx.x == 0 && s_flags) atomicOr(q.status, s_flags);
}

__global__ void __launch_bounds__(1024) zero_words_kernel(uint32_t* words, uint32_t n) {
    pdl_wait();
    for (uint32_t i = blockIdx.x * 1024u + threadIdx.x; i < n; i += gridDim.x * 1024u) words[i] = 0u;
}

uint32_t instanced_group_count(uint32_t chunks) { return (chunks + kInstGroup - 1) / kInstGroup; }

cudaError_t launch_instanced_staged(const PipeParams& p, const InstStagedParams& q, uint32_t threads, uint32_t opt,
                                    int smCount, cudaStream_t s) {
    // (a kernel, not a memset: a launch after a memset cannot be a programmatic one)
    const uint32_t words = q.groups * q.nL;
    cudaError_t e = launch_pdl(zero_words_kernel, std::min((words + 1023u) / 1024u, 1024u), 1024, 0, s, p.instHist, words);
    if (e != cudaSuccess) return e;
    if (threads == 256 && opt == 1) e = launch_decide_t<kModeInstanced, true, 256, 1>(p, 0, smCount, s);
    else if (threads == 256 && opt == 4) e = launch_decide_t<kModeInstanced, true, 256, 4>(p, 0, smCount, s);
    else if (threads == 128 && opt == 2) e = launch_decide_t<kModeInstanced, true, 128, 2>(p, 0, smCount, s);
    else if (threads == 128 && opt == 4) e = launch_decide_t<kModeInstanced, true, 128, 4>(p, 0, smCount, s);
    else if (threads == 512 && opt == 1) e = launch_decide_t<kModeInstanced, true, 512, 1>(p, 0, smCount, s);
    else e = launch_decide_t<kModeInstanced, true, kObjThreads, kObjOpt>(p, 0, smCount, s);
    if (e != cudaSuccess) return e;
    e = launch_pdl(inst_scan_kernel, (q.nL + kScanLods - 1) / kScanLods, kScanLods * kScanParts, 0, s, p.instHist, q.totals, q.groups, q.nL);
    if (e != cudaSuccess) return e;
    const uint32_t warps = inst_warps(q.nL), threads32 = warps * 32u;
    const size_t rowBytes = sizeof(uint32_t) * (warps + 2u + inst_parts(q.nL, threads32)) * inst_stride(q.nL);
    if (rowBytes > 48 * 1024) {
        // the limit is the process's, so it is never this call's own size: another thread's launch may be under way with more
        e = cudaFuncSetAttribute(inst_place_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(kInstSmem));
        if (e != cudaSuccess) return e;
    }
    return launch_pdl(inst_place_kernel, q.groups, threads32, rowBytes, s, q);
}

bool batch_shape_supported(uint32_t threads, uint32_t opt) {
    if (!(threads == 128 || threads == 256 || threads == 512)) return false;
    if (!(opt == 1 || opt == 2 || opt == 4 || opt == 8)) return false;
    return threads * opt <= 1024;
}

// A batch whose views all run one pass takes a kernel compiled for that pass: without the other
// passes' code it fits 64 registers, twice the resident warps of the per-view-mode kernel. The default
// shape's two objects per thread do not (79 registers, or spills: 213 and 237 us for the 64-view batch
// against 202), so it runs as 256 x 1 too. That batch took 303 us with the per-view-mode kernel, every view
// reading the 128 MB table from memory for itself; its floor is 45 us of memory traffic, and what is left
// is 185 instructions per 32 objects at half the issue rate.
template <int MODE>
static cudaError_t launch_batch_mode(const PipeParams& p, uint32_t threads, uint32_t blocksPerSm, int smCount,
                                     cudaStream_t s) {
    if (threads == 512) return launch_t<MODE, false, 512, 1>(p, blocksPerSm, smCount, s);
    return launch_t<MODE, false, 256, 1>(p, blocksPerSm, smCount, s);
}

cudaError_t launch_batch_cull(const PipeParams& p, uint32_t threads, uint32_t opt, uint32_t blocksPerSm, int smCount,
                              cudaStream_t s, int mode) {
    if (mode >= 0 && (threads == 256 ? opt <= 2 : threads == 512 && opt == 1)) {
        switch (mode) {
            case BLZ_MODE_FRUSTUM: return launch_batch_mode<BLZ_MODE_FRUSTUM>(p, threads, blocksPerSm, smCount, s);
            case BLZ_MODE_FIRST: return launch_batch_mode<BLZ_MODE_FIRST>(p, threads, blocksPerSm, smCount, s);
            case BLZ_MODE_LATE: return launch_batch_mode<BLZ_MODE_LATE>(p, threads, blocksPerSm, smCount, s);
            case BLZ_MODE_TEMPORAL: return launch_batch_mode<BLZ_MODE_TEMPORAL>(p, threads, blocksPerSm, smCount, s);
            default: break;
        }
    }
#define BLZ_BATCH_CASE(T, O) \
    if (threads == T && opt == O) return launch_t<kModeRuntime, false, T, O>(p, blocksPerSm, smCount, s);
    BLZ_BATCH_CASE(128, 1) BLZ_BATCH_CASE(128, 2) BLZ_BATCH_CASE(128, 4) BLZ_BATCH_CASE(128, 8)
    BLZ_BATCH_CASE(256, 1) BLZ_BATCH_CASE(256, 2) BLZ_BATCH_CASE(256, 4)
    BLZ_BATCH_CASE(512, 1) BLZ_BATCH_CASE(512, 2)
#undef BLZ_BATCH_CASE
    return cudaErrorInvalidValue;
}

// Asking for a kernel's attributes loads it.
template <typename K>
static cudaError_t load_kernel(K* kernel) {
    cudaFuncAttributes a;
    return cudaFuncGetAttributes(&a, reinterpret_cast<const void*>(kernel));
}

cudaError_t load_batch_kernels(uint32_t threads, uint32_t opt) {
    cudaError_t e = cudaSuccess;
    auto load = [&](auto* kernel) {
        if (e == cudaSuccess) e = load_kernel(kernel);
    };
    load(batch_order_kernel);
    load(batch_scan_kernel);
    load(batch_scan_warp_kernel);
    load(batch_scatter_kernel);
    if (threads == 256 && opt <= 2) {
        load(cull_decide_kernel<BLZ_MODE_FRUSTUM, false, 256, 1>);
        load(cull_decide_kernel<BLZ_MODE_TEMPORAL, false, 256, 1>);
    } else if (threads == 512 && opt == 1) {
        load(cull_decide_kernel<BLZ_MODE_FRUSTUM, false, 512, 1>);
        load(cull_decide_kernel<BLZ_MODE_TEMPORAL, false, 512, 1>);
    }
#define BLZ_BATCH_CASE(T, O) \
    if (threads == T && opt == O) load(cull_decide_kernel<kModeRuntime, false, T, O>);
    BLZ_BATCH_CASE(128, 1) BLZ_BATCH_CASE(128, 2) BLZ_BATCH_CASE(128, 4) BLZ_BATCH_CASE(128, 8)
    BLZ_BATCH_CASE(256, 1) BLZ_BATCH_CASE(256, 2) BLZ_BATCH_CASE(256, 4)
    BLZ_BATCH_CASE(512, 1) BLZ_BATCH_CASE(512, 2)
#undef BLZ_BATCH_CASE
    return e;
}

}  // namespace blz
