// binning.cu -- bin and coarse stages (stages 2 and 3 of 4): the tile lists.
//
// The reference bins with 16 persistent CTAs writing segmented linked lists
// per (bin, stream), merges the 16 streams per bin in triangle order
// (BinRaster.inl:19-469) and rasterizes each bin's list into per-tile lists
// (CoarseRaster.inl:28-809). On GB300 the tile lists are built directly, with
// one device-wide atomic counter per tile (they live in L2, 4 bytes a tile):
//
//   pairs:   records the (tile, triangle) pairs of the subtriangles in at most
//            2x2 tiles, each with its place in the tile's list, and counts
//            their bins; queues the others as items.
//   items:   records the pairs of the items and counts their tiles and bins.
//   scan:    allocates each tile's list from the counts.
//   scatter: writes the recorded pairs at their places, those of the items
//            behind the others.
//   rest:    expands the items whose pairs found no room again (in queued and
//            captured draws that may have such; a blocking one makes room and
//            reruns).
//   sort:    puts the lists of order-dependent pipes in submission order.
//
// The counters' atomics give a list's entries in no particular order. Pipes
// whose fine stage resolves visibility by keys (fine.cuh) do not depend on it;
// for the others the lists are sorted. A count -> scan -> scatter pass per
// level, bins then tiles, with every list in order (the design before) took
// for its six kernels, against these, in us: 101 / 67 on 1M small triangles at
// 1080p, 309 / 180 on an 8.4M-triangle 4x MSAA heightfield at 4K, 276 / 81 on
// 20,000 triangles of 60 pixels, 85 / 56 with the sort (11) on 300k blended
// ones.
//
// None of these kernels lets its dependent launch early (launch.h): CTAs that
// wait for it would hold slots that its own need (32-scene batch 1010 us with,
// 959 without).
//
// List entries are triangle << 3 | subtriangle (7 = the triangle's own slot),
// as in the reference. Which cells an entry goes to: its box's cells, and of
// a box larger than 2x2 cells those that the triangle may touch
// (triTouchesCell) -- for tiles, the box within each bin counts, and the bin
// must hold the entry too.
#include "cudaraster/detail/binning.cuh"
#include "cudaraster/detail/launch.h"
#include "cudaraster/detail/list_alloc.h"
#include "cudaraster/detail/per_device.h"

#include <algorithm>

namespace cr {

constexpr int kListThreads = 256;
constexpr int kListWarps = kListThreads / 32;

// Warp-level inclusive scan (of the first N lanes).
template <class T, int N = 32>
__device__ __forceinline__ T warpInclusiveScan(T v) {
    const int lane = threadIdx.x & 31;
#pragma unroll
    for (int o = 1; o < N; o <<= 1) {
        T t = __shfl_up_sync(0xFFFFFFFFu, v, o);
        if (lane >= o) v += t;
    }
    return v;
}

// A warp's 64-bit total, in 16-bit digits (the warp-wide addition takes 32 bits).
__device__ __forceinline__ U64 warpTotal(U64 v) {
    const U32 lo = __reduce_add_sync(0xFFFFFFFFu, (U32)v & 0xFFFFu), mid = __reduce_add_sync(0xFFFFFFFFu, (U32)(v >> 16) & 0xFFFFu);
    const U32 hi = __reduce_add_sync(0xFFFFFFFFu, (U32)(v >> 32));
    return ((U64)hi << 32) + ((U64)mid << 16) + lo;
}

// Queues list entry `entry` as a large or huge item.
__device__ __forceinline__ void queueLarge(const DrawDev& d, U32 entry, bool huge) {
    const S32 k = atomicAdd(&d.counters->largeItems[huge ? 1 : 0], 1);
    d.largeItems[huge ? d.maxSubtris - 1 - k : (S64)k] = entry;
}

// Up to 32 items (subtriangles) of a warp, one word per lane, to be expanded
// into (item, cell) pairs dealt evenly over the lanes.
struct ItemSmem {
    S32 incl[32];   // inclusive prefix of the items' cell counts
    U32 v[3][32];   // vertices, packed as in the triangle header
    U32 box[32];    // tile box: lx | ly << 9 | (w - 1) << 18
    U32 ext[32];    // h - 1 | (bin box of at most 2x2 bins) << 9 | first cell of the slice << 10
    U32 mul[32];    // ceil(2^32 / w) (0 for w = 1): cell k of the box is in row umulhi(k, mul)
    S32 tile0[32];  // global tile of the box's first tile
    S32 wt[32];     // tiles per row of the viewport
    S32 inst[32];
    S32 F[3][32], dx[3][32], dy[3][32];   // tile edges
};

// Edge k of a triangle over the viewport's tiles: tile (cx, cy) may be touched
// iff F + dx * cy - dy * cx >= 0 for all three. This is edgeTouchesRect on the
// tile's rectangle, whose value E + 128 (dx * cy - dy * cx) is not negative
// iff floor(E / 128) + dx * cy - dy * cx is not; |F| stays below 2^27 and the
// products below 2^26, so 32 bits hold it (20,000 triangles of 60 pixels: 57 us
// for this kernel with the 64-bit test per pair, 43 so).
__device__ __forceinline__ void tileEdge(S32 ox, S32 oy, S32 dx, S32 dy, S32 halfW, S32 halfH, S32& F) {
    const S32 side = 1 << (kTileLog2 + kSubpixelLog2);
    const S32 px = (dy > 0 ? 0 : side - 1) - halfW, py = (dx > 0 ? side - 1 : 0) - halfH;
    F = (S32)(((S64)(ox - px) * dy - (S64)(oy - py) * dx) >> (kTileLog2 + kSubpixelLog2));
}

__device__ __forceinline__ void stageItem(ItemSmem& sm, int lane, uint4 h, const TriGeom& g, const CellBox& b,
                                          bool binsSmall, U32 cell0, S32 inst, const InstanceDev* in) {
    const U32 w = (U32)(b.hx - b.lx + 1);
    sm.v[0][lane] = h.x;
    sm.v[1][lane] = h.y;
    sm.v[2][lane] = h.z;
    sm.box[lane] = (U32)b.lx | (U32)b.ly << 9 | (w - 1u) << 18;
    sm.ext[lane] = (U32)(b.hy - b.ly) | (binsSmall ? 1u << 9 : 0u) | cell0 << 10;
    sm.mul[lane] = w > 1u ? 0xFFFFFFFFu / w + 1u : 0u;
    const S32 wt = __ldg(&in->widthTiles);
    sm.tile0[lane] = __ldg(&in->tileBase) + b.ly * wt + b.lx;
    sm.wt[lane] = wt;
    sm.inst[lane] = inst;
    const S32 halfW = __ldg(&in->width) << (kSubpixelLog2 - 1), halfH = __ldg(&in->height) << (kSubpixelLog2 - 1);
    const S32 ox[3] = {g.x0, g.x1, g.x2}, oy[3] = {g.y0, g.y1, g.y2};
#pragma unroll
    for (int k = 0; k < 3; k++) {
        const int n = k == 2 ? 0 : k + 1;
        const S32 dx = ox[n] - ox[k], dy = oy[n] - oy[k];
        sm.dx[k][lane] = dx;
        sm.dy[k][lane] = dy;
        S32 F;
        tileEdge(ox[k], oy[k], dx, dy, halfW, halfH, F);
        sm.F[k][lane] = F;
    }
}

// Pair p of the `items` staged items (p below their pair count): its item j
// and global tile; returns whether the tile's list takes the entry. The
// quotient k / w = umulhi(k, ceil(2^32 / w)) is exact for k * w < 2^32 (boxes
// have at most 512 x 512 tiles).
__device__ __forceinline__ bool pairTile(const DrawDev& d, const ItemSmem& sm, S32 items, S32 p, int& j, S32& tile) {
    int jj = 0;
    if (items > 1) {
#pragma unroll
        for (int s = 16; s > 0; s >>= 1)
            if (sm.incl[jj + s - 1] <= p) jj += s;
    }
    const U32 box = sm.box[jj], ext = sm.ext[jj], mul = sm.mul[jj];
    const U32 k = (U32)(p - (jj ? sm.incl[jj - 1] : 0)) + (ext >> 10);
    const S32 w = (S32)(box >> 18) + 1;
    const S32 q = (S32)(mul ? __umulhi(k, mul) : k);
    const S32 r = (S32)k - q * w;
    const S32 lx = (S32)(box & 0x1FFu), ly = (S32)((box >> 9) & 0x1FFu);
    const S32 hx = lx + w - 1, hy = ly + (S32)(ext & 0x1FFu);
    const S32 cx = lx + r, cy = ly + q;
    j = jj;
    tile = sm.tile0[jj] + q * sm.wt[jj] + r;
    // The box within the tile's bin; of at most 2x2 tiles, all its tiles take
    // the entry if the bin does. A tile that the triangle may touch lies in a
    // bin that it may touch.
    const S32 side = 1 << d.binLog2;
    const S32 bx0 = cx & -side, by0 = cy & -side;
    const bool few = min(hx, bx0 + side - 1) - max(lx, bx0) <= 1 && min(hy, by0 + side - 1) - max(ly, by0) <= 1;
    if (!few) {
        const S32 e0 = sm.F[0][jj] + sm.dx[0][jj] * cy - sm.dy[0][jj] * cx;
        const S32 e1 = sm.F[1][jj] + sm.dx[1][jj] * cy - sm.dy[1][jj] * cx;
        const S32 e2 = sm.F[2][jj] + sm.dx[2][jj] * cy - sm.dy[2][jj] * cx;
        return (e0 | e1 | e2) >= 0;
    }
    if (ext >> 9 & 1u) return true;
    const InstanceDev* in = &d.inst[sm.inst[jj]];
    return triTouchesCell(geomFromHeader(make_uint4(sm.v[0][jj], sm.v[1][jj], sm.v[2][jj], 0u)), cx >> d.binLog2,
                          cy >> d.binLog2, d.binLog2, __ldg(&in->width), __ldg(&in->height));
}

__device__ __forceinline__ CellBox headerBox(const TriGeom& g, const InstanceDev* in) {
    return tileBox(min3i(g.x0, g.x1, g.x2), min3i(g.y0, g.y1, g.y2), max3i(g.x0, g.x1, g.x2), max3i(g.y0, g.y1, g.y2),
                   __ldg(&in->width), __ldg(&in->height), __ldg(&in->widthTiles), __ldg(&in->heightTiles),
                   __ldg(&in->samplesLog2) == 0);
}

// Instance of a triangle slot (no search for a single scene).
__device__ __forceinline__ int instanceOf(const DrawDev& d, U32 tri) {
    return d.numInstances == 1 ? 0 : findInstance64(d.triPrefix, d.numInstances, (S64)tri);
}

// ----------------------------------------------------------------- pairs
//
// A warp takes a chunk of triangles: its live subtriangles stream through a
// ring in shared memory 32 at a time, their (tile, triangle) pairs through a
// second one, so that both steps work with all lanes however many triangles
// setup culled and however many tiles each covers.

constexpr int kRing = 256;
constexpr int kSharedBins = 2048;

struct PairSmem {
    U64 pairs[kRing];    // global tile << 10 | triangle of the chunk
    U32 live[kRing];     // list entries
    U32 medium[64];      // medium items not yet queued
};

// The grid that a triangle's boxes are formed on.
struct SceneGrid {
    S32 width, height, widthTiles, heightTiles, widthBins, tileBase, binBase;
    bool centerOnly;
};
__device__ __forceinline__ SceneGrid loadGrid(const InstanceDev* in) {
    return SceneGrid{__ldg(&in->width),     __ldg(&in->height),   __ldg(&in->widthTiles), __ldg(&in->heightTiles),
                     __ldg(&in->widthBins), __ldg(&in->tileBase), __ldg(&in->binBase),    __ldg(&in->samplesLog2) == 0};
}

// Appends the list entries of triangles [next, next + 128) below end to the
// ring (which holds fewer than 32): lane l takes triangles 4 l to 4 l + 3
// (chunks start at multiples of four; the buffer is padded to whole words).
// `ahead` holds their counts, loaded since the last call, and then the next
// 128's.
__device__ __forceinline__ U32 loadCounts(const DrawDev& d, S64 first, S64 end) {
    U32 counts = first < end ? __ldg((const U32*)(d.triSubtris + first)) : 0u;
    if (first + 4 > end && first < end) counts &= (1u << (8 * (U32)(end - first))) - 1u;
    return counts;
}
__device__ __forceinline__ void refillRing(const DrawDev& d, S64 next, S64 end, U32& ahead, U32* ring, S32 head,
                                           S32& fill) {
    const int lane = threadIdx.x & 31;
    const U32 ltMask = (1u << lane) - 1u;
    const S64 first = next + 4 * lane;
    U32 counts = ahead;
    ahead = loadCounts(d, first + 128, end);
    if (__any_sync(0xFFFFFFFFu, counts & 0xFEFEFEFEu)) {
        // Clipped triangles with several subtriangles (rare): straight to
        // the large items, which have room for every subtriangle.
        for (int j = 0; j < 4; j++) {
            const U32 n = counts >> (8 * j) & 0xFFu;
            if (n < 2u) continue;
            for (U32 s = 0; s < n; s++) {
                const U32 e = (U32)(first + j) << 3 | s;
                const TriGeom g = geomFromHeader(__ldg(&d.triHeader[entrySlot(e, d.triHeader)]));
                queueLarge(d, e, headerBox(g, &d.inst[instanceOf(d, e >> 3)]).count() > kHugeCells);
            }
            counts &= ~(0xFFu << (8 * j));
        }
        __syncwarp();
    }
#pragma unroll
    for (int j = 0; j < 4; j++) {
        const bool live = counts >> (8 * j) & 1u;
        const U32 mask = __ballot_sync(0xFFFFFFFFu, live);
        if (live) ring[(head + fill + __popc(mask & ltMask)) & (kRing - 1)] = (U32)(first + j) << 3 | 7u;
        fill += __popc(mask);
    }
    __syncwarp();
}

// 32 pairs (or the chunk's last ones) between the update of their tiles'
// counters and the write of their records.
struct PairBatch {
    U64 pair;
    S32 first;     // in the head lanes of the runs of pairs on one tile: the counter before the run
    U32 heads;
    S32 n, at;     // pairs, index of the first one in the chunk
};

// Neighbouring triangles of a mesh mostly share their tile: a run of pairs on
// one tile moves its counter once.
__device__ __forceinline__ PairBatch countPairs(const DrawDev& d, const U64* ring, S32 head, S32 n, S32 at) {
    const int lane = threadIdx.x & 31;
    const U32 ltMask = (1u << lane) - 1u;
    PairBatch b;
    b.pair = lane < n ? ring[(head + lane) & (kRing - 1)] : 0ull;
    const U32 tile = (U32)(b.pair >> 10);
    const U32 before = __shfl_up_sync(0xFFFFFFFFu, tile, 1);
    const bool first = lane < n && (lane == 0 || before != tile);
    b.heads = __ballot_sync(0xFFFFFFFFu, first);
    b.first = 0;
    if (first) {
        const U32 later = b.heads & ~(ltMask | 1u << lane);
        b.first = atomicAdd(d.tileWork + ((S64)tile << d.tileWorkLog2), (later ? __ffs(later) - 1 : n) - lane);
    }
    b.n = n;
    b.at = at;
    return b;
}

__device__ __forceinline__ void writePairs(U64* pairs, const PairBatch& b) {
    const int lane = threadIdx.x & 31;
    const U32 upTo = b.heads & ((2u << lane) - 1u);
    const int head = upTo ? 31 - __clz(upTo) : 0;
    const S32 place = __shfl_sync(0xFFFFFFFFu, b.first, head) + lane - head;
    if (lane < b.n) pairs[b.at + lane] = (U64)(U32)place << 37 | b.pair;
}

// Moves up to 32 of the warp's medium items to the queue.
__device__ __forceinline__ void flushMedium(const DrawDev& d, const U32* medium, S32& fill) {
    const int lane = threadIdx.x & 31;
    const S32 n = min(fill, 32);
    S32 base = 0;
    if (lane == 0) base = atomicAdd(&d.counters->mediumItems, n);
    base = __shfl_sync(0xFFFFFFFFu, base, 0);
    if (lane < n) d.mediumItems[base + lane] = medium[fill - n + lane];
    fill -= n;
    __syncwarp();
}

// Persistent warps over chunks, taken in order as warps free up. Bound by
// latency (flags, headers and counters are three trips to L2 or beyond): a
// group's headers load while the one before it is worked on, a batch's records
// are written after the next one's counters have been issued.
__global__ void __launch_bounds__(kListThreads) pairKernel(const __grid_constant__ DrawDev d) {
    pdlWait();
    markStage(d.stageTiming, d.counters, 1);
    __shared__ PairSmem s_pair[kListWarps];
    __shared__ S32 s_bins[kSharedBins];
    if (__ldcg(&d.counters->overflow) & kOverflowSubtris) return;
    // Bins are counted in shared memory and handed over at the end, where the
    // draw's fit.
    const bool sharedBins = d.totalBins <= kSharedBins;
    if (sharedBins) {
        for (int b = threadIdx.x; b < d.totalBins; b += kListThreads) s_bins[b] = 0;
        __syncthreads();
    }
    auto countBin = [&](S32 b) {
        if (sharedBins) atomicAdd(&s_bins[b], 1); else atomicAdd(&d.binWork[b * kBinWorkStride], 1);
    };
    PairSmem& sm = s_pair[threadIdx.x >> 5];
    const int lane = threadIdx.x & 31;
    const U32 ltMask = (1u << lane) - 1u;
    const bool recordable = d.totalTiles <= kMaxRecord && d.totalTris <= kMaxRecord;
    S32 mediumFill = 0;
    // A warp's first chunk is its own, the others come from a counter (one
    // address passes 1.4 atomics per ns: 5,000 warps asking at once wait 3.5 us).
    const S32 warps = gridDim.x * kListWarps;
    S32 chunk = blockIdx.x * kListWarps + (threadIdx.x >> 5);
    while (chunk < d.numChunks) {
        S32 nextChunk = 0;   // taken now, needed at the end
        if (lane == 0 && d.numChunks > warps) nextChunk = atomicAdd(&d.counters->chunkWork, 1);
        const S64 t0 = (S64)chunk * d.chunkTris, end = min(t0 + d.chunkTris, d.totalTris);
        U64* out = d.pairs + (S64)chunk * 2 * d.chunkTris;
        // Mostly all of a chunk's triangles belong to one scene.
        const int inst0 = instanceOf(d, (U32)t0);
        const bool oneScene = inst0 == instanceOf(d, (U32)end - 1u);
        SceneGrid grid = loadGrid(&d.inst[inst0]);
        S64 next = t0;
        U32 ahead = loadCounts(d, next + 4 * lane, end);
        S32 head = 0, fill = 0;                   // live subtriangles in the ring
        S32 pairHead = 0, pairFill = 0, done = 0; // pairs in their ring, pairs taken from it
        PairBatch prev{};
        U32 entry = 0;
        uint4 h = make_uint4(0u, 0u, 0u, 0u);
        auto fetch = [&]() {   // the next group's size, its entries and headers
            while (fill < 32 && next < end) {
                refillRing(d, next, end, ahead, sm.live, head, fill);
                next += 128;
            }
            const int g = min(fill, 32);
            if (lane < g) {
                entry = sm.live[(head + lane) & (kRing - 1)];
                h = __ldg(&d.triHeader[entry >> 3]);
            }
            __syncwarp();
            head += g;
            fill -= g;
            return g;
        };
        int g = fetch();
        while (g > 0) {
            const U32 e = entry;
            const TriGeom tg = geomFromHeader(h);
            const bool valid = lane < g;
            g = fetch();
            if (!oneScene && valid) grid = loadGrid(&d.inst[instanceOf(d, e >> 3)]);
            const CellBox t = tileBox(min3i(tg.x0, tg.x1, tg.x2), min3i(tg.y0, tg.y1, tg.y2), max3i(tg.x0, tg.x1, tg.x2),
                                      max3i(tg.y0, tg.y1, tg.y2), grid.width, grid.height, grid.widthTiles,
                                      grid.heightTiles, grid.centerOnly);
            const CellBox b = t.coarser(d.binLog2);
            const bool live = valid && !b.empty();
            bool small = live && t.small() && recordable;
            bool one = small && !t.empty();
            U32 m0 = __ballot_sync(0xFFFFFFFFu, one);
            U32 mR = __ballot_sync(0xFFFFFFFFu, one && t.hx > t.lx), mD = __ballot_sync(0xFFFFFFFFu, one && t.hy > t.ly);
            S32 nR = __popc(m0), nD = nR + __popc(mR), nB = nD + __popc(mD), total = nB + __popc(mR & mD);
            if (done + pairFill + total > 2 * d.chunkTris) {
                // The chunk's room is used up (rare): the group is queued.
                small = one = false;
                m0 = mR = mD = 0u;
                total = 0;
            }
            const U64 pair = (U64)(U32)(grid.tileBase + t.ly * grid.widthTiles + t.lx) << 10 | (U64)((e >> 3) - (U32)t0);
            const S32 tail = pairHead + pairFill;
            if (one) sm.pairs[(tail + __popc(m0 & ltMask)) & (kRing - 1)] = pair;
            if (mR >> lane & 1u) sm.pairs[(tail + nR + __popc(mR & ltMask)) & (kRing - 1)] = pair + (1u << 10);
            if (mD) {
                const U64 below = pair + ((U64)(U32)grid.widthTiles << 10);
                if (mD >> lane & 1u) sm.pairs[(tail + nD + __popc(mD & ltMask)) & (kRing - 1)] = below;
                const U32 mB = mR & mD;
                if (mB >> lane & 1u) sm.pairs[(tail + nB + __popc(mB & ltMask)) & (kRing - 1)] = below + (1u << 10);
            }
            pairFill += total;
            if (small) {
                const S32 bin = grid.binBase + b.ly * grid.widthBins + b.lx;
                countBin(bin);
                if (b.hx > b.lx || b.hy > b.ly) {
                    if (b.hx > b.lx) countBin(bin + 1);
                    if (b.hy > b.ly) {
                        countBin(bin + grid.widthBins);
                        if (b.hx > b.lx) countBin(bin + grid.widthBins + 1);
                    }
                }
            }
            const bool queued = live && !small;
            if (__any_sync(0xFFFFFFFFu, queued)) {
                const S32 cells = t.count();
                const U32 mm = __ballot_sync(0xFFFFFFFFu, queued && cells <= kMediumCells);
                if (mm >> lane & 1u) sm.medium[mediumFill + __popc(mm & ltMask)] = e;
                mediumFill += __popc(mm);
                if (queued && cells > kMediumCells) queueLarge(d, e, cells > kHugeCells);
            }
            __syncwarp();
            if (mediumFill >= 32) flushMedium(d, sm.medium, mediumFill);
            while (pairFill >= 32 || (g == 0 && pairFill > 0)) {
                const S32 n = min(pairFill, 32);
                const PairBatch cur = countPairs(d, sm.pairs, pairHead, n, done);
                pairHead += n;
                pairFill -= n;
                done += n;
                writePairs(out, prev);
                prev = cur;
            }
            __syncwarp();
        }
        writePairs(out, prev);
        if (lane == 0) d.pairCount[chunk] = done;
        chunk = warps + __shfl_sync(0xFFFFFFFFu, nextChunk, 0);
    }
    if (mediumFill > 0) flushMedium(d, sm.medium, mediumFill);
    if (sharedBins) {
        __syncthreads();
        for (int b = threadIdx.x; b < d.totalBins; b += kListThreads) {
            const S32 v = s_bins[b];
            if (v) atomicAdd(&d.binWork[b * kBinWorkStride], v);
        }
    }
}

// ----------------------------------------------------------------- items
//
// A warp takes a unit of items -- a slice of one huge item's box, one large
// item, or a group of medium ones -- and expands it into (item, cell) pairs
// dealt evenly over the lanes, so lanes stay busy however uneven the boxes
// are. The units with the most pairs come first.

struct ItemUnits {
    S32 hugeSlices, hugeUnits;     // units per huge item, their units
    S32 largeSlices, largeUnits;   // likewise of the large items
    S32 medium, group;             // medium items, items per unit
    S32 total;
};

// Splits the items over `warps` warps: huge items in up to 64 slices that
// give about eight units a warp, large ones in up to 2 and medium ones in
// groups of 4 to 32 that give about one. In us of the bin stage, over 20,000
// triangles of 60 pixels, 300k blended ones, 5,000 blended of 90 pixels, 5,000
// of 6 and the 32-scene batch: 58.8, 29.2, 33.7, 17.8, 126; up to 16 slices:
// 49.6, 28.5, 37.1, 17.8, 125; large ones whole: 57.9, 32.3, 35.6, 17.8, 124, in
// up to 8: 58.5, 32.9, 36.9, 17.8, 126; groups from 1: 60.7, 29.1, 33.3, 16.8,
// 126, from 16: 58.3, 27.5, 36.4, 20.1, 126, up to 8: 59.3, 29.0, 33.5, 17.8, 135.
__device__ __forceinline__ ItemUnits planItems(const DrawDev& d, S32 warps) {
    ItemUnits u;
    const S32 large = __ldcg(&d.counters->largeItems[0]), huge = __ldcg(&d.counters->largeItems[1]);
    u.medium = __ldcg(&d.counters->mediumItems);
    u.hugeSlices = min(max(8 * warps / max(huge, 1), 1), 64);
    u.largeSlices = min(max(2 * warps / max(large, 1), 1), 2);
    u.hugeUnits = huge * u.hugeSlices;
    u.largeUnits = large * u.largeSlices;
    u.group = min(max(u.medium / warps, 4), 32);
    u.total = u.hugeUnits + u.largeUnits + (u.medium + u.group - 1) / u.group;
    return u;
}

// Stages up to 32 items in shared memory: lane l < items has list entry
// `entry`, of whose box it takes slice `slice` of `slices`; with kBins counts
// their bins (a sliced item's with its first slice). Returns the number of
// (item, cell) pairs.
template <bool kBins>
__device__ __forceinline__ S32 stageItems(const DrawDev& d, S32 items, U32 entry, S32 slice, S32 slices, ItemSmem& sm) {
    const int lane = threadIdx.x & 31;
    S32 n = 0, bins = 0;
    if (lane < items) {
        const uint4 h = __ldg(&d.triHeader[entrySlot(entry, d.triHeader)]);
        const int ii = instanceOf(d, entry >> 3);
        const InstanceDev* in = &d.inst[ii];
        const TriGeom g = geomFromHeader(h);
        const CellBox b = headerBox(g, in), bb = b.coarser(d.binLog2);
        n = b.count();
        U32 c0 = 0;
        if (slices > 1) {   // at most 2^18 cells times 64 slices
            c0 = (U32)n * (U32)slice / (U32)slices;
            n = (S32)((U32)n * (U32)(slice + 1) / (U32)slices - c0);
        }
        stageItem(sm, lane, h, g, b, bb.small(), c0, ii, in);   // (an item without cells is never looked up)
        if (kBins && slice == 0) {
            bins = bb.count();
            if (bins <= 4) {
                const bool test = !bb.small();
                const S32 wb = __ldg(&in->widthBins);
                for (S32 by = bb.ly; by <= bb.hy; by++)
                    for (S32 bx = bb.lx; bx <= bb.hx; bx++)
                        if (!test || triTouchesCell(g, bx, by, d.binLog2, __ldg(&in->width), __ldg(&in->height)))
                            atomicAdd(&d.binWork[(__ldg(&in->binBase) + by * wb + bx) * kBinWorkStride], 1);
            }
        }
    }
    const S32 incl = warpInclusiveScan(n);
    sm.incl[lane] = incl;
    __syncwarp();
    // Boxes of more than four bins: the whole warp, one item at a time.
    for (U32 m = kBins ? __ballot_sync(0xFFFFFFFFu, bins > 4) : 0u; m; m &= m - 1) {
        const int j = __ffs(m) - 1;
        const InstanceDev* in = &d.inst[sm.inst[j]];
        const S32 width = __ldg(&in->width), height = __ldg(&in->height);
        const TriGeom g = geomFromHeader(make_uint4(sm.v[0][j], sm.v[1][j], sm.v[2][j], 0u));
        const CellBox bb = headerBox(g, in).coarser(d.binLog2);
        const S32 w = bb.hx - bb.lx + 1, cnt = bb.count();
        const bool test = !bb.small();
        const S32 wb = __ldg(&in->widthBins), binBase = __ldg(&in->binBase);
        for (S32 k = lane; k < cnt; k += 32) {
            const S32 by = bb.ly + k / w, bx = bb.lx + k % w;
            if (!test || triTouchesCell(g, bx, by, d.binLog2, width, height))
                atomicAdd(&d.binWork[(binBase + by * wb + bx) * kBinWorkStride], 1);
        }
    }
    return __shfl_sync(0xFFFFFFFFu, incl, 31);
}

// A unit's items: how many, the list entry of lane l < items, and which slice
// of how many of their boxes.
__device__ __forceinline__ S32 unitItems(const DrawDev& d, const ItemUnits& iu, S32 u, U32& entry, S32& slice, S32& slices) {
    const int lane = threadIdx.x & 31;
    S32 items = 1;
    slice = 0;
    slices = 1;
    entry = 0;
    if (u < iu.hugeUnits + iu.largeUnits) {
        const bool huge = u < iu.hugeUnits;
        const S32 k = huge ? u : u - iu.hugeUnits;
        slices = huge ? iu.hugeSlices : iu.largeSlices;
        const S32 h = k / slices;
        slice = k - h * slices;
        entry = __ldcg(&d.largeItems[huge ? d.maxSubtris - 1 - h : (S64)h]);
    } else {
        const S32 first = (u - iu.hugeUnits - iu.largeUnits) * iu.group;
        items = min(iu.group, iu.medium - first);
        if (lane < items) entry = __ldcg(&d.mediumItems[first + lane]);
    }
    return items;
}

// A warp's current block of item pair records: its own first, then from a
// counter. A warp leaves at most one block partly filled. Past the last block
// nothing is written: restKernel takes the warp's pairs beyond its full blocks.
// (Block numbers are compared unsigned, so a counter past 2^31 gives none
// either.)
struct ItemBlock {
    S32 block, fill, full;
};
__device__ __forceinline__ bool isBlock(const DrawDev& d, S32 block) { return (U32)block < (U32)d.maxItemBlocks; }

// Whether every item pair has a record, by the draw's counters.
__device__ __forceinline__ bool itemsRecorded(const DrawDev& d, S32 itemWarps, S32 itemBlocks) {
    return (U32)itemWarps + (U32)itemBlocks <= (U32)d.maxItemBlocks;
}

// Records the pairs of the lanes with `hit` and counts their tiles.
__device__ __forceinline__ void recordItemPairs(const DrawDev& d, ItemBlock& blk, bool hit, U32 entry, S32 tile) {
    const int lane = threadIdx.x & 31;
    const U32 mask = __ballot_sync(0xFFFFFFFFu, hit);
    const S32 cnt = __popc(mask);
    if (cnt == 0) return;
    if (hit) atomicAdd(&d.tileItems[tile], 1);
    S32 at = blk.fill + __popc(mask & ((1u << lane) - 1u));
    S32 block = blk.block;
    blk.fill += cnt;
    if (blk.fill > kItemBlock) {
        S32 fresh = 0;
        if (lane == 0) {
            fresh = gridDim.x * kListWarps + atomicAdd(&d.counters->itemBlocks, 1);
            if (isBlock(d, block)) d.itemBlockCount[block] = kItemBlock;
        }
        fresh = __shfl_sync(0xFFFFFFFFu, fresh, 0);
        if (isBlock(d, block)) blk.full++;
        if (at >= kItemBlock) {
            block = fresh;
            at -= kItemBlock;
        }
        blk.fill -= kItemBlock;
        blk.block = fresh;
    }
    if (hit && isBlock(d, block)) d.itemPairs[(S64)block * kItemBlock + at] = (U64)entry << 32 | (U32)tile;
}

// Records the pairs of the items and counts their tiles and bins. Persistent
// warps over the units. The launch has at most d.maxItemBlocks warps.
__global__ void __launch_bounds__(kListThreads, kItemWarpsPerSM / kListWarps) itemKernel(const __grid_constant__ DrawDev d) {
    pdlWait();
    __shared__ ItemSmem s_items[kListWarps];
    if (__ldcg(&d.counters->overflow) & kOverflowSubtris) return;
    ItemSmem& sm = s_items[threadIdx.x >> 5];
    const int lane = threadIdx.x & 31;
    const S32 warps = gridDim.x * kListWarps;
    const ItemUnits iu = planItems(d, warps);
    if (blockIdx.x == 0 && threadIdx.x == 0) d.counters->numUnits = iu.total;
    ItemBlock blk{(S32)(blockIdx.x * kListWarps + (threadIdx.x >> 5)), 0, 0};
    for (S32 u = blockIdx.x * kListWarps + (threadIdx.x >> 5); u < iu.total; u += warps) {
        S32 slice, slices;
        U32 entry;
        const S32 items = unitItems(d, iu, u, entry, slice, slices);
        const S32 P = stageItems<true>(d, items, entry, slice, slices, sm);
        for (S32 base = 0; base < P; base += 32) {
            const S32 p = base + lane;
            int j = 0;
            S32 tile = 0;
            const bool hit = p < P && pairTile(d, sm, items, p, j, tile);
            const U32 e = __shfl_sync(0xFFFFFFFFu, entry, j);
            recordItemPairs(d, blk, hit, e, tile);
        }
        __syncwarp();
    }
    if (lane == 0) {
        if (isBlock(d, blk.block)) d.itemBlockCount[blk.block] = blk.fill;
        if (d.restItems) d.itemFull[blockIdx.x * kListWarps + (threadIdx.x >> 5)] = isBlock(d, blk.block) ? -1 : blk.full;
    }
    if (blockIdx.x == 0 && threadIdx.x == 0) d.counters->itemWarps = warps;
}

// ------------------------------------------------------------------ scan

// Four consecutive tiles per thread; a CTA's lists are one contiguous piece of
// the list memory, allocated with one atomic on a 64-bit total (list_alloc.h):
// a CTA whose lists do not fit flags the overflow, and no later stage reads a
// start. The first CTA also hands over the bin counts. The work arrays end
// zeroed, for the next draw.
constexpr int kScanTiles = kListThreads * 4;
constexpr int kSortRun = 256;   // lists up to this length are sorted in a warp's registers

__global__ void __launch_bounds__(kListThreads) listScanKernel(const __grid_constant__ DrawDev d) {
    pdlWait();
    markStage(d.stageTiming, d.counters, 2);
    __shared__ U64 s_warp[kListWarps];
    __shared__ U64 s_base;
    const bool failed = (__ldcg(&d.counters->overflow) & kOverflowSubtris) != 0;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    // (Loaded now, looked at when the bins are handed over.)
    const S32 itemWarps = __ldcg(&d.counters->itemWarps), itemBlocks = __ldcg(&d.counters->itemBlocks);
    const S32 t0 = blockIdx.x * kScanTiles + threadIdx.x * 4;
    S32 c[4], own[4];   // entries, and those the pair stage recorded
#pragma unroll
    for (int k = 0; k < 4; k++) {
        c[k] = own[k] = 0;
        if (t0 + k < d.totalTiles) own[k] = __ldcg(&d.tileWork[(t0 + k) << d.tileWorkLog2]);
    }
    if (t0 + 3 < d.totalTiles) {
        const int4 x = __ldcg((const int4*)(d.tileItems + t0));
        c[0] = own[0] + x.x, c[1] = own[1] + x.y, c[2] = own[2] + x.z, c[3] = own[3] + x.w;
        *(int4*)(d.tileItems + t0) = make_int4(0, 0, 0, 0);
        *(int4*)(d.tileCount + t0) = make_int4(c[0], c[1], c[2], c[3]);
    } else {
#pragma unroll
        for (int k = 0; k < 4; k++) {
            if (t0 + k < d.totalTiles) {
                c[k] = own[k] + __ldcg(&d.tileItems[t0 + k]);
                d.tileItems[t0 + k] = 0;
                d.tileCount[t0 + k] = c[k];
            }
        }
    }
#pragma unroll
    for (int k = 0; k < 4; k++)
        if (t0 + k < d.totalTiles) d.tileWork[(t0 + k) << d.tileWorkLog2] = 0;
    const S32 longest = __reduce_max_sync(0xFFFFFFFFu, max(max(c[0], c[1]), max(c[2], c[3])));
    if (lane == 0 && longest > kSortRun) atomicMax(&d.counters->longestList, longest);
    // Places modulo 2^32 (whole where the lists fit) beside 64-bit totals.
    const U64 sum = entriesOf4(c);
    const U32 incl = warpInclusiveScan((U32)sum);
    const U64 warpSum = warpTotal(sum);
    if (lane == 0) s_warp[warp] = warpSum;
    __syncthreads();
    if (warp == 0) {
        const U64 v = lane < kListWarps ? s_warp[lane] : 0ull;
        const U64 i = warpInclusiveScan<U64, kListWarps>(v);
        if (lane < kListWarps) s_warp[lane] = i - v;
        if (lane == kListWarps - 1 && !failed) {
            const U64 base = atomicAdd((unsigned long long*)&d.counters->tileTotal, (unsigned long long)i);
            atomicMax(&d.counters->tileEntries, reportedEntries(base + i));
            if (!listsFit(base + i, d.maxTileEntries)) atomicOr(&d.counters->overflow, kOverflowTile);
            s_base = base;
        }
    }
    __syncthreads();
    S32 s = (S32)((U32)s_base + (U32)s_warp[warp] + incl - (U32)sum);
    if (!failed) {
        if (t0 + 3 < d.totalTiles) {
            const int4 v = make_int4(s, s + c[0], s + c[0] + c[1], s + c[0] + c[1] + c[2]);
            *(int4*)(d.tileStart + t0) = v;
            *(int4*)(d.tileCursor + t0) = make_int4(v.x + own[0], v.y + own[1], v.z + own[2], v.w + own[3]);
        } else {
#pragma unroll
            for (int k = 0; k < 4; k++) {
                if (t0 + k < d.totalTiles) {
                    d.tileStart[t0 + k] = s;
                    d.tileCursor[t0 + k] = s + own[k];
                }
                s += c[k];
            }
        }
    }
    if (blockIdx.x == 0) {
        U64 mine = 0;
        for (S32 b = threadIdx.x; b < d.totalBins; b += kListThreads) {
            const S32 v = __ldcg(&d.binWork[b * kBinWorkStride]);
            d.binWork[b * kBinWorkStride] = 0;
            d.binCount[b] = v;
            mine += (U32)v;
        }
        mine = warpTotal(mine);
        __syncthreads();
        if (lane == 0) s_warp[warp] = mine;
        __syncthreads();
        if (threadIdx.x == 0 && !d.restItems && !itemsRecorded(d, itemWarps, itemBlocks))
            atomicOr(&d.counters->overflow, kOverflowItems);
        if (threadIdx.x == 0 && !failed) {
            U64 total = 0;
            for (int w = 0; w < kListWarps; w++) total += s_warp[w];
            d.counters->binEntries = reportedEntries(total);
            if (d.maxBinEntries >= 0 && !listsFit(total, d.maxBinEntries)) atomicOr(&d.counters->overflow, kOverflowBin);
        }
    }
}

// --------------------------------------------------------------- scatter

__device__ __forceinline__ void putEntry(const DrawDev& d, S32 idx, U32 entry) {
    if (listHolds(idx, d.maxTileEntries)) d.tileList[idx] = entry;
}

// Persistent warps: the pair records, then those of the items.
__global__ void __launch_bounds__(kListThreads) listScatterKernel(const __grid_constant__ DrawDev d) {
    pdlWait();
    if (__ldcg(&d.counters->overflow)) return;
    const int lane = threadIdx.x & 31;
    const S32 warps = gridDim.x * kListWarps, warpIdx = blockIdx.x * kListWarps + (threadIdx.x >> 5);
    for (S32 chunk = warpIdx; chunk < d.numChunks; chunk += warps) {
        const S32 count = __ldcg(&d.pairCount[chunk]);
        const U64* pairs = d.pairs + (S64)chunk * 2 * d.chunkTris;
        const U32 t0 = (U32)chunk * (U32)d.chunkTris;
        // Four pairs per lane in flight.
        for (S32 p0 = lane; p0 < count; p0 += 128) {
            U64 rec[4];
            S32 start[4];
#pragma unroll
            for (int k = 0; k < 4; k++) rec[k] = p0 + k * 32 < count ? __ldcg(&pairs[p0 + k * 32]) : 0ull;
#pragma unroll
            for (int k = 0; k < 4; k++) start[k] = __ldg(&d.tileStart[(U32)(rec[k] >> 10) & (U32)(kMaxRecord - 1)]);
#pragma unroll
            for (int k = 0; k < 4; k++)
                if (p0 + k * 32 < count)
                    putEntry(d, start[k] + (S32)(rec[k] >> 37), (t0 + ((U32)rec[k] & 1023u)) << 3 | 7u);
        }
    }
    const S32 blocks = (S32)min((U32)__ldcg(&d.counters->itemWarps) + (U32)__ldcg(&d.counters->itemBlocks), (U32)d.maxItemBlocks);
    // The items' pairs, four per lane in flight too (one per lane: the stage 23.5 us
    // instead of 22.1 on 20,000 triangles of 60 pixels, 49 / 46 on the water layer).
    constexpr int kParts = kItemBlock / 128;
    for (S64 u = warpIdx; u < (S64)blocks * kParts; u += warps) {
        const S32 block = (S32)(u / kParts), at = (S32)(u % kParts) * 128 + lane;
        const S32 count = __ldcg(&d.itemBlockCount[block]);
        const U64* pairs = d.itemPairs + (S64)block * kItemBlock;
        U64 rec[4];
        S32 place[4];
#pragma unroll
        for (int k = 0; k < 4; k++) rec[k] = at + k * 32 < count ? __ldcg(&pairs[at + k * 32]) : 0ull;
#pragma unroll
        for (int k = 0; k < 4; k++)
            if (at + k * 32 < count) place[k] = atomicAdd(&d.tileCursor[(U32)rec[k]], 1);
#pragma unroll
        for (int k = 0; k < 4; k++)
            if (at + k * 32 < count) putEntry(d, place[k], (U32)(rec[k] >> 32));
    }
}

// The item pairs without a record, straight into the lists: the item kernel's
// warps that ran out of blocks expand their units again and pass over the pairs
// of their full blocks.
__global__ void __launch_bounds__(kListThreads, kItemWarpsPerSM / kListWarps) restKernel(const __grid_constant__ DrawDev d) {
    pdlWait();
    __shared__ ItemSmem s_items[kListWarps];
    const S32 itemWarps = __ldcg(&d.counters->itemWarps);
    if (__ldcg(&d.counters->overflow) || itemsRecorded(d, itemWarps, __ldcg(&d.counters->itemBlocks))) return;
    ItemSmem& sm = s_items[threadIdx.x >> 5];
    const int lane = threadIdx.x & 31;
    const ItemUnits iu = planItems(d, itemWarps);
    for (S32 w = blockIdx.x * kListWarps + (threadIdx.x >> 5); w < itemWarps; w += gridDim.x * kListWarps) {
        const S32 full = __ldcg(&d.itemFull[w]);
        if (full < 0) continue;
        S64 recorded = (S64)full * kItemBlock;   // still to pass over
        for (S32 u = w; u < iu.total; u += itemWarps) {
            S32 slice, slices;
            U32 entry;
            const S32 items = unitItems(d, iu, u, entry, slice, slices);
            const S32 P = stageItems<false>(d, items, entry, slice, slices, sm);
            for (S32 base = 0; base < P; base += 32) {
                const S32 p = base + lane;
                int j = 0;
                S32 tile = 0;
                const bool hit = p < P && pairTile(d, sm, items, p, j, tile);
                const U32 e = __shfl_sync(0xFFFFFFFFu, entry, j);
                const U32 mask = __ballot_sync(0xFFFFFFFFu, hit);
                if (hit && __popc(mask & ((1u << lane) - 1u)) >= recorded) putEntry(d, atomicAdd(&d.tileCursor[tile], 1), e);
                recorded = max(recorded - __popc(mask), (S64)0);
            }
            __syncwarp();
        }
    }
}

// ------------------------------------------------------------------ sort
//
// A warp sorts the lists of four neighbouring tiles at a time where they have
// at most 8 entries each, of two with at most 16, and single ones of up to 256
// in registers; longer
// ones are sorted by a CTA each: runs of 256 by its warps, then merged pair by
// pair in shared memory (an entry's place in a merged run is its own index
// plus its rank in the other run: the entries of a list are distinct), up to
// kSortShared entries; lists beyond that by a radix sort through a copy in
// global memory (mostly L2; 17,000 entries in each tile of a 64x64 viewport:
// 1.15 ms a draw, 17.8 when such lists were merged in place with a bitonic
// network and two CTAs had all of them).

constexpr int kSortShared = 4096;
// Mean list length below which a warp takes four tiles at a time (coarse stage
// of the textured terrain and of the 32-scene batch: 66 and 78 us; with 64: 79
// and 78, with 4: 67 and 87).
constexpr int kSparseLists = 16;
constexpr int kSortCtas = 6;   // resident CTAs per SM

// Sorts each W consecutive lanes' values (bitonic).
template <int W>
__device__ __forceinline__ U32 laneSort(U32 v) {
    const int lane = threadIdx.x & 31;
#pragma unroll
    for (int k = 2; k <= W; k <<= 1) {
#pragma unroll
        for (int j = k >> 1; j > 0; j >>= 1) {
            const U32 o = __shfl_xor_sync(0xFFFFFFFFu, v, j);
            const bool up = k == W || (lane & k) == 0;
            v = ((lane & j) == 0) == up ? min(v, o) : max(v, o);
        }
    }
    return v;
}

// Sorts the lists of up to W entries of 32 / W tiles, the lanes of a tile
// holding its list's extent.
template <int W>
__device__ __forceinline__ void sortShort(U32* tileList, S32 n, S32 start) {
    const int at = (threadIdx.x & 31) & (W - 1);
    U32 v = at < n ? tileList[start + at] : 0xFFFFFFFFu;
    v = laneSort<W>(v);
    if (at < n) tileList[start + at] = v;
}

// Sorts 32 * E values, lane l holding values l, l + 32, ... (bitonic).
template <int E>
__device__ __forceinline__ void warpSort(U32 (&v)[E]) {
    const int lane = threadIdx.x & 31;
#pragma unroll
    for (int k = 2; k <= 32 * E; k <<= 1) {
#pragma unroll
        for (int j = k >> 1; j > 0; j >>= 1) {
            if (j >= 32) {
#pragma unroll
                for (int e = 0; e < E; e++) {
                    const int f = e ^ (j >> 5);
                    if (f > e) {
                        const bool up = ((e << 5) & k) == 0;
                        const U32 a = v[e], b = v[f];
                        v[e] = up ? min(a, b) : max(a, b);
                        v[f] = up ? max(a, b) : min(a, b);
                    }
                }
            } else {
#pragma unroll
                for (int e = 0; e < E; e++) {
                    const U32 o = __shfl_xor_sync(0xFFFFFFFFu, v[e], j);
                    const bool up = k >= 32 ? (((e << 5) & k) == 0) : ((lane & k) == 0);
                    v[e] = ((lane & j) == 0) == up ? min(v[e], o) : max(v[e], o);
                }
            }
        }
    }
}

// Sorts src[0, n), n <= 32 * E, into dst.
template <int E>
__device__ __forceinline__ void warpSortList(const U32* src, U32* dst, S32 n) {
    const int lane = threadIdx.x & 31;
    U32 v[E];
#pragma unroll
    for (int e = 0; e < E; e++) v[e] = e * 32 + lane < n ? src[e * 32 + lane] : 0xFFFFFFFFu;
    warpSort<E>(v);
#pragma unroll
    for (int e = 0; e < E; e++)
        if (e * 32 + lane < n) dst[e * 32 + lane] = v[e];
}

__device__ __forceinline__ void warpSortAny(const U32* src, U32* dst, S32 n) {
    if (n <= 32) warpSortList<1>(src, dst, n);
    else if (n <= 64) warpSortList<2>(src, dst, n);
    else if (n <= 128) warpSortList<4>(src, dst, n);
    else warpSortList<8>(src, dst, n);
}

// Sorts list[0, n), n <= kSortShared, through the two shared buffers; called
// by the whole CTA.
__device__ __forceinline__ void ctaSort(U32* list, S32 n, U32* a, U32* b) {
    for (S32 r = (threadIdx.x >> 5) * kSortRun; r < n; r += kListWarps * kSortRun)
        warpSortAny(list + r, a + r, min(n - r, kSortRun));
    __syncthreads();
    for (S32 run = kSortRun; run < n; run *= 2) {
        for (S32 i = threadIdx.x; i < n; i += kListThreads) {
            const U32 x = a[i];
            const S32 r0 = i & ~(2 * run - 1);
            const bool right = (i & run) != 0;
            const S32 o0 = right ? r0 : r0 + run;                       // the sibling run
            S32 lo = min(o0, n), hi = min(o0 + run, n);
            const S32 ofirst = lo;
            while (lo < hi) {
                const S32 mid = (lo + hi) >> 1;
                if (a[mid] < x) lo = mid + 1; else hi = mid;
            }
            b[r0 + (i & (run - 1)) + (lo - ofirst)] = x;
        }
        __syncthreads();
        U32* t = a;
        a = b;
        b = t;
    }
    for (S32 i = threadIdx.x; i < n; i += kListThreads) list[i] = a[i];
    __syncthreads();
}

// One stable pass of a radix sort over bits [shift, shift + 8) of src[0, n) into
// dst, by the whole CTA: a warp counts and then moves its own piece of the list
// (at 32 entries a step, ranked among equal digits by ballots). hist holds
// kListWarps x 256 words.
__device__ __forceinline__ void radixPass(const U32* src, U32* dst, S32 n, int shift, S32* hist, S32* sums) {
    static_assert(kListThreads == 256, "a thread per digit");
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const U32 ltMask = (1u << lane) - 1u;
    const S32 piece = (n + kListThreads - 1) / kListThreads * 32;
    const S32 begin = min(warp * piece, n), end = min(begin + piece, n);
    S32* mine = hist + warp * 256;
    for (int i = threadIdx.x; i < kListWarps * 256; i += kListThreads) hist[i] = 0;
    __syncthreads();
    for (S32 i = begin + lane; i < end; i += 128) {
        U32 v[4];
#pragma unroll
        for (int k = 0; k < 4; k++) v[k] = i + k * 32 < end ? src[i + k * 32] : 0u;
#pragma unroll
        for (int k = 0; k < 4; k++)
            if (i + k * 32 < end) atomicAdd(&mine[v[k] >> shift & 255u], 1);
    }
    __syncthreads();
    // The pieces' places among the entries of digit threadIdx.x, then the digits'.
    S32 total = 0;
    for (int w = 0; w < kListWarps; w++) {
        const S32 c = hist[w * 256 + threadIdx.x];
        hist[w * 256 + threadIdx.x] = total;
        total += c;
    }
    const S32 incl = warpInclusiveScan(total);
    if (lane == 31) sums[warp] = incl;
    __syncthreads();
    S32 base = incl - total;
    for (int w = 0; w < warp; w++) base += sums[w];
    for (int w = 0; w < kListWarps; w++) hist[w * 256 + threadIdx.x] += base;
    __syncthreads();
    for (S32 i0 = begin; i0 < end; i0 += 128) {
        U32 v[4];
#pragma unroll
        for (int k = 0; k < 4; k++) v[k] = i0 + k * 32 + lane < end ? src[i0 + k * 32 + lane] : 0u;
#pragma unroll
        for (int k = 0; k < 4; k++) {
            const bool on = i0 + k * 32 + lane < end;
            const U32 digit = v[k] >> shift & 255u;
            U32 peers = __ballot_sync(0xFFFFFFFFu, on);
#pragma unroll
            for (int b = 0; b < 8; b++) {
                const bool bit = digit >> b & 1u;
                const U32 set = __ballot_sync(0xFFFFFFFFu, bit);
                peers &= bit ? set : ~set;
            }
            const S32 at = on ? mine[digit] + __popc(peers & ltMask) : 0;
            __syncwarp();
            if (on && (peers & ltMask) == 0u) mine[digit] += __popc(peers);
            __syncwarp();
            if (on) dst[at] = v[k];
        }
    }
    __syncthreads();
}

// Sorts list[0, n) through tmp[0, n); entries are below 2^bits.
__device__ __forceinline__ void ctaSortLong(U32* list, U32* tmp, S32 n, int bits, S32* hist, S32* sums) {
    U32* src = list;
    U32* dst = tmp;
    for (int shift = 0; shift < bits; shift += 8) {
        radixPass(src, dst, n, shift, hist, sums);
        U32* t = src;
        src = dst;
        dst = t;
    }
    if (src != list) {
        for (S32 i = threadIdx.x; i < n; i += kListThreads) list[i] = src[i];
        __syncthreads();
    }
}

__global__ void __launch_bounds__(kListThreads, kSortCtas) listSortKernel(const __grid_constant__ DrawDev d, S32 tileBegin,
                                                               S32 tileEnd) {
    pdlWait();
    __shared__ U32 s_a[kSortShared], s_b[kSortShared];
    __shared__ S32 s_long[kListThreads], s_found;
    if (__ldcg(&d.counters->overflow)) return;
    const int lane = threadIdx.x & 31;
    const S32 warps = gridDim.x * kListWarps;
    const S32 quads = (tileEnd - tileBegin + 3) / 4;
    // A warp takes quads of tiles, every gridDim.x-th one per CTA. Neighbouring quads go to different CTAs: a crowded
    // viewport's long lists would otherwise pile up on a few.
    if (__ldcg(&d.counters->tileEntries) < kSparseLists * d.totalTiles) {
        // Mostly short lists: a quad at a time, its extents (of the tile lane /
        // 8) loaded during the sort of the quad before it.
        S32 quad = blockIdx.x + (threadIdx.x >> 5) * gridDim.x;
        S32 n = 0, start = 0;
        auto load = [&]() {
            const S32 tile = tileBegin + quad * 4 + (lane >> 3);
            const bool on = quad < quads && tile < tileEnd;
            n = on ? __ldg(&d.tileCount[tile]) : 0;
            start = on ? __ldg(&d.tileStart[tile]) : 0;
        };
        load();
        while (quad < quads) {
            const S32 cnt = n, first = start;
            quad += warps;
            load();
            const S32 most = __reduce_max_sync(0xFFFFFFFFu, cnt);
            if (most <= 8) {
                if (most > 1) sortShort<8>(d.tileList, cnt, first);
                continue;
            }
#pragma unroll 1
            for (int half = 0; half < 2; half++) {
                const S32 c0 = __shfl_sync(0xFFFFFFFFu, cnt, half * 16), c1 = __shfl_sync(0xFFFFFFFFu, cnt, half * 16 + 8);
                const S32 s0 = __shfl_sync(0xFFFFFFFFu, first, half * 16), s1 = __shfl_sync(0xFFFFFFFFu, first, half * 16 + 8);
                if (max(c0, c1) <= 16) {
                    sortShort<16>(d.tileList, lane < 16 ? c0 : c1, lane < 16 ? s0 : s1);
                } else {
                    if (c0 > 1 && c0 <= kSortRun) warpSortAny(d.tileList + s0, d.tileList + s0, c0);
                    if (c1 > 1 && c1 <= kSortRun) warpSortAny(d.tileList + s1, d.tileList + s1, c1);
                }
            }
        }
    } else {
        // A tile at a time, its extent loaded during the sort of the one before.
        const S32 step = gridDim.x * 4;
        S32 k = blockIdx.x * 4 + (threadIdx.x & 96) / 32 + (threadIdx.x >> 7) * step;   // tile of the range
        const S32 tiles = tileEnd - tileBegin;
        S32 n = k < tiles ? __ldg(&d.tileCount[tileBegin + k]) : 0, start = k < tiles ? __ldg(&d.tileStart[tileBegin + k]) : 0;
        while (k < tiles) {
            U32* list = d.tileList + start;
            const S32 cnt = n;
            k += (kListWarps / 4) * step;
            if (k < tiles) {
                n = __ldg(&d.tileCount[tileBegin + k]);
                start = __ldg(&d.tileStart[tileBegin + k]);
            }
            if (cnt > 1 && cnt <= kSortRun) warpSortAny(list, list, cnt);
        }
    }
    // The long lists, each by a whole CTA; a CTA looks after every gridDim.x-th
    // tile. (The warps above leave these lists alone.)
    if (__ldcg(&d.counters->longestList) <= kSortRun) return;
    const int bits = 64 - __clzll(d.totalTris * 8 - 1);
    for (S32 t0 = tileBegin + (S32)blockIdx.x; t0 < tileEnd; t0 += kListThreads * gridDim.x) {
        const S64 t = (S64)t0 + (S64)threadIdx.x * gridDim.x;
        const bool isLong = t < tileEnd && __ldg(&d.tileCount[t]) > kSortRun;
        if (threadIdx.x == 0) s_found = 0;
        if (!__syncthreads_or(isLong)) continue;
        if (isLong) s_long[atomicAdd(&s_found, 1)] = (S32)t;
        __syncthreads();
        const int found = s_found;
        for (int k = 0; k < found; k++) {
            const S32 lt = s_long[k];
            const S32 ln = __ldg(&d.tileCount[lt]), start = __ldg(&d.tileStart[lt]);
            if (ln <= kSortShared) ctaSort(d.tileList + start, ln, s_a, s_b);
            else ctaSortLong(d.tileList + start, d.sortScratch + start, ln, bits, (S32*)s_a, (S32*)s_b);
        }
        __syncthreads();
    }
}

// ------------------------------------------------------------ launchers

// The list stages after setup: bin (pairs, items) and coarse (scan, scatter).
cudaError_t launchBinning(const DrawDev& d, int numSMs, cudaStream_t stream) {
    static IntsPerDevice<2> ctas;   // resident CTAs per SM of the pair and scatter kernels
    const int pairCtas = ctas.get(0, [](int) {
        int n = 0;
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, pairKernel, kListThreads, 0);
        return n > 0 ? n : 1;
    });
    const int scatterCtas = ctas.get(1, [](int) {
        int n = 0;
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, listScatterKernel, kListThreads, 0);
        return n > 0 ? n : 1;
    });
    const int itemGrid = numSMs * (kItemWarpsPerSM / kListWarps);
    cudaError_t e = cudaSuccess;
    if (d.totalTris > 0) {
        const int pairGrid = std::min(numSMs * pairCtas, (d.numChunks + kListWarps - 1) / kListWarps);
        e = launchKernel(pairKernel, pairGrid, kListThreads, 0, stream, true, d);
        if (e == cudaSuccess) e = launchKernel(itemKernel, itemGrid, kListThreads, 0, stream, true, d);
    }
    // The scan also runs for a draw without triangles: it zeroes the counts.
    if (e == cudaSuccess)
        e = launchKernel(listScanKernel, (d.totalTiles + kScanTiles - 1) / kScanTiles, kListThreads, 0, stream, true, d);
    if (e == cudaSuccess && d.totalTris > 0)
        e = launchKernel(listScatterKernel, numSMs * scatterCtas, kListThreads, 0, stream, true, d);
    if (e == cudaSuccess && d.totalTris > 0 && d.restItems)
        e = launchKernel(restKernel, numSMs, kListThreads, 0, stream, true, d);
    return e;
}

// Sorts the lists of tiles [tileBegin, tileEnd) into submission order. A CTA to
// 32 tiles, or to every tile where the draw has at least eight triangles a
// tile and long lists are likely, which take a CTA each (20,000 blended
// triangles of 60 pixels at 200x150 574 us a draw with the former, 259 with the
// latter; 5,000 small ones at 641x479 80 and 83).
cudaError_t launchListSort(const DrawDev& d, int32_t tileBegin, int32_t tileEnd, int numSMs, cudaStream_t stream) {
    if (d.totalTris <= 0 || tileEnd <= tileBegin) return cudaSuccess;
    const int64_t tiles = (int64_t)tileEnd - tileBegin;
    const int64_t want = d.totalTris >= 8 * (int64_t)d.totalTiles ? tiles : (tiles + 4 * kListWarps - 1) / (4 * kListWarps);
    return launchKernel(listSortKernel, (unsigned)std::min<int64_t>(want, (int64_t)numSMs * kSortCtas), kListThreads, 0, stream,
                        true, d, tileBegin, tileEnd);
}

}  // namespace cr
