// fine.cuh -- fine raster kernel (stage 4 of 4).
//
// One warp owns one 8x8 tile at a time (persistent warps pulling tiles from a
// counter, as FineRaster.inl:534-552). The tile's colour and depth live in the
// warp's shared memory for the whole tile. Its triangle list is consumed in
// batches of 32; lane i fetches entry i (header, data slot, early-Z against
// the tile's current maximum depth as FineRaster.inl:229-240 or mayWin, edge
// functions at the tile origin). Then one of two algorithms runs, chosen at compile time:
//
// What bounds it: the shared-memory and L1 data pipe (70% of its wavefronts on
// 1M small triangles, 72% on the 8.4M-triangle 4x MSAA heightfield) and
// instruction issue (72%, 68%), at 30 to 38 resident warps (before). So triangles are
// kept in packed records read by 128-bit loads (two 16-bit edge steps to a
// word, an edge value in one dp2a), tiles move 8 bytes a lane, and tiles that
// no triangle touches are written without passing through shared memory. These
// took the stage from 84 to 78 us on the 1M soup (with turnOf), 107 to 96 on
// 20,000 triangles of 60 pixels, 627 to 573 on the heightfield (with pixelBox's
// tight boxes), 613 to 455 on 300k triangles at 8x MSAA, 160 to 152 on 300k
// blended ones, 471 to 449 on the textured terrain (with loadSlot32).
//
// Both paths deal the (triangle, pixel) pairs of the batch's small triangles
// (pixel box of at most fineSelfPixels pixels) over the lanes; larger
// triangles are rasterized by the 32 pixel-owning lanes, two pixels each.
//
// Ordered path (any blend shader, discard, quads):
//   coverage masks per triangle (set by the pairs, or by ballots over the
//   pixel-owning lanes for large triangles), covered pixels compacted into
//   passes of 32 fragments in submission order (FineRaster.inl:625-731), then
//   depth test, shading and blending per fragment. Fragments of one pass that
//   hit the same pixel are grouped with __match_any_sync and applied one rank
//   at a time in lane order, which is submission order. This replaces the
//   reference's reliance on lock-step warps for same-address shared-memory
//   races (FineRaster.inl:433-495, 758-851), undefined on sm_70 and later.
//   With one sample, a depth test and a fragment shader that never discards,
//   a fragment later in the batch than its pixel's minimum (depth, then
//   position) is dropped before compaction: it would fail the LESS test.
//
// Visibility path (depth test on, blend shader that ignores the destination,
//   fragment shader that never discards): the final colour and depth of a
//   sample are those of its front-most covering fragment, the earliest one in
//   submission order on equal depth -- the same result as applying every
//   fragment in order with a LESS test. Each sample keeps a 64-bit key
//   (depth << 32 | list entry + 1) that fragments lower with atomicMin, so the
//   tile's list may come in any order (entries grow in submission order; early
//   Z drops no triangle that could win, see mayWin);
//   after the list, the tile's winners are listed and each is shaded once,
//   32 at a time.
//
// MSAA keeps every sample of the tile in shared memory (reference layout:
// sample i of pixel x at word i * 8 + x of the tile row) and shades once per
// (pixel, triangle) at the centroid of the triangle's covered samples.
#pragma once

#include "../PixelPipe.hpp"
#include "device.cuh"
#include "launch.h"

#include <type_traits>

namespace cr {

constexpr int kFineMaxThreads = 256;
// Triangles whose pixel box inside the tile has at most DrawDev::fineSelfPixels
// pixels are rasterized pixel by pixel by the lanes -- their (triangle, pixel)
// pairs are dealt over all lanes; larger ones by the whole warp, two
// pixels per lane. Default: 16 pixels.
__host__ __device__ constexpr int fineSelfPixelsDefault(int, bool) { return 16; }


// A triangle of a batch in 12 words. Edge k's value at a sample whose offset
// from the tile's pixel (0, 0) centre, plus 8 subpixels on each axis, is the
// byte pair q is E[k] + A[k] * q.x + B[k] * q.y, one dp2a with the two steps
// as 16-bit halves (see packTri). Lanes read a record with 128-bit loads: all
// lanes the same one (a broadcast) on the large-triangle path; on the pair
// path lanes of a quarter warp read consecutive records, whose 48-byte stride
// puts any eight of them on distinct banks.
struct TriRec {
    uint4 q[3];   // E0 E1 E2 AB0 | AB1 AB2 zx zy | zb id box -
};

// The ordered path's per-warp state (one warp per tile).
template <int S>
struct FineWarpSmem {
    static constexpr int kTileWords = 64 << S;
    U32 color[kTileWords];
    U32 depth[kTileWords];
    TriRec rec[32];        // id: triangle index within the draw
    TriRec data[32];       // words 4 to 15 of the triangle data slots
    U32 covLo[32];
    U32 covHi[32];
    // One sample, depth test on, no discard: each pixel's minimum of
    // (depth << 32 | batch triangle) over the batch's covered fragments.
    U64 batchMin[S == 0 ? 64 : 1];
    S32 fragEnd[32];       // inclusive prefix of the small triangles' pair counts
    S32 fragHead[32];      // batch triangle whose fragments start at position i of the current pass
    F32 shared[32];
};

// The visibility path's per-warp state: no separate depth array (a key's high
// word is its sample's depth) and only the triangle words it reads.
template <int S>
struct FineVisSmem {
    static constexpr int kTileWords = 64 << S;
    U32 color[kTileWords];
    U64 key[kTileWords];        // depth << 32 | order (order << NS | coverage mask with MSAA)
    TriRec rec[32];             // id: list entry within the scene + 1
    uint2 turn[32];             // the small triangles in turn: box (packBox), batch triangle << 16 | first pair
    U32 winners[kTileWords];    // resolve: (pixel | first sample << 6 | samples won << 9)
    F32 shared[32];
};

// Compile-time shape of a pipe's fine stage.
template <class FS, class BS, int S, U32 F>
struct FineTraits {
    static constexpr bool kDepth = (F & kRenderDepth) != 0;
    static constexpr bool kQuads = (F & kRenderQuads) != 0;
    // Opaque depth-tested pipes resolve visibility with keys (see fineKernel).
    static constexpr bool kVisibility = kDepth && !kQuads && !FW::BlendShaderTraits<BS>::needsDst &&
                                        !FW::FragmentShaderTraits<FS>::mayDiscard;
    using Smem = typename std::conditional<kVisibility, FineVisSmem<S>, FineWarpSmem<S>>::type;
};

__device__ __forceinline__ int nthSetBit32(U32 m, int n) {
    int pos = 0;
#pragma unroll
    for (int w = 16; w >= 1; w >>= 1) {
        U32 lowMask = (1u << w) - 1u;
        int c = __popc(m & lowMask);
        if (n >= c) { n -= c; m >>= w; pos += w; }
    }
    return pos;
}
__device__ __forceinline__ int nthSetBit64(U32 lo, U32 hi, int n) {
    int c = __popc(lo);
    return (n < c) ? nthSetBit32(lo, n) : 32 + nthSetBit32(hi, n - c);
}

// computeBarys (FineRaster.inl:21-44)
template <int S>
__device__ __forceinline__ void computeBarys(FW::Vec3f& b, FW::Vec3f& bdx, FW::Vec3f& bdy, const U32* w,
                                             const U32* u, const U32* v, S32 sx, S32 sy) {
    F32 wr = frcp(__int2float_rn((S32)(w[0] * (U32)sx + w[1] * (U32)sy + w[2])));
    F32 uu = fmul(wr, __int2float_rn((S32)(u[0] * (U32)sx + u[1] * (U32)sy + u[2])));
    F32 vv = fmul(wr, __int2float_rn((S32)(v[0] * (U32)sx + v[1] * (U32)sy + v[2])));
    b = FW::Vec3f(fsub(fsub(1.0f, uu), vv), uu, vv);
    F32 wd = fmul(wr, (F32)(1 << (S + 1)));
    F32 udx = fmul(wd, fsub(__int2float_rn((S32)u[0]), fmul(uu, __int2float_rn((S32)w[0]))));
    F32 udy = fmul(wd, fsub(__int2float_rn((S32)u[1]), fmul(uu, __int2float_rn((S32)w[1]))));
    F32 vdx = fmul(wd, fsub(__int2float_rn((S32)v[0]), fmul(vv, __int2float_rn((S32)w[0]))));
    F32 vdy = fmul(wd, fsub(__int2float_rn((S32)v[1]), fmul(vv, __int2float_rn((S32)w[1]))));
    bdx = FW::Vec3f(fsub(-udx, vdx), udx, vdx);
    bdy = FW::Vec3f(fsub(-udy, vdy), udy, vdy);
}

__device__ __forceinline__ S32 clampEdge(S64 e) {
    const S64 lim = (S64)1 << 30;
    return (S32)(e > lim ? lim : (e < -lim ? -lim : e));
}

// Edge functions of a header relative to the tile's pixel (0, 0) centre:
// edges (v0, v1 - v0), (v1, v2 - v1), (v0, v0 - v2) as FineRaster.inl:251-275,
// bias of the fill rule (Util.inl:100) folded in. A sample at subpixel offset
// q from that centre is covered iff E[k] + A[k] * q.x + B[k] * q.y >= 0 for
// all k (the offsets stay below 2^8 and |A|, |B| below 2^17, so clamping E to
// +-2^30 keeps every sign).
struct TileEdges {
    S32 E[3], A[3], B[3];
    S32 minX, maxX, minY, maxY;   // vertex box relative to the pixel (0, 0) centre
};

__device__ __forceinline__ TileEdges tileEdges(uint4 h, S32 cx0, S32 cy0) {
    TileEdges t;
    S32 vx[3] = {lo16(h.x) - cx0, lo16(h.y) - cx0, lo16(h.z) - cx0};
    S32 vy[3] = {hi16(h.x) - cy0, hi16(h.y) - cy0, hi16(h.z) - cy0};
    t.minX = min3i(vx[0], vx[1], vx[2]);
    t.maxX = max3i(vx[0], vx[1], vx[2]);
    t.minY = min3i(vy[0], vy[1], vy[2]);
    t.maxY = max3i(vy[0], vy[1], vy[2]);
    const int oi[3] = {0, 1, 0};
    S32 ddx[3] = {vx[1] - vx[0], vx[2] - vx[1], vx[0] - vx[2]};
    S32 ddy[3] = {vy[1] - vy[0], vy[2] - vy[1], vy[0] - vy[2]};
#pragma unroll
    for (int k = 0; k < 3; k++) {
        t.A[k] = -ddy[k];
        t.B[k] = ddx[k];
    }
    // With all vertices within 2^14 subpixels (1,024 pixels) of the tile the
    // products stay within 2^29 and the values within 2^30: no 64-bit step and
    // no clamp.
    const bool near = min(t.minX, t.minY) >= -(1 << 14) && max(t.maxX, t.maxY) <= 1 << 14;
#pragma unroll
    for (int k = 0; k < 3; k++) {
        const S32 bias = ddy[k] > 0 || (ddy[k] == 0 && ddx[k] <= 0) ? 1 : 0;
        if (near)
            t.E[k] = vx[oi[k]] * ddy[k] - vy[oi[k]] * ddx[k] - bias;
        else
            t.E[k] = clampEdge((S64)vx[oi[k]] * ddy[k] - (S64)vy[oi[k]] * ddx[k] - bias);
    }
    return t;
}

__device__ __forceinline__ bool edgesCover(const S32* E, const S32* A, const S32* B, S32 qx, S32 qy) {
    return ((E[0] + A[0] * qx + B[0] * qy) | (E[1] + A[1] * qx + B[1] * qy) | (E[2] + A[2] * qx + B[2] * qy)) >= 0;
}

// Largest distance of a sample from its pixel's centre on either axis, in subpixels.
__host__ __device__ constexpr S32 sampleReach(int s) { return s == 0 ? 0 : (1 << (kSubpixelLog2 - 1)) - (1 << (kSubpixelLog2 - 1 - s)); }

// Exact sample mask of pixel (px, py) of the tile.
template <int S>
__device__ __forceinline__ U32 sampleMaskOf(const S32* E, const S32* A, const S32* B, S32 px, S32 py) {
    U32 m = 0;
#pragma unroll
    for (int i = 0; i < (1 << S); i++)
        if (edgesCover(E, A, B, (px << kSubpixelLog2) + sampleOffsetX(S, i), (py << kSubpixelLog2) + sampleOffsetY(S, i)))
            m |= 1u << i;
    return m;
}

// Steps of an edge as two signed 16-bit halves, for triangles of at most 32,767
// subpixels (2,048 pixels) across; larger ones take farEdges.
__device__ __forceinline__ bool packable(const TileEdges& t) {
    return max(t.maxX - t.minX, t.maxY - t.minY) <= 32767;
}
__device__ __forceinline__ TriRec packTri(const TileEdges& t, uint4 z, U32 id, U32 box = 0u) {
    U32 E[3], AB[3];
#pragma unroll
    for (int k = 0; k < 3; k++) {
        E[k] = (U32)(t.E[k] - 8 * (t.A[k] + t.B[k]));
        AB[k] = __byte_perm((U32)t.A[k], (U32)t.B[k], 0x5410);
    }
    return TriRec{make_uint4(E[0], E[1], E[2], AB[0]), make_uint4(AB[1], AB[2], z.x, z.y), make_uint4(z.z, id, box, 0u)};
}
// Byte pair of pixel (px, py)'s centre, and the step to sample i.
__device__ __forceinline__ S32 packedPixel(S32 px, S32 py) { return ((px | py << 8) << kSubpixelLog2) + 0x0808; }
__host__ __device__ constexpr S32 packedSample(int s, int i) { return sampleOffsetX(s, i) + 256 * sampleOffsetY(s, i); }

// Negative iff the sample at byte pair q is not covered.
__device__ __forceinline__ S32 packedEdges(uint4 r0, U32 ab1, U32 ab2, S32 q) {
    return __dp2a_lo((S32)r0.w, q, (S32)r0.x) | __dp2a_lo((S32)ab1, q, (S32)r0.y) | __dp2a_lo((S32)ab2, q, (S32)r0.z);
}
// Exact sample mask of the pixel at byte pair q.
template <int S>
__device__ __forceinline__ U32 packedMask(uint4 r0, U32 ab1, U32 ab2, S32 q) {
    U32 m = 0;
#pragma unroll
    for (int i = 0; i < (1 << S); i++)
        if (packedEdges(r0, ab1, ab2, q + packedSample(S, i)) >= 0) m |= 1u << i;
    return m;
}
// Whether the pixel can hold covered samples (exact at one sample).
template <int S>
__device__ __forceinline__ bool packedCover(uint4 r0, U32 ab1, U32 ab2, S32 q) {
    if (S == 0) return packedEdges(r0, ab1, ab2, q) >= 0;
    const U32 E[3] = {r0.x, r0.y, r0.z}, AB[3] = {r0.w, ab1, ab2};
    S32 any = 0;
#pragma unroll
    for (int k = 0; k < 3; k++)
        any |= __dp2a_lo((S32)AB[k], q, (S32)E[k]) + (abs(lo16(AB[k])) + abs(hi16(AB[k]))) * sampleReach(S);
    return any >= 0;
}
template <int S>
__device__ __forceinline__ bool edgesMayCover(const TileEdges& t, S32 px, S32 py) {
    S32 any = 0;
#pragma unroll
    for (int k = 0; k < 3; k++) {
        const S32 slack = (abs(t.A[k]) + abs(t.B[k])) * sampleReach(S);
        any |= t.E[k] + t.A[k] * (px << kSubpixelLog2) + t.B[k] * (py << kSubpixelLog2) + slack;
    }
    return any >= 0;
}

// Early Z of the visibility path. Lists come in no particular order there, so a
// triangle may be dropped only if none of its samples can win, not even a tie:
// if its lowest sample lies beyond the tile's maximum depth. The header's
// minimum is lerpError(S) = 2200 << S below the lowest vertex. Up to 2,048
// pixels across that covers the slopes' flooring to whole units per sample (at
// most half the box on each axis from its centre, where the plane is anchored:
// 2048 << S in all); the other errors stay within kZMargin: vertex depths cut
// to 24 bits (256 units) and rounded (128), the area's reciprocal (512), and in
// the anchor the cut of the gradients by 13 bits times at most 2^14 subpixels
// on each axis (8192 for the smallest area). Larger triangles are never
// dropped: their samples can lie thousands of units below the header's minimum.
constexpr U32 kZMargin = 1u << 14;
__device__ __forceinline__ U32 withZMargin(U32 z) { return z + min(kZMargin, ~z); }
// zLimit: the tile's maximum depth with the margin.
__device__ __forceinline__ bool mayWin(uint4 h, U32 zLimit) {
    if ((h.w & 0xFFFFF000u) <= zLimit) return true;
    // The extents of x and y as unsigned halves (biased, the subtraction borrows
    // nothing between them): over 32,767 subpixels?
    const U32 most = __vmaxs2(__vmaxs2(h.x, h.y), h.z) ^ 0x80008000u, least = __vmins2(__vmins2(h.x, h.y), h.z) ^ 0x80008000u;
    return ((most - least) & 0x80008000u) != 0u;
}

// Slot of a list entry's subtriangle, and the edges of a triangle that a record
// cannot hold, formed anew wherever they are needed.
__device__ __forceinline__ S64 entrySlotOf(const DrawDev& d, U32 entry) {
    const U32 tri = entry >> 3, sub = entry & 7;
    return (sub == 7) ? (S64)tri : (S64)__ldg(&d.triHeader[tri].w) + sub;
}
__device__ __forceinline__ TileEdges farEdges(const DrawDev& d, S32 listIndex, S32 cx0, S32 cy0) {
    return tileEdges(__ldg(&d.triHeader[entrySlotOf(d, __ldg(&d.tileList[listIndex]))]), cx0, cy0);
}

// 32 bytes of a triangle data slot in one load: a lane's slot is a line of its
// own, so the L1 takes a pass per lane and load (four 16-byte loads instead of
// two of these: textured terrain 453 us instead of 446, water layer 117 / 113).
__device__ __forceinline__ void loadSlot32(const uint4* p, uint4& a, uint4& b) {
    asm("ld.global.nc.v8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
        : "=r"(a.x), "=r"(a.y), "=r"(a.z), "=r"(a.w), "=r"(b.x), "=r"(b.y), "=r"(b.z), "=r"(b.w)
        : "l"(p));
}

// Depth of sample i of pixel (X, Y) (FineRaster.inl:695, 1047, 1096).
template <int S>
__device__ __forceinline__ U32 sampleDepth(U32 zx, U32 zy, U32 zb, U32 X, U32 Y, int i) {
    if (S == 0) return zx * X + zy * Y + zb;
    return zx * (U32)msaaPatternX(S, i) + zy * (U32)i + (((zx * X + zy * Y) << S) + zb);
}

// Pixel box [bx0, bx1] x [by0, by1] of the tile that can hold covered samples:
// the pixels whose samples' box meets the vertices' (padded by half a pixel, the
// 8.4M-triangle heightfield took 606 us at 4x MSAA instead of 577, and a
// textured one at 1080p 872 instead of 727).
template <int S>
__device__ __forceinline__ bool pixelBox(const TileEdges& t, S32& bx0, S32& bx1, S32& by0, S32& by1) {
    constexpr S32 pad = sampleReach(S);
    bx0 = max(0, (t.minX - pad + 15) >> kSubpixelLog2);
    bx1 = min(7, (t.maxX + pad) >> kSubpixelLog2);
    by0 = max(0, (t.minY - pad + 15) >> kSubpixelLog2);
    by1 = min(7, (t.maxY + pad) >> kSubpixelLog2);
    return bx0 <= bx1 && by0 <= by1;
}

// A small triangle's pixel box as bx0 | by0 << 4 | w << 8 | m << 12, where
// m = ceil(2^8 / w) gives the row of the box's pixel k as (k * m) >> 8, exact
// for k < 64 and w <= 8 (the error k * (m * w - 256) stays below 256). m - 1
// comes from a table in two registers, since a division takes some 20
// instructions.
__device__ __forceinline__ U32 packBox(S32 bx0, S32 by0, S32 w) {
    const U32 m = (__byte_perm(0x3F557FFFu, 0x1F242A33u, (U32)(w - 1)) & 0xFFu) + 1u;
    return (U32)bx0 | (U32)by0 << 4 | (U32)w << 8 | m << 12;
}
__device__ __forceinline__ void boxPixel(U32 box, S32 k, S32& px, S32& py) {
    const S32 q = (S32)(((U32)k * (box >> 12)) >> 8);
    px = (S32)(box & 0xFu) + k - q * (S32)((box >> 8) & 0xFu);
    py = (S32)((box >> 4) & 0xFu) + q;
}

// Pairs of a batch's small triangles, dealt to the lanes 32 a pass: a triangle
// whose first pair is `start` (-1: it has none) marks it, and pair base + lane
// belongs to the last one marked at or before it. Returns that one's turn among
// the small triangles; `before` counts those of the passes so far. Passing the
// start's lane through shared memory and the carried one by shuffles took the
// stage 80 us instead of 78 on the 1M soup, 262 / 258 on the 33.5M-triangle
// terrain and 178 / 174 on a 2x MSAA heightfield. The ordered path keeps its
// forms: there the textured terrain took 457 us with this one, 449 without.
__device__ __forceinline__ S32 turnOf(S32 start, S32 base, S32& before) {
    const U32 at = (U32)(start - base);
    const U32 marks = __reduce_or_sync(0xFFFFFFFFu, at < 32u ? 1u << at : 0u);
    const S32 turn = before + __popc(marks & (0xFFFFFFFFu >> (31 - (threadIdx.x & 31)))) - 1;
    before += __popc(marks);
    return turn;
}

// Runs the fragment shader of triangle data td (16 words) at pixel (X, Y).
template <class FS, int S, U32 F>
__device__ __forceinline__ U32 shadeFragment(const U32* td, S32 triIdx, S32 X, S32 Y, U32 sampleMask,
                                             const float4* verts, S32 stride4, volatile F32* shared, U32 laneMask,
                                             bool& discard) {
    FS fs;
    fs.m_triIdx = triIdx;
    fs.m_vertIdx = FW::Vec3i((S32)td[13], (S32)td[14], (S32)td[15]);
    fs.m_pixelPos = FW::Vec2i(X, Y);
    fs.m_vertexBytes = stride4 * 16;
    fs.m_shared = shared;
    fs.m_vertices = verts;
    fs.m_laneMask = laneMask;
    fs.m_color = 0xFF0000FFu;
    fs.m_discard = false;
    if (!(F & kRenderLerp)) {
        // Interpolation disabled => varyings at the last vertex (FineRaster.inl:71-81).
        fs.m_center = FW::Vec3f(0.0f, 0.0f, 1.0f);
        fs.m_centerDX = FW::Vec3f(0.0f);
        fs.m_centerDY = FW::Vec3f(0.0f);
        fs.m_centroid = fs.m_center;
        fs.m_centroidDX = fs.m_centerDX;
        fs.m_centroidDY = fs.m_centerDY;
    } else {
        using Reads = FW::FragmentShaderReads<FS>;
        if (Reads::center || (S == 0 && Reads::centroid))
            computeBarys<S>(fs.m_center, fs.m_centerDX, fs.m_centerDY, td + 4, td + 7, td + 10, (X * 2 + 1) << S,
                            (Y * 2 + 1) << S);
        if (S == 0) {
            fs.m_centroid = fs.m_center;
            fs.m_centroidDX = fs.m_centerDX;
            fs.m_centroidDY = fs.m_centerDY;
        } else if (Reads::centroid) {
            U32 c = centroidCode(S, sampleMask);
            computeBarys<S>(fs.m_centroid, fs.m_centroidDX, fs.m_centroidDY, td + 4, td + 7, td + 10,
                            (X << (S + 1)) + (S32)(c & 0xF), (Y << (S + 1)) + (S32)(c >> 4));
        }
    }
    fs.run();
    discard = fs.m_discard;
    return fs.m_color;
}

template <class V, class FS, class BS, int S, U32 F>
__device__ __forceinline__ void fineTiles(const DrawDev& d, int group, S32 tileBegin, S32 tileEnd) {
    constexpr int NS = 1 << S;
    constexpr int TW = 64 << S;
    using Traits = FineTraits<FS, BS, S, F>;
    constexpr bool kDepth = Traits::kDepth;
    constexpr bool kQuads = Traits::kQuads;
    constexpr bool kVisibility = Traits::kVisibility;
    extern __shared__ __align__(16) unsigned char fineSmemRaw[];
    typename Traits::Smem& sm = reinterpret_cast<typename Traits::Smem*>(fineSmemRaw)[threadIdx.x >> 5];
    const int lane = threadIdx.x & 31;
    const U32 ltMask = (1u << lane) - 1u;
    pdlWait();
    pdlTrigger();
    if (d.hostCounters != nullptr && blockIdx.x == 0 && threadIdx.x < (int)(sizeof(Counters) / 4)) {
        U32 word = reinterpret_cast<const volatile U32*>(d.counters)[threadIdx.x];
        // The last two words: when this stage began (see markStage).
        if (d.stageTiming && threadIdx.x >= (int)(sizeof(Counters) / 4) - 2) {
            const U64 t = globalNanoseconds();
            word = threadIdx.x & 1 ? (U32)(t >> 32) : (U32)t;
        }
        reinterpret_cast<volatile U32*>(d.hostCounters)[threadIdx.x] = word;
    }
    if (__ldg(&d.counters->overflow)) return;
    const S32 selfPixels = d.fineSelfPixels > 0 ? d.fineSelfPixels : fineSelfPixelsDefault(S, kVisibility);

    // A warp's tiles come from the counter in increasing order: its current
    // instance stays valid until a tile reaches the next instance's first.
    int ii = 0;
    S32 instEnd = -1;
    for (;;) {
        S32 tile = 0;
        if (lane == 0) tile = atomicAdd(&d.fineTileCounter[group], 1);
        tile = __shfl_sync(0xFFFFFFFFu, tile, 0) + tileBegin;
        if (tile >= tileEnd) break;

        if (tile >= instEnd) {
            ii = findInstance(d.tilePrefix, d.numInstances, tile);
            instEnd = __ldg(&d.tilePrefix[ii + 1]);   // the prefix has numInstances + 1 entries
        }
        const InstanceDev* in = &d.inst[ii];
        const S32 wt = __ldg(&in->widthTiles);
        const S32 lt = tile - __ldg(&in->tileBase);
        const S32 tx = lt % wt, ty = lt / wt;
        const S32 count = __ldg(&d.tileCount[tile]);
        const S32 start = __ldg(&d.tileStart[tile]);
        const bool clear = __ldg(&in->deferredClear) != 0;
        if (count == 0 && !clear) continue;

        const S32 width = __ldg(&in->width), height = __ldg(&in->height);
        const S64 rowWords = __ldg(&in->rowWords);
        U32* gColor = (U32*)__ldg((const unsigned long long*)&in->color);
        U32* gDepth = (U32*)__ldg((const unsigned long long*)&in->depth);
        const S64 tileOrigin = (S64)(ty * 8) * rowWords + (S64)tx * 8 * NS;

        // The tile's words move two per lane and step, 64 words (8 / NS rows) a
        // step, where the surfaces allow 8-byte accesses; one by one otherwise.
        const bool wide = (((U64)gColor | (U64)gDepth) & 7u) == 0;
        const S64 wideOrigin = tileOrigin + (S64)(lane / (4 * NS)) * rowWords + 2 * (lane % (4 * NS));
        const S64 wideStep = (8 / NS) * rowWords;
        if (count == 0) {
            // A cleared tile that no triangle touches.
            const U32 cc = __ldg(&in->clearColor), cd = __ldg(&in->clearDepth);
            if (wide) {
#pragma unroll
                for (int i = 0; i < NS; i++) {
                    *reinterpret_cast<uint2*>(&gColor[wideOrigin + i * wideStep]) = make_uint2(cc, cc);
                    *reinterpret_cast<uint2*>(&gDepth[wideOrigin + i * wideStep]) = make_uint2(cd, cd);
                }
            } else {
                for (int w = lane; w < TW; w += 32) {
                    const S64 g = tileOrigin + (S64)(w / (8 * NS)) * rowWords + (w % (8 * NS));
                    gColor[g] = cc;
                    gDepth[g] = cd;
                }
            }
            continue;
        }

        // Load or clear the tile (FineRaster.inl:562-580, 916-934), and its
        // maximum depth for early Z. Visibility keys start as depth << 32 (no
        // fragment yet).
        U32 tileZMax = 0;
        auto putDepth = [&](int w, U32 z) {
            if constexpr (kVisibility) sm.key[w] = (U64)z << 32; else sm.depth[w] = z;
        };
        if (clear) {
            const U32 cc = __ldg(&in->clearColor), cd = __ldg(&in->clearDepth);
#pragma unroll
            for (int w = lane; w < TW; w += 32) {
                sm.color[w] = cc;
                putDepth(w, cd);
            }
            tileZMax = cd;
        } else {
            U32 z = 0;
            if (wide) {
#pragma unroll
                for (int i = 0; i < NS; i++) {
                    const int w = 2 * lane + 64 * i;
                    const uint2 c = *reinterpret_cast<const uint2*>(&gColor[wideOrigin + i * wideStep]);
                    const uint2 dz = *reinterpret_cast<const uint2*>(&gDepth[wideOrigin + i * wideStep]);
                    *reinterpret_cast<uint2*>(&sm.color[w]) = c;
                    putDepth(w, dz.x);
                    putDepth(w + 1, dz.y);
                    z = max(z, max(dz.x, dz.y));
                }
            } else {
                for (int w = lane; w < TW; w += 32) {
                    const S64 g = tileOrigin + (S64)(w / (8 * NS)) * rowWords + (w % (8 * NS));
                    sm.color[w] = gColor[g];
                    const U32 dz = gDepth[g];
                    putDepth(w, dz);
                    z = max(z, dz);
                }
            }
            if (kDepth) tileZMax = __reduce_max_sync(0xFFFFFFFFu, z);
        }
        __syncwarp();

        // Pixel (0, 0) centre of the tile in the header frame.
        const S32 cx0 = ((tx * 8) << kSubpixelLog2) - ((width - 1) << (kSubpixelLog2 - 1));
        const S32 cy0 = ((ty * 8) << kSubpixelLog2) - ((height - 1) << (kSubpixelLog2 - 1));
        const S64 triBase = __ldg(&in->triBase);
        const S32 stride4 = __ldg(&in->stride4);
        const float4* verts = (const float4*)__ldg((const unsigned long long*)&in->vertices);

        // Visibility keys: depth << 32 | order, order = list entry within the
        // scene + 1; with MSAA the low word also carries the winner's coverage
        // mask of the pixel (order << NS | mask) where the scene's entries
        // leave room for it (at 4 samples, up to 2^25 triangles).
        const U32 entryBase = (U32)triBase << 3;
        const bool packed = S != 0 && (U32)__ldg(&in->numTris) <= (1u << (S != 0 ? 29 - NS : 0)) - 1u;

        for (S32 batch = 0; batch < count; batch += 32) {
            if constexpr (kVisibility) {
                // ---- Visibility. Every (triangle, pixel) pair of the batch's
                // triangles whose pixel box has at most selfPixels pixels is
                // dealt to the lanes in turn, 32 pairs a pass (turnOf); the
                // pair's pixel follows by an exact multiply-shift division by
                // the box width (a lane walking its own triangle's box
                // measured slower, even for boxes of one or two pixels);
                // larger triangles are rasterized by the whole warp, two
                // pixels per lane. Keys resolve by atomic minimum, so the
                // order pairs are taken in does not change a bit.
                S32 n = 0;
                U32 box = 0;
                bool big = false, far = false;
                const U32 zLimit = withZMargin(tileZMax);
                if (batch + lane < count) {
                    const U32 entry = __ldg(&d.tileList[start + batch + lane]);
                    const S64 slot = entrySlotOf(d, entry);
                    const uint4 h = __ldg(&d.triHeader[slot]);
                    if (mayWin(h, zLimit)) {
                        const TileEdges te = tileEdges(h, cx0, cy0);
                        S32 bx0, bx1, by0, by1;
                        if (pixelBox<S>(te, bx0, bx1, by0, by1)) {
                            const uint4 q0 = __ldg(&d.triData[slot * 4]);
                            const S32 w = bx1 - bx0 + 1;
                            const S32 cnt = w * (by1 - by0 + 1);
                            far = !packable(te);
                            big = !far && cnt > selfPixels;
                            if (!far && !big) n = cnt;
                            box = packBox(bx0, by0, w);
                            sm.rec[lane] = packTri(te, q0, entry - entryBase + 1u);
                        }
                    }
                }
                S32 P = 0, myStart = -1;
                const U32 smallMask = __ballot_sync(0xFFFFFFFFu, n > 0);
                if (smallMask) {
                    S32 incl = n;
#pragma unroll
                    for (int o = 1; o < 32; o <<= 1) {
                        const S32 t = __shfl_up_sync(0xFFFFFFFFu, incl, o);
                        if (lane >= o) incl += t;
                    }
                    P = __shfl_sync(0xFFFFFFFFu, incl, 31);
                    if (n > 0) {
                        myStart = incl - n;
                        sm.turn[__popc(smallMask & ltMask)] = make_uint2(box, (U32)lane << 16 | (U32)myStart);
                    }
                }
                __syncwarp();
                S32 before = 0;
                for (S32 base = 0; base < P; base += 32) {
                    const S32 turn = turnOf(myStart, base, before);
                    const S32 p = base + lane;
                    if (p >= P) continue;
                    const uint2 who = sm.turn[turn];
                    const int j = (int)(who.y >> 16);
                    S32 px, py;
                    boxPixel(who.x, p - (S32)(who.y & 0xFFFFu), px, py);
                    const uint4 r0 = sm.rec[j].q[0], r1 = sm.rec[j].q[1];
                    const U32 smask = packedMask<S>(r0, r1.x, r1.y, packedPixel(px, py));
                    if (!smask) continue;
                    const uint2 r2 = *reinterpret_cast<const uint2*>(&sm.rec[j].q[2]);
                    const U32 order = r2.y;
                    const U64 low = packed ? (order << NS | smask) : order;
                    const U32 X = (U32)(tx * 8 + px), Y = (U32)(ty * 8 + py);
                    const U32 zx = r1.z, zy = r1.w, zb = r2.x;
#pragma unroll
                    for (int i = 0; i < NS; i++) {
                        if (!(smask >> i & 1)) continue;
                        const int idx = py * 8 * NS + i * 8 + px;
                        const U64 key = ((U64)sampleDepth<S>(zx, zy, zb, X, Y, i) << 32) | low;
                        if (key < sm.key[idx]) atomicMin((unsigned long long*)&sm.key[idx], (unsigned long long)key);
                    }
                }
                __syncwarp();
                // Larger triangles: the whole warp, one at a time, in batch
                // order (each lane owns its two pixels, so plain stores
                // suffice). At one sample a lane keeps its two keys in
                // registers over all of them; the row below is 4 pixels down.
                const S32 px = lane & 7, py0 = lane >> 3, py1 = py0 + 4;
                const U32 pX = (U32)(tx * 8 + px), pY0 = (U32)(ty * 8 + py0), pY1 = pY0 + 4;
                const S32 pq0 = packedPixel(px, py0), pq1 = packedPixel(px, py1);
                U32 bigMask = __ballot_sync(0xFFFFFFFFu, big);
                if (S == 0 && bigMask) {
                    const int idx0 = py0 * 8 + px, idx1 = idx0 + 32;
                    U64 k0 = sm.key[idx0], k1 = sm.key[idx1];
                    for (; bigMask; bigMask &= bigMask - 1) {
                        const int j = __ffs(bigMask) - 1;
                        const uint4 r0 = sm.rec[j].q[0], r1 = sm.rec[j].q[1];
                        const uint2 r2 = *reinterpret_cast<const uint2*>(&sm.rec[j].q[2]);
                        const U32 z0 = r1.z * pX + r1.w * pY0 + r2.x, z1 = z0 + (r1.w << 2);
                        const U64 key0 = ((U64)z0 << 32) | r2.y, key1 = ((U64)z1 << 32) | r2.y;
                        if (packedEdges(r0, r1.x, r1.y, pq0) >= 0 && key0 < k0) k0 = key0;
                        if (packedEdges(r0, r1.x, r1.y, pq1) >= 0 && key1 < k1) k1 = key1;
                    }
                    sm.key[idx0] = k0;
                    sm.key[idx1] = k1;
                }
                auto lowerKeys = [&](U32 smask, S32 pyy, U32 Y, U32 zx, U32 zy, U32 zb, U32 order) {
                    const U64 low = packed ? (order << NS | smask) : order;
#pragma unroll
                    for (int i = 0; i < NS; i++) {
                        if (!(smask >> i & 1)) continue;
                        const int idx = pyy * 8 * NS + i * 8 + px;
                        const U64 key = ((U64)sampleDepth<S>(zx, zy, zb, pX, Y, i) << 32) | low;
                        if (key < sm.key[idx]) sm.key[idx] = key;
                    }
                };
                for (; bigMask; bigMask &= bigMask - 1) {
                    const int j = __ffs(bigMask) - 1;
                    const uint4 r0 = sm.rec[j].q[0], r1 = sm.rec[j].q[1];
                    const uint2 r2 = *reinterpret_cast<const uint2*>(&sm.rec[j].q[2]);
#pragma unroll 1
                    for (int half = 0; half < 2; half++)
                        lowerKeys(packedMask<S>(r0, r1.x, r1.y, half ? pq1 : pq0), half ? py1 : py0, half ? pY1 : pY0, r1.z,
                                  r1.w, r2.x, r2.y);
                }
                // Those whose steps a record cannot hold (over 2,048 pixels across).
                for (U32 farMask = __ballot_sync(0xFFFFFFFFu, far); farMask; farMask &= farMask - 1) {
                    const int j = __ffs(farMask) - 1;
                    const TileEdges te = farEdges(d, start + batch + j, cx0, cy0);
                    const uint4 r1 = sm.rec[j].q[1], r2 = sm.rec[j].q[2];
#pragma unroll 1
                    for (int half = 0; half < 2; half++) {
                        const S32 py = half ? py1 : py0;
                        lowerKeys(sampleMaskOf<S>(te.E, te.A, te.B, px, py), py, half ? pY1 : pY0, r1.z, r1.w, r2.x, r2.y);
                    }
                }
                __syncwarp();
                // Exact current depth maximum for the next batch's early Z.
                if (batch + 32 < count) {
                    U32 z = 0;
#pragma unroll
                    for (int w = 2 * lane; w < TW; w += 64) {
                        const ulonglong2 k = *reinterpret_cast<const ulonglong2*>(&sm.key[w]);
                        z = max(z, max((U32)(k.x >> 32), (U32)(k.y >> 32)));
                    }
                    tileZMax = __reduce_max_sync(0xFFFFFFFFu, z);
                }
            } else {
                // ---- 1. One triangle per lane: its words in shared memory, and
                // the pixels of the small ones (box of at most selfPixels pixels)
                // as (triangle, pixel) pairs dealt over the lanes, each setting
                // the triangle's coverage bit of its pixel (the masks do not
                // depend on the order the pairs are taken in).
                bool valid = batch + lane < count;
                bool self = false;     // small triangle: covered through the pairs
                bool far = false;      // its steps do not fit a record
                U32 myLo = 0, myHi = 0;
                S32 n = 0;
                sm.covLo[lane] = 0u;
                sm.covHi[lane] = 0u;
                // Batch filter (see step 2b): exact for single-sample depth-tested
                // pipes whose fragment shader never discards.
                constexpr bool kFilter = S == 0 && kDepth && !kQuads && !FW::FragmentShaderTraits<FS>::mayDiscard;
                if constexpr (kFilter) {
                    sm.batchMin[lane] = ~0ull;
                    sm.batchMin[lane + 32] = ~0ull;
                }
                if (valid) {
                    U32 entry = __ldg(&d.tileList[start + batch + lane]);
                    const U32 tri = entry >> 3;
                    const S64 slot = entrySlotOf(d, entry);
                    uint4 h = __ldg(&d.triHeader[slot]);
                    if (kDepth && (h.w & 0xFFFFF000u) >= tileZMax) valid = false;
                    if (valid) {
                        const TileEdges te = tileEdges(h, cx0, cy0);
                        const uint4* tdp = &d.triData[slot * 4];
                        uint4 q0, q1, q2, q3;
                        loadSlot32(tdp, q0, q1);
                        loadSlot32(tdp + 2, q2, q3);
                        S32 bx0, bx1, by0, by1;
                        const bool inTile = pixelBox<S>(te, bx0, bx1, by0, by1);
                        const S32 w = bx1 - bx0 + 1;
                        far = inTile && !packable(te);
                        self = !inTile || (!far && w * (by1 - by0 + 1) <= selfPixels);
                        sm.rec[lane] = packTri(te, q0, (U32)((S64)tri - triBase), inTile ? packBox(bx0, by0, w) : 0u);
                        sm.data[lane] = TriRec{q1, q2, q3};
                        // No pixel of the tile can be covered (!inTile): nothing to do.
                        if (inTile && self) n = w * (by1 - by0 + 1);
                    }
                }
                S32 P = 0;
                if (__any_sync(0xFFFFFFFFu, n > 0)) {
                    S32 incl = n;
#pragma unroll
                    for (int o = 1; o < 32; o <<= 1) {
                        const S32 t = __shfl_up_sync(0xFFFFFFFFu, incl, o);
                        if (lane >= o) incl += t;
                    }
                    sm.fragEnd[lane] = incl;
                    P = __shfl_sync(0xFFFFFFFFu, incl, 31);
                }
                __syncwarp();
                for (S32 base = 0; base < P; base += 32) {
                    const S32 p = base + lane;
                    if (p >= P) continue;
                    int j = 0;
#pragma unroll
                    for (int s2 = 16; s2 > 0; s2 >>= 1)
                        if (sm.fragEnd[j + s2 - 1] <= p) j += s2;
                    const S32 k = p - (j ? sm.fragEnd[j - 1] : 0);
                    S32 px, py;
                    boxPixel(sm.rec[j].q[2].z, k, px, py);
                    const uint4 r0 = sm.rec[j].q[0];
                    const uint2 ab = *reinterpret_cast<const uint2*>(&sm.rec[j].q[1]);
                    bool c = packedCover<S>(r0, ab.x, ab.y, packedPixel(px, py));
                    if (kDepth && S == 0 && !kQuads && c) {
                        const U32 X = (U32)(tx * 8 + px), Y = (U32)(ty * 8 + py);
                        const uint2 zxy = *reinterpret_cast<const uint2*>(&sm.rec[j].q[1].z);
                        const U32 z = zxy.x * X + zxy.y * Y + sm.rec[j].q[2].x;
                        c = z < sm.depth[py * 8 + px];
                        if constexpr (kFilter)
                            if (c) atomicMin((unsigned long long*)&sm.batchMin[py * 8 + px], ((unsigned long long)z << 32) | (U32)j);
                    }
                    if (c) {
                        const int bit = py * 8 + px;
                        atomicOr(bit < 32 ? &sm.covLo[j] : &sm.covHi[j], 1u << (bit & 31));
                    }
                }
                __syncwarp();
                if (self) {
                    myLo = sm.covLo[lane];
                    myHi = sm.covHi[lane];
                }
                U64 min0 = 0, min1 = 0;   // batch minima of this lane's pixels (lane, lane + 32)
                if constexpr (kFilter) {
                    min0 = sm.batchMin[lane];
                    min1 = sm.batchMin[lane + 32];
                }
                __syncwarp();
                const U32 coopMask = __ballot_sync(0xFFFFFFFFu, valid && !self);
                const U32 farMask = __ballot_sync(0xFFFFFFFFu, valid && far);

                // ---- 2. Large triangles, two pixels per lane.
                const S32 px = lane & 7, py0 = lane >> 3, py1 = py0 + 4;
                const U32 pX = (U32)(tx * 8 + px), pY0 = (U32)(ty * 8 + py0);
                {
                    // Single-sample depth of this lane's two pixels at the start of
                    // the batch: a fragment that fails against it fails in
                    // submission order too (depths only decrease).
                    U32 curZ0 = 0, curZ1 = 0;
                    if (kDepth && S == 0 && !kQuads) {
                        curZ0 = sm.depth[lane];
                        curZ1 = sm.depth[lane + 32];
                    }
                    const S32 pq0 = packedPixel(px, py0), pq1 = packedPixel(px, py1);
                    auto setCoverage = [&](int j, bool c0, bool c1, U32 zx, U32 zy) {
                        if (kDepth && S == 0 && !kQuads) {
                            const U32 z0 = zx * pX + zy * pY0 + sm.rec[j].q[2].x, z1 = z0 + zy * 4u;
                            c0 = c0 && (z0 < curZ0);
                            c1 = c1 && (z1 < curZ1);
                            if constexpr (kFilter) {
                                const U64 k0 = ((U64)z0 << 32) | (U32)j, k1 = ((U64)z1 << 32) | (U32)j;
                                if (c0 && k0 < min0) min0 = k0;
                                if (c1 && k1 < min1) min1 = k1;
                            }
                        }
                        const U32 lo = __ballot_sync(0xFFFFFFFFu, c0);
                        const U32 hi = __ballot_sync(0xFFFFFFFFu, c1);
                        if (lane == j) { myLo = lo; myHi = hi; }
                    };
                    for (U32 m = coopMask & ~farMask; m; m &= m - 1) {
                        const int j = __ffs(m) - 1;
                        const uint4 r0 = sm.rec[j].q[0], r1 = sm.rec[j].q[1];
                        setCoverage(j, packedCover<S>(r0, r1.x, r1.y, pq0), packedCover<S>(r0, r1.x, r1.y, pq1), r1.z, r1.w);
                    }
                    for (U32 m = farMask; m; m &= m - 1) {
                        const int j = __ffs(m) - 1;
                        const TileEdges te = farEdges(d, start + batch + j, cx0, cy0);
                        const uint2 zxy = *reinterpret_cast<const uint2*>(&sm.rec[j].q[1].z);
                        setCoverage(j, edgesMayCover<S>(te, px, py0), edgesMayCover<S>(te, px, py1), zxy.x, zxy.y);
                    }
                }
                if (kQuads) {
                    // quadCoverage (FineRaster.inl:401-406): bit of the quad's top-left pixel.
                    U64 c = ((U64)myHi << 32) | myLo;
                    c |= c >> 1;
                    c |= c >> 8;
                    c &= 0x0055005500550055ull;
                    myLo = (U32)c;
                    myHi = (U32)(c >> 32);
                }
                if constexpr (kFilter) {
                    // ---- 2b. A fragment of pixel p later in the batch than p's
                    // minimum (depth, then batch position) fails the in-order LESS
                    // test: the minimum's own fragment passes (every earlier one is
                    // deeper) and leaves the depth at or below the later one's, and
                    // without discard nothing else changes it. Triangle j keeps
                    // the pixels whose minimum is at j or later: a bit-sliced
                    // comparison of the 5-bit positions (10 ballots) against j.
                    const U32 w0 = min((U32)min0, 31u), w1 = min((U32)min1, 31u);
                    U32 gtLo = 0u, eqLo = ~0u, gtHi = 0u, eqHi = ~0u;
#pragma unroll
                    for (int b = 4; b >= 0; b--) {
                        const U32 pl = __ballot_sync(0xFFFFFFFFu, (w0 >> b) & 1u);
                        const U32 ph = __ballot_sync(0xFFFFFFFFu, (w1 >> b) & 1u);
                        const U32 jb = 0u - (((U32)lane >> b) & 1u);   // bit b of this lane's triangle j
                        gtLo |= eqLo & pl & ~jb;
                        eqLo &= ~(pl ^ jb);
                        gtHi |= eqHi & ph & ~jb;
                        eqHi &= ~(ph ^ jb);
                    }
                    myLo &= gtLo | eqLo;
                    myHi &= gtHi | eqHi;
                }
                if (!valid) { myLo = 0; myHi = 0; }

                // ---- 3. Fragment compaction in submission order.
                const S32 pop = (__popc(myLo) + __popc(myHi)) * (kQuads ? 4 : 1);
                S32 inc = pop;
#pragma unroll
                for (int o = 1; o < 32; o <<= 1) {
                    S32 t = __shfl_up_sync(0xFFFFFFFFu, inc, o);
                    if (lane >= o) inc += t;
                }
                const S32 myFragStart = inc - pop;
                S32 fragCarryJ = 0, fragCarryStart = 0;   // triangle (and its first fragment) of the last fragment so far
                sm.covLo[lane] = myLo;
                sm.covHi[lane] = myHi;
                const S32 total = __shfl_sync(0xFFFFFFFFu, inc, 31);
                __syncwarp();

                for (S32 pass = 0; pass < total; pass += 32) {
                    const S32 f = pass + lane;
                    bool act = f < total;
                    int j = 0, pixel = 0;
                    bool covered = false;
                    U32 sampleMask = 0;
                    U32 dz[NS];
                    // Triangle of fragment f: the last one whose fragments start
                    // at or before f (one OR over the warp marks the pass's
                    // starts; the triangle of the previous pass's last fragment
                    // carries over).
                    const bool startsHere = pop > 0 && myFragStart >= pass && myFragStart < pass + 32;
                    if (startsHere) sm.fragHead[myFragStart - pass] = lane;
                    const U32 startMask = __reduce_or_sync(0xFFFFFFFFu, startsHere ? 1u << (myFragStart - pass) : 0u);
                    __syncwarp();
                    const U32 upTo = startMask & (0xFFFFFFFFu >> (31 - lane));
                    int fragJ = fragCarryJ;
                    S32 fragFirst = fragCarryStart;
                    if (upTo) {
                        const int h = 31 - __clz(upTo);
                        fragJ = sm.fragHead[h];
                        fragFirst = pass + h;
                    }
                    fragCarryJ = __shfl_sync(0xFFFFFFFFu, fragJ, 31);
                    fragCarryStart = __shfl_sync(0xFFFFFFFFu, fragFirst, 31);
                    __syncwarp();   // every lane has read fragHead before the next pass rewrites it
                    if (act) {
                        j = fragJ;
                        const U32 cl = sm.covLo[j], ch = sm.covHi[j];
                        const S32 k = f - fragFirst;
                        if (kQuads) {
                            int qbit = nthSetBit64(cl, ch, k >> 2);
                            pixel = qbit + (k & 1) + ((k & 2) << 2);  // findFragment, FineRaster.inl:417-427
                        } else {
                            pixel = nthSetBit64(cl, ch, k);
                        }
                        const S32 fx = pixel & 7, fy = pixel >> 3;
                        if (S == 0 && !kQuads) {
                            sampleMask = 1;  // single-sample masks are exact
                        } else {
                            const uint4 r0 = sm.rec[j].q[0], r1 = sm.rec[j].q[1];
                            if (farMask >> j & 1u) {
                                const TileEdges te = farEdges(d, start + batch + j, cx0, cy0);
                                sampleMask = sampleMaskOf<S>(te.E, te.A, te.B, fx, fy);
                            } else {
                                sampleMask = packedMask<S>(r0, r1.x, r1.y, packedPixel(fx, fy));
                            }
                        }
                        covered = sampleMask != 0;
                        if (!kQuads && !covered) act = false;
                        const U32 X = (U32)(tx * 8 + fx), Y = (U32)(ty * 8 + fy);
                        if (kDepth) {
                            const uint2 r1 = *reinterpret_cast<const uint2*>(&sm.rec[j].q[1].z);
                            const U32 zx = r1.x, zy = r1.y, zb = sm.rec[j].q[2].x;
                            bool anyPass = false;
                            const int rowBase = fy * 8 * NS + fx;
#pragma unroll
                            for (int i = 0; i < NS; i++) {
                                dz[i] = sampleDepth<S>(zx, zy, zb, X, Y, i);
                                if ((sampleMask >> i & 1) && dz[i] < sm.depth[rowBase + i * 8]) anyPass = true;
                            }
                            if (!kQuads && !anyPass) act = false;
                            if (kQuads && !anyPass) covered = false;
                        }
                    }
                    // Shade.
                    const U32 shadeMask = __ballot_sync(0xFFFFFFFFu, act);
                    U32 src = 0;
                    bool discard = true;
                    if (act) {
                        U32 td[16];
#pragma unroll
                        for (int q = 0; q < 3; q++) {
                            const uint4 v = sm.data[j].q[q];
                            td[4 + 4 * q] = v.x; td[5 + 4 * q] = v.y; td[6 + 4 * q] = v.z; td[7 + 4 * q] = v.w;
                        }
                        src = shadeFragment<FS, S, F>(td, (S32)sm.rec[j].q[2].y, tx * 8 + (pixel & 7), ty * 8 + (pixel >> 3), sampleMask,
                                                      verts, stride4, sm.shared, shadeMask, discard);
                    }
                    // ROP: same-pixel fragments of this pass applied in lane order.
                    const bool rop = act && covered && !discard;
                    const U32 ropMask = __ballot_sync(0xFFFFFFFFu, rop);
                    if (ropMask) {
                        U32 peers = 0;
                        if (rop) peers = __match_any_sync(ropMask, pixel);
                        const int rank = __popc(peers & ltMask);
                        const int maxGroup = __reduce_max_sync(0xFFFFFFFFu, rop ? __popc(peers) : 0);
                        for (int r = 0; r < maxGroup; r++) {
                            if (rop && rank == r) {
                                const S32 fx = pixel & 7, fy = pixel >> 3;
                                const int rowBase = fy * 8 * NS + fx;
                                BS bs;
#pragma unroll
                                for (int i = 0; i < NS; i++) {
                                    if (!(sampleMask >> i & 1)) continue;
                                    const int idx = rowBase + i * 8;
                                    if (kDepth) {
                                        if (!(dz[i] < sm.depth[idx])) continue;
                                        sm.depth[idx] = dz[i];
                                    }
                                    bs.m_triIdx = (S32)sm.rec[j].q[2].y;
                                    bs.m_pixelPos = FW::Vec2i(tx * 8 + fx, ty * 8 + fy);
                                    bs.m_sampleIdx = i;
                                    bs.m_src = src;
                                    bs.m_dst = sm.color[idx];
                                    bs.m_color = 0xFF0000FFu;
                                    bs.m_writeColor = true;
                                    bs.run();
                                    if (bs.m_writeColor) sm.color[idx] = bs.m_color;
                                }
                            }
                            __syncwarp();
                        }
                    }
                }
                if (kDepth && batch + 32 < count) {
                    U32 z = 0;
                    for (int w = lane; w < TW; w += 32) z = max(z, sm.depth[w]);
                    tileZMax = __reduce_max_sync(0xFFFFFFFFu, z);
                }
                __syncwarp();
            }
        }

        if constexpr (kVisibility) {
            // ---- Resolve: shade every (pixel, winning triangle) once. Sample
            // i0 of a pixel starts a winner if no earlier sample of the pixel
            // has the same key low word (with MSAA the low word carries the
            // winner's coverage mask, so neither its edges nor its mask are
            // recomputed here). The winners of the tile are listed first (a
            // lane owns pixels lane and lane + 32), then fetched and shaded
            // 32 at a time, so lanes stay busy however unevenly the winners
            // fall on the pixels and samples.
            U32* winners = sm.winners;
            S32 nw = 0;
#pragma unroll
            for (int hh = 0; hh < 2; hh++) {
                const int p = lane + 32 * hh;
                const int rowBase = (p >> 3) * 8 * NS + (p & 7);
#pragma unroll
                for (int i0 = 0; i0 < NS; i0++) {
                    const U32 low = (U32)sm.key[rowBase + i0 * 8];
                    bool first = low != 0;
#pragma unroll
                    for (int i = 0; i < i0; i++)
                        if ((U32)sm.key[rowBase + i * 8] == low) first = false;
                    const U32 firsts = __ballot_sync(0xFFFFFFFFu, first);
                    if (first) {
                        U32 won = 0;
#pragma unroll
                        for (int i = 0; i < NS; i++)
                            if ((U32)sm.key[rowBase + i * 8] == low) won |= 1u << i;
                        winners[nw + __popc(firsts & ltMask)] = (U32)p | (U32)i0 << 6 | won << 9;
                    }
                    nw += __popc(firsts);
                }
            }
            __syncwarp();
            for (S32 w0 = 0; w0 < nw; w0 += 32) {
                if (w0 + lane >= nw) continue;
                const U32 rec = winners[w0 + lane];
                const int p = (int)(rec & 63u), i0 = (int)((rec >> 6) & 7u);
                const U32 won = rec >> 9;
                const S32 px = p & 7, py = p >> 3;
                const int rowBase = py * 8 * NS + px;
                U32 low = (U32)sm.key[rowBase + i0 * 8];
                U32 td[16];
                const U32 entry = (packed ? low >> NS : low) - 1u + entryBase;
                const U32 tri = entry >> 3;
                const S64 slot = entrySlotOf(d, entry);
                const uint4* tdp = &d.triData[slot * 4];
                uint4 q0, q1, q2, q3;
                loadSlot32(tdp, q0, q1);
                loadSlot32(tdp + 2, q2, q3);
                td[4] = q1.x; td[5] = q1.y; td[6] = q1.z; td[7] = q1.w;
                td[8] = q2.x; td[9] = q2.y; td[10] = q2.z; td[11] = q2.w;
                td[12] = q3.x; td[13] = q3.y; td[14] = q3.z; td[15] = q3.w;
                if (S != 0 && !packed) {
                    const TileEdges te = tileEdges(__ldg(&d.triHeader[slot]), cx0, cy0);
                    low = sampleMaskOf<S>(te.E, te.A, te.B, px, py);
                } else if (S != 0) {
                    low &= (1u << NS) - 1u;
                }
                bool discard;
                const S32 X = tx * 8 + px, Y = ty * 8 + py;
                const S32 triIdx = (S32)((S64)tri - triBase);
                // low now holds the winner's coverage mask of the pixel (MSAA).
                const U32 src = shadeFragment<FS, S, F>(td, triIdx, X, Y, S != 0 ? low : 1u, verts, stride4,
                                                        sm.shared, 0u, discard);
                BS bs;
#pragma unroll
                for (int i = 0; i < NS; i++) {
                    if (!(won >> i & 1)) continue;
                    const int idx = rowBase + i * 8;
                    bs.m_triIdx = triIdx;
                    bs.m_pixelPos = FW::Vec2i(X, Y);
                    bs.m_sampleIdx = i;
                    bs.m_src = src;
                    bs.m_dst = sm.color[idx];
                    bs.m_color = 0xFF0000FFu;
                    bs.m_writeColor = true;
                    bs.run();
                    if (bs.m_writeColor) sm.color[idx] = bs.m_color;
                }
            }
            __syncwarp();
        }

        // Write the tile back (FineRaster.inl:736-746).
        if (wide) {
#pragma unroll
            for (int i = 0; i < NS; i++) {
                const int w = 2 * lane + 64 * i;
                uint2 z;
                if constexpr (kVisibility) {
                    const ulonglong2 k = *reinterpret_cast<const ulonglong2*>(&sm.key[w]);
                    z = make_uint2((U32)(k.x >> 32), (U32)(k.y >> 32));
                } else {
                    z = *reinterpret_cast<const uint2*>(&sm.depth[w]);
                }
                *reinterpret_cast<uint2*>(&gColor[wideOrigin + i * wideStep]) = *reinterpret_cast<const uint2*>(&sm.color[w]);
                *reinterpret_cast<uint2*>(&gDepth[wideOrigin + i * wideStep]) = z;
            }
        } else {
            for (int w = lane; w < TW; w += 32) {
                const S64 g = tileOrigin + (S64)(w / (8 * NS)) * rowWords + (w % (8 * NS));
                gColor[g] = sm.color[w];
                if constexpr (kVisibility)
                    gDepth[g] = (U32)(sm.key[w] >> 32);
                else
                    gDepth[g] = sm.depth[w];
            }
        }
        __syncwarp();
    }
}

// The fine-stage kernel, with a register budget by kind (fine stage in us,
// budget taken against the other):
//   one sample: five resident CTAs per SM (48 registers); with quads four,
//     since their shaders spill at 48 (textured quads 395 against 416).
//   MSAA, ordered: four (textured 4x terrain 868 against 965 with the
//     compiler's own 80 registers).
//   MSAA, visibility: the compiler's own choice (4x heightfield at 4K 606
//     with 64 registers, 610 pinned to four CTAs; 8x soup 457 with 112
//     registers, 518 pinned).
template <class V, class FS, class BS, int S, U32 F>
__global__ void __launch_bounds__(kFineMaxThreads, FineTraits<FS, BS, S, F>::kQuads ? 4 : 5)
    fineKernel1(DrawDev d, int group, S32 tileBegin, S32 tileEnd) {
    fineTiles<V, FS, BS, S, F>(d, group, tileBegin, tileEnd);
}
template <class V, class FS, class BS, int S, U32 F>
__global__ void __launch_bounds__(kFineMaxThreads, 4)
    fineKernelMsaaOrdered(DrawDev d, int group, S32 tileBegin, S32 tileEnd) {
    fineTiles<V, FS, BS, S, F>(d, group, tileBegin, tileEnd);
}
template <class V, class FS, class BS, int S, U32 F>
__global__ void __launch_bounds__(kFineMaxThreads) fineKernelMsaa(DrawDev d, int group, S32 tileBegin, S32 tileEnd) {
    fineTiles<V, FS, BS, S, F>(d, group, tileBegin, tileEnd);
}
template <class V, class FS, class BS, int S, U32 F>
constexpr auto fineKernelFor() {
    if constexpr (S == 0)
        return &fineKernel1<V, FS, BS, S, F>;
    else if constexpr (FineTraits<FS, BS, S, F>::kVisibility)
        return &fineKernelMsaa<V, FS, BS, S, F>;
    else
        return &fineKernelMsaaOrdered<V, FS, BS, S, F>;
}

}  // namespace cr
