// raster_common.cuh - pixel layout and batch staging shared by the compositing kernels.
//
// Work is divided by 8x8 pixel blocks. A tile's depth-sorted list is walked in batches staged in shared
// memory; while staging, each warp votes which of its 32 entries meet a block (the Gaussian's conservative
// contributing box, SplatRec::ex / ey, and ellipse against the block), so that a block's warp walks only
// the set bits of its mask. The batch size changes how many entries are staged per barrier, not any
// result: every entry is evaluated the same way in the same order.
#pragma once

#include "paired.cuh"
#include "kernels.h"

namespace u3dg {

// The two pixels of a warp's lane in 8x8 block (bx, by): one column, rows 4 apart.
struct WarpBlock {
    int px, py0, py1;
    __device__ WarpBlock(int lane, int bx, int by) : px(bx * 8 + (lane & 7)), py0(by * 8 + (lane >> 3)), py1(py0 + 4) {}
};

// Whether the contributing ellipse of a staged entry, {d : A dx^2 + 2 B dx dy + C dy^2 <= -2 powMin}
// (power >= powMin), can reach a pixel centre of the 8x8 block [x0, x0 + 7] x [y0, y0 + 7]: the
// minimum of the quadratic over the block (zero if the block holds the mean, else on an edge, where it
// is a 1D quadratic minimised at a clamped stationary point) against the threshold widened by 4% and
// 1e-3. Rounding-explicit, so every kernel builds the same masks; conservative like the box extents,
// which are infinite for covariances whose condition number exceeds 1e4 (nothing is culled then).
// Rotated, elongated footprints meet far fewer 8x8 blocks than their axis-aligned boxes suggest.
__device__ __forceinline__ bool ellipseMeets(float mx, float my, const float4 &q, float powMin, float iA, float iC,
                                             float x0, float y0)
{
    const float X0 = __fsub_rn(x0, mx), X1 = __fadd_rn(X0, 7.0f);
    const float Y0 = __fsub_rn(y0, my), Y1 = __fadd_rn(Y0, 7.0f);
    if (X0 <= 0.0f && X1 >= 0.0f && Y0 <= 0.0f && Y1 >= 0.0f)
        return true;
    const float A = q.x, B = q.y, C = q.z;
    auto quad = [&](float dx, float dy) {
        const float cross = __fmul_rn(2.0f, __fmul_rn(__fmul_rn(B, dx), dy));
        return __fadd_rn(__fadd_rn(__fmul_rn(__fmul_rn(A, dx), dx), cross), __fmul_rn(__fmul_rn(C, dy), dy));
    };
    const float nbc = __fmul_rn(-B, iC), nba = __fmul_rn(-B, iA);
    float m = quad(X0, fminf(fmaxf(__fmul_rn(nbc, X0), Y0), Y1));
    m = fminf(m, quad(X1, fminf(fmaxf(__fmul_rn(nbc, X1), Y0), Y1)));
    m = fminf(m, quad(fminf(fmaxf(__fmul_rn(nba, Y0), X0), X1), Y0));
    m = fminf(m, quad(fminf(fmaxf(__fmul_rn(nba, Y1), X0), X1), Y1));
    return m <= __fadd_rn(__fmul_rn(-2.08f, powMin), 1e-3f);
}

template <int PB>
__device__ __forceinline__ int tileOf(const RasterArgs &a, int bx, int by)
{
    return (by * PB / a.tileSize) * a.tilesX + bx * PB / a.tileSize;
}

// Persistent scheduling: every team of threads takes work units from a device counter until none are left.
// Called by one thread of a team; returns the next unit's index (>= units: done). The last team to run out
// resets the counter for the next launch. counter[0] hands out units, counter[1] counts finished teams.
__device__ __forceinline__ int takeUnit(int units, int *counter, int teams)
{
    const int u = atomicAdd(counter, 1);
    if (u >= units) {
        __threadfence();
        if (atomicAdd(counter + 1, 1) == teams - 1) {
            atomicExch(counter, 0);
            atomicExch(counter + 1, 0);
        }
    }
    return u;
}

// Index of a pixel in its tile's segment slot (RasterArgs::ck).
__device__ __forceinline__ int slotPixel(int tileSize, int px, int py)
{
    const int x = px % tileSize, y = py % tileSize;
    return ((y >> 3) * (tileSize >> 3) + (x >> 3)) * 64 + (y & 7) * 8 + (x & 7);
}

// A list entry's raster record on its way to shared memory (p.z < 0: none).
struct StagedRecord {
    float4 p, q, c;
};

__device__ __forceinline__ StagedRecord loadRecord(const float4 *rec, int gid)
{
    StagedRecord s;
    s.p = make_float4(0.0f, 0.0f, -1.0f, -1.0f);
    s.q = s.c = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    if (gid >= 0) {
        const float4 *r = rec + size_t(gid) * 3;
        s.p = r[0];
        s.q = r[1];
        s.c = r[2];
    }
    return s;
}

// Whether a record can contribute to a pixel of the 8x8 block at (x0, y0): its box against the block,
// refined by the ellipse test where the box extents are finite (well-conditioned covariances and a
// positive minimum alpha).
__device__ __forceinline__ bool entryMeets(const StagedRecord &s, float x0, float y0)
{
    const float4 &p = s.p;
    if (p.x + p.z < x0 || p.x - p.z > x0 + 7.0f || p.y + p.w < y0 || p.y - p.w > y0 + 7.0f)
        return false;
    return !(p.z < __int_as_float(0x7f800000)) || ellipseMeets(p.x, p.y, s.q, s.c.w, __frcp_rn(s.q.x), __frcp_rn(s.q.z), x0, y0);
}

// Stages batch entry `slot` (if valid) and the masks of NG words: mask[w][g] bit b <=> entry 32g + b meets
// 8x8 block w (of WX per row) of pixel block (bx, by). Slots are a warp's lanes in order.
template <int WX, int NG>
__device__ __forceinline__ void stage(const StagedRecord &s, bool valid, int slot, float4 *sP, float4 *sQ, float4 *sR,
                                      uint32_t (*mask)[NG], int bx, int by)
{
    constexpr int PB = 8 * WX;
    if (valid) {
        // The blending loop reads the mean from sP and the exponent floor (SplatRec::powMin) from its third
        // slot; the contributing box is only needed for the masks below.
        sP[slot] = make_float4(s.p.x, s.p.y, s.c.w, s.p.w);
        sQ[slot] = s.q;
        sR[slot] = s.c;
    }
    const int group = slot >> 5, lane = slot & 31;
#pragma unroll
    for (int w = 0; w < WX * WX; ++w) {
        const uint32_t bits = __ballot_sync(0xffffffffu, valid && entryMeets(s, float(bx * PB + (w % WX) * 8), float(by * PB + (w / WX) * 8)));
        if (lane == 0)
            mask[w][group] = bits;
    }
}

// Gaussian falloff exponent at one pixel, in the reference's operation order with no fused
// multiply-add (Rasterizer.cpp:305-306), so every kernel decides contributions identically:
//   power = -0.5 * ((A dx) dx + (C dy) dy) - (B dx) dy.
// A thread's two pixels share a column, so the dx terms are computed once (columnTerms) and give the
// same roundings as computing them per pixel.
struct ColumnTerms {
    float axx; // (A dx) dx
    float bx;  // B dx
};

__device__ __forceinline__ ColumnTerms columnTerms(const float4 &Q, float dx)
{
    return {__fmul_rn(__fmul_rn(Q.x, dx), dx), __fmul_rn(Q.y, dx)};
}

__device__ __forceinline__ float powerAt(const float4 &Q, const ColumnTerms &c, float dy)
{
    const float q = __fadd_rn(c.axx, __fmul_rn(__fmul_rn(Q.z, dy), dy));
    return __fsub_rn(__fmul_rn(-0.5f, q), __fmul_rn(c.bx, dy));
}

__device__ __forceinline__ float rasterExp(float x) { return expf(x); }

__device__ __forceinline__ bool finite(float v) { return fabsf(v) < __int_as_float(0x7f800000); }

} // namespace u3dg
