// raster_bwd.cu - tile compositing backward (Rasterizer::backward pass 1, Rasterizer.cpp:353-427).
//
// Work units are (pixel block, segment) pairs: a 16x16 (or 8x8) pixel block and at most
// RasterArgs::segment consecutive entries of its tile's list, replayed back to front with the
// reference's recurrence (transmittance recovered by division, running colour accumulation, clamp
// handling) from the state the forward kept at the segment's end. Without segments a launch lasted as
// long as its heaviest tile's list, one entry after the other (on a part-trained 300k model at 640x480
// the SMs were idle 40 % of 0.33 ms; on 96x72 pixels 30 CTAs took 0.13 ms), and the transmittance
// recovered over a whole list carried the rounding of every division.
// A batch of entries is staged in shared memory with per-block masks as in the forward
// (raster_common.cuh). The 9 sums per list entry (dmean2d xy, dcovariance abc, drgb, dalpha) go through a
// reduce-scatter over a block's lanes, land in a per-block shared-memory slot, and are added over the
// 8x8 blocks in order after the batch: the result does not depend on scheduling. Each (tile, Gaussian)
// partial is stored once, at the entry's list position (a tile's partials are contiguous); entries
// behind every pixel's last contributor, where lists are long more than half, are neither written nor
// read (stop); the chain-rule kernel sums a Gaussian's partials in emission order. Tiles of 32 or 64
// pixels span 4 or 16 blocks of 16x16: each stores into its own slot array and the chain-rule kernel
// adds the slots in a fixed order, so every tile size gives deterministic gradients (no atomics).
//
// Contribution decisions (power, alpha, the cut-offs) and the transmittance recovery are computed with
// explicitly unfused operations, exactly as in the forward, so the backward visits the same entries;
// the gradient arithmetic may use fused multiply-add (gradients are compared within a relative
// tolerance). The recovery keeps the correctly rounded division: an approximate division (2 ulp) or a
// reciprocal-multiply made the backward 3 % faster but moved some colour gradients just past 1e-4
// relative to the reference's.
//
// A lane's pixels are replayed in pairs by paired FP32 instructions (paired.cuh), one float2 lane
// per pixel; the falloff exponents' sums stay scalar. A pixel that does not contribute at an entry takes
// part with alpha 0, which leaves its state as it is.

#include "raster_common.cuh"

#include <algorithm>
#include <climits>
#include <type_traits>

namespace u3dg {

namespace {

// Pixels and threads of a unit: L lanes own one 8x8 pixel block, PPL = 64 / L pixels each, in one column
// (rows r, r + L / 8, ...). L = 16: a warp holds two blocks, left and right, that walk their own entry masks
// in step, so the reduction (12 shuffles over 16 lanes), the entry's loads and the loop are paid once for two
// (block, entry) pairs and a lane adds four pixels before it. L = 32: one block per warp, which takes 1.3
// times the instructions for the same entries but 0.6 of the time for one of them.
template <int PB, int L>
struct BackwardShape {
    static constexpr int LPB = L;
    static constexpr int PPL = 64 / LPB, PAIRS = PPL / 2;
    static constexpr int WX = PB / 8, BLOCKS = WX * WX;
    static constexpr int NT = BLOCKS * LPB;
    static constexpr int BATCH = PB == 8 ? 32 : 64; // entries staged at a time (times the depth)
};

// Turns an entry's sums into dL/dmean2d and dL/dcovariance. With dPow = alpha t and w = conic (mean - pixel)
// per pixel, dmean = -sum dPow w, and the covariance's gradient, which the reference reaches through the
// conic's (Rasterizer.cpp:405-412, 432-446), is sum dPow w w^T / 2: da = sum dPow w_x^2 / 2, db = sum dPow
// w_x w_y, dc = sum dPow w_y^2 / 2. Taken through the moments of the pixel offsets instead, an elongated
// footprint's gradient is a difference of sums larger by its condition number; w has cancelled its square
// root of it already.
__device__ __forceinline__ void finishEntry(const float4 &Q, float g[kG2d])
{
    g[0] = -(Q.w * g[0]);
    g[1] = -(Q.w * g[1]);
    g[2] = 0.5f * (Q.w * g[2]);
    g[3] = Q.w * g[3];
    g[4] = 0.5f * (Q.w * g[4]);
}

// Sum of c[0..8] over the LPB lanes of a block: values 0..7 by reduce-scatter (three exchanges halve the
// values a lane holds, the rest of the lanes by a butterfly), value 8 by a butterfly. The lanes whose low
// bits (below LPB / 8) are zero get value (lane / (LPB / 8)) % 8, every lane gets v8.
template <int LPB>
__device__ __forceinline__ float blockReduce9(const float c[kG2d], int lane, float *v8)
{
    constexpr int H = LPB / 2;
    const bool bA = lane & H, bB = lane & (H / 2), bC = lane & (H / 4);
    float w4[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const float send = bA ? c[i] : c[i + 4];
        const float keep = bA ? c[i + 4] : c[i];
        w4[i] = keep + __shfl_xor_sync(0xffffffffu, send, H);
    }
    float w2[2];
#pragma unroll
    for (int i = 0; i < 2; ++i) {
        const float send = bB ? w4[i] : w4[i + 2];
        const float keep = bB ? w4[i + 2] : w4[i];
        w2[i] = keep + __shfl_xor_sync(0xffffffffu, send, H / 2);
    }
    float v;
    {
        const float send = bC ? w2[0] : w2[1];
        const float keep = bC ? w2[1] : w2[0];
        v = keep + __shfl_xor_sync(0xffffffffu, send, H / 4);
    }
#pragma unroll
    for (int o = H / 8; o > 0; o >>= 1)
        v += __shfl_xor_sync(0xffffffffu, v, o);
    float e = c[8];
#pragma unroll
    for (int o = H; o > 0; o >>= 1)
        e += __shfl_xor_sync(0xffffffffu, e, o);
    *v8 = e;
    return v;
}

// Below 2^60, so that a product of two such values, and the sums of a few, are finite.
__device__ __forceinline__ bool moderate(float v) { return fabsf(v) < 1.152921504606846976e18f; }

// Barrier of the NT threads that work on one unit.
template <int NT>
__device__ __forceinline__ void teamSync(int barrier)
{
    asm volatile("bar.sync %0, %1;" ::"r"(barrier), "r"(NT) : "memory");
}

template <int PB, int L, int BD, bool kBg>
__device__ __forceinline__ void backwardUnit(const RasterArgs &a, int block, int segment, const float *dLdRgb,
                                             const float *finalTIn, const int *nContribIn, float *partial,
                                             const int *stop, float4 *sP, float4 *sQ, float4 *sR,
                                             uint32_t (*mask)[BackwardShape<PB, L>::BATCH * BD / 32], int &sOdd,
                                             float *sBlock, int tid, int barrier)
{
    using S = BackwardShape<PB, L>;
    constexpr int NT = S::NT, LPB = S::LPB, PPL = S::PPL, PAIRS = S::PAIRS, BLOCKS = S::BLOCKS;
    constexpr int NB = S::BATCH * BD, NG = NB / 32, RS = LPB / 8; // batch entries, mask words, row step of a lane's pixels
    const int bx = block % a.blocksX, by = block / a.blocksX;
    const int lane = tid & 31, blk = tid / LPB, bl = tid % LPB;
    const int tile = tileOf<PB>(a, bx, by);
    const int start = a.tileOffsets[tile];
    // The unit's entries [jBegin, jEnd) of the tile's list.
    const int jBegin = segment * a.segment, jEnd = min(jBegin + a.segment, stop[block] - start);
    if (a.subSlots > 1) { // this block's slot array: its position in the tile, row-major
        const int per = a.tileSize / PB;
        partial += size_t((by % per) * per + bx % per) * a.subStride;
    }
    const int px = bx * PB + (blk % S::WX) * 8 + (bl & 7), py = by * PB + (blk / S::WX) * 8 + (bl >> 3);
    const float fx = float(px);
    // Replay state of the lane's pixels, a float2 lane per pixel of a pair: transmittance T and the colour
    // composited behind the current entry, which enters the gradient only through its dot product with
    // dL/dpixel (acc, one scalar per pixel: the recurrence is linear). Behind the unit's last entry, T is
    // what the forward kept where the next segment begins, and acc the colours it kept of the segments
    // behind (positive terms, added from the back) over T.
    float2 T[PAIRS], acc[PAIRS], d0[PAIRS], d1[PAIRS], d2[PAIRS], nfy[PAIRS], fb[PAIRS];
    int nC[PPL], last[PPL];
    size_t pix[PPL];
    int lastSegment = 0; // the furthest segment a pixel of the lane blends in
#pragma unroll
    for (int k = 0; k < PPL; ++k) {
        const int y = py + k * RS;
        const bool in = px < a.width && y < a.height;
        pix[k] = in ? size_t(y) * a.width + px : 0;
        last[k] = in ? nContribIn[pix[k]] : 0;
        lastSegment = max(lastSegment, (last[k] - 1) / a.segment);
    }
    float behind[PPL], t[PPL], fT[PPL], g0[PPL], g1[PPL], g2[PPL];
#pragma unroll
    for (int k = 0; k < PPL; ++k) {
        const bool in = last[k] > 0;
        g0[k] = in ? dLdRgb[pix[k] * 3] : 0.0f;
        g1[k] = in ? dLdRgb[pix[k] * 3 + 1] : 0.0f;
        g2[k] = in ? dLdRgb[pix[k] * 3 + 2] : 0.0f;
        fT[k] = in && (kBg || last[k] <= jEnd) ? finalTIn[pix[k]] : 0.0f;
        t[k] = fT[k];
        behind[k] = 0.0f;
    }
    {
        // The segments behind, for all of the lane's pixels at a time so that their loads overlap.
        const int area = a.tileSize * a.tileSize;
        const float4 *ck = a.ck + size_t(start / a.segment + tile) * area;
#pragma unroll 2
        for (int s = lastSegment; s > segment; --s) {
            float4 c[PPL];
#pragma unroll
            for (int k = 0; k < PPL; ++k)
                c[k] = last[k] > s * a.segment ? ck[size_t(s) * area + slotPixel(a.tileSize, px, py + k * RS)]
                                               : make_float4(0.0f, 0.0f, 0.0f, t[k]);
#pragma unroll
            for (int k = 0; k < PPL; ++k) {
                if (last[k] > s * a.segment) {
                    behind[k] += c[k].x * g0[k] + c[k].y * g1[k] + c[k].z * g2[k];
                    t[k] = c[k].w;
                }
            }
        }
    }
    int bMax = 0; // no pixel of this 8x8 block has a contributor at or beyond bMax: entries from there are skipped
    bool odd = false; // a huge or non-finite dL/dpixel or kept colour
#pragma unroll
    for (int k = 0; k < PPL; ++k) {
        if (last[k] > jEnd)
            behind[k] = t[k] > 0.0f ? behind[k] / t[k] : 0.0f; // (an underflown T: nothing behind is seen)
        nC[k] = min(last[k], jEnd);
        bMax = max(bMax, nC[k]);
        const float b = kBg ? -fT[k] * (a.bg[0] * g0[k] + a.bg[1] * g1[k] + a.bg[2] * g2[k]) : 0.0f;
        odd = odd || !moderate(g0[k]) || !moderate(g1[k]) || !moderate(g2[k]) || !moderate(t[k]) || !moderate(b) || !moderate(behind[k]);
        auto set = [&](float2 *v, float x) { (k & 1 ? v[k / 2].y : v[k / 2].x) = x; };
        set(T, t[k]);
        set(acc, behind[k]);
        set(d0, g0[k]);
        set(d1, g1[k]);
        set(d2, g2[k]);
        set(nfy, -float(py + k * RS));
        set(fb, b);
    }
#pragma unroll
    for (int o = LPB / 2; o > 0; o >>= 1)
        bMax = max(bMax, __shfl_xor_sync(0xffffffffu, bMax, o));
    odd = __any_sync(0xffffffffu, odd);
    const float minA = a.minAlpha;
    float *mine = sBlock + size_t(blk) * NB * kG2d;
    // The lane's store of a reduced entry: the lanes with zero low bits store value 0..7, lane 1 value 8.
    const bool storeV = (bl & (RS - 1)) == 0, store8 = bl == 1;
    const int storeAt = storeV ? (bl / RS) & 7 : 8;
    const float4 *rec = reinterpret_cast<const float4 *>(a.rec);
    for (int bEnd = jEnd; bEnd > jBegin; bEnd -= NB) {
        const int bStart = max(jBegin, bEnd - NB), cnt = bEnd - bStart;
        teamSync<NT>(barrier);
        if (tid == 0)
            sOdd = 0;
        {
            float4 *z = reinterpret_cast<float4 *>(sBlock);
            for (int k = tid; k < BLOCKS * NB * kG2d / 4; k += NT)
                z[k] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        }
        teamSync<NT>(barrier);
#pragma unroll
        for (int r = 0; r < (NB + NT - 1) / NT; ++r) {
            const int slot = r * NT + tid;
            if (slot >= NB) // whole warps
                break;
            const bool valid = slot < cnt;
            stage<S::WX, NG>(loadRecord(rec, valid ? a.entries[start + bStart + slot] : -1), valid, slot, sP, sQ, sR, mask, bx,
                          by);
            if (valid && !(moderate(sR[slot].x) && moderate(sR[slot].y) && moderate(sR[slot].z)))
                sOdd = 1;
        }
        teamSync<NT>(barrier);
        // A non-finite colour or dL/dpixel, or a product of two that is, must reach only the pixels and entries
        // that blend: then the factors of pixels that do not are replaced by zeros (0 * inf is not 0).
        const bool strict = odd || sOdd != 0;
        int k = NG;
        uint32_t bits = 0;
        int steps = 0;
#pragma unroll
        for (int g = 0; g < NG; ++g) {
            const int lim = bMax - bStart - 32 * g; // entries of this group below bMax
            steps += lim <= 0 ? 0 : __popc(mask[blk][g] & (lim < 32 ? (1u << lim) - 1u : ~0u));
        }
        if (LPB < 32)
            steps = max(steps, __shfl_xor_sync(0xffffffffu, steps, 16));
        for (int step = 0; step < steps; ++step) {
            while (bits == 0 && k > 0) {
                --k;
                const int lim = bMax - bStart - 32 * k;
                bits = lim <= 0 ? 0u : mask[blk][k] & (lim < 32 ? (1u << lim) - 1u : ~0u);
            }
            const bool has = bits != 0;
            const int hb = has ? 31 - __clz(bits) : 0;
            bits &= ~(1u << hb);
            const int jj = has ? 32 * k + hb : 0, j = has ? bStart + jj : INT_MAX;
            const float4 P = sP[jj], Q = sQ[jj];
            const float dx = __fsub_rn(P.x, fx);
            const ColumnTerms ct = columnTerms(Q, dx);
            // Falloff exponents exactly as the forward decides (powerAt's order; products paired, the sum
            // of the squares scalar; -0.5 q is exact, so one fused step rounds like the two).
            float2 dy[PAIRS], G[PAIRS], al[PAIRS];
            bool act = false;
#pragma unroll
            for (int p = 0; p < PAIRS; ++p) {
                dy[p] = add2rn(both(P.y), nfy[p]);
                const float2 cdd = mul2rn(mul2rn(both(Q.z), dy[p]), dy[p]);
                const float2 q = make_float2(__fadd_rn(ct.axx, cdd.x), __fadd_rn(ct.axx, cdd.y));
                const float2 pw = fma2rn(both(-0.5f), q, mul2rn(both(-ct.bx), dy[p]));
                G[p] = make_float2(rasterExp(pw.x), rasterExp(pw.y));
                const float2 raw = mul2rn(both(Q.w), G[p]);
                const float a0 = (raw.x < kMaxAlpha) ? raw.x : kMaxAlpha;
                const float a1 = (raw.y < kMaxAlpha) ? raw.y : kMaxAlpha;
                const bool v0 = j < nC[2 * p] && !(pw.x > 0.0f || pw.x < P.z) && !(a0 < minA);
                const bool v1 = j < nC[2 * p + 1] && !(pw.y > 0.0f || pw.y < P.z) && !(a1 < minA);
                act = act || v0 || v1;
                // A pixel that does not blend has alpha 0, which leaves its state as it is, and falloff 0;
                // a clamped alpha has a colour gradient only (falloff 0 too).
                al[p] = make_float2(v0 ? a0 : 0.0f, v1 ? a1 : 0.0f);
                G[p] = make_float2(v0 && !(raw.x > kMaxAlpha) ? G[p].x : 0.0f, v1 && !(raw.y > kMaxAlpha) ? G[p].y : 0.0f);
            }
            if (!__any_sync(0xffffffffu, act))
                continue;
            const float4 R = sR[jj];
            const float adx = Q.x * dx;
            float2 s5, s6, s7, st, sx, sy, sxx, sxy, syy;
#pragma unroll
            for (int p = 0; p < PAIRS; ++p) {
                // One back-to-front step of Rasterizer.cpp:385-416 for two pixels. Transmittance before
                // this entry: T / (1 - alpha), rounded like the division (roundedQuotient2).
                const float2 nom = add2rn(al[p], both(-1.0f)); // -(1 - alpha)
                float2 y;
                const float2 Tq = roundedQuotient2(T[p], nom, y);
                T[p] = Tq;
                const float2 w = mul2rn(al[p], Tq);
                // dAlpha = (colour . dpix - acc) T (Rasterizer.cpp:393-399) on the dot products; this entry's
                // colour then goes behind the next one.
                const float2 rd = fma2rn(both(R.z), d2[p], fma2rn(both(R.y), d1[p], mul2rn(both(R.x), d0[p])));
                const float2 s = fma2rn(acc[p], both(-1.0f), rd);
                float2 next = fma2rn(al[p], s, acc[p]);
                float2 dAl = mul2rn(s, Tq);
                if (kBg)
                    dAl = fma2rn(fb[p], y, dAl);
                float2 t = mul2rn(G[p], dAl);
                float2 wv = w, e0 = d0[p], e1 = d1[p], e2 = d2[p];
                if (strict) {
                    const bool v0 = al[p].x != 0.0f, v1 = al[p].y != 0.0f;
                    auto only = [&](const float2 &x) { return make_float2(v0 ? x.x : 0.0f, v1 ? x.y : 0.0f); };
                    next = make_float2(v0 ? next.x : acc[p].x, v1 ? next.y : acc[p].y);
                    t = make_float2(G[p].x != 0.0f ? t.x : 0.0f, G[p].y != 0.0f ? t.y : 0.0f);
                    wv = only(w);
                    e0 = only(e0);
                    e1 = only(e1);
                    e2 = only(e2);
                }
                acc[p] = next;
                // Colour sums, and the sums of t, t w and t w w^T (finishEntry).
                const float2 wx = fma2rn(both(Q.y), dy[p], both(adx)), wy = fma2rn(both(Q.z), dy[p], both(ct.bx));
                const float2 tx = mul2rn(t, wx), ty = mul2rn(t, wy);
                s5 = p ? fma2rn(wv, e0, s5) : mul2rn(wv, e0);
                s6 = p ? fma2rn(wv, e1, s6) : mul2rn(wv, e1);
                s7 = p ? fma2rn(wv, e2, s7) : mul2rn(wv, e2);
                st = p ? add2rn(st, t) : t;
                sx = p ? add2rn(sx, tx) : tx;
                sy = p ? add2rn(sy, ty) : ty;
                sxx = p ? fma2rn(tx, wx, sxx) : mul2rn(tx, wx);
                sxy = p ? fma2rn(tx, wy, sxy) : mul2rn(tx, wy);
                syy = p ? fma2rn(ty, wy, syy) : mul2rn(ty, wy);
            }
            float c[kG2d];
            c[8] = st.x + st.y;
            c[0] = sx.x + sx.y;
            c[1] = sy.x + sy.y;
            c[2] = sxx.x + sxx.y;
            c[3] = sxy.x + sxy.y;
            c[4] = syy.x + syy.y;
            c[5] = s5.x + s5.y;
            c[6] = s6.x + s6.y;
            c[7] = s7.x + s7.y;
            float v8;
            const float v = blockReduce9<LPB>(c, lane, &v8);
            if (has && (storeV || store8))
                mine[jj * kG2d + storeAt] = storeV ? v : v8;
        }
        teamSync<NT>(barrier);
#pragma unroll
        for (int r = 0; r < (NB + NT - 1) / NT; ++r) {
            const int e = r * NT + tid;
            if (e >= cnt)
                break;
            float sum[kG2d];
#pragma unroll
            for (int q = 0; q < kG2d; ++q)
                sum[q] = sBlock[e * kG2d + q];
            for (int w = 1; w < BLOCKS; ++w)
#pragma unroll
                for (int q = 0; q < kG2d; ++q)
                    sum[q] += sBlock[(size_t(w) * NB + e) * kG2d + q];
            finishEntry(sQ[e], sum);
            float4 *dst = reinterpret_cast<float4 *>(partial) + size_t(start + bStart + e) * (kPartial / 4);
            dst[0] = make_float4(sum[0], sum[1], sum[2], sum[3]);
            dst[1] = make_float4(sum[4], sum[5], sum[6], sum[7]);
            dst[2] = make_float4(sum[8], 0.0f, 0.0f, 0.0f);
        }
    }
}

// Teams of 64 threads per SM the compiler must allow for (16x16 blocks): caps registers per thread at
// 65536 / (64 * n).
#ifndef U3DG_BWD_MIN_BLOCKS
#define U3DG_BWD_MIN_BLOCKS 8
#endif

// A CTA of 16x16 blocks has 128 threads: two teams of 64 (16 lanes per 8x8 block), each with a unit of its
// own, or, where the launch has no more than `few` units (kFewUnits per SM, about one per CTA), one team of
// 128 (32 lanes). Then the launch lasts as
// long as one unit, 64 entries at about 800 cycles each by 16 lanes (a warp alone on its scheduler): 52 us
// against 38 us on 4k Gaussians at 96x72. With more units than CTAs the instructions count: at two units
// per CTA the two shapes are even (+-2 us of 60), on 300k Gaussians at 640x480 32 lanes take 169 us against
// 143. The two shapes add an entry's pixels in another order, so the line is a number of units of its own and
// not the grid: it must not move with the registers or the shared memory of one instance (the batch depths
// give the same bits).
constexpr int kFewUnits = 4;
template <int PB>
constexpr int kTeams = PB == 8 ? 1 : 2;
template <int PB>
constexpr int kThreads = PB == 8 ? 32 : 128;

template <int PB, int L, int BD, bool kBg>
__device__ __forceinline__ void backwardUnits(const RasterArgs &a, const float *dLdRgb, const float *finalTIn,
                                              const int *nContribIn, float *partial, const int *stop, const int2 *units,
                                              int count, float4 *sP, float4 *sQ, float4 *sR,
                                              uint32_t (*mask)[BackwardShape<PB, L>::BATCH * BD / 32], int &sOdd,
                                              int &sNext, float *sBlock)
{
    constexpr int NT = BackwardShape<PB, L>::NT;
    const int tid = threadIdx.x % NT, barrier = threadIdx.x / NT;
    for (;;) {
        teamSync<NT>(barrier); // every thread is done with the previous unit's shared memory
        if (tid == 0)
            sNext = takeUnit(count, a.counters, gridDim.x * (kThreads<PB> / NT));
        teamSync<NT>(barrier);
        const int u = sNext;
        if (u >= count)
            break;
        const int2 unit = units[u];
        backwardUnit<PB, L, BD, kBg>(a, unit.x, unit.y, dLdRgb, finalTIn, nContribIn, partial, stop, sP, sQ, sR, mask,
                                     sOdd, sBlock, tid, barrier);
    }
}

template <int PB, int BD, bool kBg>
__global__ void __launch_bounds__(kThreads<PB>, U3DG_BWD_MIN_BLOCKS * 64 / kThreads<PB>)
    compositeBackwardKernel(RasterArgs a, const float *dLdRgb, const float *finalTIn, const int *nContribIn,
                            float *partial, const int *stop, const int2 *units, const int *unitCount, int few)
{
    pdlEntry();
    using S = BackwardShape<PB, PB == 8 ? 32 : 16>;
    constexpr int NB = S::BATCH * BD, NG = NB / 32, TEAMS = kTeams<PB>;
    __shared__ float4 sP[TEAMS][NB];
    __shared__ float4 sQ[TEAMS][NB];
    __shared__ float4 sR[TEAMS][NB];
    __shared__ uint32_t mask[TEAMS][S::BLOCKS][NG];
    __shared__ int sOdd[TEAMS], sNext[TEAMS];
    extern __shared__ __align__(16) float sBlock[]; // per team and 8x8 block: NB entries x 9 sums
    const int count = *unitCount;
    if (PB == 8 || count <= few) {
        backwardUnits<PB, 32, BD, kBg>(a, dLdRgb, finalTIn, nContribIn, partial, stop, units, count, sP[0], sQ[0], sR[0],
                                       mask[0], sOdd[0], sNext[0], sBlock);
    } else {
        const int team = threadIdx.x / S::NT;
        backwardUnits<PB, PB == 8 ? 32 : 16, BD, kBg>(a, dLdRgb, finalTIn, nContribIn, partial, stop, units, count, sP[team], sQ[team],
                                       sR[team], mask[team], sOdd[team], sNext[team],
                                       sBlock + size_t(team) * S::BLOCKS * NB * kG2d);
    }
}

// ---------------------------------------------------------------- whole lists

// The rasterizer's own backward, for lists that are not culled: a 16x16 (or 8x8) block replays its whole list,
// two pixels of a column per thread, and sums the moments of the pixel offsets. A program that takes gradients
// from the rasterizer gets them in this order of summation: a few ill-conditioned Gaussians' (of 250k at
// 640x480) come out of sums that cancel to 1e-3 of their terms' rounding, and any other order moves those by
// up to 1e-2 of the gradients' root mean square. The trainers take units of segments (40 % of the time).
struct PixelPair {
    float2 T, nacc, lcd, nla; // transmittance, -(colour dot behind), last contributor's colour dot, -its alpha
    float2 d0, d1, d2, fy;    // dL/dpixel per channel, pixel row
    float2 fT, bgDot;         // final transmittance, background . dL/dpixel (background term only)
    int nC0, nC1;             // contributor counts
};

// dL/dmean2d and dL/dconic of an entry's summed moments (Rasterizer.cpp:405-412): dmean = -(A m_x + B m_y,
// C m_y + B m_x), dA = -m_xx / 2, dB = -m_xy, dC = -m_yy / 2.
__device__ __forceinline__ void finishMoments(const float4 &Q, float g[kG2d])
{
    const float mx = g[0], my = g[1];
    g[0] = -(Q.x * mx + Q.y * my);
    g[1] = -(Q.z * my + Q.y * mx);
    g[2] = -0.5f * g[2];
    g[3] = -g[3];
    g[4] = -0.5f * g[4];
}

__device__ __forceinline__ PixelPair initPair(bool in0, bool in1, size_t pix0, size_t pix1, float fy0, float fy1,
                                              const float *dLdRgb, const float *finalT, const int *nContrib,
                                              const float *bg)
{
    PixelPair p;
    p.nC0 = in0 ? nContrib[pix0] : 0;
    p.nC1 = in1 ? nContrib[pix1] : 0;
    p.fT = make_float2(in0 ? finalT[pix0] : 0.0f, in1 ? finalT[pix1] : 0.0f);
    p.d0 = make_float2(in0 ? dLdRgb[pix0 * 3] : 0.0f, in1 ? dLdRgb[pix1 * 3] : 0.0f);
    p.d1 = make_float2(in0 ? dLdRgb[pix0 * 3 + 1] : 0.0f, in1 ? dLdRgb[pix1 * 3 + 1] : 0.0f);
    p.d2 = make_float2(in0 ? dLdRgb[pix0 * 3 + 2] : 0.0f, in1 ? dLdRgb[pix1 * 3 + 2] : 0.0f);
    p.bgDot = make_float2(bg[0] * p.d0.x + bg[1] * p.d1.x + bg[2] * p.d2.x, bg[0] * p.d0.y + bg[1] * p.d1.y + bg[2] * p.d2.y);
    p.T = p.fT;
    p.nacc = p.lcd = p.nla = both(0.0f);
    p.fy = make_float2(fy0, fy1);
    return p;
}

template <int PB>
constexpr int kListWarps = PB * PB / 64;

template <int PB, bool kBg>
__global__ void __launch_bounds__(32 * kListWarps<PB>, 6) compositeBackwardListKernel(RasterArgs a, const float *dLdRgb,
                                                                                      const float *finalTIn,
                                                                                      const int *nContribIn, float *partial,
                                                                                      int *stop)
{
    pdlEntry();
    constexpr int NW = kListWarps<PB>, NT = 32 * NW, NB = NT, NG = NB / 32, WX = PB / 8;
    __shared__ float4 sP[NB], sQ[NB], sR[NB];
    __shared__ uint32_t mask[NW][NG];
    __shared__ int sMax;
    __shared__ __align__(16) float sWarp[NW * NB * kG2d]; // per warp: NB entries x 9 sums
    int bx = int(blockIdx.x) % a.blocksX, by = int(blockIdx.x) / a.blocksX;
    if (a.tileOrder) {
        const int per = a.tileSize / PB, t = a.tileOrder[int(blockIdx.x) / (per * per)], at = int(blockIdx.x) % (per * per);
        bx = t % a.tilesX * per + at % per;
        by = t / a.tilesX * per + at / per;
    }
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const WarpBlock wb(lane, bx * WX + warp % WX, by * WX + warp / WX);
    const int tile = tileOf<PB>(a, bx, by);
    const int start = a.tileOffsets[tile];
    const bool in0 = wb.px < a.width && wb.py0 < a.height, in1 = wb.px < a.width && wb.py1 < a.height;
    if (a.subSlots > 1) { // this block's slot array: its position in the tile, row-major
        const int per = a.tileSize / PB;
        partial += size_t((by % per) * per + bx % per) * a.subStride;
    }
    PixelPair pp = initPair(in0, in1, in0 ? size_t(wb.py0) * a.width + wb.px : 0,
                            in1 ? size_t(wb.py1) * a.width + wb.px : 0, float(wb.py0), float(wb.py1), dLdRgb,
                            finalTIn, nContribIn, a.bg);
    const float2 one2 = both(1.0f);
    const float fx = float(wb.px), minA = a.minAlpha;
    const float4 *rec = reinterpret_cast<const float4 *>(a.rec);
    if (tid == 0)
        sMax = 0;
    __syncthreads();
    const int nMax = max(pp.nC0, pp.nC1);
    if (nMax > 0)
        atomicMax(&sMax, nMax);
    // This warp's pixels have no contributor at or beyond wMax: the warp skips those entries.
    const int wMax = __reduce_max_sync(0xffffffffu, nMax);
    __syncthreads();
    const int jmax = sMax;
    if (tid == 0)
        stop[by * a.blocksX + bx] = start + jmax;
    float *myWarp = sWarp + size_t(warp) * NB * kG2d;
    for (int bEnd = jmax; bEnd > 0; bEnd -= NB) {
        const int bStart = max(0, bEnd - NB), cnt = bEnd - bStart;
        __syncthreads();
        stage<WX, NG>(loadRecord(rec, tid < cnt ? a.entries[start + bStart + tid] : -1), tid < cnt, tid, sP, sQ, sR, mask, bx, by);
        {
            float4 *z = reinterpret_cast<float4 *>(sWarp);
            for (int k = tid; k < NW * NB * kG2d / 4; k += NT)
                z[k] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        }
        __syncthreads();
        for (int k = NG - 1; k >= 0; --k) {
            uint32_t bits = mask[warp][k];
            const int lim = wMax - bStart - 32 * k; // entries of this group below wMax
            if (lim <= 0)
                continue;
            if (lim < 32)
                bits &= (1u << lim) - 1u;
            while (bits) {
                const int hb = 31 - __clz(bits);
                bits &= ~(1u << hb);
                const int jj = 32 * k + hb;
                const int j = bStart + jj;
                float c[kG2d];
#pragma unroll
                for (int q = 0; q < kG2d; ++q)
                    c[q] = 0.0f;
                bool act = false;
                if (j < pp.nC0 || j < pp.nC1) {
                    const float4 P = sP[jj], Q = sQ[jj];
                    const float dx = __fsub_rn(P.x, fx);
                    const ColumnTerms ct = columnTerms(Q, dx);
                    // Falloff exponents exactly as the forward decides (powerAt's order; products
                    // paired, sums scalar).
                    const float2 dy = make_float2(__fsub_rn(P.y, pp.fy.x), __fsub_rn(P.y, pp.fy.y));
                    const float2 cdd = mul2rn(mul2rn(both(Q.z), dy), dy);
                    const float2 bdy = mul2rn(both(ct.bx), dy);
                    const float2 hq = mul2rn(both(-0.5f), make_float2(__fadd_rn(ct.axx, cdd.x), __fadd_rn(ct.axx, cdd.y)));
                    const float2 pw = make_float2(__fsub_rn(hq.x, bdy.x), __fsub_rn(hq.y, bdy.y));
                    bool v0 = j < pp.nC0 && !(pw.x > 0.0f || pw.x < P.z);
                    bool v1 = j < pp.nC1 && !(pw.y > 0.0f || pw.y < P.z);
                    if (v0 || v1) {
                        // One back-to-front step of Rasterizer.cpp:385-416 for both pixels (a pixel that
                        // is out gets exp(0) and zero weights, and keeps its state).
                        const float2 G = make_float2(rasterExp(v0 ? pw.x : 0.0f), rasterExp(v1 ? pw.y : 0.0f));
                        const float2 raw = mul2rn(both(Q.w), G);
                        const float al0 = (raw.x < kMaxAlpha) ? raw.x : kMaxAlpha;
                        const float al1 = (raw.y < kMaxAlpha) ? raw.y : kMaxAlpha;
                        v0 = v0 && !(al0 < minA);
                        v1 = v1 && !(al1 < minA);
                        if (v0 || v1) {
                            act = true;
                            const float4 R = sR[jj];
                            // Transmittance before this entry: T / (1 - alpha), correctly rounded.
                            const float2 om = add2rn(one2, make_float2(-al0, -al1));
                            const float Tn0 = __fdiv_rn(pp.T.x, om.x), Tn1 = __fdiv_rn(pp.T.y, om.y);
                            pp.T = make_float2(v0 ? Tn0 : pp.T.x, v1 ? Tn1 : pp.T.y);
                            const float2 w = mul2rn(make_float2(v0 ? al0 : 0.0f, v1 ? al1 : 0.0f), pp.T);
                            // dAlpha = (colour . dpix - accum . dpix) T (Rasterizer.cpp:393-399), on the
                            // dot products; accum takes the previous contributor's colour first.
                            const float2 rd = fma2rn(both(R.z), pp.d2, fma2rn(both(R.y), pp.d1, mul2rn(both(R.x), pp.d0)));
                            const float2 nacc = fma2rn(pp.nla, add2rn(pp.lcd, pp.nacc), pp.nacc);
                            float2 dAl = mul2rn(add2rn(rd, nacc), pp.T);
                            pp.nacc = make_float2(v0 ? nacc.x : pp.nacc.x, v1 ? nacc.y : pp.nacc.y);
                            pp.lcd = make_float2(v0 ? rd.x : pp.lcd.x, v1 ? rd.y : pp.lcd.y);
                            pp.nla = make_float2(v0 ? -al0 : pp.nla.x, v1 ? -al1 : pp.nla.y);
                            // (An infinite dL/dpixel of a pixel that is out stays out: 0 * inf is not 0.)
                            auto only = [&](const float2 &d) { return make_float2(v0 ? d.x : 0.0f, v1 ? d.y : 0.0f); };
                            const float2 wd0 = mul2rn(w, only(pp.d0)), wd1 = mul2rn(w, only(pp.d1)), wd2 = mul2rn(w, only(pp.d2));
                            c[5] = wd0.x + wd0.y;
                            c[6] = wd1.x + wd1.y;
                            c[7] = wd2.x + wd2.y;
                            if (kBg) {
                                dAl.x += -pp.fT.x / om.x * pp.bgDot.x;
                                dAl.y += -pp.fT.y / om.y * pp.bgDot.y;
                            }
                            // A clamped alpha has a colour gradient only.
                            const bool m0 = v0 && !(raw.x > kMaxAlpha), m1 = v1 && !(raw.y > kMaxAlpha);
                            float2 t = mul2rn(G, dAl);
                            t = make_float2(m0 ? t.x : 0.0f, m1 ? t.y : 0.0f);
                            c[8] = t.x + t.y;
                            // Per-pixel moments of dPow; both pixels share dx, so dx multiplies the thread's
                            // sums once.
                            const float2 dPow = mul2rn(both(Q.w), t);
                            const float2 pdy = mul2rn(dPow, dy);
                            const float2 pdyy = mul2rn(pdy, dy);
                            c[1] = pdy.x + pdy.y;
                            c[4] = pdyy.x + pdyy.y;
                            c[0] = dx * (dPow.x + dPow.y);
                            c[2] = dx * c[0];
                            c[3] = dx * c[1];
                        }
                    }
                }
                if (__any_sync(0xffffffffu, act)) {
                    float v8;
                    const float v = blockReduce9<32>(c, lane, &v8);
                    if ((lane & 3) == 0)
                        myWarp[jj * kG2d + (lane >> 2)] = v;
                    if (lane == 1)
                        myWarp[jj * kG2d + 8] = v8;
                }
            }
        }
        __syncthreads();
        if (tid < cnt) {
            float sum[kG2d];
#pragma unroll
            for (int q = 0; q < kG2d; ++q)
                sum[q] = sWarp[tid * kG2d + q];
            for (int w = 1; w < NW; ++w)
#pragma unroll
                for (int q = 0; q < kG2d; ++q)
                    sum[q] += sWarp[(size_t(w) * NB + tid) * kG2d + q];
            finishMoments(sQ[tid], sum);
            float4 *dst = reinterpret_cast<float4 *>(partial) + size_t(start + bStart + tid) * (kPartial / 4);
            dst[0] = make_float4(sum[0], sum[1], sum[2], sum[3]);
            dst[1] = make_float4(sum[4], sum[5], sum[6], sum[7]);
            dst[2] = make_float4(sum[8], 0.0f, 0.0f, 0.0f);
        }
    }
}

// One CTA: the backward's units (block, segment) in block order, by an exclusive scan of the blocks'
// segment counts.
__global__ void __launch_bounds__(1024) backwardUnitsKernel(RasterArgs a, int pb, int *stop, int2 *units, int *unitCount)
{
    pdlEntry();
    __shared__ int warpSums[32];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int blocks = a.blocksX * a.blocksY, per = pb / 8, x8 = a.tilesX * (a.tileSize >> 3);
    int carry = 0;
    for (int b0 = 0; b0 < blocks; b0 += 1024) {
        const int b = b0 + threadIdx.x;
        int segments = 0;
        if (b < blocks) {
            const int bx = b % a.blocksX, by = b / a.blocksX;
            int most = 0;
            for (int k = 0; k < per * per; ++k) {
                const int x = bx * per + k % per, y = by * per + k / per;
                if (x * 8 < a.width && y * 8 < a.height) // 8x8 blocks outside the image have no count
                    most = max(most, a.blockMax[y * x8 + x]);
            }
            stop[b] = a.tileOffsets[(by * pb / a.tileSize) * a.tilesX + bx * pb / a.tileSize] + most;
            segments = (most + a.segment - 1) / a.segment;
        }
        int incl = segments;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int y = __shfl_up_sync(0xffffffffu, incl, o);
            if (lane >= o)
                incl += y;
        }
        if (lane == 31)
            warpSums[warp] = incl;
        __syncthreads();
        if (warp == 0) {
            int w = warpSums[lane];
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const int y = __shfl_up_sync(0xffffffffu, w, o);
                if (lane >= o)
                    w += y;
            }
            warpSums[lane] = w;
        }
        __syncthreads();
        int at = carry + incl - segments + (warp > 0 ? warpSums[warp - 1] : 0);
        for (int s = 0; s < segments; ++s)
            units[at++] = make_int2(b, s);
        carry += warpSums[31];
        __syncthreads();
    }
    if (threadIdx.x == 0)
        *unitCount = carry;
}

int multiprocessors(int device)
{
    static PerDevice count;
    return count.get(device, [&] {
        int sms = 0;
        cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device);
        return std::max(1, sms);
    });
}

} // namespace

template <int PB, int BD, bool kBg>
static void launchBackward(const RasterArgs &a, const float *dLdRgb, const float *finalT, const int *nContrib,
                           float *partial, const int *stop, const int2 *units, const int *unitCount, cudaStream_t s)
{
    using S = BackwardShape<PB, 32>;
    const size_t smem = size_t(kTeams<PB>) * S::BLOCKS * S::BATCH * BD * kG2d * sizeof(float); // 18 KB or 36 KB at PB 16
    static PerDevice allowed, resident;
    allowShared(compositeBackwardKernel<PB, BD, kBg>, smem + 16 * 1024, smem, allowed); // with the static arrays
    int device = 0;
    cudaGetDevice(&device);
    const int sms = multiprocessors(device), perSm = resident.get(device, [&] {
        int n = 0;
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, compositeBackwardKernel<PB, BD, kBg>, kThreads<PB>, smem);
        return std::max(1, n);
    });
    { launchPdl(compositeBackwardKernel<PB, BD, kBg>, sms * perSm, kThreads<PB>, smem, s, a, dLdRgb, finalT, nContrib, partial, stop, units, unitCount, kFewUnits * sms); countLaunch(); }
}

void launchBackwardUnits(const RasterArgs &a, int *stop, int2 *units, int *unitCount, cudaStream_t s)
{
    { launchPdl(backwardUnitsKernel, 1, 1024, 0, s, a, a.tileSize <= 8 ? 8 : 16, stop, units, unitCount); countLaunch(); }
}

void launchCompositeBackwardList(const RasterArgs &a, const float *dLdRgb, const float *finalT, const int *nContrib,
                                 float *partial, int *stop, cudaStream_t s)
{
    const int blocks = a.blocksX * a.blocksY;
    if (blocks <= 0)
        return;
    const bool bg = a.bg[0] != 0.0f || a.bg[1] != 0.0f || a.bg[2] != 0.0f;
    auto run = [&](auto pb, auto kBg) {
        constexpr int PB = decltype(pb)::value;
        { launchPdl(compositeBackwardListKernel<PB, decltype(kBg)::value>, blocks, 32 * kListWarps<PB>, 0, s, a, dLdRgb, finalT, nContrib, partial, stop); countLaunch(); }
    };
    auto sized = [&](auto kBg) {
        if (a.tileSize <= 8)
            run(std::integral_constant<int, 8>{}, kBg);
        else
            run(std::integral_constant<int, 16>{}, kBg);
    };
    if (bg)
        sized(std::true_type{});
    else
        sized(std::false_type{});
}

void launchCompositeBackward(const RasterArgs &a, const float *dLdRgb, const float *finalT, const int *nContrib,
                             float *partial, const int *stop, const int2 *units, const int *unitCount, cudaStream_t s)
{
    if (a.blocksX * a.blocksY <= 0)
        return;
    const bool deep = a.backwardDepth >= 2 && backwardTakesDepth(a.tileSize);
    const bool bg = a.bg[0] != 0.0f || a.bg[1] != 0.0f || a.bg[2] != 0.0f;
    auto run = [&](auto kBg) {
        constexpr bool B = decltype(kBg)::value;
        if (a.tileSize <= 8)
            deep ? launchBackward<8, 2, B>(a, dLdRgb, finalT, nContrib, partial, stop, units, unitCount, s)
                 : launchBackward<8, 1, B>(a, dLdRgb, finalT, nContrib, partial, stop, units, unitCount, s);
        else
            deep ? launchBackward<16, 2, B>(a, dLdRgb, finalT, nContrib, partial, stop, units, unitCount, s)
                 : launchBackward<16, 1, B>(a, dLdRgb, finalT, nContrib, partial, stop, units, unitCount, s);
    };
    if (bg)
        run(std::true_type{});
    else
        run(std::false_type{});
}

} // namespace u3dg
