// raster.cu - tile compositing forward (Rasterizer::forward, Rasterizer.cpp:281-329).
//
// The unit of work is an 8x8 pixel block, two pixels per lane of a warp, walking the depth-sorted list of
// the tile it lies in (all blocks of a larger tile walk the same list). Entries are staged in shared memory
// in batches with a mask of those whose contributing box and ellipse meet the block (raster_common.cuh),
// so only the set bits are walked, front to back, with the reference's cut-offs (alpha <= 0.99, skip
// alpha < minAlpha, stop when T (1 - alpha) < minTransmittance). Skipped entries are exactly those the
// reference skips for these pixels, so the output is unchanged.
//
// What an entry adds to a pixel needs its alpha, which is the same whatever lies before it, and the
// transmittance, which is one product after the other. Evaluated one entry at a time, an entry cost a
// warp's lane 320 cycles from loads over the exponential to the cut-off, and a launch lasted as long as its
// longest list took one warp (a block's last pixel terminates after about 150 entries on average, in an
// image's longest after 1,000 to 1,500; part-trained 300k model at 640x480: SMs idle 64 % of the time).
// Here the alphas of several entries are evaluated together and the path from entry to entry is the one
// product (Blend::entry). Two kernels with the same arithmetic and so the same bits:
//   compositeForwardKernel      one warp per block, four entries at a time: 190 cycles per entry
//   compositeForwardTeamKernel  four warps per block evaluate for one that blends: 70 cycles per entry, but
//                               up to a batch of entries evaluated in vain at the end of every block
// The second where blocks are too few to fill the GPU: us per launch one warp / team / before at 96x72
// pixels 46 / 27 / 71, 320x240 (1,200 blocks) 64 / 52 / 96, 480x360 (2,700) 73 / 80 / 102, 640x480 106 / 130 /
// 134.
//
// Compiled with -fmad=false: the contribution decisions (power, alpha, the transmittance cut-off) and
// the transmittance round exactly like the reference's, so the same entries contribute. The colour
// sums alone use explicit fused multiply-adds (within 1e-7 of the unfused sums; images are compared
// within 1e-5). A lane's two pixels are blended together in sm_100's paired FP32 instructions
// (add2rn / mul2rn / fma2rn, paired.cuh), which round each lane like the scalar operation.

#include "raster_common.cuh"

#include <cstdint>

namespace u3dg {

namespace {

// The alphas of one entry at a lane's two pixels (column fx, rows -nfy): the falloff exponent in powerAt's
// order (products paired, sums scalar; -0.5 q is exact, so one fused step rounds like the two). Reaches a
// pixel if the exponent is in range; its exponential is only needed then.
struct EntryPower {
    float2 pw;
    float alpha;
    bool v0, v1;
};

__device__ __forceinline__ EntryPower entryPower(const float4 &P, const float4 &Q, float fx, float2 nfy, bool on0, bool on1)
{
    const ColumnTerms ct = columnTerms(Q, __fsub_rn(P.x, fx));
    const float2 dy = add2rn(both(P.y), nfy);
    const float2 cdd = mul2rn(mul2rn(both(Q.z), dy), dy);
    const float2 q = make_float2(__fadd_rn(ct.axx, cdd.x), __fadd_rn(ct.axx, cdd.y));
    EntryPower e;
    e.pw = fma2rn(both(-0.5f), q, mul2rn(both(-ct.bx), dy));
    e.alpha = Q.w;
    e.v0 = on0 && !(e.pw.x > 0.0f || e.pw.x < P.z);
    e.v1 = on1 && !(e.pw.y > 0.0f || e.pw.y < P.z);
    return e;
}

// Negative zero where the entry is not blended.
__device__ __forceinline__ float2 entryAlpha(const EntryPower &e, float minA)
{
    const float2 raw = mul2rn(both(e.alpha), make_float2(rasterExp(e.pw.x), rasterExp(e.pw.y)));
    const float a0 = (raw.x < kMaxAlpha) ? raw.x : kMaxAlpha;
    const float a1 = (raw.y < kMaxAlpha) ? raw.y : kMaxAlpha;
    return make_float2(e.v0 && !(a0 < minA) ? a0 : -0.0f, e.v1 && !(a1 < minA) ? a1 : -0.0f);
}

// A lane's two pixels while their list is blended, front to back (Rasterizer.cpp:305-318), in paired FP32
// instructions where each lane rounds like the scalar operation. T is the running product of 1 - alpha,
// not stopped at the cut-off: it never grows, so a pixel is live exactly while T is at least the minimum,
// and the path from entry to entry is one multiplication. Tf is T before the entry that fell below it.
template <bool kKeep>
struct Blend {
    float2 T, Tf, cr, cg, cb;
    // kKeep: the colour blended since the current segment began and the transmittance it began with,
    // written when it ends (RasterArgs::ck).
    float2 lr, lg, lb, begin;
    int last0, last1, segment, left;

    __device__ __forceinline__ Blend(bool in0, bool in1, int segmentSize)
    {
        T = make_float2(in0 ? 1.0f : -1.0f, in1 ? 1.0f : -1.0f); // outside the image: never live
        Tf = begin = both(1.0f);
        cr = cg = cb = lr = lg = lb = both(0.0f);
        last0 = last1 = segment = 0;
        left = segmentSize;
    }
    // al: the entry's alphas (negative zero: not blended), idx its list position + 1. kStrict: R may hold a
    // non-finite colour, which must reach only the pixels it blends into (0 * inf is not 0): the colour is
    // taken as 0 where a pixel's weight is.
    template <bool kStrict>
    __device__ __forceinline__ void entry(const float2 &al, const float4 &R, int idx, float minT)
    {
        const float2 nT = mul2rn(T, fma2rn(al, both(-1.0f), both(1.0f)));
        const bool on0 = nT.x >= minT, on1 = nT.y >= minT;
        float2 w = mul2rn(al, T);
        w.x = on0 ? w.x : 0.0f;
        w.y = on1 ? w.y : 0.0f;
        T = nT;
        Tf.x = on0 ? nT.x : Tf.x;
        Tf.y = on1 ? nT.y : Tf.y;
        float2 r = both(R.x), g = both(R.y), b = both(R.z);
        if (kStrict) {
            const bool s0 = w.x != 0.0f, s1 = w.y != 0.0f;
            r = make_float2(s0 ? r.x : 0.0f, s1 ? r.y : 0.0f);
            g = make_float2(s0 ? g.x : 0.0f, s1 ? g.y : 0.0f);
            b = make_float2(s0 ? b.x : 0.0f, s1 ? b.y : 0.0f);
        }
        cr = fma2rn(r, w, cr);
        cg = fma2rn(g, w, cg);
        cb = fma2rn(b, w, cb);
        if (kKeep) {
            lr = fma2rn(r, w, lr);
            lg = fma2rn(g, w, lg);
            lb = fma2rn(b, w, lb);
        }
        last0 = on0 && __float_as_int(al.x) >= 0 ? idx : last0;
        last1 = on1 && __float_as_int(al.y) >= 0 ? idx : last1;
    }
    __device__ __forceinline__ void keepSegment(const RasterArgs &a, int slot0, int px, int py0, bool in0, bool in1) const
    {
        if (segment == 0)
            return;
        float4 *slot = a.ck + (size_t(slot0 + segment) * a.tileSize) * a.tileSize;
        if (in0)
            slot[slotPixel(a.tileSize, px, py0)] = make_float4(lr.x, lg.x, lb.x, begin.x);
        if (in1)
            slot[slotPixel(a.tileSize, px, py0 + 4)] = make_float4(lr.y, lg.y, lb.y, begin.y);
    }
    // Before a batch of `batch` entries (batches do not cross segments).
    __device__ __forceinline__ void beginBatch(const RasterArgs &a, int batch, int slot0, int px, int py0, bool in0, bool in1)
    {
        if (kKeep && left == 0) {
            keepSegment(a, slot0, px, py0, in0, in1);
            ++segment;
            left = a.segment;
            lr = lg = lb = both(0.0f);
            begin = Tf;
        }
        left -= batch;
    }
    __device__ __forceinline__ void store(const RasterArgs &a, int slot0, int px, int py0, bool in0, bool in1, float *rgb,
                                          float *finalT, int *nContrib) const
    {
        if (kKeep) {
            keepSegment(a, slot0, px, py0, in0, in1);
            const int most = __reduce_max_sync(0xffffffffu, max(last0, last1));
            if ((threadIdx.x & 31) == 0)
                a.blockMax[(py0 >> 3) * (a.tilesX * (a.tileSize >> 3)) + (px >> 3)] = most;
        }
        auto put = [&](int py, float T1, float r, float g, float b, int last) {
            const size_t pix = size_t(py) * a.width + px;
            rgb[pix * 3] = r + T1 * a.bg[0];
            rgb[pix * 3 + 1] = g + T1 * a.bg[1];
            rgb[pix * 3 + 2] = b + T1 * a.bg[2];
            finalT[pix] = T1;
            nContrib[pix] = last;
        };
        if (in0)
            put(py0, Tf.x, cr.x, cg.x, cb.x, last0);
        if (in1)
            put(py0 + 4, Tf.y, cr.y, cg.y, cb.y, last1);
    }
};

// One warp per 8x8 pixel block: kGroup entries at a time, first the alphas of all of them, then the
// blending. At most 96 registers, so that 20 blocks share an SM (640x480 us at groups of 1 / 2 / 4: 129 /
// 112 / 106).
constexpr int kSoloBatch = 32, kGroup = 4;

struct SoloShared {
    float4 P[kSoloBatch], Q[kSoloBatch], R[kSoloBatch];
    uint32_t mask[1][1];
};

template <bool kKeep, bool kStrict>
__device__ __forceinline__ void soloBatch(const SoloShared &sh, Blend<kKeep> &px, int first, float fx, float2 nfy, float minA,
                                          float minT)
{
    uint32_t bits = sh.mask[0][0];
    while (bits) {
        const bool on0 = px.T.x >= minT, on1 = px.T.y >= minT;
        if (!__any_sync(0xffffffffu, on0 || on1))
            break;
        float2 al[kGroup];
        int j[kGroup];
#pragma unroll
        for (int u = 0; u < kGroup; ++u) {
            const bool has = bits != 0;
            j[u] = has ? __ffs(bits) - 1 : j[0];
            bits &= bits - 1;
            al[u] = entryAlpha(entryPower(sh.P[j[u]], sh.Q[j[u]], fx, nfy, has && on0, has && on1), minA);
        }
#pragma unroll
        for (int u = 0; u < kGroup; ++u)
            px.template entry<kStrict>(al[u], sh.R[j[u]], first + j[u], minT);
    }
}

// The 8x8 block of this CTA: the tiles' blocks in tile order, or row-major blocks of the image. False outside
// the image.
__device__ __forceinline__ bool forwardBlock(const RasterArgs &a, int &bx, int &by)
{
    const int i = int(blockIdx.x);
    if (a.tileOrder) {
        const int side = a.tileSize >> 3, tile = a.tileOrder[i / (side * side)], at = i % (side * side);
        bx = tile % a.tilesX * side + at % side;
        by = tile / a.tilesX * side + at / side;
    } else {
        bx = i % a.blocksX;
        by = i / a.blocksX;
    }
    return bx < a.blocksX && by < a.blocksY;
}

template <bool kKeep>
__global__ void __launch_bounds__(32, 20) compositeForwardKernel(RasterArgs a, float *rgb, float *finalT, int *nContrib)
{
    pdlEntry();
    __shared__ SoloShared sh;
    int bx, by; // 8x8 blocks
    if (!forwardBlock(a, bx, by))
        return;
    const int lane = threadIdx.x;
    const WarpBlock wb(lane, bx, by);
    const int tile = tileOf<8>(a, bx, by);
    const int start = a.tileOffsets[tile], end = a.tileOffsets[tile + 1];
    const float fx = float(wb.px);
    const float2 nfy = make_float2(-float(wb.py0), -float(wb.py1));
    const float4 *rec = reinterpret_cast<const float4 *>(a.rec);
    const bool in0 = wb.px < a.width && wb.py0 < a.height, in1 = wb.px < a.width && wb.py1 < a.height;
    const int slot0 = kKeep ? start / a.segment + tile : 0;
    Blend<kKeep> px(in0, in1, a.segment);
    // The records of the next batch and the ids of the one after it are on their way meanwhile.
    auto idOf = [&](int b0) { return b0 + lane < end ? a.entries[b0 + lane] : -1; };
    StagedRecord next = loadRecord(rec, idOf(start));
    int gid = idOf(start + kSoloBatch);
    for (int b0 = start; b0 < end; b0 += kSoloBatch) {
        if (!__any_sync(0xffffffffu, px.T.x >= a.minTransmittance || px.T.y >= a.minTransmittance))
            break;
        px.beginBatch(a, kSoloBatch, slot0, wb.px, wb.py0, in0, in1);
        stage<1, 1>(next, b0 + lane < end, lane, sh.P, sh.Q, sh.R, sh.mask, bx, by);
        const bool odd = !finite(next.c.x) || !finite(next.c.y) || !finite(next.c.z);
        const bool strict = __any_sync(0xffffffffu, odd);
        __syncwarp();
        next = loadRecord(rec, gid);
        gid = idOf(b0 + 2 * kSoloBatch);
        if (strict)
            soloBatch<kKeep, true>(sh, px, b0 - start + 1, fx, nfy, a.minAlpha, a.minTransmittance);
        else
            soloBatch<kKeep, false>(sh, px, b0 - start + 1, fx, nfy, a.minAlpha, a.minTransmittance);
        __syncwarp();
    }
    px.store(a, slot0, wb.px, wb.py0, in0, in1, rgb, finalT, nContrib);
}

// One 8x8 pixel block by a team of warps. What an entry adds to a pixel needs its alpha, which is the same
// whatever lies before it, and the transmittance, which is one product after the other. The evaluating
// warps stage a batch of kBatch list entries and compute the alphas of those that meet the block (every
// kEval-th each, two at a time) into shared memory while the blending warp, one batch behind, takes them
// in list order through the transmittance, the cut-off and the colour sums.
constexpr int kEval = 4, kBatch = 64, kBlendGroup = 4, kEvalGroup = 2;
constexpr int kTeamThreads = 32 * (kEval + 1);
static_assert(kEval * 32 >= kBatch, "every entry of a batch has an evaluating thread");

struct TeamShared {
    float2 alpha[2][kBatch][32]; // per entry and lane: the lane's two pixels (negative zero: not blended)
    float4 P[kBatch], Q[kBatch], R[2][kBatch];
    uint32_t mask[2][1][kBatch / 32];
    int odd[2][kBatch / 32]; // a non-finite colour among a staging warp's entries
    uint2 live[2];           // the lanes whose first / second pixel is live
};

// Barriers by name, as the two roles meet at different places of the code.
__device__ __forceinline__ void evaluatorsMeet() { asm volatile("bar.sync 1, %0;" ::"n"(kEval * 32) : "memory"); }
__device__ __forceinline__ void teamMeets() { asm volatile("bar.sync 2, %0;" ::"n"(kTeamThreads) : "memory"); }

// Alphas of the batch's entries that meet the block, evaluating warp `w` of kEval. An entry that reaches no
// live pixel (on0, on1: the lane's pixels as of two batches ago) leaves the mask before its exponentials:
// towards the end of a block few pixels are live.
__device__ __forceinline__ void evaluateBatch(TeamShared &sh, int buf, int w, int lane, float fx, float2 nfy, float minA,
                                              bool on0, bool on1)
{
    static_assert(kEval == 4, "every fourth entry");
#pragma unroll
    for (int half = 0; half < kBatch / 32; ++half) {
        uint32_t mine = sh.mask[buf][0][half] & (0x11111111u << w), none = 0;
        while (mine) {
            int j[kEvalGroup];
            EntryPower e[kEvalGroup];
            bool any = false;
#pragma unroll
            for (int u = 0; u < kEvalGroup; ++u) {
                const bool has = mine != 0;
                j[u] = has ? __ffs(mine) - 1 : j[0];
                mine &= mine - 1;
                e[u] = entryPower(sh.P[32 * half + j[u]], sh.Q[32 * half + j[u]], fx, nfy, on0, on1);
                any = any || e[u].v0 || e[u].v1;
            }
            if (!__any_sync(0xffffffffu, any)) {
#pragma unroll
                for (int u = 0; u < kEvalGroup; ++u)
                    none |= 1u << j[u];
                continue;
            }
#pragma unroll
            for (int u = 0; u < kEvalGroup; ++u)
                sh.alpha[buf][32 * half + j[u]][lane] = entryAlpha(e[u], minA);
        }
        if (none && lane == 0)
            atomicAnd(&sh.mask[buf][0][half], ~none);
    }
}

template <bool kKeep, bool kStrict>
__device__ __forceinline__ void blendBatch(const TeamShared &sh, int buf, int lane, Blend<kKeep> &px, int first, float minT)
{
#pragma unroll
    for (int half = 0; half < kBatch / 32; ++half) {
        uint32_t bits = sh.mask[buf][0][half];
        while (bits) {
            int j[kBlendGroup];
            float2 al[kBlendGroup];
#pragma unroll
            for (int u = 0; u < kBlendGroup; ++u) {
                const bool has = bits != 0;
                j[u] = 32 * half + (has ? __ffs(bits) - 1 : 0);
                bits &= bits - 1;
                al[u] = sh.alpha[buf][j[u]][lane];
                if (!has)
                    al[u] = both(-0.0f);
            }
#pragma unroll
            for (int u = 0; u < kBlendGroup; ++u)
                px.template entry<kStrict>(al[u], sh.R[buf][j[u]], first + j[u], minT);
        }
    }
}

template <bool kKeep>
__global__ void __launch_bounds__(kTeamThreads, 6) compositeForwardTeamKernel(RasterArgs a, float *rgb,
                                                                                           float *finalT, int *nContrib)
{
    pdlEntry();
    __shared__ TeamShared sh;
    int bx, by; // 8x8 blocks
    if (!forwardBlock(a, bx, by))
        return;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const WarpBlock wb(lane, bx, by);
    const int tile = tileOf<8>(a, bx, by);
    const int start = a.tileOffsets[tile], end = a.tileOffsets[tile + 1];
    const int batches = (end - start + kBatch - 1) / kBatch;
    const bool in0 = wb.px < a.width && wb.py0 < a.height, in1 = wb.px < a.width && wb.py1 < a.height;
    const float minT = a.minTransmittance;
    if (warp > 0) {
        const int e = threadIdx.x - 32;
        const float fx = float(wb.px);
        const float2 nfy = make_float2(-float(wb.py0), -float(wb.py1));
        const float4 *rec = reinterpret_cast<const float4 *>(a.rec);
        auto idOf = [&](int t) {
            const int i = start + t * kBatch + e;
            return e < kBatch && i < end ? a.entries[i] : -1;
        };
        // The records of the next batch and the ids of the one after it are on their way meanwhile.
        bool on0 = in0, on1 = in1;
        StagedRecord next = loadRecord(rec, idOf(0));
        int gid = idOf(1);
        for (int t = 0; t < batches; ++t) {
            const int buf = t & 1;
            if (e < kBatch) {
                const bool valid = start + t * kBatch + e < end;
                stage<1, kBatch / 32>(next, valid, e, sh.P, sh.Q, sh.R[buf], sh.mask[buf], bx, by);
                const bool odd = !finite(next.c.x) || !finite(next.c.y) || !finite(next.c.z);
                const bool any = __any_sync(0xffffffffu, odd);
                if (lane == 0)
                    sh.odd[buf][e >> 5] = any;
            }
            evaluatorsMeet();
            next = loadRecord(rec, gid);
            gid = idOf(t + 2);
            evaluateBatch(sh, buf, warp - 1, lane, fx, nfy, a.minAlpha, on0, on1);
            teamMeets(); // batch t is evaluated, batch t - 1 blended
            if (t > 0) {
                const uint2 live = sh.live[buf ^ 1];
                if (!(live.x | live.y))
                    return; // and so does the blending warp
                on0 = live.x >> lane & 1u;
                on1 = live.y >> lane & 1u;
            }
        }
        return;
    }
    const int slot0 = kKeep ? start / a.segment + tile : 0;
    Blend<kKeep> px(in0, in1, a.segment);
    if (batches > 0)
        teamMeets(); // batch 0 is evaluated
    for (int t = 0; t < batches; ++t) {
        const int buf = t & 1;
        px.beginBatch(a, kBatch, slot0, wb.px, wb.py0, in0, in1);
        if (sh.odd[buf][0] | sh.odd[buf][1])
            blendBatch<kKeep, true>(sh, buf, lane, px, t * kBatch + 1, minT);
        else
            blendBatch<kKeep, false>(sh, buf, lane, px, t * kBatch + 1, minT);
        if (t + 1 == batches)
            break;
        const uint2 live = make_uint2(__ballot_sync(0xffffffffu, px.T.x >= minT), __ballot_sync(0xffffffffu, px.T.y >= minT));
        if (lane == 0)
            sh.live[buf] = live;
        teamMeets(); // batch t + 1 is evaluated, this one's buffers are free
        if (!(live.x | live.y))
            break;
    }
    px.store(a, slot0, wb.px, wb.py0, in0, in1, rgb, finalT, nContrib);
}

// Blocks up to which the team is faster: us by a team / one warp with lists of trained models (80k to 150k
// Gaussians) at 1,200 blocks 51.5 / 63.7, 1,530 58.1 / 63.7, 1,900 65.1 / 69.0, 2,080 68.1 / 69.5, 2,352 73.0 / 71.8,
// 2,700 79.6 / 73.1. (With the short lists of 20k Gaussians one warp is faster from below 1,900 on: 48.6 / 39.9;
// the host does not know the lists' lengths.)
constexpr int kTeamLimit = 2048;
// Blocks up to which all teams run at once (6 on each of a B200's 148 SMs), so that their order does not matter. Beyond,
// the longest lists go first: forward of 1,200 blocks 55.8 -> 51.4 us, of 2,700 75.8 -> 73.0, of 4,800 104.1 ->
// 100.0; of 108 blocks 26.8 -> 27.2, and the lists 34.6 -> 35.1.
constexpr int kTeamsResident = 888;

} // namespace

bool forwardOrdersTiles(int tiles, int tileSize) { return tiles * (tileSize / 8) * (tileSize / 8) > kTeamsResident; }

template <bool kKeep>
static void launchForward(const RasterArgs &a, float *rgb, float *finalT, int *nContrib, cudaStream_t s)
{
    const int blocks = a.blocksX * a.blocksY, side = a.tileSize / 8;
    const int grid = a.tileOrder ? a.tilesX * ((a.height + a.tileSize - 1) / a.tileSize) * side * side : blocks;
    if (blocks <= kTeamLimit)
        { launchPdl(compositeForwardTeamKernel<kKeep>, grid, kTeamThreads, 0, s, a, rgb, finalT, nContrib); countLaunch(); }
    else
        { launchPdl(compositeForwardKernel<kKeep>, grid, 32, 0, s, a, rgb, finalT, nContrib); countLaunch(); }
}

void launchCompositeForward(const RasterArgs &a, float *rgb, float *finalT, int *nContrib, cudaStream_t s)
{
    RasterArgs f = a;
    f.blocksX = (a.width + 7) / 8;
    f.blocksY = (a.height + 7) / 8;
    if (f.blocksX * f.blocksY <= 0)
        return;
    if (a.segment > 0)
        launchForward<true>(f, rgb, finalT, nContrib, s);
    else
        launchForward<false>(f, rgb, finalT, nContrib, s);
}

} // namespace u3dg
