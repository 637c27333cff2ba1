// kernels.h - host-side launch interface of the CUDA kernels (no torch, plain pointers).
#pragma once

#include "common.cuh"
#include "per_device.h"

#include <utility>

namespace u3dg {

// Programmatic dependent launch (sm_90+): the kernels of a training step are launched with
// cudaLaunchAttributeProgrammaticStreamSerialization, so the GPU may launch a kernel as soon as every CTA
// of the previous kernel in the stream has exited, before that kernel's completion and memory flush are
// signalled to the stream; each such kernel starts with pdlEntry(), which waits until the previous
// kernel has completed and its memory is visible (griddepcontrol.wait). No kernel triggers its
// dependents early (griddepcontrol.launch_dependents): measured on a 300k-Gaussian 640x480 step, an
// early trigger let waiting CTAs occupy SM slots the running kernel's tail still needed (1.297 ms per
// step against 1.276 without it). Ordering is the plain stream order's; what overlaps is one kernel's
// launch and CTA set-up with the previous one's completion. In a kernel launched without the attribute
// the instruction does nothing.
__device__ __forceinline__ void pdlEntry()
{
    asm volatile("griddepcontrol.wait;" ::: "memory");
}

// Launches `kernel` on stream s with programmatic stream serialisation (see pdlEntry; the kernel must
// call pdlEntry() before it reads anything an earlier kernel wrote).
template <typename... KArgs, typename... Args>
inline void launchPdl(void (*kernel)(KArgs...), dim3 grid, dim3 block, size_t smem, cudaStream_t s, Args &&...args)
{
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid;
    cfg.blockDim = block;
    cfg.dynamicSmemBytes = smem;
    cfg.stream = s;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    cudaLaunchKernelEx(&cfg, kernel, std::forward<Args>(args)...);
}

// Lets a kernel that is about to use `need` bytes of shared memory, static arrays among them, have up to `most`
// of dynamic shared memory on the current device, where `need` is above the default 48 KB.
template <class K>
inline void allowShared(K kernel, size_t need, size_t most, PerDevice &done)
{
    if (need <= 48 * 1024)
        return;
    int device = 0;
    cudaGetDevice(&device);
    done.get(device, [&] {
        cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, int(most));
        return 1;
    });
}

// Device-side sizes of one bin pass. The host never waits for them inside a step: it reads the
// struct back asynchronously and checks it one step later.
struct BinCounts {
    int total;     // tile-Gaussian intersections found by the scan
    int effTotal;  // intersections actually binned: total, or 0 after an overflow / abort
    int abortIter; // -1, or the first step whose intersections did not fit (sticky until cleared)
    int need;      // largest intersection count that did not fit
    int pad[4];
};

// The values of one training step that change from step to step (view, target image, iteration,
// Adam step sizes). Launches given a StepDesc read them from device memory instead of their by-value
// arguments, so a captured CUDA graph of training steps serves any views and learning rates.
struct StepDesc {
    u3dg_camera cam;
    const uint8_t *target; // the view's uint8 image
    int iteration;         // iteration count before the step (0-based step index)
    float stepSize[5];     // Adam: lr / bc1 per group
    float invSqrtBc2;
    int pad[2];
};

// Outputs of the projection kernel, one entry per Gaussian.
struct ProjOut {
    SplatRec *rec;      // raster record (valid where radius > 0)
    uint32_t *depthKey; // float bits of the camera-space depth; 0xFFFFFFFF when not visible
    float *depth;       // camera-space depth (valid where radius > 0)
    int4 *rect;         // tile rectangle x0, y0, x1, y1 (exclusive)
    int *radius;        // 0 = not visible
    uint8_t *flags;     // bit0/1: J clamped in x/y; bit2..4: colour clamped
    float4 *cov2d;      // 2D covariance a, b, c (including eps2d), for inspection
    int *tileCount;     // tiles the Gaussian is listed in (0 when not visible)
    uint32_t *rowTab;   // tile culling: the first rows' spans (tile_cull.cuh, listedTiles); may be null
    int cullTiles;      // 1: list only the tiles the contributing ellipse reaches (then rowTab is set)
};

// Arguments of the chain-rule kernel (backward pass 2), optionally fused with Adam.
struct ChainArgs {
    Params params;
    int n;
    u3dg_camera cam;
    u3dg_raster_settings st;
    const int *radius;
    const SplatRec *rec;
    const uint8_t *flags;
    const int *offs;      // per Gaussian: first intersection in emission order
    const int *tileCount; // per Gaussian: its intersections
    const int2 *listPos;  // per intersection, in emission order: position in the tile lists, tile
    const int *stop;      // per backward block: the list position behind its pixels' last contributor
    const float *partial; // per list position below its block's stop: 9 summed 2D gradients (kPartial
                          // floats; subSlots arrays)
    int subSlots;         // slot arrays of partial (RasterArgs::subSlots), subStride floats apart
    size_t subStride;
    int tilesX, blocksX;  // tiles per row; backward blocks per row
    const BinCounts *counts; // the kernel does nothing when counts->abortIter >= 0
    float *gradAccum;     // |dL/dmean2d| NDC statistic (may be null)
    int *gradCount;       // visibility count (may be null)
    bool conics;          // partials of launchCompositeBackwardList
    bool alone;           // TileBins::alone
    // Non-Adam mode, conics: the Gaussians by depth rank, and space for 9 sums per Gaussian (partialSumKernel;
    // else the chain rule gathers the partials itself).
    const uint32_t *order;
    float *sums;
    Params grads;         // non-Adam mode: gradients are added here
    Params m, v;          // Adam mode: moments
    float stepSize[5];    // Adam mode: lr / bc1 per group
    float invSqrtBc2;
    const StepDesc *desc; // when set: cam, stepSize and invSqrtBc2 come from here
};

// gaussian.cu
// desc (may be null): the camera comes from desc->cam (no spherical harmonics in that mode).
void launchProject(const Params &P, int n, const u3dg_camera &cam, const u3dg_raster_settings &st, int tilesX,
                   int tilesY, const float *shRest, int shDegree, const ProjOut &out, cudaStream_t s,
                   const StepDesc *desc = nullptr);
void launchChain(const ChainArgs &a, bool adam, cudaStream_t s);
void launchAdamSegment(float *p, const float *g, float *m, float *v, int len, float stepSize, float invSqrtBc2,
                       cudaStream_t s);
void launchDensifyClassify(const Params &P, int n, const float *gradAccum, const int *gradCount, float extent,
                           float splitScale, float pruneOpacity, float gradThreshold, int opacityWasReset, int *keep,
                           int *cost, cudaStream_t s);
void launchDensifySelect(int n, const int *cost, const int *costScan, long long budget, int *firstSecond, int *keep,
                         int *accCost, int *isSplit, cudaStream_t s);
void launchDensifyWrite(const Params &P, const Params &M, const Params &V, const Params &P2, const Params &M2,
                        const Params &V2, int n, const int *keep, const int *keepScan, const int *accCost,
                        const int *accScan, const int *isSplit, const int *splitScan, int keptTotal,
                        const float *normals, float log16, cudaStream_t s);
// Skipped when counts (may be null) records an aborted step.
void launchOpacityReset(float *opac, float *mOpac, float *vOpac, int n, float cap, const BinCounts *counts,
                        cudaStream_t s);

// binning.cu
// The depth sort: stable sort of the n 32-bit keys (four 8-bit passes; ties keep index order), items
// kept as (key, index) pairs between passes (pairsA / pairsB: n each); sortedIds receives the
// indices in key order. hist needs binHistEntries(n, 0) entries.
void radixSortDepth(const uint32_t *keys, uint2 *pairsA, uint2 *pairsB, uint32_t *sortedIds, int n, int *hist,
                    cudaStream_t s);
// The capacity check of a bin pass on its intersection count (see BinCounts).
struct ScanCapacity {
    int capacity;
    BinCounts *counts;
    int iteration;
    const StepDesc *desc;
};
// Tile lists of up to 2048 tiles (binsByTile) from the depth order: the Gaussians' tiles in rank order,
// stably by tile.
struct TileBins {
    const uint32_t *sortedIds; // Gaussian id per depth rank
    const int *tileCount;      // per Gaussian: tiles it is listed in
    const int4 *rect;
    int n, tilesX, tiles;
    const SplatRec *cullRec; // tile culling: the records and row tables; else null
    int tileSize;
    const uint32_t *rowTab;
    int *tileOffsets; // tiles + 1
    int *tileOrder;   // tiles, the longest lists first (in 64 steps of length; may be null)
    int *entries;     // per list position: Gaussian id
    int2 *listPos;    // per emission: list position, tile (may be null)
    int *offsById;    // per Gaussian: first emission (may be null)
    bool alone;       // nothing else is on the GPU: few Gaussians may be spread over more threads than they fill
};
bool binsByTile(int tiles);
// hist needs binHistEntries(n, tiles) entries, tileTotals radixDigits(), chunkTotals binChunkEntries(n).
void binByTile(const TileBins &b, int *hist, int *tileTotals, int *chunkTotals, const ScanCapacity &cap, cudaStream_t s);
size_t binHistEntries(int n, int tiles);
size_t binChunkEntries(int n);
// With more tiles the intersections are written out (launchEmit) and sorted by tile id in 8-bit passes:
// stable LSD radix sort of (key, value) pairs on key bits [0, bits); the item count is read on the device
// from *nDev (at most nMax); the initial values are the item indices. Result in *keysOut / *valsOut (one
// of the two buffers). Returns the number of passes; hist needs radixHistEntries(nMax) entries and
// rowTotals radixDigits().
int radixBlocks(int nMax);
size_t radixHistEntries(int nMax);
int radixDigits();
int radixSortPairs(uint32_t *keysA, uint32_t *keysB, uint32_t *valsA, uint32_t *valsB, const int *nDev, int nMax,
                   int bits, int *hist, int *rowTotals, uint32_t **keysOut, uint32_t **valsOut, cudaStream_t s);
// Exclusive prefix sum of n ints: out[0..n], out[n] = total. partial needs scanPartialEntries(n).
size_t scanPartialEntries(int n);
void exclusiveScan(const int *in, int *out, int n, int *partial, cudaStream_t s);
// The scan of in[perm[i]] (the per-Gaussian tile counts in depth-rank order), fused with the bin pass's
// capacity check (launchCapacityCheck on the total out[n], done by the scan's last kernel).
// outById[perm[i]] gets out[i].
void exclusiveScanChecked(const int *in, const uint32_t *perm, int *out, int *outById, int n, int *partial,
                          const ScanCapacity &cap, cudaStream_t s);
// Entries of the per-Gaussian row table of tile culling (ProjOut::rowTab) for n Gaussians.
size_t cullRowEntries(size_t n);
// Checks *total against the intersection capacity (see BinCounts); exclusiveScanChecked does the same
// inside its last kernel.
void launchCapacityCheck(const int *total, int capacity, BinCounts *c, int iteration, cudaStream_t s,
                         const StepDesc *desc = nullptr);
// Emission of the intersections in depth-rank order: tile key and Gaussian id per intersection (the
// tiles that the projection counted, ProjOut::tileCount).
void launchEmit(const uint32_t *sortedIds, const int *offs, const int4 *rect, int n, const BinCounts *c, int capacity,
                int tilesX, const SplatRec *cullRec, int tileSize, const uint32_t *rowTab, uint32_t *keys, int *emitGid,
                cudaStream_t s);
// After that sort: the Gaussian id of every sorted entry, the list position and tile of every emission
// (listPos may be null) and the tile offsets (a binary search in the sorted keys).
void launchFinalizeBins(const uint32_t *sortedKeys, const uint32_t *sortedEmit, const int *emitGid, const BinCounts *c,
                        int capacity, int tiles, int *entries, int2 *listPos, int *tileOffsets, cudaStream_t s);

// raster.cu
struct RasterArgs {
    const int *tileOffsets;
    const int *entries; // per tile-sorted entry: Gaussian id
    const int *tileOrder; // the order in which the forward takes the tiles (null: row-major pixel blocks)
    const SplatRec *rec;
    int width, height, tileSize, tilesX;
    float bg[3];
    float minAlpha, minTransmittance;
    // Pixel blocks of the backward (PB x PB, PB = 8 for tile size 8, else 16).
    int blocksX, blocksY;
    int *counters; // 2 ints, zero between launches: the backward's units handed out, CTAs done
    // What a forward keeps for the backward (segment > 0; 0: images only). A tile's list is cut every
    // `segment` entries; for each segment but the first that a pixel reaches, ck holds the colour the
    // pixel blends in it and its transmittance before it, so that the backward can replay every segment
    // by itself. Slot tileOffsets[tile] / segment + tile + s holds segment s of a tile, a float4 per
    // pixel (8x8 blocks row-major, pixels row-major within). blockMax: per 8x8 block, its pixels'
    // largest contributor count.
    int segment;
    float4 *ck;
    int *blockMax;
    int backwardDepth;     // list entries staged per thread per batch, backward: 1 or 2 (same results)
    // Tiles larger than the backward's 16x16 pixel block are covered by several CTAs: each writes its
    // sums into its own slot array (slot = the block's position in its tile, row-major), subSlots
    // arrays of subStride floats apart, and the chain rule adds a Gaussian's slots in slot order.
    int subSlots;
    size_t subStride;
};
// Work of the backward: (pixel block, segment) of every segment with a contributor into units,
// their number into unitCount, and per pixel block the list position behind its last contributor into
// stop.
void launchBackwardUnits(const RasterArgs &a, int *stop, int2 *units, int *unitCount, cudaStream_t s);
// Whether the forward of so many tiles takes them in the order of their list lengths (RasterArgs::tileOrder).
bool forwardOrdersTiles(int tiles, int tileSize);
void launchCompositeForward(const RasterArgs &a, float *rgb, float *finalT, int *nContrib, cudaStream_t s);
// partial: kPartial floats per list position, in a.subSlots slot arrays. Partials from a block's stop on
// are not written: they are zero, and ChainArgs' reader skips them.
void launchCompositeBackward(const RasterArgs &a, const float *dLdRgb, const float *finalT, const int *nContrib,
                             float *partial, const int *stop, const int2 *units, const int *unitCount,
                             cudaStream_t s);
// Whether RasterArgs::backwardDepth makes a difference to launchCompositeBackward: at tiles of 16 a segment of 64
// entries is one batch.
inline bool backwardTakesDepth(int tileSize) { return tileSize != 16; }
// The same over whole lists: partials hold dL/dmean2d and dL/dconic, stop is written, and a forward with
// segment 0 is enough.
void launchCompositeBackwardList(const RasterArgs &a, const float *dLdRgb, const float *finalT, const int *nContrib,
                                 float *partial, int *stop, cudaStream_t s);

// loss.cu
struct LossScratch {
    float *abc;        // 3 maps x 3 channels x P
    double *blockSums; // 3 doubles per block: l1, ssim, squared error
    int blocks;
};
int lossBlocks(int width, int height);
// target is either float (targetF) or uint8 (targetU8, converted as float(u8) * (1/255f)).
// desc (may be null): the uint8 target comes from desc->target.
// Also reduces the block sums into the step's LossValue / PSNR and updates the EMA stats (may be null;
// Trainer.cpp:88-92) unless counts (may be null) records an aborted step. out3 (may be null) gets
// total, l1, ssim; psnrOut (may be null) the PSNR. With desc, iteration is desc->iteration + 1.
void launchLoss(const float *render, const float *targetF, const uint8_t *targetU8, int width, int height, float lambda,
                float *grad, const LossScratch &ls, DevStats *stats, int iteration, const BinCounts *counts, float *out3,
                float *psnrOut, cudaStream_t s, const StepDesc *desc = nullptr);
// PSNR of the render against a uint8 target, accumulated in double (evaluatePsnr).
void launchPsnrU8(const float *render, const uint8_t *target, size_t count, double *sumOut, cudaStream_t s);
void launchPsnrF(const float *a, const float *b, size_t count, double *sumOut, cudaStream_t s);
// TrainImage::quantize on the device: lround(clamp(v, 0, 1) * 255) per value.
void launchQuantize(const float *rgb, size_t count, uint8_t *out, cudaStream_t s);

} // namespace u3dg
