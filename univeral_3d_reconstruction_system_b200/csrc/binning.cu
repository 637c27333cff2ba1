// binning.cu - tile binning on the GPU (Rasterizer::binTiles, Rasterizer.cpp:206-261).
//
// The reference sorts the visible Gaussians by the float bits of their depth with a stable LSD
// radix sort (ties keep index order), then buckets them per tile in that order, so every tile list
// is depth-sorted. Here the same order comes from two stable sorts:
//   1. (depth bits, Gaussian id) over all Gaussians -> depth rank; invisible ones get key
//      0xFFFFFFFF and sort last: four passes of 8 bits, a histogram and a scatter kernel each, or
//      one kernel for up to 4096 Gaussians (radixSortDepth);
//   2. the ranks' intersections, in rank order, by tile. Up to 2048 tiles (binByTile) they are never
//      written out: a chunk of ranks counts its intersections per tile, the counts are scanned over the
//      chunks, and the chunk then goes through its intersections again and writes each one's Gaussian id
//      straight to its place in the tile lists. With more tiles they are emitted in rank order (an
//      exclusive scan of per-rank tile counts gives each Gaussian its slots), keyed by tile id, and
//      sorted by radix passes on the tile id.
// Within a tile the rank order, i.e. (depth bits, id), survives, which is exactly the reference's list.
// Emission order, in which the chain rule adds up a Gaussian's partials, is rank order too.
//
// The intersection count is only known on the device, so nothing here waits for the host: a capacity
// check on the count turns an overflow into empty lists plus a flag the host reads later (it then grows
// the buffers and replays the step). Grids of the first path follow the host-known Gaussian count; those
// of the second are sized for the capacity.
//
// In-block ranks of the stable scatters come from warp votes: each warp ranks its items among
// equal digits and the warps' counts per digit are added in warp order.

#include "tile_cull.cuh"

#include <algorithm>
#include <climits>

namespace u3dg {

namespace {

constexpr int kThreads = 256;
constexpr int kItemsPerThread = 4;
constexpr int kTile = kThreads * kItemsPerThread; // items per block round
constexpr int kWarps = kThreads / 32;
// Blocks of a radix pass at most (each owns a contiguous chunk of the items in rounds of kTile).
#ifndef U3DG_RADIX_MAX_BLOCKS
#define U3DG_RADIX_MAX_BLOCKS (148 * 6)
#endif
constexpr int kMaxBlocks = U3DG_RADIX_MAX_BLOCKS;
constexpr int kWideBits = 11; // one pass sorts tile ids up to 2048; other sorts use 8-bit digits

// Block-wide exclusive scan of one int per thread (blockDim == 256); returns the block total.
__device__ __forceinline__ int blockExclusiveScan(int v, int &total)
{
    __shared__ int warpSums[kWarps];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    int x = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int y = __shfl_up_sync(0xffffffffu, x, o);
        if (lane >= o)
            x += y;
    }
    if (lane == 31)
        warpSums[warp] = x;
    __syncthreads();
    if (warp == 0) {
        int w = lane < kWarps ? warpSums[lane] : 0;
#pragma unroll
        for (int o = 1; o < kWarps; o <<= 1) {
            const int y = __shfl_up_sync(0xffffffffu, w, o);
            if (lane >= o)
                w += y;
        }
        if (lane < kWarps)
            warpSums[lane] = w; // inclusive
    }
    __syncthreads();
    total = warpSums[kWarps - 1];
    const int before = warp > 0 ? warpSums[warp - 1] : 0;
    __syncthreads();
    return before + x - v;
}

// The contiguous item range of block b when n items are split over G blocks in rounds of kTile.
__device__ __forceinline__ void chunkOf(int n, int G, int b, int &begin, int &end)
{
    const long long per = (long long)G * kTile;
    const int rounds = int((n + per - 1) / per);
    const long long chunk = (long long)rounds * kTile;
    begin = int(std::min<long long>(n, b * chunk));
    end = int(std::min<long long>(n, begin + chunk));
}

template <int DB>
__global__ void __launch_bounds__(kThreads) radixHistKernel(const uint32_t *keys, const int *nPtr, int shift, int *hist, int G)
{
    pdlEntry();
    constexpr int R = 1 << DB;
    __shared__ int counts[R];
    for (int d = threadIdx.x; d < R; d += kThreads)
        counts[d] = 0;
    __syncthreads();
    int begin, end;
    chunkOf(*nPtr, G, blockIdx.x, begin, end);
    for (int i = begin + threadIdx.x; i < end; i += kThreads)
        atomicAdd(&counts[(keys[i] >> shift) & uint32_t(R - 1)], 1);
    __syncthreads();
    for (int d = threadIdx.x; d < R; d += kThreads)
        hist[size_t(d) * G + blockIdx.x] = counts[d];
}

// One block per digit: exclusive scan of that digit's row of G block counts; rowTotals[d] = sum.
__global__ void __launch_bounds__(kThreads) radixRowScanKernel(int *hist, int G, int *rowTotals)
{
    pdlEntry();
    int *row = hist + size_t(blockIdx.x) * G;
    int carry = 0;
    for (int c0 = 0; c0 < G; c0 += kThreads) {
        const int i = c0 + threadIdx.x;
        const int v = i < G ? row[i] : 0;
        int total;
        const int ex = blockExclusiveScan(v, total);
        if (i < G)
            row[i] = carry + ex;
        carry += total;
    }
    if (threadIdx.x == 0)
        rowTotals[blockIdx.x] = carry;
}

// Stable scatter of one pass with 2^DB digits. Per round of kTile items, each warp ranks its items
// among equal digits with match-any votes and keeps per-digit counts (at most 128, one byte) in shared
// memory; an item's position is its digit's base + the counts of the warps before it (they hold
// earlier items) + its rank in its warp. After the round the last item of each (warp, digit) advances
// the digit's base and clears that count, so only the touched counts are reset.
template <int DB>
__global__ void __launch_bounds__(kThreads) radixScatterKernel(const uint32_t *keysIn, const uint32_t *valsIn,
                                                               uint32_t *keysOut, uint32_t *valsOut, const int *nPtr,
                                                               int shift, const int *hist, const int *rowTotals, int G)
{
    pdlEntry();
    const int n = *nPtr;
    constexpr int R = 1 << DB;
    __shared__ uint8_t warpCounts[kWarps][R];
    __shared__ int base[R];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    int begin, end;
    chunkOf(n, G, blockIdx.x, begin, end);
    for (int k = threadIdx.x; k < kWarps * R; k += kThreads)
        (&warpCounts[0][0])[k] = 0;
    {
        // Digit base: exclusive scan of the digit totals, plus this block's row prefix.
        int carry = 0;
        for (int c0 = 0; c0 < R; c0 += kThreads) {
            const int d = c0 + threadIdx.x;
            int total;
            const int ex = blockExclusiveScan(rowTotals[d], total);
            base[d] = carry + ex + hist[size_t(d) * G + blockIdx.x];
            carry += total;
        }
    }
    __syncthreads();
    const uint32_t lanesBelow = (1u << lane) - 1u;
    uint8_t *myCounts = warpCounts[warp];
    for (int r0 = begin; r0 < end; r0 += kTile) {
        const int first = r0 + warp * (32 * kItemsPerThread);
        uint32_t key[kItemsPerThread], val[kItemsPerThread];
        int digit[kItemsPerThread], local[kItemsPerThread];
#pragma unroll
        for (int r = 0; r < kItemsPerThread; ++r) {
            const int i = first + r * 32 + lane;
            const bool valid = i < end;
            key[r] = valid ? keysIn[i] : 0u;
            val[r] = valid ? (valsIn ? valsIn[i] : uint32_t(i)) : 0u;
            const int d = valid ? int((key[r] >> shift) & uint32_t(R - 1)) : R;
            digit[r] = d;
            local[r] = 0;
            const uint32_t peers = __match_any_sync(0xffffffffu, d);
            int before = 0;
            if (valid) {
                before = myCounts[d];
                local[r] = before + __popc(peers & lanesBelow);
            }
            __syncwarp();
            if (valid && lane == __ffs(peers) - 1)
                myCounts[d] = uint8_t(before + __popc(peers));
            __syncwarp();
        }
        __syncthreads();
        bool last[kItemsPerThread];
#pragma unroll
        for (int r = 0; r < kItemsPerThread; ++r) {
            const int d = digit[r];
            last[r] = false;
            if (d < R) {
                int cross = 0;
                for (int w = 0; w < warp; ++w)
                    cross += warpCounts[w][d];
                const int pos = base[d] + cross + local[r];
                keysOut[pos] = key[r];
                valsOut[pos] = val[r];
                last[r] = local[r] == int(myCounts[d]) - 1;
            }
        }
        __syncthreads();
#pragma unroll
        for (int r = 0; r < kItemsPerThread; ++r)
            if (last[r])
                atomicAdd(&base[digit[r]], int(myCounts[digit[r]]));
        __syncthreads();
#pragma unroll
        for (int r = 0; r < kItemsPerThread; ++r)
            if (last[r])
                myCounts[digit[r]] = 0;
        __syncthreads();
    }
}

// Capacity check of a bin pass on its intersection count t: the usable count is t, or 0 when t
// exceeds the intersection buffers or a previous step already aborted (the abort is sticky until the
// host clears it). iteration identifies the aborted step for the host.
__device__ __forceinline__ void checkCapacity(int t, int capacity, BinCounts *c, int iteration, const StepDesc *desc)
{
    if (desc)
        iteration = desc->iteration;
    const bool over = t < 0 || t > capacity;
    if (over) {
        if (c->abortIter < 0)
            c->abortIter = iteration;
        c->need = max(c->need, t < 0 ? INT_MAX : t);
    }
    c->total = t;
    c->effTotal = (over || c->abortIter >= 0) ? 0 : t;
}

// Exclusive scan, reduce-then-scan over a host-known n.
constexpr int kScanTile = kThreads * 8;

// The scan's input element i: in[i], or in[perm[i]] with a permutation (the per-Gaussian tile counts
// taken in depth-rank order).
__device__ __forceinline__ int scanInput(const int *in, const uint32_t *perm, int i)
{
    return in[perm ? int(perm[i]) : i];
}

__global__ void __launch_bounds__(kThreads) scanReduceKernel(const int *in, const uint32_t *perm, int n, int *partial)
{
    pdlEntry();
    const int base = blockIdx.x * kScanTile;
    int s = 0;
#pragma unroll
    for (int r = 0; r < 8; ++r) {
        const int i = base + r * kThreads + threadIdx.x;
        if (i < n)
            s += scanInput(in, perm, i);
    }
    int total;
    blockExclusiveScan(s, total);
    if (threadIdx.x == 0)
        partial[blockIdx.x] = total;
}

__global__ void __launch_bounds__(kThreads) scanPartialKernel(int *partial, int B)
{
    pdlEntry();
    int carry = 0;
    for (int c0 = 0; c0 < B; c0 += kThreads) {
        const int i = c0 + threadIdx.x;
        const int v = i < B ? partial[i] : 0;
        int total;
        const int ex = blockExclusiveScan(v, total);
        if (i < B)
            partial[i] = carry + ex;
        carry += total;
    }
    if (threadIdx.x == 0)
        partial[B] = carry;
}

// cap.counts (may be null): block 0 also runs the bin pass's capacity check on the total.
__global__ void __launch_bounds__(kThreads) scanDownsweepKernel(const int *in, const uint32_t *perm, int *out, int *outById, int n,
                                                                const int *partial, int B, ScanCapacity cap)
{
    pdlEntry();
    const int base = blockIdx.x * kScanTile + threadIdx.x * 8;
    int v[8];
    int s = 0;
#pragma unroll
    for (int r = 0; r < 8; ++r) {
        v[r] = (base + r < n) ? scanInput(in, perm, base + r) : 0;
        s += v[r];
    }
    int total;
    int run = blockExclusiveScan(s, total) + partial[blockIdx.x];
#pragma unroll
    for (int r = 0; r < 8; ++r) {
        if (base + r < n) {
            out[base + r] = run;
            if (outById)
                outById[perm[base + r]] = run;
        }
        run += v[r];
    }
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        out[n] = partial[B];
        if (cap.counts != nullptr)
            checkCapacity(partial[B], cap.capacity, cap.counts, cap.iteration, cap.desc);
    }
}

// Capacity check of a bin pass on its scan total (checkCapacity), when the scan had no kernels to
// fold it into.
__global__ void capacityKernel(const int *total, int capacity, BinCounts *c, int iteration, const StepDesc *desc)
{
    pdlEntry();
    checkCapacity(*total, capacity, c, iteration, desc);
}

// ---------------------------------------------------------------- depth sort

// A pass is two kernels over chunks of the items: chunk histograms (hist[chunk][digit], so a chunk's row
// and the rows of a digit range are contiguous), and a scatter whose blocks add up the rows themselves.
// Every block reads every row, so the chunks are kept to about one per SM (148 rows of 1 KB: 22 MB from L2
// per pass) and the rows are dealt out to four groups of the block's threads.
constexpr int kDigits = 256;
constexpr int kDepthThreads = 1024, kDepthWarps = kDepthThreads / 32, kDepthGroups = kDepthThreads / kDigits;
constexpr int kDepthItems = 2;
constexpr int kDepthTile = kDepthThreads * kDepthItems;
constexpr int kDepthChunks = 160;

// The lanes of the warp with the same digit d (0 .. 255, or kDigits for none). Nine votes: match-any takes
// about 64 cycles of the SM per warp on 32 different digits (tile lists of 4k Gaussians 47 us, 44.6 with votes,
// of 300k 116 and 113.5).
__device__ __forceinline__ uint32_t digitPeers(int d)
{
    uint32_t peers = 0xffffffffu;
#pragma unroll
    for (int b = 0; b < 9; ++b) {
        const uint32_t set = __ballot_sync(0xffffffffu, d >> b & 1);
        peers &= d >> b & 1 ? set : ~set;
    }
    return peers;
}

__device__ __forceinline__ uint32_t depthDigit(uint32_t key, int shift) { return (key >> shift) & uint32_t(kDigits - 1); }

// Stable ranks of a warp's items (32 consecutive ones per round) among those with the same digit, and the
// digits' counts, which start at zero. left: items from this lane's first one on.
template <int kItems>
__device__ __forceinline__ void rankInWarp(const uint2 (&item)[kItems], int shift, int left, uint16_t *counts,
                                           int (&local)[kItems])
{
    const int lane = threadIdx.x & 31;
    uint32_t peers[kItems];
#pragma unroll
    for (int r = 0; r < kItems; ++r)
        peers[r] = digitPeers(r * 32 < left ? int(depthDigit(item[r].x, shift)) : kDigits);
#pragma unroll
    for (int r = 0; r < kItems; ++r) {
        const bool valid = r * 32 < left;
        const int d = int(depthDigit(item[r].x, shift));
        const int seen = counts[d];
        local[r] = seen + __popc(peers[r] & ((1u << lane) - 1u));
        __syncwarp();
        if (valid && lane == __ffs(peers[r]) - 1)
            counts[d] = uint16_t(seen + __popc(peers[r]));
        __syncwarp();
    }
}

__global__ void __launch_bounds__(kDepthThreads) depthHistKernel(const uint32_t *keys, const uint2 *pairs, int n, int shift,
                                                                 int chunk, int *hist)
{
    pdlEntry();
    __shared__ int counts[kDigits];
    if (threadIdx.x < kDigits)
        counts[threadIdx.x] = 0;
    __syncthreads();
    const int begin = blockIdx.x * chunk, end = min(n, begin + chunk), lane = threadIdx.x & 31;
    for (int i0 = begin; i0 < end; i0 += kDepthThreads) {
        const int i = i0 + threadIdx.x;
        const int d = i < end ? int(depthDigit(pairs ? pairs[i].x : keys[i], shift)) : kDigits;
        // One addition per distinct digit of a warp: the upper digits of depths hold few values.
        const uint32_t peers = digitPeers(d);
        if (d < kDigits && lane == __ffs(peers) - 1)
            atomicAdd(&counts[d], __popc(peers));
    }
    __syncthreads();
    if (threadIdx.x < kDigits)
        hist[blockIdx.x * kDigits + threadIdx.x] = counts[threadIdx.x];
}

// Where a pass of the depth sort keeps its items: (key, value) pairs in and out, so each item is one
// load and one scattered 8-byte store; the last pass writes the values only (the keys are done).
struct PairIO {
    const uint2 *in;    // when null: the keys, valued by their index
    uint2 *out;         // when set: write (key, value) pairs
    uint32_t *valsOnly; // when set: write the values only
};

__global__ void __launch_bounds__(kDepthThreads) depthScatterKernel(const uint32_t *keys, int n, int shift, int chunk,
                                                                    const int *hist, PairIO io)
{
    pdlEntry();
    __shared__ uint16_t counts[kDepthWarps][kDigits];
    __shared__ int base[kDigits], before[kDepthGroups][kDigits], all[kDepthGroups][kDigits], warpSums[kDigits / 32];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int begin = blockIdx.x * chunk, end = min(n, begin + chunk);
    {
        // This chunk's first position of a digit: all items of lower digits, plus the digit's in the chunks
        // before.
        const int d = tid % kDigits, group = tid / kDigits;
        int sumBefore = 0, sumAll = 0;
#pragma unroll 8
        for (int c = group; c < int(gridDim.x); c += kDepthGroups) {
            const int v = hist[c * kDigits + d];
            sumAll += v;
            sumBefore += c < int(blockIdx.x) ? v : 0;
        }
        before[group][d] = sumBefore;
        all[group][d] = sumAll;
        __syncthreads();
        int total = 0, scan = 0;
        if (tid < kDigits) {
#pragma unroll
            for (int g = 0; g < kDepthGroups; ++g)
                total += all[g][tid];
            scan = total;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const int y = __shfl_up_sync(0xffffffffu, scan, o);
                if (lane >= o)
                    scan += y;
            }
            if (lane == 31)
                warpSums[warp] = scan;
        }
        __syncthreads();
        if (tid < kDigits) {
            int at = scan - total;
            for (int w = 0; w < warp; ++w)
                at += warpSums[w];
#pragma unroll
            for (int g = 0; g < kDepthGroups; ++g)
                at += before[g][tid];
            base[tid] = at;
        }
    }
    for (int r0 = begin; r0 < end; r0 += kDepthTile) {
        const int first = r0 + warp * (32 * kDepthItems);
        uint2 item[kDepthItems];
        int local[kDepthItems];
#pragma unroll
        for (int r = 0; r < kDepthItems; ++r) {
            const int i = first + r * 32 + lane;
            item[r] = i >= end ? make_uint2(0u, 0u) : io.in ? io.in[i] : make_uint2(keys[i], uint32_t(i));
        }
#pragma unroll
        for (int k = 0; k < kDigits / 32; ++k)
            counts[warp][k * 32 + lane] = 0;
        __syncwarp();
        rankInWarp<kDepthItems>(item, shift, end - first - lane, counts[warp], local);
        __syncthreads();
        int run = 0; // digit `tid`: the warps' counts to what the warps before hold
        if (tid < kDigits) {
#pragma unroll 8
            for (int w = 0; w < kDepthWarps; ++w) {
                const int c = counts[w][tid];
                counts[w][tid] = uint16_t(run);
                run += c;
            }
        }
        __syncthreads();
#pragma unroll
        for (int r = 0; r < kDepthItems; ++r) {
            if (first + r * 32 + lane >= end)
                continue;
            const int d = int(depthDigit(item[r].x, shift));
            const int pos = base[d] + counts[warp][d] + local[r];
            if (io.out)
                io.out[pos] = item[r];
            else
                io.valsOnly[pos] = item[r].y;
        }
        __syncthreads();
        if (tid < kDigits)
            base[tid] += run;
    }
}

// Few items: all four passes in one CTA, the items in its registers (a warp's ones consecutive) and exchanged
// through shared memory; bound by the latency of its steps (3.5 us per pass). 4k items: sort and tile lists
// 44.6 us with eight launches, 35.5 with this one; 6k (8 items a thread): even, 12k: 48.0 and 61.0. So it takes
// what 4 items a thread hold.
constexpr int kSmallItems = 4, kSmallSort = kSmallItems * kDepthThreads;

__global__ void __launch_bounds__(kDepthThreads) depthSortSmallKernel(const uint32_t *keys, int n, uint32_t *sortedIds)
{
    pdlEntry();
    extern __shared__ __align__(16) uint8_t shared[];
    uint2 *exchange = reinterpret_cast<uint2 *>(shared);
    uint16_t(*counts)[kDigits] = reinterpret_cast<uint16_t(*)[kDigits]>(exchange + kSmallItems * kDepthThreads);
    __shared__ int groups[kDepthGroups][kDigits], warpSums[kDigits / 32];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, first = warp * (32 * kSmallItems) + lane;
    uint2 item[kSmallItems];
#pragma unroll
    for (int r = 0; r < kSmallItems; ++r) {
        const int i = first + r * 32;
        item[r] = make_uint2(i < n ? keys[i] : 0u, uint32_t(i));
    }
    for (int shift = 0; shift < 32; shift += 8) {
        int local[kSmallItems];
#pragma unroll
        for (int k = 0; k < kDigits / 32; ++k)
            counts[warp][k * 32 + lane] = 0;
        __syncwarp();
        rankInWarp<kSmallItems>(item, shift, n - first, counts[warp], local);
        __syncthreads();
        {
            // A digit's counts of a group of warps to what the group's warps before hold.
            const int d = tid % kDigits, group = tid / kDigits;
            constexpr int per = kDepthWarps / kDepthGroups;
            int c[per], sum = 0;
#pragma unroll
            for (int w = 0; w < per; ++w)
                c[w] = counts[group * per + w][d];
#pragma unroll
            for (int w = 0; w < per; ++w) {
                counts[group * per + w][d] = uint16_t(sum);
                sum += c[w];
            }
            groups[group][d] = sum;
        }
        __syncthreads();
        int total = 0, scan = 0;
        if (tid < kDigits) {
#pragma unroll
            for (int g = 0; g < kDepthGroups; ++g)
                total += groups[g][tid];
            scan = total;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const int y = __shfl_up_sync(0xffffffffu, scan, o);
                if (lane >= o)
                    scan += y;
            }
            if (lane == 31)
                warpSums[warp] = scan;
        }
        __syncthreads();
        if (tid < kDigits) {
            int at = scan - total;
            for (int w = 0; w < warp; ++w)
                at += warpSums[w];
#pragma unroll
            for (int g = 0; g < kDepthGroups; ++g) {
                const int c = groups[g][tid];
                groups[g][tid] = at; // the group's first position of the digit
                at += c;
            }
        }
        __syncthreads();
#pragma unroll
        for (int r = 0; r < kSmallItems; ++r)
            if (first + r * 32 < n) {
                const int d = int(depthDigit(item[r].x, shift));
                const int pos = groups[warp / (kDepthWarps / kDepthGroups)][d] + counts[warp][d] + local[r];
                if (shift < 24)
                    exchange[pos] = item[r];
                else
                    sortedIds[pos] = item[r].y;
            }
        if (shift < 24) {
            __syncthreads();
#pragma unroll
            for (int r = 0; r < kSmallItems; ++r)
                if (first + r * 32 < n)
                    item[r] = exchange[first + r * 32];
        }
    }
}

// ---------------------------------------------------------------- tile lists of up to 2048 tiles

// A block of T threads takes a chunk of ranks, each of its warps R consecutive ones (at most one per lane). Few
// Gaussians are cut finer, as a warp goes through its ranks' tiles one after the other and 512 ranks to a block
// would leave most of the chip idle. Sort and lists, us, by 512 / 64 / 32 ranks to a block (32 / 32 / 8 to a warp):
// 5,000 Gaussians at 640x480 389 / 142 / 96, 5,000 at 400x304 in tiles of 8 652 / 208 / 126, without culling 380 /
// 340 / 175, 1,000 at 200x150 81 / 50 / 40, 15,000 at 640x480 221 / 104 / 82, 4,000 at 96x72 36 / 34 / 32. Beyond,
// blocks of 512 keep the counts that are scanned few (300k at 640x480: 586 rows of 1,200); and where other work
// fills the chip, their warps have no idle lanes (16 scenes at once 4,260 steps per second, 4,200 by 32).
constexpr int kMaxTiles = 1 << kWideBits;
template <int T, int R>
struct RankShape {
    static constexpr int THREADS = T, WARPS = T / 32, PER_WARP = R, CHUNK = WARPS * R;
};
using ManyRanks = RankShape<512, 32>;
using FewRanks = RankShape<128, 8>;
constexpr int kFewGaussians = 16384;

template <class S>
int rankChunks(int n)
{
    return std::max(1, (n + S::CHUNK - 1) / S::CHUNK);
}

// The rank of a thread, n where it has none.
template <class S>
__device__ __forceinline__ int rankOf(int chunk, int n)
{
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    return lane < S::PER_WARP ? min(n, chunk * S::CHUNK + warp * S::PER_WARP + lane) : n;
}

// The k-th tile (row-major) in which Gaussian g with rectangle q is listed.
__device__ __forceinline__ int2 listedTile(const SplatRec *cullRec, const uint32_t *rowTab, int tileSize, int g,
                                           const int4 &q, int k)
{
    if (cullRec == nullptr) {
        const int wdt = q.z - q.x;
        return make_int2(q.x + k % wdt, q.y + k / wdt);
    }
    // The k-th reachable tile: the Gaussian's row table (one 32-byte row, two vector loads; entries past its
    // rows are unused), then (rows beyond it, rare) the rows' spans.
    const uint4 *tab = reinterpret_cast<const uint4 *>(rowTab + size_t(g) * kCullRows);
    const uint4 t0 = tab[0], t1 = tab[1];
    const uint32_t tv[kCullRows] = {t0.x, t0.y, t0.z, t0.w, t1.x, t1.y, t1.z, t1.w};
    const int rows = q.w - q.y;
    int before = 0;
#pragma unroll
    for (int i = 0; i < kCullRows; ++i) {
        if (i >= rows)
            break;
        const int through = int(tv[i] & 0xffffu);
        if (k < through)
            return make_int2(int(tv[i] >> 16) + (k - before), q.y + i);
        before = through;
    }
    k -= before;
    const CullShape cs = cullShape(cullRec, g);
    for (int row = q.y + kCullRows; row < q.w; ++row) {
        int c0, c1;
        cullSpan(cs, q, row, tileSize, c0, c1);
        if (k < c1 - c0)
            return make_int2(c0 + k, row);
        k -= c1 - c0;
    }
    return make_int2(q.x, q.y);
}

// A rank's Gaussian: its rectangle and, culling, the first rows' spans in registers.
struct Listed {
    int gid = 0, count = 0;
    int4 q = make_int4(0, 0, 0, 0);
    uint32_t tab[kCullRows] = {};
};

__device__ __forceinline__ Listed loadListed(const uint32_t *sortedIds, const int *tileCount, const int4 *rect,
                                             const uint32_t *rowTab, bool cull, int r, int n)
{
    Listed l;
    if (r < n) {
        l.gid = int(sortedIds[r]);
        l.count = tileCount[l.gid];
        l.q = rect[l.gid];
        if (cull) {
            const uint4 *t = reinterpret_cast<const uint4 *>(rowTab + size_t(l.gid) * kCullRows);
            const uint4 t0 = t[0], t1 = t[1];
            const uint32_t v[kCullRows] = {t0.x, t0.y, t0.z, t0.w, t1.x, t1.y, t1.z, t1.w};
#pragma unroll
            for (int i = 0; i < kCullRows; ++i)
                l.tab[i] = v[i];
        }
    }
    return l;
}

// f(tile) for every tile of the rank, row-major.
template <class F>
__device__ __forceinline__ void eachTile(const Listed &l, const SplatRec *cullRec, int tileSize, int tilesX, F &&f)
{
    if (l.count == 0)
        return;
    if (cullRec == nullptr) {
        for (int row = l.q.y; row < l.q.w; ++row)
            for (int c = l.q.x; c < l.q.z; ++c)
                f(row * tilesX + c);
        return;
    }
    const int rows = l.q.w - l.q.y;
    int before = 0;
#pragma unroll
    for (int i = 0; i < kCullRows; ++i) {
        if (i >= rows)
            break;
        const int through = int(l.tab[i] & 0xffffu), t0 = (l.q.y + i) * tilesX + int(l.tab[i] >> 16);
        for (int c = 0; c < through - before; ++c)
            f(t0 + c);
        before = through;
    }
    if (rows > kCullRows) {
        const CullShape cs = cullShape(cullRec, l.gid);
        for (int row = l.q.y + kCullRows; row < l.q.w; ++row) {
            int c0, c1;
            cullSpan(cs, l.q, row, tileSize, c0, c1);
            for (int c = c0; c < c1; ++c)
                f(row * tilesX + c);
        }
    }
}

// hist[chunk][tile]: intersections of the chunk's ranks per tile; chunkTotals[chunk]: all of them.
template <class S>
__global__ void __launch_bounds__(S::THREADS) tileCountKernel(TileBins b, int *hist, int *chunkTotals)
{
    pdlEntry();
    extern __shared__ int counts[]; // per tile
    __shared__ int total;
    for (int d = threadIdx.x; d < b.tiles; d += S::THREADS)
        counts[d] = 0;
    if (threadIdx.x == 0)
        total = 0;
    const Listed l = loadListed(b.sortedIds, b.tileCount, b.rect, b.rowTab, b.cullRec != nullptr,
                                rankOf<S>(blockIdx.x, b.n), b.n);
    __syncthreads();
    eachTile(l, b.cullRec, b.tileSize, b.tilesX, [&](int tile) { atomicAdd(&counts[tile], 1); });
    const int sum = __reduce_add_sync(0xffffffffu, l.count); // at most 32 * kMaxTiles
    if ((threadIdx.x & 31) == 0)
        atomicAdd(&total, sum);
    __syncthreads();
    if (threadIdx.x == 0)
        chunkTotals[blockIdx.x] = total;
    for (int d = threadIdx.x; d < b.tiles; d += S::THREADS)
        hist[size_t(blockIdx.x) * b.tiles + d] = counts[d];
}

// Blocks of 32 tiles (a warp's lanes) by 32 groups of chunks: hist to the tile's intersections in the chunks
// before, in place, and tileTotals. The last block: chunkTotals to the chunks' first emission, in place,
// and the capacity check on their sum.
constexpr int kScanThreads = 1024, kScanGroups = kScanThreads / 32;

__global__ void __launch_bounds__(kScanThreads) tileScanKernel(int *hist, int chunks, int tiles, int *tileTotals,
                                                               int *chunkTotals, ScanCapacity cap)
{
    pdlEntry();
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    if (int(blockIdx.x) == int(gridDim.x) - 1) {
        if (warp > 0)
            return;
        long long carry = 0;
        for (int c0 = 0; c0 < chunks; c0 += 32) {
            const int c = c0 + lane, v = c < chunks ? chunkTotals[c] : 0; // at most 512 * kMaxTiles = 2^20
            int incl = v;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const int y = __shfl_up_sync(0xffffffffu, incl, o);
                if (lane >= o)
                    incl += y;
            }
            if (c < chunks)
                chunkTotals[c] = int(min(carry + incl - v, (long long)INT_MAX));
            carry += __shfl_sync(0xffffffffu, incl, 31);
        }
        if (lane == 0)
            checkCapacity(int(min(carry, (long long)INT_MAX)), cap.capacity, cap.counts, cap.iteration, cap.desc);
        return;
    }
    __shared__ int groupSums[kScanGroups][32];
    const int t = blockIdx.x * 32 + lane, per = (chunks + kScanGroups - 1) / kScanGroups;
    const int c0 = warp * per, c1 = min(chunks, c0 + per);
    int sum = 0;
    if (t < tiles) {
#pragma unroll 8
        for (int c = c0; c < c1; ++c)
            sum += hist[size_t(c) * tiles + t];
    }
    groupSums[warp][lane] = sum;
    __syncthreads();
    if (t >= tiles)
        return;
    int run = 0;
    for (int w = 0; w < warp; ++w)
        run += groupSums[w][lane];
    if (warp == kScanGroups - 1)
        tileTotals[t] = run + sum;
#pragma unroll 8
    for (int c = c0; c < c1; ++c) {
        const int v = hist[size_t(c) * tiles + t];
        hist[size_t(c) * tiles + t] = run;
        run += v;
    }
}

// Writes the chunk's Gaussian ids to the tile lists (and, with listPos, where each emission went, and with
// offsById each Gaussian's first emission). The chunk first lists its ranks' intersections (tile and lane, in
// rank order) and counts them per warp and tile, the counts are added up over the block's warps in order, and each
// warp then goes through its list, 32 intersections at a time, ranking equal tiles by match-any votes, with
// no barrier on the way. A chunk with more than kListed intersections lists so many at a time, and enumerates its
// ranks' tiles again for each; without culling, where a rank's k-th tile is a division away, it finds each one's
// rank by a search over the warp's lanes instead. Block 0 writes the tile offsets.
constexpr int kListed = 10240; // 20 KB; 512 ranks have about 4,000 on a 300k model at 640x480
static_assert(kMaxTiles * 32 == 65536, "a tile and a lane fit in 16 bits");

// Tiles by descending list length, in kLengths steps of the longest (one block): the forward
// starts the longest lists first. Within a step the order is open; it changes no result.
constexpr int kLengths = 64;

template <class S>
__device__ __forceinline__ void orderTiles(const int *lengths, int tiles, int *order)
{
    __shared__ int longest, count[kLengths];
    const int tid = threadIdx.x;
    if (tid == 0)
        longest = 0;
    if (tid < kLengths)
        count[tid] = 0;
    __syncthreads();
    int most = 0;
    for (int d = tid; d < tiles; d += S::THREADS)
        most = max(most, lengths[d]);
    most = __reduce_max_sync(0xffffffffu, most);
    if ((tid & 31) == 0)
        atomicMax(&longest, most);
    __syncthreads();
    const float scale = float(kLengths) / (float(longest) + 1.0f);
    auto step = [&](int d) { return kLengths - 1 - min(kLengths - 1, int(float(lengths[d]) * scale)); };
    for (int d = tid; d < tiles; d += S::THREADS)
        atomicAdd(&count[step(d)], 1);
    __syncthreads();
    if (tid == 0) {
        int run = 0;
        for (int k = 0; k < kLengths; ++k) {
            const int c = count[k];
            count[k] = run;
            run += c;
        }
    }
    __syncthreads();
    for (int d = tid; d < tiles; d += S::THREADS)
        order[atomicAdd(&count[step(d)], 1)] = d;
}

template <class S, bool kCull>
__global__ void __launch_bounds__(S::THREADS, S::THREADS == 128 ? 5 : kCull ? 2 : 3)
    tileScatterKernel(TileBins b, const int *hist, const int *tileTotals, const int *chunkFirst, const BinCounts *bc)
{
    pdlEntry();
    constexpr int kRankWarps = S::WARPS;
    extern __shared__ int dyn[];
    const int tiles = b.tiles, stride = (tiles + 1) / 2 * 2;
    int *base = dyn;                                                      // per tile: the chunk's first position
    uint16_t *offset = reinterpret_cast<uint16_t *>(dyn + stride);        // per warp and tile: the warp's next, from base
    __shared__ int warpSums[kRankWarps], scanSums[kRankWarps];
    __shared__ uint16_t listed[kListed];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int chunk = int(blockIdx.x) - (b.tileOrder ? 1 : 0); // the first block orders the tiles
    if (chunk < 0) {
        orderTiles<S>(tileTotals, tiles, b.tileOrder);
        return;
    }
    if (bc->effTotal <= 0) { // nothing listed, or an overflow
        if (chunk == 0)
            for (int d = tid; d <= tiles; d += S::THREADS)
                b.tileOffsets[d] = 0;
        // A backward takes its loop bounds from the first emissions, of unseen Gaussians too.
        if (b.offsById && rankOf<S>(chunk, b.n) < b.n)
            b.offsById[b.sortedIds[rankOf<S>(chunk, b.n)]] = 0;
        return;
    }
    const Listed l = loadListed(b.sortedIds, b.tileCount, b.rect, b.rowTab, kCull, rankOf<S>(chunk, b.n), b.n);
    for (int k = tid; k < kRankWarps * stride / 2; k += S::THREADS)
        reinterpret_cast<uint32_t *>(offset)[k] = 0;
    auto warpScan = [&](int v) {
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int y = __shfl_up_sync(0xffffffffu, v, o);
            if (lane >= o)
                v += y;
        }
        return v;
    };
    const int incl = warpScan(l.count), o = incl - l.count; // the rank's first intersection in its warp
    if (lane == 31)
        warpSums[warp] = incl;
    // The tile lists' starts: every thread scans consecutive tiles.
    const int per = (tiles + S::THREADS - 1) / S::THREADS;
    int own = 0;
    for (int k = 0; k < per; ++k)
        own += tid * per + k < tiles ? tileTotals[tid * per + k] : 0;
    const int scan = warpScan(own);
    if (lane == 31)
        scanSums[warp] = scan;
    __syncthreads();
    int start = scan - own, l0 = 0, all = 0; // l0: the warp's first intersection in the chunk
#pragma unroll
    for (int w = 0; w < kRankWarps; ++w) {
        start += w < warp ? scanSums[w] : 0;
        l0 += w < warp ? warpSums[w] : 0;
        all += warpSums[w];
    }
    const int e0 = chunkFirst[chunk];
    for (int k = 0; k < per; ++k) {
        const int d = tid * per + k;
        if (d >= tiles)
            break;
        base[d] = start + hist[size_t(chunk) * tiles + d];
        if (chunk == 0)
            b.tileOffsets[d] = start;
        start += tileTotals[d];
        if (chunk == 0 && d == tiles - 1)
            b.tileOffsets[tiles] = start;
    }
    if (b.offsById && rankOf<S>(chunk, b.n) < b.n)
        b.offsById[l.gid] = e0 + l0 + o;
    uint16_t *mine = offset + warp * stride;
    const int items = __shfl_sync(0xffffffffu, incl, 31);
    const uint32_t below = (1u << lane) - 1u;
    const int first = l0 + o; // the rank's first intersection in the chunk
    const bool search = !kCull && all > kListed;
    const int window = search ? all : kListed;
    for (int from = 0; from < all; from += window) {
        const int to = from + window;
        if (from > 0)
            __syncthreads(); // the warps are done with the last ones listed
        if (from == 0 || (first < to && first + l.count > from)) {
            int at = first - from;
            eachTile(l, kCull ? b.cullRec : nullptr, b.tileSize, b.tilesX, [&](int tile) {
                // (Two tiles share a word; a warp's ranks add at most 32 to each.)
                if (from == 0)
                    atomicAdd(reinterpret_cast<uint32_t *>(mine) + (tile >> 1), 1u << (16 * (tile & 1)));
                if (at >= 0 && at < kListed)
                    listed[at] = uint16_t(tile << 5 | lane);
                ++at;
            });
        }
        __syncthreads();
        if (from == 0) {
            for (int d = tid; d < tiles; d += S::THREADS) {
                int run = 0; // at most S::CHUNK
#pragma unroll
                for (int w = 0; w < kRankWarps; ++w) {
                    const int c = offset[w * stride + d];
                    offset[w * stride + d] = uint16_t(run);
                    run += c;
                }
            }
            __syncthreads();
        }
        const int end = min(l0 + items, to);
        for (int i0 = max(l0, from); i0 < end; i0 += 32) {
            const int i = i0 + lane;
            int gid, tile = kMaxTiles;
            if (!search) {
                const int v = i < end ? listed[i - from] : 0;
                gid = __shfl_sync(0xffffffffu, l.gid, v & 31);
                if (i < end)
                    tile = v >> 5;
            } else {
                int owner = 0; // the last lane whose first intersection is not above i (empty ranks share the next one's)
#pragma unroll
                for (int step = 16; step > 0; step >>= 1)
                    if (__shfl_sync(0xffffffffu, first, owner + step) <= i)
                        owner += step;
                const int k = i - __shfl_sync(0xffffffffu, first, owner);
                gid = __shfl_sync(0xffffffffu, l.gid, owner);
                const int x = __shfl_sync(0xffffffffu, l.q.x, owner), y = __shfl_sync(0xffffffffu, l.q.y, owner);
                const int wide = __shfl_sync(0xffffffffu, l.q.z, owner) - x;
                if (i < end)
                    tile = (y + k / wide) * b.tilesX + x + k % wide;
            }
            const uint32_t peers = __match_any_sync(0xffffffffu, tile);
            int seen = 0;
            if (i < end) {
                seen = mine[tile];
                const int pos = base[tile] + seen + __popc(peers & below);
                b.entries[pos] = gid;
                if (b.listPos)
                    b.listPos[e0 + i] = make_int2(pos, tile);
            }
            __syncwarp();
            if (i < end && lane == __ffs(peers) - 1)
                mine[tile] = uint16_t(seen + __popc(peers));
            __syncwarp();
        }
    }
}

// One warp per 32 consecutive depth ranks (grid-stride): the warp writes its ranks' intersections in
// order, 32 at a time. Each lane finds the rank of its intersection as the last of the warp's 32 start
// offsets not above it (a binary search over lanes with shuffles; empty ranks share their start with
// the next rank, so the search lands on the rank that owns the slot), then its tile in that rank's
// rectangle (row-major, as the reference's ty/tx loops).
__global__ void __launch_bounds__(256) emitKernel(const uint32_t *sortedIds, const int *offs, const int4 *rect, int n,
                                                  const BinCounts *c, int tilesX, const SplatRec *cullRec, int tileSize,
                                                  const uint32_t *rowTab, uint32_t *keys, int *emitGid)
{
    pdlEntry();
    const int total = c->effTotal;
    if (total <= 0)
        return;
    const int lane = threadIdx.x & 31;
    const int warps = int((gridDim.x * blockDim.x) >> 5);
    for (int w = int((blockIdx.x * blockDim.x + threadIdx.x) >> 5); w * 32 < n; w += warps) {
        const int r = w * 32 + lane;
        const bool valid = r < n;
        const int o = valid ? offs[r] : INT_MAX;
        int g = 0;
        int4 q = make_int4(0, 0, 1, 1);
        if (valid) {
            g = int(sortedIds[r]);
            q = rect[g];
        }
        const int first = offs[w * 32], last = min(offs[min(w * 32 + 32, n)], total);
        for (int e0 = first; e0 < last; e0 += 32) {
            const int e = e0 + lane;
            int l = 0;
#pragma unroll
            for (int step = 16; step > 0; step >>= 1) {
                const int oc = __shfl_sync(0xffffffffu, o, l + step);
                if (oc <= e)
                    l += step;
            }
            const int ol = __shfl_sync(0xffffffffu, o, l);
            const int gl = __shfl_sync(0xffffffffu, g, l);
            const int qx = __shfl_sync(0xffffffffu, q.x, l), qy = __shfl_sync(0xffffffffu, q.y, l);
            const int qz = __shfl_sync(0xffffffffu, q.z, l), qw = __shfl_sync(0xffffffffu, q.w, l);
            if (e < last) {
                const int2 t = listedTile(cullRec, rowTab, tileSize, gl, make_int4(qx, qy, qz, qw), e - ol);
                keys[e] = uint32_t(t.y * tilesX + t.x);
                emitGid[e] = gl;
            }
        }
    }
}

__global__ void finalizeKernel(const uint32_t *sortedKeys, const uint32_t *sortedEmit, const int *emitGid,
                               const BinCounts *c, int *entries, int2 *listPos)
{
    pdlEntry();
    const int total = c->effTotal;
    for (int s = blockIdx.x * blockDim.x + threadIdx.x; s < total; s += gridDim.x * blockDim.x) {
        const uint32_t e = sortedEmit[s];
        entries[s] = emitGid[e];
        if (listPos)
            listPos[e] = make_int2(s, int(sortedKeys[s]));
    }
}

__global__ void tileOffsetsKernel(const uint32_t *sortedKeys, const BinCounts *c, int tiles, int *tileOffsets)
{
    pdlEntry();
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t > tiles)
        return;
    const int total = c->effTotal;
    int lo = 0, hi = total; // first s with key >= t
    while (lo < hi) {
        const int mid = (lo + hi) >> 1;
        if (int(sortedKeys[mid]) < t)
            lo = mid + 1;
        else
            hi = mid;
    }
    tileOffsets[t] = (t == tiles) ? total : lo;
}

inline int grid(long long n, int t) { return int((n + t - 1) / t); }

} // namespace

int radixBlocks(int nMax) { return std::max(1, std::min(kMaxBlocks, (nMax + kTile - 1) / kTile)); }

size_t radixHistEntries(int nMax) { return size_t(1 << 8) * size_t(radixBlocks(nMax)); }

int radixDigits() { return kMaxTiles; }

bool binsByTile(int tiles) { return tiles <= kMaxTiles; }

int radixSortPairs(uint32_t *keysA, uint32_t *keysB, uint32_t *valsA, uint32_t *valsB, const int *nDev, int nMax,
                   int bits, int *hist, int *rowTotals, uint32_t **keysOut, uint32_t **valsOut, cudaStream_t s)
{
    uint32_t *kin = keysA, *kout = keysB, *vout = valsB;
    const uint32_t *vin = nullptr;
    const int G = radixBlocks(nMax);
    int passes = 0;
    for (int shift = 0; shift < bits; shift += 8, ++passes) {
        { launchPdl(radixHistKernel<8>, G, kThreads, 0, s, kin, nDev, shift, hist, G); countLaunch(); }
        { launchPdl(radixRowScanKernel, 1 << 8, kThreads, 0, s, hist, G, rowTotals); countLaunch(); }
        { launchPdl(radixScatterKernel<8>, G, kThreads, 0, s, kin, vin, kout, vout, nDev, shift, hist, rowTotals, G); countLaunch(); }
        uint32_t *nk = kin;
        kin = kout;
        kout = nk;
        vin = vout;
        vout = (vout == valsB) ? valsA : valsB;
    }
    *keysOut = kin;
    *valsOut = const_cast<uint32_t *>(vin);
    return passes;
}

// Items per depth chunk: whole tiles, at most kDepthChunks chunks.
static int depthChunk(int n) { return kDepthTile * std::max(1, (n + kDepthTile * kDepthChunks - 1) / (kDepthTile * kDepthChunks)); }

void radixSortDepth(const uint32_t *keys, uint2 *pairsA, uint2 *pairsB, uint32_t *sortedIds, int n, int *hist,
                    cudaStream_t s)
{
    if (n <= 0)
        return;
    if (n <= kSmallSort) {
        constexpr size_t shared = kSmallSort * sizeof(uint2) + size_t(kDepthWarps) * kDigits * sizeof(uint16_t);
        static PerDevice allowed;
        allowShared(depthSortSmallKernel, shared + 8192, shared, allowed); // with the static arrays
        { launchPdl(depthSortSmallKernel, 1, kDepthThreads, shared, s, keys, n, sortedIds); countLaunch(); }
        return;
    }
    const int chunk = depthChunk(n), G = (n + chunk - 1) / chunk;
    const uint2 *pin = nullptr;
    uint2 *bufs[2] = {pairsA, pairsB};
    for (int pass = 0; pass < 4; ++pass) {
        const int shift = 8 * pass;
        const PairIO io{pin, pass < 3 ? bufs[pass & 1] : nullptr, pass < 3 ? nullptr : sortedIds};
        { launchPdl(depthHistKernel, G, kDepthThreads, 0, s, keys, pin, n, shift, chunk, hist); countLaunch(); }
        { launchPdl(depthScatterKernel, G, kDepthThreads, 0, s, keys, n, shift, chunk, hist, io); countLaunch(); }
        pin = io.out;
    }
}

// For up to n Gaussians (few of them can be cut into more chunks than many).
size_t binChunkEntries(int n) { return size_t(std::max(rankChunks<ManyRanks>(n), rankChunks<FewRanks>(std::min(n, kFewGaussians)))); }

size_t binHistEntries(int n, int tiles)
{
    const size_t depth = size_t(kDepthChunks) * kDigits;
    return binsByTile(tiles) ? std::max(depth, binChunkEntries(n) * size_t(std::max(tiles, 1))) : depth;
}

template <class S, bool kCull>
static void launchBins(const TileBins &b, int *hist, int *tileTotals, int *chunkTotals, const ScanCapacity &cap, cudaStream_t s)
{
    const int G = rankChunks<S>(b.n), stride = (b.tiles + 1) / 2 * 2;
    constexpr size_t perTile = sizeof(int) + S::WARPS * sizeof(uint16_t); // 36 or 12 bytes
    static PerDevice allowed;
    allowShared(tileScatterKernel<S, kCull>, stride * perTile + 24 * 1024, size_t(kMaxTiles) * perTile, allowed); // with the static arrays
    { launchPdl(tileCountKernel<S>, G, S::THREADS, b.tiles * sizeof(int), s, b, hist, chunkTotals); countLaunch(); }
    { launchPdl(tileScanKernel, (b.tiles + 31) / 32 + 1, kScanThreads, 0, s, hist, G, b.tiles, tileTotals, chunkTotals, cap); countLaunch(); }
    { launchPdl(tileScatterKernel<S, kCull>, G + (b.tileOrder ? 1 : 0), S::THREADS, stride * perTile, s, b, hist, tileTotals, chunkTotals, cap.counts); countLaunch(); }
}

void binByTile(const TileBins &b, int *hist, int *tileTotals, int *chunkTotals, const ScanCapacity &cap, cudaStream_t s)
{
    const bool few = b.alone && b.n <= kFewGaussians, cull = b.cullRec != nullptr;
    const auto launch = few ? (cull ? launchBins<FewRanks, true> : launchBins<FewRanks, false>)
                            : (cull ? launchBins<ManyRanks, true> : launchBins<ManyRanks, false>);
    launch(b, hist, tileTotals, chunkTotals, cap, s);
}

size_t scanPartialEntries(int n) { return size_t((n + kScanTile - 1) / kScanTile) + 1; }

static void scanLaunches(const int *in, const uint32_t *perm, int *out, int *outById, int n, int *partial,
                         const ScanCapacity &cap, cudaStream_t s)
{
    const int B = (n + kScanTile - 1) / kScanTile;
    { launchPdl(scanReduceKernel, B, kThreads, 0, s, in, perm, n, partial); countLaunch(); }
    { launchPdl(scanPartialKernel, 1, kThreads, 0, s, partial, B); countLaunch(); }
    { launchPdl(scanDownsweepKernel, B, kThreads, 0, s, in, perm, out, outById, n, partial, B, cap); countLaunch(); }
}

void exclusiveScan(const int *in, int *out, int n, int *partial, cudaStream_t s)
{
    if (n <= 0) {
        cudaMemsetAsync(out, 0, sizeof(int), s);
        return;
    }
    scanLaunches(in, nullptr, out, nullptr, n, partial, ScanCapacity{0, nullptr, 0, nullptr}, s);
}

void exclusiveScanChecked(const int *in, const uint32_t *perm, int *out, int *outById, int n, int *partial,
                          const ScanCapacity &cap, cudaStream_t s)
{
    if (n <= 0) {
        cudaMemsetAsync(out, 0, sizeof(int), s);
        launchCapacityCheck(out, cap.capacity, cap.counts, cap.iteration, s, cap.desc);
        return;
    }
    scanLaunches(in, perm, out, outById, n, partial, cap, s);
}

size_t cullRowEntries(size_t n) { return n * kCullRows; }


void launchCapacityCheck(const int *total, int capacity, BinCounts *c, int iteration, cudaStream_t s,
                         const StepDesc *desc)
{
    { launchPdl(capacityKernel, 1, 1, 0, s, total, capacity, c, iteration, desc); countLaunch(); }
}

void launchEmit(const uint32_t *sortedIds, const int *offs, const int4 *rect, int n, const BinCounts *c, int capacity,
                int tilesX, const SplatRec *cullRec, int tileSize, const uint32_t *rowTab, uint32_t *keys, int *emitGid,
                cudaStream_t s)
{
    if (n > 0 && capacity > 0)
        { launchPdl(emitKernel, std::min(grid((long long)(n + 31) / 32 * 32, 256), 148 * 16), 256, 0, s, sortedIds, offs, rect, n, c, tilesX, cullRec, tileSize, rowTab, keys, emitGid); countLaunch(); }
}

void launchFinalizeBins(const uint32_t *sortedKeys, const uint32_t *sortedEmit, const int *emitGid, const BinCounts *c,
                        int capacity, int tiles, int *entries, int2 *listPos, int *tileOffsets, cudaStream_t s)
{
    if (capacity > 0)
        { launchPdl(finalizeKernel, std::min(grid(capacity, 256), 148 * 16), 256, 0, s, sortedKeys, sortedEmit, emitGid, c, entries, listPos); countLaunch(); }
    { launchPdl(tileOffsetsKernel, grid(tiles + 1, 256), 256, 0, s, sortedKeys, c, tiles, tileOffsets); countLaunch(); }
}

} // namespace u3dg
