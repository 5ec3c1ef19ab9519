// Parallel primitives (see prims.cuh). Counts come from device memory; grids from capacities.

#include "cluster.cuh"
#include "prims.cuh"

#include <mutex>
#include <vector>

namespace avbdg {

namespace {

constexpr int kScanThreads = 256;
constexpr int kScanItems = 8;
constexpr int kScanTile = kScanThreads * kScanItems;
constexpr int kTopThreads = 1024;
// Small capacities (the stores of single worlds up to some thousand bodies) are scanned by a single block in
// one launch, without clusters up to its reach: the three-launch form's fixed cost dominates there.
constexpr int kSmallThreads = 1024;
constexpr int kSmallItems = 16;
constexpr int kSmallScanCap = kSmallThreads * kSmallItems;
// Larger ones, up to kClusterScanCap, by one cluster: its CTAs hold up to 131,072 values at a time and tell
// one another their sums. Microseconds here and by the other forms: 16,384 values 3.5 / 7.4 (one block), 30,000
// 3.8 / 7.0 (three launches), 65,537 5.0 / 7.2; 452,000, in four turns, 23.3 / 12.8.
constexpr int kBlockScanCap = 4096;
constexpr int kClusterScanCap = 1 << 17;
constexpr int kClusterItems = 8;

__device__ __forceinline__ int loadCount(const int *d_n, int capacity) {
    if (!d_n)
        return capacity;
    const int n = *d_n;
    return n < capacity ? n : capacity;
}

// Block-wide exclusive scan of one value per thread; returns the prefix, writes the total.
template <int THREADS>
__device__ __forceinline__ int blockExclusiveScan(int v, int *smemWarp, int &total) {
    const int lane = threadIdx.x & 31;
    const int warp = threadIdx.x >> 5;
    int x = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int y = __shfl_up_sync(0xffffffffu, x, o);
        if (lane >= o)
            x += y;
    }
    if (lane == 31)
        smemWarp[warp] = x;
    __syncthreads();
    if (warp == 0) {
        constexpr int W = THREADS / 32;
        int s = lane < W ? smemWarp[lane] : 0;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int y = __shfl_up_sync(0xffffffffu, s, o);
            if (lane >= o)
                s += y;
        }
        if (lane < W)
            smemWarp[lane] = s;
    }
    __syncthreads();
    const int warpPrefix = warp > 0 ? smemWarp[warp - 1] : 0;
    total = smemWarp[THREADS / 32 - 1];
    __syncthreads();
    return warpPrefix + x - v;
}

__global__ void scanReduceKernel(const int *in, int capacity, const int *d_n, int *blockSums) {
    pdlWait();
    pdlTrigger();
    __shared__ int warpSums[kScanThreads / 32];
    const int n = loadCount(d_n, capacity);
    const int base = blockIdx.x * kScanTile + threadIdx.x * kScanItems;
    int s = 0;
#pragma unroll
    for (int k = 0; k < kScanItems; k++) {
        const int i = base + k;
        if (i < n)
            s += in[i];
    }
    int total;
    blockExclusiveScan<kScanThreads>(s, warpSums, total);
    if (threadIdx.x == 0)
        blockSums[blockIdx.x] = total;
}

__global__ void scanTopKernel(int *blockSums, int numBlocks, int *d_total) {
    pdlWait();
    pdlTrigger();
    __shared__ int warpSums[kTopThreads / 32];
    const int per = (numBlocks + kTopThreads - 1) / kTopThreads;
    const int first = threadIdx.x * per;
    int s = 0;
    for (int k = 0; k < per; k++) {
        const int i = first + k;
        if (i < numBlocks)
            s += blockSums[i];
    }
    int total;
    int prefix = blockExclusiveScan<kTopThreads>(s, warpSums, total);
    for (int k = 0; k < per; k++) {
        const int i = first + k;
        if (i < numBlocks) {
            const int v = blockSums[i];
            blockSums[i] = prefix;
            prefix += v;
        }
    }
    if (threadIdx.x == 0 && d_total)
        *d_total = total;
}

// The whole scan in one block: each thread holds kSmallItems consecutive values (read before any
// write, so `in` may alias `out`), exactly the prefixes the three-launch form writes.
__global__ void __launch_bounds__(kSmallThreads) scanSmallKernel(const int *in, int *out, int capacity,
                                                                 const int *d_n, int *d_total) {
    pdlWait();
    pdlTrigger();
    __shared__ int warpSums[kSmallThreads / 32];
    const int n = loadCount(d_n, capacity);
    const int base = threadIdx.x * kSmallItems;
    int v[kSmallItems];
    int s = 0;
#pragma unroll
    for (int k = 0; k < kSmallItems; k++) {
        const int i = base + k;
        v[k] = i < n ? in[i] : 0;
        s += v[k];
    }
    int total;
    int prefix = blockExclusiveScan<kSmallThreads>(s, warpSums, total);
#pragma unroll
    for (int k = 0; k < kSmallItems; k++) {
        const int i = base + k;
        if (i < n)
            out[i] = prefix;
        prefix += v[k];
    }
    if (threadIdx.x == 0 && d_total)
        *d_total = total;
}

// The whole scan by one cluster (`in` may alias `out`: a value is read before any CTA's next barrier and
// written after it by the same thread).
__global__ void __launch_bounds__(kSmallThreads) scanClusterKernel(const int *in, int *out, int capacity, const int *d_n, int *d_total) {
    pdlWait();
    pdlTrigger();
    __shared__ int warpSums[kSmallThreads / 32], totals[2][kMaxTeam];
    const int n = loadCount(d_n, capacity), rank = clusterRank(), size = clusterSize(), lanes = size * kSmallThreads;
    clusterArrive(); // a CTA's shared memory is another's to write once it runs: waited for before the first turn's sums
    int run = 0, turn = 0;
    for (int first = 0, per; first < n; first += lanes * per, turn ^= 1) {
        per = min(kClusterItems, (n - first + lanes - 1) / lanes);
        const int base = first + (rank * kSmallThreads + static_cast<int>(threadIdx.x)) * per;
        int v[kClusterItems], s = 0;
#pragma unroll
        for (int k = 0; k < kClusterItems; k++) {
            v[k] = k < per && base + k < n ? in[base + k] : 0;
            s += v[k];
        }
        int total;
        int prefix = run + blockExclusiveScan<kSmallThreads>(s, warpSums, total);
        if (first == 0)
            clusterWait();
        if (static_cast<int>(threadIdx.x) < size)
            storeClusterInt(mapShared(sharedAddress(&totals[turn][rank]), threadIdx.x), total);
        clusterSync(size); // (a turn's sums are read before anyone writes those of the turn after the next)
        for (int k = 0; k < size; k++) {
            prefix += k < rank ? totals[turn][k] : 0;
            run += totals[turn][k];
        }
#pragma unroll
        for (int k = 0; k < kClusterItems; k++) {
            if (k < per && base + k < n)
                out[base + k] = prefix;
            prefix += v[k];
        }
    }
    if (n <= 0)
        clusterWait();
    if (rank == 0 && threadIdx.x == 0 && d_total)
        *d_total = run;
}

__global__ void scanDownKernel(const int *in, int *out, int capacity, const int *d_n, const int *blockSums) {
    pdlWait();
    pdlTrigger();
    __shared__ int warpSums[kScanThreads / 32];
    const int n = loadCount(d_n, capacity);
    const int base = blockIdx.x * kScanTile + threadIdx.x * kScanItems;
    int v[kScanItems];
    int s = 0;
#pragma unroll
    for (int k = 0; k < kScanItems; k++) {
        const int i = base + k;
        v[k] = i < n ? in[i] : 0;
        s += v[k];
    }
    int total;
    int prefix = blockExclusiveScan<kScanThreads>(s, warpSums, total) + blockSums[blockIdx.x];
#pragma unroll
    for (int k = 0; k < kScanItems; k++) {
        const int i = base + k;
        if (i < n)
            out[i] = prefix;
        prefix += v[k];
    }
}

// ---------------------------------------------------------------------------------------------
// Radix sort: 8-bit digits, tiles of 256 threads x 8 keys, stable ranking by warp votes.
//
// A pass counts each tile's digits, scans the counts along the tiles (a block a digit) and scatters.
// In the scatter a warp ranks its 256 consecutive keys without meeting the others; the tile is then
// put in digit order in shared memory, so neighbouring lanes write neighbouring keys, and every tile
// finds the digits' bases from their 256 totals itself. A million keys a pass, kernels alone: 24.6 us
// when each of eight rounds met three block barriers and scattered from registers, with the counts
// scanned as one array of 131,072; 15.4 us this way (16 MB through L2). A single tile (stores of up
// to 2048 bodies) needs neither count nor scan: one launch a pass.
// ---------------------------------------------------------------------------------------------

constexpr int kRadixThreads = 256;
constexpr int kRadixWarps = kRadixThreads / 32;
constexpr int kRadixRounds = 8;
constexpr int kRadixTile = kRadixThreads * kRadixRounds;
constexpr int kRadixBins = 256;

// A tile's counts, at hist[digit * numBlocks + tile].
__global__ void __launch_bounds__(kRadixThreads) radixHistKernel(const uint64_t *keys, int capacity, const int *d_n, int shift,
                                                                 uint32_t mask, int numBlocks, int *hist) {
    pdlWait();
    pdlTrigger();
    __shared__ int h[kRadixBins];
    h[threadIdx.x] = 0;
    __syncthreads();
    const int n = loadCount(d_n, capacity);
    const int base = blockIdx.x * kRadixTile + threadIdx.x;
    uint64_t key[kRadixRounds];
#pragma unroll
    for (int r = 0; r < kRadixRounds; r++)
        key[r] = base + r * kRadixThreads < n ? keys[base + r * kRadixThreads] : 0;
#pragma unroll
    for (int r = 0; r < kRadixRounds; r++)
        if (base + r * kRadixThreads < n)
            atomicAdd(&h[(key[r] >> shift) & mask], 1);
    __syncthreads();
    hist[threadIdx.x * numBlocks + blockIdx.x] = h[threadIdx.x];
}

// Block d: the exclusive prefix of digit d's counts along the tiles, in place, and their total.
__global__ void __launch_bounds__(kRadixThreads) radixScanKernel(int *hist, int numBlocks, int *totals) {
    pdlWait();
    pdlTrigger();
    __shared__ int warpSums[kRadixWarps];
    constexpr int kItems = 4;
    int *row = hist + static_cast<size_t>(blockIdx.x) * numBlocks;
    int run = 0;
    for (int first = 0; first < numBlocks; first += kRadixThreads * kItems) {
        const int base = first + threadIdx.x * kItems;
        int v[kItems], s = 0;
#pragma unroll
        for (int k = 0; k < kItems; k++) {
            v[k] = base + k < numBlocks ? row[base + k] : 0;
            s += v[k];
        }
        int total;
        int prefix = run + blockExclusiveScan<kRadixThreads>(s, warpSums, total);
#pragma unroll
        for (int k = 0; k < kItems; k++) {
            if (base + k < numBlocks)
                row[base + k] = prefix;
            prefix += v[k];
        }
        run += total;
    }
    if (threadIdx.x == 0)
        totals[blockIdx.x] = run;
}

__global__ void __launch_bounds__(kRadixThreads)
        radixScatterKernel(const uint64_t *keysIn, const uint32_t *valsIn, uint64_t *keysOut, uint32_t *valsOut, int capacity,
                           const int *d_n, int shift, uint32_t mask, int numBlocks, const int *hist, const int *totals) {
    pdlWait();
    pdlTrigger();
    __shared__ int warpCount[kRadixWarps][kRadixBins];
    __shared__ int place[kRadixBins]; // a digit's place in the output, less its place in the tile
    __shared__ int warpSums[kRadixWarps];
    __shared__ uint64_t tileKeys[kRadixTile];
    __shared__ uint32_t tileVals[kRadixTile];
    const int n = loadCount(d_n, capacity);
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int first = static_cast<int>(blockIdx.x) * kRadixTile, base = first + warp * (32 * kRadixRounds) + lane;
    uint64_t key[kRadixRounds];
    uint32_t val[kRadixRounds];
#pragma unroll
    for (int r = 0; r < kRadixRounds; r++) {
        const int i = base + 32 * r;
        key[r] = i < n ? keysIn[i] : 0;
        val[r] = i < n && valsIn ? valsIn[i] : 0u;
    }
    for (int b = lane; b < kRadixBins; b += 32)
        warpCount[warp][b] = 0;
    __syncwarp();
    // Each key's rank among the warp's earlier keys of its digit.
    int rank[kRadixRounds];
#pragma unroll
    for (int r = 0; r < kRadixRounds; r++) {
        const bool valid = base + 32 * r < n;
        const uint32_t d = static_cast<uint32_t>((key[r] >> shift) & mask);
        uint32_t peers = __ballot_sync(0xffffffffu, valid);
#pragma unroll
        for (int b = 0; b < 8; b++) { // (eight votes take less than one match of scattered digits)
            const uint32_t ones = __ballot_sync(0xffffffffu, (d >> b) & 1u);
            peers &= (d >> b) & 1u ? ones : ~ones;
        }
        const int below = __popc(peers & ((1u << lane) - 1u));
        rank[r] = valid ? warpCount[warp][d] + below : 0;
        __syncwarp();
        if (valid && below == 0)
            warpCount[warp][d] += __popc(peers);
        __syncwarp();
    }
    __syncthreads();
    // Thread b: digit b's warps in order, its place in the tile and in the output.
    {
        int mine = 0;
#pragma unroll
        for (int w = 0; w < kRadixWarps; w++) {
            const int c = warpCount[w][threadIdx.x];
            warpCount[w][threadIdx.x] = mine;
            mine += c;
        }
        int total;
        const int inTile = blockExclusiveScan<kRadixThreads>(mine, warpSums, total);
        int out = inTile;
        if (numBlocks > 1)
            out = blockExclusiveScan<kRadixThreads>(totals[threadIdx.x], warpSums, total) +
                  hist[threadIdx.x * numBlocks + blockIdx.x];
#pragma unroll
        for (int w = 0; w < kRadixWarps; w++)
            warpCount[w][threadIdx.x] += inTile;
        place[threadIdx.x] = out - inTile;
    }
    __syncthreads();
#pragma unroll
    for (int r = 0; r < kRadixRounds; r++)
        if (base + 32 * r < n) {
            const int at = warpCount[warp][(key[r] >> shift) & mask] + rank[r];
            tileKeys[at] = key[r];
            tileVals[at] = val[r];
        }
    __syncthreads();
    const int count = min(kRadixTile, n - first);
#pragma unroll
    for (int r = 0; r < kRadixRounds; r++) {
        const int i = r * kRadixThreads + threadIdx.x;
        if (i < count) {
            const uint64_t k = tileKeys[i];
            const int to = place[(k >> shift) & mask] + i;
            keysOut[to] = k;
            if (valsOut)
                valsOut[to] = tileVals[i];
        }
    }
}

// ---------------------------------------------------------------------------------------------
// The distinct keys of a sorted array: a key counts where it differs from the one before. Both passes
// read the keys (the second from L2) rather than keep a flag and a rank for each.
// ---------------------------------------------------------------------------------------------

__device__ __forceinline__ bool firstOfKey(const uint64_t *keys, int i, int n) { return i < n && (i == 0 || keys[i] != keys[i - 1]); }

__global__ void __launch_bounds__(kRadixThreads) uniqueCountKernel(const uint64_t *keys, int n, int *blockSums) {
    pdlWait();
    pdlTrigger();
    __shared__ int warpSums[kRadixWarps];
    const int base = blockIdx.x * kRadixTile + threadIdx.x;
    int mine = 0;
#pragma unroll
    for (int r = 0; r < kRadixRounds; r++)
        mine += firstOfKey(keys, base + r * kRadixThreads, n) ? 1 : 0;
    int total;
    blockExclusiveScan<kRadixThreads>(mine, warpSums, total);
    if (threadIdx.x == 0)
        blockSums[blockIdx.x] = total;
}

__global__ void __launch_bounds__(kRadixThreads) uniqueScatterKernel(const uint64_t *keys, int n, const int *blockSums, uint64_t *out) {
    pdlWait();
    pdlTrigger();
    __shared__ int counts[kRadixRounds * kRadixWarps];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, base = blockIdx.x * kRadixTile + threadIdx.x;
    unsigned hits[kRadixRounds];
#pragma unroll
    for (int r = 0; r < kRadixRounds; r++) {
        hits[r] = __ballot_sync(0xffffffffu, firstOfKey(keys, base + r * kRadixThreads, n));
        if (lane == 0)
            counts[r * kRadixWarps + warp] = __popc(hits[r]);
    }
    __syncthreads();
    if (warp == 0) { // two counts a lane
        static_assert(kRadixRounds * kRadixWarps == 64, "two counts a lane");
        const int a = counts[2 * lane], b = counts[2 * lane + 1];
        int upTo = a + b;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int y = __shfl_up_sync(0xffffffffu, upTo, o);
            if (lane >= o)
                upTo += y;
        }
        const int before = blockSums[blockIdx.x] + upTo - a - b;
        counts[2 * lane] = before;
        counts[2 * lane + 1] = before + a;
    }
    __syncthreads();
#pragma unroll
    for (int r = 0; r < kRadixRounds; r++)
        if ((hits[r] >> lane) & 1u)
            out[counts[r * kRadixWarps + warp] + __popc(hits[r] & ((1u << lane) - 1u))] = keys[base + r * kRadixThreads];
}

template <typename T>
__global__ void copyKernel(const T *src, T *dst, int capacity, const int *d_n) {
    pdlWait();
    pdlTrigger();
    const int n = loadCount(d_n, capacity);
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x)
        dst[i] = src[i];
}

// ---------------------------------------------------------------------------------------------
// Segmented sort
// ---------------------------------------------------------------------------------------------

constexpr int kSmallSeg = 32;
constexpr int kMidSegThreads = 256;
constexpr int kMidSegCap = 8192;
constexpr int kBigBlocks = 64;
constexpr int kBigTile = 2048;

template <typename T>
__global__ void segSmallKernel(T *data, const int *start, int segCapacity, const int *d_segments, int *longList,
                               int *longCount) {
    pdlWait();
    pdlTrigger();
    const int ns = loadCount(d_segments, segCapacity);
    for (int s = blockIdx.x * blockDim.x + threadIdx.x; s < ns; s += gridDim.x * blockDim.x) {
        const int b = start[s], e = start[s + 1];
        const int len = e - b;
        if (len <= 1)
            continue;
        if (len > kSmallSeg) {
            longList[atomicAdd(longCount, 1)] = s;
            continue;
        }
        for (int i = b + 1; i < e; i++) {
            const T x = data[i];
            int j = i - 1;
            while (j >= b && data[j] > x) {
                data[j + 1] = data[j];
                j--;
            }
            data[j + 1] = x;
        }
    }
}

template <typename T>
__global__ void segMidKernel(T *data, const int *start, const int *longList, const int *longCount) {
    pdlWait();
    pdlTrigger();
    extern __shared__ unsigned char smemRaw[];
    T *buf = reinterpret_cast<T *>(smemRaw);
    const int nl = *longCount;
    for (int k = blockIdx.x; k < nl; k += gridDim.x) {
        const int s = longList[k];
        const int b = start[s], len = start[s + 1] - start[s];
        if (len > kMidSegCap)
            continue;
        for (int i = threadIdx.x; i < len; i += blockDim.x)
            buf[i] = data[b + i];
        __syncthreads();
        for (int i = threadIdx.x; i < len; i += blockDim.x) {
            const T x = buf[i];
            int rank = 0;
            for (int j = 0; j < len; j++)
                rank += buf[j] < x ? 1 : 0;
            data[b + rank] = x;
        }
        __syncthreads();
    }
}

template <typename T>
__global__ void segBigCopyKernel(const T *data, T *tmp, const int *start, const int *longList, const int *longCount) {
    pdlWait();
    pdlTrigger();
    const int nl = *longCount;
    for (int k = 0; k < nl; k++) {
        const int s = longList[k];
        const int b = start[s], len = start[s + 1] - start[s];
        if (len <= kMidSegCap)
            continue;
        for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < len; i += gridDim.x * blockDim.x)
            tmp[b + i] = data[b + i];
    }
}

template <typename T>
__global__ void segBigRankKernel(T *data, const T *tmp, const int *start, const int *longList, const int *longCount) {
    pdlWait();
    pdlTrigger();
    __shared__ T tile[kBigTile];
    const int nl = *longCount;
    for (int k = 0; k < nl; k++) {
        const int s = longList[k];
        const int b = start[s], len = start[s + 1] - start[s];
        if (len <= kMidSegCap)
            continue;
        for (int i0 = blockIdx.x * blockDim.x; i0 < len; i0 += gridDim.x * blockDim.x) {
            const int i = i0 + threadIdx.x;
            const T x = i < len ? tmp[b + i] : T(0);
            int rank = 0;
            for (int t0 = 0; t0 < len; t0 += kBigTile) {
                __syncthreads();
                for (int j = threadIdx.x; j < kBigTile && t0 + j < len; j += blockDim.x)
                    tile[j] = tmp[b + t0 + j];
                __syncthreads();
                const int tl = len - t0 < kBigTile ? len - t0 : kBigTile;
                if (i < len)
                    for (int j = 0; j < tl; j++)
                        rank += tile[j] < x ? 1 : 0;
            }
            if (i < len)
                data[b + rank] = x;
        }
    }
}

} // namespace

size_t scanScratchBytes(int capacity) {
    const int blocks = divUp(capacity > 0 ? capacity : 1, kScanTile);
    return static_cast<size_t>(blocks) * sizeof(int) + 256;
}

size_t radixScratchBytes(int capacity) {
    const int blocks = divUp(capacity > 0 ? capacity : 1, kRadixTile);
    return (static_cast<size_t>(blocks) + 1) * kRadixBins * sizeof(int);
}

size_t uniqueScratchBytes(int count) { return static_cast<size_t>(divUp(count > 0 ? count : 1, kRadixTile)) * sizeof(int); }

int smCount() {
    static PerDevice counts;
    const int device = currentDevice();
    return counts.get(device, [device] {
        int sms = 0;
        cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device);
        return sms > 0 ? sms : 1;
    });
}

static int scanTeam() {
    static PerDevice teams;
    return teams.get(currentDevice(), [] { return allowTeam(reinterpret_cast<const void *>(scanClusterKernel), kSmallThreads, 0); });
}

void scanExclusive(const int *in, int *out, int capacity, const int *d_n, int *d_total, void *scratch,
                   cudaStream_t stream) {
    const int largest = capacity > kBlockScanCap && capacity <= kClusterScanCap ? scanTeam() : 1;
    if (largest > 1) {
        int team = 2;
        while (team < largest && team * 2 * kSmallThreads < capacity)
            team *= 2;
        const TeamLaunch l(team, 1, kSmallThreads, 0, stream);
        ++launchCount();
        cudaLaunchKernelEx(&l.cfg, scanClusterKernel, in, out, capacity, d_n, d_total);
        return;
    }
    if (capacity <= kSmallScanCap) {
        ++launchCount(); launchK(scanSmallKernel, 1, kSmallThreads, 0, stream, in, out, capacity, d_n, d_total);
        return;
    }
    const int blocks = divUp(capacity > 0 ? capacity : 1, kScanTile);
    int *blockSums = static_cast<int *>(scratch);
    ++launchCount(); launchK(scanReduceKernel, blocks, kScanThreads, 0, stream, in, capacity, d_n, blockSums);
    ++launchCount(); launchK(scanTopKernel, 1, kTopThreads, 0, stream, blockSums, blocks, d_total);
    ++launchCount(); launchK(scanDownKernel, blocks, kScanThreads, 0, stream, in, out, capacity, d_n, blockSums);
}

void radixSortPairs(uint64_t *keys, uint32_t *values, uint64_t *keysAlt, uint32_t *valuesAlt, int capacity,
                    const int *d_n, int beginBit, int endBit, void *scratch, cudaStream_t stream) {
    const int blocks = divUp(capacity > 0 ? capacity : 1, kRadixTile);
    int *totals = static_cast<int *>(scratch), *hist = totals + kRadixBins;
    uint64_t *kin = keys, *kout = keysAlt;
    uint32_t *vin = values, *vout = valuesAlt;
    int passes = 0;
    for (int bit = beginBit; bit < endBit; bit += 8) {
        const int bits = endBit - bit < 8 ? endBit - bit : 8;
        const uint32_t mask = (1u << bits) - 1u;
        if (blocks > 1) {
            ++launchCount();
            launchK(radixHistKernel, blocks, kRadixThreads, 0, stream, kin, capacity, d_n, bit, mask, blocks, hist);
            ++launchCount();
            launchK(radixScanKernel, kRadixBins, kRadixThreads, 0, stream, hist, blocks, totals);
        }
        ++launchCount();
        launchK(radixScatterKernel, blocks, kRadixThreads, 0, stream, kin, vin, kout, vout, capacity, d_n, bit, mask, blocks, hist,
                totals);
        uint64_t *tk = kin;
        kin = kout;
        kout = tk;
        uint32_t *tv = vin;
        vin = vout;
        vout = tv;
        passes++;
    }
    if (passes & 1) {
        const int grid = divUp(capacity > 0 ? capacity : 1, 256) < 1184 ? divUp(capacity > 0 ? capacity : 1, 256) : 1184;
        ++launchCount(); launchK(copyKernel<uint64_t>, grid, 256, 0, stream, kin, keys, capacity, d_n);
        if (values) {
            ++launchCount();
            launchK(copyKernel<uint32_t>, grid, 256, 0, stream, vin, values, capacity, d_n);
        }
    }
}

void uniqueSorted(const uint64_t *keys, int n, uint64_t *out, int *d_count, void *scratch, cudaStream_t stream) {
    const int blocks = divUp(n, kRadixTile);
    int *blockSums = static_cast<int *>(scratch);
    ++launchCount(); launchK(uniqueCountKernel, blocks, kRadixThreads, 0, stream, keys, n, blockSums);
    ++launchCount(); launchK(scanTopKernel, 1, kTopThreads, 0, stream, blockSums, blocks, d_count);
    ++launchCount(); launchK(uniqueScatterKernel, blocks, kRadixThreads, 0, stream, keys, n, blockSums, out);
}

template <typename T>
static void segmentedSort(T *data, const int *start, int segCapacity, const int *d_segments, int *longList,
                          int *longCount, T *tmp, cudaStream_t stream) {
    const int grid = divUp(segCapacity > 0 ? segCapacity : 1, 256);
    ++launchCount(); launchK(segSmallKernel<T>, grid < 4096 ? grid : 4096, 256, 0, stream, data, start, segCapacity, d_segments, longList,
                                                                   longCount);
    const size_t smem = kMidSegCap * sizeof(T);
    ++launchCount(); launchK(segMidKernel<T>, 152, kMidSegThreads, smem, stream, data, start, longList, longCount);
    if (tmp) {
        ++launchCount(); launchK(segBigCopyKernel<T>, kBigBlocks, 256, 0, stream, data, tmp, start, longList, longCount);
        ++launchCount(); launchK(segBigRankKernel<T>, kBigBlocks, 256, 0, stream, data, tmp, start, longList, longCount);
    }
}

void preparePrimitives() {
    cudaFuncSetAttribute(segMidKernel<uint32_t>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                         static_cast<int>(kMidSegCap * sizeof(uint32_t)));
    cudaFuncSetAttribute(segMidKernel<uint64_t>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                         static_cast<int>(kMidSegCap * sizeof(uint64_t)));
    scanTeam();
}

int residentGrid(const void *kernel, int block, size_t smem, int want) {
    struct Entry {
        int device;
        const void *kernel;
        int block;
        size_t smem;
        int blocks;
    };
    static std::mutex mu;
    static std::vector<Entry> cache;
    int dev = 0;
    cudaGetDevice(&dev);
    int blocks = 0;
    {
        std::lock_guard<std::mutex> lock(mu);
        for (const Entry &e : cache)
            if (e.device == dev && e.kernel == kernel && e.block == block && e.smem == smem)
                blocks = e.blocks;
        if (blocks == 0) {
            int sms = 0, perSm = 0;
            cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
            cudaOccupancyMaxActiveBlocksPerMultiprocessor(&perSm, kernel, block, smem);
            blocks = (sms > 0 ? sms : 1) * (perSm > 0 ? perSm : 1);
            cache.push_back(Entry{dev, kernel, block, smem, blocks});
        }
    }
    return want < 1 ? 1 : (want < blocks ? want : blocks);
}

void segmentedSortU32(uint32_t *data, uint32_t *tmp, const int *start, int segCapacity, const int *d_segments,
                      int *longList, int *longCount, cudaStream_t stream) {
    segmentedSort<uint32_t>(data, start, segCapacity, d_segments, longList, longCount, tmp, stream);
}

void segmentedSortU64(uint64_t *data, uint64_t *tmp, const int *start, int segCapacity, const int *d_segments,
                      int *longList, int *longCount, cudaStream_t stream) {
    segmentedSort<uint64_t>(data, start, segCapacity, d_segments, longList, longCount, tmp, stream);
}

} // namespace avbdg
