// Update set, colouring and the substep (godot-avbd src/avbd/solver_solve.cpp,
// src/avbd/solver_step.cpp:79-105,195-316, src/avbd/manifold.cpp:465-671, src/avbd/joint.cpp,
// src/avbd/types.hpp:147-201, src/avbd/maths.h:156-343).
//
// Primal, block-Jacobi ("overflow") bodies: the reference computes each round's per-contact force
// cache once per manifold (preCompute), then every overflow body stamps its incident manifolds
// from that cache in adjacency order and solves its 6x6 block against the round's pose snapshot.
// Here one kernel per manifold computes the dual update AND, from the same poses, the next
// round's per-side block contributions ("stamps"); one kernel per body then sums its stamps in
// adjacency order, solves the LDL^T in registers and applies the relaxed delta. Both steps keep
// the reference's operation order, so the result is bit-identical.
//
// Coloured (Gauss-Seidel) bodies recompute their manifold terms from the current poses at every
// touch; the reference's "first touch uses the dual's cache" rule yields the same floats.

#include "gridsync.cuh"
#include "kernels.cuh"
#include "prims.cuh"
#include "project.cuh"
#include "solve.cuh"

namespace avbdg {

namespace {

constexpr int kThreads = 256;
constexpr int kSolveThreads = 128;
constexpr int kQueueThreads = 128; // items per round-queue tile

__device__ __forceinline__ int divUpDev(int a, int b) { return (a + b - 1) / b; }

__global__ void stampsKernel(Dev d, StepParams p, int mixedOnly) {
    pdlWait();
    pdlTrigger();
    const int n = d.ctr[C_LIVE];
    for (int m = blockIdx.x * blockDim.x + threadIdx.x; m < n; m += gridDim.x * blockDim.x)
        stampsAt(d, p, mixedOnly, m);
}

template <bool STAMPS, bool ARM>
__global__ void __launch_bounds__(512) dualKernel(Dev d, StepParams p, real decay) { pdlWait(); pdlTrigger(); // 512: largest tuned block
    const int live = d.ctr[C_LIVE];
    for (int m = blockIdx.x * blockDim.x + threadIdx.x; m < live; m += gridDim.x * blockDim.x)
        dualAt<STAMPS, ARM>(d, p, decay, m);
}

__global__ void forceDualKernel(Dev d, StepParams p) {
    pdlWait();
    pdlTrigger();
    const int f = blockIdx.x * blockDim.x + threadIdx.x;
    if (f < d.ctr[C_FORCES])
        forceDualAt(d, p, f);
}

// One round's colour passes in one cooperative launch: colours in order, each a grid-stride loop
// over its list, a grid barrier after each but the last non-empty one. Every block reads the same
// counts (nothing writes them during the sweep), so all blocks skip the same empty colours.
__global__ void __launch_bounds__(kSolveThreads) colourSweepKernel(Dev d, StepParams p, int armsFromDual) {
    pdlWait();
    pdlTrigger();
    int last = -1;
    for (int c = 0; c < kMaxColours; c++)
        if (d.colourCount[c] > 0)
            last = c;
    const int stride = gridDim.x * blockDim.x;
    for (int c = 0; c <= last; c++) {
        const int cnt = d.colourCount[c];
        if (cnt == 0)
            continue;
        for (int k = blockIdx.x * blockDim.x + threadIdx.x; k < cnt; k += stride)
            colourBodyAt(d, p, d.colourList[c * d.NB + k], armsFromDual);
        if (c < last && !gridSync(d))
            return;
    }
}

#ifdef AVBDG_FP64
#define AVBDG_SOLVE_BOUNDS __launch_bounds__(kSolveThreads)
#else
#define AVBDG_SOLVE_BOUNDS __launch_bounds__(kSolveThreads, 8) // 64 registers: 8 blocks an SM
#endif
// Overflow bodies are walked in slot order (coalesced body loads); the overflow colour has no list.
template <bool FORCES, bool QUOTIENTS>
__global__ void AVBDG_SOLVE_BOUNDS
        overflowSolveKernel(const __grid_constant__ Dev d, const __grid_constant__ StepParams p, int inPlace) {
    pdlWait();
    pdlTrigger();
    const int g = blockIdx.x * blockDim.x + threadIdx.x;
    if (g < d.ctr[C_BODIES])
        solveAt<FORCES, true, QUOTIENTS>(d, p, g, inPlace);
}

// ---- the round loop as one persistent launch over a tile queue ----
//
// In a store without forces or coloured bodies, round r's body solve in world w needs only the
// stamps round r-1's dual wrote for w, and round r's dual needs only that round's solves in w;
// worlds never read each other. One launch runs all the rounds: tiles (round, phase, world, chunk)
// are handed out in that order by one counter, a tile waits (bounded by waitLimit) until its world
// has completed the previous phase, runs one item per thread and counts itself done; the last
// chunk of a phase advances the world's stage. Every tile a tile waits for was handed out earlier
// to a block that is running (cooperative launch), so the waits end. Worlds move through their
// rounds independently instead of every world waiting at each kernel boundary. The per-item work
// is the separate kernels' (solveAt, dualAt, with coherent loads), so the results are the same.
__device__ __forceinline__ int worldOfTile(const int *pre, int nWorlds, int t) {
    int lo = 0, hi = nWorlds - 1; // the largest w with pre[w] <= t (every world has a chunk)
    while (lo < hi) {
        const int mid = (lo + hi + 1) >> 1;
        if (pre[mid] <= t)
            lo = mid;
        else
            hi = mid - 1;
    }
    return lo;
}

template <bool ARM>
__global__ void __launch_bounds__(kQueueThreads, 4) roundQueueKernel(Dev d, StepParams p, QueueRounds qr) {
    pdlWait();
    pdlTrigger();
    __shared__ int sTile, sOk;
    const int nWorlds = d.ctr[C_WORLDS];
    const int ts = d.ctr[C_QSOLVE], td = d.ctr[C_QDUAL];
    const int perRound = ts + td;
    const int total = qr.rounds * perRound;
    const int *sPre = d.qPre, *dPre = d.qPre + (d.WW + 1);
    volatile int *errors = d.ctr + C_ERRORS;
    for (;;) {
        if (threadIdx.x == 0)
            sTile = static_cast<int>(atomicAdd(d.qTicket, 1u));
        __syncthreads();
        const int t = sTile;
        __syncthreads();
        if (t >= total)
            return;
        const int r = t / perRound;
        int u = t - r * perRound;
        const bool solve = u < ts;
        if (!solve)
            u -= ts;
        const int *pre = solve ? sPre : dPre;
        const int w = worldOfTile(pre, nWorlds, u);
        const int chunk = u - pre[w];
        const int q = 2 * r + (solve ? 0 : 1); // phases of world w completed before this tile may run
        if (threadIdx.x == 0) {
            sOk = 1;
            long long spins = 0;
            while (static_cast<int>(ldAcquireU32(reinterpret_cast<const unsigned *>(d.qStage + w))) < q) {
                if (++spins > d.waitLimit || (*errors & kErrQueueTimeout)) {
                    atomicOr(d.ctr + C_ERRORS, kErrQueueTimeout);
                    sOk = 0;
                    break;
                }
                __nanosleep(32);
            }
            __threadfence();
        }
        __syncthreads();
        if (!sOk)
            return;
        if (solve) {
            const int g = d.wBase[w] + chunk * kQueueThreads + threadIdx.x;
            if (((qr.newtonMask >> r) & 1u) && g < d.wBase[w] + d.wCount[w])
                solveAt<false, false>(d, p, g, 1);
        } else {
            const int k = d.wManStart[w] + chunk * kQueueThreads + threadIdx.x;
            if (k < d.wManStart[w + 1]) {
                const int m = d.wManList[k];
                if ((qr.stampMask >> r) & 1u)
                    dualAt<true, ARM, false>(d, p, qr.decay[r], m);
                else
                    dualAt<false, ARM, false>(d, p, qr.decay[r], m);
            }
        }
        __syncthreads();
        if (threadIdx.x == 0) {
            __threadfence(); // the tile's writes before its count
            if (atomicAdd(d.qDone + w, 1) + 1 == pre[w + 1] - pre[w]) {
                d.qDone[w] = 0;
                __threadfence();
                stReleaseU32(reinterpret_cast<unsigned *>(d.qStage + w), static_cast<unsigned>(q + 1));
            }
        }
    }
}

// Each live manifold into its world's group (the order inside a group does not matter: every
// manifold's dual reads and writes only its own state and its bodies' stamp entries).
__global__ void worldManCountKernel(Dev d) {
    pdlWait();
    pdlTrigger();
    const int n = d.ctr[C_LIVE];
    for (int m = blockIdx.x * blockDim.x + threadIdx.x; m < n; m += gridDim.x * blockDim.x)
        atomicAdd(&d.wManStart[d.meta[d.live.ab[m].x].x], 1);
}

__global__ void worldManFillKernel(Dev d) {
    pdlWait();
    pdlTrigger();
    const int n = d.ctr[C_LIVE];
    for (int m = blockIdx.x * blockDim.x + threadIdx.x; m < n; m += gridDim.x * blockDim.x) {
        const int w = d.meta[d.live.ab[m].x].x;
        d.wManList[d.wManStart[w] + atomicAdd(&d.wManFill[w], 1)] = m;
    }
}

// Chunks of each world's solve and dual phases (at least one each, so every phase of every world
// has a tile that advances its stage), zero past the last world; the stages start at zero.
__global__ void queueChunksKernel(Dev d) {
    pdlWait();
    pdlTrigger();
    const int nWorlds = d.ctr[C_WORLDS];
    const int w = blockIdx.x * blockDim.x + threadIdx.x;
    if (w > d.WW)
        return;
    int cs = 0, cd = 0;
    if (w < nWorlds) {
        cs = divUpDev(d.wCount[w], kQueueThreads);
        cd = divUpDev(d.wManStart[w + 1] - d.wManStart[w], kQueueThreads);
        cs = cs > 0 ? cs : 1;
        cd = cd > 0 ? cd : 1;
        d.qStage[w] = 0;
        d.qDone[w] = 0;
    }
    d.qPre[w] = cs;
    d.qPre[d.WW + 1 + w] = cd;
}

__global__ void overflowApplyKernel(Dev d, StepParams p) {
    pdlWait();
    pdlTrigger();
    const int g = blockIdx.x * blockDim.x + threadIdx.x;
    if (g < d.ctr[C_BODIES] && d.meta[g].x >= 0)
        overflowApplyAt(d, p, g);
}

__global__ void warmstartKernel(Dev d, StepParams p) {
    pdlWait();
    pdlTrigger();
    stampPhase(d);
    const int n = d.ctr[C_BODIES];
    const int g = blockIdx.x * blockDim.x + threadIdx.x;
    if (g < n && d.meta[g].x >= 0)
        warmstartAt(d, p, g);
}

__global__ void finishKernel(Dev d, StepParams p, int idle) {
    pdlWait();
    pdlTrigger();
    const int n = d.ctr[C_BODIES];
    const int g = blockIdx.x * blockDim.x + threadIdx.x;
    if (g < n && d.meta[g].x >= 0)
        finishAt(d, p, g, idle);
    if (g < d.WW)
        d.wActive[g] = 0; // until the projection finds manifolds to move
}

// The counters to the host's memory. As a kernel behind the step's others it starts when they end; a copy,
// like a memset between kernels, costs the work around it some microseconds of order (publish: 13 us a step;
// each memset 5-8), which is why the kernels of a step clear each other's counts.
__global__ void publishKernel(int *ctr, int *to) {
    if (threadIdx.x == 0)
        *reinterpret_cast<unsigned long long *>(ctr + C_CLOCK + 8) = nowNs(); // the step's end
    __syncthreads();
    if (threadIdx.x < C_COUNT)
        to[threadIdx.x] = ctr[threadIdx.x];
}

// ---- update set and colouring (solver_solve.cpp:263-424) ----

__global__ void contactOnlyInitKernel(Dev d) {
    pdlWait();
    pdlTrigger();
    const int g = blockIdx.x * blockDim.x + threadIdx.x;
    if (g < d.WW)
        d.wColour[g] = 0;
    if (g <= kMaxColours)
        d.colourCount[g] = 0;
    if (g >= d.ctr[C_BODIES])
        return;
    const bool dyn = d.meta[g].x >= 0 && d.x[g].w > 0.0f, update = selectBody(d, g, dyn);
    d.contactOnly[g] = 1;
    d.upd[g] = update ? 1 : 0;
    d.colour[g] = update ? kUncoloured : (dyn ? kNotUpdated : kOverflowColour);
}

__global__ void contactOnlyMarkKernel(Dev d) {
    pdlWait();
    pdlTrigger();
    const int f = blockIdx.x * blockDim.x + threadIdx.x;
    if (f >= d.ctr[C_FORCES])
        return;
    const int2 ab = d.fAB[f];
    if (ab.x >= 0)
        d.contactOnly[ab.x] = 0;
    if (ab.y >= 0)
        d.contactOnly[ab.y] = 0;
    d.wColour[d.meta[ab.y].x] = 1;
}

// One Jones-Plassmann attempt with list-order priority: a body is coloured once every earlier
// (lower list position) neighbour in the update set is, with the smallest colour none of them
// uses (the sequential greedy of colourGraph, reproduced exactly). A body still waiting counts
// itself in *waiting.
__device__ __forceinline__ unsigned loadColour(const uint8_t *p) {
    unsigned v;
    asm volatile("ld.acquire.gpu.global.u8 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
    return v;
}

__device__ __forceinline__ void publishColour(uint8_t *p, unsigned v) {
    asm volatile("st.release.gpu.global.u8 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}

constexpr int kColourThreads = 512;

// Greedy colouring (solver_solve.cpp:365-424) as a dataflow in one cooperative launch: bodies are
// taken in increasing list position; each waits until its earlier dynamic neighbours have
// published their colours, takes the smallest colour none of them has (or the overflow colour)
// and publishes it. That is the sequential greedy assignment; the body with the smallest
// uncoloured list position can always proceed, so the waits end (each is bounded anyway).
// Worlds that no force touches hold only contact-only bodies, which go to the overflow colour
// whatever their greedy colour, so they are not coloured at all (unless every body is coloured).
__global__ void __launch_bounds__(kColourThreads) colourFlowKernel(Dev d, int everyWorld) {
    pdlWait();
    pdlTrigger();
    const int n = d.ctr[C_BODIES];
    const int stride = gridDim.x * blockDim.x;
    volatile int *errors = d.ctr + C_ERRORS;
    for (int p = blockIdx.x * blockDim.x + threadIdx.x; p < n; p += stride) {
        const int g = d.lpToBody[p];
        if (g < 0 || d.meta[g].x < 0 || !inUpdate(d, g))
            continue;
        if (!everyWorld && !d.wColour[d.meta[g].x]) {
            publishColour(d.colour + g, kOverflowColour);
            continue;
        }
        unsigned used = 0;
        for (int e = d.adjStart[g]; e < d.adjStart[g + 1]; e++) {
            const int h = adjInfoOther(d.adjInfo[e]);
            if (h < 0 || !inUpdate(d, h) || listPos(d, h) >= p)
                continue;
            unsigned c;
            long long spins = 0;
            while ((c = loadColour(d.colour + h)) == kUncoloured) {
                if (++spins > d.waitLimit || (*errors & kErrColourTimeout)) {
                    atomicOr(d.ctr + C_ERRORS, kErrColourTimeout);
                    return;
                }
                __nanosleep(64);
            }
            if (c < kMaxColours)
                used |= 1u << c;
        }
        unsigned c = kOverflowColour;
        for (int k = 0; k < kMaxColours; k++)
            if (!(used & (1u << k))) {
                c = static_cast<unsigned>(k);
                break;
            }
        publishColour(d.colour + g, c);
    }
}

// The same colouring, a block a world, for worlds of up to kColourWorldMost bodies: colours and earlier
// neighbours lie in shared memory, and a warp looks at all its waiting bodies in turn, so a hop from
// a body to the next costs one such pass (0.1 us) instead of a trip through L2 and the turns of the
// warp's other waiting lanes (2 us): a 1653-box pile with a chain of 32 72 -> 21 us, 600 bodies with ragdolls
// 33 -> 9.
constexpr int kColourWorldMost = 4096;
constexpr int kColourWorldThreads = 1024;
constexpr int kColourHeld = kColourWorldMost / kColourWorldThreads; // bodies a thread
constexpr int kColourNear = 16;  // earlier neighbours in shared memory; a body with more reads them all from L2
constexpr size_t kColourBodyBytes = sizeof(uint16_t) * kColourNear + 2;

__global__ void __launch_bounds__(kColourWorldThreads) colourWorldKernel(const __grid_constant__ Dev d, int everyWorld, int most) {
    pdlWait();
    pdlTrigger();
    extern __shared__ uint16_t nearList[]; // most x kColourNear, then the counts and the colours
    uint8_t *nearCount = reinterpret_cast<uint8_t *>(nearList + static_cast<size_t>(most) * kColourNear);
    volatile uint8_t *colours = nearCount + most;
    __shared__ int stopped;
    const int nWorlds = d.ctr[C_WORLDS];
    for (int world = blockIdx.x; world < nWorlds; world += gridDim.x) {
        const int base = d.wBase[world], cnt = d.wCount[world];
        if (cnt <= 0)
            continue;
        if (!everyWorld && !d.wColour[world]) {
            for (int i = threadIdx.x; i < cnt; i += blockDim.x)
                if (inUpdate(d, base + i))
                    d.colour[base + i] = kOverflowColour;
            continue;
        }
        __syncthreads(); // the world before has been read
        if (threadIdx.x == 0)
            stopped = 0;
        // A later slot is an earlier list position.
        for (int i = threadIdx.x; i < cnt; i += blockDim.x) {
            const int g = base + i;
            const bool update = inUpdate(d, g);
            int n = 0;
            const int e1 = update ? d.adjStart[g + 1] : 0;
            for (int e = update ? d.adjStart[g] : 0; e < e1; e += 4) {
                int h[4], in[4];
#pragma unroll
                for (int k = 0; k < 4; k++)
                    h[k] = e + k < e1 ? adjInfoOther(d.adjInfo[e + k]) : -1;
#pragma unroll
                for (int k = 0; k < 4; k++)
                    in[k] = h[k] > g && inUpdate(d, h[k]);
#pragma unroll
                for (int k = 0; k < 4; k++)
                    if (in[k]) {
                        if (n < kColourNear)
                            nearList[i * kColourNear + n] = static_cast<uint16_t>(h[k] - base);
                        n = min(n + 1, kColourNear + 1);
                    }
            }
            nearCount[i] = static_cast<uint8_t>(n);
            colours[i] = kUncoloured;
        }
        __syncthreads();
        unsigned used[kColourHeld] = {};
        int next[kColourHeld] = {}; // its first neighbour not seen yet; done: -1
        bool open = false;
#pragma unroll
        for (int k = 0; k < kColourHeld; k++) {
            const int i = cnt - 1 - static_cast<int>(threadIdx.x + k * blockDim.x); // in list order
            next[k] = i >= 0 && inUpdate(d, base + i) ? (nearCount[i] > kColourNear ? d.adjStart[base + i] : 0) : -1;
            open = open || next[k] >= 0;
        }
        long long passed = 0;
        bool late = false;
        while (__any_sync(0xffffffffu, open)) {
            open = false;
            bool waits = false;
#pragma unroll
            for (int k = 0; k < kColourHeld; k++) {
                if (next[k] < 0)
                    continue;
                const int i = cnt - 1 - static_cast<int>(threadIdx.x + k * blockDim.x);
                const bool far = nearCount[i] > kColourNear;
                const int end = far ? d.adjStart[base + i + 1] : nearCount[i];
                for (; next[k] < end; next[k]++) {
                    int h;
                    if (far) {
                        h = adjInfoOther(d.adjInfo[next[k]]) - base;
                        if (h <= i || !inUpdate(d, base + h))
                            continue;
                    } else {
                        h = nearList[i * kColourNear + next[k]];
                    }
                    const unsigned c = colours[h];
                    if (c == kUncoloured)
                        break;
                    if (c < kMaxColours)
                        used[k] |= 1u << c;
                }
                if (next[k] < end) {
                    open = waits = true;
                    continue;
                }
                unsigned c = kOverflowColour;
#pragma unroll
                for (int q = kMaxColours - 1; q >= 0; q--)
                    c = used[k] & (1u << q) ? c : static_cast<unsigned>(q);
                colours[i] = static_cast<uint8_t>(c);
                next[k] = -1;
            }
            if (waits && ++passed > d.waitLimit) {
                late = true;
                stopped = 1;
            }
            if (late || *const_cast<volatile int *>(&stopped))
                open = false;
        }
        if (late)
            atomicOr(d.ctr + C_ERRORS, kErrColourTimeout);
        __syncthreads();
        for (int i = threadIdx.x; i < cnt; i += blockDim.x)
            if (inUpdate(d, base + i))
                d.colour[base + i] = colours[i];
    }
}

__global__ void colourListKernel(Dev d, int contactOnlyOverflow) {
    pdlWait();
    pdlTrigger();
    const int n = d.ctr[C_BODIES];
    const int g = blockIdx.x * blockDim.x + threadIdx.x;
    if (g >= n || d.meta[g].x < 0 || !inUpdate(d, g))
        return;
    uint8_t c = d.colour[g];
    if (contactOnlyOverflow && d.contactOnly[g])
        c = kOverflowColour;
    if (c > kOverflowColour) // left uncoloured by a colouring that timed out (the step reports it)
        c = kOverflowColour;
    d.colour[g] = c;
    // One atomic per warp and colour (the overflow colour is counted, not listed).
    const unsigned active = __activemask();
    const unsigned peers = __match_any_sync(active, static_cast<int>(c));
    const int leader = __ffs(peers) - 1;
    const int lane = threadIdx.x & 31;
    int base = 0;
    if (lane == leader)
        base = atomicAdd(&d.colourCount[c], __popc(peers));
    base = __shfl_sync(peers, base, leader);
    if (c < kOverflowColour)
        d.colourList[c * d.NB + base + __popc(peers & ((1u << lane) - 1u))] = g;
}

} // namespace

static int grid(int n) { return divUp(n > 0 ? n : 1, kThreads); }
static int queueGridMax();

void launchContactOnly(const Dev &d, cudaStream_t s) {
    const int most = d.NB > d.WW ? d.NB : d.WW;
    ++launchCount(); launchK(contactOnlyInitKernel, grid(most > kMaxColours ? most : kMaxColours + 1), kThreads, 0, s, d);
    ++launchCount(); launchK(contactOnlyMarkKernel, grid(d.FF), kThreads, 0, s, d);
}

static int g_colourBlocks = 0;

int colourGridBlocks() {
    if (g_colourBlocks == 0) {
        int dev = 0, sms = 0, perSm = 0;
        cudaGetDevice(&dev);
        cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&perSm, colourFlowKernel, kColourThreads, 0);
        g_colourBlocks = sms * (perSm < 1 ? 1 : (perSm > 2 ? 2 : perSm));
        if (g_colourBlocks < 1)
            g_colourBlocks = 1;
    }
    return g_colourBlocks;
}

bool dualBlockFits(int block) {
    return blockFits(dualKernel<false, false>, block) && blockFits(dualKernel<true, false>, block) &&
           blockFits(dualKernel<false, true>, block) && blockFits(dualKernel<true, true>, block);
}

bool solveBlockFits(int block) {
    return blockFits(overflowSolveKernel<false, true>, block) && blockFits(overflowSolveKernel<true, true>, block) &&
           blockFits(overflowSolveKernel<false, false>, block) && blockFits(overflowSolveKernel<true, false>, block);
}

static int g_sweepBlocks = 0;

static int sweepGridMax() {
    if (g_sweepBlocks == 0) {
        int dev = 0, sms = 0, perSm = 0;
        cudaGetDevice(&dev);
        cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&perSm, colourSweepKernel, kSolveThreads, 0);
        g_sweepBlocks = sms * (perSm < 1 ? 1 : perSm);
    }
    return g_sweepBlocks;
}

void prepareKernels() {
    worldTeamMax();
    worldPairsMost();
    prepareWorldContacts();
    sweepGridMax();
    queueGridMax();
    projectionGridBlocks();
    preparePrimitives();
    prepareNarrowPhase();
    brakeGridBlocks();
    colourGridBlocks();
    cudaFuncSetAttribute(colourWorldKernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                         static_cast<int>(kColourBodyBytes * kColourWorldMost));
}

int colourWorldMost() { return kColourWorldMost; }

void launchColour(const Dev &d, bool needGreedy, bool everyWorld, int largest, cudaStream_t s) {
    if (!needGreedy)
        return;
    if (largest > 0) {
        const int most = 4 * smCount(), blocks = d.WW < most ? d.WW : most;
        ++launchCount();
        launchK(colourWorldKernel, blocks, kColourWorldThreads, kColourBodyBytes * static_cast<size_t>(largest), s, d,
                everyWorld ? 1 : 0, largest);
        return;
    }
    // No more blocks than the store's bodies can fill.
    const int want = divUp(d.NB > 0 ? d.NB : 1, kColourThreads), most = colourGridBlocks();
    Dev dd = d;
    int every = everyWorld ? 1 : 0;
    void *args[] = {&dd, &every};
    ++launchCount();
    cudaLaunchCooperativeKernel(reinterpret_cast<void *>(colourFlowKernel), dim3(want < most ? want : most),
                                dim3(kColourThreads), args, 0, s);
}

void launchColourLists(const Dev &d, int contactOnlyOverflow, cudaStream_t s) {
    ++launchCount(); launchK(colourListKernel, grid(d.NB), kThreads, 0, s, d, contactOnlyOverflow);
}

void launchWarmstartBodies(const Dev &d, const StepParams &p, cudaStream_t s) {
    ++launchCount(); launchK(warmstartKernel, grid(d.NB), kThreads, 0, s, d, p);
}

void launchFinishBodies(const Dev &d, const StepParams &p, bool idle, cudaStream_t s) {
    ++launchCount(); launchK(finishKernel, grid(d.NB > d.WW ? d.NB : d.WW), kThreads, 0, s, d, p, idle ? 1 : 0);
}

void launchPublish(const Dev &d, int *to, cudaStream_t s) {
    static_assert(C_COUNT <= kThreads, "one block");
    ++launchCount(); // in plain stream order: it comes behind a graph as often as behind a kernel
    publishKernel<<<1, kThreads, 0, s>>>(d.ctr, to);
}

void launchStamps(const Dev &d, const StepParams &p, bool mixedOnly, cudaStream_t s) {
    ++launchCount(); launchK(stampsKernel, residentGrid(stampsKernel, kThreads, grid(d.MM)), kThreads, 0, s, d, p, mixedOnly ? 1 : 0);
}

void launchColourSweep(const Dev &d, const StepParams &p, bool armsFromDual, cudaStream_t s) {
    // With contact-only bodies in the overflow colour, a coloured body has a force of its own and a
    // force touches at most two bodies, so the grid (and its barrier) scales with the forces.
    const int bound = p.contactOnlyOverflow && d.FF < d.NB / 2 ? 2 * d.FF : d.NB;
    const int want = divUp(bound > 0 ? bound : 1, kSolveThreads), most = sweepGridMax();
    const int blocks = want < most ? want : most;
    cudaMemsetAsync(d.gridBar, 0, sizeof(unsigned), s);
    Dev dd = d;
    StepParams pp = p;
    int arms = armsFromDual ? 1 : 0;
    void *args[] = {&dd, &pp, &arms};
    ++launchCount();
    cudaLaunchCooperativeKernel(reinterpret_cast<void *>(colourSweepKernel), dim3(blocks), dim3(kSolveThreads),
                                args, 0, s);
}

template <bool FORCES>
static void solveLaunch(const Dev &d, const StepParams &p, bool inPlace, int block, cudaStream_t s) {
    // Stores of several waves of bodies wait on memory: there the plain divisions' fewer registers count
    // (441,690 bodies: 52.4 us a round plain, 55.9 with grouped quotients); smaller ones wait on a body's
    // chain (65,537 bodies: 9.9 plain, 9.4 grouped).
    if (d.NB > 131072)
        launchK(overflowSolveKernel<FORCES, false>, divUp(d.NB, block), block, 0, s, d, p, inPlace ? 1 : 0);
    else
        launchK(overflowSolveKernel<FORCES, true>, divUp(d.NB, block), block, 0, s, d, p, inPlace ? 1 : 0);
}

void launchOverflowSolve(const Dev &d, const StepParams &p, bool inPlace, bool forces, int block, cudaStream_t s) {
    ++launchCount();
    forces ? solveLaunch<true>(d, p, inPlace, block, s) : solveLaunch<false>(d, p, inPlace, block, s);
}

static int g_queueBlocks = 0;

static int queueGridMax() {
    if (g_queueBlocks == 0) {
        int dev = 0, sms = 0, perSm = 0, perSmArm = 0;
        cudaGetDevice(&dev);
        cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&perSm, roundQueueKernel<false>, kQueueThreads, 0);
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&perSmArm, roundQueueKernel<true>, kQueueThreads, 0);
        perSm = perSm < perSmArm ? perSm : perSmArm;
        g_queueBlocks = sms * (perSm < 1 ? 1 : perSm);
    }
    return g_queueBlocks;
}

void launchRoundQueue(const Dev &d, const StepParams &p, const QueueRounds &qr, cudaStream_t s) {
    const int cap = static_cast<int>(static_cast<size_t>(d.WW) + 1);
    cudaMemsetAsync(d.wManStart, 0, sizeof(int) * static_cast<size_t>(cap), s);
    cudaMemsetAsync(d.wManFill, 0, sizeof(int) * static_cast<size_t>(d.WW), s);
    ++launchCount(); launchK(worldManCountKernel, residentGrid(worldManCountKernel, kThreads, grid(d.MM)), kThreads, 0, s, d);
    scanExclusive(d.wManStart, d.wManStart, cap, nullptr, nullptr, d.scanScratch, s);
    ++launchCount(); launchK(worldManFillKernel, residentGrid(worldManFillKernel, kThreads, grid(d.MM)), kThreads, 0, s, d);
    ++launchCount(); launchK(queueChunksKernel, divUp(cap, kThreads), kThreads, 0, s, d);
    scanExclusive(d.qPre, d.qPre, cap, nullptr, d.ctr + C_QSOLVE, d.scanScratch, s);
    scanExclusive(d.qPre + cap, d.qPre + cap, cap, nullptr, d.ctr + C_QDUAL, d.scanScratch, s);
    cudaMemsetAsync(d.qTicket, 0, sizeof(unsigned), s);
    Dev dd = d;
    StepParams pp = p;
    QueueRounds q = qr;
    void *args[] = {&dd, &pp, &q};
    ++launchCount();
    cudaLaunchCooperativeKernel(p.armCache ? reinterpret_cast<void *>(roundQueueKernel<true>)
                                           : reinterpret_cast<void *>(roundQueueKernel<false>),
                                dim3(queueGridMax()), dim3(kQueueThreads), args, 0, s);
}

void launchOverflowApply(const Dev &d, const StepParams &p, cudaStream_t s) {
    ++launchCount();
    launchK(overflowApplyKernel, grid(d.NB), kThreads, 0, s, d, p);
}

template <bool STAMPS, bool ARM>
static void dualLaunch(const Dev &d, const StepParams &p, real decay, int block, cudaStream_t s) {
    const int blocks = residentGrid(dualKernel<STAMPS, ARM>, block, divUp(d.MM, block));
    launchK(dualKernel<STAMPS, ARM>, blocks, block, 0, s, d, p, decay);
}

void launchDual(const Dev &d, const StepParams &p, bool stamps, real decay, int block, cudaStream_t s) {
    ++launchCount();
    if (p.armCache)
        stamps ? dualLaunch<true, true>(d, p, decay, block, s) : dualLaunch<false, true>(d, p, decay, block, s);
    else
        stamps ? dualLaunch<true, false>(d, p, decay, block, s) : dualLaunch<false, false>(d, p, decay, block, s);
}

void launchForceDual(const Dev &d, const StepParams &p, bool forces, cudaStream_t s) {
    if (!forces)
        return;
    ++launchCount(); launchK(forceDualKernel, grid(d.FF), kThreads, 0, s, d, p);
}

} // namespace avbdg
