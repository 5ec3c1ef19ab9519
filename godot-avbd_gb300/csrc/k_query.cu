// Spatial queries of one world (godot-avbd src/avbd/solver_query.cpp): ray picks and box overlap
// collection. The reference scans the body list; here every (ray, body) pair is one thread and the
// nearest hit per ray is an atomic minimum over (distance, list position), so the winner is the
// reference's (the first body in list order among equal distances). Overlap flags are compacted in
// list order.

#include <cfloat>

#include "kernels.cuh"
#include "prims.cuh"

namespace avbdg {

namespace {

constexpr int kThreads = 256;

__device__ __forceinline__ f3 localHalfExtent(const Dev &d, int g) {
    const real4 s = d.size[g];
    const int shape = (d.meta[g].w >> 18) & 0x3;
    return shape == 1 ? f3{s.x, s.x, s.x} : (shape == 2 ? f3{s.x, s.x, s.z * 0.5f} : scale(xyz(s), 0.5f));
}

// What the ray test reads of a body.
struct RayBody {
    f3 x;
    q4 q;
    f3 half; // x: a sphere's radius
    bool sphere;
};
__device__ __forceinline__ RayBody rayBody(const Dev &d, int g) {
    return RayBody{xyz(d.x[g]), asq(d.q[g]), localHalfExtent(d, g), ((d.meta[g].w >> 18) & 0x3) == 1};
}

// The reference's per-body ray test (solver_query.cpp:48-133): distance in units of `dir` or
// +infinity, and the hit point in the body's frame.
__device__ real rayTest(const RayBody &body, f3 origin, f3 dir, f3 &local) {
    const real inf = bitsf(0x7f800000);
    const q4 inv = qconj(body.q);
    const f3 o = qrot(inv, sub(origin, body.x));
    const f3 dd = qrot(inv, dir);
    if (body.sphere) {
        const real r = body.half.x;
        const real b = dot(o, dd);
        const real c = length2(o) - r * r;
        const real disc = b * b - c;
        if (disc < 0.0f)
            return inf;
        const real sq = msqrt(disc);
        real t = -b - sq;
        if (t < 0.0f)
            t = -b + sq;
        if (t < 0.0f)
            return inf;
        local = add(o, scale(dd, t));
        return t;
    }
    const f3 half = body.half;
    real tEnter = 0.0f, tExit = inf;
    for (int i = 0; i < 3; ++i) {
        const real di = at(dd, i), oi = at(o, i), hi = at(half, i);
        if (mabs(di) < 1.0e-6f) {
            if (oi < -hi || oi > hi)
                return inf;
            continue;
        }
        const real invD = 1.0f / di;
        real t0 = (-hi - oi) * invD;
        real t1 = (hi - oi) * invD;
        if (t0 > t1) {
            const real tmp = t0;
            t0 = t1;
            t1 = tmp;
        }
        tEnter = smax(tEnter, t0);
        tExit = smin(tExit, t1);
        if (tEnter > tExit)
            return inf;
    }
    const real tHit = tEnter >= 0.0f ? tEnter : tExit;
    if (tHit < 0.0f)
        return inf;
    local = add(o, scale(dd, tHit));
    return tHit;
}

// The rays' origins, then their directions.
__device__ __forceinline__ f3 rayOrigin(const float *rays, int r) { return f3{rays[3 * r], rays[3 * r + 1], rays[3 * r + 2]}; }
__device__ __forceinline__ f3 rayDirection(const float *rays, int nRays, int r) { return rayOrigin(rays + 3 * static_cast<size_t>(nRays), r); }

__global__ void pickResetKernel(unsigned long long *best, int rays) {
    pdlWait();
    pdlTrigger();
    const int r = blockIdx.x * blockDim.x + threadIdx.x;
    if (r < rays)
        best[r] = ~0ull;
}

// A hit's key = (distance bits, list position), distances >= 0 compare as integers (-0 counts as +0, as
// the reference's comparisons do).
__device__ __forceinline__ void putHit(unsigned long long *best, real dist, unsigned listPosition) {
    if (dist < bitsf(0x7f800000))
        atomicMin(best, (static_cast<unsigned long long>(static_cast<unsigned>(fbits(dist + 0.0f))) << 32) | listPosition);
}

// Few pairs: a thread each.
__global__ void pickKernel(Dev d, int base, int count, const float *rays, int nRays, unsigned mask,
                           unsigned long long *best) {
    pdlWait();
    pdlTrigger();
    const long long t = static_cast<long long>(blockIdx.x) * blockDim.x + threadIdx.x;
    if (t >= static_cast<long long>(nRays) * count)
        return;
    const int r = static_cast<int>(t / count);
    const int g = base + static_cast<int>(t % count);
    if ((static_cast<unsigned>(d.meta[g].y) & mask) == 0)
        return;
    f3 local;
    const real dist = rayTest(rayBody(d, g), rayOrigin(rays, r), rayDirection(rays, nRays, r), local);
    putHit(best + r, dist, static_cast<unsigned>(listPos(d, g) - base));
}

// Many pairs: a thread a ray against a tile of bodies in shared memory. Nearly every pair is far apart,
// which a cross product shows: the line through o along the unit d passes the origin at |o x d|. A pair
// is left out only where that is clearly more than the body's bounding radius (limit below, with |o|^2
// as the scale of what rounding may do, and more than it does). The others go to a queue of
// their warp, and the whole test runs on 32 of them at a time. Rays that are not of unit length and
// bodies whose orientation is not are never left out; a NaN leaves nothing out.
// 4096 rays, 1653 bodies: a thread per pair 53 us, bound by the three divisions and the branches
// of 6.8 M whole tests; 16 us this way.
constexpr int kPickBodies = 64;

__global__ void __launch_bounds__(kThreads) pickTileKernel(const __grid_constant__ Dev d, int base, int count, const float *rays,
                                                           int nRays, unsigned mask, unsigned long long *best) {
    pdlWait();
    pdlTrigger();
    __shared__ RayBody bodies[kPickBodies];
    __shared__ real4 spheres[kPickBodies]; // centre, squared radius with its margin
    __shared__ unsigned places[kPickBodies];
    __shared__ f3 origins[kThreads], dirs[kThreads];
    __shared__ uint16_t queues[kThreads / 32][64];
    __shared__ int found;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int r = blockIdx.x * kThreads + threadIdx.x, rayBase = r - lane;
    const real inf = bitsf(0x7f800000);
    const bool on = r < nRays;
    const f3 o = on ? rayOrigin(rays, r) : f3{0, 0, 0}, dir = on ? rayDirection(rays, nRays, r) : f3{0, 0, 0};
    origins[threadIdx.x] = o;
    dirs[threadIdx.x] = dir;
    if (threadIdx.x == 0)
        found = 0;
    __syncthreads();
    const int i = blockIdx.y * kPickBodies + threadIdx.x;
    if (threadIdx.x < kPickBodies && i < count) {
        const int g = base + i;
        if ((static_cast<unsigned>(d.meta[g].y) & mask) != 0) {
            const RayBody b = rayBody(d, g);
            const real r2 = b.sphere ? b.half.x * b.half.x : length2(b.half), qq = qlength2(b.q);
            const int at = atomicAdd(&found, 1);
            bodies[at] = b;
            spheres[at] = f4(b.x, mabs(qq - 1.0f) <= 1.0e-5f ? 1.02f * r2 : inf);
            places[at] = static_cast<unsigned>(listPos(d, g) - base);
        }
    }
    __syncthreads();
    const bool unit = mabs(length2(dir) - 1.0f) <= 1.0e-5f;
    uint16_t *queue = queues[warp];
    int queued = 0;
    const int n = found;
    const auto test = [&](int k) {
        const int entry = queue[k], from = 32 * warp + (entry & 31), b = entry >> 5;
        f3 local;
        putHit(best + rayBase + (entry & 31), rayTest(bodies[b], origins[from], dirs[from], local), places[b]);
    };
    for (int b = 0; b < n; b++) {
        const real4 s = spheres[b];
        const f3 rel = sub(o, xyz(s)), c = cross(rel, dir);
        const bool far = unit && length2(c) > s.w + 2.0e-4f * length2(rel);
        const unsigned near = __ballot_sync(0xffffffffu, on && !far);
        if (near >> lane & 1u)
            queue[queued + __popc(near & ((1u << lane) - 1u))] = static_cast<uint16_t>(b << 5 | lane);
        queued += __popc(near);
        __syncwarp();
        if (queued >= 32) {
            test(lane);
            __syncwarp();
            if (lane < queued - 32)
                queue[lane] = queue[32 + lane];
            queued -= 32;
            __syncwarp();
        }
    }
    if (lane < queued)
        test(lane);
}

__global__ void pickResultKernel(Dev d, int base, int count, const float *rays, int nRays,
                                 const unsigned long long *best, int *outBody, float *outLocal) {
    pdlWait();
    pdlTrigger();
    const int r = blockIdx.x * blockDim.x + threadIdx.x;
    if (r >= nRays)
        return;
    const unsigned long long key = best[r];
    if (key == ~0ull) {
        outBody[r] = -1;
        outLocal[3 * r] = outLocal[3 * r + 1] = outLocal[3 * r + 2] = 0.0f;
        return;
    }
    const int g = base + (count - 1 - static_cast<int>(key & 0xffffffffu)); // list position -> slot
    f3 local{0, 0, 0};
    rayTest(rayBody(d, g), rayOrigin(rays, r), rayDirection(rays, nRays, r), local);
    outBody[r] = g - base;
    outLocal[3 * r] = local.x;
    outLocal[3 * r + 1] = local.y;
    outLocal[3 * r + 2] = local.z;
}

// Overlap flag per list position of the world (collectAABB's test, solver_query.cpp:154-170).
__global__ void overlapFlagKernel(Dev d, int base, int count, f3 lo, f3 hi, unsigned mask, int *flags) {
    pdlWait();
    pdlTrigger();
    const int p = blockIdx.x * blockDim.x + threadIdx.x;
    if (p >= count)
        return;
    const int g = base + (count - 1 - p);
    int hit = 0;
    if ((static_cast<unsigned>(d.meta[g].y) & mask) != 0) {
        const m3 rot = qmat(asq(d.q[g]));
        const f3 h = localHalfExtent(d, g);
        const f3 wx{(mabs(rot.c0.x) * h.x + mabs(rot.c1.x) * h.y) + mabs(rot.c2.x) * h.z,
                    (mabs(rot.c0.y) * h.x + mabs(rot.c1.y) * h.y) + mabs(rot.c2.y) * h.z,
                    (mabs(rot.c0.z) * h.x + mabs(rot.c1.z) * h.y) + mabs(rot.c2.z) * h.z};
        const f3 c = xyz(d.x[g]);
        const f3 bmin = sub(c, wx), bmax = add(c, wx);
        hit = !(bmin.x > hi.x || bmin.y > hi.y || bmin.z > hi.z || lo.x > bmax.x || lo.y > bmax.y || lo.z > bmax.z);
    }
    flags[p] = hit;
}

__global__ void overlapScatterKernel(int base, int count, const int *flags, const int *rank, int capacity,
                                     int *out) {
    pdlWait();
    pdlTrigger();
    const int p = blockIdx.x * blockDim.x + threadIdx.x;
    if (p >= count || !flags[p])
        return;
    if (rank[p] < capacity)
        out[rank[p]] = count - 1 - p; // list position -> creation index
}

} // namespace

// From about a million pairs a ray's thread against a tile of bodies is faster. Kernel alone, microseconds
// there and as a thread per pair: 1653 bodies 512 rays 10.2 / 8.7, 1024 rays 10.1 / 14.5, 8192 rays
// 28.8 / 97.5; 30,000 bodies 64 rays 15.1 / 16.1, 512 rays 32.4 / 110; 50 bodies 8192 rays 8.7 / 5.6.
constexpr long long kTilePairs = 1 << 20;
constexpr int kTileRays = 64;

void launchPick(const Dev &d, int base, int count, const float *rays, int nRays, unsigned mask,
                unsigned long long *best, int *outBody, float *outLocal, cudaStream_t s) {
    ++launchCount(); launchK(pickResetKernel, divUp(nRays > 0 ? nRays : 1, kThreads), kThreads, 0, s, best, nRays);
    const long long pairs = static_cast<long long>(nRays) * count;
    if (pairs >= kTilePairs && nRays >= kTileRays && divUp(count, kPickBodies) < 65536) {
        ++launchCount();
        launchK(pickTileKernel, dim3(divUp(nRays, kThreads), divUp(count, kPickBodies)), kThreads, 0, s, d, base, count, rays, nRays,
                mask, best);
    } else if (pairs > 0) {
        ++launchCount();
        launchK(pickKernel, static_cast<unsigned>((pairs + kThreads - 1) / kThreads), kThreads, 0, s, d, base, count, rays,
                                                                                              nRays, mask, best);
    }
    ++launchCount();
    launchK(pickResultKernel, divUp(nRays > 0 ? nRays : 1, kThreads), kThreads, 0, s, d, base, count, rays, nRays, best,
                                                                                 outBody, outLocal);
}

void launchCollectAabb(const Dev &d, int base, int count, f3 lo, f3 hi, unsigned mask, int *flags, int *rank,
                       int *total, void *scanScratch, int capacity, int *out, cudaStream_t s) {
    ++launchCount();
    launchK(overlapFlagKernel, divUp(count > 0 ? count : 1, kThreads), kThreads, 0, s, d, base, count, lo, hi, mask, flags);
    scanExclusive(flags, rank, count, nullptr, total, scanScratch, s);
    ++launchCount();
    launchK(overlapScatterKernel, divUp(count > 0 ? count : 1, kThreads), kThreads, 0, s, base, count, flags, rank, capacity,
                                                                                    out);
}

} // namespace avbdg
