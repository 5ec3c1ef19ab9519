// The step from the brake to the rebase as one launch, a thread-block cluster per world.
//
// Everything after the adjacency and the colouring is local to a world: the brake sweep, the body
// warm start, the rounds, the finish, the projection and the rebase. On stores of ordinary worlds
// these phases are bound by latency, not by bandwidth: a few hundred bodies are one thread's serial
// chain of L2 round trips in each of ~30 kernels, with most SMs idle. Here one cluster of CTAs keeps
// a world for all of them and meets at hardware cluster barriers, the world's state lies in the
// cluster's distributed shared memory, and each phase spreads it over more threads than the separate
// launches do, with the same sums in the same order:
//
//   state     each CTA owns a range of the world's bodies (poses, step constants, the stamp records
//             of their adjacency entries) and a range of its manifolds (basis, contacts); contact
//             lanes read the two poses from their owners' shared memory and store the stamp records
//             there, so a round makes no trip to L2.
//   contacts  a lane a contact, whole manifolds packed into warps. The lanes leave their stamp terms
//             in shared memory and the warp's lanes add them, four sums a lane, in contact order
//             from zero.
//   bodies    the block's thirty sums are one lane each: a warp adds a body's stamp records in entry
//             order; a thread per body then factorises.
//   colours   the coloured bodies are dealt round the CTAs, wherever their state lies. A lane takes a
//             contact of one's manifolds or a part of one of its forces, lanes of a kind together in a
//             warp; a warp a body then adds the terms in adjacency order.
//   brake     a single CTA of the cluster runs the sweep, level by level of its dependencies, with the
//             world's velocities in shared memory.
//
// Of every four warps three take contacts and one takes bodies: what is left of a phase is one warp's
// instruction stream, and a scheduler that runs one phase's code keeps it in its instruction cache.
//
// A world whose parts do not fit in shared memory is left, whole, to worldWideKernel, which runs the
// separate launches' per-item functions on the global arrays in the same order.

#include <algorithm>

#include "cluster.cuh"
#include "kernels.cuh"
#include "prims.cuh"
#include "project.cuh"
#include "solve.cuh"

namespace avbdg {

namespace {

constexpr int kMaxWorldThreads = 512;
constexpr int kWideThreads = 256;
constexpr int kTaskManifolds = 8; // manifolds a task of 32 contact slots may hold: 96 groups of four sums
// A contact's stamp terms in shared memory: twelve groups of four (0, 1: the part both sides share;
// 2-6: side A; 7-11: side B), padded so that eight lanes' 16-byte accesses hit distinct banks.
constexpr int kRowReals = 52;
constexpr int kBlkReals = 31; // a body's thirty block sums, padded
constexpr int kVelReals = 6;

// Flags of a live manifold, constant over a step (bits 8-11: its contacts).
enum : int {
    kMfAwake = 1,  // a side is awake (dual pass)
    kMfSideA = 2,  // overflow sides: take stamps
    kMfSideB = 4,
    kMfMixed = 8,  // a coloured body touches it
    kMfMoveA = 16, // movable sides (brake, projection)
    kMfMoveB = 32,
    kMfMassA = 64, // sides with mass: they have adjacency entries
    kMfMassB = 128,
    kMfCountShift = 8
};
// A manifold with contacts and a movable side.
__device__ __forceinline__ bool mfActive(int f) { return (f & (kMfMoveA | kMfMoveB)) != 0 && (f >> kMfCountShift) != 0; }

// What a body's neighbours read of it (kRecF4 values, at its owner): the rotation's columns (w: the
// step's displacement, a component each), the step's rotation vector, position and mass,
// orientation, moment.
enum : int { kRecAng = 3, kRecX = 4, kRecQ = 5, kRecMoment = 6, kRecF4 = 7 };
// Its step constants: inertial position and orientation, step-start position and orientation.
enum : int { kConXi = 0, kConQi = 1, kConX0 = 2, kConQ0 = 3, kConF4 = 4 };
// Body flags: colour, in the update set, movable, has a force, axis locks.
enum : int { kBiColour = 0xf, kBiUpdate = 16, kBiMovable = 32, kBiForce = 64, kBiLocks = 8 };

// The world a cluster works on and this CTA's part of it, with the byte offsets of its arrays.
struct World {
    int rank, size;        // this CTA's place in the cluster
    int base, cnt;         // bodies
    int m0, n;             // live manifolds
    int f0, f1;            // forces
    int per, b0, nb;       // bodies a CTA; this CTA's
    int mlo, nm;           // this CTA's manifolds
    int e0;                // its bodies' first adjacency entry
    int tasks, conStride;  // contact tasks; bytes of one contact array
    int levelsFit;         // the brake's levels lie in shared memory (else in a global array)
    int sums, info, entry, rec, con, stamps; // bodies
    int mf, link, basis, cap, taskFirst;     // manifolds
    int slots, contacts;                     // contact slots
    // The coloured bodies dealt to this CTA, by colour, their blocks and their terms.
    int colourList, colourBlocks, termFirst, terms, termOrder, termKinds;
    int colourAt[kMaxColours + 1]; // first of each colour in the list
    int groupAt[kMaxColours + 1];  // first group of terms of each colour
    int rec0, con0;                // this CTA's address of the pose records and step constants
};

__device__ __forceinline__ real4 loadCluster(unsigned a) {
    real4 v;
#ifdef AVBDG_FP64
    asm volatile("ld.shared::cluster.v2.f64 {%0, %1}, [%2];" : "=d"(v.x), "=d"(v.y) : "r"(a));
    asm volatile("ld.shared::cluster.v2.f64 {%0, %1}, [%2];" : "=d"(v.z), "=d"(v.w) : "r"(a + 16));
#else
    asm volatile("ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(a));
#endif
    return v;
}
__device__ __forceinline__ void storeCluster(unsigned a, real4 v) {
#ifdef AVBDG_FP64
    asm volatile("st.shared::cluster.v2.f64 [%0], {%1, %2};" ::"r"(a), "d"(v.x), "d"(v.y) : "memory");
    asm volatile("st.shared::cluster.v2.f64 [%0], {%1, %2};" ::"r"(a + 16), "d"(v.z), "d"(v.w) : "memory");
#else
    asm volatile("st.shared::cluster.v4.f32 [%0], {%1, %2, %3, %4};" ::"r"(a), "f"(v.x), "f"(v.y), "f"(v.z), "f"(v.w) : "memory");
#endif
}
__device__ __forceinline__ void maxClusterInt(unsigned a, int v) {
    asm volatile("red.shared::cluster.max.s32 [%0], %1;" ::"r"(a), "r"(v) : "memory");
}
constexpr unsigned kF4 = sizeof(real4);

// Warps by role: of every four, the last is a body warp, the others contact warps.
__device__ __forceinline__ bool bodyWarp() { return ((threadIdx.x >> 5) & 3) == 3; }
__device__ __forceinline__ int contactWarp() { return static_cast<int>((threadIdx.x >> 5) - (threadIdx.x >> 7)); }
__device__ __forceinline__ int contactWarps() { return static_cast<int>(3 * (blockDim.x >> 7)); }
// Threads in body order: the body warps' first.
__device__ __forceinline__ int bodyThread() {
    const int w = bodyWarp() ? static_cast<int>(threadIdx.x >> 7) : static_cast<int>(blockDim.x >> 7) + contactWarp();
    return 32 * w + static_cast<int>(threadIdx.x & 31);
}

template <typename T>
__device__ __forceinline__ T *arrayAt(unsigned char *smem, int offset) {
    return reinterpret_cast<T *>(smem + offset);
}

__device__ __forceinline__ void putPose(real4 *r, f3 x, real mass, q4 q, f3 x0, q4 q0) {
    const f3 dl = sub(x, x0), da = qdiff(q, q0);
    const m3 rot = qmat(q);
    r[0] = f4(rot.c0, dl.x);
    r[1] = f4(rot.c1, dl.y);
    r[2] = f4(rot.c2, dl.z);
    r[kRecAng] = f4(da, 0.0f);
    r[kRecX] = f4(x, mass);
    r[kRecQ] = f4(q);
}

// What the contact terms need of a body's pose (loadPose's values).
struct PoseRec {
    f3 dLin, dAng;
    m3 rot;
};

__device__ __forceinline__ PoseRec readPose(unsigned a) {
    const real4 c0 = loadCluster(a), c1 = loadCluster(a + kF4), c2 = loadCluster(a + 2 * kF4), e = loadCluster(a + kRecAng * kF4);
    return PoseRec{f3{c0.w, c1.w, c2.w}, xyz(e), m3{xyz(c0), xyz(c1), xyz(c2)}};
}

// ---- contact phases ----

enum : int { kStampsOverflow, kStampsMixed, kDual, kDualStamps };

// Side groups 2-6 of a stamp record: fw.z, the angular block, its right-hand side, the cross block.
__device__ __forceinline__ void putSide(real4 *row, const SideTerms &t, real fwz) {
    row[0] = mk4(fwz, t.h[0], t.h[1], t.h[2]);
    row[1] = mk4(t.h[3], t.h[4], t.h[5], t.rc.x);
    row[2] = mk4(t.rc.y, t.rc.z, t.rs.c0.x, t.rs.c0.y);
    row[3] = mk4(t.rs.c0.z, t.rs.c1.x, t.rs.c1.y, t.rs.c1.z);
    row[4] = mk4(t.rs.c2.x, t.rs.c2.y, t.rs.c2.z, 0.0f);
}

// Sides of a manifold that take stamps in a phase.
__device__ __forceinline__ int stampSides(int flags, int mode) {
    const bool mixed = (flags & kMfMixed) != 0;
    if (mode == kDual || mixed != (mode == kStampsMixed))
        return 0;
    if (mode == kDualStamps && !(flags & kMfAwake))
        return 0;
    return flags & (kMfSideA | kMfSideB);
}

// Stamps of the manifolds with overflow sides (computeStamps), or the dual pass with or without the
// next round's stamps (dualAt): the same terms, a lane a contact. Contact state that the colour
// passes also read and write (a mixed manifold's) stays in the global arrays.
template <bool ARM, bool COLOURS>
__device__ __forceinline__ void contactPhase(const Dev &d, const StepParams &p, const World &w, unsigned char *smem, int mode,
                                             real decay) {
    const ManifoldBuf &L = d.live;
    const int lane = threadIdx.x & 31, cw = contactWarp(), warps = contactWarps(), tasks = w.tasks, mlo = w.mlo;
    const int conStride = w.conStride;
    real *rows = arrayAt<real>(smem, 0) + cw * 32 * kRowReals;
    real4 *row = reinterpret_cast<real4 *>(rows + lane * kRowReals);
    const int2 *mf = arrayAt<int2>(smem, w.mf);
    const uint4 *links = arrayAt<uint4>(smem, w.link);
    const real4 *bases = arrayAt<real4>(smem, w.basis);
    real4 *caps = arrayAt<real4>(smem, w.cap);
    const int *first = arrayAt<int>(smem, w.taskFirst);
    const uint16_t *slots = arrayAt<uint16_t>(smem, w.slots);
    unsigned char *contacts = smem + w.contacts;
    const bool update = mode == kDual || mode == kDualStamps;
    for (int task = cw; task < tasks; task += warps) {
        const int slot = 32 * task + lane;
        const int v = slots[slot];
        const int j = v >> 3, c = v & 7, m = mlo + j;
        const int flags = v != 0xffff ? mf[j].x : 0;
        const int sides = stampSides(flags, mode);
        const bool on = update ? (flags & kMfAwake) != 0 : sides != 0;
        const bool resident = !(COLOURS && (flags & kMfMixed));
        bool capture = false; // this lane takes its manifold's new capture
        f3 capA{}, capB{};
        if (on) {
            const uint4 link = links[j];
            const PoseRec A = readPose(link.x), B = readPose(link.y);
            const real4 b04 = bases[3 * j];
            const f3 r0 = xyz(b04), r1 = xyz(bases[3 * j + 1]), r2 = xyz(bases[3 * j + 2]);
            const real mu = b04.w;
            real4 *con = reinterpret_cast<real4 *>(contacts + slot * sizeof(real4));
            const auto at = [&](int k) -> real4 & { return *reinterpret_cast<real4 *>(reinterpret_cast<unsigned char *>(con) + k * conStride); };
            const int ci = COLOURS || ARM ? cslot(d, m, c) : 0;
            const real4 rA4 = at(0), rB4 = at(1);
            const f3 C0 = xyz(at(2));
            f3 k = xyz(resident ? at(3) : L.k[ci]);
            const real4 lam4 = resident ? at(4) : L.lam[ci];
            bool driftUsable = false;
            if (ARM && update) {
                const real4 cA = resident ? caps[2 * j] : L.capA[m], cB = resident ? caps[2 * j + 1] : L.capB[m];
                const bool held = resident ? cA.w != 0.0f : L.armFlag[m] != 0;
                const f3 dA = sub(A.rot.c0, xyz(cA)), dB = sub(B.rot.c0, xyz(cB));
                driftUsable = held && length2(dA) <= p.armRebuild2 && length2(dB) <= p.armRebuild2;
            }
            const auto putArms = [&](f3 a, f3 b) {
                if (resident) {
                    at(5) = f4(a, 0.0f);
                    at(6) = f4(b, 0.0f);
                } else {
                    L.armA[ci] = f4(a, 0.0f);
                    L.armB[ci] = f4(b, 0.0f);
                }
            };
            f3 rAw, rBw;
            if (ARM && driftUsable) {
                rAw = xyz(resident ? at(5) : L.armA[ci]);
                rBw = xyz(resident ? at(6) : L.armB[ci]);
            } else {
                rAw = mul(A.rot, xyz(rA4));
                rBw = mul(B.rot, xyz(rB4));
                if (ARM)
                    putArms(rAw, rBw);
            }
            const f3 bracket = sub(add(sub(A.dLin, B.dLin), cross(A.dAng, rAw)), cross(B.dAng, rBw));
            f3 C = contactError(p, C0, bracket, r0, r1, r2);
            f3 lam = xyz(lam4);
            if (update) {
                if (decay < 1.0f)
                    k = lclampv(scale(k, decay), PENALTY_MIN, PENALTY_MAX);
                real stick = lam4.w;
                f3 F = add(cmul(k, C), lam);
                const Cone cone = clampForce(F, mu);
                lam = F;
                const real beta = p.betaLin * rA4.w;
                if (F.x < 0)
                    k.x = smin(k.x + beta * mabs(C.x), PENALTY_MAX);
                if (cone.scale <= cone.bounds) {
                    k.y = smin(k.y + beta * mabs(C.y), PENALTY_MAX);
                    k.z = smin(k.z + beta * mabs(C.z), PENALTY_MAX);
                    stick = length2d(C.y, C.z) < STICK_THRESH ? 1.0f : 0.0f;
                }
                if (resident) {
                    at(3) = f4(k, 0.0f);
                    at(4) = f4(lam, stick);
                } else {
                    L.k[ci] = f4(k, 0.0f);
                    L.lam[ci] = f4(lam, stick);
                }
            }
            if (sides) {
                if (ARM && update) {
                    // Overflow phase A precomputes with fresh arms, whatever the dual used.
                    if (driftUsable) {
                        rAw = mul(A.rot, xyz(rA4));
                        rBw = mul(B.rot, xyz(rB4));
                        const f3 bracketF = sub(add(sub(A.dLin, B.dLin), cross(A.dAng, rAw)), cross(B.dAng, rBw));
                        C = contactError(p, C0, bracketF, r0, r1, r2);
                    }
                    putArms(rAw, rBw);
                }
                f3 F = add(cmul(k, C), lam);
                clampForce(F, mu);
                real S[6];
                basisHessianD(r0, r1, r2, k, S);
                const f3 fw = add(add(scale(r0, F.x), scale(r1, F.y)), scale(r2, F.z));
                row[0] = mk4(S[0], S[1], S[2], S[3]);
                row[1] = mk4(S[4], S[5], fw.x, fw.y);
                if (sides & kMfSideA)
                    putSide(row + 2, sideTerms(S, rAw, fw), fw.z);
                if (sides & kMfSideB)
                    putSide(row + 7, sideTerms(S, rBw, fw), fw.z);
            }
            if (ARM && update && !driftUsable && c == 0) {
                capture = true;
                capA = A.rot.c0;
                capB = B.rot.c0;
            }
        }
        __syncwarp();
        if (ARM && capture) { // every lane of the manifold has read the old one
            if (resident) {
                caps[2 * j] = f4(capA, 1.0f);
                caps[2 * j + 1] = f4(capB, 0.0f);
            } else {
                L.capA[m] = f4(capA, 0.0f);
                L.capB[m] = f4(capB, 0.0f);
                L.armFlag[m] = 1;
            }
        }
        if (mode == kDual)
            continue;
        // The sums over each manifold's contacts, in contact order from zero: twelve groups a manifold.
        const int j0 = first[task], items = 12 * (first[task + 1] - j0);
        for (int i = lane; i < items; i += 32) {
            const int man = i / 12, grp = i - 12 * man;
            const int2 f = mf[j0 + man];
            const int sd = stampSides(f.x, mode);
            if (!(sd & (grp < 2 ? kMfSideA | kMfSideB : (grp < 7 ? kMfSideA : kMfSideB))))
                continue;
            const real4 *from = reinterpret_cast<const real4 *>(rows + (f.y & 31) * kRowReals) + grp;
            real4 a = mk4(0, 0, 0, 0);
            for (int k = f.x >> kMfCountShift; k > 0; k--, from += kRowReals / 4) {
                const real4 t = *from;
                a.x += t.x;
                a.y += t.y;
                a.z += t.z;
                a.w += t.w;
            }
            const uint4 link = links[j0 + man];
            const int r = grp < 7 ? grp : grp - 5;
            if (grp < 7 && (sd & kMfSideA))
                storeCluster(link.z + r * kF4, a);
            if ((grp < 2 || grp >= 7) && (sd & kMfSideB)) { // side B's right-hand sides are negated (storeStamp)
                const real s01 = r == 4 ? -1.0f : 1.0f, s23 = r == 1 ? -1.0f : 1.0f;
                storeCluster(link.w + r * kF4, mk4(a.x * (r == 2 ? -1.0f : s01), a.y * s01, a.z * s23, a.w * (r == 3 ? -1.0f : s23)));
            }
        }
        __syncwarp();
    }
}

// ---- body phases ----

// Block sum i (0..29) of a body and the stamp value it takes: the record's 27 values in order, then
// the angular block's mirrored entries (makeBlock's are not exactly symmetric).
__device__ __forceinline__ int stampIndex(int i) { return i < 27 ? i : (i == 27 ? 10 : (i == 28 ? 11 : 13)); }

__device__ __forceinline__ void putBlock(real *b, const Blk &k) {
    const real v[30] = {k.lin.c0.x, k.lin.c0.y, k.lin.c0.z, k.lin.c1.y, k.lin.c1.z, k.lin.c2.z, k.rl.x, k.rl.y, k.rl.z,
                        k.ang.c0.x, k.ang.c0.y, k.ang.c0.z, k.ang.c1.y, k.ang.c1.z, k.ang.c2.z, k.ra.x, k.ra.y, k.ra.z,
                        k.crs.c0.x, k.crs.c0.y, k.crs.c0.z, k.crs.c1.x, k.crs.c1.y, k.crs.c1.z,
                        k.crs.c2.x, k.crs.c2.y, k.crs.c2.z, k.ang.c1.x, k.ang.c2.x, k.ang.c2.y};
#pragma unroll
    for (int i = 0; i < 30; i++)
        b[i] = v[i];
}

__device__ __forceinline__ Blk getBlock(const real *b) {
    Blk k;
    k.lin = mcols(f3{b[0], b[1], b[2]}, f3{b[1], b[3], b[4]}, f3{b[2], b[4], b[5]});
    k.rl = f3{b[6], b[7], b[8]};
    k.ang = mcols(f3{b[9], b[10], b[11]}, f3{b[27], b[12], b[13]}, f3{b[28], b[29], b[14]});
    k.ra = f3{b[15], b[16], b[17]};
    k.crs = mcols(f3{b[18], b[19], b[20]}, f3{b[21], b[22], b[23]}, f3{b[24], b[25], b[26]});
    return k;
}

__device__ __forceinline__ bool overflowBody(int info) { return (info & (kBiUpdate | kBiColour)) == (kBiUpdate | kOverflowColour); }

// A body's new pose: to its record, and to the global arrays where other phases read it there.
__device__ __forceinline__ void movePose(const Dev &d, const World &w, unsigned char *smem, int i, f3 x, real mass, q4 q, bool global) {
    const real4 *con = arrayAt<real4>(smem, w.con) + kConF4 * i;
    putPose(arrayAt<real4>(smem, w.rec) + kRecF4 * i, x, mass, q, xyz(con[kConX0]), asq(con[kConQ0]));
    if (global) {
        d.x[w.b0 + i] = f4(x, mass);
        d.q[w.b0 + i] = f4(q);
    }
}

// Where the records of a body of the world (counted from its first) lie.
struct BodyPlace {
    unsigned rec, con;
};
__device__ __forceinline__ BodyPlace placeOf(const World &w, int i) {
    const int o = i / w.per, k = i - o * w.per;
    return BodyPlace{mapShared(w.rec0, o) + kF4 * kRecF4 * k, mapShared(w.con0, o) + kF4 * kConF4 * k};
}

// The blocks of the bodies to solve before their forces and manifolds (makeBlock, from the body's own
// pose): while a round's contact tasks run, the body warps already prepare the next round's.
template <bool COLOURS>
__device__ __forceinline__ void startBlocks(const StepParams &p, const World &w, unsigned char *smem) {
    const int *info = arrayAt<int>(smem, w.info);
    const int nb = w.nb, coloured = COLOURS ? w.colourAt[kMaxColours] : 0;
    for (int k = bodyThread(); k < nb + coloured; k += blockDim.x) {
        if (COLOURS && k < coloured) {
            const BodyPlace at = placeOf(w, arrayAt<uint16_t>(smem, w.colourList)[k]);
            const real4 x4 = loadCluster(at.rec + kRecX * kF4);
            putBlock(arrayAt<real>(smem, w.colourBlocks) + k * kBlkReals,
                     makeBlock(x4.w, xyz(loadCluster(at.rec + kRecMoment * kF4)), p.dtSq, xyz(x4),
                               xyz(loadCluster(at.con + kConXi * kF4)), asq(loadCluster(at.rec + kRecQ * kF4)),
                               asq(loadCluster(at.con + kConQi * kF4))));
            continue;
        }
        const int i = k - coloured;
        if (!overflowBody(info[i]))
            continue;
        const real4 *r = arrayAt<real4>(smem, w.rec) + kRecF4 * i, *con = arrayAt<real4>(smem, w.con) + kConF4 * i;
        const real4 x4 = r[kRecX];
        putBlock(arrayAt<real>(smem, w.sums) + i * kBlkReals,
                 makeBlock(x4.w, xyz(r[kRecMoment]), p.dtSq, xyz(x4), xyz(con[kConXi]), asq(r[kRecQ]), asq(con[kConQi])));
    }
}

// The forces of overflow bodies (they come first in an adjacency) onto their blocks: bodies past the
// last colour are rare.
__device__ __forceinline__ void overflowForces(const Dev &d, const StepParams &p, const World &w, unsigned char *smem) {
    const int *info = arrayAt<int>(smem, w.info), *entry = arrayAt<int>(smem, w.entry);
    const int nf = nForcesDev(d);
    for (int i = threadIdx.x; i < w.nb; i += blockDim.x) {
        if (!overflowBody(info[i]) || !(info[i] & kBiForce))
            continue;
        real *sum = arrayAt<real>(smem, w.sums) + i * kBlkReals;
        Blk blk = getBlock(sum);
        for (int e = entry[i]; e < entry[i + 1]; e++) {
            const int seq = static_cast<int>(d.adjSeq[e]);
            if (seq >= nf)
                break;
            jointStamp(d, p, nf - 1 - seq, w.b0 + i, blk);
        }
        putBlock(sum, blk);
    }
    __syncthreads();
}

// Overflow bodies of this CTA: add the stamp records, factorise, apply (solveAt). Bodies with a force
// leave their step in dLin/dAng for applyPhase.
template <bool COLOURS>
__device__ __forceinline__ void solvePhase(const Dev &d, const StepParams &p, const World &w, unsigned char *smem) {
    const int *info = arrayAt<int>(smem, w.info), *entry = arrayAt<int>(smem, w.entry);
    real *sums = arrayAt<real>(smem, w.sums);
    const int nb = w.nb, lane = threadIdx.x & 31;
    {
        const int e0 = w.e0, idx = stampIndex(lane < 30 ? lane : 0);
        const real *rec = arrayAt<real>(smem, w.stamps) + idx;
        constexpr int R = 4 * kStampF4;
        for (int i = threadIdx.x >> 5; i < nb; i += blockDim.x >> 5) {
            if (!overflowBody(info[i]) || lane >= 30)
                continue;
            int e = entry[i] - e0;
            const int e1 = entry[i + 1] - e0;
            if (COLOURS && (info[i] & kBiForce)) {
                const int nf = nForcesDev(d);
                while (e < e1 && static_cast<int>(d.adjSeq[e0 + e]) < nf)
                    e++;
            }
            real v = sums[i * kBlkReals + lane];
            const real *o = rec + e * R;
            for (; e + 4 <= e1; e += 4, o += 4 * R) {
                const real s0 = o[0], s1 = o[R], s2 = o[2 * R], s3 = o[3 * R];
                v = (((v + s0) + s1) + s2) + s3;
            }
            for (; e < e1; e++, o += R)
                v = v + *o;
            sums[i * kBlkReals + lane] = v;
        }
    }
    __syncthreads();
    for (int i = bodyThread(); i < nb; i += blockDim.x) {
        if (!overflowBody(info[i]))
            continue;
        f3 dl, da;
        if (!solveBlockFast(getBlock(sums + i * kBlkReals), dl, da)) {
            const Delta r = solveSlow(getBlock(sums + i * kBlkReals));
            dl = r.ok ? r.dl : f3{0, 0, 0};
            da = r.ok ? r.da : f3{0, 0, 0};
        }
        if (COLOURS && (info[i] & kBiForce)) {
            const int g = w.b0 + i;
            d.dLin[g] = f4(dl, 0.0f);
            d.dAng[g] = f4(da, 0.0f);
            continue;
        }
        const real4 *r = arrayAt<real4>(smem, w.rec) + kRecF4 * i;
        const real4 x4 = r[kRecX];
        movePose(d, w, smem, i, add(xyz(x4), scale(dl, p.jacobiRelax)), x4.w, qintegrate(asq(r[kRecQ]), scale(da, p.jacobiRelax)),
                 COLOURS);
    }
}

__device__ __forceinline__ void applyPhase(const Dev &d, const StepParams &p, const World &w, unsigned char *smem) {
    for (int i = threadIdx.x; i < w.nb; i += blockDim.x) {
        const int g = w.b0 + i;
        const int info = arrayAt<int>(smem, w.info)[i];
        if (!overflowBody(info) || !(info & kBiForce))
            continue;
        const real4 *r = arrayAt<real4>(smem, w.rec) + kRecF4 * i;
        const real4 x4 = r[kRecX];
        movePose(d, w, smem, i, add(xyz(x4), scale(xyz(d.dLin[g]), p.jacobiRelax)), x4.w,
                 qintegrate(asq(r[kRecQ]), scale(xyz(d.dAng[g]), p.jacobiRelax)), true);
    }
}

// ---- colours (solver_step.cpp:209-229) ----
//
// A coloured body's block is its start (startBlocks), then its forces' terms, then its manifolds', in
// adjacency order. Each is a list of terms fixed for the step: a force's parts (a ball joint's linear
// stamp, its geometric stiffness and its angular stamp; a spring; a generic joint's constraint and spring
// of each axis that has them) and a manifold side's contacts (the same terms recomputeSide adds). A
// term is a lane's work and leaves its thirty values in a row of shared memory, in order; thirty lanes
// then add the rows, a manifold's contacts summed from zero first. A colour is a chain of one body's
// latencies (poses over the cluster, a term's code, the sum, the factorisation), so its terms are sorted by
// kind, a warp to a kind, and its bodies are dealt round the CTAs (ragdolls lie side by side in a store).
// A level of 600 bodies with 114 coloured ones took 92 us a round in the separate sweep; 27k cycles (13 us)
// a colour with each body at its owner and one warp taking its kinds in turn; 16k this way, of which the
// terms take half and the factorisation a fifth.

// Kinds of terms.
enum : int { kTermContact, kTermBallLinear, kTermBallGeometric, kTermBallAngular, kTermSpring, kTermLinear, kTermAngular, kTermKinds };
// A term: its kind, force (or contact and manifold), and the records of its bodies A and B (0: none).
struct __align__(16) Term {
    int flags, id;
    unsigned recA, recB;
    int manifold, row; // row: its place in the world's list of this CTA
};
enum : int {
    kTermKind = 0xf,
    kTermFirst = 16, kTermLast = 32, // of a manifold's contacts
    kTermSideB = 64,                 // the body is B
    kTermDualArms = 128,             // arm cache: after a dual, the first touch takes the arms it left
    kTermPart = 8                    // (shift) a generic joint's axis 0-2, + 4 for its spring
};
constexpr int kRowMark = 51; // place of the flags in a row

struct TermPose {
    f3 x;
    q4 q;
};
__device__ __forceinline__ TermPose termPose(unsigned rec) {
    if (!rec)
        return TermPose{f3{0, 0, 0}, q4{0.0f, 0.0f, 0.0f, 1.0f}};
    return TermPose{xyz(loadCluster(rec + kRecX * kF4)), asq(loadCluster(rec + kRecQ * kF4))};
}

// ballStamp's parts (joint.cpp:80-175).
// What a part does not touch stays -0, which no sum feels.
__device__ __forceinline__ void ballPart(const Dev &d, const StepParams &p, int f, int kind, bool isA, const Term &t, Blk &k) {
    const real4 par = d.fPar[f];
    const TermPose A = termPose(t.recA), B = termPose(t.recB);
    if (kind == kTermBallAngular) {
        const f3 ka = xyz(d.fKA[f]);
        if (!(length2(ka) > 0))
            return;
        const m3 K = mdiag(ka.x, ka.y, ka.z);
        f3 C = scale(qdiff(A.q, B.q), par.w);
        if (isinf(par.y))
            C = sub(C, scale(xyz(d.fC0A[f]), p.alpha));
        const f3 F = add(mul(K, C), xyz(d.fLA[f]));
        const m3 base = isA ? mdiag(1, 1, 1) : mcols(f3{0, 0, 0}, f3{0, -1, 0}, f3{0, 0, -1});
        const m3 jAng = mscale(base, par.w);
        k.ang = mul(mul(transpose(jAng), K), jAng);
        k.ra = mul(transpose(jAng), F);
        return;
    }
    const f3 kl = xyz(d.fKL[f]);
    if (!(length2(kl) > 0))
        return;
    const m3 K = mdiag(kl.x, kl.y, kl.z);
    const f3 rA = xyz(d.fRA[f]), rB = xyz(d.fRB[f]);
    const f3 rotA = qrot(A.q, rA), rotB = qrot(B.q, rB);
    f3 C = sub(t.recA ? add(A.x, rotA) : rA, add(B.x, rotB));
    if (isinf(par.x))
        C = sub(C, scale(xyz(d.fC0L[f]), p.alpha));
    const f3 F = add(mul(K, C), xyz(d.fLL[f]));
    if (kind == kTermBallGeometric) {
        const f3 rr = isA ? rotA : neg(rotB);
        const m3 H = madd(madd(mscale(geometricStiffness(0, rr), F.x), mscale(geometricStiffness(1, rr), F.y)),
                          mscale(geometricStiffness(2, rr), F.z));
        k.ang = mdiag(H.c0.x, H.c1.y, H.c2.z);
        return;
    }
    const m3 I = mdiag(1, 1, 1);
    const m3 jLin = isA ? I : mneg(I);
    const f3 r = isA ? neg(rotA) : rotB;
    const m3 jAng = mcols(f3{0, r.z, -r.y}, f3{-r.z, 0, r.x}, f3{r.y, -r.x, 0});
    const m3 jLinT = transpose(jLin);
    const m3 jAngT = transpose(jAng);
    const m3 jAngTk = mul(jAngT, K);
    k.lin = mul(mul(jLinT, K), jLin);
    k.ang = mul(jAngTk, jAng);
    k.crs = mul(jAngTk, jLin);
    k.rl = mul(jLinT, F);
    k.ra = mul(jAngT, F);
}

// springStamp (spring.cpp:31-70).
__device__ __forceinline__ void springPart(const Dev &d, int f, bool isA, const Term &t, Blk &k) {
    const real4 par = d.fPar[f];
    const TermPose A = termPose(t.recA), B = termPose(t.recB);
    const f3 rA = qrot(A.q, xyz(d.fRA[f])), rB = qrot(B.q, xyz(d.fRB[f]));
    const f3 dv = sub(add(A.x, rA), add(B.x, rB));
    const real len = length(dv);
    if (len <= 1.0e-6f)
        return;
    const f3 n = divs(dv, len);
    const real C = len - par.y;
    const real force = par.x * C;
    const f3 jLin = isA ? n : neg(n);
    const f3 jAng = isA ? cross(rA, n) : neg(cross(rB, n));
    k.lin = mscale(outerprod(jLin, jLin), par.x);
    k.ang = mscale(outerprod(jAng, jAng), par.x);
    k.crs = mscale(outerprod(jAng, jLin), par.x);
    k.rl = scale(jLin, force);
    k.ra = scale(jAng, force);
}

// One axis' constraint or spring of a generic joint (genericStamp, stampAxis).
template <bool angular>
__device__ __forceinline__ void genericPart(const Dev &d, const StepParams &p, int f, int part, bool isA, const Term &t, Blk &k) {
    const int i = part & 3;
    const bool spring = (part & 4) != 0;
    const int2 ab = d.fAB[f];
    const TermPose A = termPose(t.recA), B = termPose(t.recB);
    const real sign = isA ? 1.0f : -1.0f;
    const f3 rA = xyz(d.fRA[f]), rAWorld = qrot(A.q, rA), rBWorld = qrot(B.q, xyz(d.fRB[f]));
    const f3 axis = qrot(A.q, unitAxis(i));
    const GAxis ax = loadAxis(d, f, angular ? 3 + i : i);
    f3 jLin{0, 0, 0}, jAng;
    real value;
    if (angular) {
        real ang[3];
        genericAnglesOf(d, f, A.q, B.q, ang);
        value = i == 0 ? ang[0] : (i == 1 ? ang[1] : ang[2]);
        jAng = scale(axis, sign);
    } else {
        const f3 anchorA = t.recA ? add(A.x, rAWorld) : rA;
        value = at(qrot(qconj(A.q), sub(anchorA, add(B.x, rBWorld))), i);
        jLin = scale(axis, sign);
        jAng = cross(isA ? rAWorld : rBWorld, jLin);
    }
    real stiffness, F;
    if (spring) {
        const f3 wA = ab.x >= 0 ? xyz(d.w[ab.x]) : f3{0, 0, 0}, wB = xyz(d.w[ab.y]);
        real rate;
        if (angular) {
            rate = dot(sub(wA, wB), axis);
        } else {
            const f3 vA = ab.x >= 0 ? add(xyz(d.v[ab.x]), cross(wA, rAWorld)) : f3{0, 0, 0};
            const f3 vB = add(xyz(d.v[ab.y]), cross(wB, rBWorld));
            rate = dot(sub(vA, vB), axis);
        }
        const real Cs = value - ax.springEq;
        F = ax.springK * Cs - ax.springDamp * rate;
        stiffness = ax.springK;
    } else {
        real C;
        if (!axisForce(ax, value, p.alpha, C, F))
            return;
        stiffness = ax.penalty;
    }
    k.lin = mscale(outerprod(jLin, jLin), stiffness);
    k.ang = mscale(outerprod(jAng, jAng), stiffness);
    k.crs = mscale(outerprod(jAng, jLin), stiffness);
    k.rl = scale(jLin, F);
    k.ra = scale(jAng, F);
}

// A contact's terms of one side at the current poses (recomputeSide): its 27 values in record order.
template <bool ARM>
__device__ __forceinline__ void contactTerm(const Dev &d, const StepParams &p, const Term &t, int armsFromDual, real4 *row) {
    const ManifoldBuf &L = d.live;
    const int m = t.manifold, ci = t.id;
    const real4 rA4 = L.rA[ci], rB4 = L.rB[ci], b04 = L.b0[m];
    const f3 r0 = xyz(b04), r1 = xyz(L.b1[m]), r2 = xyz(L.b2[m]), C0 = xyz(L.C0[ci]), k = xyz(L.k[ci]), lam = xyz(L.lam[ci]);
    const PoseRec A = readPose(t.recA), B = readPose(t.recB);
    f3 rAw, rBw;
    if (ARM && armsFromDual && (t.flags & kTermDualArms)) {
        rAw = xyz(L.armA[ci]);
        rBw = xyz(L.armB[ci]);
    } else {
        rAw = mul(A.rot, xyz(rA4));
        rBw = mul(B.rot, xyz(rB4));
        if (ARM) {
            L.armA[ci] = f4(rAw, 0.0f);
            L.armB[ci] = f4(rBw, 0.0f);
        }
    }
    const f3 bracket = sub(add(sub(A.dLin, B.dLin), cross(A.dAng, rAw)), cross(B.dAng, rBw));
    const f3 C = contactError(p, C0, bracket, r0, r1, r2);
    f3 F = add(cmul(k, C), lam);
    clampForce(F, b04.w);
    real S[6];
    basisHessianD(r0, r1, r2, k, S);
    const f3 fw = add(add(scale(r0, F.x), scale(r1, F.y)), scale(r2, F.z));
    row[0] = mk4(S[0], S[1], S[2], S[3]);
    row[1] = mk4(S[4], S[5], fw.x, fw.y);
    const SideTerms side = sideTerms(S, t.flags & kTermSideB ? rBw : rAw, fw);
    putSide(row + 2, side, fw.z);
    real *r = reinterpret_cast<real *>(row);
    r[27] = side.h[1]; // the angular block's mirrored entries
    r[28] = side.h[2];
    r[29] = side.h[4];
}

// The rows a pass holds: a colour's terms in the CTA are taken in groups of this many.
__device__ __forceinline__ int passRows() { return 32 * contactWarps(); }

template <bool ARM>
__device__ __forceinline__ void colourPhase(const Dev &d, const StepParams &p, const World &w, unsigned char *smem, int colours,
                                            int armsFromDual, real (*carries)[32]) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, warps = blockDim.x >> 5, group = passRows();
    real *rows = arrayAt<real>(smem, 0);
    const int *termFirst = arrayAt<int>(smem, w.termFirst);
    const Term *terms = arrayAt<Term>(smem, w.terms);
    const uint16_t *order = arrayAt<uint16_t>(smem, w.termOrder);
    const bool rhs = (lane >= 6 && lane < 9) || (lane >= 15 && lane < 18);
    for (int c = 0; c < kMaxColours; c++) {
        if (!((colours >> c) & 1))
            continue;
        const int k0 = w.colourAt[c], k1 = w.colourAt[c + 1];
        const int first = k0 < k1 ? termFirst[k0] : 0, last = k0 < k1 ? termFirst[k1] : 0;
        for (int from = first, pass = 0; k0 < k1 && (pass == 0 || from < last); from += group, pass++) {
            const int to = min(from + group, last);
            // A body that goes on hands its sums to the next pass. In one pass the body that came over reads the last
            // one's while another warp may write the next one's: two in turn.
            real *carried = carries[(pass + 1) & 1], *carry = carries[pass & 1];
            // Terms: warps take up to 32 of a kind.
            const uint16_t *kinds = arrayAt<uint16_t>(smem, w.termKinds) + (w.groupAt[c] + pass) * (kTermKinds + 1);
            for (int task = warp, kind = 0, before = 0; kind < kTermKinds; kind++) {
                const int a = kinds[kind], n = kinds[kind + 1] - a, tasks = (n + 31) >> 5;
                for (; task < before + tasks; task += warps) {
                    const int at = 32 * (task - before) + lane;
                    if (at >= n)
                        continue;
                    const Term t = terms[order[from + a + at]];
                    real *row = rows + (t.row - from) * kRowReals;
                    const bool isA = !(t.flags & kTermSideB);
                    if (kind == kTermContact) {
                        contactTerm<ARM>(d, p, t, armsFromDual, reinterpret_cast<real4 *>(row));
                    } else {
                        Blk b;
                        const f3 none{-0.0f, -0.0f, -0.0f};
                        b.lin = b.ang = b.crs = mcols(none, none, none);
                        b.rl = b.ra = none;
                        if (kind == kTermSpring)
                            springPart(d, t.id, isA, t, b);
                        else if (kind == kTermLinear)
                            genericPart<false>(d, p, t.id, t.flags >> kTermPart, isA, t, b);
                        else if (kind == kTermAngular)
                            genericPart<true>(d, p, t.id, t.flags >> kTermPart, isA, t, b);
                        else
                            ballPart(d, p, t.id, kind, isA, t, b);
                        putBlock(row, b);
                    }
                    *reinterpret_cast<int *>(row + kRowMark) = t.flags;
                }
                before += tasks;
            }
            __syncthreads();
            // Sums, a warp a body; a body whose terms go on in the next group leaves its sums for it.
            for (int k = k0 + warp; k < k1; k += warps) {
                const int t0 = termFirst[k], t1 = termFirst[k + 1];
                const bool done = t1 <= from + group && (t1 > from || pass == 0);
                if (!done && !(t0 < to && t1 > from))
                    continue;
                real *sums = arrayAt<real>(smem, w.colourBlocks) + k * kBlkReals;
                real v = lane < 30 ? sums[lane] : 0.0f, acc = t0 < from ? carried[lane] : 0.0f;
                const real *r = rows + (max(t0, from) - from) * kRowReals, *end = rows + (min(t1, to) - from) * kRowReals;
#pragma unroll 4
                for (; r < end; r += kRowReals) {
                    const int mark = *reinterpret_cast<const int *>(r + kRowMark);
                    // A force's term alone (-0 + x is x), a manifold's contacts from zero.
                    acc = (mark & kTermFirst ? (mark & kTermKind ? -0.0f : 0.0f) : acc) + r[lane];
                    const real next = v + (rhs && (mark & (kTermKind | kTermSideB)) == kTermSideB ? -acc : acc);
                    v = mark & kTermLast ? next : v;
                }
                if (lane < 30)
                    sums[lane] = v;
                if (!done) {
                    carry[lane] = acc;
                    continue;
                }
                __syncwarp();
                if (lane == 0) {
                    const int i = arrayAt<uint16_t>(smem, w.colourList)[k];
                    const BodyPlace at = placeOf(w, i);
                    const real4 x4 = loadCluster(at.rec + kRecX * kF4), q4v = loadCluster(at.rec + kRecQ * kF4);
                    const real4 x0 = loadCluster(at.con + kConX0 * kF4), q0 = loadCluster(at.con + kConQ0 * kF4);
                    f3 dl, da;
                    if (!solveBlockFast(getBlock(sums), dl, da)) {
                        const Delta s = solveSlow(getBlock(sums));
                        dl = s.ok ? s.dl : f3{0, 0, 0};
                        da = s.ok ? s.da : f3{0, 0, 0};
                    }
                    const f3 x = add(xyz(x4), dl);
                    const q4 q = qintegrate(asq(q4v), da);
                    real4 rec[kRecMoment];
                    putPose(rec, x, x4.w, q, xyz(x0), asq(q0));
#pragma unroll
                    for (int j = 0; j < kRecMoment; j++)
                        storeCluster(at.rec + j * kF4, rec[j]);
                    d.x[w.base + i] = rec[kRecX];
                    d.q[w.base + i] = rec[kRecQ];
                }
            }
            if (to < last)
                __syncthreads();
        }
        clusterSync(w.size);
    }
}

// A force's dual pass by eight lanes: a generic joint's axes one each, any other force by the first. The
// CTAs' last body warps take four forces each first: the first ones start the next round's blocks.
__device__ __forceinline__ void forceDuals(const Dev &d, const StepParams &p, const World &w) {
    const int last = static_cast<int>(blockDim.x >> 7) - 1 - static_cast<int>(threadIdx.x >> 7), axis = threadIdx.x & 7;
    const int first = w.f0 + 4 * (w.rank + w.size * last) + (static_cast<int>(threadIdx.x & 31) >> 3);
    for (int f = first; f < w.f1; f += 4 * w.size * static_cast<int>(blockDim.x >> 7)) {
        if (d.fKind[f] == kForceGeneric) {
            if (axis < 6)
                genericDualAxis(d, p, f, axis);
        } else if (axis == 0) {
            forceDualAt(d, p, f);
        }
    }
}

// The terms of an adjacency entry of coloured body `g`, counted and given to `put`.
template <typename RecOf, typename Put>
__device__ __forceinline__ int entryTerms(const Dev &d, int g, int e, RecOf recOf, Put put) {
    const int nf = nForcesDev(d), seq = static_cast<int>(d.adjSeq[e]), v = d.adjInfo[e], o = adjInfoOther(v), side = adjInfoSide(v);
    const unsigned own = recOf(g), other = o >= 0 ? recOf(o) : 0;
    Term t{side ? kTermSideB : 0, 0, side ? other : own, side ? own : other, 0, 0};
    int n = 0;
    const auto add = [&](int flags) {
        Term a = t;
        a.flags |= flags;
        put(n++, a);
    };
    if (seq >= nf) {
        t.manifold = seq - nf;
        const int count = d.live.count[t.manifold];
        if (!(o >= 0 && inUpdate(d, o) && d.colour[o] < d.colour[g]))
            t.flags |= kTermDualArms;
        for (int c = 0; c < count; c++) {
            t.id = cslot(d, t.manifold, c);
            add(kTermContact | (c == 0 ? kTermFirst : 0) | (c + 1 == count ? kTermLast : 0));
        }
        return n;
    }
    t.id = nf - 1 - seq;
    t.flags |= kTermFirst | kTermLast;
    const int kind = d.fKind[t.id];
    if (kind == kForceBall) {
        add(kTermBallLinear);
        add(kTermBallGeometric);
        add(kTermBallAngular);
    } else if (kind == kForceSpring) {
        add(kTermSpring);
    } else if (kind == kForceGeneric) {
        for (int i = 0; i < 6; i++) { // axis i / 2, linear then angular
            const GAxis ax = loadAxis(d, t.id, (i >> 1) + 3 * (i & 1));
            const int flags = (i & 1 ? kTermAngular : kTermLinear) | (i >> 1) << kTermPart;
            if (ax.mode == kAxisLocked || ax.mode == kAxisLimited)
                add(flags);
            if (ax.springK > 0.0f)
                add(flags | 4 << kTermPart);
        }
    }
    return n;
}

// A body's entries by a warp: `put(n, term)` numbers its terms in order; their count.
template <typename RecOf, typename Put>
__device__ __forceinline__ int bodyTerms(const Dev &d, int g, RecOf recOf, Put put) {
    const int lane = threadIdx.x & 31, e1 = d.adjStart[g + 1];
    int n = 0;
    for (int e0 = d.adjStart[g]; e0 < e1; e0 += 32) {
        const int mine = e0 + lane < e1 ? entryTerms(d, g, e0 + lane, [](int) { return 0u; }, [](int, const Term &) {}) : 0;
        int upTo = mine;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int y = __shfl_up_sync(0xffffffffu, upTo, o);
            if (lane >= o)
                upTo += y;
        }
        const int from = n + upTo - mine;
        if (e0 + lane < e1)
            entryTerms(d, g, e0 + lane, recOf, [&](int k, const Term &t) { put(from + k, t); });
        n += __shfl_sync(0xffffffffu, upTo, 31);
    }
    return n;
}

// The first force whose body B is in slot `g` or later (forces lie in world order, as bodies do).
__device__ __forceinline__ int firstForce(const Dev &d, int nf, int g) {
    int lo = 0, hi = nf;
    while (lo < hi) {
        const int mid = (lo + hi) >> 1;
        if (d.fAB[mid].y < g)
            lo = mid + 1;
        else
            hi = mid;
    }
    return lo;
}

// ---- brake (solver_projection.cpp:96-167) ----

// A candidate's predecessor on a movable body is the candidate before it among the body's manifolds
// (live order, after its forces); candidates are in mSpec, their predecessors start at none.
__device__ __forceinline__ void brakePredecessors(const Dev &d, int m0, int g) {
    const int nf = nForcesDev(d);
    int last = -1;
    const int e1 = d.adjStart[g + 1];
    for (int e = d.adjStart[g]; e < e1; e += 4) {
        int m[4], spec[4], side[4];
#pragma unroll
        for (int k = 0; k < 4; k++) {
            m[k] = e + k < e1 ? static_cast<int>(d.adjSeq[e + k]) - nf : -1;
            side[k] = e + k < e1 ? adjInfoSide(d.adjInfo[e + k]) : 0;
        }
#pragma unroll
        for (int k = 0; k < 4; k++)
            spec[k] = m[k] >= 0 ? d.mSpec[m[k]] : 0;
#pragma unroll
        for (int k = 0; k < 4; k++)
            if (spec[k]) {
                reinterpret_cast<int *>(d.specPred)[2 * static_cast<size_t>(m[k]) + side[k]] = last;
                last = m[k] - m0;
            }
    }
}

__device__ __forceinline__ f3 xorLane(f3 v) {
    return f3{__shfl_xor_sync(0xffffffffu, v.x, 1), __shfl_xor_sync(0xffffffffu, v.y, 1), __shfl_xor_sync(0xffffffffu, v.z, 1)};
}

// One side's response to a patch: the torque axis' compliance and the angular response per unit of
// impulse.
__device__ __forceinline__ real patchResponse(f3 I0, q4 q, f3 patch, real invN, f3 nrm, f3 &response) {
    const Inertia I = inertia(I0);
    const f3 t = qrot(qconj(q), cross(scale(patch, invN), nrm));
    response = angularResponse(I, q, t);
    return angularCompliance(I, t);
}

// A candidate's part of the sweep that does not depend on the velocities, found before it and kept in
// the staging buffer, which is free after the compaction: per contact the arm of each side (rA, rB; w
// the target velocity -gap / window), and for all open contacts braking together, as they nearly always
// do if any does: b0 = normal, K; b1 = side A's angular response per unit of impulse, 1 / contacts;
// b2 = side B's response, the open contacts' bits; C0 of contact 0 = the inverse masses, then each
// side's axis locks, plus kBrakeMoves where it is movable. (Small whole numbers are exact.)
constexpr int kBrakeMoves = 65536;

__device__ __forceinline__ real brakeSideFlags(const Dev &d, int g) {
    return static_cast<real>((d.meta[g].w & 0xffff) + (movable(d, g) ? kBrakeMoves : 0));
}

// Both sides of manifold m by one thread.
__device__ __forceinline__ void brakePrepareAt(const Dev &d, int m, real window) {
    const ManifoldBuf &L = d.live, &S = d.stage;
    const int2 ab = L.ab[m];
    const real4 xa4 = d.x[ab.x], xb4 = d.x[ab.y];
    const q4 qa = asq(d.q[ab.x]), qb = asq(d.q[ab.y]);
    const bool moveA = movable(d, ab.x), moveB = movable(d, ab.y);
    const real massA = moveA ? 1.0f / xa4.w : 0.0f, massB = moveB ? 1.0f / xb4.w : 0.0f;
    const f3 nrm = xyz(L.b0[m]);
    f3 patchA{0, 0, 0}, patchB{0, 0, 0}, responseA{0, 0, 0}, responseB{0, 0, 0};
    int open = 0;
    for (int k = 0; k < L.count[m]; k++) {
        const int ci = cslot(d, m, k);
        const f3 rA = qrot(qa, xyz(L.rA[ci])), rB = qrot(qb, xyz(L.rB[ci]));
        const real gap = dot(nrm, sub(add(xyz(xa4), rA), add(xyz(xb4), rB)));
        S.rA[ci] = f4(rA, -gap / window);
        S.rB[ci] = f4(rB, -gap / window);
        if (gap > 0.0f) {
            patchA = add(patchA, rA);
            patchB = add(patchB, rB);
            open |= 1 << k;
        }
    }
    const real invN = 1.0f / static_cast<real>(__popc(open));
    const real cA = moveA ? patchResponse(xyz(d.moment[ab.x]), qa, patchA, invN, nrm, responseA) : 0.0f;
    const real cB = moveB ? patchResponse(xyz(d.moment[ab.y]), qb, patchB, invN, nrm, responseB) : 0.0f;
    S.b0[m] = f4(nrm, massA + massB + cA + cB);
    S.b1[m] = f4(responseA, invN);
    S.b2[m] = f4(responseB, static_cast<real>(open));
    S.C0[cslot(d, m, 0)] = mk4(massA, massB, brakeSideFlags(d, ab.x), brakeSideFlags(d, ab.y));
}

constexpr int kBrakeLevels = 1024; // deeper dependency chains leave the candidates in live order

// The brake's Gauss-Seidel sweep over manifolds [m0, m0 + n) in one CTA, by levels. A candidate's level
// is one more than its deepest predecessor's; candidates of a level share no movable body, so they
// brake together, with a block barrier between levels. They are sorted by level, so a level costs only
// the warps it fills. Two lanes a candidate, one a side, half a block of candidates at a time; what
// does not depend on the velocities is prepared (brakePrepareAt). The world's velocities are in `vel`
// (six a body), an int per manifold in `level`. A candidate that finds a predecessor without a level
// more than waitLimit times reports the timeout and the sweep is left out.
// Longest chains of the timed worlds: 4 (420-box walls), 23 (1653-box pile), 53 candidates (a wall
// dropped on a wall). Taken as a dataflow instead, in which every lane ran when its predecessors were
// done, a warp made a pass for nearly every lane: 43, 170 and 150 us a sweep.
// `pose(g, q, moment)` reads a body's orientation and moment.
template <typename PoseOf>
__device__ __forceinline__ void brakeSweep(const Dev &d, int base, int cnt, int m0, int n, real *vel, int *level, PoseOf pose) {
    __shared__ int counts[kMaxWorldThreads / 32], levelAt[kBrakeLevels], deepestLevel, stopped;
    const ManifoldBuf &L = d.live, &S = d.stage;
    const int lane = threadIdx.x & 31;
    // The candidates in live order.
    int *list = d.specList + m0, *sorted = d.pairValid + m0;
    int total = 0;
    for (int first = 0; first < n; first += blockDim.x) {
        const int ml = first + threadIdx.x;
        const bool spec = ml < n && d.mSpec[m0 + ml];
        if (ml < n)
            level[ml] = 0;
        const unsigned hits = __ballot_sync(0xffffffffu, spec);
        if (lane == 0)
            counts[threadIdx.x >> 5] = __popc(hits);
        __syncthreads();
        int before = 0, all = 0;
        for (int k = 0; k < static_cast<int>(blockDim.x >> 5); k++) {
            before += k < static_cast<int>(threadIdx.x >> 5) ? counts[k] : 0;
            all += counts[k];
        }
        if (spec)
            list[total + before + __popc(hits & ((1u << lane) - 1u))] = ml;
        total += all;
        __syncthreads();
    }
    if (total == 0)
        return;
    for (int i = threadIdx.x; i < cnt; i += blockDim.x) {
        const real4 v = d.v[base + i], w = d.w[base + i];
        real *o = vel + kVelReals * i;
        o[0] = v.x, o[1] = v.y, o[2] = v.z, o[3] = w.x, o[4] = w.y, o[5] = w.z;
    }
    for (int k = threadIdx.x; k < kBrakeLevels; k += blockDim.x)
        levelAt[k] = 0;
    if (threadIdx.x == 0)
        deepestLevel = stopped = 0;
    __syncthreads();
    // Levels as a dataflow: a candidate settles once its predecessors have.
    {
        volatile int *settled = level;
        constexpr int kHeld = 2; // candidates a thread holds in registers
        int held[kHeld];
        int2 pred[kHeld];
#pragma unroll
        for (int c = 0; c < kHeld; c++) {
            const int k = threadIdx.x + c * blockDim.x;
            held[c] = k < total ? list[k] : -1;
            pred[c] = held[c] >= 0 ? d.specPred[m0 + held[c]] : make_int2(-1, -1);
        }
        int mine = 0;
        const auto settle = [&](int ml, int2 p) {
            const int a = p.x < 0 ? 0 : settled[p.x], b = p.y < 0 ? 0 : settled[p.y];
            if ((p.x >= 0 && !a) || (p.y >= 0 && !b))
                return false;
            settled[ml] = 1 + max(a, b);
            mine = max(mine, 1 + max(a, b));
            return true;
        };
        long long passed = 0;
        int turns = 0;
        bool open = true, late = false;
        while (__any_sync(0xffffffffu, open)) {
            open = false;
#pragma unroll
            for (int c = 0; c < kHeld; c++)
                if (held[c] >= 0) {
                    if (settle(held[c], pred[c]))
                        held[c] = -1;
                    else
                        open = true;
                }
            for (int k = threadIdx.x + kHeld * blockDim.x; k < total; k += blockDim.x)
                if (!settled[list[k]])
                    open = !settle(list[k], d.specPred[m0 + list[k]]) || open;
            if (open && ++passed > d.waitLimit) {
                late = true;
                open = false;
            }
            if (late)
                stopped = 1;
            if ((++turns & 255) == 0 && *const_cast<volatile int *>(&stopped))
                open = false;
        }
        if (late)
            atomicOr(d.ctr + C_ERRORS, kErrBrakeTimeout);
        if (__syncthreads_or(late))
            return;
        atomicMax(&deepestLevel, mine);
    }
    __syncthreads();
    const int deepest = deepestLevel;
    const bool bySort = deepest < kBrakeLevels;
    if (bySort) {
        for (int k = threadIdx.x; k < total; k += blockDim.x)
            atomicAdd(&levelAt[level[list[k]]], 1);
        __syncthreads();
        if (threadIdx.x < 32) { // first place of each level
            int run = 0;
            for (int k0 = 0; k0 <= deepest; k0 += 32) {
                const int c = k0 + lane <= deepest ? levelAt[k0 + lane] : 0;
                int upTo = c;
#pragma unroll
                for (int o = 1; o < 32; o <<= 1) {
                    const int y = __shfl_up_sync(0xffffffffu, upTo, o);
                    if (lane >= o)
                        upTo += y;
                }
                if (k0 + lane <= deepest)
                    levelAt[k0 + lane] = run + upTo - c;
                run += __shfl_sync(0xffffffffu, upTo, 31);
            }
        }
        __syncthreads();
        for (int k = threadIdx.x; k < total; k += blockDim.x) {
            const int ml = list[k];
            sorted[atomicAdd(&levelAt[level[ml]], 1)] = ml;
        }
        __syncthreads();
    }
    const int *order = bySort ? sorted : list;
    const int side = threadIdx.x & 1, half = static_cast<int>(blockDim.x) / 2;
    for (int first = 0; first < total; first += half) {
        const int k0 = first + static_cast<int>(threadIdx.x >> 1);
        int g = base, locks = 0, open = 0, turn = 0;
        bool move = false;
        real invMass = 0.0f, invN = 0.0f, K = 0.0f;
        f3 nrm{0, 0, 0}, response{0, 0, 0}, arm[kMaxContacts];
        real target[kMaxContacts];
        if (k0 < total) {
            const int ml = order[k0], m = m0 + ml;
            turn = level[ml];
            const int2 ab = L.ab[m];
            const real4 b0 = S.b0[m], b1 = S.b1[m], b2 = S.b2[m], sides = S.C0[cslot(d, m, 0)];
            const real4 *arms = side == 0 ? S.rA : S.rB;
#pragma unroll
            for (int k = 0; k < 4; k++) { // (those past the manifold's contacts are not open)
                const real4 a = arms[cslot(d, m, k)];
                arm[k] = xyz(a);
                target[k] = a.w;
            }
            nrm = xyz(b0);
            K = b0.w;
            invN = b1.w;
            response = side == 0 ? xyz(b1) : xyz(b2);
            open = static_cast<int>(b2.w);
            invMass = side == 0 ? sides.x : sides.y;
            locks = static_cast<int>(side == 0 ? sides.z : sides.w);
            move = locks >= kBrakeMoves;
            g = side == 0 ? ab.x : ab.y;
#pragma unroll
            for (int k = 4; k < kMaxContacts; k++)
                if ((open >> k) & 1) {
                    const real4 a = arms[cslot(d, m, k)];
                    arm[k] = xyz(a);
                    target[k] = a.w;
                }
        }
        // Side B sees the pair's differences and the normal both negated: the same products.
        const f3 along = side == 0 ? nrm : neg(nrm);
        const int most = __reduce_max_sync(0xffffffffu, 32 - __clz(open));
        const int from = bySort ? level[order[first]] : 1, to = bySort ? level[order[min(first + half, total) - 1]] : deepest;
        for (int now = from; now <= to; now++) {
            if (__any_sync(0xffffffffu, turn == now)) {
                real *at = vel + kVelReals * (g - base);
                const f3 v{at[0], at[1], at[2]}, w{at[3], at[4], at[5]};
                real velErr = 0.0f;
                int braked = 0;
#pragma unroll
                for (int k = 0; k < kMaxContacts; k++)
                    if (k < most) {
                        const f3 own = add(v, cross(w, arm[k]));
                        const real vn = dot(sub(own, xorLane(own)), along);
                        if (((open >> k) & 1) && vn < target[k]) {
                            velErr += target[k] - vn;
                            braked |= 1 << k;
                        }
                    }
                const bool some = turn == now && braked != 0 && braked != open; // not all of the open contacts
                if (__any_sync(0xffffffffu, some)) {
                    f3 sum{0, 0, 0};
#pragma unroll
                    for (int k = 0; k < kMaxContacts; k++)
                        if ((braked >> k) & 1)
                            sum = add(sum, arm[k]);
                    real compliance = 0.0f;
                    if (some) {
                        invN = 1.0f / static_cast<real>(__popc(braked));
                        if (move) {
                            q4 q;
                            f3 moment;
                            pose(g, q, moment);
                            compliance = patchResponse(moment, q, sum, invN, nrm, response);
                        }
                    }
                    const real oMass = __shfl_xor_sync(0xffffffffu, invMass, 1), oComp = __shfl_xor_sync(0xffffffffu, compliance, 1);
                    if (some)
                        K = side == 0 ? invMass + oMass + compliance + oComp : oMass + invMass + oComp + compliance;
                }
                if (turn == now && braked && move) {
                    const real j = velErr * invN / K;
                    f3 dv = scale(nrm, invMass * j), dw = scale(response, j);
                    maskLocked(locks & 0xff, dv);
                    maskLocked((locks >> 8) & 0xff, dw);
                    const f3 nv = side == 0 ? add(v, dv) : sub(v, dv), nw = side == 0 ? add(w, dw) : sub(w, dw);
                    at[0] = nv.x, at[1] = nv.y, at[2] = nv.z, at[3] = nw.x, at[4] = nw.y, at[5] = nw.z;
                }
            }
            __syncthreads();
        }
    }
    for (int i = threadIdx.x; i < cnt; i += blockDim.x) {
        const int g = base + i;
        if (!movable(d, g))
            continue;
        const real *o = vel + kVelReals * i;
        d.v[g] = mk4(o[0], o[1], o[2], d.v[g].w);
        d.w[g] = mk4(o[3], o[4], o[5], 0.0f);
    }
}

__device__ __forceinline__ void brakePhase(const Dev &d, const World &w, unsigned char *smem, real window) {
    const ManifoldBuf &S = d.stage;
    const int lane = threadIdx.x & 31;
    const int2 *mf = arrayAt<int2>(smem, w.mf);
    real *rows = arrayAt<real>(smem, 0) + contactWarp() * 32 * kRowReals;
    real4 *row = reinterpret_cast<real4 *>(rows + lane * kRowReals);
    if (!bodyWarp())
        for (int task = contactWarp(); task < w.tasks; task += contactWarps()) {
            const int slot = 32 * task + lane, v = arrayAt<uint16_t>(smem, w.slots)[slot], j = v >> 3;
            bool open = false;
            if (v != 0xffff && mfActive(mf[j].x)) {
                const uint4 link = arrayAt<uint4>(smem, w.link)[j];
                const f3 nrm = xyz(arrayAt<real4>(smem, w.basis)[3 * j]);
                const unsigned char *con = smem + w.contacts + slot * sizeof(real4);
                const f3 xa = xyz(loadCluster(link.x + kRecX * kF4)), xb = xyz(loadCluster(link.y + kRecX * kF4));
                const f3 rA = qrot(asq(loadCluster(link.x + kRecQ * kF4)), xyz(*reinterpret_cast<const real4 *>(con)));
                const f3 rB = qrot(asq(loadCluster(link.y + kRecQ * kF4)), xyz(*reinterpret_cast<const real4 *>(con + w.conStride)));
                const real gap = dot(nrm, sub(add(xa, rA), add(xb, rB)));
                open = gap > 0.0f;
                const int ci = cslot(d, w.mlo + j, v & 7);
                const real4 a = f4(rA, -gap / window), b = f4(rB, -gap / window);
                row[0] = a;
                row[1] = b;
                S.rA[ci] = a;
                S.rB[ci] = b;
            }
            const unsigned hit = __ballot_sync(0xffffffffu, open);
            // Two lanes a manifold: its response to all open contacts (brakePrepareAt).
            const int j0 = arrayAt<int>(smem, w.taskFirst)[task], j1 = arrayAt<int>(smem, w.taskFirst)[task + 1];
            const int jm = j0 + (lane >> 1), side = lane & 1, m = w.mlo + jm;
            const int2 f = jm < j1 ? mf[jm] : make_int2(0, 0);
            const unsigned mine = (hit >> (f.y & 31)) & ((1u << (f.x >> kMfCountShift)) - 1u);
            real invN = 0.0f, invMass = 0.0f, compliance = 0.0f;
            f3 nrm{0, 0, 0}, response{0, 0, 0};
            const bool move = (f.x & (side == 0 ? kMfMoveA : kMfMoveB)) != 0;
            int flags = 0;
            __syncwarp();
            if (mine) {
                f3 patch{0, 0, 0};
                for (int k = 0; k < f.x >> kMfCountShift; k++)
                    if ((mine >> k) & 1)
                        patch = add(patch, xyz(reinterpret_cast<const real4 *>(rows + ((f.y & 31) + k) * kRowReals)[side]));
                invN = 1.0f / static_cast<real>(__popc(mine));
                nrm = xyz(arrayAt<real4>(smem, w.basis)[3 * jm]);
                const uint4 link = arrayAt<uint4>(smem, w.link)[jm];
                const unsigned rec = side == 0 ? link.x : link.y;
                const int2 ab = d.live.ab[m];
                flags = (d.meta[side == 0 ? ab.x : ab.y].w & 0xffff) + (move ? kBrakeMoves : 0);
                if (move) {
                    invMass = 1.0f / loadCluster(rec + kRecX * kF4).w;
                    compliance = patchResponse(xyz(loadCluster(rec + kRecMoment * kF4)), asq(loadCluster(rec + kRecQ * kF4)), patch,
                                               invN, nrm, response);
                }
            }
            const real oMass = __shfl_xor_sync(0xffffffffu, invMass, 1), oComp = __shfl_xor_sync(0xffffffffu, compliance, 1);
            const int oFlags = __shfl_xor_sync(0xffffffffu, flags, 1);
            if (jm < j1 && side == 0) {
                d.mSpec[m] = mine ? 1 : 0;
                d.specPred[m] = make_int2(-1, -1);
            }
            if (mine && side == 0) {
                S.b0[m] = f4(nrm, invMass + oMass + compliance + oComp);
                S.b1[m] = f4(response, invN);
                S.C0[cslot(d, m, 0)] = mk4(invMass, oMass, static_cast<real>(flags), static_cast<real>(oFlags));
            } else if (mine) {
                S.b2[m] = f4(response, static_cast<real>(mine));
            }
            __syncwarp();
        }
    clusterSync(w.size);
    for (int i = threadIdx.x; i < w.nb; i += blockDim.x)
        if (arrayAt<int>(smem, w.info)[i] & kBiMovable)
            brakePredecessors(d, w.m0, w.b0 + i);
    clusterSync(w.size);
    if (w.rank == 0) {
        int *level = w.levelsFit ? arrayAt<int>(smem, static_cast<int>(sizeof(real)) * kVelReals * w.cnt) : d.mActive + w.m0;
        const unsigned rec0 = sharedAddress(smem + w.rec);
        const int base = w.base, per = w.per;
        brakeSweep(d, base, w.cnt, w.m0, w.n, arrayAt<real>(smem, 0), level, [&](int g, q4 &q, f3 &moment) {
            const int i = g - base, owner = i / per;
            const unsigned rec = mapShared(rec0, owner) + kF4 * kRecF4 * (i - owner * per);
            q = asq(loadCluster(rec + kRecQ * kF4));
            moment = xyz(loadCluster(rec + kRecMoment * kF4));
        });
    }
    clusterSync(w.size);
}

// ---- projection (solver_projection.cpp:169-280) ----

// A pass's corrections: a lane a contact finds its arms and depth, then two lanes a manifold (side A,
// side B) add the corrected contacts' in contact order and respond, into the first two values of the
// side's stamp record (w of the first: the side's sign, 0 = none). The deepest patch goes to `deepest`
// of every CTA of the cluster.
__device__ __forceinline__ void projectManifolds(const Dev &d, const StepParams &p, const World &w, unsigned char *smem,
                                                 unsigned deepest) {
    if (bodyWarp())
        return;
    const int lane = threadIdx.x & 31, side = lane & 1;
    real *rows = arrayAt<real>(smem, 0) + contactWarp() * 32 * kRowReals;
    real4 *row = reinterpret_cast<real4 *>(rows + lane * kRowReals);
    const int2 *mf = arrayAt<int2>(smem, w.mf);
    const uint4 *links = arrayAt<uint4>(smem, w.link);
    const real4 *bases = arrayAt<real4>(smem, w.basis);
    int most = 0;
    for (int task = contactWarp(); task < w.tasks; task += contactWarps()) {
        const int slot = 32 * task + lane, v = arrayAt<uint16_t>(smem, w.slots)[slot], j = v >> 3;
        if (v != 0xffff && mfActive(mf[j].x)) {
            const uint4 link = links[j];
            const f3 nrm = xyz(bases[3 * j]);
            const real4 *con = arrayAt<real4>(smem, w.contacts) + slot;
            const m3 rotA{xyz(loadCluster(link.x)), xyz(loadCluster(link.x + kF4)), xyz(loadCluster(link.x + 2 * kF4))};
            const m3 rotB{xyz(loadCluster(link.y)), xyz(loadCluster(link.y + kF4)), xyz(loadCluster(link.y + 2 * kF4))};
            const f3 rA = mul(rotA, xyz(con[0]));
            const f3 rB = mul(rotB, xyz(*reinterpret_cast<const real4 *>(reinterpret_cast<const unsigned char *>(con) + w.conStride)));
            const real rawDepth = -dot(nrm, sub(add(xyz(loadCluster(link.x + kRecX * kF4)), rA),
                                                add(xyz(loadCluster(link.y + kRecX * kF4)), rB)));
            row[0] = f4(rA, rawDepth - p.projSlop);
            row[1] = f4(rB, 0.0f);
        }
        __syncwarp();
        const int j0 = arrayAt<int>(smem, w.taskFirst)[task], j1 = arrayAt<int>(smem, w.taskFirst)[task + 1];
        const int jm = j0 + (lane >> 1); // up to eight manifolds a task
        const int2 f = jm < j1 ? mf[jm] : make_int2(0, 0);
        const bool on = mfActive(f.x), move = on && (f.x & (side == 0 ? kMfMoveA : kMfMoveB));
        f3 patch{0, 0, 0};
        real patchDepth = 0.0f;
        int corrected = 0;
        if (on) {
            const real4 *r = reinterpret_cast<const real4 *>(rows + (f.y & 31) * kRowReals);
            for (int c = f.x >> kMfCountShift; c > 0; c--, r += kRowReals / 4) {
                const real4 a = r[0];
                if (a.w > 0.0f) {
                    patch = add(patch, xyz(side == 0 ? a : r[1]));
                    patchDepth += a.w;
                    corrected++;
                }
            }
        }
        real invN = 0.0f, compliance = 0.0f, invMass = 0.0f;
        f3 nrm{0, 0, 0}, tq{0, 0, 0};
        Inertia I{};
        q4 q{0, 0, 0, 1};
        uint4 link{};
        if (jm < j1)
            link = links[jm];
        if (corrected) {
            invN = 1.0f / static_cast<real>(corrected);
            nrm = xyz(bases[3 * jm]);
            if (move) {
                const unsigned rec = side == 0 ? link.x : link.y;
                I = inertia(xyz(loadCluster(rec + kRecMoment * kF4)));
                q = asq(loadCluster(rec + kRecQ * kF4));
                invMass = 1.0f / loadCluster(rec + kRecX * kF4).w;
                tq = qrot(qconj(q), cross(scale(patch, invN), nrm));
                compliance = angularCompliance(I, tq);
            }
        }
        const real oMass = __shfl_xor_sync(0xffffffffu, invMass, 1), oComp = __shfl_xor_sync(0xffffffffu, compliance, 1);
        if (f.x & (side == 0 ? kMfMassA : kMfMassB)) {
            const unsigned out = side == 0 ? link.z : link.w;
            if (corrected && move) {
                const real K = side == 0 ? invMass + oMass + compliance + oComp : oMass + invMass + oComp + compliance;
                const real dp = p.projBeta * patchDepth * invN / K;
                storeCluster(out, f4(scale(nrm, invMass * dp), side == 0 ? 1.0f : -1.0f));
                storeCluster(out + kF4, f4(scale(angularResponse(I, q, tq), dp), 0.0f));
            } else {
                storeCluster(out, mk4(0.0f, 0.0f, 0.0f, 0.0f));
            }
        }
        if (corrected)
            most = max(most, fbits(patchDepth * invN));
        __syncwarp();
    }
    most = __reduce_max_sync(0xffffffffu, most);
    if (most && lane < w.size)
        maxClusterInt(mapShared(deepest, lane), most);
}

// One body's averaged correction (projBodyAt).
__device__ __forceinline__ void projectBody(const Dev &d, const StepParams &p, const World &w, unsigned char *smem, int i, int info) {
    const int nf = nForcesDev(d);
    f3 sl{0, 0, 0}, sa{0, 0, 0};
    int cnt = 0;
    int e = arrayAt<int>(smem, w.entry)[i];
    const int e1 = arrayAt<int>(smem, w.entry)[i + 1];
    while (nf > 0 && e < e1 && static_cast<int>(d.adjSeq[e]) < nf)
        e++; // forces come first
    const real4 *r = arrayAt<real4>(smem, w.stamps) + (e - w.e0) * kStampF4;
    for (; e < e1; e++, r += kStampF4) {
        const real4 cl = r[0];
        if (cl.w == 0.0f)
            continue;
        const f3 ca = xyz(r[1]);
        cnt++;
        if (cl.w > 0.0f) {
            sl = add(sl, xyz(cl));
            sa = add(sa, ca);
        } else {
            sl = sub(sl, xyz(cl));
            sa = sub(sa, ca);
        }
    }
    const real invCount = 1.0f / static_cast<real>(cnt > 1 ? cnt : 1);
    f3 dl = scale(sl, invCount);
    f3 da = scale(sa, invCount);
    const int locks = info >> kBiLocks;
    maskLocked(locks & 0xff, dl);
    maskLocked((locks >> 8) & 0xff, da);
    const real cap = p.projMaxCorr;
    if (cap > 0.0f) {
        const real moved = length(dl);
        if (moved > cap)
            dl = scale(dl, cap / moved);
        const real turned = length(da);
        if (turned > cap)
            da = scale(da, cap / turned);
    }
    const real4 *rec = arrayAt<real4>(smem, w.rec) + kRecF4 * i;
    const real4 x4 = rec[kRecX];
    movePose(d, w, smem, i, add(xyz(x4), dl), x4.w, qintegrate(asq(rec[kRecQ]), da), true);
}

// `deepest`: two words a CTA, zero on entry; passes alternate between them.
__device__ __forceinline__ void projectionPhase(const Dev &d, const StepParams &p, const World &w, unsigned char *smem, real tolerance,
                                                int *deepest) {
    for (int it = 0; it < p.projIters; it++) {
        projectManifolds(d, p, w, smem, sharedAddress(deepest + (it & 1)));
        clusterSync(w.size);
        const bool last = bitsf(*const_cast<volatile int *>(deepest + (it & 1))) <= tolerance;
        for (int i = bodyThread(); i < w.nb; i += blockDim.x) {
            const int info = arrayAt<int>(smem, w.info)[i];
            if (info & kBiMovable)
                projectBody(d, p, w, smem, i, info);
        }
        if (threadIdx.x == 0)
            deepest[(it + 1) & 1] = 0;
        clusterSync(w.size);
        if (last)
            return;
    }
}

// Rebase (ManifoldStore::rebase), a lane a contact.
__device__ __forceinline__ void rebasePhase(const Dev &d, const StepParams &p, const World &w, unsigned char *smem) {
    for (int slot = threadIdx.x; slot < 32 * w.tasks; slot += blockDim.x) {
        const int v = arrayAt<uint16_t>(smem, w.slots)[slot], j = v >> 3;
        if (v == 0xffff)
            continue;
        const uint4 link = arrayAt<uint4>(smem, w.link)[j];
        const real4 *basis = arrayAt<real4>(smem, w.basis) + 3 * j;
        unsigned char *con = smem + w.contacts + slot * sizeof(real4);
        const auto at = [&](int k) -> real4 & { return *reinterpret_cast<real4 *>(con + k * w.conStride); };
        const f3 pA = add(xyz(loadCluster(link.x + kRecX * kF4)), qrot(asq(loadCluster(link.x + kRecQ * kF4)), xyz(at(0))));
        const f3 pB = add(xyz(loadCluster(link.y + kRecX * kF4)), qrot(asq(loadCluster(link.y + kRecQ * kF4)), xyz(at(1))));
        f3 C0 = add(basisMulD(xyz(basis[0]), xyz(basis[1]), xyz(basis[2]), sub(pA, pB)), f3{COLLISION_MARGIN, 0, 0});
        if (C0.x < -p.maxPen)
            C0.x = -p.maxPen;
        at(2) = f4(C0, 0.0f);
        d.live.C0[cslot(d, w.mlo + j, v & 7)] = f4(C0, 0.0f);
    }
}

// ---- setup ----

__device__ __forceinline__ int manifoldFlags(const Dev &d, int2 ab, int n) {
    const PairFlags f = loadPairFlags<true>(d, ab);
    int v = (f.awakeA || f.awakeB) ? kMfAwake : 0;
    v |= (f.sides & kSideA) ? kMfSideA : 0;
    v |= (f.sides & kSideB) ? kMfSideB : 0;
    v |= f.touches ? kMfMixed : 0;
    v |= d.x[ab.x].w > 0.0f ? kMfMassA | (inUpdate(d, ab.x) ? kMfMoveA : 0) : 0;
    v |= d.x[ab.y].w > 0.0f ? kMfMassB | (inUpdate(d, ab.y) ? kMfMoveB : 0) : 0;
    return v | n << kMfCountShift;
}

struct SetupShared {
    int fits[kMaxTeam], active[kMaxTeam], entry0[kMaxTeam];
    int tasks, colourCount[kMaxColours + 1], colourBase[kMaxColours + 1];
};

// Deals the world's coloured bodies, by colour and then slot, round the CTAs; a world's CTAs find the same.
__device__ __forceinline__ void dealColours(const Dev &d, World &w, unsigned char *smem, SetupShared &sh, bool fits) {
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, warps = blockDim.x >> 5;
    int *warpColours = arrayAt<int>(smem, 0) + warp * (kMaxColours + 1); // scratch
    const auto colourOf = [&](int i) {
        return i < w.cnt && inUpdate(d, w.base + i) && d.colour[w.base + i] < kMaxColours ? d.colour[w.base + i] : kMaxColours;
    };
    if (threadIdx.x <= kMaxColours)
        sh.colourCount[threadIdx.x] = 0;
    __syncthreads();
    for (int i = threadIdx.x; i < w.cnt; i += blockDim.x)
        if (colourOf(i) < kMaxColours)
            atomicAdd(&sh.colourCount[colourOf(i)], 1);
    __syncthreads();
    int start = 0;
    for (int c = 0; c <= kMaxColours; c++) { // the first of this CTA at or after the colour's start
        w.colourAt[c] = (start - w.rank + w.size - 1) / w.size;
        w.groupAt[c] = 0;
        if (threadIdx.x == 0)
            sh.colourBase[c] = start;
        start += c < kMaxColours ? sh.colourCount[c] : 0;
    }
    for (int i0 = 0; i0 < w.cnt; i0 += blockDim.x) {
        const int i = i0 + static_cast<int>(threadIdx.x), c = colourOf(i);
        if (lane <= kMaxColours)
            warpColours[lane] = 0;
        __syncwarp();
        const unsigned peers = __match_any_sync(0xffffffffu, c);
        const int below = __popc(peers & ((1u << lane) - 1));
        if (below == 0)
            warpColours[c] = __popc(peers);
        __syncthreads();
        if (threadIdx.x < kMaxColours) {
            int at = sh.colourBase[threadIdx.x];
            for (int k = 0; k < warps; k++) {
                int &n = arrayAt<int>(smem, 0)[k * (kMaxColours + 1) + threadIdx.x];
                const int first = at;
                at += n;
                n = first;
            }
            sh.colourBase[threadIdx.x] = at;
        }
        __syncthreads();
        if (fits && c < kMaxColours) {
            const int at = warpColours[c] + below;
            if (at % w.size == w.rank)
                arrayAt<uint16_t>(smem, w.colourList)[at / w.size] = static_cast<uint16_t>(i);
        }
        __syncthreads();
    }
}

// The terms of this CTA's coloured bodies and, a group at a time, their order by kind.
__device__ __forceinline__ void listTerms(const Dev &d, const World &w, unsigned char *smem) {
    const uint16_t *list = arrayAt<uint16_t>(smem, w.colourList);
    const int *termFirst = arrayAt<int>(smem, w.termFirst);
    Term *terms = arrayAt<Term>(smem, w.terms);
    const int bodies = w.colourAt[kMaxColours];
    for (int k = threadIdx.x >> 5; k < bodies; k += blockDim.x >> 5) {
        const int first = termFirst[k];
        bodyTerms(
                d, w.base + list[k], [&](int b) { return placeOf(w, b - w.base).rec; },
                [&](int n, const Term &t) {
                    terms[first + n] = t;
                    terms[first + n].row = first + n;
                });
    }
    __syncthreads();
    const int rows = passRows();
    for (int c = 0; c < kMaxColours; c++) {
        const int first = termFirst[w.colourAt[c]], last = termFirst[w.colourAt[c + 1]];
        for (int e = first + static_cast<int>(threadIdx.x); e < last; e += blockDim.x) {
            const int from = e - (e - first) % rows, to = min(from + rows, last), kind = terms[e].flags & kTermKind;
            int at = from;
            for (int k = from; k < to; k++) {
                const int other = terms[k].flags & kTermKind;
                at += other < kind || (other == kind && k < e) ? 1 : 0;
            }
            arrayAt<uint16_t>(smem, w.termOrder)[at] = static_cast<uint16_t>(e);
        }
        const int groups = w.groupAt[c + 1] - w.groupAt[c];
        for (int k = threadIdx.x; k < groups * (kTermKinds + 1); k += blockDim.x) {
            const int g = k / (kTermKinds + 1), kind = k - g * (kTermKinds + 1), from = first + g * rows, to = min(from + rows, last);
            int before = 0;
            for (int e = from; e < to; e++)
                before += (terms[e].flags & kTermKind) < kind ? 1 : 0;
            arrayAt<uint16_t>(smem, w.termKinds)[w.groupAt[c] * (kTermKinds + 1) + k] = static_cast<uint16_t>(before);
        }
    }
}


__device__ __forceinline__ int carve(int &at, size_t bytes) {
    const int p = at;
    at += static_cast<int>((bytes + 31) & ~static_cast<size_t>(31));
    return p;
}

// This CTA's part of the world, its state loaded; agrees with the cluster's other CTAs whether every
// part fits in shared memory (false: the world is left to worldWideKernel) and whether any manifold
// is active (`active`).
template <bool ARM, bool COLOURS>
__device__ __forceinline__ bool setupWorld(const Dev &d, const WorldRun &r, World &shared, unsigned char *smem, SetupShared &sh,
                                           bool &active) {
    const ManifoldBuf &L = d.live;
    World w = shared;
    w.per = (w.cnt + w.size - 1) / w.size;
    w.b0 = min(w.base + w.rank * w.per, w.base + w.cnt);
    w.nb = min(w.per, w.base + w.cnt - w.b0);
    const int mper = (w.n + w.size - 1) / w.size;
    w.mlo = min(w.m0 + w.rank * mper, w.m0 + w.n);
    w.nm = min(mper, w.m0 + w.n - w.mlo);
    w.e0 = d.adjStart[w.b0];
    const int ne = d.adjStart[w.b0 + w.nb] - w.e0, end = static_cast<int>(r.smemBytes);
    // A part this large cannot fit; its sizes in bytes would not fit an int either.
    bool fits = ne < 65536 && w.nm < 8191;
    // The same offsets in every CTA up to the stamps, so neighbours find a body's record and entries.
    // The brake runs before or after the rounds, so the world's velocities and levels lie over
    // what only they need: the contact rows, the block sums and the step constants.
    int at = static_cast<int>(r.rowBytes);
    w.sums = carve(at, sizeof(real) * kBlkReals * w.per);
    w.con = carve(at, kF4 * kConF4 * w.per);
    const int vel = static_cast<int>(sizeof(real)) * kVelReals * w.cnt;
    w.levelsFit = w.n < 8192;
    at = max(at, (vel + (w.levelsFit ? 4 * w.n : 0) + 31) & ~31);
    w.info = carve(at, sizeof(int) * w.per);
    w.entry = carve(at, sizeof(int) * (w.per + 1));
    w.rec = carve(at, kF4 * kRecF4 * w.per);
    w.rec0 = static_cast<int>(sharedAddress(smem + w.rec));
    w.con0 = static_cast<int>(sharedAddress(smem + w.con));
    w.colourList = carve(at, COLOURS ? sizeof(uint16_t) * w.per : 0);
    w.termFirst = carve(at, COLOURS ? sizeof(int) * (w.per + 1) : 0);
    w.stamps = carve(at, fits ? kF4 * kStampF4 * ne : 0);
    const int nm = fits ? w.nm : 0;
    w.mf = carve(at, sizeof(int2) * nm);
    w.link = carve(at, sizeof(uint4) * nm);
    w.basis = carve(at, kF4 * 3 * nm);
    w.cap = carve(at, ARM ? kF4 * 2 * nm : 0);
    w.taskFirst = carve(at, sizeof(int) * (nm + 1));
    fits = fits && at <= end;
    int2 *mf = arrayAt<int2>(smem, w.mf);
    active = false;
    if (fits)
        for (int j = threadIdx.x; j < w.nm; j += blockDim.x) {
            const int flags = manifoldFlags(d, L.ab[w.mlo + j], L.count[w.mlo + j]);
            mf[j] = make_int2(flags, 0);
            active = active || mfActive(flags);
        }
    active = __syncthreads_or(active) != 0;
    w.tasks = 0;
    if (fits) {
        // Pack whole manifolds into tasks of 32 contact slots, in order.
        if (threadIdx.x < 32) {
            int *first = arrayAt<int>(smem, w.taskFirst);
            int j0 = 0, task = 0;
            while (j0 < w.nm) {
                const int lane = threadIdx.x, j = j0 + lane;
                const int n = j < w.nm && lane < kTaskManifolds ? mf[j].x >> kMfCountShift : 33;
                int upTo = n;
#pragma unroll
                for (int o = 1; o < kTaskManifolds; o <<= 1) {
                    const int y = __shfl_up_sync(0xffffffffu, upTo, o);
                    if (lane >= o)
                        upTo += y;
                }
                const int taken = __popc(__ballot_sync(0xffffffffu, lane < kTaskManifolds && upTo <= 32));
                if (lane < taken)
                    mf[j].y = 32 * task + upTo - n;
                if (lane == 0)
                    first[task] = j0;
                j0 += taken;
                task++;
            }
            if (threadIdx.x == 0) {
                first[task] = w.nm;
                sh.tasks = task;
            }
        }
        __syncthreads();
        w.tasks = sh.tasks;
        w.slots = carve(at, sizeof(uint16_t) * 32 * w.tasks);
        w.conStride = static_cast<int>(kF4) * 32 * w.tasks;
        w.contacts = carve(at, static_cast<size_t>(ARM ? 7 : 5) * w.conStride);
        fits = at <= end;
    }
    if (COLOURS) {
        dealColours(d, w, smem, sh, fits);
        w.colourBlocks = carve(at, sizeof(real) * kBlkReals * w.colourAt[kMaxColours]);
        fits = fits && at <= end;
        if (fits) {
            int *termFirst = arrayAt<int>(smem, w.termFirst), *count = arrayAt<int>(smem, w.sums); // scratch
            const int bodies = w.colourAt[kMaxColours];
            for (int k = threadIdx.x >> 5; k < bodies; k += blockDim.x >> 5) {
                const int n = bodyTerms(d, w.base + arrayAt<uint16_t>(smem, w.colourList)[k], [](int) { return 0u; }, [](int, const Term &) {});
                if ((threadIdx.x & 31) == 0)
                    count[k] = n;
            }
            __syncthreads();
            for (int k = threadIdx.x; k <= bodies; k += blockDim.x) {
                int before = 0;
                for (int j = 0; j < k; j++)
                    before += count[j];
                termFirst[k] = before;
            }
            __syncthreads();
            const int terms = termFirst[bodies];
            for (int c = 0; c < kMaxColours; c++) {
                const int n = termFirst[w.colourAt[c + 1]] - termFirst[w.colourAt[c]];
                w.groupAt[c + 1] = w.groupAt[c] + max(1, (n + passRows() - 1) / passRows());
            }
            w.termKinds = carve(at, sizeof(uint16_t) * (kTermKinds + 1) * w.groupAt[kMaxColours]);
            w.termOrder = carve(at, sizeof(uint16_t) * terms);
            fits = terms < 65536 && at <= end;
            w.terms = carve(at, fits ? sizeof(Term) * terms : 0);
            fits = fits && at <= end;
        }
    }
    if (static_cast<int>(threadIdx.x) < w.size) {
        storeClusterInt(mapShared(sharedAddress(&sh.fits[w.rank]), threadIdx.x), fits ? 1 : 0);
        storeClusterInt(mapShared(sharedAddress(&sh.active[w.rank]), threadIdx.x), active ? 1 : 0);
        storeClusterInt(mapShared(sharedAddress(&sh.entry0[w.rank]), threadIdx.x), w.e0);
    }
    clusterSync(w.size);
    active = false;
    for (int k = 0; k < w.size; k++) {
        fits = fits && sh.fits[k];
        active = active || sh.active[k];
    }
    if (!fits)
        return false;
    int *info = arrayAt<int>(smem, w.info), *entry = arrayAt<int>(smem, w.entry);
    for (int i = threadIdx.x; i <= w.nb; i += blockDim.x) {
        const int g = w.b0 + i;
        entry[i] = d.adjStart[g];
        if (i == w.nb)
            break;
        const real4 x4 = d.x[g];
        const bool update = inUpdate(d, g);
        info[i] = (d.colour[g] & kBiColour) | (update ? kBiUpdate : 0) | (update && x4.w > 0.0f ? kBiMovable : 0) |
                  (COLOURS && bodyHasForce(d, g, nForcesDev(d)) ? kBiForce : 0) | (d.meta[g].w & 0xffff) << kBiLocks;
        real4 *rec = arrayAt<real4>(smem, w.rec) + kRecF4 * i;
        rec[kRecX] = x4;
        rec[kRecQ] = d.q[g];
        rec[kRecMoment] = d.moment[g];
    }
    uint16_t *slots = arrayAt<uint16_t>(smem, w.slots);
    for (int k = threadIdx.x; k < 32 * w.tasks; k += blockDim.x)
        slots[k] = 0xffff;
    const unsigned rec0 = sharedAddress(smem + w.rec), stamps0 = sharedAddress(smem + w.stamps);
    for (int j = threadIdx.x; j < w.nm; j += blockDim.x) {
        const int m = w.mlo + j;
        const int2 ab = L.ab[m], slot = d.stampSlot[m];
        real4 *basis = arrayAt<real4>(smem, w.basis) + 3 * j;
        basis[0] = L.b0[m];
        basis[1] = L.b1[m];
        basis[2] = L.b2[m];
        const int flags = mf[j].x;
        const int ia = ab.x - w.base, ib = ab.y - w.base, oa = ia / w.per, ob = ib / w.per;
        uint4 link;
        link.x = mapShared(rec0, oa) + kF4 * kRecF4 * (ia - oa * w.per);
        link.y = mapShared(rec0, ob) + kF4 * kRecF4 * (ib - ob * w.per);
        link.z = flags & kMfMassA ? mapShared(stamps0, oa) + kF4 * kStampF4 * (slot.x - sh.entry0[oa]) : 0;
        link.w = flags & kMfMassB ? mapShared(stamps0, ob) + kF4 * kStampF4 * (slot.y - sh.entry0[ob]) : 0;
        arrayAt<uint4>(smem, w.link)[j] = link;
        if (ARM) {
            real4 *cap = arrayAt<real4>(smem, w.cap) + 2 * j;
            const real4 cA = L.capA[m];
            cap[0] = mk4(cA.x, cA.y, cA.z, L.armFlag[m] ? 1.0f : 0.0f);
            cap[1] = L.capB[m];
        }
    }
    __syncthreads();
    for (int j = threadIdx.x; j < w.nm; j += blockDim.x) {
        const int2 v = mf[j];
        for (int c = 0; c < v.x >> kMfCountShift; c++)
            slots[v.y + c] = static_cast<uint16_t>(j << 3 | c);
    }
    __syncthreads();
    for (int k = threadIdx.x; k < 32 * w.tasks; k += blockDim.x) {
        const int v = slots[k];
        if (v == 0xffff)
            continue;
        const int ci = cslot(d, w.mlo + (v >> 3), v & 7);
        unsigned char *con = smem + w.contacts + k * sizeof(real4);
        const auto at = [&](int a) -> real4 & { return *reinterpret_cast<real4 *>(con + a * w.conStride); };
        at(0) = L.rA[ci];
        at(1) = L.rB[ci];
        at(2) = L.C0[ci];
        at(3) = L.k[ci];
        at(4) = L.lam[ci];
        if (ARM) {
            at(5) = L.armA[ci];
            at(6) = L.armB[ci];
        }
    }
    if (COLOURS)
        listTerms(d, w, smem);
    if (threadIdx.x == 0)
        shared = w;
    clusterSync(w.size);
    return true;
}

// Contact state the rounds changed, back to the global arrays (rebasePhase writes C0 itself).
template <bool ARM, bool COLOURS>
__device__ __forceinline__ void storeContacts(const Dev &d, const World &w, unsigned char *smem) {
    const ManifoldBuf &L = d.live;
    const int2 *mf = arrayAt<int2>(smem, w.mf);
    for (int k = threadIdx.x; k < 32 * w.tasks; k += blockDim.x) {
        const int v = arrayAt<uint16_t>(smem, w.slots)[k];
        if (v == 0xffff || (COLOURS && (mf[v >> 3].x & kMfMixed))) // a mixed manifold's is there
            continue;
        const int ci = cslot(d, w.mlo + (v >> 3), v & 7);
        const unsigned char *con = smem + w.contacts + k * sizeof(real4);
        const auto at = [&](int a) { return *reinterpret_cast<const real4 *>(con + a * w.conStride); };
        L.k[ci] = at(3);
        L.lam[ci] = at(4);
        if (ARM) {
            L.armA[ci] = at(5);
            L.armB[ci] = at(6);
        }
    }
    if (ARM)
        for (int j = threadIdx.x; j < w.nm; j += blockDim.x) {
            if (COLOURS && (mf[j].x & kMfMixed))
                continue;
            const int m = w.mlo + j;
            const real4 *cap = arrayAt<real4>(smem, w.cap) + 2 * j;
            L.capA[m] = mk4(cap[0].x, cap[0].y, cap[0].z, 0.0f);
            L.capB[m] = cap[1];
            L.armFlag[m] = cap[0].w != 0.0f ? 1 : 0;
        }
}

template <bool COLOURS, bool ARM>
__global__ void __launch_bounds__(kMaxWorldThreads, 1)
        worldKernel(const __grid_constant__ Dev d, const __grid_constant__ StepParams p, const __grid_constant__ WorldRun r) {
    pdlWait();
    pdlTrigger();
    stampPhase(d);
    extern __shared__ __align__(32) unsigned char smem[];
    __shared__ int shared[4], deepest[2];
    __shared__ real carry[2][32];
    __shared__ SetupShared sh;
    // The world's description is uniform and wide: it is kept in shared memory, and a phase reads what
    // it needs.
    __shared__ World w;
    if (threadIdx.x == 0) {
        w.rank = clusterRank();
        w.size = clusterSize();
    }
    __syncthreads();
    const int size = w.size, nWorlds = d.ctr[C_WORLDS];
    const int clusters = static_cast<int>(gridDim.x) / size;
    for (int world = static_cast<int>(blockIdx.x) / size; world < nWorlds; world += clusters) {
        if (d.wCount[world] <= 0)
            continue;
        clusterSync(size); // every CTA runs, and has left the world before
        if (threadIdx.x == 0) {
            const int m0 = r.multiWorld ? d.wMan[world] : 0;
            w.base = d.wBase[world];
            w.cnt = d.wCount[world];
            w.m0 = m0;
            w.n = (r.multiWorld ? d.wMan[world + 1] : d.ctr[C_LIVE]) - m0;
            w.f0 = w.f1 = 0;
        }
        if (threadIdx.x < 2)
            deepest[threadIdx.x] = 0;
        if (threadIdx.x < 4)
            shared[threadIdx.x] = 0;
        __syncthreads();
        int colours = 0;
        if (COLOURS) {
            const int nf = nForcesDev(d);
            if (threadIdx.x < 2)
                shared[2 + threadIdx.x] = r.multiWorld ? firstForce(d, nf, w.base + (threadIdx.x ? w.cnt : 0))
                                                       : (threadIdx.x ? nf : 0);
            int mine = 0;
            for (int i = threadIdx.x; i < w.cnt; i += blockDim.x) {
                const int g = w.base + i;
                if (inUpdate(d, g) && d.colour[g] < kMaxColours)
                    mine |= 1 << d.colour[g];
            }
            if (mine)
                atomicOr(&shared[1], mine);
            __syncthreads();
            colours = shared[1];
            if (threadIdx.x == 0) {
                w.f0 = shared[2];
                w.f1 = shared[3];
            }
            __syncthreads();
        }
        bool active;
        const bool fits = setupWorld<ARM, COLOURS>(d, r, w, smem, sh, active);
        if (threadIdx.x == 0 && w.rank == 0)
            d.wStop[world] = fits ? 1 : 0; // 0: worldWideKernel's
        if (!fits)
            continue;
        for (int step = 0;; step++) {
            const bool finished = step == r.substeps; // the brake runs once more after the last substep
            if (step > 0 && !finished) {
                rebasePhase(d, p, w, smem);
                if (!r.brake) // (whose barriers keep the poses that the rebase reads)
                    clusterSync(size);
            }
            if (r.brake)
                brakePhase(d, w, smem, r.substeps > 1 && !finished ? r.dt * static_cast<real>(r.substeps - step) : p.collisionDt);
            if (finished)
                break;
            if (r.stampSolve && w.rank == 0 && threadIdx.x == 0)
                stampSolve(d);
            for (int i = threadIdx.x; i < w.nb; i += blockDim.x) {
                const int g = w.b0 + i;
                warmstartAt(d, p, g);
                const real4 x4 = d.x[g], x0 = d.x0[g], q0 = d.q0[g];
                real4 *con = arrayAt<real4>(smem, w.con) + kConF4 * i;
                con[kConXi] = d.xi[g];
                con[kConQi] = d.qi[g];
                con[kConX0] = x0;
                con[kConQ0] = q0;
                putPose(arrayAt<real4>(smem, w.rec) + kRecF4 * i, xyz(x4), x4.w, asq(d.q[g]), xyz(x0), asq(q0));
            }
            clusterSync(size);
            for (int it = -1; it < r.rounds; it++) { // -1: the first stamps
                const bool newton = it >= 0 && it < r.newtonRounds;
                if (newton) {
                    if (COLOURS) {
                        if (colours) {
                            colourPhase<ARM>(d, p, w, smem, colours, it > 0 ? 1 : 0, carry);
                            if (!bodyWarp())
                                contactPhase<ARM, COLOURS>(d, p, w, smem, kStampsMixed, 1.0f);
                            clusterSync(size);
                        }
                        overflowForces(d, p, w, smem);
                    }
                    solvePhase<COLOURS>(d, p, w, smem);
                    clusterSync(size);
                    if (COLOURS && w.f1 > w.f0) {
                        applyPhase(d, p, w, smem);
                        clusterSync(size);
                    }
                }
                if (!bodyWarp())
                    contactPhase<ARM, COLOURS>(d, p, w, smem,
                                               it < 0 ? kStampsOverflow : (it + 1 < r.newtonRounds ? kDualStamps : kDual),
                                               newton || it < 0 ? 1.0f : p.stiffnessDecay);
                if (COLOURS && it >= 0 && bodyWarp())
                    forceDuals(d, p, w);
                if (it + 1 < r.newtonRounds)
                    startBlocks<COLOURS>(p, w, smem); // the poses of this phase are where the next solve starts
                clusterSync(size);
            }
            const int idle = step + 1 == r.substeps ? 1 : 0;
            for (int i = threadIdx.x; i < w.nb; i += blockDim.x) {
                const int g = w.b0 + i;
                const real4 *rec = arrayAt<real4>(smem, w.rec) + kRecF4 * i;
                d.x[g] = rec[kRecX];
                d.q[g] = rec[kRecQ];
                finishAt(d, p, g, idle);
            }
            clusterSync(size);
        }
        storeContacts<ARM, COLOURS>(d, w, smem);
        if (r.project && active)
            projectionPhase(d, p, w, smem, r.tolerance, deepest);
        rebasePhase(d, p, w, smem);
        clusterSync(size); // no CTA leaves while another reads its shared memory
    }
}

// ---- worlds that do not fit ----

// The same phases for the worlds worldKernel left (wStop 0), on the global arrays with the separate
// launches' functions, a cluster a world.
template <bool COLOURS, bool ARM>
__global__ void __launch_bounds__(kWideThreads)
        worldWideKernel(const __grid_constant__ Dev d, const __grid_constant__ StepParams p, const __grid_constant__ WorldRun r) {
    pdlWait();
    pdlTrigger();
    extern __shared__ __align__(32) unsigned char smem[];
    const int rank = clusterRank(), size = clusterSize();
    const int nWorlds = d.ctr[C_WORLDS];
    const int clusters = static_cast<int>(gridDim.x) / size;
    const int tid = rank * static_cast<int>(blockDim.x) + static_cast<int>(threadIdx.x), threads = size * static_cast<int>(blockDim.x);
    for (int world = static_cast<int>(blockIdx.x) / size; world < nWorlds; world += clusters) {
        if (d.wCount[world] <= 0 || d.wStop[world])
            continue;
        const int base = d.wBase[world], end = base + d.wCount[world];
        const int m0 = r.multiWorld ? d.wMan[world] : 0, m1 = r.multiWorld ? d.wMan[world + 1] : d.ctr[C_LIVE];
        const int nf = nForcesDev(d);
        const int f0 = COLOURS && r.multiWorld ? firstForce(d, nf, base) : 0, f1 = COLOURS && r.multiWorld ? firstForce(d, nf, end) : nf;
        int *deepest = d.wMaxDepth + 2 * world;
        if (tid == 0) {
            d.wActive[world] = 0;
            deepest[0] = deepest[1] = 0;
        }
        clusterSync(size);
        for (int step = 0;; step++) {
            const bool finished = step == r.substeps;
            if (step > 0 && !finished)
                for (int m = m0 + tid; m < m1; m += threads)
                    rebaseAt(d, p, m);
            for (int m = m0 + tid; m < m1; m += threads) {
                projActiveAt(d, m);
                d.specPred[m] = make_int2(-1, -1);
            }
            clusterSync(size);
            if (r.brake) {
                const real window = r.substeps > 1 && !finished ? r.dt * static_cast<real>(r.substeps - step) : p.collisionDt;
                for (int g = base + tid; g < end; g += threads)
                    if (movable(d, g))
                        brakePredecessors(d, m0, g);
                for (int m = m0 + tid; m < m1; m += threads)
                    if (d.mSpec[m])
                        brakePrepareAt(d, m, window);
                clusterSync(size);
                if (rank == 0)
                    brakeSweep(d, base, end - base, m0, m1 - m0, arrayAt<real>(smem, 0), d.mActive + m0,
                               [&](int g, q4 &q, f3 &moment) {
                                   q = asq(d.q[g]);
                                   moment = xyz(d.moment[g]);
                               });
                clusterSync(size);
            }
            if (finished)
                break;
            if (r.stampSolve && tid == 0)
                stampSolve(d);
            for (int g = base + tid; g < end; g += threads)
                warmstartAt(d, p, g);
            clusterSync(size);
            for (int m = m0 + tid; m < m1; m += threads)
                stampsAt(d, p, 0, m);
            clusterSync(size);
            for (int it = 0; it < r.rounds; it++) {
                const bool newton = it < r.newtonRounds;
                if (newton) {
                    if (COLOURS) {
                        for (int c = 0; c < kMaxColours; c++) {
                            if (d.colourCount[c] == 0)
                                continue;
                            for (int g = base + tid; g < end; g += threads)
                                if (inUpdate(d, g) && d.colour[g] == c)
                                    colourBodyAt(d, p, g, it > 0 ? 1 : 0);
                            clusterSync(size);
                        }
                        for (int m = m0 + tid; m < m1; m += threads)
                            stampsAt(d, p, 1, m);
                        clusterSync(size);
                    }
                    for (int g = base + tid; g < end; g += threads)
                        solveAt<COLOURS, false>(d, p, g, f1 > f0 ? 0 : 1);
                    clusterSync(size);
                    if (COLOURS && f1 > f0) {
                        for (int g = base + tid; g < end; g += threads)
                            overflowApplyAt(d, p, g);
                        clusterSync(size);
                    }
                }
                const real decay = newton ? 1.0f : p.stiffnessDecay;
                for (int m = m0 + tid; m < m1; m += threads) {
                    if (it + 1 < r.newtonRounds)
                        dualAt<true, ARM, false>(d, p, decay, m);
                    else
                        dualAt<false, ARM, false>(d, p, decay, m);
                }
                if (COLOURS)
                    for (int f = f0 + tid; f < f1; f += threads)
                        forceDualAt(d, p, f);
                clusterSync(size);
            }
            for (int g = base + tid; g < end; g += threads)
                finishAt(d, p, g, step + 1 == r.substeps ? 1 : 0);
            clusterSync(size);
        }
        if (r.project && *const_cast<volatile int *>(d.wActive + world))
            for (int it = 0; it < p.projIters; it++) {
                for (int m = m0 + tid; m < m1; m += threads) {
                    int of = -1, depthBits = 0;
                    projManifoldAt(d, p, m, of, depthBits);
                    if (of >= 0)
                        atomicMax(deepest + (it & 1), depthBits);
                }
                clusterSync(size);
                const bool last = bitsf(*const_cast<volatile int *>(deepest + (it & 1))) <= r.tolerance;
                for (int g = base + tid; g < end; g += threads)
                    projBodyAt(d, p, g);
                if (tid == 0)
                    deepest[(it + 1) & 1] = 0;
                clusterSync(size);
                if (last)
                    break;
            }
        for (int m = m0 + tid; m < m1; m += threads)
            rebaseAt(d, p, m);
        clusterSync(size);
    }
}

using WorldKernel = void (*)(Dev, StepParams, WorldRun);

WorldKernel worldKernelFor(bool colours, bool arm) {
    return colours ? (arm ? worldKernel<true, true> : worldKernel<true, false>)
                   : (arm ? worldKernel<false, true> : worldKernel<false, false>);
}

WorldKernel wideKernelFor(bool colours, bool arm) {
    return colours ? (arm ? worldWideKernel<true, true> : worldWideKernel<true, false>)
                   : (arm ? worldWideKernel<false, true> : worldWideKernel<false, false>);
}

// Dynamic shared memory a CTA may have beside the static part, of 227 KB together.
#ifdef AVBDG_FP64
constexpr int kSmemMost = 221 * 1024;
#else
constexpr int kSmemMost = 222 * 1024;
#endif

} // namespace

int worldTeamMax() {
    static PerDevice teams;
    return teams.get(currentDevice(), [] {
        int team = kMaxTeam;
        for (int c = 0; c < 4; c++) {
            team = std::min(team, allowTeam(reinterpret_cast<const void *>(worldKernelFor(c & 1, c & 2)), kMaxWorldThreads, kSmemMost));
            team = std::min(team, allowTeam(reinterpret_cast<const void *>(wideKernelFor(c & 1, c & 2)), kWideThreads, kSmemMost));
        }
        return team;
    });
}

namespace {

// CTAs a world: enough that a CTA has about 24 bodies (their contacts then take one pass of its
// contact warps), as far as the GPU's SMs go round the worlds (a CTA fills one).
int worldTeam(int worlds, int bodies) {
    const int largest = worldTeamMax(), sms = smCount();
    int team = 1;
    while (team < largest && team * 24 < bodies && 2 * team * worlds <= sms)
        team *= 2;
    return team;
}

int worldThreads(int team, int bodies) { return bodies > 64 * team ? 384 : kMaxWorldThreads; }

size_t worldRows(int threads) { return sizeof(real) * static_cast<size_t>(threads / 4 * 3) * kRowReals; }

} // namespace

// A launch takes as long as its largest world, a fixed part and about 2 us a body of its CTAs; the
// separate launches take about 0.45-0.65 ms a step on these stores whatever their worlds are. Measured,
// microseconds a step here and there:
//   one world     211 bodies 286 / 456, 1261 (walls) 483 / 536, 2000 (pile) 578 / 676; where the parts do
//                 not fit in shared memory, 1681 (walls) 637 / 551, 3000 (pile) 775 / 754
//   with forces   600 bodies with ragdolls and springs 703 / 1680, a 1653-box pile with a chain 673 / 915
//   many worlds   64 of 8-64 bodies 300 / 537, 256 of them 461 / 606, 512: 622 / 650, 1024: 945 / 751;
//                 128 of 8-128 539 / 525, 64 of 8-256 540 / 528 (both 128 bodies a CTA)
//   some worlds   32 of 64-512 353 / 540, 16 of 64-1024 394 / 527, 8 of 256-2048 415 / 533, 4 of 500-2048
//                 387 / 509 (all 128 bodies a CTA); 9 of 1000-2048 (256 a CTA, too many for one) 685 / 586
// So worlds of up to 72 bodies a CTA, or 128 where four CTAs and more share a world, in up to three waves of
// CTAs, and a single world while it fits.
// The fit is an estimate, from the store's mean density and without the terms of bodies that are coloured though no
// force touches them (contact_only_overflow 0), and the host is not told which worlds did not fit. It need not be:
// worldWideKernel, to which they are left, took no longer than the separate launches in any store tried:
//   uneven worlds 300 bodies within one another and 1200 apart 902 / 1050, 16 worlds of 500 with 120 so 542 / 591
//   all coloured  900 bodies 1025 / 2612, 1100: 1526 / 2601, 2000: 2690 / 3024, 8 worlds of 900 1344 / 3212, 4 of 1900
//                 3100 / 3322
//   with forces   150 bodies within one another, 12 forces 1074 / 3181, 100 forces 2153 / 3404
bool worldsTake(int worlds, int bodies, double density, double forces) {
    const int team = worldTeam(worlds, bodies), per = divUp(bodies, team);
    if (worlds * team > 3 * smCount() || (worlds > 1 && per > (team >= 4 ? 128 : 72)))
        return false;
    // Shared memory a CTA needs: its bodies, their stamp records (two a manifold), its manifolds and
    // their contacts (four a manifold and what packing leaves empty).
    // With forces: a second block, and about eight terms a side of each.
    const double body = sizeof(real) * kBlkReals * (forces > 0 ? 2 : 1) + kF4 * (kConF4 + kRecF4) + 8 + forces * 16 * (sizeof(Term) + 2);
    const double manifold = 2.0 * kF4 * kStampF4 + kF4 * 3 + 28 + 4.7 * (kF4 * 5 + 2);
    return worldRows(worldThreads(team, bodies)) + per * (body + density * manifold) < 0.99 * kSmemMost;
}

void launchWorlds(const Dev &d, const StepParams &p, const WorldRun &run, int worlds, int bodies, cudaStream_t s) {
    const int team = worldTeam(worlds, bodies);
    const int threads = worldThreads(team, bodies);
    WorldRun r = run;
    r.rowBytes = static_cast<unsigned>(worldRows(threads));
    r.smemBytes = kSmemMost;
    const TeamLaunch l(team, worlds, threads, r.smemBytes, s);
    ++launchCount();
    cudaLaunchKernelEx(&l.cfg, worldKernelFor(r.colours, p.armCache != 0), d, p, r);
    const TeamLaunch wide(team, worlds, kWideThreads, sizeof(real) * kVelReals * static_cast<size_t>(bodies), s);
    ++launchCount();
    cudaLaunchKernelEx(&wide.cfg, wideKernelFor(r.colours, p.armCache != 0), d, p, r);
}

} // namespace avbdg
