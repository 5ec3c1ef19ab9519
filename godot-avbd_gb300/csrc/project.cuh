// Device functions of the speculative brake and the positional projection, shared by the separate
// launches (k_proj.cu) and the per-world launch (k_world.cu) (godot-avbd
// src/avbd/solver_projection.cpp:67-281).
#pragma once

#include "kernels.cuh"

namespace avbdg {

namespace {

// Whether body g joins the step's update set (solver_solve.cpp:296-339): movable bodies (`dyn`), minus idle
// sleepers (mode 1) and untouched, motionless bodies that start asleep (mode 2); a mode-2 sleeper
// otherwise wakes here. Reads the adjacency of this step.
__device__ __forceinline__ bool selectBody(const Dev &d, int g, bool dyn) {
    if (!dyn)
        return false;
    const int mode = (d.meta[g].w >> 16) & 0x3;
    const int2 s = d.sleep[g];
    if (mode == 1)
        return s.x == 0;
    if (mode == 2) {
        if (!s.x && length2(xyz(d.v[g])) == 0.0f && d.adjStart[g] == d.adjStart[g + 1])
            return false;
        if (s.x)
            d.sleep[g] = make_int2(0, s.y);
    }
    return true;
}

// Movable and in this step's update set (solver_projection.cpp:87, 105-106, 194-195).
__device__ __forceinline__ bool movable(const Dev &d, int g) { return d.x[g].w > 0.0f && inUpdate(d, g); }

__device__ __forceinline__ real angularCompliance(f3 I, f3 axis) {
    real sum = 0.0f;
    if (I.x > 0.0f)
        sum += axis.x * axis.x / I.x;
    if (I.y > 0.0f)
        sum += axis.y * axis.y / I.y;
    if (I.z > 0.0f)
        sum += axis.z * axis.z / I.z;
    return sum;
}

__device__ __forceinline__ f3 angularResponse(f3 I, q4 q, f3 axis) {
    f3 out{0.0f, 0.0f, 0.0f};
    if (I.x > 0.0f)
        out.x = axis.x / I.x;
    if (I.y > 0.0f)
        out.y = axis.y / I.y;
    if (I.z > 0.0f)
        out.z = axis.z / I.z;
    return qrot(q, out);
}

// The same with the moments' reciprocals found ahead of the quotients (dmath.cuh), where one thread's
// chain of divisions is what a sweep waits for.
struct Inertia {
    f3 I;
    Divisor x, y, z;
    bool ok;
};

__device__ __forceinline__ Inertia inertia(f3 I) {
    Inertia r;
    r.I = I;
    r.ok = true;
    // A moment that is not positive takes no quotient: any divisor will do.
    r.x = divisor(I.x > 0.0f ? I.x : 1.0f, r.ok);
    r.y = divisor(I.y > 0.0f ? I.y : 1.0f, r.ok);
    r.z = divisor(I.z > 0.0f ? I.z : 1.0f, r.ok);
    return r;
}

// a / moments, component by component, where the moment is positive (0 elsewhere).
__device__ __forceinline__ f3 perInertia(const Inertia &I, f3 a) {
    bool ok = I.ok;
    f3 q{quotient(a.x, I.x, ok), quotient(a.y, I.y, ok), quotient(a.z, I.z, ok)};
    if (!ok)
        q = f3{a.x / I.I.x, a.y / I.I.y, a.z / I.I.z};
    return f3{I.I.x > 0.0f ? q.x : 0.0f, I.I.y > 0.0f ? q.y : 0.0f, I.I.z > 0.0f ? q.z : 0.0f};
}

__device__ __forceinline__ real angularCompliance(const Inertia &I, f3 axis) {
    const f3 q = perInertia(I, cmul(axis, axis));
    real sum = 0.0f;
    if (I.I.x > 0.0f)
        sum += q.x;
    if (I.I.y > 0.0f)
        sum += q.y;
    if (I.I.z > 0.0f)
        sum += q.z;
    return sum;
}

__device__ __forceinline__ f3 angularResponse(const Inertia &I, q4 q, f3 axis) { return qrot(q, perInertia(I, axis)); }

// ---- projection (solver_projection.cpp:169-280) ----

// projectionActive membership and "can brake" (an open gap at the current poses).
__device__ __forceinline__ void projActiveAt(Dev d, int m) {
    if (m >= d.ctr[C_LIVE])
        return;
    const ManifoldBuf L = d.live;
    const int2 ab = L.ab[m];
    const int n = L.count[m];
    const bool active = n > 0 && (movable(d, ab.x) || movable(d, ab.y));
    uint8_t spec = 0;
    if (active) {
        int *flag = &d.wActive[d.meta[ab.x].x]; // a flag: one store, no atomic traffic on a shared word
        if (*flag == 0)
            *flag = 1;
        const f3 nrm = xyz(L.b0[m]);
        const f3 xa = xyz(d.x[ab.x]), xb = xyz(d.x[ab.y]);
        const q4 qa = asq(d.q[ab.x]), qb = asq(d.q[ab.y]);
        for (int k = 0; k < n; k++) {
            const int ci = cslot(d, m, k);
            const f3 rA = qrot(qa, xyz(L.rA[ci]));
            const f3 rB = qrot(qb, xyz(L.rB[ci]));
            const real gap = dot(nrm, sub(add(xa, rA), add(xb, rB)));
            if (gap > 0.0f) {
                spec = 1;
                break;
            }
        }
    }
    d.mSpec[m] = spec;
    d.mActive[m] = spec;
}

// Returns the patch's mean depth bits for the world's early-exit maximum through `depthBits`
// (left alone when the manifold corrects nothing).
__device__ __forceinline__ void projManifoldAt(Dev d, StepParams p, int m, int &world, int &depthBits) {
    if (m >= d.ctr[C_LIVE])
        return;
    const ManifoldBuf L = d.live;
    const int2 ab = L.ab[m];
    const int a = ab.x, b = ab.y;
    const int w = d.meta[a].x;
    if (d.wStop[w]) // a stopped world's bodies skip the body pass, which reads these entries
        return;
    // The adjacency entries of sides A and B; only bodies with mass have entries (a static side's
    // slot is not written by the adjacency build and is not touched here).
    const int2 slot = d.stampSlot[m];
    const real4 xa4 = d.x[a], xb4 = d.x[b];
    if (xa4.w > 0.0f)
        d.projLin[slot.x].w = 0.0f;
    if (xb4.w > 0.0f)
        d.projLin[slot.y].w = 0.0f;
    const bool moveA = movable(d, a), moveB = movable(d, b);
    const int n = L.count[m];
    if (n == 0 || (!moveA && !moveB))
        return;
    const real invMassA = moveA ? 1.0f / xa4.w : 0.0f;
    const real invMassB = moveB ? 1.0f / xb4.w : 0.0f;
    const f3 nrm = xyz(L.b0[m]);
    const q4 qa = asq(d.q[a]), qb = asq(d.q[b]);
    const f3 xa = xyz(xa4), xb = xyz(xb4);
    const m3 rotA = qmat(qa), rotB = qmat(qb);
    f3 patchRA{0, 0, 0}, patchRB{0, 0, 0};
    real patchDepth = 0.0f;
    int corrected = 0;
    for (int k = 1; k < n; k++) { // the later contacts' arms, requested before the in-order loop
        prefetchL1(&L.rA[cslot(d, m, k)]);
        prefetchL1(&L.rB[cslot(d, m, k)]);
    }
    for (int k = 0; k < n; k++) {
        const int ci = cslot(d, m, k);
        const f3 rA = mul(rotA, xyz(L.rA[ci]));
        const f3 rB = mul(rotB, xyz(L.rB[ci]));
        const real rawDepth = -dot(nrm, sub(add(xa, rA), add(xb, rB)));
        const real depth = rawDepth - p.projSlop;
        if (depth > 0.0f) {
            patchRA = add(patchRA, rA);
            patchRB = add(patchRB, rB);
            patchDepth += depth;
            corrected++;
        }
    }
    if (corrected == 0)
        return;
    const real invN = 1.0f / static_cast<real>(corrected);
    world = w;
    depthBits = fbits(patchDepth * invN); // positive: the bits order like the floats
    const f3 IA = xyz(d.moment[a]), IB = xyz(d.moment[b]);
    const f3 tA = moveA ? qrot(qconj(qa), cross(scale(patchRA, invN), nrm)) : f3{0, 0, 0};
    const f3 tB = moveB ? qrot(qconj(qb), cross(scale(patchRB, invN), nrm)) : f3{0, 0, 0};
    const real K = invMassA + invMassB + (moveA ? angularCompliance(IA, tA) : 0.0f) +
                    (moveB ? angularCompliance(IB, tB) : 0.0f);
    const real dp = p.projBeta * patchDepth * invN / K;
    if (moveA) {
        d.projLin[slot.x] = f4(scale(nrm, invMassA * dp), 1.0f);
        d.projAng[slot.x] = f4(scale(angularResponse(IA, qa, tA), dp), 0.0f);
    }
    if (moveB) {
        d.projLin[slot.y] = f4(scale(nrm, invMassB * dp), -1.0f);
        d.projAng[slot.y] = f4(scale(angularResponse(IB, qb, tB), dp), 0.0f);
    }
}

// One body's averaged correction of a pass: its contributions in adjacency order, capped, applied.
__device__ __forceinline__ void projBodyAt(const Dev &d, const StepParams &p, int g) {
    // The checks' loads go out together (valid reads of body g), then its world's stop flag.
    const int world = d.meta[g].x;
    const real mass = d.x[g].w;
    const bool updated = inUpdate(d, g);
    if ((world < 0) | !((mass > 0.0f) & updated))
        return;
    if (d.wStop[world])
        return;
    const int nf = d.ctr[C_FORCES];
    f3 sl{0, 0, 0}, sa{0, 0, 0};
    int cnt = 0;
    // Each manifold entry holds the contribution for this body (w: +1 side A, -1 side B, 0 none).
    for (int e = d.adjStart[g]; e < d.adjStart[g + 1]; e++) {
        if (nf > 0 && static_cast<int>(d.adjSeq[e]) < nf)
            continue;
        const real4 cl = d.projLin[e];
        if (cl.w == 0.0f)
            continue;
        const f3 ca = xyz(d.projAng[e]);
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
    const int locks = d.meta[g].w;
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
    const real4 x4 = d.x[g];
    d.x[g] = f4(add(xyz(x4), dl), x4.w);
    d.q[g] = f4(qintegrate(asq(d.q[g]), da));
}

// ---- rebase (ManifoldStore::rebase, manifold.cpp:448-461) ----

// mul(basis, v) with the basis stored as rows.
__device__ __forceinline__ f3 basisMul(f3 r0, f3 r1, f3 r2, f3 v) {
    return f3{(r0.x * v.x + r0.y * v.y) + r0.z * v.z, (r1.x * v.x + r1.y * v.y) + r1.z * v.z,
              (r2.x * v.x + r2.y * v.y) + r2.z * v.z};
}

__device__ __forceinline__ void rebaseAt(Dev d, StepParams p, int m) {
    if (m >= d.ctr[C_LIVE])
        return;
    const ManifoldBuf L = d.live;
    const int2 ab = L.ab[m];
    const f3 xa = xyz(d.x[ab.x]), xb = xyz(d.x[ab.y]);
    const q4 qa = asq(d.q[ab.x]), qb = asq(d.q[ab.y]);
    const f3 r0 = xyz(L.b0[m]), r1 = xyz(L.b1[m]), r2 = xyz(L.b2[m]);
    const int n = L.count[m];
    for (int c = 0; c < n; c++) {
        const int ci = cslot(d, m, c);
        const f3 pA = add(xa, qrot(qa, xyz(L.rA[ci])));
        const f3 pB = add(xb, qrot(qb, xyz(L.rB[ci])));
        f3 C0 = add(basisMul(r0, r1, r2, sub(pA, pB)), f3{COLLISION_MARGIN, 0, 0});
        if (C0.x < -p.maxPen)
            C0.x = -p.maxPen;
        L.C0[ci] = f4(C0, 0.0f);
    }
}

} // namespace

} // namespace avbdg
