// Colour sweeps without barriers: the warm start and the solve sweeps of the
// manifolds outside island groups, and of islands too large for one CTA's
// shared memory, ordered visit by visit.
//
// The colour-ordered Gauss-Seidel sequence only orders two visits when they
// share a dynamic body.  A launch (or a grid barrier) per colour orders all of
// them: a sweep of a few thousand manifolds costs the launch, and one of
// sixty thousand leaves the last wave of every colour half empty.  Here each
// body's velocity carries a tag, in the fourth word of its linear and of its
// angular 16-byte word, that names the visit whose turn it is: the manifold's
// place among the body's manifolds in slot order, plus the sweep times their
// number.  A visit starts when both bodies' words name it, and leaves them
// naming the next.  The sequence at each body is the colour order's, so the
// results are the same bits.
//
// A manifold that stops being active (half of them by the last sweep of a
// resting pile) has nothing to do in later sweeps.  The tag of a body with up
// to kFlowMask manifolds therefore also carries the set of those still active,
// and the turn passes over the others; only the visit whose turn it is
// changes the set.
//
// Velocity and tag travel in one 128-bit relaxed access, which is single-copy
// atomic: a word with the expected tag holds the velocity that goes with it,
// and no fence is needed.  Everything else a visit writes (impulses, state) is
// read again only by the same thread, or after the launch.
//
// Progress: a warp takes its 16-slot chunks of one colour in sweep-major,
// colour-major order, and the launch is cooperative, so every warp is
// resident; the earliest unfinished chunk never waits for a later one.  A
// wait that sees no tag change for kFlowSpinLimit polls reports a timeout
// and ends its warp.
#include <cuda_runtime.h>

#include <algorithm>
#include <type_traits>
#include <vector>

#include "../../include/bepugpu.h"
#include "bepugpu_internal.h"
#include "groups_device.cuh"
#include "solver_device.cuh"

namespace bepugpu {

namespace {

constexpr int kFlowThreads = 128;
constexpr int kFlowChunk = 16;  // manifolds a warp visits at once, two lanes each
constexpr int kFlowSpinLimit = 1 << 21;

// A body's word: its velocity and its tag.
__device__ __forceinline__ float4 LoadWord(const float4* p) {
    unsigned long long lo, hi;
    asm volatile("{\n\t.reg .b128 q;\n\tld.relaxed.gpu.global.b128 q, [%2];\n\tmov.b128 {%0, %1}, q;\n\t}"
                 : "=l"(lo), "=l"(hi)
                 : "l"(p)
                 : "memory");
    return make_float4(__uint_as_float((unsigned)lo), __uint_as_float((unsigned)(lo >> 32)),
                       __uint_as_float((unsigned)hi), __uint_as_float((unsigned)(hi >> 32)));
}
__device__ __forceinline__ void StoreWord(float4* p, float4 v, unsigned tag) {
    const unsigned long long lo = ((unsigned long long)__float_as_uint(v.y) << 32) | __float_as_uint(v.x);
    const unsigned long long hi = ((unsigned long long)tag << 32) | __float_as_uint(v.z);
    asm volatile("{\n\t.reg .b128 q;\n\tmov.b128 q, {%1, %2};\n\tst.relaxed.gpu.global.b128 [%0], q;\n\t}" ::"l"(p),
                 "l"(lo), "l"(hi)
                 : "memory");
}

// Tags.  A body with at most kFlowMask manifolds, in a step of at most
// kFlowMaskSweeps sweeps: the turn (sweep times the body's manifolds plus the
// place) in the low 16 bits, the active manifolds' places above.  Others: the
// turn in all 32 bits.
constexpr unsigned kFlowMask = 16, kFlowMaskSweeps = 4095;
__device__ __forceinline__ bool Masked(unsigned degree, unsigned sweeps) {
    return degree <= kFlowMask && sweeps <= kFlowMaskSweeps;
}
// One end of a visit: its body's words and the turn it waits for.
struct FlowEnd {
    float4 v, w;
    unsigned degree, place, turn;
    bool masked, ready;
    __device__ __forceinline__ void Poll(const FlowTables& f, int body) {
        v = LoadWord(f.lin + body);
        w = LoadWord(f.ang + body);
        const unsigned tag = __float_as_uint(v.w);
        ready = tag == __float_as_uint(w.w) && (masked ? tag & 0xffffu : tag) == turn;
    }
    // The words after the visit, naming the body's next one; true when the
    // body has none left.
    __device__ __forceinline__ bool Pass(const FlowTables& f, int body, bool active, unsigned t, unsigned sweeps) {
        const unsigned tag = __float_as_uint(v.w);
        unsigned next;
        bool done;
        if (masked) {
            unsigned set = tag >> 16;
            if (!active) set &= ~(1u << place);
            const unsigned later = set & ~((2u << place) - 1u);  // after this one in the sweep
            const unsigned sweep = later ? t : t + 1;
            next = (set << 16) | (sweep * degree + (unsigned)__ffs((int)(later ? later : set)) - 1u);
            done = set == 0 || sweep >= sweeps;
        } else {
            next = turn + 1;
            done = next == sweeps * degree;
        }
        StoreWord(f.lin + body, v, next);
        StoreWord(f.ang + body, w, next);
        return done;
    }
};

// After the prestep: numbers each body's manifolds that have anything to
// solve (a manifold without an active child leaves its bodies as they are in
// every sweep) in slot order, and gives the body's first one the turn.
// list (null: every body): the n bodies to number.
__global__ void k_flow_order(ManifoldSoA m, BodySoA b, FlowTables f, const int32_t* __restrict__ list, int bodies,
                             unsigned first, unsigned sweeps) {
    const int q = blockIdx.x * blockDim.x + threadIdx.x;
    if (q >= bodies) return;
    const int i = list ? list[q] : q;
    const int begin = f.csrBegin[i], end = f.csrBegin[i + 1];
    unsigned n = 0;
    for (int k = begin; k < end; k++) {
        const int e = f.csr[k];
        const uint2 st = m.state[e >> 1];
        const bool on = (st.x & kGroupActive) && st.y != ~0u;
        ((int*)f.visit)[e] = on ? (int)n : -1;
        n += on ? 1 : 0;
    }
    if (!n) return;
    f.degree[i] = (int)n;
    const unsigned turn = first * n, tag = Masked(n, sweeps) ? (((1u << n) - 1u) << 16) | turn : turn;
    const float4 v = b.vlin[i], w = b.vang[i];
    f.lin[i] = make_float4(v.x, v.y, v.z, __uint_as_float(tag));
    f.ang[i] = make_float4(w.x, w.y, w.z, __uint_as_float(tag));
}

// One end's share of a manifold's visit.  Lanes 2 i and 2 i + 1 of a warp run
// one visit: the even lane holds body A, the odd one body B.  Each computes
// its body's half of every relative velocity and applies its body's half of
// every impulse; the halves meet in one shuffle, and both lanes then run the
// same child arithmetic on the same values (the sums commute, and a sign
// multiplies exactly, so every bit is SolveManifold's).  A visit is one chain
// of dependent operations, so half the instructions in it is what shortens a
// turn; the lanes' loads halve with them.
struct HalfLanes {
    float4 j0[4];       // linear jacobian of this end (B: A's negated), w = bias
    float4 j[4];        // angular jacobian, w = softness
    float v2i[4];
    float4 r, l1, l2;   // sliding: signed arm, w = friction; rows of linear A, w = M12, M21
    float4 row1, row2;  // angular rows, w = M22, twist velocityToImpulse
    float4 n, lev;      // twist: axis, w = friction; lever arms
    float m11;
    float4 acc, f;      // accumulated impulses
};
__device__ __forceinline__ float OfA(float own, bool second) {  // lane A's value, in both lanes
    const float other = __shfl_xor_sync(0xffffffffu, own, 1);
    return second ? other : own;
}
__device__ __forceinline__ float OfB(float own, bool second) {
    const float other = __shfl_xor_sync(0xffffffffu, own, 1);
    return second ? own : other;
}
__device__ __forceinline__ float4 Signed(float4 v, float sign) {
    return make_float4(sign * v.x, sign * v.y, sign * v.z, v.w);
}
// Every lane of the warp calls it (shuffles); a manifold's two lanes pass the
// same st and children.
__device__ __forceinline__ void LoadHalf(const ManifoldSoA& m, int s, uint32_t st, uint32_t children, bool second,
                                         HalfLanes& H) {
    const int cap = m.capacity;
    const float sign = second ? -1.f : 1.f;
    const bool friction = !(st & kContactFriction);
    const bool sliding = friction && ChildOn(children, kSlidingChild), twist = friction && ChildOn(children, kTwistChild);
    const float4 zero = make_float4(0.f, 0.f, 0.f, 0.f);
    if (children != ~0u) {
        H.acc = m.penacc[s];
        H.f = m.fricacc[s];
    }
#pragma unroll
    for (int k = 0; k < 4; k++) {
        const bool on = ChildOn(children, k);
        H.j0[k] = H.j[k] = zero;
        if (on || (k == 0 && twist)) H.j0[k] = m.pj0[k * cap + s];
        if (on) H.j[k] = (second ? m.pj2 : m.pj1)[k * cap + s];
    }
    H.r = H.row1 = H.row2 = zero;
    if (sliding) {
        H.r = (second ? m.s1 : m.s0)[s];
        H.l1 = m.saxis[s];
        H.l2 = m.s3[s];
    }
    if (sliding || twist) {
        H.row1 = (second ? m.s6 : m.s4)[s];
        H.row2 = (second ? m.s7 : m.s5)[s];
    }
    if (twist) H.lev = m.lever[s];
#pragma unroll
    for (int k = 0; k < 4; k++) {
        const float w = H.j[k].w;  // A: softness, B: velocityToImpulse
        H.v2i[k] = OfB(w, second);
        H.j[k].w = OfA(w, second);
    }
    H.n = make_float4(-H.j0[0].x, -H.j0[0].y, -H.j0[0].z, OfB(H.row1.w, second));
    H.row1.w = OfA(H.row1.w, second);
    H.row2.w = OfA(H.row2.w, second);
    H.m11 = OfB(H.r.w, second);
    H.r.w = OfA(H.r.w, second);
    H.r = Signed(H.r, sign);
#pragma unroll
    for (int k = 0; k < 4; k++) H.j0[k] = Signed(H.j0[k], sign);
}
__device__ __forceinline__ void ApplyHalf(BodyState& b, float impulse, float4 linear, float4 angular) {
    ApplyLinear(b, impulse * linear.x, impulse * linear.y, impulse * linear.z);
    ApplyAngular(b, impulse * angular.x, impulse * angular.y, impulse * angular.z);
}
__device__ __forceinline__ float VelocityHalf(const BodyState& b, float4 linear, float4 angular) {
    return b.vx * linear.x + b.vy * linear.y + b.vz * linear.z + b.wx * angular.x + b.wy * angular.y + b.wz * angular.z;
}
// WarmStartManifold for one end.
__device__ __forceinline__ void WarmHalf(const ManifoldSoA& m, int s, BodyState& b, uint2 state, bool second,
                                         const HalfLanes& H) {
    const int cap = m.capacity;
    const float sign = second ? -1.f : 1.f;
    const float accs[4] = {H.acc.x, H.acc.y, H.acc.z, H.acc.w};
#pragma unroll
    for (int k = 0; k < 4; k++)
        if (ChildOn(state.y, k)) ApplyHalf(b, accs[k], H.j0[k], H.j[k]);
    if (state.x & kContactFriction) {
#pragma unroll
        for (int k = 0; k < 4; k++) {
            if (!ChildOn(state.y, 4 + k)) continue;
            const float4 fr = m.cfr[k * cap + s];
            ApplyHalf(b, fr.w, Signed(fr, sign), (second ? m.cfb : m.cfa)[k * cap + s]);
        }
        return;
    }
    if (!ChildOn(state.y, kSlidingChild)) return;  // no contacts
    const float ax = H.f.x, ay = H.f.y;
    ApplyLinear(b, sign * (ax * H.l1.x + ay * H.l2.x), sign * (ax * H.l1.y + ay * H.l2.y),
                sign * (ax * H.l1.z + ay * H.l2.z));
    ApplyAngular(b, ax * H.row1.x + ay * H.row2.x, ax * H.row1.y + ay * H.row2.y, ax * H.row1.z + ay * H.row2.z);
    ApplyAngular(b, sign * (H.f.z * H.n.x), sign * (H.f.z * H.n.y), sign * (H.f.z * H.n.z));
}
// The warp's lanes whose visit solves a child (both lanes of a visit), for the
// shuffles inside SolveHalf: penetration 0..3, contact friction 0..3, sliding
// and twist apart, since a warp may hold NONCONVEX manifolds beside convex ones.
struct ChildLanes {
    unsigned penetration[4], friction[4], sliding, twist;
};
__device__ __forceinline__ ChildLanes LanesOf(uint32_t st, uint32_t children) {
    ChildLanes c;
    const bool nonConvex = st & kContactFriction;
#pragma unroll
    for (int k = 0; k < 4; k++) {
        c.penetration[k] = __ballot_sync(0xffffffffu, ChildOn(children, k));
        c.friction[k] = __ballot_sync(0xffffffffu, nonConvex && ChildOn(children, 4 + k));
    }
    c.sliding = __ballot_sync(0xffffffffu, !nonConvex && ChildOn(children, kSlidingChild));
    c.twist = __ballot_sync(0xffffffffu, !nonConvex && ChildOn(children, kTwistChild));
    return c;
}
// SolveManifold for one end.
__device__ __forceinline__ void SolveHalf(const ManifoldSoA& m, int s, BodyState& b, uint2& state, bool second,
                                          const StepParams& p, const HalfLanes& H, const ChildLanes& lanes) {
    const int cap = m.capacity;
    const float sign = second ? -1.f : 1.f;
    uint32_t st = state.x, children = state.y;
    const uint32_t iter = (st >> kIterShift) + 1;
    st = (st & 0xffffu) | (iter << kIterShift);
    const uint32_t on = children;
    uint32_t still = 0;
    auto account = [&](int c, float r) { still |= r < p.minimumImpulse ? 1u << (4 * c) : 0u; };
    auto both = [](unsigned lanesOn, float own) { return own + __shfl_xor_sync(lanesOn, own, 1); };
    float accs[4] = {H.acc.x, H.acc.y, H.acc.z, H.acc.w};
    float4 f = H.f;
#pragma unroll
    for (int k = 0; k < 4; k++) {
        if (!ChildOn(on, k)) continue;
        const float rv = both(lanes.penetration[k], VelocityHalf(b, H.j0[k], H.j[k]));
        float lambda = (rv - H.j0[k].w + H.j[k].w * accs[k]) * H.v2i[k];
        const float prev = accs[k];
        accs[k] = Maxf(0, accs[k] + lambda);
        lambda = accs[k] - prev;
        ApplyHalf(b, lambda, H.j0[k], H.j[k]);
        account(k, fabsf(lambda));
    }
    if (st & kContactFriction) {
#pragma unroll
        for (int k = 0; k < 4; k++) {
            if (!ChildOn(on, 4 + k)) continue;
            float4 fr = m.cfr[k * cap + s];
            const float4 fa = m.cfa[k * cap + s], fb = m.cfb[k * cap + s];
            const float4 own = second ? fb : fa, linear = Signed(fr, sign);
            float lambda = both(lanes.friction[k], VelocityHalf(b, linear, own)) * fa.w;
            const float prev = fr.w, maxForce = fb.w * accs[k];
            fr.w = Clampf(fr.w + lambda, -maxForce, maxForce);
            lambda = fr.w - prev;
            ApplyHalf(b, lambda, linear, own);
            account(4 + k, fabsf(lambda));
            m.cfr[k * cap + s] = fr;  // by both lanes, the same value
        }
    } else {
        if (ChildOn(on, kSlidingChild)) {
            const float dvx = both(lanes.sliding, sign * b.vx + (b.wy * H.r.z) - (b.wz * H.r.y));
            const float dvy = both(lanes.sliding, sign * b.vy + (b.wz * H.r.x) - (b.wx * H.r.z));
            const float dvz = both(lanes.sliding, sign * b.vz + (b.wx * H.r.y) - (b.wy * H.r.x));
            float lxv = dvx * H.l1.x + dvy * H.l1.y + dvz * H.l1.z;
            float lyv = dvx * H.l2.x + dvy * H.l2.y + dvz * H.l2.z;
            const float x = lxv;
            lxv = x * H.m11 + lyv * H.l2.w;       // M11, M21
            lyv = x * H.l1.w + lyv * H.row1.w;    // M12, M22
            const float px = f.x, py = f.y;
            f.x += lxv;
            f.y += lyv;
            float length = f.x * f.x + f.y * f.y;
            float maximumFrictionForce = accs[0] + accs[1] + accs[2] + accs[3];
            maximumFrictionForce *= H.r.w;
            if (length > maximumFrictionForce * maximumFrictionForce) {
                length = maximumFrictionForce / SqrtOfFloat(length);
                f.x *= length;
                f.y *= length;
            }
            lxv = f.x - px;
            lyv = f.y - py;
            ApplyLinear(b, sign * (lxv * H.l1.x + lyv * H.l2.x), sign * (lxv * H.l1.y + lyv * H.l2.y),
                        sign * (lxv * H.l1.z + lyv * H.l2.z));
            ApplyAngular(b, lxv * H.row1.x + lyv * H.row2.x, lxv * H.row1.y + lyv * H.row2.y,
                         lxv * H.row1.z + lyv * H.row2.z);
            account(kSlidingChild, fabsf(lxv) + fabsf(lyv));
        }
        if (ChildOn(on, kTwistChild)) {
            // A's part minus B's, in both lanes
            const float own = b.wx * H.n.x + b.wy * H.n.y + b.wz * H.n.z;
            const float other = __shfl_xor_sync(lanes.twist, own, 1);
            float lambda = ((second ? other : own) - (second ? own : other)) * H.row2.w;
            const float prev = f.z;
            float maximumFrictionForce =
                H.lev.x * accs[0] + H.lev.y * accs[1] + H.lev.z * accs[2] + H.lev.w * accs[3];
            maximumFrictionForce *= H.n.w;
            f.z = Clampf(f.z + lambda, -maximumFrictionForce, maximumFrictionForce);
            lambda = f.z - prev;
            ApplyAngular(b, sign * (lambda * H.n.x), sign * (lambda * H.n.y), sign * (lambda * H.n.z));
            account(kTwistChild, fabsf(lambda));
        }
    }
    st = AccountChildren(st, children, still, p);
    // both lanes write the same values, and read their own back in the next sweep
    m.penacc[s] = make_float4(accs[0], accs[1], accs[2], accs[3]);
    m.fricacc[s] = f;
    state = make_uint2(st, children);
}

// Sweeps [first, sweeps); sweep 0 is the warm start.
// Bound by the turns' latency in small and deep scenes (a visit and one trip
// through L2 per turn) and by the lanes' trips through L2 in large ones (76 MB
// a sweep at 188,667 manifolds).  128 registers, 16 warps an SM; 20 warps spill
// and measured 11 % slower.  Against launches per colour and sweep: the frame
// of a 5,750-box pile 307 -> 151 us, of a 1,000-box one (in one CTA before)
// 225 -> 104 us, four frames of the settling 65,536-box heap 4.35 -> 3.98 ms
// against one lane per manifold (8 warps an SM), the packed 65,536-box pile
// four steps 2,890 -> 1,860 us (1,973 with one lane).
__global__ void __launch_bounds__(kFlowThreads, 4) k_flow(ManifoldSoA m, BodySoA b, StepParams p, FlowTables f,
                                                       unsigned first, unsigned sweeps) {
    const int lane = threadIdx.x & 31;
    const bool second = lane & 1;  // this lane's end: A, or B
    // consecutive chunks on different CTAs: a scene of few chunks spreads over the SMs
    const int warp = (threadIdx.x >> 5) * gridDim.x + blockIdx.x, warps = gridDim.x * (kFlowThreads / 32);
    const float4 zero = make_float4(0.f, 0.f, 0.f, 0.f);
    for (unsigned t = first; t < sweeps; t++)
        for (int c = warp; c < f.chunkCount; c += warps) {
            const int2 range = f.chunks[c];
            const int s = range.x + (lane >> 1);
            const int2 visit = s < range.y ? f.visit[s] : make_int2(-1, -1);
            const bool listed = visit.x >= 0 || visit.y >= 0;
            uint2 state = listed ? m.state[s] : make_uint2(0u, ~0u);
            const bool active = state.x & kGroupActive;
            // the visit's iteration past a limit only ends the manifold (Solver.cs:285-314)
            const int iter = (int)(state.x >> kIterShift) + 1;
            const bool runs = active && (t == 0 || (iter <= p.iterationLimit && iter <= p.maximumIterationCount));
            const int4 h = listed ? m.head[s] : make_int4(-1, -1, 0, 0);
            const int body = second ? h.y : h.x;
            const bool dynamic = state.x & (second ? kDynB : kDynA);
            FlowEnd E;
            E.v = E.w = zero;
            E.place = (unsigned)(second ? visit.y : visit.x);
            const bool turns = listed && (int)E.place >= 0;
            E.degree = turns ? (unsigned)f.degree[body] : 0u;
            E.masked = Masked(E.degree, sweeps);
            E.turn = t * E.degree + E.place;
            // a stopped manifold only takes its turn at bodies without a set
            const bool at = turns && (active || !E.masked);
            if (!__any_sync(0xffffffffu, at)) continue;
            E.ready = !at;
            // everything that no other visit writes during the sweeps, before the wait
            HalfLanes H;
            const uint32_t children = runs ? state.y : ~0u;
            LoadHalf(m, s, state.x, children, second, H);
            const ChildLanes lanes = LanesOf(state.x, children);
            float4 ia = zero, ic = zero;
            float mass = 0.f, last = 0.f;  // inverse mass, inertia M33
            if (runs && !turns && body >= 0) {
                E.v = b.vlin[body];
                E.w = b.vang[body];
            }
            if (runs && dynamic) {
                ia = b.inv0[body];
                ic = b.inv1[body];
                mass = b.vlin[body].w;
                last = b.vang[body].w;
            }
            unsigned seen = 0;
            for (int spins = 0;; spins++) {
                if (!E.ready) E.Poll(f, body);
                if (__all_sync(0xffffffffu, E.ready)) break;
                const unsigned now = __float_as_uint(E.v.w) + __float_as_uint(E.w.w);
                if (__any_sync(0xffffffffu, now != seen)) spins = 0;
                seen = now;
                if (spins > kFlowSpinLimit) {
                    *(volatile int*)f.error = BEPUGPU_TIMEOUT;
                    return;
                }
            }
            if (runs) {
                BodyState own;
                MakeBody(make_float4(E.v.x, E.v.y, E.v.z, mass), make_float4(E.w.x, E.w.y, E.w.z, last), ia, ic, own);
                if (t == 0) WarmHalf(m, s, own, state, second, H);
                else SolveHalf(m, s, own, state, second, p, H, lanes);
                if (dynamic) {
                    E.v.x = own.vx; E.v.y = own.vy; E.v.z = own.vz;
                    E.w.x = own.wx; E.w.y = own.wy; E.w.z = own.wz;
                }
            } else if (active) {
                state.x = ((state.x & 0xffffu) | ((uint32_t)iter << kIterShift)) & ~kGroupActive;
            }
            // the body's last visit leaves the velocity in the scene's lanes
            if (at && E.Pass(f, body, state.x & kGroupActive, t, sweeps) && dynamic) {
                b.vlin[body] = make_float4(E.v.x, E.v.y, E.v.z, b.vlin[body].w);
                b.vang[body] = make_float4(E.w.x, E.w.y, E.w.z, b.vang[body].w);
            }
            if (active && t > 0) m.state[s] = state;
        }
}

// The body of sorted entry k: -1 before the first, `bodies` past the last.
__device__ __forceinline__ int BodyOfEntry(const unsigned long long* __restrict__ entries, int count, int bodies, int k) {
    return k < 0 ? -1 : (k < count && entries[k] != ~0ull ? (int)(entries[k] >> 32) : bodies);
}
// The tables from the constraint upload's slots [0, n) and those from g0 on: a
// (dynamic body, slot << 1 | end) entry for each end, ~0 without one, sorted by
// body.  The slots ascend and the sort is stable, so a body's entries end in
// slot order.  Nothing when the sort gave up (*err).
__global__ void k_flow_entries(ManifoldSoA m, BodySoA b, int n, int g0, int slots, unsigned long long* entries) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= slots) return;
    const int s = i < n ? i : g0 + i - n;
    const int4 h = m.head[s];
    const auto entry = [&](int body, int end) {
        const bool moves = body >= 0 && b.pos[body].w != 0.f;
        return moves ? ((unsigned long long)(unsigned)body << 32) | (unsigned)(s << 1 | end) : ~0ull;
    };
    entries[2 * (size_t)i] = entry(h.x, 0);
    entries[2 * (size_t)i + 1] = entry(h.y, 1);
}
__global__ void k_flow_slots(const unsigned long long* __restrict__ entries, int count, int bodies, FlowTables f,
                             const int* __restrict__ err) {
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k > count || *err) return;
    const int body = BodyOfEntry(entries, count, bodies, k);
    for (int i = BodyOfEntry(entries, count, bodies, k - 1) + 1; i <= body; i++) f.csrBegin[i] = k;
    if (body < bodies) f.csr[k] = (int)(entries[k] & 0xffffffffu);
}

// update_pairs' side of the tables, from its (dynamic body, entry) keys
// sorted by body: where each body's entries start, and the entries as
// slot << 1 | end in slot order.  Nothing when the slots' sort gave up (*err).
__global__ void k_flow_csr(const unsigned long long* __restrict__ entries, int count, int bodies,
                           const int2* __restrict__ ends, const int* __restrict__ slotOf, FlowTables f,
                           const int* __restrict__ err) {
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k > count || *err) return;
    // the bodies after the previous entry's, up to this one's, start here
    const int body = BodyOfEntry(entries, count, bodies, k);
    for (int i = BodyOfEntry(entries, count, bodies, k - 1) + 1; i <= body; i++) f.csrBegin[i] = k;
    if (body == bodies) return;
    const int entry = (int)(entries[k] & 0xffffffffu), slot = slotOf[entry];
    int first = k, rank = 0;
    while (first > 0 && (int)(entries[first - 1] >> 32) == body) first--;
    for (int q = first; q < count && entries[q] != ~0ull && (int)(entries[q] >> 32) == body; q++)
        rank += slotOf[(int)(entries[q] & 0xffffffffu)] < slot ? 1 : 0;
    f.csr[first + rank] = (slot << 1) | (ends[entry].x == body ? 0 : 1);
}

}  // namespace

std::vector<int2> FlowChunks(const std::vector<int32_t>& colourOffsets) {
    std::vector<int2> chunks;
    for (size_t c = 0; c + 1 < colourOffsets.size(); c++)
        for (int32_t s = colourOffsets[c]; s < colourOffsets[c + 1]; s += kFlowChunk)
            chunks.push_back(make_int2(s, std::min(s + kFlowChunk, colourOffsets[c + 1])));
    return chunks;
}

#define CK(call)                                                                              \
    do {                                                                                      \
        cudaError_t e_ = (call);                                                              \
        if (e_ != cudaSuccess) {                                                              \
            ctx->SetError("%s failed: %s (%s:%d)", #call, cudaGetErrorString(e_), __FILE__, __LINE__); \
            return BEPUGPU_CUDA_ERROR;                                                        \
        }                                                                                     \
    } while (0)

const GroupClass* FlowGroups(const GroupPlan& plan) {
    const GroupClass& c = plan.global;
    const bool large = c.end > c.begin &&
                       GroupSmemBytes(true, c.maxLocal, c.maxManifolds, 0, plan.nonConvexLanes) > kGroupSmemBudget;
    return large ? &c : nullptr;
}

// The tables' places in their block; returns the block's size.
size_t Scene::RebaseFlow() {
    const size_t B = maxBodies ? maxBodies : 1, M = maxManifolds ? maxManifolds : 1;
    size_t bytes = 0;
    auto take = [&](auto*& p, size_t n) {
        p = flowBlock ? reinterpret_cast<std::remove_reference_t<decltype(p)>>((char*)flowBlock + bytes) : nullptr;
        bytes += (n * sizeof(*p) + 255) & ~(size_t)255;
    };
    take(flow.chunks, M);
    take(flow.visit, M);
    take(flow.csr, 2 * M);
    take(flow.degree, B);
    take(flow.csrBegin, B + 1);
    take(flow.sort, SortBlocks(2 * M) * kSortBins + 1);
    take(flow.lin, B);
    take(flow.ang, B);
    return bytes;
}
bepugpu_status Scene::NeedFlow(Context* ctx) {
    if (flowBlock) return BEPUGPU_OK;
    const size_t bytes = RebaseFlow();
    const cudaError_t e = heap->Alloc(bytes, &flowBlock);
    if (e != cudaSuccess) {
        flowBlock = nullptr;
        ctx->SetError("solve sweeps: %zu bytes of tables: %s", bytes, cudaGetErrorString(e));
        return e == cudaErrorMemoryAllocation ? BEPUGPU_OUT_OF_MEMORY : BEPUGPU_CUDA_ERROR;
    }
    flowBytes = bytes;
    RebaseFlow();
    return BEPUGPU_OK;
}

// After the records' upload, whose heads and staging buffer it uses.  On the
// host, two walks over the records in slot order were a twelfth of the upload of
// a pile of 65,536 boxes: 14.8 ms, 13.7 this way.
bepugpu_status Scene::UploadFlow(Context* ctx) {
    // slots [0, n) and [g0, g1); beside joints the sweep path runs colour by colour
    const int n = groupPlan.jointGlobalCount ? 0 : groupPlan.globalCount;
    const GroupClass* large = FlowGroups(groupPlan);
    const int g0 = large ? groupPlan.groups[large->begin].mBegin : n, g1 = large ? groupPlan.groups[large->end - 1].mEnd : n;
    flow.chunkCount = flow.groupChunkCount = 0;
    if (n == 0 && g1 == g0) return BEPUGPU_OK;
    bepugpu_status st = NeedFlow(ctx);
    if (st != BEPUGPU_OK) return st;
    // the groups' chunks colour by colour over all of them
    std::vector<int2> groupChunks;
    for (int c = 0; large; c++) {
        bool any = false;
        for (int k = large->begin; k < large->end; k++) {
            const GroupDesc& g = groupPlan.groups[k];
            if (c >= g.cCount) continue;
            any = true;
            const int32_t* off = groupPlan.colourOffsets.data() + g.cBegin;
            for (int32_t s = off[c]; s < off[c + 1]; s += kFlowChunk)
                groupChunks.push_back(make_int2(g.mBegin + s, g.mBegin + std::min(s + kFlowChunk, off[c + 1])));
        }
        if (!any) break;
    }
    std::vector<int2> chunks;
    if (n) chunks = FlowChunks(manifoldOffsets);
    const size_t sweepChunks = chunks.size();
    chunks.insert(chunks.end(), groupChunks.begin(), groupChunks.end());
    st = UploadFlowChunks(ctx, chunks, groupPlan.slotOf.size());
    if (st != BEPUGPU_OK) return st;
    const int slots = n + g1 - g0, T = 256;
    const size_t keys = 2 * (size_t)slots;
    auto* entries = (unsigned long long*)staging;  // 32 bytes a slot; a manifold record is larger
    static_assert(sizeof(bepugpu_manifold) >= 32, "the entries and the sort's second buffer fit the staged records");
    int* status = flow.sort + SortBlocks(keys) * kSortBins;
    CK(cudaMemsetAsync(status, 0, sizeof(int), stream));
    CK(MarkExpired(status, BEPUGPU_WAIT_TABLES));
    k_flow_entries<<<(slots + T - 1) / T, T, 0, stream>>>(m, b, n, g0, slots, entries);
    CK(cudaGetLastError());
    CK(RadixSort(this, entries, entries + keys, nullptr, keys, SortPlan(0, 0, BitsFor((size_t)b.count + 1)),
                 (unsigned*)flow.sort, status, stream));
    k_flow_slots<<<(int)((keys + T) / T), T, 0, stream>>>(entries, (int)keys, b.count, flow, status);
    CK(cudaGetLastError());
    int gaveUp = 0;
    CK(cudaMemcpyAsync(&gaveUp, status, sizeof(int), cudaMemcpyDeviceToHost, stream));
    CK(cudaStreamSynchronize(stream));
    if (gaveUp) {
        CK(cudaMemsetAsync(SortCounter(), 0, sizeof(unsigned), stream));
        ctx->SetError("upload_constraints: the sort of the sweeps' visits did not finish");
        return BEPUGPU_TIMEOUT;
    }
    flow.chunkCount = (int)sweepChunks;
    flow.groupChunkCount = (int)groupChunks.size();
    return BEPUGPU_OK;
}

// The caller keeps the chunks until the stream has passed the copy.
bepugpu_status Scene::UploadFlowChunks(Context* ctx, const std::vector<int2>& chunks, size_t slots) {
    if (chunks.empty()) return BEPUGPU_OK;
    if (!flowStatus) CK(words->Take(&flowStatus));  // outside any stream capture
    if (!flowBlocksPerSm) CK(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&flowBlocksPerSm, k_flow, kFlowThreads, 0));
    CK(cudaHostGetDevicePointer((void**)&flow.error, flowStatus, 0));
    // the ends without a dynamic body keep visit -1
    CK(cudaMemsetAsync(flow.visit, 0xff, sizeof(int2) * slots, stream));
    CK(cudaMemcpyAsync(flow.chunks, chunks.data(), sizeof(int2) * chunks.size(), cudaMemcpyHostToDevice, stream));
    return BEPUGPU_OK;
}

bepugpu_status Scene::BuildFlowOnDevice(Context* ctx, const unsigned long long* entries, int count, const int2* ends,
                                        const int* slots, const int* status) {
    k_flow_csr<<<(count + 1 + 255) / 256, 256, 0, stream>>>(entries, count, b.count, ends, slots, flow, status);
    CK(cudaGetLastError());
    return BEPUGPU_OK;
}

bepugpu_status LaunchFlow(Context* ctx, Scene* s, const StepParams& p, bool groups, bool warm, int* launches) {
    FlowTables f = s->flow;
    const int32_t* list = nullptr;
    int nb = s->b.count;
    if (groups) {
        const GroupPlan& plan = s->groupPlan;
        const GroupDesc &first = plan.groups[plan.global.begin], &last = plan.groups[plan.global.end - 1];
        list = s->groupBodiesDev + first.bBegin;
        nb = last.bEnd - first.bBegin;
        f.chunks += f.chunkCount;
        f.chunkCount = f.groupChunkCount;
    }
    if (f.chunkCount == 0) {
        ctx->SetError("solve sweeps: no tables (the last constraint upload failed)");
        return BEPUGPU_INVALID_OPERATION;
    }
    const int resident = s->flowBlocksPerSm * ctx->smCount;
    if (resident < 1) {
        ctx->SetError("solve sweeps: no resident CTA (%d an SM of %d)", s->flowBlocksPerSm, ctx->smCount);
        return BEPUGPU_CUDA_ERROR;
    }
    const unsigned sweeps = (unsigned)p.iterationLimit + 1;
    k_flow_order<<<(nb + 127) / 128, 128, 0, s->stream>>>(s->m, s->b, f, list, nb, warm ? 0u : 1u, sweeps);
    if (launches) (*launches)++;
    cudaLaunchConfig_t cfg = {};
    // a warp per chunk on its own CTA while the CTAs last
    cfg.gridDim = dim3((unsigned)std::min(resident, f.chunkCount));
    cfg.blockDim = dim3(kFlowThreads);
    cfg.stream = s->stream;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeCooperative;
    attr[0].val.cooperative = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    // sweep 0 is the warm start
    CK(cudaLaunchKernelEx(&cfg, k_flow, s->m, s->b, p, f, warm ? 0u : 1u, sweeps));
    if (launches) (*launches)++;
    return BEPUGPU_OK;
}

bepugpu_status FlowStatus(Context* ctx, Scene* s) {
    if (!s->flowStatus || !*(volatile int*)s->flowStatus) return BEPUGPU_OK;
    *(volatile int*)s->flowStatus = 0;
    ctx->SetError("solve sweeps of scene %d: a wait for an earlier visit ran out", s->id);
    return BEPUGPU_TIMEOUT;
}

StatusWords::~StatusWords() {
    for (int* p : pages_) cudaFreeHost(p);
}
cudaError_t StatusWords::Take(int** word) {
    if (free_.empty()) {
        constexpr int kWords = 1024;
        int* page = nullptr;
        const cudaError_t e = cudaHostAlloc((void**)&page, sizeof(int) * kWords, cudaHostAllocMapped);
        if (e != cudaSuccess) return e;
        pages_.push_back(page);
        free_.reserve(kWords * pages_.size());  // Give never allocates
        for (int k = kWords - 1; k >= 0; k--) free_.push_back(page + k);
    }
    *word = free_.back();
    free_.pop_back();
    **word = 0;
    return cudaSuccess;
}

}  // namespace bepugpu
