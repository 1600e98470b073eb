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
// Progress: a warp takes its 32-slot chunks of one colour in sweep-major,
// colour-major order, and the launch is cooperative, so every warp is
// resident; the earliest unfinished chunk never waits for a later one.  A
// wait that sees no tag change for kFlowSpinLimit polls reports a timeout
// and ends its warp.
#include <cuda_runtime.h>

#include <algorithm>
#include <vector>

#include "../../include/bepugpu.h"
#include "bepugpu_internal.h"
#include "groups_device.cuh"
#include "solver_device.cuh"

namespace bepugpu {

namespace {

constexpr int kFlowThreads = 128;
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

// Sweeps [first, sweeps); sweep 0 is the warm start.
// Bound by the turns' latency in small scenes (a turn is a visit of about 1 us
// plus one trip through L2) and by the lanes' trips through L2 in large ones
// (76 MB a sweep at 188,667 manifolds).  180 registers, 8 warps an SM; held to
// 168 for 12 warps it measured 11 % slower, at 32- or 64-thread CTAs the same.
// A step of the packed piles, launches per colour against this kernel: 15,789
// manifolds 228 -> 93 us, 188,667 manifolds 590 -> 332 us (without the sets of
// active manifolds 175 and 390 us).
__global__ void __launch_bounds__(kFlowThreads) k_flow(ManifoldSoA m, BodySoA b, StepParams p, FlowTables f,
                                                       unsigned first, unsigned sweeps) {
    const int lane = threadIdx.x & 31;
    // consecutive chunks on different CTAs: a scene of few chunks spreads over the SMs
    const int warp = (threadIdx.x >> 5) * gridDim.x + blockIdx.x, warps = gridDim.x * (kFlowThreads / 32);
    const float4 zero = make_float4(0.f, 0.f, 0.f, 0.f);
    for (unsigned t = first; t < sweeps; t++)
        for (int c = warp; c < f.chunkCount; c += warps) {
            const int2 range = f.chunks[c];
            const int s = range.x + lane;
            const int2 visit = s < range.y ? f.visit[s] : make_int2(-1, -1);
            uint2 state = make_uint2(0u, 0u);
            if (visit.x >= 0 || visit.y >= 0) state = m.state[s];
            const bool active = state.x & kGroupActive;
            int4 h = make_int4(-1, -1, 0, 0);
            FlowEnd A, B;
            A.v = A.w = B.v = B.w = zero;
            A.degree = B.degree = 0;
            if (visit.x >= 0 || visit.y >= 0) {
                h = m.head[s];
                if (visit.x >= 0) A.degree = (unsigned)f.degree[h.x];
                if (visit.y >= 0) B.degree = (unsigned)f.degree[h.y];
            }
            A.masked = Masked(A.degree, sweeps);
            B.masked = Masked(B.degree, sweeps);
            // a stopped manifold only takes its turn at bodies without a set
            const bool atA = visit.x >= 0 && (active || !A.masked), atB = visit.y >= 0 && (active || !B.masked);
            if (!__any_sync(0xffffffffu, atA || atB)) continue;
            A.place = (unsigned)visit.x;
            B.place = (unsigned)visit.y;
            A.turn = t * A.degree + A.place;
            B.turn = t * B.degree + B.place;
            A.ready = !atA;
            B.ready = !atB;
            SolveLanes L;
            float4 aa = zero, ca = zero, ab = zero, cb = zero;
            float massA = 0.f, massB = 0.f, lastA = 0.f, lastB = 0.f;  // inverse mass, inertia M33
            if (active) {
                // everything that no other thread writes during the sweeps, before the wait
                LoadSolveLanes(m, s, state.x, state.y, L);
                if (visit.x < 0 && h.x >= 0) {
                    A.v = b.vlin[h.x];
                    A.w = b.vang[h.x];
                }
                if (visit.y < 0 && h.y >= 0) {
                    B.v = b.vlin[h.y];
                    B.w = b.vang[h.y];
                }
                if (state.x & kDynA) {
                    aa = b.inv0[h.x];
                    ca = b.inv1[h.x];
                    massA = b.vlin[h.x].w;
                    lastA = b.vang[h.x].w;
                }
                if (state.x & kDynB) {
                    ab = b.inv0[h.y];
                    cb = b.inv1[h.y];
                    massB = b.vlin[h.y].w;
                    lastB = b.vang[h.y].w;
                }
            }
            unsigned seen = 0;
            for (int spins = 0;; spins++) {
                if (!A.ready) A.Poll(f, h.x);
                if (!B.ready) B.Poll(f, h.y);
                if (__all_sync(0xffffffffu, A.ready && B.ready)) break;
                const unsigned now = __float_as_uint(A.v.w) + __float_as_uint(A.w.w) + __float_as_uint(B.v.w) +
                                     __float_as_uint(B.w.w);
                if (__any_sync(0xffffffffu, now != seen)) spins = 0;
                seen = now;
                if (spins > kFlowSpinLimit) {
                    *(volatile int*)f.error = BEPUGPU_TIMEOUT;
                    return;
                }
            }
            if (active) {
                BodyState bodyA, bodyB;
                MakeBody(make_float4(A.v.x, A.v.y, A.v.z, massA), make_float4(A.w.x, A.w.y, A.w.z, lastA), aa, ca, bodyA);
                MakeBody(make_float4(B.v.x, B.v.y, B.v.z, massB), make_float4(B.w.x, B.w.y, B.w.z, lastB), ab, cb, bodyB);
                if (t == 0) {
                    WarmStartManifold(m, s, bodyA, bodyB, state, L);
                } else {
                    SolveManifold(m, s, bodyA, bodyB, state, p, &L);
                    m.state[s] = state;
                }
                if (state.x & kDynA) {
                    A.v.x = bodyA.vx; A.v.y = bodyA.vy; A.v.z = bodyA.vz;
                    A.w.x = bodyA.wx; A.w.y = bodyA.wy; A.w.z = bodyA.wz;
                }
                if (state.x & kDynB) {
                    B.v.x = bodyB.vx; B.v.y = bodyB.vy; B.v.z = bodyB.vz;
                    B.w.x = bodyB.wx; B.w.y = bodyB.wy; B.w.z = bodyB.wz;
                }
            }
            const bool still = state.x & kGroupActive;  // active in the next sweep
            // the body's last visit leaves the velocity in the scene's lanes
            if (atA && A.Pass(f, h.x, still, t, sweeps) && (state.x & kDynA)) {
                b.vlin[h.x] = make_float4(A.v.x, A.v.y, A.v.z, b.vlin[h.x].w);
                b.vang[h.x] = make_float4(A.w.x, A.w.y, A.w.z, b.vang[h.x].w);
            }
            if (atB && B.Pass(f, h.y, still, t, sweeps) && (state.x & kDynB)) {
                b.vlin[h.y] = make_float4(B.v.x, B.v.y, B.v.z, b.vlin[h.y].w);
                b.vang[h.y] = make_float4(B.w.x, B.w.y, B.w.z, b.vang[h.y].w);
            }
        }
}

// update_pairs' side of the tables, from its (dynamic body, entry) keys
// sorted by body: where each body's entries start, and the entries as
// slot << 1 | end in slot order.
__device__ __forceinline__ int BodyOfEntry(const unsigned long long* __restrict__ entries, int count, int bodies, int k) {
    return k < 0 ? -1 : (k < count && entries[k] != ~0ull ? (int)(entries[k] >> 32) : bodies);
}
__global__ void k_flow_csr(const unsigned long long* __restrict__ entries, int count, int bodies,
                           const int2* __restrict__ ends, const int* __restrict__ slotOf, FlowTables f) {
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k > count) return;
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
        for (int32_t s = colourOffsets[c]; s < colourOffsets[c + 1]; s += 32)
            chunks.push_back(make_int2(s, std::min(s + 32, colourOffsets[c + 1])));
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

bepugpu_status Scene::UploadFlow(Context* ctx, const int32_t* a, const int32_t* b) {
    // slots [0, n) and [g0, g1)
    const int n = groupPlan.globalCount;
    const GroupClass* large = FlowGroups(groupPlan);
    const int g0 = large ? groupPlan.groups[large->begin].mBegin : n, g1 = large ? groupPlan.groups[large->end - 1].mEnd : n;
    flow.chunkCount = flow.groupChunkCount = 0;
    if (n == 0 && g1 == g0) return BEPUGPU_OK;
    std::vector<int32_t> recordOf(groupPlan.slotOf.size(), -1);
    for (size_t i = 0; i < groupPlan.slotOf.size(); i++) recordOf[groupPlan.slotOf[i]] = (int32_t)i;
    const int nb = this->b.count;
    std::vector<int32_t> begin(nb + 1, 0);
    auto moving = [&](int32_t e) { return e >= 0 && hostDynamic[e]; };
    auto slots = [&](auto visit) {
        for (int s = 0; s < n; s++) visit(s, a[recordOf[s]], b[recordOf[s]]);
        for (int s = g0; s < g1; s++) visit(s, a[recordOf[s]], b[recordOf[s]]);
    };
    slots([&](int, int32_t x, int32_t y) {
        if (moving(x)) begin[x + 1]++;
        if (moving(y)) begin[y + 1]++;
    });
    for (int i = 0; i < nb; i++) begin[i + 1] += begin[i];
    std::vector<int32_t> at(begin.begin(), begin.end() - 1), csr(begin[nb]);
    slots([&](int s, int32_t x, int32_t y) {
        if (moving(x)) csr[at[x]++] = s << 1;
        if (moving(y)) csr[at[y]++] = (s << 1) | 1;
    });
    CK(cudaMemcpyAsync(flow.csrBegin, begin.data(), sizeof(int32_t) * begin.size(), cudaMemcpyHostToDevice, stream));
    CK(cudaMemcpyAsync(flow.csr, csr.data(), sizeof(int32_t) * csr.size(), cudaMemcpyHostToDevice, stream));
    // the groups' chunks colour by colour over all of them
    std::vector<int2> groupChunks;
    for (int c = 0; large; c++) {
        bool any = false;
        for (int k = large->begin; k < large->end; k++) {
            const GroupDesc& g = groupPlan.groups[k];
            if (c >= g.cCount) continue;
            any = true;
            const int32_t* off = groupPlan.colourOffsets.data() + g.cBegin;
            for (int32_t s = off[c]; s < off[c + 1]; s += 32)
                groupChunks.push_back(make_int2(g.mBegin + s, g.mBegin + std::min(s + 32, off[c + 1])));
        }
        if (!any) break;
    }
    return UploadFlowChunks(ctx, groupChunks);
}

bepugpu_status Scene::UploadFlowChunks(Context* ctx, const std::vector<int2>& groupChunks) {
    std::vector<int2> chunks = FlowChunks(manifoldOffsets);
    flow.chunkCount = (int)chunks.size();
    flow.groupChunkCount = (int)groupChunks.size();
    chunks.insert(chunks.end(), groupChunks.begin(), groupChunks.end());
    if (chunks.empty()) return BEPUGPU_OK;
    if (!ctx->flowError) {  // once a context, outside any stream capture
        CK(cudaHostAlloc((void**)&ctx->flowError, sizeof(int), cudaHostAllocMapped));
        *ctx->flowError = 0;
        CK(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&ctx->flowBlocksPerSm, k_flow, kFlowThreads, 0));
    }
    CK(cudaHostGetDevicePointer((void**)&flow.error, ctx->flowError, 0));
    // the ends without a dynamic body keep visit -1
    CK(cudaMemsetAsync(flow.visit, 0xff, sizeof(int2) * groupPlan.slotOf.size(), stream));
    CK(cudaMemcpyAsync(flow.chunks, chunks.data(), sizeof(int2) * chunks.size(), cudaMemcpyHostToDevice, stream));
    CK(cudaStreamSynchronize(stream));
    return BEPUGPU_OK;
}

bepugpu_status Scene::BuildFlowOnDevice(Context* ctx, const unsigned long long* entries, int count, const int2* ends,
                                        const int* slots) {
    k_flow_csr<<<(count + 1 + 255) / 256, 256, 0, stream>>>(entries, count, b.count, ends, slots, flow);
    CK(cudaGetLastError());
    return UploadFlowChunks(ctx, {});
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
    const unsigned sweeps = (unsigned)p.iterationLimit + 1;
    k_flow_order<<<(nb + 127) / 128, 128, 0, s->stream>>>(s->m, s->b, f, list, nb, warm ? 0u : 1u, sweeps);
    if (launches) (*launches)++;
    cudaLaunchConfig_t cfg = {};
    // a warp per chunk on its own CTA while the CTAs last
    cfg.gridDim = dim3((unsigned)std::max(1, std::min(ctx->flowBlocksPerSm * ctx->smCount, f.chunkCount)));
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

bepugpu_status FlowStatus(Context* ctx) {
    if (!ctx->flowError || !*(volatile int*)ctx->flowError) return BEPUGPU_OK;
    *ctx->flowError = 0;
    ctx->SetError("solve sweeps: a wait for an earlier visit ran out");
    return BEPUGPU_TIMEOUT;
}

}  // namespace bepugpu
