// The narrow phase's pair bookkeeping on the device: the manifold list of a
// scene follows the broad phase's pair set without a host round trip, as the
// reference's NarrowPhase keeps a pair handler per overlap
// (NarrowPhaseSystems/NarrowPhase.cs:143-178 adds one for a new overlap,
// :254-332 drops a pair whose boxes stopped overlapping), and the solver list
// is recoloured on the device.
//
//   1. the broad phase leaves the pair keys sorted in device memory;
//   2. the old records' keys go into a hash table, where each pair looks
//      itself up: found, its records are kept, else it is new;
//   3. prefix sums give the new list: the kept records in their order, then
//      the new pairs ascending;
//   4. the colouring -- the smallest colour no earlier entry sharing a dynamic
//      body took, the host's greedy colouring in list order -- runs as
//      Jones-Plassmann with the list index as priority: an entry takes its
//      colour once the entries before it at each of its dynamic bodies have
//      theirs, which is exactly the greedy choice; one cooperative launch, the
//      entries polling the ones before them;
//   5. slots follow the colour-major order (a sort of (colour, index) keys) and
//      the records' lanes move to them, new records start empty.
#include <cuda_runtime.h>

#include <algorithm>
#include <climits>
#include <cstring>
#include <vector>

#include "../../include/bepugpu.h"
#include "bepugpu_internal.h"
#include "scan_device.cuh"
#include "solver_device.cuh"

namespace bepugpu {

// Device buffers of bepugpu_update_pairs, grown as needed.
struct PairBuffers {
    float4* material = nullptr;  // per body: kinetic, static friction, bounciness
    int32_t materialCount = 0;
    void* block = nullptr;
    size_t blockBytes = 0;
    int* colouring = nullptr;  // the last call's colours, then their order; the scene's capacity of each
    ~PairBuffers() {
        cudaFree(colouring);
        cudaFree(material);
        cudaFree(block);
    }
};

// The entries' colours and their order that the last update_pairs kept.  They
// are read by bepugpu_get_colouring alone, so the call itself does not wait for
// them: copying them and the slots into host vectors on each call was 70 of
// the 1,000 us a settling heap's frame of 82,000 pairs takes.
cudaError_t Scene::FetchColouring() {
    if (!colouringOnDevice) return cudaSuccess;
    const size_t n = colouringEntries, bytes = sizeof(int32_t) * n;
    std::vector<int32_t> colour(n), order(n);
    cudaError_t e = cudaSuccess;
    if (n && ((e = cudaMemcpyAsync(colour.data(), pairs->colouring, bytes, cudaMemcpyDeviceToHost, stream)) ||
              (e = cudaMemcpyAsync(order.data(), pairs->colouring + n, bytes, cudaMemcpyDeviceToHost, stream)) ||
              (e = cudaStreamSynchronize(stream))))
        return e;
    colouring.colour.swap(colour);
    colouring.order.swap(order);
    colouringOnDevice = false;
    return cudaSuccess;
}

void ReleasePairs(Scene* s) {
    delete s->pairs;
    s->pairs = nullptr;
}

namespace {

constexpr int kScanBlock = 256, kScanItems = 4, kScanTile = kScanBlock * kScanItems;
constexpr int kLanes = 25;  // head, cpos x4, cnrm x4, offA x4, offB x4, mat, penacc, fricacc, saxis, cfr x4

// Exclusive scan of one tile per block; tile totals to sums.
__global__ void k_scan_tiles(const int* __restrict__ in, int* __restrict__ out, int n, int* __restrict__ sums) {
    __shared__ int warpSums[32];
    const int base = blockIdx.x * kScanTile + threadIdx.x * kScanItems;
    int v[kScanItems], t = 0;
#pragma unroll
    for (int k = 0; k < kScanItems; k++) {
        v[k] = base + k < n ? in[base + k] : 0;
        t += v[k];
    }
    const int incl = BlockInclusiveSum(t, warpSums);
    int run = incl - t;
#pragma unroll
    for (int k = 0; k < kScanItems; k++) {
        if (base + k < n) out[base + k] = run;
        run += v[k];
    }
    if (threadIdx.x == blockDim.x - 1) sums[blockIdx.x] = incl;
}
__global__ void k_scan_add(int* __restrict__ out, int n, const int* __restrict__ sums) {
    const int i = blockIdx.x * kScanTile + threadIdx.x;
    const int add = sums[blockIdx.x];
    for (int k = 0; k < kScanItems; k++) {
        const int j = i + k * kScanBlock;
        if (j < n) out[j] += add;
    }
}

// 64-bit key of a pair: lower body << 32 | higher body.
__device__ __forceinline__ unsigned long long PairKey(int a, int b) {
    const int lo = min(a, b), hi = max(a, b);
    return ((unsigned long long)(unsigned)lo << 32) | (unsigned)hi;
}
// The hash table of the old records: open addressing over a power of two of
// slots, at least twice the records; a slot is the record's key and, in rec,
// its index.  Two records of one pair take a slot each.
__device__ __forceinline__ unsigned HashOf(unsigned long long key, unsigned slots) {
    return (unsigned)((key * 0x9E3779B97F4A7C15ull) >> 32) & (slots - 1);
}
__global__ void k_old_table(ManifoldSoA m, const int32_t* __restrict__ slotOf, int n, unsigned long long* table,
                            int* rec, unsigned slots) {
    const int r = blockIdx.x * blockDim.x + threadIdx.x;
    if (r >= n) return;
    const int4 h = m.head[slotOf[r]];
    const unsigned long long key = PairKey(h.x, h.y);
    for (unsigned at = HashOf(key, slots);; at = (at + 1) & (slots - 1))
        if (atomicCAS(table + at, ~0ull, key) == ~0ull) {
            rec[at] = r;
            return;
        }
}
// fresh[p]: pair p is new; kept[r] (zero before): record r's pair is still reported.
__global__ void k_membership(const unsigned long long* __restrict__ table, const int* __restrict__ rec, unsigned slots,
                             const unsigned long long* __restrict__ pairs, int nPairs, int* kept, int* fresh) {
    const int p = blockIdx.x * blockDim.x + threadIdx.x;
    if (p >= nPairs) return;
    const unsigned long long key = pairs[p];
    bool known = false;
    for (unsigned at = HashOf(key, slots); table[at] != ~0ull; at = (at + 1) & (slots - 1))
        if (table[at] == key) {
            kept[rec[at]] = 1;
            known = true;
        }
    fresh[p] = known ? 0 : 1;
}

// The new list: record i's bodies (A, B as the record keeps them), its flags
// and its old slot (-1 for a new pair).
struct NewRecords {
    int2* ends;
    uint32_t* flags;
    int32_t* oldSlot;
};
__global__ void k_list_kept(ManifoldSoA m, const int32_t* __restrict__ slotOf, int nOld, const int* __restrict__ kept,
                            const int* __restrict__ keptAt, NewRecords out) {
    const int r = blockIdx.x * blockDim.x + threadIdx.x;
    if (r >= nOld || !kept[r]) return;
    const int s = slotOf[r], i = keptAt[r];
    const int4 h = m.head[s];
    out.ends[i] = make_int2(h.x, h.y);
    out.flags[i] = (uint32_t)h.z >> 8;
    out.oldSlot[i] = s;
}
// A new pair's record: the box first in a box-sphere pair (BoxSpherePairHandler),
// NONCONVEX for a pair with a sphere (SpherePairHandler.cs:28, BoxSpherePairHandler.cs:28).
__global__ void k_list_fresh(const unsigned long long* __restrict__ pairs, int nPairs, const int* __restrict__ fresh,
                             const int* __restrict__ freshAt, int kept, const float4* __restrict__ shape,
                             NewRecords out) {
    const int p = blockIdx.x * blockDim.x + threadIdx.x;
    if (p >= nPairs || !fresh[p]) return;
    int a = (int)(pairs[p] >> 32), b = (int)(pairs[p] & 0xffffffffu);
    const int ta = __float_as_int(shape[a].w), tb = __float_as_int(shape[b].w);
    if (ta == BEPUGPU_SHAPE_SPHERE && tb == BEPUGPU_SHAPE_BOX) {
        const int t = a;
        a = b;
        b = t;
    }
    const bool sphere = ta == BEPUGPU_SHAPE_SPHERE || tb == BEPUGPU_SHAPE_SPHERE;
    const int i = kept + freshAt[p];
    out.ends[i] = make_int2(a, b);
    out.flags[i] = BEPUGPU_MANIFOLD_ACTIVE | BEPUGPU_MANIFOLD_SOLVER_RULE | BEPUGPU_MANIFOLD_GENERATED |
                   (sphere ? BEPUGPU_MANIFOLD_NONCONVEX : 0u);
    out.oldSlot[i] = -1;
}

// Colouring.  entries: (dynamic body << 32 | entry) for each dynamic end of
// each entry, sorted; at[i]: the entry's positions there for its ends A and
// B, -1 for an end without a dynamic body.
__global__ void k_colour_entries(const int2* __restrict__ ends, int n, BodySoA b, unsigned long long* entries,
                                 int* colour) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const int2 e = ends[i];
    const bool da = e.x >= 0 && b.pos[e.x].w != 0.f, db = e.y >= 0 && b.pos[e.y].w != 0.f;
    entries[2 * i] = da ? ((unsigned long long)(unsigned)e.x << 32) | (unsigned)i : ~0ull;
    entries[2 * i + 1] = db ? ((unsigned long long)(unsigned)e.y << 32) | (unsigned)i : ~0ull;
    colour[i] = -1;
}
// (entries that a sort left half moved when its wait ran out may name none of
// the n entries; the colouring then returns at once.)
__global__ void k_colour_positions(const unsigned long long* __restrict__ entries, int count, const int2* __restrict__ ends,
                                   int n, int2* at) {
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= count) return;
    const unsigned long long key = entries[k];
    if (key == ~0ull) return;
    const int body = (int)(key >> 32), i = (int)(key & 0xffffffffu);
    if ((unsigned)i >= (unsigned)n) return;
    if (ends[i].x == body) at[i].x = k;
    else at[i].y = k;
}
// The colouring: every entry waits until the entries before it at its dynamic
// bodies are coloured, then takes the smallest colour none of them has.  A
// thread takes its entries in list order and every thread is resident
// (cooperative launch), so the first uncoloured entry is never waiting; only
// the colours themselves pass between threads, each read past L1, and a stale
// one reads as uncoloured.  An entry keeps its place in its walk over the
// entries before it, so a poll is one trip and each of them is read once, four
// at a time; only an entry that finds 64 colours taken walks again, 256 colours
// a walk.  A warp that polls kColourSpinLimit times while no entry anywhere is
// coloured (*progress) ends with *err, and its entries keep colour -1; nothing
// reads a colour once *err is set.
// Bound by the polls' trips through L2 along the longest chain.  82,000 entries
// of a settling heap took 80 us with a walk from the start in every poll (270
// with a launch for each of 32 rounds); four frames of it 3,450 -> 3,275 us
// with this walk and the slots' single sort pass.  With a walk from the start
// 560 bodies that all overlap ran into the limit; they take 0.1 s.
constexpr int kColourSpinLimit = 1 << 22;
__device__ __forceinline__ int PeekColour(const int* colour, int i) { return *(volatile const int*)(colour + i); }
// Up to four entries of `body` from q down: q moves past the coloured ones,
// their colours go to `take`; false at one that is not coloured.  q is -1 at
// the body's first entry.
template <class Take>
__device__ __forceinline__ bool WalkEntries(const unsigned long long* __restrict__ entries, const int* colour,
                                            unsigned body, int& q, Take take) {
    bool mine[4];
    int c[4];
#pragma unroll
    for (int u = 0; u < 4; u++) {
        const unsigned long long entry = q - u >= 0 ? entries[q - u] : ~0ull;
        mine[u] = (unsigned)(entry >> 32) == body;
        c[u] = mine[u] ? PeekColour(colour, (int)(entry & 0xffffffffu)) : 0;
    }
#pragma unroll
    for (int u = 0; u < 4; u++) {
        if (!mine[u]) {
            q = -1;
            return true;
        }
        if (c[u] < 0) return false;
        take(c[u]);
        q--;
    }
    return true;
}
__global__ void k_colour_entries_in_order(const unsigned long long* __restrict__ entries, const int2* __restrict__ at,
                                          int n, int* colour, int* progress, int* err) {
    if (*(volatile int*)err) return;  // the entries are not sorted
    const int stride = gridDim.x * blockDim.x;
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i - (int)(threadIdx.x & 31) < n; i += stride) {
        bool done = i >= n;
        const int2 pos = done ? make_int2(-1, -1) : at[i];
        const int ks[2] = {pos.x, pos.y};
        unsigned body[2];
        int q[2];
#pragma unroll
        for (int e = 0; e < 2; e++) {
            body[e] = ks[e] >= 0 ? (unsigned)(entries[ks[e]] >> 32) : 0u;
            q[e] = ks[e] - 1;  // below zero: nothing to wait for
        }
        unsigned long long used = 0;
        int seen = -1;
        for (int spins = 0; !__all_sync(0xffffffffu, done); spins++) {
            if (spins > kColourSpinLimit) {
                const int now = __shfl_sync(0xffffffffu, *(volatile int*)progress, 0);
                if (now == seen) {
                    *(volatile int*)err = BEPUGPU_TIMEOUT;
                    return;
                }
                seen = now;
                spins = 0;
            }
            int chosen = -1;
            if (!done) {
                bool ready = true;
#pragma unroll
                for (int e = 0; e < 2; e++)
                    while (ready && q[e] >= 0)
                        ready = WalkEntries(entries, colour, body[e], q[e], [&](int c) {
                            if (c < 64) used |= 1ull << c;
                        });
                if (ready && ~used) chosen = __ffsll((long long)~used) - 1;
                for (int from = 64; ready && chosen < 0; from += 256) {
                    unsigned long long more[4] = {0, 0, 0, 0};
#pragma unroll
                    for (int e = 0; e < 2; e++)
                        for (int w = ks[e] - 1; w >= 0;)
                            WalkEntries(entries, colour, body[e], w, [&](int c) {
                                const unsigned k = (unsigned)(c - from);
#pragma unroll
                                for (unsigned g = 0; g < 4; g++)
                                    if (k >> 6 == g) more[g] |= 1ull << (k & 63);
                            });
#pragma unroll
                    for (int g = 3; g >= 0; g--)
                        if (~more[g]) chosen = from + 64 * g + __ffsll((long long)~more[g]) - 1;
                }
                if (chosen >= 0) {
                    *(volatile int*)(colour + i) = chosen;
                    done = true;
                }
            }
            if (__any_sync(0xffffffffu, chosen >= 0) && (threadIdx.x & 31) == 0) atomicAdd(progress, 1);
        }
    }
}
// Entries per colour; the colours up to kColourBins through shared memory.
// Nothing when a wait ran out: some entries then have no colour.
constexpr int kColourBins = 1024;
__global__ void k_colour_count(const int* __restrict__ colour, int n, int* counts, int* maxColour,
                               const int* __restrict__ err) {
    __shared__ int bins[kColourBins];
    __shared__ int top;
    if (*err) return;
    for (int k = threadIdx.x; k < kColourBins; k += blockDim.x) bins[k] = 0;
    if (threadIdx.x == 0) top = 0;
    __syncthreads();
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const int c = colour[i];
        if (c < kColourBins) atomicAdd(bins + c, 1);
        else atomicAdd(counts + c, 1);
        atomicMax(&top, c);
    }
    __syncthreads();
    for (int k = threadIdx.x; k < kColourBins; k += blockDim.x)
        if (bins[k]) atomicAdd(counts + k, bins[k]);
    if (threadIdx.x == 0) atomicMax(maxColour, top);
}
__global__ void k_slot_keys(const int* __restrict__ colour, int n, unsigned long long* keys) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) keys[i] = ((unsigned long long)(unsigned)colour[i] << 32) | (unsigned)i;
}
// (keys of a sort whose wait ran out may name none of the n entries)
__global__ void k_slots(const unsigned long long* __restrict__ keys, int n, int* slotOf, int* order) {
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= n) return;
    const int i = (int)(keys[k] & 0xffffffffu);
    if ((unsigned)i >= (unsigned)n) return;
    slotOf[i] = k;
    order[k] = i;
}

// A record's input lanes at its new slot of the scratch copy (capacity n):
// a kept record's lanes as a download and upload would carry them, a new
// record's empty with the blended material (MaterialManager.cs:77-85).
// Nothing when the slots' sort gave up: not every entry has a slot then.
__global__ void k_move_lanes(ManifoldSoA m, NewRecords rec, const int* __restrict__ newSlot, int n,
                             const float4* __restrict__ material, float4* scratch, const int* __restrict__ err) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n || *err) return;
    const int ns = newSlot[i], os = rec.oldSlot[i], cap = m.capacity;
    const int2 e = rec.ends[i];
    const uint32_t flags = rec.flags[i];
    float4* L = scratch;
    auto at = [&](int lane) -> float4& { return L[(size_t)lane * n + ns]; };
    const float4 zero = make_float4(0.f, 0.f, 0.f, 0.f);
    if (os < 0) {
        at(0) = make_float4(__int_as_float(e.x), __int_as_float(e.y), __int_as_float((int)(flags << 8)),
                            __int_as_float(i));
        for (int lane = 1; lane < kLanes; lane++) at(lane) = zero;
        const float4 ma = material[e.x], mb = material[e.y];
        at(17) = make_float4(ma.x * mb.x, ma.y * mb.y, ma.z * mb.z, 0.f);
        return;
    }
    const int4 h = m.head[os];
    const int count = h.z & 0xff;
    at(0) = make_float4(__int_as_float(h.x), __int_as_float(h.y), __int_as_float(h.z), __int_as_float(i));
    const bool nonConvex = flags & BEPUGPU_MANIFOLD_NONCONVEX;
    for (int k = 0; k < 4; k++) {
        const bool live = k < count;
        const float4 ob = m.offB[k * cap + os];
        at(1 + k) = live ? m.cpos[k * cap + os] : zero;
        at(5 + k) = live ? m.cnrm[k * cap + os] : zero;
        at(9 + k) = live ? m.offA[k * cap + os] : zero;
        at(13 + k) = live ? make_float4(ob.x, ob.y, ob.z, 0.f) : zero;
        at(21 + k) = live && nonConvex ? m.cfr[k * cap + os] : zero;
    }
    const float4 mat = m.mat[os], pa = m.penacc[os], f = m.fricacc[os], ax = m.saxis[os];
    at(17) = make_float4(mat.x, mat.y, mat.z, 0.f);
    at(18) = make_float4(count > 0 ? pa.x : 0.f, count > 1 ? pa.y : 0.f, count > 2 ? pa.z : 0.f,
                         count > 3 ? pa.w : 0.f);
    at(19) = make_float4(count > 0 ? f.x : 0.f, count > 0 ? f.y : 0.f, count > 0 ? f.z : 0.f, f.w);
    at(20) = make_float4(ax.x, ax.y, ax.z, 0.f);
}
// The scratch copy back into the scene's lanes, slots [0, n), and the entries'
// slots, colours and order beside them; nothing when the slots' sort gave up.
struct KeptColouring {
    const int *slotOf, *colour, *order;  // scratch
    int *sceneSlotOf, *colouring;        // the scene's: slots; colours, then order
};
__global__ void k_lanes_back(ManifoldSoA m, const float4* __restrict__ scratch, int n, int32_t* genSlots,
                             KeptColouring keep, const int* __restrict__ err) {
    const int s = blockIdx.x * blockDim.x + threadIdx.x;
    if (s >= n || *err) return;
    keep.sceneSlotOf[s] = keep.slotOf[s];
    keep.colouring[s] = keep.colour[s];
    keep.colouring[n + s] = keep.order[s];
    const int cap = m.capacity;
    auto L = [&](int lane) { return scratch[(size_t)lane * n + s]; };
    const float4 h = L(0);
    m.head[s] = make_int4(__float_as_int(h.x), __float_as_int(h.y), __float_as_int(h.z), __float_as_int(h.w));
    for (int k = 0; k < 4; k++) {
        m.cpos[k * cap + s] = L(1 + k);
        m.cnrm[k * cap + s] = L(5 + k);
        m.offA[k * cap + s] = L(9 + k);
        m.offB[k * cap + s] = L(13 + k);
        m.cfr[k * cap + s] = L(21 + k);
    }
    m.mat[s] = L(17);
    m.penacc[s] = L(18);
    m.fricacc[s] = L(19);
    m.saxis[s] = L(20);
    m.state[s] = make_uint2(0u, 0u);
    genSlots[s] = s;
}

}  // namespace

#define CK(call)                                                                              \
    do {                                                                                      \
        cudaError_t e_ = (call);                                                              \
        if (e_ != cudaSuccess) {                                                              \
            ctx->SetError("%s failed: %s (%s:%d)", #call, cudaGetErrorString(e_), __FILE__, __LINE__); \
            return BEPUGPU_CUDA_ERROR;                                                        \
        }                                                                                     \
    } while (0)

namespace {

// Exclusive scan of n ints (in and out may not alias); *total receives the sum.
bepugpu_status ExclusiveScan(Context* ctx, const int* in, int* out, int n, int* scratch, int* total, cudaStream_t st) {
    if (n <= 0) {
        CK(cudaMemsetAsync(total, 0, sizeof(int), st));
        return BEPUGPU_OK;
    }
    const int tiles = (n + kScanTile - 1) / kScanTile;
    int* sums = scratch;
    k_scan_tiles<<<tiles, kScanBlock, 0, st>>>(in, out, n, sums);
    CK(cudaGetLastError());
    if (tiles == 1) {
        CK(cudaMemcpyAsync(total, sums, sizeof(int), cudaMemcpyDeviceToDevice, st));
        return BEPUGPU_OK;
    }
    int* scanned = sums + tiles;
    bepugpu_status r = ExclusiveScan(ctx, sums, scanned, tiles, scanned + tiles, total, st);
    if (r != BEPUGPU_OK) return r;
    k_scan_add<<<tiles, kScanBlock, 0, st>>>(out, n, scanned);
    CK(cudaGetLastError());
    return BEPUGPU_OK;
}

// Bump allocator over one block of device memory.
struct Carve {
    char* base;
    size_t used = 0;
    template <class T>
    T* take(size_t count) {
        T* p = (T*)(base + used);
        used += (count * sizeof(T) + 255) & ~(size_t)255;
        return p;
    }
};

}  // namespace

// The colouring of n entries with ends[] (host-side greedy rule, on the
// device): colour[i], order (colour-major, list order inside a colour),
// per-colour offsets into order.  Needs the buffers of one call.
struct DeviceColouring {
    int* colour;
    int* order;
    int* slotOf;
    const unsigned long long* entries = nullptr;  // (dynamic body << 32 | entry), sorted, 2 n of them (~0: none)
    const int* status = nullptr;  // device: set when the slots' sort gave up (its end is not waited for)
    int colours = 0;
    std::vector<int32_t> offsets;
};

// A sort's or the colouring's wait ran out: blocks that gave up leave the
// barrier counter where it was, so it starts again from zero.
static bepugpu_status GaveUp(Context* ctx, Scene* s, const char* what) {
    CK(cudaMemsetAsync(s->SortCounter(), 0, sizeof(unsigned), s->stream));
    ctx->SetError("update_pairs: %s did not finish", what);
    return BEPUGPU_TIMEOUT;
}

static bepugpu_status ColourOnDevice(Context* ctx, Scene* s, const int2* ends, int n, Carve& c, DeviceColouring& out) {
    const cudaStream_t st = s->stream;
    const int T = 256;
    out.colour = c.take<int>(n);
    out.order = c.take<int>(n);
    out.slotOf = c.take<int>(n);
    out.colours = 0;
    out.offsets.assign(1, 0);
    if (n == 0) return BEPUGPU_OK;
    auto* entries = c.take<unsigned long long>(2 * (size_t)n);
    auto* other = c.take<unsigned long long>(2 * (size_t)n);  // the sorts' second buffer
    auto* keys = c.take<unsigned long long>(n);
    auto* at = c.take<int2>(n);
    unsigned* hist = c.take<unsigned>(kSortHistWords);
    // counts[0, n]: entries per colour; then the highest colour, the status and the colouring's progress
    int* counts = c.take<int>((size_t)n + 4);
    int *maxColour = counts + n + 1, *err = counts + n + 2;
    CK(cudaMemsetAsync(counts, 0, sizeof(int) * ((size_t)n + 4), st));
    CK(s->MarkExpired(err, BEPUGPU_WAIT_COLOURING));
    k_colour_entries<<<(n + T - 1) / T, T, 0, st>>>(ends, n, s->b, entries, out.colour);
    // by body alone: the entries start in list order and the sort is stable
    // (entries of no dynamic body have every bit set: one value more than the bodies)
    CK(RadixSort(s, entries, other, nullptr, 2 * (size_t)n, SortPlan(0, 0, BitsFor((size_t)s->b.count + 1)), hist, err,
                 st));
    out.entries = entries;
    CK(cudaMemsetAsync(at, 0xff, sizeof(int2) * n, st));
    k_colour_positions<<<(int)((2 * (size_t)n + T - 1) / T), T, 0, st>>>(entries, 2 * n, ends, n, at);
    CK(cudaGetLastError());
    if (!ctx->colourBlocksPerSm)
        CK(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&ctx->colourBlocksPerSm, k_colour_entries_in_order, T, 0));
    {
        cudaLaunchConfig_t cfg = {};
        cfg.gridDim = dim3((unsigned)std::max(1, std::min((n + T - 1) / T, ctx->colourBlocksPerSm * ctx->smCount)));
        cfg.blockDim = dim3(T);
        cfg.stream = st;
        cudaLaunchAttribute attr[1];
        attr[0].id = cudaLaunchAttributeCooperative;
        attr[0].val.cooperative = 1;
        cfg.attrs = attr;
        cfg.numAttrs = 1;
        CK(cudaLaunchKernelEx(&cfg, k_colour_entries_in_order, (const unsigned long long*)entries, (const int2*)at, n,
                              out.colour, err + 1, err));
    }
    k_colour_count<<<std::min((n + T - 1) / T, ctx->smCount), T, 0, st>>>(out.colour, n, counts, maxColour, err);
    CK(cudaGetLastError());
    int tail[2];  // the highest colour, the status
    const int listed = std::min(n, kColourBins);
    std::vector<int32_t> hc(listed);
    CK(cudaMemcpyAsync(tail, maxColour, sizeof(tail), cudaMemcpyDeviceToHost, st));
    CK(cudaMemcpyAsync(hc.data(), counts, sizeof(int) * listed, cudaMemcpyDeviceToHost, st));
    CK(cudaStreamSynchronize(st));
    if (tail[1]) return GaveUp(ctx, s, "the colouring");
    out.colours = tail[0] + 1;
    if (out.colours > listed) {
        hc.resize(out.colours);
        CK(cudaMemcpyAsync(hc.data(), counts, sizeof(int) * out.colours, cudaMemcpyDeviceToHost, st));
        CK(cudaStreamSynchronize(st));
    }
    // slots: entries sorted by colour, in list order inside one
    k_slot_keys<<<(n + T - 1) / T, T, 0, st>>>(out.colour, n, keys);
    // up to 512 colours are one digit: one pass of about 12 us, which ends in `other`, where an even number took 24
    const SortDigits byColour = SortPlan(0, 0, BitsFor((size_t)out.colours), true);
    out.status = err;
    CK(s->MarkExpired(err, BEPUGPU_WAIT_SLOTS));
    CK(RadixSort(s, keys, other, nullptr, (size_t)n, byColour, hist, err, st));
    k_slots<<<(n + T - 1) / T, T, 0, st>>>(byColour.passes & 1 ? other : keys, n, out.slotOf, out.order);
    CK(cudaGetLastError());
    out.offsets.assign(out.colours + 1, 0);
    for (int k = 0; k < out.colours; k++) out.offsets[k + 1] = out.offsets[k] + hc[k];
    return BEPUGPU_OK;
}

}  // namespace bepugpu

using namespace bepugpu;

extern "C" bepugpu_status bepugpu_set_materials(bepugpu_context* c, int32_t id, const float* materials,
                                                uint32_t count) {
    auto* ctx = reinterpret_cast<Context*>(c);
    if (!ctx) return BEPUGPU_INVALID_ARGUMENT;
    cudaSetDevice(ctx->device);
    Scene* s = FindScene(ctx, id);
    if (!s) return SceneMissing(ctx, id);
    if (count != (uint32_t)s->b.count || (count && !materials)) {
        ctx->SetError("set_materials: three floats for each of the %d bodies", s->b.count);
        return BEPUGPU_INVALID_ARGUMENT;
    }
    if (!s->pairs) s->pairs = new PairBuffers();
    PairBuffers& P = *s->pairs;
    if (P.materialCount < (int32_t)count) {
        cudaFree(P.material);
        P.material = nullptr;
        P.materialCount = 0;
        CK(cudaMalloc(&P.material, sizeof(float4) * std::max<uint32_t>(count, 1)));
        P.materialCount = (int32_t)count;
    }
    std::vector<float4> h(count);
    for (uint32_t i = 0; i < count; i++) h[i] = make_float4(materials[3 * i], materials[3 * i + 1], materials[3 * i + 2], 0.f);
    if (count) CK(cudaMemcpyAsync(P.material, h.data(), sizeof(float4) * count, cudaMemcpyHostToDevice, s->stream));
    CK(cudaStreamSynchronize(s->stream));
    return BEPUGPU_OK;
}

extern "C" bepugpu_status bepugpu_update_pairs(bepugpu_context* c, int32_t id, float dt, uint32_t* manifold_count) {
    NvtxRange range("bepugpu_update_pairs");
    auto* ctx = reinterpret_cast<Context*>(c);
    if (!ctx) return BEPUGPU_INVALID_ARGUMENT;
    cudaSetDevice(ctx->device);
    Scene* s = FindScene(ctx, id);
    if (!s) return SceneMissing(ctx, id);
    if (!(dt >= 0) || !std::isfinite(dt)) {
        ctx->SetError("update_pairs: dt must be >= 0 and finite");
        return BEPUGPU_INVALID_ARGUMENT;
    }
    if (s->jointCount != 0 || s->generatedCount != s->m.count) {
        ctx->SetError("update_pairs: the scene's constraints must all be GENERATED manifolds");
        return BEPUGPU_INVALID_OPERATION;
    }
    if (!s->pairs || s->pairs->materialCount < s->b.count) {
        ctx->SetError("update_pairs: set the bodies' materials first (bepugpu_set_materials)");
        return BEPUGPU_INVALID_OPERATION;
    }
    unsigned found = 0;
    bepugpu_status st0 = RunBroadPhase(ctx, s, dt, found);
    if (st0 != BEPUGPU_OK) return st0;
    const int nPairs = (int)found, nOld = s->m.count;
    if ((uint32_t)nPairs > s->maxManifolds) {
        ctx->SetError("update_pairs: %d pairs exceed the scene's capacity of %u manifolds", nPairs, s->maxManifolds);
        return BEPUGPU_INVALID_OPERATION;
    }
    const unsigned long long* pairs = BroadPhasePairs(s);
    const cudaStream_t st = s->stream;
    PairBuffers& P = *s->pairs;
    // scratch: keys, flags and scans, the new list, the colouring, the moved lanes
    const int nMax = std::max(std::max(nPairs, nOld), 1);
    unsigned tableSlots = 64;
    while (tableSlots < 2 * (unsigned)nMax) tableSlots *= 2;
    const size_t want = 256 * 64 + (sizeof(unsigned long long) + sizeof(int)) * (size_t)tableSlots +
                        sizeof(unsigned long long) * 5 * (size_t)nMax +
                        sizeof(int) * (14 * (size_t)nMax + 64 + kSortHistWords) +
                        sizeof(float4) * kLanes * (size_t)nMax + sizeof(int2) * 2 * (size_t)nMax;
    if (P.blockBytes < want) {
        cudaFree(P.block);
        P.block = nullptr;
        P.blockBytes = 0;
        const size_t bytes = want + want / 4;
        cudaError_t e = cudaMalloc(&P.block, bytes);
        if (e != cudaSuccess) {
            ctx->SetError("update_pairs: %zu bytes of scratch: %s", bytes, cudaGetErrorString(e));
            return e == cudaErrorMemoryAllocation ? BEPUGPU_OUT_OF_MEMORY : BEPUGPU_CUDA_ERROR;
        }
        P.blockBytes = bytes;
    }
    if (!P.colouring) {
        const size_t bytes = 2 * sizeof(int) * std::max<size_t>(s->maxManifolds, 1);
        cudaError_t e = cudaMalloc(&P.colouring, bytes);
        if (e != cudaSuccess) {
            ctx->SetError("update_pairs: %zu bytes for the colouring: %s", bytes, cudaGetErrorString(e));
            return e == cudaErrorMemoryAllocation ? BEPUGPU_OUT_OF_MEMORY : BEPUGPU_CUDA_ERROR;
        }
    }
    if (nPairs) {
        bepugpu_status fs = s->NeedFlow(ctx);
        if (fs != BEPUGPU_OK) return fs;
    }
    Carve cv{(char*)P.block};
    const int T = 256;
    auto* table = cv.take<unsigned long long>(tableSlots);
    int* tableRec = cv.take<int>(tableSlots);
    int* kept = cv.take<int>(nMax);
    int* keptAt = cv.take<int>(nMax);
    int* fresh = cv.take<int>(nMax);
    int* freshAt = cv.take<int>(nMax);
    int* scanScratch = cv.take<int>(2 * (size_t)nMax + 64);
    int* totals = cv.take<int>(2);
    NewRecords rec{cv.take<int2>(nMax), cv.take<uint32_t>(nMax), cv.take<int32_t>(nMax)};
    CK(cudaMemsetAsync(table, 0xff, sizeof(unsigned long long) * tableSlots, st));
    if (nOld) {
        CK(cudaMemsetAsync(kept, 0, sizeof(int) * nOld, st));
        k_old_table<<<(nOld + T - 1) / T, T, 0, st>>>(s->m, s->slotOf, nOld, table, tableRec, tableSlots);
    }
    if (nPairs)
        k_membership<<<(nPairs + T - 1) / T, T, 0, st>>>(table, tableRec, tableSlots, pairs, nPairs, kept, fresh);
    CK(cudaGetLastError());
    bepugpu_status sr = ExclusiveScan(ctx, kept, keptAt, nOld, scanScratch, totals, st);
    if (sr != BEPUGPU_OK) return sr;
    sr = ExclusiveScan(ctx, fresh, freshAt, nPairs, scanScratch, totals + 1, st);
    if (sr != BEPUGPU_OK) return sr;
    int tot[2] = {0, 0};
    CK(cudaMemcpyAsync(tot, totals, sizeof(tot), cudaMemcpyDeviceToHost, st));
    CK(cudaStreamSynchronize(st));
    const int nKept = tot[0], n = tot[0] + tot[1];
    if (n != nPairs) {
        ctx->SetError("update_pairs: %d kept and %d new records for %d pairs", tot[0], tot[1], nPairs);
        return BEPUGPU_CUDA_ERROR;
    }
    if (nOld) k_list_kept<<<(nOld + T - 1) / T, T, 0, st>>>(s->m, s->slotOf, nOld, kept, keptAt, rec);
    if (nPairs)
        k_list_fresh<<<(nPairs + T - 1) / T, T, 0, st>>>(pairs, nPairs, fresh, freshAt, nKept, s->shape, rec);
    CK(cudaGetLastError());
    DeviceColouring col;
    sr = ColourOnDevice(ctx, s, rec.ends, n, cv, col);
    if (sr != BEPUGPU_OK) return sr;
    auto* scratch = cv.take<float4>((size_t)kLanes * nMax);
    if (cv.used > P.blockBytes) {
        ctx->SetError("update_pairs: scratch overrun (%zu of %zu bytes)", cv.used, P.blockBytes);
        return BEPUGPU_CUDA_ERROR;
    }
    // Everything so far went to scratch.  The scene changes from here on: in
    // kernels that look at the status themselves, and on the host and in the
    // tables it uploads once the status has been read.
    const std::vector<int2> chunks = FlowChunks(col.offsets);
    if (n) {
        k_move_lanes<<<(n + T - 1) / T, T, 0, st>>>(s->m, rec, col.slotOf, n, P.material, scratch, col.status);
        const KeptColouring keep{col.slotOf, col.colour, col.order, s->slotOf, P.colouring};
        k_lanes_back<<<(n + T - 1) / T, T, 0, st>>>(s->m, scratch, n, s->genSlotsDev, keep, col.status);
        CK(cudaGetLastError());
        bepugpu_status fs = s->BuildFlowOnDevice(ctx, col.entries, 2 * n, rec.ends, col.slotOf, col.status);
        if (fs != BEPUGPU_OK) return fs;
        int status = 0;
        CK(cudaMemcpyAsync(&status, col.status, sizeof(int), cudaMemcpyDeviceToHost, st));
        CK(cudaStreamSynchronize(st));
        if (status) return GaveUp(ctx, s, "the slots' sort");
    }
    // the scene's bookkeeping: every manifold on the colour-sweep path
    if (s->islands) ReleaseIslands(s);
    const bool hadGroups = !s->groupPlan.groups.empty();
    GroupPlan& plan = s->groupPlan;
    plan = GroupPlan();
    plan.globalOffsets = col.offsets;
    plan.globalCount = n;
    plan.jointGlobalOffsets.assign(col.colours + 1, 0);
    plan.jointSlotOf.clear();
    s->colouring.colours = col.colours;
    s->colouring.offsets = col.offsets;
    s->colouringOnDevice = true;
    s->colouringEntries = n;
    s->manifoldOffsets = col.offsets;
    s->flow.chunkCount = s->flow.groupChunkCount = 0;
    bepugpu_status fs = s->UploadFlowChunks(ctx, chunks, (size_t)n);
    if (fs != BEPUGPU_OK) return fs;
    s->flow.chunkCount = (int)chunks.size();
    s->jointOffsets.assign(col.colours + 1, 0);
    s->m.count = n;
    s->generatedCount = n;
    s->hostGenPairs.clear();  // the shapes' pair check of bepugpu_upload_shapes applies to uploaded records only
    CK(cudaMemcpyAsync(s->colourOffsetsDev, col.offsets.data(), sizeof(int32_t) * col.offsets.size(),
                       cudaMemcpyHostToDevice, st));
    CK(cudaStreamSynchronize(st));
    if (hadGroups) {  // the bodies groups stepped go back to the sweep path's body stages
        s->hostOwned.assign(s->b.count, 0);
        s->dampDirty = true;
        bepugpu_status rs = s->RebuildSweepBodies(ctx);
        if (rs != BEPUGPU_OK) return rs;
    }
    s->version++;
    if (manifold_count) *manifold_count = (uint32_t)n;
    return BEPUGPU_OK;
}
