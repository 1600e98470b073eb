// Radix sort of 64-bit keys in one cooperative launch.
//
// The broad phase and the pair bookkeeping sort a few hundred thousand keys of
// which 18 to 36 bits vary, with the number of keys known on the device only.
// Each pass takes one digit of up to nine bits, least significant first and
// stable: a block counts its tile's digits, a grid barrier, every block adds
// up the blocks' counts to its own digit offsets, and moves its tile in order
// (ranks from __match_any_sync inside a warp, a prefix over the warps).  Four
// passes are seven barriers in one launch.
// Bound by the barriers and the passes' trips through L2, not by bandwidth: a
// barrier that counts up and is polled for itself, in place of one that resets
// and then releases, took the broad phase of 65,536 boxes (some 230,000 cell
// entries by 18 bits and 150,000 pairs by 34) from 219 to 206 us; the bitonic
// network before it took 57 launches and 451.  64 blocks: with 32 the tiles'
// serial ranking, with 128 the barriers cost more (235 and 237 us a broad phase
// against 222, before the change of barrier; 100 blocks 218 against 206 after).
#include <cuda_runtime.h>

#include <algorithm>

#include "bepugpu_internal.h"
#include "grid_barrier.cuh"
#include "scan_device.cuh"

namespace bepugpu {

namespace {

constexpr int kSortThreads = 1024, kSortWarps = kSortThreads / 32;
constexpr int kSortDigitBits = 9;
static_assert(kSortBins == 1 << kSortDigitBits, "a digit's values");

__global__ void __launch_bounds__(kSortThreads) k_radix_sort(unsigned long long* keys, unsigned long long* other,
                                                             const unsigned* __restrict__ count, unsigned capacity,
                                                             SortDigits digits, unsigned* hist, unsigned* counter,
                                                             int* err) {
    __shared__ unsigned base[kSortBins];
    __shared__ __align__(16) unsigned short warpCount[kSortWarps][kSortBins];
    __shared__ int warpSums[32];
    unsigned arrived = 0;
    const unsigned n = count ? min(*count, capacity) : capacity;
    const unsigned tile = (n + gridDim.x - 1) / gridDim.x;
    const unsigned begin = min(n, blockIdx.x * tile), end = min(n, begin + tile);
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    unsigned long long *src = keys, *dst = other;
    for (int pass = 0; pass < digits.passes; pass++) {
        const int shift = digits.shift[pass];
        const unsigned mask = (1u << digits.bits[pass]) - 1u;
        const bool bin = tid <= (int)mask;  // this thread's digit value
        if (tid < kSortBins) base[tid] = 0;
        __syncthreads();
        // keys come from other blocks' passes: past L1
        for (unsigned i = begin + tid; i < end; i += kSortThreads)
            atomicAdd(base + ((unsigned)(__ldcg(src + i) >> shift) & mask), 1u);
        __syncthreads();
        if (bin) hist[blockIdx.x * kSortBins + tid] = base[tid];
        if (!CountBarrier(counter, arrived, err)) return;
        unsigned total = 0, before = 0;
        if (bin) {
#pragma unroll 16
            for (int k = 0; k < kSortBlocks; k++) {  // rows of absent blocks are skipped, not waited for
                const unsigned v = k < (int)gridDim.x ? __ldcg(hist + k * kSortBins + tid) : 0u;
                before += k < (int)blockIdx.x ? v : 0u;
                total += v;
            }
        }
        const unsigned upTo = (unsigned)BlockInclusiveSum((int)total, warpSums);
        if (bin) base[tid] = upTo - total + before;
        for (unsigned first = begin; first < end; first += kSortThreads) {
            for (int k = tid; k < kSortWarps * kSortBins / 8; k += kSortThreads)
                ((uint4*)&warpCount[0][0])[k] = make_uint4(0u, 0u, 0u, 0u);
            __syncthreads();
            const unsigned i = first + tid;
            const unsigned long long key = i < end ? __ldcg(src + i) : 0ull;
            const unsigned digit = i < end ? (unsigned)(key >> shift) & mask : (unsigned)kSortBins;
            const unsigned same = __match_any_sync(0xffffffffu, digit);
            const int rank = __popc(same & ((1u << lane) - 1u));
            if (i < end && rank == 0) warpCount[warp][digit] = (unsigned short)__popc(same);
            __syncthreads();
            unsigned sum = 0;
            if (bin) {
                unsigned c[kSortWarps];
#pragma unroll
                for (int k = 0; k < kSortWarps; k++) c[k] = warpCount[k][tid];
#pragma unroll
                for (int k = 0; k < kSortWarps; k++) {
                    warpCount[k][tid] = (unsigned short)sum;
                    sum += c[k];
                }
            }
            __syncthreads();
            const unsigned to = i < end ? base[digit] + warpCount[warp][digit] + rank : n;
            if (to < n) dst[to] = key;
            __syncthreads();
            if (bin) base[tid] += sum;
        }
        if (pass + 1 < digits.passes && !CountBarrier(counter, arrived, err)) return;
        unsigned long long* t = src;
        src = dst;
        dst = t;
    }
    FinishGridBarriers(counter, arrived);
}

}  // namespace

SortDigits SortPlan(int lowFrom, int lowBits, int highBits, bool odd) {
    SortDigits d{};
    const auto parts = [](int bits) { return (bits + kSortDigitBits - 1) / kSortDigitBits; };
    int low = parts(lowBits), high = parts(highBits);
    if (!odd && ((low + high) & 1)) (highBits > lowBits ? high : low)++;  // an even number of passes ends in `keys`
    const auto add = [&](int from, int bits, int n) {
        for (int k = 0; k < n; k++) {
            const int at = bits * k / n, to = bits * (k + 1) / n;
            d.shift[d.passes] = from + at;
            d.bits[d.passes++] = to - at;
        }
    };
    add(lowFrom, lowBits, low);
    add(32, highBits, high);
    return d;
}

int BitsFor(size_t values) {
    int bits = 1;
    while (((size_t)1 << bits) < values) bits++;
    return bits;
}

cudaError_t RadixSort(const Scene* s, unsigned long long* keys, unsigned long long* other, const unsigned* count,
                      size_t capacity, const SortDigits& digits, unsigned* hist, int* err, cudaStream_t st) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)SortBlocks(capacity));
    cfg.blockDim = dim3(kSortThreads);
    cfg.stream = st;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeCooperative;
    attr[0].val.cooperative = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, k_radix_sort, keys, other, count, (unsigned)capacity, digits, hist,
                              s->SortCounter(), err);
}

}  // namespace bepugpu
