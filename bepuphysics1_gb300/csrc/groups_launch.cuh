// The island-group kernel and its launches, instantiated for the in-kernel
// prologue (groups.cu) and the split one (groups_prestepped.cu).
#pragma once

#include <cuda_runtime.h>

#include <algorithm>

#include "../../include/bepugpu.h"
#include "bepugpu_internal.h"
#include "groups_device.cuh"
#include "solver_device.cuh"

namespace bepugpu {

template <bool kCensus, bool kShared, int kJoints, bool kPrestepped>
__global__ void k_groups(ManifoldSoA m, BodySoA b, JointSoA j, StepParams p, uint32_t flags, GroupTables t,
                         int groupBase, int Bc, int Lc, int Jc, unsigned long long* census, bool nonConvex) {
    extern __shared__ float4 smem[];
    const GroupDesc g = t.groups[groupBase + blockIdx.x];
    GroupStep<kCensus, kShared, kJoints, kPrestepped>(m, b, j, p, flags, t, g, Bc, Lc, Jc, smem, census, nonConvex);
}

inline int ClassThreads(const GroupClass& c, int override_) {
    if (override_ > 0) return override_;
    int t = ((c.maxColourMembers + 31) / 32) * 32;
    return std::min(std::max(t, 32), 256);
}

template <bool kShared, int kJoints, bool kPrestepped>
bepugpu_status LaunchClass(Context* ctx, Scene* s, const GroupClass& c, const StepParams& p, uint32_t flags,
                           bool count, GroupTables t, cudaStream_t stream, int* launches) {
    if (c.end <= c.begin) return BEPUGPU_OK;
    const int Bc = std::max(c.maxLocal, 1), Lc = std::max(c.maxManifolds, 1), Jc = std::max(c.maxJoints, 1);
    const bool nonConvex = s->groupPlan.nonConvexLanes;
    size_t smemBytes = GroupSmemBytes(kShared, Bc, Lc, kJoints ? Jc : 0, nonConvex);
    cudaError_t e = cudaSuccess;
    if (smemBytes > 48 * 1024) {
        e = cudaFuncSetAttribute(k_groups<false, kShared, kJoints, kPrestepped>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 (int)smemBytes);
        if (e == cudaSuccess)
            e = cudaFuncSetAttribute(k_groups<true, kShared, kJoints, kPrestepped>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                     (int)smemBytes);
        if (e != cudaSuccess) {
            ctx->SetError("group kernel shared memory %zu bytes: %s", smemBytes, cudaGetErrorString(e));
            return BEPUGPU_CUDA_ERROR;
        }
    }
    const unsigned blocks = (unsigned)(c.end - c.begin);
    int threads = ClassThreads(c, s->groupThreadsOverride);
    if (kJoints && s->groupThreadsOverride <= 0) {
        // More warps for the joints' types while every group stays resident: in
        // one warp the types of a colour run one after another.  384 chains of
        // the added types: 189 -> 132 us a step with the launches beside each
        // other; 256 threads measured the same.
        for (int t = 128; t > threads; t /= 2) {
            int perSm = 0;
            if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&perSm, k_groups<false, kShared, kJoints, kPrestepped>, t,
                                                              smemBytes) == cudaSuccess &&
                blocks <= (unsigned)(perSm * ctx->smCount)) {
                threads = t;
                break;
            }
        }
    }
    // the thread's last error must be this launch's own
    const cudaError_t earlier = cudaGetLastError();
    if (count)
        k_groups<true, kShared, kJoints, kPrestepped><<<blocks, threads, smemBytes, stream>>>(
            s->m, s->b, s->j, p, flags, t, c.begin, Bc, Lc, Jc, s->Census(), nonConvex);
    else
        k_groups<false, kShared, kJoints, kPrestepped><<<blocks, threads, smemBytes, stream>>>(
            s->m, s->b, s->j, p, flags, t, c.begin, Bc, Lc, Jc, nullptr, nonConvex);
    if (launches) (*launches)++;
    e = cudaGetLastError();
    if (e != cudaSuccess) {
        ctx->SetError("group kernel launch (%u CTAs of %d threads, %zu bytes of shared memory): %s%s%s", blocks,
                      threads, smemBytes, cudaGetErrorString(e), earlier != cudaSuccess ? "; earlier error: " : "",
                      earlier != cudaSuccess ? cudaGetErrorString(earlier) : "");
        return BEPUGPU_CUDA_ERROR;
    }
    return BEPUGPU_OK;
}


// Every kind of group: without joints, then with (any joint type when
// addedJointTypes, else the classic ones only).
template <bool kPrestepped>
bepugpu_status LaunchClasses(Context* ctx, Scene* s, const StepParams& p, uint32_t flags, bool count, GroupTables t,
                             int* launches) {
    const GroupPlan& g = s->groupPlan;
    const bool contacts = g.shared.end > g.shared.begin || g.global.end > g.global.begin;
    // Joint and contact groups share no dynamic body: the joint launches, the
    // longer ones, run on a stream (a branch of a captured graph) of their own.
    const bool beside = g.groupJoints && contacts && s->sideStream;
    const cudaStream_t jq = beside ? s->sideStream : s->stream;
    bepugpu_status st = BEPUGPU_OK;
    auto order = [&](cudaEvent_t done, cudaStream_t from, cudaStream_t to) {
        if (!beside || st != BEPUGPU_OK) return;
        cudaError_t e = cudaEventRecord(done, from);
        if (e == cudaSuccess) e = cudaStreamWaitEvent(to, done, 0);
        if (e != cudaSuccess) {
            ctx->SetError("group streams: %s", cudaGetErrorString(e));
            st = BEPUGPU_CUDA_ERROR;
        }
    };
    order(s->evSide[0], s->stream, jq);
    if (s->addedJointTypes) {
        if (st == BEPUGPU_OK)
            st = LaunchClass<true, 2, kPrestepped>(ctx, s, g.sharedJoints, p, flags, count, t, jq, launches);
        if (st == BEPUGPU_OK)
            st = LaunchClass<false, 2, kPrestepped>(ctx, s, g.globalJoints, p, flags, count, t, jq, launches);
    } else {
        if (st == BEPUGPU_OK)
            st = LaunchClass<true, 1, kPrestepped>(ctx, s, g.sharedJoints, p, flags, count, t, jq, launches);
        if (st == BEPUGPU_OK)
            st = LaunchClass<false, 1, kPrestepped>(ctx, s, g.globalJoints, p, flags, count, t, jq, launches);
    }
    if (st == BEPUGPU_OK) st = LaunchClass<true, 0, kPrestepped>(ctx, s, g.shared, p, flags, count, t, s->stream, launches);
    // (the census of an instrumented step counts the visits of the group kernel)
    if (st == BEPUGPU_OK)
        st = !count && FlowGroups(g)
                 ? LaunchFlowGroups(ctx, s, p, flags, t, kPrestepped, launches)
                 : LaunchClass<false, 0, kPrestepped>(ctx, s, g.global, p, flags, count, t, s->stream, launches);
    order(s->evSide[1], jq, s->stream);
    return st;
}

}  // namespace bepugpu
