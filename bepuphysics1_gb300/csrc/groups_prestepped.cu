// The island-group kernels of the split prologue (groups_launch.cuh with
// kPrestepped): a translation unit of their own, so the two sets compile side
// by side.
#include "groups_launch.cuh"

namespace bepugpu {

bepugpu_status LaunchPrestepped(Context* ctx, Scene* s, const StepParams& p, uint32_t flags, bool count,
                                const GroupTables& t, int* launches) {
    return LaunchClasses<true>(ctx, s, p, flags, count, t, launches);
}

}  // namespace bepugpu
