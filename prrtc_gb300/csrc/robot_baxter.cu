// Kernels for pRRTC's baxter robot (model: robots/baxter_fkcc.cuh).
#include "device_common.cuh"
#include "robots/baxter_fkcc.cuh"
#include "robot_kernels.cuh"

PRRTC_GEN_ADAPTER(GenBaxter, gen_baxter)

namespace prrtc {
// Within 1e-8 m of contact a verdict depends on how the exact form's products
// are contracted.  Baxter's edges of more than 96 points have it from a build
// with 64 registers and the form compiled in; the called form, which shorter
// edges have, differs from it on 2.5 % of configurations bisected onto contact
// (the other robots' builds agree).  2^14 edges of 128 points in clutter 2.29 ms,
// 2.09 with the called form (5.66 testing every obstacle).
template <>
struct LongEdges<GenBaxter> {
    using Ctx = SingleCheckCtx;
    static constexpr int kMinBlocks = 8;
};

RobotOps robot_ops_baxter() { return RobotKernels<GenBaxter>::ops(GenBaxter::kDof); }
}  // namespace prrtc
