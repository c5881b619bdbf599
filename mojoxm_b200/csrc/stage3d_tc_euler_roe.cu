// Explicit instantiation of the tensor-core 3D stage for one physics.
#include "stage3d_tc_launch.cuh"

namespace mxm {
using PhysF = EulerD<float, FLUX_ROE>;
MXM_INST_TC(PhysF)
}  // namespace mxm
