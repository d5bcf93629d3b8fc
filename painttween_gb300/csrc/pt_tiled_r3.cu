// pt_tiled_r3.cu -- tiled patch-distance kernels instantiated for patch radius 3.
#include "pt_energy.cuh"

namespace pt {
cudaError_t launch_tiled_3(int kind, int tm, const Params& P, const TileMaps& M, PatchPlanes work, int arg,
                           uint32_t pass_id, float* out, int wide, bool dependent, cudaStream_t s) {
    return ptk::launch_tiled_r<3>(kind, tm, P, M, work, arg, pass_id, out, wide, dependent, s);
}
}  // namespace pt
