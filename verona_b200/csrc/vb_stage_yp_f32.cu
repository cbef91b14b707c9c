// FP32-bulk 2D stages on packed pairs (vb_stage_yp.cuh), a unit of its own for
// the build; flags as vb_stage_f32.cu.
#include "vb_stage_yp.cuh"

namespace vb {
cudaError_t launch_stage_yp(int rec, int rs, const StageParams& p, const StageBufs<float>& b, cudaStream_t s) {
    return dispatch_stage_yp(rec, rs, p, b, s);
}
bool encode_stage_row_tmap(void* out, const float* P, const Grid& g) { return encode_yp_tmap(out, P, g); }
}  // namespace vb
