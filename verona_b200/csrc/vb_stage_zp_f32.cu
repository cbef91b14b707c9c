// FP32-bulk 3D stages on packed pairs (vb_stage_zp.cuh), a unit of its own for
// the build; flags as vb_stage_f32.cu, whose k_c2p it launches. The dispatch stands
// here and not in the header: any function that is no template would put every
// instantiation of k_stage_zp into each unit that includes the header for the
// packed arithmetic.
#include "vb_stage_zp.cuh"

namespace vb {
extern template cudaError_t launch_c2p<float>(const StageParams&, const StageBufs<float>&, cudaStream_t);
cudaError_t launch_stage_zp(int rec, int rs, const StageParams& p, const StageBufs<float>& b, cudaStream_t s) {
    if (rec == REC_MINMOD) return dispatch_stage_zp_rec<REC_MINMOD>(rs, p, b, s);
    if (rec == REC_PPM) return dispatch_stage_zp_rec<REC_PPM>(rs, p, b, s);
    return dispatch_stage_zp_rec<REC_WENOZ>(rs, p, b, s);
}
}  // namespace vb
