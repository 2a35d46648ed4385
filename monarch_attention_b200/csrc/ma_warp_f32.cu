// fp32 on the tensor path: the warp-level stage kernels on fp32 operands, and their single launch for few heads.
#include <math.h>

#include "ma_warp_common.cuh"

#include "ma_warp_kernels.inc"
#include "ma_warp_head.inc"

namespace ma {

bool tf32x3_supported(const Geometry& g, int qk_dtype, int v_dtype, const char** why) {
  if (qk_dtype != MA_B200_F32 || v_dtype != MA_B200_F32) { *why = "needs f32 for q, k and v"; return false; }
  if (g.B > 128 || g.M > 128) { *why = "needs block size and block count of at most 128"; return false; }
  return tile_shape_supported(g, 4, why);
}

cudaError_t launch_warp_stage_f32(const Geometry& g, StageKind kind, bool first, cudaStream_t stream) {
  return launch_warp_kp<float>(g, kind, first, stream);
}

}  // namespace ma
