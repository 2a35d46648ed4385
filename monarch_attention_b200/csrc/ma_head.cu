#include "ma_head.inc"

namespace ma {

cudaError_t launch_head_resident_f16(const Geometry& g, cudaStream_t stream);  // ma_head_f16.cu

bool head_resident_supported(const Geometry& g, int qk_dtype, int v_dtype, const char** why) {
  if (!warp_supported(g, qk_dtype, v_dtype, why)) return false;
  if (g.B > 32 || g.M > 32) { *why = "needs block size and block count of at most 32"; return false; }
  return true;
}

cudaError_t launch_head_resident(const Geometry& g, int qk_dtype, cudaStream_t stream) {
  if (qk_dtype == MA_B200_BF16) return launch_head_dtype<__nv_bfloat16>(g, stream);
  return launch_head_resident_f16(g, stream);
}

}  // namespace ma
