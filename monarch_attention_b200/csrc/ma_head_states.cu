// bf16 instances of the kernel that recomputes the backward pass's stage inputs, in a file of their own to compile in parallel.
#include "ma_head.inc"

namespace ma {

cudaError_t launch_head_states_f16(const Geometry& g, const BackwardStates& s, cudaStream_t stream);  // ma_head_states_f16.cu

// Where that is faster than a launch per stage: small tiles, or few heads, whose parts have an SM each.  One iteration is one launch
// either way.  Forward and backward, us, single launch / launch per stage: 168 heads of 16 x 16 x 32, three iterations, 84 / 98, 720 204 /
// 239; 768 of 15 x 14 x 64 with two 220 / 235, 240 of 32 x 16 with three 279 / 293, 192 of 10 x 30 x 80 163 / 160; 48 of 32 x 32 x 64
// with three 158.5 / 166, 72 of 30 x 30 x 72 with two 152.4 / 153.4; many heads of long blocks on the other side: 96 of 32 x 32 x 80
// with two 243 / 233, 156 of 30 x 30 x 64 with three 411 / 399.
bool head_states_pay(const Geometry& g, int dtype) {
  if (dtype == MA_B200_F32 || g.T == 1 || g.B > 32 || g.M > 32) return false;
  if (g.D != 32 && g.D != 64 && g.D != 72 && g.D != 80) return false;
  return g.B <= 16 || g.M <= 16 || g.E * g.H * ((g.B + 15) / 16) <= sm_count();
}

cudaError_t launch_head_states(const Geometry& g, int dtype, const BackwardStates& s, cudaStream_t stream) {
  if (dtype == MA_B200_F16) return launch_head_states_f16(g, s, stream);
  return launch_states_dtype<__nv_bfloat16>(g, KeptArgs{s.al, s.ar, s.y, s.cl, s.cr, s.mat, s.vec}, stream);
}

}  // namespace ma
