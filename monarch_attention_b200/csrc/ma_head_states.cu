// bf16 instances of the kernel that recomputes the backward pass's stage inputs, in a file of their own to compile in parallel.
#include "ma_head.inc"

namespace ma {

cudaError_t launch_head_states_f16(const Geometry& g, const BackwardStates& s, cudaStream_t stream);  // ma_head_states_f16.cu

// Where that is faster than a launch per stage whatever the number of heads: both tiles of up to 16, or one of them and a width of up to
// 64.  The shape of a head alone decides, as the two differ in the last bits and a head's gradients are the same in any batch and on
// any rank.  One iteration is one launch either way.  Forward and backward by the single launch over a launch per stage, 4 to 720
// heads, two and three iterations, geometric mean (least gain): tiles of 16 x 16, widths 32 and 64, 0.77 to 0.87 (0.95), 72 and 80
// 0.84 to 0.92 (1.00); 16 x 32 and 32 x 16, width 32, 0.84 to 0.88 (1.00), width 64 0.88 to 0.94 (1.016, and 1.044 and 1.026 at 48 heads of
// 8 x 32 and 10 x 30); 72 and 80 would have 0.90 to 1.00 (1.12).  Tiles of 32 x 32: 0.92 to 1.01 (1.13), faster with some numbers of
// heads and slower with others (us, two iterations: 75 of 32 x 32 x 72 204 / 188, 96 of 32 x 32 x 80 239 / 229; with three 48 of 32 x 32 x
// 64 142 / 154).  On this side, us: 144 of 16 x 16 x 32, three iterations, 64 / 83, 720 198 / 228; with two 720 of 15 x 14 x 64 200 / 215, 144 of
// 29 x 16 x 64 112 / 120.  Widths that have no tiles of their own in the head-resident kernel keep the stage launches.
bool head_states_pay(const Geometry& g, int dtype) {
  if (dtype == MA_B200_F32 || g.T == 1 || g.B > 32 || g.M > 32) return false;
  const bool small = g.B <= 16 && g.M <= 16, narrow = g.D == 32 || g.D == 64;
  return (small && (narrow || g.D == 72 || g.D == 80)) || (narrow && (g.B <= 16 || g.M <= 16));
}

cudaError_t launch_head_states(const Geometry& g, int dtype, const BackwardStates& s, cudaStream_t stream) {
  if (dtype == MA_B200_F16) return launch_head_states_f16(g, s, stream);
  return launch_states_dtype<__nv_bfloat16>(g, KeptArgs{s.al, s.ar, s.y, s.cl, s.cr, s.mat, s.vec}, stream);
}

}  // namespace ma
