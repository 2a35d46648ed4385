// Warp-level tensor-core stage kernels for 16-bit inputs with block size and block count up to 128:
// the ViT / RoBERTa / DiT shapes (b = 14..32, N <= 1024, D = 64 or 72) and the b = 64 op sweep.
//
// By bytes these shapes are HBM-bound (intensity ~1.25*b FLOP/B) and their blocks are far smaller than
// a tcgen05 tile, so the job here is to move each operand once, with every row masked / zero-padded in
// flight, and to keep the small contractions on tensor cores: mma.sync m16n8k16 with fp32
// accumulation, fragments read from padded shared-memory tiles with ldmatrix.  Measured, the tiles
// are so small that instruction issue (address arithmetic, softmax, staging) is what bounds them.  One CTA works on one
// tile - (head, key block m) for the right-factor stages, (head, column j) for the left-factor and
// output stages - with one warp per 16 rows.  The row softmax runs on the accumulator fragments
// (a row lives in one quad of lanes), and the normalised factor goes back into the second
// contraction straight from registers (right-factor / output) or through a shared-memory tile that
// is read transposed (left-factor, which contracts over the rows).
//
// Semantics follow the reference stage for stage (reference: ma/ma_torch.py:10-62): invalid keys at
// -inf, row maximum clamped from below at eps, eps in the denominator, floor at FLT_MIN, fully
// masked key blocks give ~0 factors and logit 0, invalid queries zeroed in the left-factor stage
// only, padding rows dropped on output.
#include <math.h>

#include "ma_warp_common.cuh"

// Explicit launcher templates are declared before use in ma_warp_kernels.inc and defined in
// ma_warp_wide.inc, so the public entry points have to come last.
#include "ma_warp_kernels.inc"
#include "ma_warp_wide.inc"

namespace ma {

cudaError_t launch_warp_stage_f32(const Geometry& g, StageKind kind, bool first, cudaStream_t stream);  // ma_warp_f32.cu

bool warp_supported(const Geometry& g, int qk_dtype, int v_dtype, const char** why) {
  if (qk_dtype != v_dtype || (qk_dtype != MA_B200_BF16 && qk_dtype != MA_B200_F16)) {
    *why = "needs bf16 or f16 for q, k and v";
    return false;
  }
  return tile_shape_supported(g, 8, why);
}

cudaError_t launch_warp_stage(const Geometry& g, int qk_dtype, StageKind kind, bool first, cudaStream_t stream) {
  if (qk_dtype == MA_B200_BF16) return launch_warp_kp<__nv_bfloat16>(g, kind, first, stream);
  if (qk_dtype == MA_B200_F32) return launch_warp_stage_f32(g, kind, first, stream);
  return launch_warp_kp<__half>(g, kind, first, stream);
}

}  // namespace ma
