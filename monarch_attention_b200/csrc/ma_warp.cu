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
#include "ma_warp_head.inc"
#include "ma_warp_wide.inc"
