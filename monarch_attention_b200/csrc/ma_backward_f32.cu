// fp32 instances of the backward kernels, in a file of their own to compile in parallel.
#include "ma_backward.inc"

namespace ma {

cudaError_t backward_stage_f32(const BackwardArgs& a, BackwardStage st, size_t* smem_out, cudaStream_t stream) {
  return backward_kp<float>(a, st, smem_out, stream);
}

}  // namespace ma
