// fp16 instances of the kernel that recomputes the backward pass's stage inputs, in a file of their own to compile in parallel.
#include "ma_head.inc"

namespace ma {

cudaError_t launch_head_states_f16(const Geometry& g, const BackwardStates& s, cudaStream_t stream) {
  return launch_states_dtype<__half>(g, KeptArgs{s.al, s.ar, s.y, s.cl, s.cr, s.mat, s.vec}, stream);
}

}  // namespace ma
