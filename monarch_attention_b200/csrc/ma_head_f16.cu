// fp16 instances of the head-resident kernel, in a file of their own to compile in parallel.
#include "ma_head.inc"

namespace ma {

cudaError_t launch_head_resident_f16(const Geometry& g, cudaStream_t stream) { return launch_head_dtype<__half>(g, stream); }

}  // namespace ma
