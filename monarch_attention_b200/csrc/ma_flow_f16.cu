// fp16 instances of the single-launch tile kernels, in a file of their own to compile in parallel.
#include "ma_flow.inc"

namespace ma {

cudaError_t launch_flow_f16(const Geometry& g, int* counters, int* host_status, bool wait_expiry, cudaStream_t stream) {
  return launch_flow_dtype<__half>(g, MA_B200_F16, counters, host_status, wait_expiry, stream);
}

}  // namespace ma
