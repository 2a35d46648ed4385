// The single-launch form of the tcgen05 tile kernels (ma_flow.inc): which calls take it, and its bf16 instances.
#include "ma_flow.inc"

namespace ma {

cudaError_t launch_flow_f16(const Geometry& g, int* counters, int* host_status, bool wait_expiry, cudaStream_t stream);  // ma_flow_f16.cu

// Blocks of up to 128 in both directions (256 keys would leave room for one CTA per SM beside the ring), and a list of tiles
// that an int can count.
bool flow_supported(const Geometry& g) {
  return g.B <= 128 && g.M <= 128 && (long long)g.E * g.H * 2 * 128 * g.T < 0x7fffffffLL;
}

cudaError_t launch_flow(const Geometry& g, int dtype, int* counters, int* host_status, bool wait_expiry, cudaStream_t stream) {
  if (dtype == MA_B200_BF16) return launch_flow_dtype<__nv_bfloat16>(g, dtype, counters, host_status, wait_expiry, stream);
  return launch_flow_f16(g, counters, host_status, wait_expiry, stream);
}

}  // namespace ma
