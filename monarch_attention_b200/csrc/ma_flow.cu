// The single-launch form of the tcgen05 tile kernels (ma_flow.inc): which calls take it, and its bf16 instances.
#include "ma_flow.inc"

namespace ma {

cudaError_t launch_flow_f16(const Geometry& g, int* counters, int* host_status, bool wait_expiry, cudaStream_t stream);  // ma_flow_f16.cu

namespace {
__global__ void clear_kernel(uint4* p, int n) {
  grid_wait();
  dependents_may_start();  // (not before: see grid_wait's comment on tensor memory)
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) p[i] = make_uint4(0u, 0u, 0u, 0u);
}
}  // namespace

// The kernel behind this one comes up and sets up its tensor memory meanwhile, which it cannot do under a memset.
cudaError_t launch_clear(void* p, size_t bytes, cudaStream_t stream) {
  int pieces = (int)((bytes + 15) / 16);
  void* params[] = {(void*)&p, (void*)&pieces};
  return launch_kernel((const void*)clear_kernel, dim3(std::min(32, (pieces + 2047) / 2048)), dim3(256), params, 0, stream);
}

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
