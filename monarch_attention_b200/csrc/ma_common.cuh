// Shared definitions for the MonarchAttention kernels (sm_100a).
#pragma once

#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include <atomic>
#include <map>
#include <mutex>
#include <utility>

#include "../../include/monarch_attention_b200.h"

namespace ma {

constexpr float kEps = 1e-12f;            // eps of the right-factor stages (reference: ma/ma_torch.py:10)
constexpr float kTiny = 1.17549435e-38f;  // smallest normal fp32: floor of the right-factor entries (:18)

// A strided (E,H,N,W) view; strides in elements, innermost stride 1.
struct View4 {
  const void* ptr;
  long long se, sh, sn;
};

// Everything a stage kernel needs to know about one forward call.
struct Geometry {
  int E, H, N, D, Dv;
  int B, M;        // block size, number of blocks
  int pad_off;     // padded position p = m*B + j maps to token p - pad_off
  int T;
  float sm_scale;  // (float)(1/sqrt(D))
  View4 q, k, v, out;
  const uint8_t* mask;  // (E,N) values of mask_type, non-zero = valid; or nullptr
  long long mask_se;    // elements
  int mask_type;        // MA_B200_MASK_*
  // stage-to-stage state (workspace)
  void* ar;   // (EH, M, B, D)  qk dtype
  float* cr;  // (EH, M, B)
  void* al;   // (EH, B, M, D)  qk dtype
  float* cl;  // (EH, B, M)
  void* y;    // (EH, B, M, Dv) v dtype
  int* status;  // device flag, 0 = fine
};

enum StageKind { kStageRight = 0, kStageRightWithV = 1, kStageLeft = 2, kStageOutput = 3 };

template <typename T>
struct Cvt;
template <>
struct Cvt<float> {
  static __device__ __forceinline__ float to_f(float x) { return x; }
  static __device__ __forceinline__ float from_f(float x) { return x; }
};
template <>
struct Cvt<__nv_bfloat16> {
  static __device__ __forceinline__ float to_f(__nv_bfloat16 x) { return __bfloat162float(x); }
  static __device__ __forceinline__ __nv_bfloat16 from_f(float x) { return __float2bfloat16_rn(x); }
};
template <>
struct Cvt<__half> {
  static __device__ __forceinline__ float to_f(__half x) { return __half2float(x); }
  static __device__ __forceinline__ __half from_f(float x) { return __float2half_rn(x); }
};

// Round an fp32 value through storage type T and back (the reference rounds every
// contraction result to the storage dtype before the fp32 softmax arithmetic).
template <typename T>
__device__ __forceinline__ float round_through(float x) {
  return Cvt<T>::to_f(Cvt<T>::from_f(x));
}

// Lets `fn` use up to `bytes` of dynamic shared memory on the current device.  The runtime call takes longer than
// queuing a launch, so it is made only when a larger size than before is asked for.
inline cudaError_t allow_dynamic_smem(const void* fn, size_t bytes) {
  if (bytes <= 48 * 1024) return cudaSuccess;
  static std::mutex mutex;
  static std::map<std::pair<int, const void*>, size_t> allowed;
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return e;
  std::lock_guard<std::mutex> lock(mutex);
  size_t& have = allowed[{dev, fn}];
  if (bytes <= have) return cudaSuccess;
  e = cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
  if (e == cudaSuccess) have = bytes;
  return e;
}

// Stage kernels that follow one another ask for one split of an SM's memory, all of it shared memory.  The driver chooses it by what a
// kernel needs, and an SM empties before it changes: stages whose tiles differ (16 x 48 keys beside 64, left factor beside right) then
// wait for one another in full, whatever the launches allow.  Warp-level kernels on 16-bit tensors, us, with the driver's choice / with one
// split: 4 heads of 40 x 49 x 64, one iteration, 13.5 / 8.8 (9.5 when both stages padded their keys to 64), of 33 x 48 12.6 / 7.9, of 32 x 32
// with two 20.4 / 14.1, 12 of 33 x 48 x 64 with three 43.9 / 33.9; 374 calls and training steps 0.955 as a geometric mean, 1.04 at the most.
// The fp32 kernels spill into the L1 cache that is left and keep the driver's choice (4 heads of 120 x 120 x 64, one iteration, 194 / 200).
// `done`: devices that have been told, a bit each.
inline cudaError_t prefer_shared_memory(const void* fn, std::atomic<unsigned long long>& done) {
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess || dev >= 64) return e;
  if (done.load(std::memory_order_relaxed) >> dev & 1) return cudaSuccess;
  e = cudaFuncSetAttribute(fn, cudaFuncAttributePreferredSharedMemoryCarveout, cudaSharedmemCarveoutMaxShared);
  if (e == cudaSuccess) done.fetch_or(1ull << dev, std::memory_order_relaxed);
  return e;
}

// Multiprocessors of the current device (where there is none, as in a layout query: those of a B200).
inline int sm_count() {
  static std::atomic<int> counts[64];
  int dev = 0, n = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return 148;
  if ((n = counts[dev].load(std::memory_order_relaxed)) == 0 &&
      cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev) == cudaSuccess)
    counts[dev].store(n, std::memory_order_relaxed);
  return n > 0 ? n : 148;
}

// Whether the mask lets token n of batch element e through.  The callers' masks come as booleans, integers or floats
// (-0.0 is zero); reading them as they are saves a conversion kernel in front of every call.
__device__ __forceinline__ bool mask_lets(const Geometry& g, int e, int n) {
  if (g.mask == nullptr) return true;
  const long long i = (long long)e * g.mask_se + n;
  switch (g.mask_type) {
    case MA_B200_MASK_I64: return reinterpret_cast<const unsigned long long*>(g.mask)[i] != 0;
    case MA_B200_MASK_F32: return (reinterpret_cast<const uint32_t*>(g.mask)[i] & 0x7fffffffu) != 0;
    case MA_B200_MASK_I32: return reinterpret_cast<const uint32_t*>(g.mask)[i] != 0;
    case MA_B200_MASK_F16: return (reinterpret_cast<const uint16_t*>(g.mask)[i] & 0x7fffu) != 0;
    case MA_B200_MASK_I16: return reinterpret_cast<const uint16_t*>(g.mask)[i] != 0;
    case MA_B200_MASK_F64: return (reinterpret_cast<const unsigned long long*>(g.mask)[i] << 1) != 0;
    default: return g.mask[i] != 0;
  }
}

// Kernels are launched with programmatic dependence on whatever precedes them in the stream, another library's kernel included:
// the GPU then prepares the launch while that kernel ends, and the kernel waits at its start (grid_wait), before it touches
// memory, until everything before it is complete and visible.  A plain launch costs more than its work here: launches of a
// kernel that spins for t us follow one another every ceil((t + 2) / 2.05) * 2.05 us (2 us: 4.11, 3: 6.16, 10: 12.31, 16: 18.45; 148 and
// 768 CTAs), with the dependence every t + 0.8 (148 CTAs) to t + 1.0 (768), and 2.05 at the least.
// A stage kernel that another stage follows also lets that one's CTAs come up at once (stage_begin), under its own tail: 256 fp32
// tokens, two launches, 15.4 to 13.3 us; six launches 84 to 75.  The last kernel of a call does not, so that a small grid behind
// it finds all SMs free and spreads evenly, nor do the tcgen05 tile kernels: their early CTAs took instruction fetch from the
// running stage.
// A kernel that allocates tensor memory does so behind grid_wait, or behind a kernel that has passed its own: a kernel in front
// that lets its dependents start before it has tensor memory of its own would wait for ours, and we for its end.
inline cudaError_t launch_kernel(const void* fn, dim3 grid, dim3 block, void** args, size_t smem, cudaStream_t stream, int cluster = 1) {
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = grid;
  cfg.blockDim = block;
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  cudaLaunchAttribute attrs[2] = {};
  attrs[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attrs[0].val.programmaticStreamSerializationAllowed = 1;
  attrs[1].id = cudaLaunchAttributeClusterDimension;
  attrs[1].val.clusterDim.x = cluster;
  attrs[1].val.clusterDim.y = attrs[1].val.clusterDim.z = 1;
  cfg.attrs = attrs;
  cfg.numAttrs = cluster > 1 ? 2 : 1;
  return cudaLaunchKernelExC(&cfg, fn, args);
}
__device__ __forceinline__ void grid_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void dependents_may_start() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
__device__ __forceinline__ void stage_begin() {
  dependents_may_start();
  grid_wait();
}

// Host-side launchers implemented by the kernel translation units.
// Each returns cudaSuccess or the launch error.
// Test hook: 1 = the generic family always runs its general (warp-per-row) form.
void generic_set_general_form_only(int on);
cudaError_t launch_generic_stage(const Geometry& g, int qk_dtype, int v_dtype, StageKind kind, bool first,
                                 cudaStream_t stream);
size_t generic_stage_smem_bytes(const Geometry& g, StageKind kind);

// Warp-level tensor-core stage kernels (block size and count <= 256, D <= 80).
bool warp_supported(const Geometry& g, int qk_dtype, int v_dtype, const char** why);
// The same kernels on fp32 tensors (products of split operands on the tf32 tensor path).
bool tf32x3_supported(const Geometry& g, int qk_dtype, int v_dtype, const char** why);
cudaError_t launch_warp_stage(const Geometry& g, int qk_dtype, StageKind kind, bool first, cudaStream_t stream);

// Backward pass (ma_backward.cu): byte offsets in its workspace; al, ar, cl, cr hold one entry per iteration.
struct BackwardLayout {
  size_t mat, vec;  // bytes of one (EH, M*B, D) tensor / (EH, M*B) vector
  size_t al, ar, cl, cr, y, dal, dy, dar, dcl, dcr, dq_acc, dk_acc, total;
};
bool backward_supported(const Geometry& g, int qk_dtype, int v_dtype, const char** why);
BackwardLayout backward_layout(const Geometry& g, int qk_dtype);
cudaError_t launch_backward(const Geometry& g, int dtype, const View4& dz, const View4& dq, const View4& dk, const View4& dv,
                            void* workspace, cudaStream_t stream);

// Head-resident kernel: all stages of a head in one launch, block size and count up to 32 (ma_head.cu).
bool head_resident_supported(const Geometry& g, int qk_dtype, int v_dtype, const char** why);
cudaError_t launch_head_resident(const Geometry& g, int qk_dtype, cudaStream_t stream);
// The same kernel under the narrower limits of the HEAD_FUSED family.
bool head_fused_supported(const Geometry& g, int qk_dtype, int v_dtype, const char** why);

// Tensor-core (tcgen05) path.
bool tc_supported(const Geometry& g, int qk_dtype, int v_dtype, const char** why);
// The TMA tensor maps of one call.  tc_plan_get copies them into *plan, from a cache when the same
// pointers, strides and sizes were seen before; tc_plan_create always encodes (heap object).
struct TcPlan;
int tc_plan_get(const Geometry& g, int qk_dtype, TcPlan* plan, const char** err);
int tc_plan_create(const Geometry& g, int qk_dtype, TcPlan** plan, const char** err);
void tc_plan_destroy(TcPlan* plan);
// All stages of the fp32 tensor path (TF32X3) in one launch, for block size and count up to 32 (ma_warp_head.inc).
bool head_f32_pays(const Geometry& g);
cudaError_t launch_head_f32(const Geometry& g, cudaStream_t stream);
// The stage inputs of the backward pass in one launch, where the head-resident kernel has tiles for the shape (ma_head_states.cu): al
// and y (EH, B, M, D), ar (EH, M, B, D), cl (EH, B, M), cr (EH, M, B); those of an iteration `mat` and `vec` bytes behind those of
// the one before, ar and cr from the second iteration on.
struct BackwardStates {
  char *al, *ar, *y;
  float *cl, *cr;
  long long mat, vec;
};
bool head_states_pay(const Geometry& g, int dtype);
cudaError_t launch_head_states(const Geometry& g, int dtype, const BackwardStates& s, cudaStream_t stream);
// Persistent fused kernel: stages [stage_begin, stage_end) of the 2T stages in one cooperative launch.
size_t fused_counter_bytes(const Geometry& g);
// (spin_limit: iterations of the dependency wait before it gives up, 0 = default; for the wait-expiry self-test.)
cudaError_t launch_fused(const TcPlan* plan, const Geometry& g, int* counters, int stage_begin, int stage_end,
                         int wait_deps, int spin_limit, cudaStream_t stream);
// Device address of the mapped host word that a kernel whose bounded wait gave up stores its code in (nullptr: none).
int* host_status_word(int device);
// tcgen05 stage kernels, one 128-row tile per CTA: block size and count up to 256, D <= 64, masks and padding (ma_tile.cu).
bool tile_supported(const Geometry& g, int qk_dtype, int v_dtype, const char** why);
// wait_expiry (self-test): a wait of every CTA runs out.
cudaError_t launch_tile_stage(const Geometry& g, int dtype, StageKind kind, bool first, int* host_status, bool wait_expiry, cudaStream_t stream);
// Their single-launch form, all stages of a call, for block size and count up to 128 (ma_flow.cu); counters: (E*H, 2T)
// zeroed ints, as the status block.  wait_expiry (self-test): the first stage is left out, so that the waits for it run out.
bool flow_supported(const Geometry& g);
// `bytes` from p on to zero, rounded up to whole pieces of 16; p on a 16-byte boundary.
cudaError_t launch_clear(void* p, size_t bytes, cudaStream_t stream);
cudaError_t launch_flow(const Geometry& g, int dtype, int* counters, int* host_status, bool wait_expiry, cudaStream_t stream);
// Code of a bounded device-side wait that gave up on `device` since the last poll (0 = none); reads a mapped
// host word, so it needs no synchronisation.
int fused_poll_status(int device);

}  // namespace ma
