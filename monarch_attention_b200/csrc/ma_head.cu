#include "ma_head.inc"

namespace ma {

cudaError_t launch_head_resident_f16(const Geometry& g, cudaStream_t stream);  // ma_head_f16.cu

bool head_resident_supported(const Geometry& g, int qk_dtype, int v_dtype, const char** why) {
  if (!warp_supported(g, qk_dtype, v_dtype, why)) return false;
  if (g.B > 32 || g.M > 32) { *why = "needs block size and block count of at most 32"; return false; }
  return true;
}

// The limits that callers of HEAD_FUSED know: Q, K, V, al and y of the head, in rows spaced by eight elements, and what a
// kernel of sixteen warps kept beside them, within 227 KB.  (The kernel that had the name took 39.2 us for 64 images of 12 heads of
// 197 tokens and 10.7 us for one; this one takes 22.7 and 9.0.)
bool head_fused_supported(const Geometry& g, int qk_dtype, int v_dtype, const char** why) {
  auto no = [&](const char* w) { *why = w; return false; };
  if (!warp_supported(g, qk_dtype, v_dtype, why)) return false;
  if (g.T != 1) return no("single-launch head kernel handles one iteration (T = 1)");
  if (g.B > 32 || g.M > 32 || g.D > 64) return no("needs block size and block count <= 32 and D <= 64");
  const size_t kc = g.B > 16 ? 32 : 16, kd = g.M > 16 ? 32 : 16, rows = (size_t)g.B * g.M, pitch = (g.D > 32 ? 64 : 32) + 8;
  const size_t elements = (5 * rows + 2 * kc + 2 * kd + 16 + 1 + 16 * 16) * pitch;
  if (2 * elements + 4 * ((rows + 3) / 4 * 4 + 16 * (kc > kd ? kc : kd)) > 227 * 1024)
    return no("the head's Q, K, V, al and y do not fit in shared memory");
  return true;
}

cudaError_t launch_head_resident(const Geometry& g, int qk_dtype, cudaStream_t stream) {
  if (qk_dtype == MA_B200_BF16) return launch_head_dtype<__nv_bfloat16>(g, stream);
  return launch_head_resident_f16(g, stream);
}

}  // namespace ma
