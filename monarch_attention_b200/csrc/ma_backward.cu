// Backward pass: which problems it takes, its workspace, its launches, and the bf16 instances of its kernels (ma_backward.inc).
#include "ma_backward.inc"

namespace ma {

cudaError_t backward_stage_f16(const BackwardArgs& a, BackwardStage st, size_t* smem_out, cudaStream_t stream);  // ma_backward_f16.cu
cudaError_t backward_stage_f32(const BackwardArgs& a, BackwardStage st, size_t* smem_out, cudaStream_t stream);  // ma_backward_f32.cu

namespace {

cudaError_t backward_stage(const BackwardArgs& a, int dtype, BackwardStage st, size_t* smem_out, cudaStream_t stream) {
  if (dtype == MA_B200_BF16) return backward_kp<__nv_bfloat16>(a, st, smem_out, stream);
  if (dtype == MA_B200_F16) return backward_stage_f16(a, st, smem_out, stream);
  return backward_stage_f32(a, st, smem_out, stream);
}

size_t align256(size_t x) { return (x + 255) / 256 * 256; }

}  // namespace

bool backward_supported(const Geometry& g, int qk_dtype, int v_dtype, const char** why) {
  const bool ok = qk_dtype == MA_B200_F32 ? tf32x3_supported(g, qk_dtype, v_dtype, why) : warp_supported(g, qk_dtype, v_dtype, why);
  if (!ok) return false;
  // fp32: the operand tiles of a 128 x 128 stage would need 360 KB of shared memory
  const int most = qk_dtype == MA_B200_F32 ? 64 : 128;
  if (g.B > most || g.M > most) { *why = "needs block size and block count of at most 128 (fp32: 64)"; return false; }
  BackwardArgs a{};
  a.g = g;
  const BackwardStage stages[] = {kBackOutput, kBackRightWithV};  // the ones that need the most shared memory
  for (BackwardStage st : stages) {
    size_t smem = 0;
    backward_stage(a, qk_dtype, st, &smem, nullptr);
    if (smem > kMaxSmem) { *why = "a tile of the backward pass does not fit in shared memory"; return false; }
  }
  return true;
}

BackwardLayout backward_layout(const Geometry& g, int qk_dtype) {
  const size_t EH = (size_t)g.E * g.H, rows = EH * g.M * g.B, es = qk_dtype == MA_B200_F32 ? 4 : 2;
  const size_t mat = align256(rows * g.D * es), vec = align256(rows * sizeof(float)), acc = align256(rows * g.D * sizeof(float));
  BackwardLayout L;
  size_t off = 256;  // status word
  auto take = [&](size_t n) { const size_t o = off; off += n; return o; };
  L.mat = mat;
  L.vec = vec;
  L.al = take(mat * g.T);
  L.ar = take(mat * (g.T - 1));
  L.cl = take(vec * g.T);
  L.cr = take(vec * (g.T - 1));
  L.y = take(mat);
  L.dal = take(mat);
  L.dy = take(mat);
  L.dar = take(g.T > 1 ? mat : 0);
  L.dcl = take(vec);
  L.dcr = take(g.T > 1 ? vec : 0);
  L.dq_acc = take(acc);
  L.dk_acc = take(g.T > 1 ? acc : 0);
  L.total = off;
  return L;
}

cudaError_t launch_backward(const Geometry& g0, int dtype, const View4& dz, const View4& dq, const View4& dk, const View4& dv,
                            void* workspace, cudaStream_t stream) {
  const BackwardLayout L = backward_layout(g0, dtype);
  char* ws = static_cast<char*>(workspace);
  auto at_iteration = [&](int right_it, int col_it) {  // stage inputs: ar, cr of right_it (> 0), al, cl of col_it
    Geometry g = g0;
    g.status = reinterpret_cast<int*>(ws);
    g.ar = right_it > 0 ? ws + L.ar + L.mat * (right_it - 1) : nullptr;
    g.cr = right_it > 0 ? reinterpret_cast<float*>(ws + L.cr + L.vec * (right_it - 1)) : nullptr;
    g.al = ws + L.al + L.mat * col_it;
    g.cl = reinterpret_cast<float*>(ws + L.cl + L.vec * col_it);
    g.y = ws + L.y;
    return g;
  };
  cudaError_t e;
  const int T = g0.T;
  // ---- the forward stages, every iteration's state kept ---------------------------------------------------
  if (head_states_pay(g0, dtype)) {
    const BackwardStates s{ws + L.al, ws + L.ar, ws + L.y, reinterpret_cast<float*>(ws + L.cl), reinterpret_cast<float*>(ws + L.cr),
                           (long long)L.mat, (long long)L.vec};
    if ((e = launch_head_states(at_iteration(0, 0), dtype, s, stream)) != cudaSuccess) return e;
  } else {
    for (int t = 0; t < T; ++t) {
      if ((e = launch_warp_stage(at_iteration(t, t), dtype, t == T - 1 ? kStageRightWithV : kStageRight, t == 0, stream)) != cudaSuccess)
        return e;
      if (t < T - 1)
        if ((e = launch_warp_stage(at_iteration(t + 1, t), dtype, kStageLeft, false, stream)) != cudaSuccess) return e;
    }
  }
  // ---- and back -------------------------------------------------------------------------------------------
  BackwardArgs a{};
  a.dz = dz; a.dq = dq; a.dk = dk; a.dv = dv;
  a.dal = ws + L.dal; a.dy = ws + L.dy; a.dar = ws + L.dar;
  a.dcl = reinterpret_cast<float*>(ws + L.dcl);
  a.dcr = reinterpret_cast<float*>(ws + L.dcr);
  a.dq_acc = reinterpret_cast<float*>(ws + L.dq_acc);
  a.dk_acc = reinterpret_cast<float*>(ws + L.dk_acc);
  for (int t = T - 1; t >= 0; --t) {
    a.g = at_iteration(t, t);
    a.first = t == 0;
    a.accumulate = t < T - 1;
    if (t == T - 1) {
      if ((e = backward_stage(a, dtype, kBackOutput, nullptr, stream)) != cudaSuccess) return e;
      if ((e = backward_stage(a, dtype, kBackRightWithV, nullptr, stream)) != cudaSuccess) return e;
    } else {
      // left-factor update of iteration t: al, cl of t in, ar, cr of t + 1 out
      if ((e = backward_stage(a, dtype, kBackLeft, nullptr, stream)) != cudaSuccess) return e;
      if ((e = backward_stage(a, dtype, kBackRight, nullptr, stream)) != cudaSuccess) return e;
    }
  }
  return cudaSuccess;
}

}  // namespace ma
