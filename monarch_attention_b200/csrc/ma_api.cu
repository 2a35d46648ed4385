// C ABI of the library: argument validation, workspace layout, kernel selection and the
// stage driver  (T-1) x [right-factor, left-factor], right-factor-with-V, output
// (reference: ma/ma_torch.py:100-105).
#include <math.h>
#include <stdio.h>
#include <string.h>

#include <string>

#include "ma_common.cuh"
#include "ma_tc_plan.cuh"

namespace {

thread_local std::string g_last_error;

int fail(int code, const std::string& msg) {
  g_last_error = msg;
  return code;
}

size_t dtype_size(int dt) {
  switch (dt) {
    case MA_B200_F32: return 4;
    case MA_B200_BF16: return 2;
    case MA_B200_F16: return 2;
    default: return 0;
  }
}

size_t align_up(size_t x, size_t a) { return (x + a - 1) / a * a; }

int validate(const ma_b200_problem* p, bool need_pointers) {
  if (p == nullptr) return fail(MA_B200_INVALID_ARGUMENT, "problem is NULL");
  if (p->abi_version != MA_B200_ABI_VERSION)
    return fail(MA_B200_INVALID_ARGUMENT, "abi_version mismatch: got " + std::to_string(p->abi_version));
  if (p->E <= 0 || p->H <= 0 || p->N <= 0 || p->D <= 0 || p->Dv <= 0)
    return fail(MA_B200_INVALID_ARGUMENT, "E, H, N, D, Dv must be positive");
  if (p->block_size <= 0) return fail(MA_B200_INVALID_ARGUMENT, "block_size must be positive");
  if (p->num_steps <= 0) return fail(MA_B200_INVALID_ARGUMENT, "num_steps must be positive");
  if (dtype_size(p->qk_dtype) == 0 || dtype_size(p->v_dtype) == 0)
    return fail(MA_B200_INVALID_ARGUMENT, "unknown dtype");
  if (!(p->qk_dtype == p->v_dtype || p->v_dtype == MA_B200_F32))
    return fail(MA_B200_UNSUPPORTED, "v_dtype must equal qk_dtype or be f32");
  if (p->kernel < MA_B200_KERNEL_AUTO || p->kernel > MA_B200_KERNEL_TILE || p->kernel == 4)
    return fail(MA_B200_INVALID_ARGUMENT, "unknown kernel family");
  if ((long long)p->E * p->H > 0x7fffffffLL / 2) return fail(MA_B200_INVALID_ARGUMENT, "E*H too large");
  if (need_pointers) {
    if (!p->q.ptr || !p->k.ptr || !p->v.ptr || !p->out.ptr)
      return fail(MA_B200_INVALID_ARGUMENT, "q, k, v and out must be non-NULL");
    const ma_b200_tensor* ts[4] = {&p->q, &p->k, &p->v, &p->out};
    const char* names[4] = {"q", "k", "v", "out"};
    for (int i = 0; i < 4; ++i) {
      if (ts[i]->stride_e < 0 || ts[i]->stride_h < 0 || ts[i]->stride_n < 0)
        return fail(MA_B200_INVALID_ARGUMENT, std::string(names[i]) + ": negative stride");
      const size_t es = dtype_size(i < 2 ? p->qk_dtype : p->v_dtype);
      if (reinterpret_cast<uintptr_t>(ts[i]->ptr) % es != 0)
        return fail(MA_B200_INVALID_ARGUMENT, std::string(names[i]) + ": pointer not aligned to its element size");
    }
    const int W = p->Dv;
    if (p->out.stride_n < W && p->N > 1) return fail(MA_B200_INVALID_ARGUMENT, "out rows overlap (stride_n < Dv)");
    if (p->mask != nullptr && p->mask_stride_e < 0) return fail(MA_B200_INVALID_ARGUMENT, "mask: negative stride");
  }
  return MA_B200_OK;
}

ma::Geometry make_geometry(const ma_b200_problem* p, int mask_type = MA_B200_MASK_U8) {
  ma::Geometry g;
  memset(&g, 0, sizeof(g));
  g.E = p->E; g.H = p->H; g.N = p->N; g.D = p->D; g.Dv = p->Dv;
  g.B = p->block_size;
  g.M = (p->N + p->block_size - 1) / p->block_size;
  g.pad_off = p->pre_pad ? g.M * g.B - g.N : 0;
  g.T = p->num_steps;
  g.sm_scale = (float)(1.0 / sqrt((double)p->D));
  auto view = [](const ma_b200_tensor& t) {
    ma::View4 v;
    v.ptr = t.ptr; v.se = t.stride_e; v.sh = t.stride_h; v.sn = t.stride_n;
    return v;
  };
  g.q = view(p->q); g.k = view(p->k); g.v = view(p->v); g.out = view(p->out);
  g.mask = p->mask;
  g.mask_type = mask_type;
  g.mask_se = p->mask_stride_e;
  return g;
}

// Whether the warp-level kernels are expected to take a problem faster than the tcgen05 tile kernels: those work on tiles of
// 128 x 64 or 128 x 128 whatever the blocks fill of them, so that blocks just above 32, a long side beside a short one,
// narrow heads and few heads are better off with 16-row warps and two launches.  Microseconds of one iteration, fitted to 1008 pairs
// of calls (36 shapes of 8 to 128, widths 32 and 64, 4 to 256 heads, one and two iterations, replayed from a graph): a tile takes 8.2 ns of
// the GPU's time beside 10.9 us; a padded element of a warp-level tile, keys and rows to the next multiple of 16, takes 3.13 ps in the
// right-factor stage and 1.62 in the left-factor or output stage, 0.55 of that in heads of up to 32, beside 3.8 us.  What the rule takes
// is 0.1 % more than the faster one of each pair as a geometric mean, and 11 pairs lose more than 5 %: us, warp-level / tile, 96 heads of
// 96 x 33 x 32, two iterations, 171 / 150 the most that is lost by the warp-level kernels, 16 of 49 x 49 x 64 34.9 / 39.9 by the tiles.
// (Before, keys counted as 16, 32, 64 or 128, as the kernels once padded them, and one cost for both stages: 1.9 % and 123 pairs; 4 heads
// of 72 x 72 x 64, one iteration, 12.4 / 18.5 and 128 of 128 x 16 x 64 122 / 89 were on the wrong side.)
bool warp_beats_tiles(const ma::Geometry& g, double heads) {
  if (g.B > 128 || g.M > 128) return false;  // (the warp-level kernels then walk a row twice: never the faster ones)
  auto padded = [](int x) { return (double)((x + 15) & ~15); };
  const double right = heads * g.M * padded(g.B) * padded(g.B), left = heads * g.B * padded(g.M) * padded(g.M);
  const double tiles = heads * ((g.B <= 64 ? (g.M + 1) / 2 : g.M) + (g.M <= 64 ? (g.B + 1) / 2 : g.B));
  const double warp_us = 3.8 + (3.13e-6 * right + 1.62e-6 * left) * (g.D <= 32 ? 0.55 : 1.0);
  return warp_us < tiles * 8.2e-3 + 10.9;
}

// AUTO goes by the shape of a head and by how many heads there are.  `heads`: the (batch, head) pairs of the whole call, of
// which `p` may be a part: families differ in the order of their sums, so the parts of one call take the same one.
int resolve_kernel(const ma_b200_problem* p, const ma::Geometry& g, long long heads, int* kernel) {
  const char* why = "";
  const bool tc_ok = ma::tc_supported(g, p->qk_dtype, p->v_dtype, &why);
  const bool wants_tc = p->kernel == MA_B200_KERNEL_TCGEN05 || p->kernel == MA_B200_KERNEL_TCGEN05_STAGED;
  if (wants_tc && !tc_ok)
    return fail(MA_B200_UNSUPPORTED, std::string("tcgen05 path cannot run this problem: ") + why);
  const char* why_w = "";
  const bool warp_ok = ma::warp_supported(g, p->qk_dtype, p->v_dtype, &why_w);
  if (p->kernel == MA_B200_KERNEL_WARP_MMA && !warp_ok)
    return fail(MA_B200_UNSUPPORTED, std::string("warp-level tensor-core path cannot run this problem: ") + why_w);
  const char* why_h = "";
  const bool head_ok = ma::head_fused_supported(g, p->qk_dtype, p->v_dtype, &why_h);
  if (p->kernel == MA_B200_KERNEL_HEAD_FUSED && !head_ok)
    return fail(MA_B200_UNSUPPORTED, std::string("one-CTA-per-head kernel cannot run this problem: ") + why_h);
  const char* why_r = "";
  const bool resident_ok = ma::head_resident_supported(g, p->qk_dtype, p->v_dtype, &why_r);
  if (p->kernel == MA_B200_KERNEL_HEAD_RESIDENT && !resident_ok)
    return fail(MA_B200_UNSUPPORTED, std::string("head-resident kernel cannot run this problem: ") + why_r);
  const char* why_t = "";
  const bool tile_ok = ma::tile_supported(g, p->qk_dtype, p->v_dtype, &why_t);
  if (p->kernel == MA_B200_KERNEL_TILE && !tile_ok)
    return fail(MA_B200_UNSUPPORTED, std::string("tcgen05 tile kernels cannot run this problem: ") + why_t);
  const char* why_x = "";
  const bool tf32_ok = ma::tf32x3_supported(g, p->qk_dtype, p->v_dtype, &why_x);
  if (p->kernel == MA_B200_KERNEL_TF32X3 && !tf32_ok)
    return fail(MA_B200_UNSUPPORTED, std::string("fp32 tensor-core path cannot run this problem: ") + why_x);
  // Heads narrower than 24 leave most of a 16-wide contraction step of the fp32 tensor path padded or give it one
  // step per tile; the thread-per-logit kernels are as fast there.
  const bool tf32_pays = tf32_ok && g.D >= 24;
  // The fused kernel takes one tile at a time through an SM, quickly; the tile kernels take four, each more slowly, and do
  // 1.2 to 1.4 times as many in a time.  So the fused kernel is the faster one while a stage is few rounds of one tile per
  // SM.  Measured (us, fused / tile kernels, replayed from a graph, both with their programmatic launches) over 0.4 to 8.7 tiles per SM
  // and stage, blocks of 64 and 128: with two iterations 38.9 / 41.6 and 43.4 / 48.1 at 3.5, 47.3 / 48.8 and 55.5 / 57.0 at 5.2, 48.5 / 49.6
  // (blocks of 64) at 5.4, 50.4 / 49.8 at 5.6, 54.1 / 50.8 and 65.2 / 61.6 at 6.1, 74 / 52 and 72 / 65 at 6.9; with three 66.5 / 67.3 and 79 / 87 at
  // 5.2, 68.5 / 67.7 at 5.4, 75.8 / 69.0 and 91.7 / 91.2 at 6.1: the line is at 5.5.  With one, whose two stages leave the tile kernels' list
  // fewer waits, 14.1 / 15.9 and 15.5 / 17.6 at 0.9, 17.2 / 17.7 and 18.8 / 19.9 at 1.7, 19.6 / 18.9 at 2.2, 21.0 / 20.0 and 23.2 / 22.4 at 2.6: the
  // line is at 2.
  const bool few_tiles = tc_ok && heads * p->N / 64 <= (long long)ma::sm_count() * (p->num_steps == 1 ? 4 : 11);
  // Head widths other than 32, 64, 72 and 80 have one tile size for both kinds of stage in the head-resident kernel: with one side of
  // up to 16 beside a longer one the warp-level kernels pad less, and win once the heads no longer fit the SMs in one round.
  // Head-resident over warp-level, 112 calls each (8 x 20 to 32 x 5, 149 to 1000 heads, one and two iterations, replayed from a graph): width
  // 40 1.24 as a geometric mean (10 x 30, one iteration, 149 heads 1.64; 16 x 17, two, 592 heads 0.88), 48 1.25, 56 1.26, 24 1.12.  Width 80, with
  // tiles of its own, 0.81 (1.05 the most, 300 heads of 16 x 17 with one) would be faster on the other side of this line; it stays because
  // test_parts_gpu.py needs a part of 200 heads of 10 x 30 x 80 to be of another family than the whole.
  const bool lopsided = (g.B <= 16) != (g.M <= 16) && g.D != 32 && g.D != 64 && g.D != 72 && heads > ma::sm_count();
  if (p->kernel == MA_B200_KERNEL_AUTO)
    *kernel = few_tiles ? MA_B200_KERNEL_TCGEN05
              : resident_ok && !lopsided ? MA_B200_KERNEL_HEAD_RESIDENT
              : tile_ok && !(warp_ok && warp_beats_tiles(g, (double)heads)) ? MA_B200_KERNEL_TILE
              : warp_ok          ? MA_B200_KERNEL_WARP_MMA
              : tf32_pays        ? MA_B200_KERNEL_TF32X3
                                 : MA_B200_KERNEL_GENERIC;
  else *kernel = p->kernel;
  if (*kernel == MA_B200_KERNEL_GENERIC) {
    const size_t need = ma::generic_stage_smem_bytes(g, g.B > g.M ? ma::kStageRight : ma::kStageLeft);
    if (need > 200 * 1024)
      return fail(MA_B200_UNSUPPORTED, "generic path: block size or block count too large for shared memory");
    if (g.M > 65535 || g.B > 65535)  // gridDim.y; E*H sits on gridDim.x (limit 2^31 - 1, checked in validate)
      return fail(MA_B200_UNSUPPORTED, "generic path: grid too large");
  }
  return MA_B200_OK;
}

int layout_of(const ma_b200_problem* p, ma_b200_workspace_layout* L) {
  int rc = validate(p, false);
  if (rc != MA_B200_OK) return rc;
  ma::Geometry g = make_geometry(p);
  int kernel = 0;
  rc = resolve_kernel(p, g, (long long)p->E * p->H, &kernel);
  if (rc != MA_B200_OK) return rc;
  const size_t EH = (size_t)p->E * p->H, MB = (size_t)g.M * g.B;
  const size_t qs = dtype_size(p->qk_dtype), vs = dtype_size(p->v_dtype);
  size_t off = 0;
  L->status = off; off = align_up(off + 256, 256);
  L->counters = off; off = align_up(off + EH * 2 * (size_t)p->num_steps * sizeof(int), 256);
  L->ar = off;     off = align_up(off + (p->num_steps > 1 ? EH * MB * p->D * qs : 0), 256);
  L->cr = off;     off = align_up(off + (p->num_steps > 1 ? EH * MB * sizeof(float) : 0), 256);
  L->al = off;     off = align_up(off + EH * MB * p->D * qs, 256);
  L->cl = off;     off = align_up(off + EH * MB * sizeof(float), 256);
  L->y = off;      off = align_up(off + EH * MB * p->Dv * vs, 256);
  L->total = off;
  L->M = g.M;
  L->kernel = kernel;
  return MA_B200_OK;
}

int check_mask_type(const ma_b200_problem* p, int mask_type) {
  static const int bytes[] = {1, 2, 4, 8, 2, 4, 8};
  if (mask_type < MA_B200_MASK_U8 || mask_type > MA_B200_MASK_F64) return fail(MA_B200_INVALID_ARGUMENT, "unknown mask type");
  if (p != nullptr && reinterpret_cast<uintptr_t>(p->mask) % bytes[mask_type] != 0)
    return fail(MA_B200_INVALID_ARGUMENT, "mask: pointer not aligned to its element size");
  return MA_B200_OK;
}

int run_forward(const ma_b200_problem* p, int mask_type, void* workspace, size_t workspace_bytes, void* stream_v, float* stage_ms,
                int n_stage_ms) {
  int rc = validate(p, true);
  if (rc == MA_B200_OK) rc = check_mask_type(p, mask_type);
  if (rc != MA_B200_OK) return rc;
  ma_b200_workspace_layout L;
  rc = layout_of(p, &L);
  if (rc != MA_B200_OK) return rc;
  if (workspace == nullptr) return fail(MA_B200_INVALID_ARGUMENT, "workspace is NULL");
  if (reinterpret_cast<uintptr_t>(workspace) % 256 != 0)
    return fail(MA_B200_INVALID_ARGUMENT, "workspace must be 256-byte aligned");
  if (workspace_bytes < L.total)
    return fail(MA_B200_WORKSPACE_TOO_SMALL, "workspace has " + std::to_string(workspace_bytes) + " bytes, need " +
                                                 std::to_string(L.total));
  cudaStream_t stream = reinterpret_cast<cudaStream_t>(stream_v);
  ma::Geometry g = make_geometry(p, mask_type);
  char* ws = reinterpret_cast<char*>(workspace);
  g.status = reinterpret_cast<int*>(ws + L.status);
  g.ar = ws + L.ar;
  g.cr = reinterpret_cast<float*>(ws + L.cr);
  g.al = ws + L.al;
  g.cl = reinterpret_cast<float*>(ws + L.cl);
  g.y = ws + L.y;

  auto cuda_fail = [&](cudaError_t e, const char* what) {
    return fail(MA_B200_CUDA_ERROR, std::string(what) + ": " + cudaGetErrorString(e));
  };
  // Status word and stage-completion counters start at zero.  The stage kernels that wait for nothing clear the
  // status word themselves (a memset in front of them is 1.5 us on the stream, as much as a small kernel), and the
  // single-launch tile kernels have a kernel before them that clears both.
  cudaError_t ce = cudaSuccess;
  const bool flow = L.kernel == MA_B200_KERNEL_TILE && ma::flow_supported(g);
  if (L.kernel != MA_B200_KERNEL_WARP_MMA && L.kernel != MA_B200_KERNEL_TF32X3 && L.kernel != MA_B200_KERNEL_HEAD_RESIDENT &&
      L.kernel != MA_B200_KERNEL_HEAD_FUSED && L.kernel != MA_B200_KERNEL_TILE) {
    ce = ma::launch_clear(ws + L.status, L.ar - L.status, stream);
    if (ce != cudaSuccess) return cuda_fail(ce, "clearing status and counters");
  }
  int* counters = reinterpret_cast<int*>(ws + L.counters);

  ma::TcPlan plan_store;
  const ma::TcPlan* plan = nullptr;
  if (L.kernel == MA_B200_KERNEL_TCGEN05 || L.kernel == MA_B200_KERNEL_TCGEN05_STAGED) {
    const char* err = "";
    rc = ma::tc_plan_get(g, p->qk_dtype, &plan_store, &err);
    if (rc != MA_B200_OK) return fail(rc, std::string("tcgen05 plan: ") + err);
    plan = &plan_store;
  }

  int* host_status = nullptr;
  if (L.kernel == MA_B200_KERNEL_TILE) {
    int dev = 0;
    if ((ce = cudaGetDevice(&dev)) != cudaSuccess) return cuda_fail(ce, "cudaGetDevice");
    host_status = ma::host_status_word(dev);
  }

  const int n_stages = 2 * p->num_steps;
  cudaEvent_t* ev = nullptr;
  if (stage_ms != nullptr) {
    ev = new cudaEvent_t[n_stages + 1];
    for (int i = 0; i <= n_stages; ++i) cudaEventCreate(&ev[i]);
    cudaEventRecord(ev[0], stream);
  }
  int stage_idx = 0;
  auto launch = [&](ma::StageKind kind, bool first) -> cudaError_t {
    cudaError_t e;
    if (L.kernel == MA_B200_KERNEL_TCGEN05_STAGED)
      e = ma::launch_fused(plan, g, counters, stage_idx, stage_idx + 1, 0, 0, stream);
    else if (L.kernel == MA_B200_KERNEL_TILE)
      e = ma::launch_tile_stage(g, p->qk_dtype, kind, first, host_status, false, stream);
    else if (L.kernel == MA_B200_KERNEL_WARP_MMA || L.kernel == MA_B200_KERNEL_TF32X3)
      e = ma::launch_warp_stage(g, p->qk_dtype, kind, first, stream);
    else e = ma::launch_generic_stage(g, p->qk_dtype, p->v_dtype, kind, first, stream);
    ++stage_idx;
    if (ev != nullptr) cudaEventRecord(ev[stage_idx], stream);
    return e;
  };

  bool single = false;
  auto one_launch = [&] {  // all stages in one launch: their time is the first entry, the others are 0
    single = true;
    if (ev != nullptr) cudaEventRecord(ev[1], stream);
  };

  rc = MA_B200_OK;
  bool first = true;
  if (L.kernel == MA_B200_KERNEL_HEAD_FUSED || L.kernel == MA_B200_KERNEL_HEAD_RESIDENT) {
    ce = ma::launch_head_resident(g, p->qk_dtype, stream);
    if (ce != cudaSuccess) rc = cuda_fail(ce, "head-resident kernel");
    one_launch();
  } else if (L.kernel == MA_B200_KERNEL_TF32X3 && ma::head_f32_pays(g)) {
    ce = ma::launch_head_f32(g, stream);
    if (ce != cudaSuccess) rc = cuda_fail(ce, "fp32 tensor path in one launch");
    one_launch();
  } else if (flow) {
    ce = ma::launch_flow(g, p->qk_dtype, counters, host_status, false, stream);
    if (ce != cudaSuccess) rc = cuda_fail(ce, "tile kernels in one launch");
    one_launch();
  } else if (L.kernel == MA_B200_KERNEL_TCGEN05) {
    // every stage in one persistent launch
    ce = ma::launch_fused(plan, g, counters, 0, n_stages, 1, 0, stream);
    if (ce != cudaSuccess) rc = cuda_fail(ce, "fused kernel");
    one_launch();
  } else {
  for (int t = 0; t + 1 < p->num_steps && rc == MA_B200_OK; ++t) {
    if ((ce = launch(ma::kStageRight, first)) != cudaSuccess) { rc = cuda_fail(ce, "right-factor stage"); break; }
    first = false;
    if ((ce = launch(ma::kStageLeft, false)) != cudaSuccess) { rc = cuda_fail(ce, "left-factor stage"); break; }
  }
  if (rc == MA_B200_OK && (ce = launch(ma::kStageRightWithV, first)) != cudaSuccess)
    rc = cuda_fail(ce, "right-factor stage with V");
  if (rc == MA_B200_OK && (ce = launch(ma::kStageOutput, false)) != cudaSuccess) rc = cuda_fail(ce, "output stage");
  }

  if (ev != nullptr) {
    if (rc == MA_B200_OK) {
      ce = cudaStreamSynchronize(stream);
      if (ce != cudaSuccess) rc = cuda_fail(ce, "cudaStreamSynchronize");
      for (int i = 0; i < n_stages && i < n_stage_ms && rc == MA_B200_OK; ++i) {
        stage_ms[i] = 0.f;
        if (!single || i == 0) cudaEventElapsedTime(&stage_ms[i], ev[i], ev[i + 1]);
      }
    }
    for (int i = 0; i <= n_stages; ++i) cudaEventDestroy(ev[i]);
    delete[] ev;
  }
  return rc;
}

}  // namespace

extern "C" {

size_t ma_b200_workspace_bytes(const ma_b200_problem* p) {
  ma_b200_workspace_layout L;
  if (layout_of(p, &L) != MA_B200_OK) return 0;
  return L.total;
}

int ma_b200_workspace_layout_of(const ma_b200_problem* p, ma_b200_workspace_layout* layout) {
  if (layout == nullptr) return fail(MA_B200_INVALID_ARGUMENT, "layout is NULL");
  return layout_of(p, layout);
}

int ma_b200_kernel_of_part(const ma_b200_problem* part, int64_t heads) {
  if (validate(part, false) != MA_B200_OK) return 0;
  if (heads < (int64_t)part->E * part->H || heads > 0x7fffffffLL) {
    fail(MA_B200_INVALID_ARGUMENT, "heads must count at least the part's own E*H, and fit 31 bits");
    return 0;
  }
  int kernel = 0;
  return resolve_kernel(part, make_geometry(part), heads, &kernel) == MA_B200_OK ? kernel : 0;
}

int ma_b200_forward(const ma_b200_problem* p, void* workspace, size_t workspace_bytes, void* stream) {
  return run_forward(p, MA_B200_MASK_U8, workspace, workspace_bytes, stream, nullptr, 0);
}

int ma_b200_forward_typed_mask(const ma_b200_problem* p, int mask_type, void* workspace, size_t workspace_bytes, void* stream) {
  return run_forward(p, mask_type, workspace, workspace_bytes, stream, nullptr, 0);
}

int ma_b200_forward_timed(const ma_b200_problem* p, void* workspace, size_t workspace_bytes, void* stream,
                          float* stage_ms, int32_t n_stage_ms) {
  if (stage_ms == nullptr || n_stage_ms <= 0) return fail(MA_B200_INVALID_ARGUMENT, "stage_ms is NULL or empty");
  return run_forward(p, MA_B200_MASK_U8, workspace, workspace_bytes, stream, stage_ms, n_stage_ms);
}

size_t ma_b200_backward_workspace_bytes(const ma_b200_problem* p) {
  if (validate(p, false) != MA_B200_OK) return 0;
  const ma::Geometry g = make_geometry(p);
  const char* why = "";
  if (!ma::backward_supported(g, p->qk_dtype, p->v_dtype, &why)) {
    fail(MA_B200_UNSUPPORTED, std::string("backward kernels cannot run this problem: ") + why);
    return 0;
  }
  return ma::backward_layout(g, p->qk_dtype).total;
}

int ma_b200_backward(const ma_b200_problem* p, const ma_b200_gradients* gr, void* workspace, size_t workspace_bytes,
                     void* stream) {
  return ma_b200_backward_typed_mask(p, MA_B200_MASK_U8, gr, workspace, workspace_bytes, stream);
}

int ma_b200_backward_typed_mask(const ma_b200_problem* p, int mask_type, const ma_b200_gradients* gr, void* workspace,
                                size_t workspace_bytes, void* stream) {
  if (p == nullptr || gr == nullptr) return fail(MA_B200_INVALID_ARGUMENT, "problem or gradients is NULL");
  ma_b200_problem q = *p;
  q.out = gr->grad_out;  // takes the output's place in the checks of pointers and alignment
  if (q.out.stride_n < q.Dv) q.out.stride_n = q.Dv;  // (read only: rows may repeat)
  int rc = validate(&q, true);
  if (rc == MA_B200_OK) rc = check_mask_type(&q, mask_type);
  if (rc != MA_B200_OK) return rc;
  ma::Geometry g = make_geometry(&q, mask_type);
  g.out.sn = gr->grad_out.stride_n;
  const char* why = "";
  if (!ma::backward_supported(g, p->qk_dtype, p->v_dtype, &why))
    return fail(MA_B200_UNSUPPORTED, std::string("backward kernels cannot run this problem: ") + why);
  const size_t need = ma::backward_layout(g, p->qk_dtype).total;
  if (workspace == nullptr || reinterpret_cast<uintptr_t>(workspace) % 256 != 0)
    return fail(MA_B200_INVALID_ARGUMENT, "workspace is NULL or not 256-byte aligned");
  if (workspace_bytes < need)
    return fail(MA_B200_WORKSPACE_TOO_SMALL, "workspace has " + std::to_string(workspace_bytes) + " bytes, need " + std::to_string(need));
  const ma_b200_tensor* outs[3] = {&gr->dq, &gr->dk, &gr->dv};
  const size_t es = dtype_size(p->qk_dtype), per = 16 / es;
  ma::View4 v[3];
  for (int i = 0; i < 3; ++i) {
    const ma_b200_tensor& t = *outs[i];
    v[i].ptr = t.ptr; v[i].se = t.stride_e; v[i].sh = t.stride_h; v[i].sn = t.stride_n;
    if (t.ptr == nullptr) continue;
    if (reinterpret_cast<uintptr_t>(t.ptr) % 16 != 0 || t.stride_n % per != 0 || t.stride_h % per != 0 || t.stride_e % per != 0 ||
        t.stride_e < 0 || t.stride_h < 0 || (t.stride_n < p->D && p->N > 1))
      return fail(MA_B200_INVALID_ARGUMENT, "dq, dk, dv: rows must not overlap and must start on 16-byte boundaries");
  }
  const cudaError_t ce = ma::launch_backward(g, p->qk_dtype, g.out, v[0], v[1], v[2], workspace, reinterpret_cast<cudaStream_t>(stream));
  if (ce != cudaSuccess) return fail(MA_B200_CUDA_ERROR, std::string("backward pass: ") + cudaGetErrorString(ce));
  return MA_B200_OK;
}

int ma_b200_device_status(void* workspace, void* stream) {
  if (workspace == nullptr) return fail(MA_B200_INVALID_ARGUMENT, "workspace is NULL");
  int flag = 0;
  cudaError_t ce = cudaMemcpyAsync(&flag, workspace, sizeof(int), cudaMemcpyDeviceToHost,
                                   reinterpret_cast<cudaStream_t>(stream));
  if (ce == cudaSuccess) ce = cudaStreamSynchronize(reinterpret_cast<cudaStream_t>(stream));
  if (ce != cudaSuccess) return fail(MA_B200_CUDA_ERROR, std::string("device_status: ") + cudaGetErrorString(ce));
  if (flag != 0)
    return fail(MA_B200_DEVICE_WAIT_EXPIRED, "device flag = " + std::to_string(flag) + " (a bounded wait expired)");
  return MA_B200_OK;
}

int ma_b200_poll_device_status(int device) {
  const int code = ma::fused_poll_status(device);
  if (code != 0)
    return fail(MA_B200_DEVICE_WAIT_EXPIRED, "device " + std::to_string(device) + ": wait " + std::to_string(code) +
                                                 " of a kernel gave up; the output of that call is undefined");
  return MA_B200_OK;
}

void ma_b200_selftest_generic_general_form(int on) { ma::generic_set_general_form_only(on); }

int ma_b200_selftest_wait_expiry(const ma_b200_problem* p, void* workspace, size_t workspace_bytes, void* stream_v) {
  int rc = validate(p, true);
  if (rc != MA_B200_OK) return rc;
  ma_b200_problem q = *p;
  if (q.kernel != MA_B200_KERNEL_TILE) q.kernel = MA_B200_KERNEL_TCGEN05;
  ma_b200_workspace_layout L;
  rc = layout_of(&q, &L);
  if (rc != MA_B200_OK) return rc;
  if (workspace == nullptr || reinterpret_cast<uintptr_t>(workspace) % 256 != 0 || workspace_bytes < L.total)
    return fail(MA_B200_INVALID_ARGUMENT, "workspace is NULL, misaligned or too small");
  cudaStream_t stream = reinterpret_cast<cudaStream_t>(stream_v);
  ma::Geometry g = make_geometry(&q);
  char* ws = reinterpret_cast<char*>(workspace);
  g.status = reinterpret_cast<int*>(ws + L.status);
  g.ar = ws + L.ar; g.cr = reinterpret_cast<float*>(ws + L.cr);
  g.al = ws + L.al; g.cl = reinterpret_cast<float*>(ws + L.cl);
  g.y = ws + L.y;
  cudaError_t ce = cudaMemsetAsync(ws + L.status, 0, L.ar - L.status, stream);
  if (ce != cudaSuccess) return fail(MA_B200_CUDA_ERROR, cudaGetErrorString(ce));
  if (q.kernel == MA_B200_KERNEL_TILE) {
    int dev = 0;
    if ((ce = cudaGetDevice(&dev)) != cudaSuccess) return fail(MA_B200_CUDA_ERROR, cudaGetErrorString(ce));
    int* const host_status = ma::host_status_word(dev);
    // The single launch: its first stage is left out, and every CTA waits for that.  The kernels of a launch each: the
    // first stage, with an operand that no CTA asks for.
    ce = ma::flow_supported(g) ? ma::launch_flow(g, q.qk_dtype, reinterpret_cast<int*>(ws + L.counters), host_status, true, stream)
                               : ma::launch_tile_stage(g, q.qk_dtype, q.num_steps > 1 ? ma::kStageRight : ma::kStageRightWithV, true,
                                                       host_status, true, stream);
    if (ce != cudaSuccess) return fail(MA_B200_CUDA_ERROR, std::string("tile kernels: ") + cudaGetErrorString(ce));
    return MA_B200_OK;
  }
  ma::TcPlan plan;
  const char* err = "";
  rc = ma::tc_plan_get(g, q.qk_dtype, &plan, &err);
  if (rc != MA_B200_OK) return fail(rc, std::string("tcgen05 plan: ") + err);
  // Stage 1 alone, waiting on completion counters of stage 0 that nothing will ever raise: every
  // producer runs out of patience after a few hundred microseconds and the CTAs return.
  ce = ma::launch_fused(&plan, g, reinterpret_cast<int*>(ws + L.counters), 1, 2, 1, 4096, stream);
  if (ce != cudaSuccess) return fail(MA_B200_CUDA_ERROR, std::string("fused kernel: ") + cudaGetErrorString(ce));
  return MA_B200_OK;
}

const char* ma_b200_status_string(int status) {
  switch (status) {
    case MA_B200_OK: return "ok";
    case MA_B200_INVALID_ARGUMENT: return "invalid argument";
    case MA_B200_UNSUPPORTED: return "unsupported configuration";
    case MA_B200_CUDA_ERROR: return "CUDA error";
    case MA_B200_DEVICE_WAIT_EXPIRED: return "device-side bounded wait expired";
    case MA_B200_WORKSPACE_TOO_SMALL: return "workspace too small";
    default: return "unknown status";
  }
}

const char* ma_b200_last_error(void) { return g_last_error.c_str(); }

int32_t ma_b200_abi_version(void) { return MA_B200_ABI_VERSION; }

}  // extern "C"
