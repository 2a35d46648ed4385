// ma_b200_forward_host: the forward pass for q, k, v and the result in HOST memory.
//
// For the long-sequence workloads the PCIe copies around a call cost far more than the kernels
// (134 MB against 0.14 ms of compute for N = 16384 and 16 heads).  Every (batch, head) pair is
// independent in every stage, so the call is cut into chunks of a few heads and pipelined over
// three streams owned by the library -
//     copy-in : H2D q, k, v of chunk i+1
//     compute : ma_b200_forward on chunk i (device staging buffers, some heads of one batch element or several whole
//               elements; the kernel family of the whole call, so that the result has the bits of one call on device tensors)
//     copy-out: D2H result of chunk i-1
// - with three staging slots in caller-provided device memory and events between the streams.
// PCIe is full duplex, so the steady state is bound by the larger copy direction alone; the chunks of
// the last batch element shrink towards the end so that little is left exposed after the last copy-in.
// A chunk costs the host 25 us (three copies, a launch, a copy and the events between them), and the copy engines some
// more, so small chunks are bound by that: heads of a few kilobytes are grouped across batch elements (the caller says how many).
// The whole pipeline is queued from one host thread without waiting for the GPU; on return the
// caller's stream has been made to wait for the last copy.
#include <mutex>
#include <string>

#include "ma_common.cuh"

namespace {

constexpr int kSlots = 3;
constexpr int kMaxDevices = 64;
constexpr size_t kAlign = 256;

struct Pipes {
  bool ready = false;
  cudaStream_t in = nullptr, comp = nullptr, out = nullptr;
  cudaEvent_t start = nullptr, loaded[kSlots] = {}, computed[kSlots] = {}, stored[kSlots] = {}, done_comp = nullptr,
              done_out = nullptr;
  // what the previous call on this device laid out in the scratch (a streamed call may only overlap a
  // previous call that used the same slots)
  const void* last_scratch = nullptr;
  size_t last_qk_bytes = 0, last_slot_bytes = 0, last_total = 0;
};
Pipes g_pipes[kMaxDevices];
std::mutex g_pipes_mutex;
thread_local std::string g_host_error;

size_t round_up(size_t x) { return (x + kAlign - 1) / kAlign * kAlign; }
size_t elem_size(int dtype) { return dtype == MA_B200_F32 ? 4 : 2; }

void clamp_chunk(int E, int H, int heads, int elements, int* hc, int* ec) {
  *hc = heads < H ? heads : H;
  *ec = *hc < H ? 1 : elements < E ? elements : E;
}

struct HostLayout {
  int hc;                                // heads per chunk (clamped to H)
  int ec;                                // batch elements per chunk (more than one only with all heads)
  size_t qk_bytes, v_bytes;              // one staging tensor of a slot
  size_t slot_bytes, mask_off, mask_bytes, ws_off, ws_bytes, total;
};

// 0 on success; fills the layout of the device scratch for this problem.
int host_layout(const ma_b200_problem* p, int heads_per_chunk, int elements_per_chunk, HostLayout* L, std::string* err) {
  if (p == nullptr) { *err = "problem is null"; return MA_B200_INVALID_ARGUMENT; }
  if (heads_per_chunk < 1) { *err = "heads_per_chunk must be at least 1"; return MA_B200_INVALID_ARGUMENT; }
  if (elements_per_chunk < 1) { *err = "elements_per_chunk must be at least 1"; return MA_B200_INVALID_ARGUMENT; }
  if (p->E < 1 || p->H < 1 || p->N < 1 || p->D < 1 || p->Dv < 1) { *err = "E, H, N, D, Dv must be positive"; return MA_B200_INVALID_ARGUMENT; }
  clamp_chunk(p->E, p->H, heads_per_chunk, elements_per_chunk, &L->hc, &L->ec);
  L->qk_bytes = round_up((size_t)L->ec * L->hc * p->N * p->D * elem_size(p->qk_dtype));
  L->v_bytes = round_up((size_t)L->ec * L->hc * p->N * p->Dv * elem_size(p->v_dtype));
  L->slot_bytes = 2 * L->qk_bytes + 2 * L->v_bytes;  // q, k, v, result
  L->mask_off = kSlots * L->slot_bytes;
  L->mask_bytes = p->mask != nullptr ? round_up((size_t)p->E * p->N) : 0;
  L->ws_off = L->mask_off + L->mask_bytes;
  // workspace of the largest chunk problem (pointers are not looked at by the size query)
  ma_b200_problem sub = *p;
  sub.E = L->ec;
  sub.H = L->hc;
  sub.q.ptr = sub.k.ptr = sub.v.ptr = sub.out.ptr = nullptr;
  sub.q.stride_e = sub.k.stride_e = (int64_t)L->hc * p->N * p->D;
  sub.q.stride_h = sub.k.stride_h = (int64_t)p->N * p->D;
  sub.q.stride_n = sub.k.stride_n = p->D;
  sub.v.stride_e = sub.out.stride_e = (int64_t)L->hc * p->N * p->Dv;
  sub.v.stride_h = sub.out.stride_h = (int64_t)p->N * p->Dv;
  sub.v.stride_n = sub.out.stride_n = p->Dv;
  sub.mask = nullptr;
  sub.mask_stride_e = 0;
  L->ws_bytes = ma_b200_workspace_bytes(&sub);
  if (L->ws_bytes == 0) { *err = std::string("chunk problem rejected: ") + ma_b200_last_error(); return MA_B200_INVALID_ARGUMENT; }
  L->ws_bytes = round_up(L->ws_bytes);
  L->total = L->ws_off + L->ws_bytes;
  return MA_B200_OK;
}

int get_pipes(Pipes** out, std::string* err) {
  int dev = -1;
  cudaError_t ce = cudaGetDevice(&dev);
  if (ce != cudaSuccess) { *err = std::string("cudaGetDevice: ") + cudaGetErrorString(ce); return MA_B200_CUDA_ERROR; }
  if (dev < 0 || dev >= kMaxDevices) { *err = "device ordinal out of range"; return MA_B200_UNSUPPORTED; }
  std::lock_guard<std::mutex> lock(g_pipes_mutex);
  Pipes& P = g_pipes[dev];
  if (!P.ready) {
    auto ev = [&](cudaEvent_t* e) { return cudaEventCreateWithFlags(e, cudaEventDisableTiming); };
    bool ok = cudaStreamCreateWithFlags(&P.in, cudaStreamNonBlocking) == cudaSuccess &&
              cudaStreamCreateWithFlags(&P.comp, cudaStreamNonBlocking) == cudaSuccess &&
              cudaStreamCreateWithFlags(&P.out, cudaStreamNonBlocking) == cudaSuccess && ev(&P.start) == cudaSuccess &&
              ev(&P.done_comp) == cudaSuccess && ev(&P.done_out) == cudaSuccess;
    for (int i = 0; i < kSlots && ok; ++i)
      ok = ev(&P.loaded[i]) == cudaSuccess && ev(&P.computed[i]) == cudaSuccess && ev(&P.stored[i]) == cudaSuccess;
    if (!ok) { *err = std::string("creating streams / events: ") + cudaGetErrorString(cudaGetLastError()); return MA_B200_CUDA_ERROR; }
    P.ready = true;
  }
  *out = &P;
  return MA_B200_OK;
}

// Heads [h0, h0 + heads) of the batch elements [e, e + elements); more than one element only with all their heads.
struct Chunk {
  int e, elements, h0, heads;
};
int ceil_div(int a, int b) { return (a + b - 1) / b; }
// The chunk behind `c` (e = E: there is none); c = {0, 0, 0, 0} gives the first.  Chunks of `ec` elements where they have all hc = H
// heads, else of hc heads.  The last batch element tapers off when it is by itself: a chunk is cut to half of what is left, but not below
// `least` heads; what that leaves may be fewer.  Small heads (least > 1): chunks of an earlier element are as even as they can be.
// Measured, us: 6 x 20 heads of 2300 x 64 in chunks of 15 and 5 / 10 and 10 2476 / 2419, 3 x 16 15 and 1 / 8 and 8 1032 / 1002, 2 x 24 of 1500
// x 64 714 / 699.  Not so at the end, where a small last chunk leaves little to copy out: 12 heads of 3000 x 64 in chunks of 6, 5, 1 / 6, 6
// 378 / 396, 16 of 2300 x 64 8, 7, 1 / 8, 8 389 / 402; nor over elements: 52 x 12 of 93 x 64 in fp32 14, 14, 14, 10 / 13, 13, 13, 13 1077 / 1119.
Chunk next_chunk(const Chunk& c, int E, int H, int hc, int ec, int least) {
  const bool more = c.elements == 1 && c.h0 + c.heads < H;  // of the same element
  Chunk n{more ? c.e : c.e + c.elements, 1, more ? c.h0 + c.heads : 0, 0};
  if (n.e >= E) return n;
  const int left = H - n.h0;
  if (ec > 1) n.elements = ec < E - n.e ? ec : E - n.e;
  if (n.elements > 1 || n.e < E - 1) {
    n.heads = least > 1 ? ceil_div(left, ceil_div(left, hc)) : left < hc ? left : hc;
  } else {
    n.heads = left < hc ? left : hc;
    if (n.heads > least && n.heads > left / 2) n.heads = left / 2 > least ? left / 2 : least;
  }
  return n;
}

// Copies `heads` heads of each of `elements` batch elements between a strided host tensor and a dense staging
// buffer (elements, heads, N, W).  One copy where they are dense in host memory, one (pitched) copy per
// head otherwise.
cudaError_t copy_heads(void* dev, const ma_b200_tensor& host, int e, int elements, int h0, int heads, int N, int W, size_t es,
                       bool to_device, cudaStream_t s) {
  if (elements > 1) {
    if (host.stride_n == W && host.stride_h == (int64_t)N * W && host.stride_e == heads * host.stride_h) {
      heads *= elements;  // (whole elements: h0 is 0)
    } else {
      for (int i = 0; i < elements; ++i)
        if (const cudaError_t ce = copy_heads(static_cast<char*>(dev) + (size_t)i * heads * N * W * es, host, e + i, 1, h0, heads, N, W, es, to_device, s);
            ce != cudaSuccess)
          return ce;
      return cudaSuccess;
    }
  }
  char* hbase = static_cast<char*>(const_cast<void*>(host.ptr)) + ((int64_t)e * host.stride_e + (int64_t)h0 * host.stride_h) * (int64_t)es;
  const bool rows_dense = host.stride_n == W;
  const bool heads_dense = rows_dense && (heads == 1 || host.stride_h == (int64_t)N * W);
  const cudaMemcpyKind kind = to_device ? cudaMemcpyHostToDevice : cudaMemcpyDeviceToHost;
  if (heads_dense) {
    const size_t bytes = (size_t)heads * N * W * es;
    return to_device ? cudaMemcpyAsync(dev, hbase, bytes, kind, s) : cudaMemcpyAsync(hbase, dev, bytes, kind, s);
  }
  for (int h = 0; h < heads; ++h) {
    char* hp = hbase + (int64_t)h * host.stride_h * (int64_t)es;
    char* dp = static_cast<char*>(dev) + (size_t)h * N * W * es;
    cudaError_t ce;
    if (rows_dense) {
      ce = to_device ? cudaMemcpyAsync(dp, hp, (size_t)N * W * es, kind, s) : cudaMemcpyAsync(hp, dp, (size_t)N * W * es, kind, s);
    } else {
      ce = to_device ? cudaMemcpy2DAsync(dp, (size_t)W * es, hp, (size_t)host.stride_n * es, (size_t)W * es, N, kind, s)
                     : cudaMemcpy2DAsync(hp, (size_t)host.stride_n * es, dp, (size_t)W * es, (size_t)W * es, N, kind, s);
    }
    if (ce != cudaSuccess) return ce;
  }
  return cudaSuccess;
}

}  // namespace

extern "C" {

MA_B200_API const char* ma_b200_host_last_error(void) { return g_host_error.c_str(); }

MA_B200_API size_t ma_b200_host_scratch_bytes_grouped(const ma_b200_problem* p, int heads_per_chunk, int elements_per_chunk) {
  HostLayout L;
  g_host_error.clear();
  if (host_layout(p, heads_per_chunk, elements_per_chunk, &L, &g_host_error) != MA_B200_OK) return 0;
  return L.total;
}

MA_B200_API size_t ma_b200_host_scratch_bytes(const ma_b200_problem* p, int heads_per_chunk) {
  return ma_b200_host_scratch_bytes_grouped(p, heads_per_chunk, 1);
}

MA_B200_API int ma_b200_host_chunk_plan(int E, int H, int heads_per_chunk, int elements_per_chunk, int least_heads, int32_t* chunks,
                                        int capacity) {
  g_host_error.clear();
  if (E < 0 || H < 0 || heads_per_chunk < 1 || elements_per_chunk < 1 || least_heads < 1) {
    g_host_error = "E and H must not be negative, heads_per_chunk, elements_per_chunk and least_heads at least 1";
    return -1;
  }
  int hc, ec, n = 0;
  clamp_chunk(E, H, heads_per_chunk, elements_per_chunk, &hc, &ec);
  if (E == 0 || H == 0) return 0;
  for (Chunk c = next_chunk({0, 0, 0, 0}, E, H, hc, ec, least_heads); c.e < E; c = next_chunk(c, E, H, hc, ec, least_heads), ++n)
    if (n < capacity) {
      chunks[3 * n] = c.e;
      chunks[3 * n + 1] = c.h0;
      chunks[3 * n + 2] = c.elements * c.heads;
    }
  return n;
}

MA_B200_API int ma_b200_forward_host_grouped(const ma_b200_problem* p, int heads_per_chunk, int elements_per_chunk, int least_heads,
                                             int streamed, void* device_scratch, size_t scratch_bytes, void* stream_v) {
  g_host_error.clear();
  HostLayout L;
  int rc = host_layout(p, heads_per_chunk, elements_per_chunk, &L, &g_host_error);
  if (rc != MA_B200_OK) return rc;
  if (least_heads < 1) {
    g_host_error = "least_heads must be at least 1";
    return MA_B200_INVALID_ARGUMENT;
  }
  if (p->q.ptr == nullptr || p->k.ptr == nullptr || p->v.ptr == nullptr || p->out.ptr == nullptr) {
    g_host_error = "q, k, v and out must be host pointers";
    return MA_B200_INVALID_ARGUMENT;
  }
  if (device_scratch == nullptr || scratch_bytes < L.total) {
    g_host_error = "device scratch too small: need " + std::to_string(L.total) + " bytes";
    return MA_B200_WORKSPACE_TOO_SMALL;
  }
  if (reinterpret_cast<uintptr_t>(device_scratch) % kAlign != 0) {
    g_host_error = "device scratch must be 256-byte aligned";
    return MA_B200_INVALID_ARGUMENT;
  }
  Pipes* P = nullptr;
  rc = get_pipes(&P, &g_host_error);
  if (rc != MA_B200_OK) return rc;
  cudaStream_t caller = reinterpret_cast<cudaStream_t>(stream_v);
  char* base = static_cast<char*>(device_scratch);
  const size_t es_qk = elem_size(p->qk_dtype), es_v = elem_size(p->v_dtype);
  auto fail = [&](cudaError_t ce, const char* what) {
    g_host_error = std::string(what) + ": " + cudaGetErrorString(ce);
    return MA_B200_CUDA_ERROR;
  };
  cudaError_t ce;
#define MA_TRY(call, what) \
  if ((ce = (call)) != cudaSuccess) return fail(ce, what)

  // A streamed call may start copying in while the previous call on this device is still computing and
  // copying out, provided that call used the scratch in the same way (same slots: the per-slot events then
  // order every reuse); anything else is ordered after what the caller has already queued on its stream,
  // which includes the end of the previous call.
  const bool overlap = streamed != 0 && P->last_scratch == device_scratch && P->last_qk_bytes == L.qk_bytes && P->last_slot_bytes == L.slot_bytes &&
                       P->last_total == L.total;
  P->last_scratch = device_scratch;
  P->last_qk_bytes = L.qk_bytes;  // (a slot of the same size with its tensors elsewhere: copying in would run over a result on its way out)
  P->last_slot_bytes = L.slot_bytes;
  P->last_total = L.total;
  if (!overlap) {
    MA_TRY(cudaEventRecord(P->start, caller), "cudaEventRecord(start)");
    MA_TRY(cudaStreamWaitEvent(P->in, P->start, 0), "cudaStreamWaitEvent(in, start)");
    MA_TRY(cudaStreamWaitEvent(P->comp, P->start, 0), "cudaStreamWaitEvent(comp, start)");
    MA_TRY(cudaStreamWaitEvent(P->out, P->start, 0), "cudaStreamWaitEvent(out, start)");
  } else if (p->mask != nullptr) {
    // the mask has one place in the scratch: the previous call's kernels must have read theirs
    MA_TRY(cudaStreamWaitEvent(P->in, P->done_comp, 0), "cudaStreamWaitEvent(in, done_comp)");
  }
  unsigned char* mask_dev = nullptr;
  if (p->mask != nullptr) {
    mask_dev = reinterpret_cast<unsigned char*>(base + L.mask_off);
    const size_t pitch = (size_t)p->mask_stride_e;
    if (pitch == (size_t)p->N || p->E == 1) {
      MA_TRY(cudaMemcpyAsync(mask_dev, p->mask, (size_t)p->E * p->N, cudaMemcpyHostToDevice, P->in), "mask upload");
    } else {
      MA_TRY(cudaMemcpy2DAsync(mask_dev, p->N, p->mask, pitch, p->N, p->E, cudaMemcpyHostToDevice, P->in), "mask upload");
    }
  }

  int i = 0, kernel = 0;  // one kernel family for all chunks: the one of a call on device tensors with all heads
  auto behind = [&](const Chunk& c) { return next_chunk(c, p->E, p->H, L.hc, L.ec, least_heads); };
  for (Chunk c = behind({0, 0, 0, 0}); c.e < p->E; c = behind(c), ++i) {
    const int e = c.e, ne = c.elements, h0 = c.h0, nh = c.heads;
    const int slot = i % kSlots;
    char* sq = base + (size_t)slot * L.slot_bytes;
    char* sk = sq + L.qk_bytes;
    char* sv = sk + L.qk_bytes;
    char* so = sv + L.v_bytes;
    // copy in: the kernels of the chunk that used this slot last have read q, k, v
    if (i >= kSlots || overlap) MA_TRY(cudaStreamWaitEvent(P->in, P->computed[slot], 0), "wait(in, computed)");
    MA_TRY(copy_heads(sq, p->q, e, ne, h0, nh, p->N, p->D, es_qk, true, P->in), "H2D q");
    MA_TRY(copy_heads(sk, p->k, e, ne, h0, nh, p->N, p->D, es_qk, true, P->in), "H2D k");
    MA_TRY(copy_heads(sv, p->v, e, ne, h0, nh, p->N, p->Dv, es_v, true, P->in), "H2D v");
    MA_TRY(cudaEventRecord(P->loaded[slot], P->in), "record(loaded)");
    // compute: inputs landed, and the previous result of this slot has left it
    MA_TRY(cudaStreamWaitEvent(P->comp, P->loaded[slot], 0), "wait(comp, loaded)");
    if (i >= kSlots || overlap) MA_TRY(cudaStreamWaitEvent(P->comp, P->stored[slot], 0), "wait(comp, stored)");
    ma_b200_problem sub = *p;
    sub.E = ne;
    sub.H = nh;
    sub.q = {sq, (int64_t)nh * p->N * p->D, (int64_t)p->N * p->D, p->D};
    sub.k = {sk, (int64_t)nh * p->N * p->D, (int64_t)p->N * p->D, p->D};
    sub.v = {sv, (int64_t)nh * p->N * p->Dv, (int64_t)p->N * p->Dv, p->Dv};
    sub.out = {so, (int64_t)nh * p->N * p->Dv, (int64_t)p->N * p->Dv, p->Dv};
    sub.mask = mask_dev != nullptr ? mask_dev + (size_t)e * p->N : nullptr;
    sub.mask_stride_e = mask_dev != nullptr ? p->N : 0;
    if (kernel == 0) kernel = ma_b200_kernel_of_part(&sub, (int64_t)p->E * p->H);
    if (kernel != 0) sub.kernel = kernel;  // (0: ma_b200_forward says why)
    rc = ma_b200_forward(&sub, base + L.ws_off, L.ws_bytes, P->comp);
    if (rc != MA_B200_OK) {
      g_host_error = std::string("chunk forward: ") + ma_b200_last_error();
      return rc;
    }
    MA_TRY(cudaEventRecord(P->computed[slot], P->comp), "record(computed)");
    // copy out
    MA_TRY(cudaStreamWaitEvent(P->out, P->computed[slot], 0), "wait(out, computed)");
    MA_TRY(copy_heads(so, p->out, e, ne, h0, nh, p->N, p->Dv, es_v, false, P->out), "D2H result");
    MA_TRY(cudaEventRecord(P->stored[slot], P->out), "record(stored)");
  }
  // the caller's stream continues once the last kernel and the last copy are done
  MA_TRY(cudaEventRecord(P->done_comp, P->comp), "record(done_comp)");
  MA_TRY(cudaEventRecord(P->done_out, P->out), "record(done_out)");
  MA_TRY(cudaStreamWaitEvent(caller, P->done_comp, 0), "wait(caller, done_comp)");
  MA_TRY(cudaStreamWaitEvent(caller, P->done_out, 0), "wait(caller, done_out)");
#undef MA_TRY
  return MA_B200_OK;
}

MA_B200_API int ma_b200_forward_host(const ma_b200_problem* p, int heads_per_chunk, void* device_scratch,
                                     size_t scratch_bytes, void* stream_v) {
  return ma_b200_forward_host_grouped(p, heads_per_chunk, 1, 1, 0, device_scratch, scratch_bytes, stream_v);
}

MA_B200_API int ma_b200_forward_host_streamed(const ma_b200_problem* p, int heads_per_chunk, void* device_scratch,
                                              size_t scratch_bytes, void* stream_v) {
  return ma_b200_forward_host_grouped(p, heads_per_chunk, 1, 1, 1, device_scratch, scratch_bytes, stream_v);
}

}  // extern "C"
