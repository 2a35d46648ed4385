// Shared by the tcgen05 tile kernels (ma_tile.cu, one launch per stage) and their single-launch form (ma_flow.inc): TMA
// wrappers, the passes over a tile row in tensor memory, and the tensor maps.
#pragma once

#include <cuda.h>
#include <math.h>
#include <string.h>

#include <algorithm>
#include <mutex>
#include <type_traits>

#include "ma_common.cuh"
#include "ma_sm100.cuh"

namespace ma {
namespace {

using namespace sm100;

constexpr int kRows = 128;         // rows of a tile
constexpr uint32_t kRowBytes = 128;  // 64 elements, zero-filled past D
constexpr float kGone = -1e30f;    // exponent of a column that does not exist or is masked

constexpr bool is_right(StageKind k) { return k == kStageRight || k == kStageRightWithV; }

// Element pair rounded to storage and back.
template <typename T>
__device__ __forceinline__ void round_pair(float& a, float& b);
template <>
__device__ __forceinline__ void round_pair<__nv_bfloat16>(float& a, float& b) {
  const uint32_t u = pack2<__nv_bfloat16>(a, b);
  a = __uint_as_float(u << 16);
  b = __uint_as_float(u & 0xffff0000u);
}
template <>
__device__ __forceinline__ void round_pair<__half>(float& a, float& b) {
  const float2 f = unpack2<__half>(pack2<__half>(a, b));
  a = f.x;
  b = f.y;
}

__device__ __forceinline__ void tma_load_4d(uint32_t dst, const CUtensorMap* map, uint32_t bar, int c0, int c1, int c2, int c3) {
  asm volatile(
      "cp.async.bulk.tensor.4d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4, %5}], [%6];" ::"r"(dst),
      "l"(map), "r"(c0), "r"(c1), "r"(c2), "r"(c3), "r"(bar)
      : "memory");
}
__device__ __forceinline__ void tma_store_4d(const CUtensorMap* map, uint32_t src, int c0, int c1, int c2, int c3) {
  asm volatile("cp.async.bulk.tensor.4d.global.shared::cta.bulk_group [%0, {%2, %3, %4, %5}], [%1];" ::"l"(map), "r"(src), "r"(c0),
               "r"(c1), "r"(c2), "r"(c3)
               : "memory");
}
__device__ __forceinline__ void tma_store_5d(const CUtensorMap* map, uint32_t src, int c0, int c1, int c2, int c3, int c4) {
  asm volatile("cp.async.bulk.tensor.5d.global.shared::cta.bulk_group [%0, {%2, %3, %4, %5, %6}], [%1];" ::"l"(map), "r"(src), "r"(c0),
               "r"(c1), "r"(c2), "r"(c3), "r"(c4)
               : "memory");
}
__device__ __forceinline__ float lg2(float x) {
  float y;
  asm("lg2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
__device__ __forceinline__ float rcp_fast(float x) {
  float y;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}

__device__ __forceinline__ bool token_valid(const Geometry& g, int e, int p) {
  const int n = p - g.pad_off;
  if (n < 0 || n >= g.N) return false;
  return mask_lets(g, e, n);
}

// Calls f(values, c) for the 16-column pieces c of a row of tensor memory (nch: its 32-column chunks), the next piece's
// load in flight behind the arithmetic of the present one.
template <typename F>
__device__ __forceinline__ void for_chunks(uint32_t t, int nch, F f) {
  float a[16], b[16];
  tmem_ld16_nowait(t, a);
#pragma unroll 1
  for (int c = 0; c < 2 * nch; c += 2) {
    tmem_wait_ld16(a);
    tmem_ld16_nowait(t + 16 * c + 16, b);
    f(a, c);
    tmem_wait_ld16(b);
    if (c + 2 < 2 * nch) tmem_ld16_nowait(t + 16 * c + 32, a);
    f(b, c + 1);
  }
}

struct Max4 {
  float m0 = -INFINITY, m1 = -INFINITY, m2 = -INFINITY, m3 = -INFINITY;
  __device__ __forceinline__ void take(const float (&v)[16]) {
#pragma unroll
    for (int i = 0; i < 16; i += 8) {
      m0 = max3(m0, v[i], v[i + 1]);
      m1 = max3(m1, v[i + 2], v[i + 3]);
      m2 = max3(m2, v[i + 4], v[i + 5]);
      m3 = max3(m3, v[i + 6], v[i + 7]);
    }
  }
  __device__ __forceinline__ float get() const { return fmaxf(fmaxf(m0, m1), fmaxf(m2, m3)); }
};
struct Sum2 {
  float2 a = make_float2(0.f, 0.f), b = make_float2(0.f, 0.f);
  __device__ __forceinline__ float get() const { return (a.x + a.y) + (b.x + b.y); }
};

// The row passes.  t_s: the row's columns of S, t_p: its half of the columns as 16-bit pairs.
// MASKED: some column of the chunks holds no key; the result is then the maximum of scale * S + bias, else that of S.
template <bool MASKED>
__device__ __forceinline__ float row_max(uint32_t t_s, int nch, const float* bias, float scale) {
  Max4 m;
  for_chunks(t_s, nch, [&](float(&v)[16], int c) {
    if (MASKED) {
#pragma unroll
      for (int i = 0; i < 16; i += 4) {
        const float4 b = *reinterpret_cast<const float4*>(bias + 16 * c + i);
        const float2 p = fma2(make_float2(v[i], v[i + 1]), make_float2(scale, scale), make_float2(b.x, b.y));
        const float2 q = fma2(make_float2(v[i + 2], v[i + 3]), make_float2(scale, scale), make_float2(b.z, b.w));
        v[i] = p.x; v[i + 1] = p.y; v[i + 2] = q.x; v[i + 3] = q.y;
      }
    }
    m.take(v);
  });
  return m.get();
}

// Right-factor rows: e = 2^(mul * round(S) - off) over S, sum of e and of e log2 e.
template <typename T, bool MASKED>
__device__ __forceinline__ void right_exps(uint32_t t_s, int nch, const float* bias, float mul, float off, float& sum, float& ent) {
  Sum2 s, n;
  for_chunks(t_s, nch, [&](float(&v)[16], int c) {
#pragma unroll
    for (int i = 0; i < 16; i += 4) {
      round_pair<T>(v[i], v[i + 1]);
      round_pair<T>(v[i + 2], v[i + 3]);
      float2 ua = fma2(make_float2(v[i], v[i + 1]), make_float2(mul, mul), make_float2(-off, -off));
      float2 ub = fma2(make_float2(v[i + 2], v[i + 3]), make_float2(mul, mul), make_float2(-off, -off));
      if (MASKED) {
        const float4 b = *reinterpret_cast<const float4*>(bias + 16 * c + i);
        ua = make_float2(b.x == 0.f ? ua.x : kGone, b.y == 0.f ? ua.y : kGone);
        ub = make_float2(b.z == 0.f ? ub.x : kGone, b.w == 0.f ? ub.y : kGone);
      }
      const float2 ea = make_float2(ex2(ua.x), ex2(ua.y)), eb = make_float2(ex2(ub.x), ex2(ub.y));
      s.a = add2(s.a, ea);
      s.b = add2(s.b, eb);
      n.a = fma2(ea, ua, n.a);
      n.b = fma2(eb, ub, n.b);
      v[i] = ea.x; v[i + 1] = ea.y; v[i + 2] = eb.x; v[i + 3] = eb.y;
    }
    tmem_st16(t_s + 16 * c, *reinterpret_cast<const uint32_t(*)[16]>(&v[0]));
  });
  tmem_wait_st();
  sum = s.get();
  ent = n.get();
}

// Column rows: sum of e = 2^(log2e * round(S) + bias - off); STORE: e over S.
template <typename T, bool STORE>
__device__ __forceinline__ float column_exps(uint32_t t_s, int nch, const float* bias, float off) {
  Sum2 s;
  for_chunks(t_s, nch, [&](float(&v)[16], int c) {
#pragma unroll
    for (int i = 0; i < 16; i += 4) {
      const float4 b = *reinterpret_cast<const float4*>(bias + 16 * c + i);
      round_pair<T>(v[i], v[i + 1]);
      round_pair<T>(v[i + 2], v[i + 3]);
      const float2 ua = add2(fma2(make_float2(v[i], v[i + 1]), make_float2(kLog2e, kLog2e), make_float2(b.x, b.y)), make_float2(-off, -off));
      const float2 ub = add2(fma2(make_float2(v[i + 2], v[i + 3]), make_float2(kLog2e, kLog2e), make_float2(b.z, b.w)), make_float2(-off, -off));
      v[i] = ex2(ua.x); v[i + 1] = ex2(ua.y); v[i + 2] = ex2(ub.x); v[i + 3] = ex2(ub.y);
      s.a = add2(s.a, make_float2(v[i], v[i + 1]));
      s.b = add2(s.b, make_float2(v[i + 2], v[i + 3]));
    }
    if (STORE) tmem_st16(t_s + 16 * c, *reinterpret_cast<const uint32_t(*)[16]>(&v[0]));
  });
  if (STORE) tmem_wait_st();
  return s.get();
}

constexpr float kFar = 1048576.f;
constexpr float kLeastShift = 0.1f * kGone;

template <int N>
__device__ __forceinline__ float max_of(const float (&v)[N]) {
  Max4 m;
  m.take(v);
  return m.get();
}
__device__ __forceinline__ bool is_far(const Sum2& s) { return fmaxf(fmaxf(s.a.x, s.a.y), fmaxf(s.b.x, s.b.y)) > kFar; }
// The columns before piece c times f.
__device__ __forceinline__ void scale_columns(uint32_t t_s, int c, float f) {
  tmem_wait_st();
#pragma unroll 1
  for (int i = 0; i < c; ++i) {
    float v[16];
    tmem_ld16_nowait(t_s + 16 * i, v);
    tmem_wait_ld16(v);
#pragma unroll
    for (int k = 0; k < 16; ++k) v[k] *= f;
    tmem_st16(t_s + 16 * i, *reinterpret_cast<const uint32_t(*)[16]>(&v[0]));
  }
  tmem_wait_st();
}

// Column rows where columns are missing (bias kGone): the maximum would need the biases too, and with them its pass takes as
// long as that of the exponentials.  Any off within a few powers of two of the row's largest exponent gives the same
// quotients, so it is taken from the first 16 columns, and raised to the maximum of later ones (what was formed before is scaled
// down) where a sum of 16 passes 2^20; a row sum in fp32 is good to 2^127, so nothing has been lost by then.  48 heads of 7683
// tokens in fp16, blocks of 64, masked, calls back to back on three sets of inputs: 171 us instead of 174 with a pass for the
// maximum; on one set 159 instead of 160.  (Where no column is missing that pass is as fast: the check costs what it saves.)  Logits below the range of the storage type are -inf, and 16 such columns would make the shift -inf and e NaN:
// it stays above kLeastShift, far below any other logit and far above a missing column's.  STORE: e over S.
template <typename T, bool STORE>
__device__ __forceinline__ float masked_column_exps(uint32_t t_s, int nch, const float* bias, float& off) {
  Sum2 s;
  off = 0.f;
  for_chunks(t_s, nch, [&](float(&v)[16], int c) {
    Sum2 cs;
    auto logits = [&] {
#pragma unroll
      for (int i = 0; i < 16; i += 4) {
        const float4 b = *reinterpret_cast<const float4*>(bias + 16 * c + i);
        round_pair<T>(v[i], v[i + 1]);
        round_pair<T>(v[i + 2], v[i + 3]);
        const float2 ua = fma2(make_float2(v[i], v[i + 1]), make_float2(kLog2e, kLog2e), make_float2(b.x, b.y));
        const float2 ub = fma2(make_float2(v[i + 2], v[i + 3]), make_float2(kLog2e, kLog2e), make_float2(b.z, b.w));
        v[i] = ua.x; v[i + 1] = ua.y; v[i + 2] = ub.x; v[i + 3] = ub.y;
      }
    };
    auto exps = [&] {
#pragma unroll
      for (int i = 0; i < 16; i += 4) {
        const float2 ua = add2(make_float2(v[i], v[i + 1]), make_float2(-off, -off));
        const float2 ub = add2(make_float2(v[i + 2], v[i + 3]), make_float2(-off, -off));
        v[i] = ex2(ua.x); v[i + 1] = ex2(ua.y); v[i + 2] = ex2(ub.x); v[i + 3] = ex2(ub.y);
        const float2 ea = make_float2(v[i], v[i + 1]), eb = make_float2(v[i + 2], v[i + 3]);
        cs.a = i == 0 ? ea : add2(cs.a, ea);
        cs.b = i == 0 ? eb : add2(cs.b, eb);
      }
    };
    logits();
    if (c == 0) off = fmaxf(max_of(v), kLeastShift);
    exps();
    const bool far = is_far(cs);
    if (__any_sync(0xffffffffu, far)) {
      tmem_ld16_nowait(t_s + 16 * c, v);
      tmem_wait_ld16(v);
      logits();
      const float to = far ? fmaxf(max_of(v), off) : off, f = ex2(off - to);  // (a row goes by its own columns: f = 1 in the others)
      if (STORE) scale_columns(t_s, c, f);
      s.a = mul2(s.a, make_float2(f, f));
      s.b = mul2(s.b, make_float2(f, f));
      off = to;
      exps();
    }
    s.a = add2(s.a, cs.a);
    s.b = add2(s.b, cs.b);
    if (STORE) tmem_st16(t_s + 16 * c, *reinterpret_cast<const uint32_t(*)[16]>(&v[0]));
  });
  if (STORE) tmem_wait_st();
  return s.get();
}

// P = e * inv, e as left over S.
template <typename T>
__device__ __forceinline__ void normalise(uint32_t t_s, uint32_t t_p, int nch, float inv) {
  for_chunks(t_s, nch, [&](float(&v)[16], int c) {
    uint32_t pk[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      const float2 r = mul2(make_float2(v[2 * i], v[2 * i + 1]), make_float2(inv, inv));
      pk[i] = pack2<T>(r.x, r.y);
    }
    tmem_st8(t_p + 8 * c, pk);
  });
}

// ---------------------------------------------------------------------------------------------------
// Host side: tensor maps
// ---------------------------------------------------------------------------------------------------
typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*, const cuuint64_t*,
                                  const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle,
                                  CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

EncodeTiledFn encode_fn() {
  static EncodeTiledFn fn = nullptr;
  static std::once_flag once;
  std::call_once(once, [] {
    void* p = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPointByVersion("cuTensorMapEncodeTiled", &p, 12000, cudaEnableDefault, &q) == cudaSuccess &&
        q == cudaDriverEntryPointSuccess)
      fn = reinterpret_cast<EncodeTiledFn>(p);
  });
  return fn;
}

// Everything that enters a tensor map.  Encoding takes about as long as queuing a launch, and a program calls with the
// same buffers again and again, so the last maps are kept (a fixed number, found by comparing all of the description).
struct MapKey {
  const void* base;
  cuuint64_t dims[5], strides[4];
  cuuint32_t box[5];
  int rank, dtype, device;
};
struct MapEntry { MapKey key; CUtensorMap map; unsigned long long hash; };
constexpr int kMapCache = 256;  // direct-mapped
MapEntry g_maps[kMapCache];
std::mutex g_maps_mutex;

unsigned long long hash_key(const MapKey& k) {
  const unsigned char* p = reinterpret_cast<const unsigned char*>(&k);
  unsigned long long h = 1469598103934665603ull, w;
  for (size_t i = 0; i + 8 <= sizeof(MapKey); i += 8) {
    memcpy(&w, p + i, 8);
    h = (h ^ w) * 1099511628211ull;
    h ^= h >> 29;
  }
  return h | 1;
}

bool make_map(CUtensorMap* out, int dtype, const void* base, int rank, const cuuint64_t* dims, const cuuint64_t* strides_bytes,
              const cuuint32_t* box) {
  MapKey k;
  memset(&k, 0, sizeof(k));
  k.base = base; k.rank = rank; k.dtype = dtype;
  if (cudaGetDevice(&k.device) != cudaSuccess) return false;
  for (int i = 0; i < rank; ++i) { k.dims[i] = dims[i]; k.box[i] = box[i]; }
  for (int i = 0; i + 1 < rank; ++i) {
    k.strides[i] = strides_bytes[i];
    // a dimension of one entry may carry any stride; give the encoder a legal one
    if (k.dims[i + 1] == 1 && (k.strides[i] == 0 || k.strides[i] % 16 != 0)) k.strides[i] = 128;
  }
  const unsigned long long h = hash_key(k);
  MapEntry& m = g_maps[(h >> 8) % kMapCache];
  std::lock_guard<std::mutex> lock(g_maps_mutex);
  if (m.hash == h && memcmp(&m.key, &k, sizeof(k)) == 0) { *out = m.map; return true; }
  const cuuint32_t estr[5] = {1, 1, 1, 1, 1};
  const CUtensorMapDataType dt = dtype == MA_B200_BF16 ? CU_TENSOR_MAP_DATA_TYPE_BFLOAT16 : CU_TENSOR_MAP_DATA_TYPE_FLOAT16;
  if (encode_fn()(&m.map, dt, rank, const_cast<void*>(base), k.dims, k.strides, k.box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                  CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) != CUDA_SUCCESS) {
    m.hash = 0;
    return false;
  }
  m.key = k;
  m.hash = h;
  *out = m.map;
  return true;
}

// (D, tokens, H, E) view of a user tensor
bool token_map(CUtensorMap* m, int dtype, const Geometry& g, const View4& t, int rows) {
  const cuuint64_t dims[4] = {(cuuint64_t)g.D, (cuuint64_t)g.N, (cuuint64_t)g.H, (cuuint64_t)g.E};
  const cuuint64_t str[3] = {(cuuint64_t)t.sn * 2, (cuuint64_t)t.sh * 2, (cuuint64_t)t.se * 2};
  const cuuint32_t box[4] = {64, (cuuint32_t)rows, 1, 1};
  return make_map(m, dtype, t.ptr, 4, dims, str, box);
}
// (D, B, whole rows of B tokens, H, E) view: a box takes one column
bool column_map(CUtensorMap* m, int dtype, const Geometry& g, const View4& t, int rows) {
  const cuuint64_t dims[5] = {(cuuint64_t)g.D, (cuuint64_t)g.B, (cuuint64_t)(g.N / g.B), (cuuint64_t)g.H, (cuuint64_t)g.E};
  const cuuint64_t str[4] = {(cuuint64_t)t.sn * 2, (cuuint64_t)t.sn * 2 * g.B, (cuuint64_t)t.sh * 2, (cuuint64_t)t.se * 2};
  const cuuint32_t box[5] = {64, 1, (cuuint32_t)rows, 1, 1};
  return make_map(m, dtype, t.ptr, 5, dims, str, box);
}
// (D, rows of a head, E*H, 1) view of a state tensor
bool state_map(CUtensorMap* m, int dtype, const Geometry& g, const void* base, int rows) {
  const cuuint64_t n = (cuuint64_t)g.B * g.M, eh = (cuuint64_t)g.E * g.H;
  const cuuint64_t dims[4] = {(cuuint64_t)g.D, n, eh, 1};
  const cuuint64_t str[3] = {(cuuint64_t)g.D * 2, n * g.D * 2, n * g.D * 2 * eh};
  const cuuint32_t box[4] = {64, (cuuint32_t)rows, 1, 1};
  return make_map(m, dtype, base, 4, dims, str, box);
}
// (D, inner, outer, E*H) view of a state tensor whose rows (outer, inner) are written one `inner` at a time
bool strided_state_map(CUtensorMap* m, int dtype, const Geometry& g, const void* base, int inner, int outer, int rows) {
  const cuuint64_t row = (cuuint64_t)g.D * 2;
  const cuuint64_t dims[4] = {(cuuint64_t)g.D, (cuuint64_t)inner, (cuuint64_t)outer, (cuuint64_t)g.E * g.H};
  const cuuint64_t str[3] = {row, row * inner, row * inner * outer};
  const cuuint32_t box[4] = {64, 1, (cuuint32_t)rows, 1};
  return make_map(m, dtype, base, 4, dims, str, box);
}

}  // namespace
}  // namespace ma
