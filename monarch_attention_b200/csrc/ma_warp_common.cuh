// Warp-level building blocks shared by the stage kernels (ma_warp.cu) and the backward kernels (ma_backward.cu):
// ldmatrix / mma.sync wrappers, the asynchronous tile loader, and the 16 x 16 fragment operations of one
// element type.
#pragma once

#include "ma_common.cuh"

namespace ma {
namespace {

__device__ __forceinline__ uint32_t smem_addr(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }

__device__ __forceinline__ void ldsm_x4(uint32_t addr, uint32_t (&r)[4]) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0, %1, %2, %3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
               : "r"(addr));
}
__device__ __forceinline__ void ldsm_x2(uint32_t addr, uint32_t (&r)[2]) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x2.shared.b16 {%0, %1}, [%2];" : "=r"(r[0]), "=r"(r[1]) : "r"(addr));
}
__device__ __forceinline__ void ldsm_x2_trans(uint32_t addr, uint32_t (&r)[2]) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x2.trans.shared.b16 {%0, %1}, [%2];" : "=r"(r[0]), "=r"(r[1]) : "r"(addr));
}
__device__ __forceinline__ void ldsm_x4_trans(uint32_t addr, uint32_t (&r)[4]) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0, %1, %2, %3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
               : "r"(addr));
}

template <typename T>
__device__ __forceinline__ void mma16816(float (&c)[4], const uint32_t (&a)[4], const uint32_t (&b)[2]);
template <>
__device__ __forceinline__ void mma16816<__nv_bfloat16>(float (&c)[4], const uint32_t (&a)[4], const uint32_t (&b)[2]) {
  asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, "
               "{%0, %1, %2, %3};"
               : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
               : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b[0]), "r"(b[1]));
}
template <>
__device__ __forceinline__ void mma16816<__half>(float (&c)[4], const uint32_t (&a)[4], const uint32_t (&b)[2]) {
  asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, "
               "{%0, %1, %2, %3};"
               : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
               : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b[0]), "r"(b[1]));
}

template <typename T>
__device__ __forceinline__ uint32_t pack_pair(float lo, float hi);
template <>
__device__ __forceinline__ uint32_t pack_pair<__nv_bfloat16>(float lo, float hi) {
  __nv_bfloat162 v = __floats2bfloat162_rn(lo, hi);
  return *reinterpret_cast<uint32_t*>(&v);
}
template <>
__device__ __forceinline__ uint32_t pack_pair<__half>(float lo, float hi) {
  __half2 v = __floats2half2_rn(lo, hi);
  return *reinterpret_cast<uint32_t*>(&v);
}

__device__ __forceinline__ float quad_max(float v) {
  v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, 1));
  return fmaxf(v, __shfl_xor_sync(0xffffffffu, v, 2));
}
__device__ __forceinline__ float quad_sum(float v) {
  v += __shfl_xor_sync(0xffffffffu, v, 1);
  return v + __shfl_xor_sync(0xffffffffu, v, 2);
}

// Sums over the eight lanes lane/4 of N values per lane (N a power of two, at least 4), by halving: a step sends one
// half of the values to the partner and keeps the other, so N values take about N shuffles instead of 3 N.  Returns
// the index of the first of the values left in this lane; N/8 values are left (one, twice over, when N = 4).
template <int N>
__device__ __forceinline__ int reduce_rows(float (&v)[N], int lane) {
  int base = 0;
  int n = N;
#pragma unroll
  for (int d = 16; d >= 4; d >>= 1) {
    if (n > 1) {
      const bool up = (lane & d) != 0;
      n >>= 1;
#pragma unroll
      for (int i = 0; i < N / 2; ++i)
        if (i < n) {
          const float send = up ? v[i] : v[i + n], keep = up ? v[i + n] : v[i];
          v[i] = keep + __shfl_xor_sync(0xffffffffu, send, d);
        }
      if (up) base += n;
    } else {
      v[0] += __shfl_xor_sync(0xffffffffu, v[0], d);
    }
  }
  return base;
}

// Copies `rows` rows of `width` elements (whole 16-byte pieces) into a shared tile with row pitch `pitch` elements,
// zero-filling rows that do not exist, columns past width and rows [rows, rpad).  Threads tid of nthreads cooperate.  The
// copies are asynchronous (cp.async, 16 bytes each, zero-fill by giving a source size of 0): a thread queues all of its
// pieces without waiting; tiles_commit_and_wait() must be called before the tile is read.
// Every source these kernels have is an arithmetic progression of rows: row r comes from element
// offset (n0 + r*nstep)*row_stride of `base` and exists iff r < rows and 0 <= n0 + r*nstep < n_limit
// (token index inside the sequence; for the dense state tensors n0 = 0, nstep = 1, n_limit = rows).
// fp32: eight threads share a row, and a thread takes every eighth piece of it, so that all but the first of a row's copies
// differ from it by constants.  The fp32 stage kernels are bound by their instructions, and those that worked out a row and a
// column for every piece were 300 of 2530 (16 x 16 x 72) for each tile (67.3 instead of 72 us for 128 heads of 256 x 72, three
// iterations).  16-bit types, whose rows are one or two lines: one piece after the other, with row, column chunk, token index
// and source offset carried along by additions only; shared rows were slower there (64 x 12 heads of 197 x 64: 39.1 instead of
// 37.1 us; 8 x 16 of 2025 x 80: 115 instead of 107).  Together with store_rows' stores from fragments, which the backward kernels
// share, a training step in fp32 went from 479 to 461 us (4 x 12 heads of 1024 x 64, three iterations) and from 1058 to 996 (2 x 12
// of 4096 x 64, two).
template <typename T, int CHUNKS>  // CHUNKS: 16-byte pieces of a padded row
__device__ __forceinline__ void load_rows(T* tile, int pitch, int rows, int rpad, int width, const T* base, int n0,
                                          int nstep, int n_limit, long long row_stride, int tid, int nthreads,
                                          const void* any_valid_global) {
  constexpr int kPer = 16 / (int)sizeof(T);  // elements of a piece
  if constexpr (sizeof(T) == 4) {
    constexpr int L = 8;
    const int q = tid % L;
    for (int r = tid / L; r < rpad; r += nthreads / L) {
      const int n = n0 + r * nstep;
      const bool ok = r < rows && (unsigned)n < (unsigned)n_limit;
      const T* src = (ok ? base + (long long)n * row_stride : static_cast<const T*>(any_valid_global)) + q * kPer;
      const uint32_t dst = smem_addr(tile + r * pitch + q * kPer);
#pragma unroll
      for (int c = 0; c < CHUNKS; c += L) {
        if (c + L > CHUNKS && c + q >= CHUNKS) break;
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst + 16u * c), "l"(src + c * kPer),
                     "r"(ok && (c + q) * kPer < width ? 16u : 0u)
                     : "memory");
      }
    }
  } else {
    int r = tid / CHUNKS, c = tid - r * CHUNKS;
    const int dr = nthreads / CHUNKS, dc = nthreads - dr * CHUNKS;
    int n = n0 + r * nstep;
    const T* src = base + (long long)n * row_stride;
    uint32_t dst = smem_addr(tile + r * pitch);
    const int dn = dr * nstep;
    const long long dsrc = (long long)dn * row_stride, step1 = (long long)nstep * row_stride;
    const uint32_t ddst = (uint32_t)(dr * pitch) * (uint32_t)sizeof(T), dst1 = (uint32_t)pitch * (uint32_t)sizeof(T);
    while (r < rpad) {
      const bool ok = r < rows && c * kPer < width && (unsigned)n < (unsigned)n_limit;
      const void* gsrc = ok ? static_cast<const void*>(src + c * kPer) : any_valid_global;
      asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst + (uint32_t)(c << 4)), "l"(gsrc),
                   "r"(ok ? 16u : 0u)
                   : "memory");
      c += dc; r += dr; n += dn; src += dsrc; dst += ddst;
      if (c >= CHUNKS) { c -= CHUNKS; ++r; n += nstep; src += step1; dst += dst1; }
    }
  }
}
__device__ __forceinline__ void tiles_commit_and_wait() {
  asm volatile("cp.async.commit_group;" ::: "memory");
  asm volatile("cp.async.wait_group 0;" ::: "memory");
}

// The first kernel of a call zeroes the workspace's status word, so that no separate clear has to be queued.
__device__ __forceinline__ void clear_status(const Geometry& g) {
  if (threadIdx.x == 0 && blockIdx.x == 0 && blockIdx.y == 0) *g.status = 0;
}

__device__ __forceinline__ bool pos_valid(const Geometry& g, int e, int p) {
  const int n = p - g.pad_off;
  if (n < 0 || n >= g.N) return false;
  return mask_lets(g, e, n);
}
// Row of a user tensor for padded position p, given the (e, h) base pointer: nullptr for padding.
template <typename T>
__device__ __forceinline__ const T* head_base(const View4& t, int e, int h) {
  return reinterpret_cast<const T*>(t.ptr) + (long long)e * t.se + (long long)h * t.sh;
}
// ---------------------------------------------------------------------------------------------------
// Contractions of one warp on 16 x 16 pieces of one element type: A (16 x 16) times B (16 x 16, as two n8 tiles)
// into two m16n8 fp32 accumulator tiles.  16-bit types: one m16n8k16 per n8 tile.  fp32: operands split into a
// tf32 part and the tf32 of the remainder, three m16n8k8 per n8 tile and k8 step (small products first), which keeps
// about 22 bits of every operand; the plain fp32 pipes would need 32 x as many instructions for the same tile.
// Accumulator element layout (both): c[0], c[1] = row lane/4, columns 2*(lane%4), +1; c[2], c[3] = row + 8.
// ---------------------------------------------------------------------------------------------------
template <typename T>
struct Tile {
  struct A { uint32_t r[4]; };
  struct B { uint32_t r[4]; };
  // A[m][k] = s[m * pitch + k]
  static __device__ __forceinline__ void load_a(A& a, const T* s, int pitch, int lane) {
    ldsm_x4(smem_addr(s + ((lane & 7) + ((lane >> 3) & 1) * 8) * pitch + (lane >> 4) * 8), a.r);
  }
  // A[m][k] = s[k * pitch + m]
  static __device__ __forceinline__ void load_a_t(A& a, const T* s, int pitch, int lane) {
    ldsm_x4_trans(smem_addr(s + ((lane & 7) + (lane >> 4) * 8) * pitch + ((lane >> 3) & 1) * 8), a.r);
  }
  // B[k][n] = s[n * pitch + k]
  static __device__ __forceinline__ void load_b_nk(B& b, const T* s, int pitch, int lane) {
    ldsm_x4(smem_addr(s + ((lane & 7) + (lane >> 4) * 8) * pitch + ((lane >> 3) & 1) * 8), b.r);
  }
  // B[k][n] = s[k * pitch + n]
  static __device__ __forceinline__ void load_b_kn(B& b, const T* s, int pitch, int lane) {
    ldsm_x4_trans(smem_addr(s + ((lane & 7) + ((lane >> 3) & 1) * 8) * pitch + (lane >> 4) * 8), b.r);
  }
  static __device__ __forceinline__ void from_acc(A& a, const float (&c0)[4], const float (&c1)[4]) {
    a.r[0] = pack_pair<T>(c0[0], c0[1]);
    a.r[1] = pack_pair<T>(c0[2], c0[3]);
    a.r[2] = pack_pair<T>(c1[0], c1[1]);
    a.r[3] = pack_pair<T>(c1[2], c1[3]);
  }
  static __device__ __forceinline__ void mma(float (&c0)[4], float (&c1)[4], const A& a, const B& b) {
    const uint32_t b0[2] = {b.r[0], b.r[1]}, b1[2] = {b.r[2], b.r[3]};
    mma16816<T>(c0, a.r, b0);
    mma16816<T>(c1, a.r, b1);
  }
  static __device__ __forceinline__ void store_pair(T* p, float lo, float hi) {
    *reinterpret_cast<uint32_t*>(p) = pack_pair<T>(lo, hi);
  }
};

__device__ __forceinline__ void mma1688_tf32(float (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3,
                                             uint32_t b0, uint32_t b1) {
  asm volatile("mma.sync.aligned.m16n8k8.row.col.f32.tf32.tf32.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, "
               "{%0, %1, %2, %3};"
               : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
               : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}

// The k index inside a k8 step is permuted so that a step's columns are those of one accumulator tile: k = t is
// column 2t, k = t + 4 is column 2t + 1 (t = lane % 4), for A and B alike.
template <>
struct Tile<float> {
  struct A { float hi[8], lo[8]; };  // [step][a0..a3]
  struct B { float hi[8], lo[8]; };  // [n8 tile][step][b0, b1]
  static __device__ __forceinline__ void split(float x, float& hi, float& lo) {
    // round to nearest at 11 bits, twice (the tensor path ignores the bits below, so the remainder's need not be
    // cleared); rounding instead of cutting takes the result's error from 3e-6 to 5e-7, the plain fp32 kernels' own
    hi = __uint_as_float((__float_as_uint(x) + 0x1000u) & 0xffffe000u);
    lo = __uint_as_float(__float_as_uint(x - hi) + 0x1000u);
  }
  static __device__ __forceinline__ void load_a(A& a, const float* s, int pitch, int lane) {
    const float* p = s + (lane >> 2) * pitch + 2 * (lane & 3);
#pragma unroll
    for (int st = 0; st < 2; ++st) {
      const float2 x = *reinterpret_cast<const float2*>(p + 8 * st);
      const float2 y = *reinterpret_cast<const float2*>(p + 8 * pitch + 8 * st);
      split(x.x, a.hi[4 * st], a.lo[4 * st]);
      split(y.x, a.hi[4 * st + 1], a.lo[4 * st + 1]);
      split(x.y, a.hi[4 * st + 2], a.lo[4 * st + 2]);
      split(y.y, a.hi[4 * st + 3], a.lo[4 * st + 3]);
    }
  }
  static __device__ __forceinline__ void load_a_t(A& a, const float* s, int pitch, int lane) {
    const float* p = s + 2 * (lane & 3) * pitch + (lane >> 2);
#pragma unroll
    for (int st = 0; st < 2; ++st) {
      split(p[(8 * st) * pitch], a.hi[4 * st], a.lo[4 * st]);
      split(p[(8 * st) * pitch + 8], a.hi[4 * st + 1], a.lo[4 * st + 1]);
      split(p[(8 * st + 1) * pitch], a.hi[4 * st + 2], a.lo[4 * st + 2]);
      split(p[(8 * st + 1) * pitch + 8], a.hi[4 * st + 3], a.lo[4 * st + 3]);
    }
  }
  static __device__ __forceinline__ void load_b_nk(B& b, const float* s, int pitch, int lane) {
    const float* p = s + (lane >> 2) * pitch + 2 * (lane & 3);
#pragma unroll
    for (int n = 0; n < 2; ++n)
#pragma unroll
      for (int st = 0; st < 2; ++st) {
        const float2 x = *reinterpret_cast<const float2*>(p + 8 * n * pitch + 8 * st);
        split(x.x, b.hi[4 * n + 2 * st], b.lo[4 * n + 2 * st]);
        split(x.y, b.hi[4 * n + 2 * st + 1], b.lo[4 * n + 2 * st + 1]);
      }
  }
  static __device__ __forceinline__ void load_b_kn(B& b, const float* s, int pitch, int lane) {
    const float* p = s + 2 * (lane & 3) * pitch + (lane >> 2);
#pragma unroll
    for (int n = 0; n < 2; ++n)
#pragma unroll
      for (int st = 0; st < 2; ++st) {
        split(p[(8 * st) * pitch + 8 * n], b.hi[4 * n + 2 * st], b.lo[4 * n + 2 * st]);
        split(p[(8 * st + 1) * pitch + 8 * n], b.hi[4 * n + 2 * st + 1], b.lo[4 * n + 2 * st + 1]);
      }
  }
  static __device__ __forceinline__ void from_acc(A& a, const float (&c0)[4], const float (&c1)[4]) {
#pragma unroll
    for (int st = 0; st < 2; ++st) {
      const float(&c)[4] = st == 0 ? c0 : c1;
      split(c[0], a.hi[4 * st], a.lo[4 * st]);
      split(c[2], a.hi[4 * st + 1], a.lo[4 * st + 1]);
      split(c[1], a.hi[4 * st + 2], a.lo[4 * st + 2]);
      split(c[3], a.hi[4 * st + 3], a.lo[4 * st + 3]);
    }
  }
  static __device__ __forceinline__ void mma_part(float (&c)[4], const float* a, const float* b) {
    mma1688_tf32(c, __float_as_uint(a[0]), __float_as_uint(a[1]), __float_as_uint(a[2]), __float_as_uint(a[3]),
                 __float_as_uint(b[0]), __float_as_uint(b[1]));
  }
  // The tensor path aligns a step's products and its accumulator input to the largest of them and cuts the rest
  // off, so a long chain of steps on one accumulator drifts.  Every 16 products therefore start from zero (small
  // parts first) and are added to the running sum by an ordinary rounded addition.
  static __device__ __forceinline__ void mma(float (&c0)[4], float (&c1)[4], const A& a, const B& b) {
    float t0[4] = {0.f, 0.f, 0.f, 0.f}, t1[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
    for (int st = 0; st < 2; ++st) {
      mma_part(t0, a.lo + 4 * st, b.hi + 2 * st);
      mma_part(t1, a.lo + 4 * st, b.hi + 4 + 2 * st);
      mma_part(t0, a.hi + 4 * st, b.lo + 2 * st);
      mma_part(t1, a.hi + 4 * st, b.lo + 4 + 2 * st);
    }
#pragma unroll
    for (int st = 0; st < 2; ++st) {
      mma_part(t0, a.hi + 4 * st, b.hi + 2 * st);
      mma_part(t1, a.hi + 4 * st, b.hi + 4 + 2 * st);
    }
#pragma unroll
    for (int i = 0; i < 4; ++i) { c0[i] += t0[i]; c1[i] += t1[i]; }
  }
  static __device__ __forceinline__ void store_pair(float* p, float lo, float hi) {
    *reinterpret_cast<float2*>(p) = make_float2(lo, hi);
  }
};

constexpr float kWLog2e = 1.4426950408889634f;
constexpr float kWLn2 = 0.6931471805599453f;

__device__ __forceinline__ float fast_ex2(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}

// exp(t) for t <= 0: the 16-bit pipelines round the result to 8 or 11 bits right after, fp32 takes the
// full-precision function.
template <typename T>
__device__ __forceinline__ float exp_of(float t) { return fast_ex2(t * kWLog2e); }
template <>
__device__ __forceinline__ float exp_of<float>(float t) { return expf(t); }
template <typename T>
__device__ __forceinline__ float log_of(float x) { return __logf(x); }
template <>
__device__ __forceinline__ float log_of<float>(float x) { return logf(x); }

// S[16 x KP] (fp32 fragments) = A[16 x DP] * Bt[KP x DP]^T for one warp.  sA points at the warp's first
// row; both tiles are row-major with pitch PITCH elements.
template <typename T, int KP, int DP, int PITCH>
__device__ __forceinline__ void warp_gemm_abt(float (&s)[KP / 8][4], const T* sA, const T* sB, int lane) {
#pragma unroll
  for (int nt = 0; nt < KP / 8; ++nt) s[nt][0] = s[nt][1] = s[nt][2] = s[nt][3] = 0.f;
#pragma unroll
  for (int kk = 0; kk < DP / 16; ++kk) {
    typename Tile<T>::A a;
    Tile<T>::load_a(a, sA + kk * 16, PITCH, lane);
#pragma unroll
    for (int np = 0; np < KP / 16; ++np) {
      typename Tile<T>::B b;
      Tile<T>::load_b_nk(b, sB + np * 16 * PITCH + kk * 16, PITCH, lane);
      Tile<T>::mma(s[2 * np], s[2 * np + 1], a, b);
    }
  }
}

// A softmax factor (accumulator fragments of a 16 x KP tile) kept for the contractions that consume it:
// 16-bit types as packed A fragments, fp32 as it is (the split into two tf32 parts is redone per use).
template <typename T, int KP>
struct Factor {
  typename Tile<T>::A p[KP / 16];
  __device__ __forceinline__ void set(const float (&s)[KP / 8][4]) {
#pragma unroll
    for (int kt = 0; kt < KP / 16; ++kt) Tile<T>::from_acc(p[kt], s[2 * kt], s[2 * kt + 1]);
  }
  __device__ __forceinline__ const typename Tile<T>::A& get(int kt) const { return p[kt]; }
};
template <int KP>
struct Factor<float, KP> {
  float s[KP / 8][4];
  __device__ __forceinline__ void set(const float (&x)[KP / 8][4]) {
#pragma unroll
    for (int nt = 0; nt < KP / 8; ++nt)
#pragma unroll
      for (int i = 0; i < 4; ++i) s[nt][i] = x[nt][i];
  }
  __device__ __forceinline__ Tile<float>::A get(int kt) const {
    Tile<float>::A a;
    Tile<float>::from_acc(a, s[2 * kt], s[2 * kt + 1]);
    return a;
  }
};

// O[16 x DP] = P[16 x KP] * V[KP x DP], V row-major.
template <typename T, int KP, int DP, int PITCH>
__device__ __forceinline__ void warp_gemm_pv(float (&o)[DP / 8][4], const Factor<T, KP>& p, const T* sV, int lane) {
#pragma unroll
  for (int nt = 0; nt < DP / 8; ++nt) o[nt][0] = o[nt][1] = o[nt][2] = o[nt][3] = 0.f;
#pragma unroll
  for (int kt = 0; kt < KP / 16; ++kt) {
    const typename Tile<T>::A a = p.get(kt);
#pragma unroll
    for (int np = 0; np < DP / 16; ++np) {
      typename Tile<T>::B b;
      Tile<T>::load_b_kn(b, sV + kt * 16 * PITCH + np * 16, PITCH, lane);
      Tile<T>::mma(o[2 * np], o[2 * np + 1], a, b);
    }
  }
}

// Writes a warp's 16 x D accumulator tile to global rows; row_ptr(r) gives the destination of row r (0..15) or nullptr to
// skip it.  fp32: straight from the fragments, four lanes writing 32 consecutive bytes of a row.  16-bit types: the fragments
// go to a 16-row staging area in shared memory (the warp's own, no longer needed operand rows), then every lane copies 16-byte
// pieces, so that each 128-byte row is written by eight consecutive lanes.
template <typename T, int DP, int PITCH, typename RowFn>
__device__ __forceinline__ void store_rows(const float (&o)[DP / 8][4], T* stage, RowFn row_ptr, int D, int lane,
                                           float post_scale, bool double_round) {
  const int gq = lane >> 2, t = lane & 3;
  if constexpr (sizeof(T) == 4) {
    T* const rows[2] = {row_ptr(gq), row_ptr(gq + 8)};
    __syncwarp();
#pragma unroll
    for (int nt = 0; nt < DP / 8; ++nt) {
      const int c = nt * 8 + 2 * t;
      if (c >= D) break;
      if (rows[0] != nullptr) Tile<T>::store_pair(rows[0] + c, o[nt][0] * post_scale, o[nt][1] * post_scale);
      if (rows[1] != nullptr) Tile<T>::store_pair(rows[1] + c, o[nt][2] * post_scale, o[nt][3] * post_scale);
    }
    __syncwarp();
    return;
  }
  // The reference rounds the product to storage before scaling it (ma/ma_torch.py:21).  Scaling by a power
  // of two (1/sqrt(D) for D = 16, 64, 256) commutes with rounding, so one rounding gives the same bits.
  const bool two_roundings = double_round && (__float_as_uint(post_scale) & 0x007fffffu) != 0u;
  __syncwarp();
#pragma unroll
  for (int nt = 0; nt < DP / 8; ++nt) {
    const int c = nt * 8 + 2 * t;
    float v0 = o[nt][0], v1 = o[nt][1], v2 = o[nt][2], v3 = o[nt][3];
    if (two_roundings) {
      v0 = round_through<T>(v0); v1 = round_through<T>(v1); v2 = round_through<T>(v2); v3 = round_through<T>(v3);
    }
    Tile<T>::store_pair(stage + gq * PITCH + c, v0 * post_scale, v1 * post_scale);
    Tile<T>::store_pair(stage + (gq + 8) * PITCH + c, v2 * post_scale, v3 * post_scale);
  }
  __syncwarp();
  constexpr int kPer = 16 / (int)sizeof(T), chunks = DP / kPer;  // compile-time, so the row / column split below is shifts
#pragma unroll
  for (int i0 = 0; i0 < 16 * chunks; i0 += 32) {
    const int i = i0 + lane;
    const int r = i / chunks, c = (i - r * chunks) * kPer;
    T* dst = (i < 16 * chunks && c < D) ? row_ptr(r) : nullptr;
    if (dst != nullptr) *reinterpret_cast<uint4*>(dst + c) = *reinterpret_cast<const uint4*>(stage + r * PITCH + c);
  }
}

template <typename T>
constexpr int kF = (int)(sizeof(float) / sizeof(T));  // elements of T in a float
template <typename T, int DP>
struct RowPieces { static constexpr int n = DP * (int)sizeof(T) / 16; };

// Row softmax of the logits s[l, m] = round(<q, al>) - cl[m] held as accumulator fragments.
template <typename T, int KP>
__device__ __forceinline__ void column_softmax_tail(float (&s)[KP / 8][4], const float* nbias, int lane) {
  const int t = lane & 3;
  float mx_lo = -INFINITY, mx_hi = -INFINITY;
#pragma unroll
  for (int nt = 0; nt < KP / 8; ++nt) {
    const float2 bb = *reinterpret_cast<const float2*>(nbias + nt * 8 + 2 * t);  // 8-byte aligned: 2t is even
    const float b0 = bb.x, b1 = bb.y;  // -cl[m], or -inf beyond M
    s[nt][0] = round_through<T>(s[nt][0]) + b0;
    s[nt][1] = round_through<T>(s[nt][1]) + b1;
    s[nt][2] = round_through<T>(s[nt][2]) + b0;
    s[nt][3] = round_through<T>(s[nt][3]) + b1;
    mx_lo = fmaxf(mx_lo, fmaxf(s[nt][0], s[nt][1]));
    mx_hi = fmaxf(mx_hi, fmaxf(s[nt][2], s[nt][3]));
  }
  mx_lo = quad_max(mx_lo);
  mx_hi = quad_max(mx_hi);
  float sum_lo = 0.f, sum_hi = 0.f;
#pragma unroll
  for (int nt = 0; nt < KP / 8; ++nt) {
    s[nt][0] = exp_of<T>(s[nt][0] - mx_lo);
    s[nt][1] = exp_of<T>(s[nt][1] - mx_lo);
    s[nt][2] = exp_of<T>(s[nt][2] - mx_hi);
    s[nt][3] = exp_of<T>(s[nt][3] - mx_hi);
    sum_lo += s[nt][0] + s[nt][1];
    sum_hi += s[nt][2] + s[nt][3];
  }
  const float inv_lo = 1.0f / quad_sum(sum_lo), inv_hi = 1.0f / quad_sum(sum_hi);
#pragma unroll
  for (int nt = 0; nt < KP / 8; ++nt) {
    s[nt][0] *= inv_lo; s[nt][1] *= inv_lo; s[nt][2] *= inv_hi; s[nt][3] *= inv_hi;
  }
}

// ---------------------------------------------------------------------------------------------------
// Logits of the left-factor and output stages for one warp: rows l of column j against all m,
// w[l,m] = <q[l,j], al[j,m]> - cl[j,m], softmax over m.  Returns the normalised probabilities in s.
// ---------------------------------------------------------------------------------------------------
template <typename T, int KP, int DP, int PITCH>
__device__ __forceinline__ void column_softmax(float (&s)[KP / 8][4], const T* sQw, const T* sAL, const float* nbias,
                                               int lane) {
  warp_gemm_abt<T, KP, DP, PITCH>(s, sQw, sAL, lane);
  column_softmax_tail<T, KP>(s, nbias, lane);
}

}  // namespace
}  // namespace ma
