// Backward pass: gradients of the forward pass with respect to q, k and v.
//
// The stages are those of the forward pass in reverse order, each on the same tiles: output (column j), right-factor
// with V (block m), then for every earlier iteration left-factor (column j) and right-factor (block m).  The stage
// inputs (ar, cr, al, cl of every iteration, y) are recomputed by the forward stage kernels into the workspace, the
// factors are recomputed tile by tile from them and never stored.  Notation as in the forward kernels: R[j, i] and
// L[l, m] are the right and left factor, X and W their logits.
//   output:        dL = dz y^T,                dy = L^T dz,   dW = L o (dL - rowsum(L o dL)),
//                  dal = dW^T q,  dq = dW al,  dcl = -colsum(dW)
//   left-factor:   dL = dcr + q dar^T (valid queries only),   dW as above,
//                  dal = dW^T q,  dq += L dar + dW al,  dcl = -colsum(dW)
//   right-factor:  dR = s dal k^T + dcl (ln R + 1) [+ dy v^T], dX = R o (dR - rowsum(R o dR)),  c = s / (cr + eps),
//                  dar = c dX k,  dk += s R^T dal + (c dX)^T ar,  [dv = R^T dy],  dcr = -rowsum(dX o X) / (cr + eps)
//   the first right-factor stage has ar = q and cr = 1: dq += dar.
//
// One CTA per tile, one warp per 16 rows, as in the forward kernels: a first phase works on rows (factor, logit
// gradient, and the contraction over keys straight from registers) and leaves the factor and the logit gradient in
// shared memory in the storage type, a second phase contracts them over the rows with the operands read transposed.
// dq and dk collect contributions of several stages in fp32; every element has exactly one writer per stage, so the
// sums need no atomics and come out the same on every run.
//
// What bounds it: at 4 x 12 heads of 1024 tokens and three iterations each of the launches is 4-6 us of which the
// tensor work is under 1 us; the differentiable tensor operations this replaces were ~150 launches that wrote every
// factor and its gradients to memory in fp32.
#include <math.h>

#include <string>

#include "ma_warp_common.cuh"

namespace ma {
namespace {

struct BackwardArgs {
  Geometry g;            // q, k, v and the stage's ar, cr, al, cl, y
  View4 dz, dq, dk, dv;  // user tensors; dq / dk / dv may have a null pointer (not wanted)
  void *dal, *dy, *dar;  // (EH, B, M, D), (EH, B, M, D), (EH, M, B, D), storage type
  float *dcl, *dcr;      // (EH, B, M), (EH, M, B)
  float *dq_acc, *dk_acc;  // (EH, B, M, D) and (EH, M, B, D): the tiles that add to them own consecutive rows
  int first;             // right-factor: first iteration (ar = q, cr = 1)
  int accumulate;        // right-factor: dk_acc holds the later iterations' sum
};

// acc[16 x DP] += A^T[16 x rows] * Bm[rows x DP]; sA points at the warp's 16 columns of a [rows][pitch_a] tile.
template <typename T, int DP, int PITCH>
__device__ __forceinline__ void warp_gemm_atb(float (&o)[DP / 8][4], const T* sA, int pitch_a, const T* sB, int rows16,
                                              int lane) {
  for (int lt = 0; lt < rows16; ++lt) {
    typename Tile<T>::A a;
    Tile<T>::load_a_t(a, sA + lt * 16 * pitch_a, pitch_a, lane);
#pragma unroll
    for (int np = 0; np < DP / 16; ++np) {
      typename Tile<T>::B b;
      Tile<T>::load_b_kn(b, sB + lt * 16 * PITCH + np * 16, PITCH, lane);
      Tile<T>::mma(o[2 * np], o[2 * np + 1], a, b);
    }
  }
}

template <typename T, int KP, int DP, int PITCH>
__device__ __forceinline__ void warp_gemm_pv_add(float (&o)[DP / 8][4], const Factor<T, KP>& p, const T* sV, int lane) {
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

// Asks for the 16 fp32 rows a warp will add to much later (each lane for half a row or less), so that the addition does
// not wait for memory: the kernels are bound by such waits, not by bandwidth or arithmetic.
template <typename RowFn>
__device__ __forceinline__ void prefetch_rows_f32(RowFn row_ptr, int D, int lane) {
  const float* p = row_ptr(lane >> 1);
  if (p == nullptr) return;
  for (int c = (lane & 1) * 32; c < D; c += 64) asm volatile("prefetch.global.L1 [%0];" ::"l"(p + c));
}

template <int DP>
__device__ __forceinline__ void zero_acc(float (&o)[DP / 8][4]) {
#pragma unroll
  for (int nt = 0; nt < DP / 8; ++nt) o[nt][0] = o[nt][1] = o[nt][2] = o[nt][3] = 0.f;
}

// Rows of a fp32 accumulator array as fragments.  All loads are asked for before the first one is used: addition by addition, with
// the stores between them, each waited for memory by itself: forward and backward of 4 x 12 heads of 1024 x 64, three iterations, 197 ->
// 172 us (the kernels that add, 21-24 -> 15-17); 2 x 12 of 4096 411 -> 361; 8 x 16 of 256 x 72 in fp32 291 -> 250.
template <int DP>
struct RowsF32 {
  float2 v[2][DP / 8];
  template <typename RowFn>
  __device__ __forceinline__ void load(RowFn row_ptr, int D, int lane) {
    const int gq = lane >> 2, t = lane & 3;
#pragma unroll
    for (int half = 0; half < 2; ++half) {
      const float* p = row_ptr(gq + 8 * half);
#pragma unroll
      for (int nt = 0; nt < DP / 8; ++nt) {
        const int c = nt * 8 + 2 * t;
        v[half][nt] = p != nullptr && c < D ? *reinterpret_cast<const float2*>(p + c) : make_float2(0.f, 0.f);
      }
    }
  }
  __device__ __forceinline__ void add_to(float (&o)[DP / 8][4]) const {
#pragma unroll
    for (int nt = 0; nt < DP / 8; ++nt) {
      o[nt][0] += v[0][nt].x; o[nt][1] += v[0][nt].y;
      o[nt][2] += v[1][nt].x; o[nt][3] += v[1][nt].y;
    }
  }
};
template <int DP, typename RowFn>
__device__ __forceinline__ void store_rows_f32(const float (&o)[DP / 8][4], RowFn row_ptr, int D, int lane) {
  const int gq = lane >> 2, t = lane & 3;
#pragma unroll
  for (int half = 0; half < 2; ++half) {
    float* p = row_ptr(gq + 8 * half);
    if (p == nullptr) continue;
#pragma unroll
    for (int nt = 0; nt < DP / 8; ++nt) {
      const int c = nt * 8 + 2 * t;
      if (c < D) *reinterpret_cast<float2*>(p + c) = make_float2(o[nt][2 * half], o[nt][2 * half + 1]);
    }
  }
}
// o += rows of a fp32 array.
template <int DP, typename RowFn>
__device__ __forceinline__ void add_rows_f32(float (&o)[DP / 8][4], RowFn row_ptr, int D, int lane) {
  RowsF32<DP> rows;
  rows.load(row_ptr, D, lane);
  rows.add_to(o);
}
// add: memory += o, else memory = o.
template <int DP, typename RowFn>
__device__ __forceinline__ void update_rows_f32(float (&o)[DP / 8][4], RowFn row_ptr, int D, int lane, bool add) {
  if (add) add_rows_f32<DP>(o, row_ptr, D, lane);
  store_rows_f32<DP>(o, row_ptr, D, lane);
}

template <typename T>
__device__ __forceinline__ T* user_row_or_null(const View4& t, const Geometry& g, int e, int h, int p) {
  const int n = p - g.pad_off;
  if (t.ptr == nullptr || n < 0 || n >= g.N) return nullptr;
  return reinterpret_cast<T*>(const_cast<void*>(t.ptr)) + (long long)e * t.se + (long long)h * t.sh + (long long)n * t.sn;
}

// ---------------------------------------------------------------------------------------------------
// Output stage (OUT) or left-factor stage, column j.  grid = (B, E*H), one warp per 16 rows l.
// ---------------------------------------------------------------------------------------------------
template <typename T, int KP, int DP>
constexpr size_t column_elems(bool out, int RP) {
  return (size_t)(RP + 2 * KP + (out ? RP : 0)) * (DP + 8) + (size_t)RP * (KP + 8) * (out ? 2 : 1) +
         (size_t)kF<T> * (2 * KP + KP * (RP / 16));
}

template <typename T, int KP, int DP, bool OUT>
__global__ void __launch_bounds__(2 * KP) backward_column_kernel(const BackwardArgs a) {
  constexpr int PITCH = DP + 8, PP = KP + 8;
  stage_begin();
  extern __shared__ __align__(16) uint8_t smem[];
  const Geometry& g = a.g;
  const int eh = blockIdx.y, e = eh / g.H, h = eh - e * g.H, j = blockIdx.x;
  const int B = g.B, M = g.M, D = g.D, tid = threadIdx.x, nth = blockDim.x, RP = nth >> 1;  // 16 rows per warp
  T* sQ = reinterpret_cast<T*>(smem);
  T* sAL = sQ + RP * PITCH;
  T* sX = sAL + KP * PITCH;                       // y[j] or dar[:, j]
  T* sDZ = sX + KP * PITCH;                       // OUT only
  T* sW = sDZ + (OUT ? RP * PITCH : 0);           // [RP][PP] gradient of the logits
  T* sP = sW + RP * PP;                           // [RP][PP] factor (OUT only)
  float* nbias = reinterpret_cast<float*>(sP + (OUT ? RP * PP : 0));
  float* dcrs = nbias + KP;
  float* cpart = dcrs + KP;                       // [warps][KP]

  const T* qh = head_base<T>(g.q, e, h);
  load_rows<T, RowPieces<T, DP>::n>(sQ, PITCH, M, RP, D, qh, j - g.pad_off, B, g.N, g.q.sn, tid, nth, g.q.ptr);
  const long long col = ((long long)eh * B + j) * M;
  load_rows<T, RowPieces<T, DP>::n>(sAL, PITCH, M, KP, D, reinterpret_cast<const T*>(g.al) + col * D, 0, 1, M, D, tid, nth, g.q.ptr);
  if (OUT) {
    load_rows<T, RowPieces<T, DP>::n>(sX, PITCH, M, KP, D, reinterpret_cast<const T*>(g.y) + col * D, 0, 1, M, D, tid, nth, g.q.ptr);
    load_rows<T, RowPieces<T, DP>::n>(sDZ, PITCH, M, RP, D, head_base<T>(a.dz, e, h), j - g.pad_off, B, g.N, a.dz.sn, tid, nth, g.q.ptr);
  } else {
    load_rows<T, RowPieces<T, DP>::n>(sX, PITCH, M, KP, D, reinterpret_cast<const T*>(a.dar) + (long long)eh * M * B * D, j, B, M * B, D,
                                      tid, nth, g.q.ptr);
  }
  const int warp = tid >> 5, lane = tid & 31, gq = lane >> 2, t = lane & 3, row0 = warp * 16;
  const int l_lo = row0 + gq, l_hi = l_lo + 8;
  float ok_lo = 1.f, ok_hi = 1.f;
  auto dq_row = [&](int r) -> float* {
    const int l = row0 + r;
    return l < M ? a.dq_acc + (((long long)eh * B + j) * M + l) * D : nullptr;
  };
  if (!OUT) {
    ok_lo = pos_valid(g, e, l_lo * B + j) ? 1.f : 0.f;
    ok_hi = pos_valid(g, e, l_hi * B + j) ? 1.f : 0.f;
    prefetch_rows_f32(dq_row, D, lane);
  }
  for (int i = tid; i < KP; i += nth) {
    nbias[i] = i < M ? -g.cl[col + i] : -INFINITY;
    if (!OUT) dcrs[i] = i < M ? a.dcr[((long long)eh * M + i) * B + j] : 0.f;
  }
  tiles_commit_and_wait();
  __syncthreads();

  {
    float s[KP / 8][4], d[KP / 8][4];
    column_softmax<T, KP, DP, PITCH>(s, sQ + row0 * PITCH, sAL, nbias, lane);
    warp_gemm_abt<T, KP, DP, PITCH>(d, (OUT ? sDZ : sQ) + row0 * PITCH, sX, lane);
    float de_lo = 0.f, de_hi = 0.f;
#pragma unroll
    for (int nt = 0; nt < KP / 8; ++nt) {
      if (!OUT) {
        const float2 c = *reinterpret_cast<const float2*>(dcrs + nt * 8 + 2 * t);
        d[nt][0] = (d[nt][0] + c.x) * ok_lo; d[nt][1] = (d[nt][1] + c.y) * ok_lo;
        d[nt][2] = (d[nt][2] + c.x) * ok_hi; d[nt][3] = (d[nt][3] + c.y) * ok_hi;
      }
      de_lo = fmaf(s[nt][0], d[nt][0], fmaf(s[nt][1], d[nt][1], de_lo));
      de_hi = fmaf(s[nt][2], d[nt][2], fmaf(s[nt][3], d[nt][3], de_hi));
    }
    de_lo = quad_sum(de_lo);
    de_hi = quad_sum(de_hi);
    float cs[KP / 4];
#pragma unroll
    for (int nt = 0; nt < KP / 8; ++nt) {
      const int c = nt * 8 + 2 * t;
      d[nt][0] = s[nt][0] * (d[nt][0] - de_lo); d[nt][1] = s[nt][1] * (d[nt][1] - de_lo);
      d[nt][2] = s[nt][2] * (d[nt][2] - de_hi); d[nt][3] = s[nt][3] * (d[nt][3] - de_hi);
      Tile<T>::store_pair(sW + l_lo * PP + c, d[nt][0], d[nt][1]);
      Tile<T>::store_pair(sW + l_hi * PP + c, d[nt][2], d[nt][3]);
      if (OUT) {
        Tile<T>::store_pair(sP + l_lo * PP + c, s[nt][0], s[nt][1]);
        Tile<T>::store_pair(sP + l_hi * PP + c, s[nt][2], s[nt][3]);
      } else {
        s[nt][0] *= ok_lo; s[nt][1] *= ok_lo; s[nt][2] *= ok_hi; s[nt][3] *= ok_hi;
      }
      cs[2 * nt] = d[nt][0] + d[nt][2];
      cs[2 * nt + 1] = d[nt][1] + d[nt][3];
    }
    const int base = reduce_rows<KP / 4>(cs, lane);
#pragma unroll
    for (int i = 0; i < (KP / 32 > 0 ? KP / 32 : 1); ++i) {
      const int x = base + i;
      cpart[warp * KP + (x >> 1) * 8 + 2 * t + (x & 1)] = cs[i];
    }
    float o[DP / 8][4];
    zero_acc<DP>(o);
    if (!OUT) {
      Factor<T, KP> f;
      f.set(s);
      warp_gemm_pv_add<T, KP, DP, PITCH>(o, f, sX, lane);
    }
    Factor<T, KP> f;
    f.set(d);
    warp_gemm_pv_add<T, KP, DP, PITCH>(o, f, sAL, lane);
    update_rows_f32<DP>(o, dq_row, D, lane, !OUT);
  }
  __syncthreads();

  // rows m of this warp: dal = dW^T q, dy = L^T dz (staging in the al tile, which nothing reads any more)
  {
    float o[DP / 8][4];
    zero_acc<DP>(o);
    warp_gemm_atb<T, DP, PITCH>(o, sW + row0, PP, sQ, RP / 16, lane);
    T* dal = reinterpret_cast<T*>(a.dal) + col * D;
    store_rows<T, DP, PITCH>(o, sAL + row0 * PITCH, [&](int r) -> T* { return row0 + r < M ? dal + (long long)(row0 + r) * D : nullptr; },
                             D, lane, 1.0f, false);
  }
  if (OUT) {
    float o[DP / 8][4];
    zero_acc<DP>(o);
    warp_gemm_atb<T, DP, PITCH>(o, sP + row0, PP, sDZ, RP / 16, lane);
    T* dy = reinterpret_cast<T*>(a.dy) + col * D;
    store_rows<T, DP, PITCH>(o, sAL + row0 * PITCH, [&](int r) -> T* { return row0 + r < M ? dy + (long long)(row0 + r) * D : nullptr; },
                             D, lane, 1.0f, false);
  }
  for (int m = tid; m < M; m += nth) {
    float acc = 0.f;
    for (int w = 0; w < RP / 16; ++w) acc += cpart[w * KP + m];
    a.dcl[col + m] = -acc;
  }
}

// ---------------------------------------------------------------------------------------------------
// Right-factor stage, block m.  grid = (M, E*H), one warp per 16 rows j.
// ---------------------------------------------------------------------------------------------------
template <typename T, int KP, int DP>
constexpr size_t right_elems(bool with_v, int RP) {
  return (size_t)(2 * RP + KP + (with_v ? KP + RP : 0)) * (DP + 8) + (size_t)2 * RP * (KP + 8) + (size_t)kF<T> * KP;
}

// CTAs per SM that the 16-bit instances for up to 32 keys (the fine-tuning shapes) are compiled for: without V ten, at 96
// registers; with V seven, which is what shared memory holds at width 64 (28.3 KB each), so that no register is given up for more.
// 8 x 16 heads of 1024 tokens at width 72, two iterations: 334.7 us with ten for both kinds (the instances with V then
// spill at widths above 64), 332.2 left to the compiler, 331.4 as it is; 4 x 12 heads at width 64, three iterations: 193.0, 193.7, 192.0.
// The fp32 instances for up to 64 keys take all 255 registers and spill (264 bytes a thread at width 64, 736 with V; 864 and
// 1240 at width 80): the logit and factor rows of a warp alone are 2 x 32 registers, their split halves as many again.  They are
// still worth having: forward and backward of 2 x 12 heads of 4096 tokens, two iterations, 973 us against 3425 by tensor
// operations at width 64, 1506 against 4009 at width 80.
constexpr int right_ctas(int element_bytes, int KP, bool with_v) { return KP == 32 && element_bytes == 2 ? (with_v ? 7 : 10) : 1; }

template <typename T, int KP, int DP, bool WITH_V>
__global__ void __launch_bounds__(2 * KP, right_ctas(sizeof(T), KP, WITH_V)) backward_right_kernel(const BackwardArgs a) {
  constexpr int PITCH = DP + 8, PP = KP + 8;
  if (!a.first) dependents_may_start();
  grid_wait();
  extern __shared__ __align__(16) uint8_t smem[];
  const Geometry& g = a.g;
  const int eh = blockIdx.y, e = eh / g.H, h = eh - e * g.H, m = blockIdx.x;
  const int B = g.B, M = g.M, D = g.D, tid = threadIdx.x, nth = blockDim.x, RP = nth >> 1;
  T* sA = reinterpret_cast<T*>(smem);
  T* sDAL = sA + RP * PITCH;
  T* sK = sDAL + RP * PITCH;
  T* sV = sK + KP * PITCH;                        // WITH_V only, as sDY
  T* sDY = sV + (WITH_V ? KP * PITCH : 0);
  T* sP = sDY + (WITH_V ? RP * PITCH : 0);        // [RP][PP] factor
  T* sG = sP + RP * PP;                           // [RP][PP] c * gradient of the logits
  float* kbias = reinterpret_cast<float*>(sG + RP * PP);

  const long long blk = ((long long)eh * M + m) * B;  // row of (m, 0) in the (EH, M, B) arrays
  if (a.first)
    load_rows<T, RowPieces<T, DP>::n>(sA, PITCH, B, RP, D, head_base<T>(g.q, e, h), m * B - g.pad_off, 1, g.N, g.q.sn, tid, nth, g.q.ptr);
  else
    load_rows<T, RowPieces<T, DP>::n>(sA, PITCH, B, RP, D, reinterpret_cast<const T*>(g.ar) + blk * D, 0, 1, B, D, tid, nth, g.q.ptr);
  load_rows<T, RowPieces<T, DP>::n>(sK, PITCH, B, KP, D, head_base<T>(g.k, e, h), m * B - g.pad_off, 1, g.N, g.k.sn, tid, nth, g.q.ptr);
  const long long st = (long long)eh * B * M;       // (EH, B, M) arrays: row (j, m) is st + j*M + m
  load_rows<T, RowPieces<T, DP>::n>(sDAL, PITCH, B, RP, D, reinterpret_cast<const T*>(a.dal) + (st + m) * D, 0, 1, B, (long long)M * D,
                                    tid, nth, g.q.ptr);
  if (WITH_V) {
    load_rows<T, RowPieces<T, DP>::n>(sV, PITCH, B, KP, D, head_base<T>(g.v, e, h), m * B - g.pad_off, 1, g.N, g.v.sn, tid, nth, g.q.ptr);
    load_rows<T, RowPieces<T, DP>::n>(sDY, PITCH, B, RP, D, reinterpret_cast<const T*>(a.dy) + (st + m) * D, 0, 1, B, (long long)M * D,
                                      tid, nth, g.q.ptr);
  }
  const int warp = tid >> 5, lane = tid & 31, gq = lane >> 2, t = lane & 3, row0 = warp * 16;
  const int r_lo = row0 + gq, r_hi = r_lo + 8;
  const float cr_lo = (a.first || r_lo >= B ? 1.0f : g.cr[blk + r_lo]) + kEps;
  const float cr_hi = (a.first || r_hi >= B ? 1.0f : g.cr[blk + r_hi]) + kEps;
  const float dcl_lo = r_lo < B ? a.dcl[st + (long long)r_lo * M + m] : 0.f;
  const float dcl_hi = r_hi < B ? a.dcl[st + (long long)r_hi * M + m] : 0.f;
  auto dq_row = [&](int r) -> float* { return row0 + r < B ? a.dq_acc + (st + (long long)(row0 + r) * M + m) * D : nullptr; };
  auto dk_row = [&](int r) -> float* { return row0 + r < B ? a.dk_acc + (blk + row0 + r) * D : nullptr; };
  if (a.first) prefetch_rows_f32(dq_row, D, lane);
  if (a.accumulate) prefetch_rows_f32(dk_row, D, lane);
  for (int i = tid; i < KP; i += nth) kbias[i] = (i < B && pos_valid(g, e, m * B + i)) ? 0.f : -INFINITY;
  tiles_commit_and_wait();
  __syncthreads();

  float row_grad[DP / 8][4];  // dar, or dq of the first stage: stored after the next barrier, from where the key tile was
  {
    float s[KP / 8][4], d[KP / 8][4];
    warp_gemm_abt<T, KP, DP, PITCH>(d, sDAL + row0 * PITCH, sK, lane);
#pragma unroll
    for (int nt = 0; nt < KP / 8; ++nt) {
      d[nt][0] *= g.sm_scale; d[nt][1] *= g.sm_scale; d[nt][2] *= g.sm_scale; d[nt][3] *= g.sm_scale;
    }
    if (WITH_V) {
      warp_gemm_abt<T, KP, DP, PITCH>(s, sDY + row0 * PITCH, sV, lane);
#pragma unroll
      for (int nt = 0; nt < KP / 8; ++nt) {
        d[nt][0] += s[nt][0]; d[nt][1] += s[nt][1]; d[nt][2] += s[nt][2]; d[nt][3] += s[nt][3];
      }
    }
    warp_gemm_abt<T, KP, DP, PITCH>(s, sA + row0 * PITCH, sK, lane);
    const float c_lo = g.sm_scale / cr_lo, c_hi = g.sm_scale / cr_hi;
    float mx_lo = -INFINITY, mx_hi = -INFINITY;
#pragma unroll
    for (int nt = 0; nt < KP / 8; ++nt) {
      const float2 bb = *reinterpret_cast<const float2*>(kbias + nt * 8 + 2 * t);
      s[nt][0] = fmaf(round_through<T>(s[nt][0]), c_lo, bb.x);
      s[nt][1] = fmaf(round_through<T>(s[nt][1]), c_lo, bb.y);
      s[nt][2] = fmaf(round_through<T>(s[nt][2]), c_hi, bb.x);
      s[nt][3] = fmaf(round_through<T>(s[nt][3]), c_hi, bb.y);
      mx_lo = fmaxf(mx_lo, fmaxf(s[nt][0], s[nt][1]));
      mx_hi = fmaxf(mx_hi, fmaxf(s[nt][2], s[nt][3]));
    }
    mx_lo = fmaxf(quad_max(mx_lo), kEps);  // lower clamp on the row maximum, as in the forward pass
    mx_hi = fmaxf(quad_max(mx_hi), kEps);
    // e = exp(t), t = X - max; d becomes dR without its row constant dcl (1 - ln(sum)); sums for the row quantities
    float S_lo = 0.f, S_hi = 0.f, Sd_lo = 0.f, Sd_hi = 0.f, St_lo = 0.f, St_hi = 0.f, Sdt_lo = 0.f, Sdt_hi = 0.f;
#pragma unroll
    for (int nt = 0; nt < KP / 8; ++nt) {
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const float tt = fmaxf(s[nt][i] - (i < 2 ? mx_lo : mx_hi), -1e4f);  // exp is 0 there, and products stay finite
        const float ex = exp_of<T>(tt);
        const float dd = fmaf(i < 2 ? dcl_lo : dcl_hi, tt, d[nt][i]);
        s[nt][i] = ex;
        d[nt][i] = dd;
        const float ed = ex * dd;
        if (i < 2) { S_lo += ex; St_lo = fmaf(ex, tt, St_lo); Sd_lo += ed; Sdt_lo = fmaf(ed, tt, Sdt_lo); }
        else { S_hi += ex; St_hi = fmaf(ex, tt, St_hi); Sd_hi += ed; Sdt_hi = fmaf(ed, tt, Sdt_hi); }
      }
    }
    S_lo = quad_sum(S_lo); S_hi = quad_sum(S_hi); Sd_lo = quad_sum(Sd_lo); Sd_hi = quad_sum(Sd_hi);
    St_lo = quad_sum(St_lo); St_hi = quad_sum(St_hi); Sdt_lo = quad_sum(Sdt_lo); Sdt_hi = quad_sum(Sdt_hi);
    const float i_lo = 1.0f / (S_lo + kEps), i_hi = 1.0f / (S_hi + kEps);
    const float k_lo = dcl_lo * (1.f - log_of<T>(S_lo + kEps)), k_hi = dcl_hi * (1.f - log_of<T>(S_hi + kEps));
    const float de_lo = i_lo * fmaf(k_lo, S_lo, Sd_lo), de_hi = i_hi * fmaf(k_hi, S_hi, Sd_hi);  // rowsum(R o dR)
    if (!a.first && t == 0) {
      // rowsum(dX o X) with X = t + max: sum R dR t - de sum R t + max de (1 - sum R)
      const float x_lo = i_lo * (fmaf(k_lo, St_lo, Sdt_lo) - de_lo * St_lo) + mx_lo * de_lo * (1.f - S_lo * i_lo);
      const float x_hi = i_hi * (fmaf(k_hi, St_hi, Sdt_hi) - de_hi * St_hi) + mx_hi * de_hi * (1.f - S_hi * i_hi);
      if (r_lo < B) a.dcr[blk + r_lo] = -x_lo / cr_lo;
      if (r_hi < B) a.dcr[blk + r_hi] = -x_hi / cr_hi;
    }
    const float o_lo = k_lo - de_lo, o_hi = k_hi - de_hi;
#pragma unroll
    for (int nt = 0; nt < KP / 8; ++nt) {
      const int c = nt * 8 + 2 * t;
      s[nt][0] *= i_lo; s[nt][1] *= i_lo; s[nt][2] *= i_hi; s[nt][3] *= i_hi;
      d[nt][0] = c_lo * (s[nt][0] * (d[nt][0] + o_lo)); d[nt][1] = c_lo * (s[nt][1] * (d[nt][1] + o_lo));
      d[nt][2] = c_hi * (s[nt][2] * (d[nt][2] + o_hi)); d[nt][3] = c_hi * (s[nt][3] * (d[nt][3] + o_hi));
      Tile<T>::store_pair(sP + r_lo * PP + c, s[nt][0], s[nt][1]);
      Tile<T>::store_pair(sP + r_hi * PP + c, s[nt][2], s[nt][3]);
      Tile<T>::store_pair(sG + r_lo * PP + c, d[nt][0], d[nt][1]);
      Tile<T>::store_pair(sG + r_hi * PP + c, d[nt][2], d[nt][3]);
    }
    zero_acc<DP>(row_grad);
    Factor<T, KP> f;
    f.set(d);
    warp_gemm_pv_add<T, KP, DP, PITCH>(row_grad, f, sK, lane);
  }
  __syncthreads();

  T* stage = sK + row0 * PITCH;  // (the key tile has been read)
  if (a.first) {
    add_rows_f32<DP>(row_grad, dq_row, D, lane);
    store_rows<T, DP, PITCH>(row_grad, stage, [&](int r) -> T* {
      return row0 + r < B ? user_row_or_null<T>(a.dq, g, e, h, m * B + row0 + r) : nullptr;
    }, D, lane, 1.0f, false);
  } else {
    T* dar = reinterpret_cast<T*>(a.dar) + blk * D;
    store_rows<T, DP, PITCH>(row_grad, stage, [&](int r) -> T* { return row0 + r < B ? dar + (long long)(row0 + r) * D : nullptr; }, D,
                             lane, 1.0f, false);
  }

  // keys i of this warp
  {
    float o[DP / 8][4];
    zero_acc<DP>(o);
    warp_gemm_atb<T, DP, PITCH>(o, sP + row0, PP, sDAL, RP / 16, lane);
#pragma unroll
    for (int nt = 0; nt < DP / 8; ++nt) {
      o[nt][0] *= g.sm_scale; o[nt][1] *= g.sm_scale; o[nt][2] *= g.sm_scale; o[nt][3] *= g.sm_scale;
    }
    warp_gemm_atb<T, DP, PITCH>(o, sG + row0, PP, sA, RP / 16, lane);
    if (a.first) {
      if (a.accumulate) add_rows_f32<DP>(o, dk_row, D, lane);
      store_rows<T, DP, PITCH>(o, stage, [&](int r) -> T* {
        return row0 + r < B ? user_row_or_null<T>(a.dk, g, e, h, m * B + row0 + r) : nullptr;
      }, D, lane, 1.0f, false);
    } else {
      update_rows_f32<DP>(o, dk_row, D, lane, a.accumulate != 0);
    }
  }
  if (WITH_V) {
    float o[DP / 8][4];
    zero_acc<DP>(o);
    warp_gemm_atb<T, DP, PITCH>(o, sP + row0, PP, sDY, RP / 16, lane);
    store_rows<T, DP, PITCH>(o, stage, [&](int r) -> T* {
      return row0 + r < B ? user_row_or_null<T>(a.dv, g, e, h, m * B + row0 + r) : nullptr;
    }, D, lane, 1.0f, false);
  }
}

enum BackwardStage { kBackOutput, kBackLeft, kBackRight, kBackRightWithV };

constexpr size_t kMaxSmem = 227 * 1024;

template <typename T, int KP, int DP>
size_t backward_smem(const Geometry& g, BackwardStage st) {
  const bool right = st == kBackRight || st == kBackRightWithV;
  const int RP = ((right ? g.B : g.M) + 15) & ~15;
  return (right ? right_elems<T, KP, DP>(st == kBackRightWithV, RP) : column_elems<T, KP, DP>(st == kBackOutput, RP)) * sizeof(T);
}

// g.E == 0: only the shared memory of the stage is wanted.
template <typename T, int KP, int DP>
cudaError_t backward_launch(const BackwardArgs& a, BackwardStage st, size_t* smem_out, cudaStream_t stream) {
  const Geometry& g = a.g;
  const bool right = st == kBackRight || st == kBackRightWithV;
  const size_t smem = backward_smem<T, KP, DP>(g, st);
  if (smem_out != nullptr) { *smem_out = smem; return cudaSuccess; }
  const void* fn = nullptr;
  switch (st) {
    case kBackOutput: fn = (const void*)backward_column_kernel<T, KP, DP, true>; break;
    case kBackLeft: fn = (const void*)backward_column_kernel<T, KP, DP, false>; break;
    case kBackRight: fn = (const void*)backward_right_kernel<T, KP, DP, false>; break;
    case kBackRightWithV: fn = (const void*)backward_right_kernel<T, KP, DP, true>; break;
  }
  if (const cudaError_t e = allow_dynamic_smem(fn, smem); e != cudaSuccess) return e;
  const int rows = right ? g.B : g.M;
  void* args[] = {(void*)&a};
  return launch_kernel(fn, dim3(right ? g.M : g.B, g.E * g.H), dim3(2 * ((rows + 15) & ~15)), args, smem, stream);
}

template <typename T, int KP>
cudaError_t backward_dp(const BackwardArgs& a, BackwardStage st, size_t* smem_out, cudaStream_t stream) {
  if (a.g.D <= 32) return backward_launch<T, KP, 32>(a, st, smem_out, stream);
  if (a.g.D <= 64) return backward_launch<T, KP, 64>(a, st, smem_out, stream);
  return backward_launch<T, KP, 80>(a, st, smem_out, stream);
}

template <typename T>
cudaError_t backward_kp(const BackwardArgs& a, BackwardStage st, size_t* smem_out, cudaStream_t stream) {
  const bool right = st == kBackRight || st == kBackRightWithV;
  const int keys = right ? a.g.B : a.g.M;
  if (keys <= 16) return backward_dp<T, 16>(a, st, smem_out, stream);
  if (keys <= 32) return backward_dp<T, 32>(a, st, smem_out, stream);
  if constexpr (sizeof(T) == 2) {
    if (keys > 64) return backward_dp<T, 128>(a, st, smem_out, stream);
  }
  return backward_dp<T, 64>(a, st, smem_out, stream);
}

cudaError_t backward_stage(const BackwardArgs& a, int dtype, BackwardStage st, size_t* smem_out, cudaStream_t stream) {
  if (dtype == MA_B200_BF16) return backward_kp<__nv_bfloat16>(a, st, smem_out, stream);
  if (dtype == MA_B200_F16) return backward_kp<__half>(a, st, smem_out, stream);
  return backward_kp<float>(a, st, smem_out, stream);
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
  for (int t = 0; t < T; ++t) {
    if ((e = launch_warp_stage(at_iteration(t, t), dtype, t == T - 1 ? kStageRightWithV : kStageRight, t == 0, stream)) != cudaSuccess)
      return e;
    if (t < T - 1)
      if ((e = launch_warp_stage(at_iteration(t + 1, t), dtype, kStageLeft, false, stream)) != cudaSuccess) return e;
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
