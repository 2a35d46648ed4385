// tcgen05 stage kernels for 16-bit tensors and D <= 64, one launch per stage: persistent CTAs, three per SM (two for 256 keys),
// each on one 128-row tile at a time with one thread per tile row and a control warp.  They take the calls whose block size
// or block count is above 128 (the instances for 64 and 128 keys: the other side of such a call); up to 128 on both sides
// all stages are one launch of ma_flow.inc.
//
// A tile is one key block m (or two, of up to 64 tokens) in the right-factor stages, one column j (or two) in the
// left-factor and output stages.  A CTA loads its operands by TMA, forms S = A B^T in tensor memory, turns it row by row
// into the factor P (16-bit, written over S), contracts P with an operand tile and stores the rows by TMA:
//   right-factor:  A = q or ar rows j, B = k rows i;  al = s P k,  y = P v      (reference: ma/ma_torch.py:10-23, :38-52)
//   output:        A = q rows l,       B = al rows m; z = P y                   (:55-62)
//   left-factor:   the contraction runs over the rows l of the factor, so P^T is needed.  S = q al^T only gives the row
//                  statistics lse[l]; then S' = al q^T is formed (the tensor pipe has time: 128 cycles) and
//                  P^T[m, l] = exp(S'[m, l] - cl[m] - lse[l]) comes out with its rows where the contraction wants
//                  them, and cr[m] is a sum along a thread's own row, before rounding, in fp32   (:26-35)
// A thread owns a whole row, so no statistics are exchanged, and everything a warp does is a plain instruction stream;
// the waits of one CTA (loads, tensor pipe, tensor memory) are covered by the other CTAs of the SM instead of by a
// pipeline of specialised warps.  What bounds it: at 256 keys the latency of the row passes, with eight row warps on an SM.  A
// right-factor tile of 128 x 256 takes its CTA 10600 cycles (16 heads of 65536 tokens: 8192 tiles on 296 places in 155 us; the
// stages of two iterations 155-157, 253, 183-186, 159), 5300 of the SM's per tile; the pipe of exponentials and conversions, 32
// lanes a clock, needs 2048, and the row passes alone take 2950 with eight warps on an SM.  (Tensor instructions behind a test of
// the lane's number instead of an elected lane: 163, 258, 196, 165.  Rows stored by their threads instead of by TMA took 1700
// cycles of that chain; launching the next stage early, by programmatic dependent launch, cost the running stage its instruction
// cache: 18000 cycles for the first tile instead of 9000.)
//
// Rounding points are the reference's: S is rounded to storage before the softmax, P is normalised in fp32 and then
// rounded.  Ragged ends, padding and masks: rows that do not exist are zero-filled by TMA (or by hand, where a column's
// last row would lie behind the end of the tensor), columns that do not exist get an exponent of -1e30.
#include "ma_tile_common.cuh"

namespace ma {
namespace {

struct TileMaps { CUtensorMap a, b, v, s0, s1; };  // operands, and where the rows (al or ar or z, and y) go

struct TileArgs {
  int tiles, total;  // tiles per head, and of all heads
  int first;         // right-factor: first iteration (A = q, cr = 1)
  int clear;         // this launch clears the status word
  int* host_status;  // mapped host word for a wait that gave up, or nullptr
};

// NK: key columns of a row's unit, rounded up: 64 (two units per tile), 128 or 256.
// Shared memory: a staging tile, operand slots A, B and V; the kinds without V have a second slot for the operand that is
// released last.
constexpr int tile_a_rows(int nk, StageKind kind) { return kind == kStageLeft && nk == 256 ? 256 : kRows; }
constexpr int tile_b_rows(int nk) { return nk == 256 ? 256 : kRows; }
constexpr int tile_ctas(int nk) { return nk == 256 ? 2 : 3; }  // CTAs per SM
constexpr bool tile_has_v(StageKind kind) { return kind == kStageRightWithV || kind == kStageOutput; }
constexpr int tile_slot_rows(int nk, StageKind kind) {
  return tile_a_rows(nk, kind) * (kind == kStageLeft && nk != 256 ? 2 : 1) + tile_b_rows(nk) * (kind == kStageLeft ? 1 : 2);
}
constexpr uint32_t kAuxBytes = (2 + 1) * 256 * 4 + 128;  // two column vectors, the row statistics of the left-factor stage, barriers
constexpr uint32_t tile_smem(int nk, StageKind kind) { return (kRows + tile_slot_rows(nk, kind)) * kRowBytes + kAuxBytes + 1024; }

struct Tile {
  int eh, e, h, u0, row_base;
};

// mbarriers of a CTA.  Every phase of one is waited for by all its waiters before the next can complete.
enum {
  kBarA = 0,     // [2] operand slot A filled (the second only where A alternates)
  kBarB = 2,     // [2] operand slot B filled
  kBarV = 4,     // operand slot V filled
  kBarS = 5,     // S in tensor memory
  kBarP = 6,     // S read and P written by the 128 row threads
  kBarO = 7,     // O in tensor memory
  kBarE = 8,     // O read and staged in shared memory by the 128 row threads
  kBarFree = 9,  // staging tile read by the store
  kBarDrain = 10,  // after a wait that gave up: the tensor pipe has finished
  kTileBars = 11
};
constexpr int kRowBarrier = 1;  // named barrier of the row threads
constexpr int kTileThreads = kRows + 32;

// HOLD: the self-test's instance, in which a CTA never asks for its first operand and soon gives up waiting for it (as a
// run-time switch it cost the timed instances 0.6 %: 16 heads of 50176 tokens 681 against 685 us).
template <typename T, int NK, StageKind KIND, bool HOLD>
__global__ void __launch_bounds__(kTileThreads, tile_ctas(NK))
    tile_kernel(const __grid_constant__ TileMaps maps, const Geometry g, const TileArgs args) {
  constexpr bool kRight = is_right(KIND), kHasV = tile_has_v(KIND), kLeft = KIND == kStageLeft;
  constexpr int kFmt = std::is_same<T, __nv_bfloat16>::value ? 1 : 0;
  constexpr int kUnits = NK == 64 ? 2 : 1;         // blocks (columns) per tile
  constexpr int kBRows = tile_b_rows(NK), kARows = tile_a_rows(NK, KIND);
  constexpr int kCols = NK == 64 ? 128 : NK;       // columns of S
  constexpr int kVec = kCols / kRows;              // entries of the column vector per thread
  constexpr uint32_t kTmemO = kCols / 2;           // P takes the first half of S's columns, O follows
  constexpr bool kSplitRows = NK == 256 && !kLeft;  // a unit's rows take two tiles
  constexpr int kChunks = NK == 256 && kLeft ? 2 : 1;  // left-factor: 128-row chunks of the rows l, and of the rows m
  constexpr bool kTwoA = kLeft && NK != 256, kTwoB = KIND == kStageRight;
  extern __shared__ uint8_t smem_raw[];
  const uint32_t stage = (smem_u32(smem_raw) + 1023u) & ~1023u;  // staging tile of the stores, then the operand slots
  uint8_t* base_ptr = smem_raw + (stage - smem_u32(smem_raw));
  const uint32_t slots = stage + kRows * kRowBytes;
  constexpr uint32_t kABytes = kARows * kRowBytes, kBBytes = kBRows * kRowBytes;
  constexpr uint32_t kOffAux = kRows * kRowBytes + tile_slot_rows(NK, KIND) * kRowBytes;
  auto slot_a = [&](int i) { return slots + (kTwoA && (i & 1) ? kABytes + kBBytes : 0u); };
  auto slot_b = [&](int i) { return slots + kABytes + (kTwoB && (i & 1) ? kBBytes : 0u); };
  const uint32_t slot_v = slots + kABytes + kBBytes;
  float* const vec = reinterpret_cast<float*>(base_ptr + kOffAux);  // [2][256] per key column, log2 units: 0 or -cl, kGone where there is none
  float* const lse = vec + 2 * 256;                                 // left-factor: per row l, log2 units
  const uint32_t bars = stage + kOffAux + 3 * 256 * 4;
  auto bar = [&](int b) { return bars + 8u * (uint32_t)b; };
  volatile int* abort_flag = reinterpret_cast<volatile int*>(base_ptr + kOffAux + 3 * 256 * 4 + 8 * kTileBars);
  volatile uint32_t* tmem_slot = reinterpret_cast<volatile uint32_t*>(base_ptr + kOffAux + 3 * 256 * 4 + 8 * kTileBars + 8);

  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int B = g.B, M = g.M, D = g.D;
  const int units = kRight ? M : B, keys = kRight ? B : M;     // units of the head; rows and columns of a unit
  const int nch = NK == 64 ? 2 : (keys + 31) >> 5;              // 32-column chunks that hold keys
  // Every token of the padded sequence is there and no chunk is partly empty: nothing to mask.
  const bool plain = g.mask == nullptr && g.N == M * B && keys == 32 * nch;
  const int whole = g.N / B;                                     // whole rows of B tokens (see column_start)
  const int my_tiles = args.total > (int)blockIdx.x ? (args.total - 1 - (int)blockIdx.x) / (int)gridDim.x + 1 : 0;
  auto tile_at = [&](int i) {
    const int t = (int)blockIdx.x + i * (int)gridDim.x;
    Tile w;
    w.eh = t / args.tiles;
    const int r = t - w.eh * args.tiles;
    w.e = w.eh / g.H;
    w.h = w.eh - w.e * g.H;
    w.u0 = kSplitRows ? r >> 1 : r * kUnits;
    w.row_base = kSplitRows ? (r & 1) * kRows : 0;
    return w;
  };
  // Column x (block size B, front padding pad): the row r of its tile is token r*B + jj, jj = x - pad, or where that is
  // negative jj = x - pad + B - the column's first row is padding then and is left out.  Tensor maps see the tokens as
  // whole rows of B; a token of the row behind the last whole one is handled by hand.
  auto column_start = [&](int x) { return x < g.pad_off ? x - g.pad_off + B : x - g.pad_off; };
  auto give_up = [&](int code) {
    *abort_flag = 1;
    if (atomicCAS(g.status, 0, code) == 0 && args.host_status != nullptr) {
      *reinterpret_cast<volatile int*>(args.host_status) = code;
      __threadfence_system();
    }
  };
  // Every wait is bounded, and one that gives up ends the others of the CTA.  The vote brings the lanes of a warp back
  // together (the tensor-memory instructions need that) and of one mind.
  auto wait = [&](int b, uint32_t phase) {
    const bool r = __all_sync(0xffffffffu, mbar_wait_abortable(bar(b), phase & 1u, abort_flag));
    if (!r) *abort_flag = 1;
    return r;
  };

  if (tid == 0) {
    for (int i = 0; i < kTileBars; ++i) mbar_init(bar(i), i == kBarP || i == kBarE ? kRows : 1);
    *abort_flag = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  grid_wait();
  if (args.clear && blockIdx.x == 0 && tid == 0) *g.status = 0;
  if (warp == 4) {
    __syncwarp();
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(stage + kOffAux + 3 * 256 * 4 + 8 * kTileBars + 8),
                 "r"(kCols)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = *tmem_slot;

  if (warp == 4) {
    // =========================== control warp: loads, tensor pipe, stores ====================================
    // (a unit past the end reads zeros)
    int la = 0, lb = 0, lv = 0;  // loads queued (lane 0)
    auto load_a = [&](int i) {
      if (lane != 0 || i >= my_tiles) return;
      la = i + 1;
      const Tile w = tile_at(i);
      const uint32_t b = bar(kBarA + (kTwoA ? i & 1 : 0));
      mbar_expect_tx(b, kABytes);
      for (int u = 0; u < kUnits; ++u) {
        const int x = w.u0 + u;
        const uint32_t dst = slot_a(i) + u * 64 * kRowBytes;
        if (!kRight) tma_load_5d(dst, &maps.a, b, 0, column_start(x), w.row_base, w.h, w.e);
        else if (args.first) tma_load_4d(dst, &maps.a, b, 0, x * B - g.pad_off + w.row_base, w.h, w.e);
        else tma_load_4d(dst, &maps.a, b, 0, x * B + w.row_base, w.eh, 0);
      }
    };
    auto load_b = [&](int i) {
      if (lane != 0 || i >= my_tiles) return;
      lb = i + 1;
      const Tile w = tile_at(i);
      const uint32_t b = bar(kBarB + (kTwoB ? i & 1 : 0));
      mbar_expect_tx(b, kBBytes);
      for (int u = 0; u < kUnits; ++u) {
        const int x = w.u0 + u;
        const uint32_t dst = slot_b(i) + u * 64 * kRowBytes;
        if (kRight) tma_load_4d(dst, &maps.b, b, 0, x * B - g.pad_off, w.h, w.e);
        else tma_load_4d(dst, &maps.b, b, 0, x * M, w.eh, 0);
      }
    };
    auto load_v = [&](int i) {
      if (!kHasV || lane != 0 || i >= my_tiles) return;
      lv = i + 1;
      const Tile w = tile_at(i);
      mbar_expect_tx(bar(kBarV), kBBytes);
      for (int u = 0; u < kUnits; ++u) {
        const int x = w.u0 + u;
        const uint32_t dst = slot_v + u * 64 * kRowBytes;
        if (kRight) tma_load_4d(dst, &maps.v, bar(kBarV), 0, x * B - g.pad_off, w.h, w.e);
        else tma_load_4d(dst, &maps.v, bar(kBarV), 0, x * M, w.eh, 0);
      }
    };
    // S = A B^T over the features, both K-major
    auto issue_abt = [&](uint32_t a, uint32_t b) {
      tc_fence_after();
      constexpr uint32_t idesc = instr_desc(kFmt, 0, 0, kCols, kRows);
      const uint32_t da = smem_desc_lo(a, 16), db = smem_desc_lo(b, 16);
      if (elect_one()) {
#pragma unroll
        for (int kk = 0; kk < 4; ++kk)
          if (16 * kk < D) mma_f16_lo(tmem, da + kk * 2, db + kk * 2, idesc, kk > 0);
        mma_commit(bar(kBarS));
      }
    };
    // O[128 x 64] = P X, P in tensor memory, X row-major [keys][64]
    auto issue_px = [&](uint32_t x) {
      tc_fence_after();
      constexpr uint32_t idesc = instr_desc(kFmt, 0, 1, 64, kRows);
      const uint32_t dx = smem_desc_lo(x, kRows * kRowBytes);
      const int steps = kUnits == 2 ? 8 : (keys + 15) >> 4;
      if (elect_one()) {
#pragma unroll
        for (int kk = 0; kk < kCols / 16; ++kk)
          if (kk < steps) mma_f16_ts(tmem + kTmemO, tmem + kk * 8, dx + kk * 128, idesc, kk > 0);
        mma_commit(bar(kBarO));
      }
    };
    // Staged rows of tile i to memory (rows past the end are clipped by the map); frees the staging tile.
    auto store = [&](const CUtensorMap* m, int i, int row0) {
      if (lane != 0) return;
      const Tile w = tile_at(i);
      for (int u = 0; u < kUnits; ++u) {
        const int x = w.u0 + u;
        if (x >= units) continue;
        const uint32_t src = stage + u * 64 * kRowBytes;
        if (KIND == kStageOutput) tma_store_5d(m, src, 0, column_start(x), w.row_base + row0, w.h, w.e);
        else tma_store_4d(m, src, 0, x, w.row_base + row0, w.eh);
      }
      asm volatile("cp.async.bulk.commit_group;" ::: "memory");
      asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory");
      mbar_arrive(bar(kBarFree));
    };

    if (!HOLD) load_a(0);
    load_b(0);
    load_v(0);
    if (kTwoA) load_a(1);
    if (kTwoB) load_b(1);
    uint32_t ns = 0, np = 0, no = 0, ne = 0;  // phases of S, P, O, E waited for
    bool ok = !HOLD || __all_sync(0xffffffffu, mbar_wait_abortable(bar(kBarA), 0, abort_flag, 4096));
    for (int i = 0; ok && i < my_tiles; ++i) {
      ok = wait(kBarA + (kTwoA ? i & 1 : 0), kTwoA ? i >> 1 : i) && wait(kBarB + (kTwoB ? i & 1 : 0), kTwoB ? i >> 1 : i);
      if (!ok) break;
      if (!kRight && g.N != whole * B) {  // the token of the row behind the last whole one (its place was zero-filled)
        const Tile w = tile_at(i);
        for (int u = 0; u < kUnits; ++u) {
          const int x = w.u0 + u, n = whole * B + column_start(x), r = whole - w.row_base;
          if (x < units && n < g.N && r >= 0 && r < (kUnits == 2 ? 64 : kARows) && lane < D / 8) {
            const T* src = reinterpret_cast<const T*>(g.q.ptr) + (long long)w.e * g.q.se + (long long)w.h * g.q.sh + (long long)n * g.q.sn;
            *reinterpret_cast<uint4*>(base_ptr + (slot_a(i) - stage) + swz(r + u * 64, lane)) = *reinterpret_cast<const uint4*>(src + lane * 8);
            fence_async_smem();
          }
        }
        __syncwarp();
      }
      issue_abt(slot_a(i), slot_b(i));
      if (i > 0) store(KIND == kStageRightWithV ? &maps.s1 : &maps.s0, i - 1, (kChunks - 1) * kRows);  // left over from the tile before
      if (kLeft) {
        for (int rc = 0; rc < kChunks && ok; ++rc) {  // statistics of the rows l
          if (rc > 0) issue_abt(slot_a(i) + rc * kRows * kRowBytes, slot_b(i));
          ok = wait(kBarS, ns++) && wait(kBarP, np++);
        }
        for (int mc = 0; mc < kChunks && ok; ++mc) {  // rows m
          issue_abt(slot_b(i) + mc * kRows * kRowBytes, slot_a(i));
          ok = wait(kBarS, ns++);
          if (ok && mc == kChunks - 1) load_b(i + 1);
          ok = ok && wait(kBarP, np++);
          if (!ok) break;
          issue_px(slot_a(i));
          ok = wait(kBarO, no++);
          if (ok && mc == kChunks - 1) load_a(kTwoA ? i + 2 : i + 1);
          ok = ok && wait(kBarE, ne++);
          if (ok && mc < kChunks - 1) store(&maps.s0, i, mc * kRows);
        }
        if (!ok) break;
      } else {
        ok = wait(kBarS, ns++);
        if (!ok) break;
        load_a(i + 1);
        if (KIND == kStageOutput) load_b(i + 1);
        ok = wait(kBarP, np++) && (KIND != kStageOutput || wait(kBarV, i));
        if (!ok) break;
        issue_px(KIND == kStageOutput ? slot_v : slot_b(i));
        ok = wait(kBarO, no++);
        if (!ok) break;
        if (KIND == kStageRight) load_b(i + 2);
        if (KIND == kStageRightWithV) load_b(i + 1);
        if (KIND == kStageOutput) load_v(i + 1);
        ok = wait(kBarE, ne++);
        if (KIND == kStageRightWithV && ok) {  // y takes the place of al
          ok = wait(kBarV, i);
          if (!ok) break;
          issue_px(slot_v);
          store(&maps.s0, i, 0);
          ok = wait(kBarO, no++);
          if (!ok) break;
          load_v(i + 1);
          ok = wait(kBarE, ne++);
        }
        if (!ok) break;
      }
    }
    if (!ok) {
      if (lane == 0) {
        give_up(701);
        // own copies have landed before the CTA leaves
        constexpr int na = kTwoA ? 2 : 1, nb = kTwoB ? 2 : 1;  // (one slot has one load in flight)
        for (int i = max(la - na, HOLD ? 1 : 0); i < la; ++i) (void)mbar_wait(bar(kBarA + (kTwoA ? i & 1 : 0)), (uint32_t)(kTwoA ? i >> 1 : i) & 1u);
        for (int i = max(lb - nb, 0); i < lb; ++i) (void)mbar_wait(bar(kBarB + (kTwoB ? i & 1 : 0)), (uint32_t)(kTwoB ? i >> 1 : i) & 1u);
        if (lv > 0) (void)mbar_wait(bar(kBarV), (uint32_t)(lv - 1) & 1u);
      }
      __syncwarp();
      if (elect_one()) {  // the contractions that were issued have read their operands and written tensor memory
        mma_commit(bar(kBarDrain));
        (void)mbar_wait(bar(kBarDrain), 0);
      }
    } else if (my_tiles > 0) {
      store(KIND == kStageRightWithV ? &maps.s1 : &maps.s0, my_tiles - 1, (kChunks - 1) * kRows);
    }
    if (lane == 0) asm volatile("cp.async.bulk.wait_group 0;" ::: "memory");
    __syncwarp();
  } else {
    // =========================== row threads ==================================================================
    const int unit = kUnits == 2 ? tid >> 6 : 0, r_unit = kUnits == 2 ? tid & 63 : tid;
    const uint32_t lane_base = (uint32_t)(warp * 32) << 16;
    const uint32_t col0 = kUnits == 2 ? 64u * unit : 0u;
    const uint32_t t_s = tmem + lane_base + col0;  // this row's columns of S
    const uint32_t t_p = tmem + lane_base + (col0 >> 1);
    // ---- the tile's column vector (this thread's entries), read one tile ahead and left as it is in memory, so that
    // nothing waits for the load before it is needed -------------------------------------------------------------
    auto column_vector = [&](int i, float(&v)[kVec]) {
      if (i >= my_tiles || (kRight && plain)) return;
      const Tile w = tile_at(i);
#pragma unroll
      for (int k = 0; k < kVec; ++k) {
        const int s = tid + k * kRows, x = w.u0 + (kUnits == 2 ? s >> 6 : 0), c = kUnits == 2 ? s & 63 : s;
        v[k] = -kGone;
        if (x < units && c < keys) {
          if (!kRight) v[k] = g.cl[((long long)w.eh * B + x) * M + c];
          else if (token_valid(g, w.e, x * B + c)) v[k] = 0.f;
        }
      }
    };
    // Leaves the vector of tile i in shared memory; true if a column inside the chunks is missing.
    auto put_vector = [&](int i, const float(&v)[kVec]) {
      bool missing = false;
      if (i < my_tiles && !(kRight && plain)) {
#pragma unroll
        for (int k = 0; k < kVec; ++k) {
          const int s = tid + k * kRows, c = kUnits == 2 ? s & 63 : s;
          const bool gone = v[k] == -kGone;
          vec[(i & 1) * 256 + s] = gone ? kGone : kRight ? 0.f : -v[k] * kLog2e;
          missing = missing || (gone && c < nch * 32);
        }
      }
      return missing;
    };
    // normaliser of this thread's row (right-factor) or validity of its query (left-factor), read one tile ahead too
    auto row_scalar = [&](int i, float(&v)[kChunks]) {
      if (i >= my_tiles || KIND == kStageOutput || (kRight && args.first)) return;
      const Tile w = tile_at(i);
      const int x = w.u0 + unit;
#pragma unroll
      for (int k = 0; k < kChunks; ++k) {
        const int r = r_unit + w.row_base + k * kRows;
        if (kRight) {
          v[k] = x < units && r < keys ? g.cr[((long long)w.eh * M + x) * B + r] : 1.0f;
        } else {
          const int n = r * B + column_start(x);
          v[k] = x < units && r < keys && n < g.N && mask_lets(g, w.e, n) ? 1.0f : 0.0f;
        }
      }
    };
    uint32_t ns = 0, no = 0, ne = 0;  // phases of S and O waited for, rows staged
    // 64 accumulator columns of this thread's row into the staging tile (scaled: times sm_scale after a rounding of its own
    // where the scale is no power of two); `direct`: where the row goes if the store's tensor map does not reach it.
    auto stage_row = [&](bool scaled, T* direct) {
      const bool two = (__float_as_uint(g.sm_scale) & 0x007fffffu) != 0u;
      bool ok = wait(kBarO, no++);
      tc_fence_after();
      if (ok && ne > 0) ok = wait(kBarFree, ne - 1);
      ++ne;
#pragma unroll
      for (int half = 0; half < 2; ++half) {
        float o[32];
        tmem_ld32_nowait(tmem + lane_base + kTmemO + 32 * half, o);
        tmem_wait_ld(o);
        uint32_t k[16];
#pragma unroll
        for (int j = 0; j < 16; ++j) {
          float2 t = make_float2(o[2 * j], o[2 * j + 1]);
          if (scaled) {
            if (two) round_pair<T>(t.x, t.y);
            t = mul2(t, make_float2(g.sm_scale, g.sm_scale));
          }
          k[j] = pack2<T>(t.x, t.y);
        }
#pragma unroll
        for (int c = 0; c < 4; ++c) {
          st_shared_v4(stage + swz(tid, 4 * half + c), k[4 * c], k[4 * c + 1], k[4 * c + 2], k[4 * c + 3]);
          if (direct != nullptr && 32 * half + 8 * c < D)
            *reinterpret_cast<uint4*>(direct + 32 * half + 8 * c) = make_uint4(k[4 * c], k[4 * c + 1], k[4 * c + 2], k[4 * c + 3]);
        }
      }
      fence_async_smem();
      tc_fence_before();
      mbar_arrive(bar(kBarE));
      return ok;
    };
    auto zero_rest = [&] {  // two units per tile: the columns of P that belong to the other unit
      if (kUnits == 2) {
        uint32_t z[16];
#pragma unroll
        for (int i = 0; i < 16; ++i) z[i] = 0u;
        const uint32_t other = tmem + lane_base + ((col0 ^ 64u) >> 1);
        tmem_st16(other, z);
        tmem_st16(other + 16, z);
      }
    };
    auto p_ready = [&] {
      tmem_wait_st();
      tc_fence_before();
      mbar_arrive(bar(kBarP));
    };

    float next_vec[kVec], next_row[kChunks];
#pragma unroll
    for (int k = 0; k < kVec; ++k) next_vec[k] = -kGone;
#pragma unroll
    for (int k = 0; k < kChunks; ++k) next_row[k] = 1.0f;
    column_vector(0, next_vec);
    row_scalar(0, next_row);
    bool missing = put_vector(0, next_vec);
    bool ok = true;

    // (a row thread leaves this loop only where all of them meet, so none is left alone at a barrier)
    for (int i = 0; i < my_tiles; ++i) {
      const Tile w = tile_at(i);
      const float* my_vec = vec + (i & 1) * 256 + col0;
      const int x = w.u0 + unit, r_in = r_unit + w.row_base;  // this row's block or column, and its place there
      const bool live = x < units && r_in < keys;
      const bool warp_live = __any_sync(0xffffffffu, live);
      float my_row[kChunks];
#pragma unroll
      for (int k = 0; k < kChunks; ++k) my_row[k] = next_row[k];
      // the vector is there for all; and all agree whether to go on, and whether something has to be masked
      if (named_barrier_or(kRowBarrier, kRows, !ok)) break;
      const bool masked = plain ? false : named_barrier_or(kRowBarrier, kRows, missing);
      column_vector(i + 1, next_vec);
      row_scalar(i + 1, next_row);
      // e over S (STORE) and its sum, against a shift: the maximum of S, plus a bound on -cl (an entropy of at most 256 outcomes: 8 in
      // powers of two).  Any shift within a few powers of two of the true maximum gives the same quotients.
      auto column_sum = [&](auto store, float& off) {
        constexpr bool kStore = decltype(store)::value;
        if (masked) return masked_column_exps<T, kStore>(t_s, nch, my_vec, off);
        off = fmaf(row_max<false>(t_s, nch, my_vec, 1.0f), kLog2e, 8.0f);
        return column_exps<T, kStore>(t_s, nch, my_vec, off);
      };

      ok = wait(kBarS, ns++);
      tc_fence_after();
      if (kRight) {
        float stat = 0.f;
        if (warp_live) {
          // x = sm_scale * round(S) / (cr + eps) in powers of two, maximum clamped from below
          const float mul = g.sm_scale / ((args.first ? 1.0f : my_row[0]) + kEps) * kLog2e;
          const float top = masked ? row_max<true>(t_s, nch, my_vec, 1.0f) : row_max<false>(t_s, nch, my_vec, 1.0f);
          const float off = fmaxf(round_through<T>(top) * mul, kEps * kLog2e);
          float sum, ent;
          if (masked) right_exps<T, true>(t_s, nch, my_vec, mul, off, sum, ent);
          else right_exps<T, false>(t_s, nch, my_vec, mul, off, sum, ent);
          const float dn = sum + kEps, inv = rcp_fast(dn);
          normalise<T>(t_s, t_p, nch, inv);
          zero_rest();
          stat = (kLn2 * ent - __logf(dn) * sum) * inv;  // sum_i r_i ln r_i, r_i = e_i / dn
        }
        p_ready();
        if (live) g.cl[((long long)w.eh * B + r_in) * M + x] = stat;
        missing = put_vector(i + 1, next_vec);
        ok = stage_row(true, nullptr) && ok;
        if (KIND == kStageRightWithV) ok = stage_row(false, nullptr) && ok;
      }

      if (KIND == kStageOutput) {
        if (warp_live) {
          float off;
          normalise<T>(t_s, t_p, nch, rcp_fast(column_sum(std::true_type(), off)));
          zero_rest();
        }
        p_ready();
        missing = put_vector(i + 1, next_vec);
        const int n = r_in * B + column_start(x);
        T* direct = nullptr;  // (padding rows are dropped, ma/ma_torch.py:108: their place is behind the end of the map)
        if (live && r_in == whole && n < g.N)
          direct = reinterpret_cast<T*>(const_cast<void*>(g.out.ptr)) + (long long)w.e * g.out.se + (long long)w.h * g.out.sh + (long long)n * g.out.sn;
        ok = stage_row(false, direct) && ok;
      }

      if (kLeft) {
#pragma unroll 1
        for (int rc = 0; rc < kChunks; ++rc) {
          if (rc > 0) {
            ok = wait(kBarS, ns++) && ok;
            tc_fence_after();
          }
          float z = 1e30f;  // 2^-z = 0: rows that do not exist and invalid queries contribute nothing
          if (warp_live) {
            float off;
            const float sum = column_sum(std::false_type(), off);
            if (my_row[rc] != 0.f) z = off + lg2(sum);
          }
          lse[tid + rc * kRows] = z;
          p_ready();
        }
        if (named_barrier_or(kRowBarrier, kRows, !ok)) break;  // every lse is there
        const float* my_lse = lse + col0;
#pragma unroll 1
        for (int mc = 0; mc < kChunks; ++mc) {
          ok = wait(kBarS, ns++) && ok;
          tc_fence_after();
          const int m = r_in + mc * kRows;
          float cr = 0.f;
          if (warp_live) {
            const float own = my_vec[m], mine = own > kGone ? own : 0.f;  // -cl[m]
            Sum2 s;
            for_chunks(t_s, nch, [&](float(&v)[16], int c) {
              uint32_t pk[8];
#pragma unroll
              for (int k = 0; k < 16; k += 4) {
                const float4 b = *reinterpret_cast<const float4*>(my_lse + 16 * c + k);
                round_pair<T>(v[k], v[k + 1]);
                round_pair<T>(v[k + 2], v[k + 3]);
                const float2 ua = sub2(fma2(make_float2(v[k], v[k + 1]), make_float2(kLog2e, kLog2e), make_float2(mine, mine)), make_float2(b.x, b.y));
                const float2 ub = sub2(fma2(make_float2(v[k + 2], v[k + 3]), make_float2(kLog2e, kLog2e), make_float2(mine, mine)), make_float2(b.z, b.w));
                const float2 ea = make_float2(ex2(ua.x), ex2(ua.y)), eb = make_float2(ex2(ub.x), ex2(ub.y));
                s.a = add2(s.a, ea);  // before rounding (ma/ma_torch.py:32)
                s.b = add2(s.b, eb);
                pk[k / 2] = pack2<T>(ea.x, ea.y);
                pk[k / 2 + 1] = pack2<T>(eb.x, eb.y);
              }
              tmem_st8(t_p + 8 * c, pk);
            });
            zero_rest();
            cr = s.get();
          }
          p_ready();
          if (x < units && m < keys) g.cr[((long long)w.eh * M + m) * B + x] = cr;
          if (mc == kChunks - 1) missing = put_vector(i + 1, next_vec);
          ok = stage_row(false, nullptr) && ok;
        }
      }
    }
    if (!ok) give_up(702);
  }

  tc_fence_before();
  __syncthreads();
  if (warp == 4) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(kCols) : "memory");
}

// ---------------------------------------------------------------------------------------------------
// Host side: launches
// ---------------------------------------------------------------------------------------------------
template <typename T, int NK, StageKind KIND>
cudaError_t launch_tile_typed(const Geometry& g, const TileMaps& maps, const TileArgs& args_in, bool hold, cudaStream_t stream) {
  const int units = is_right(KIND) ? g.M : g.B;
  TileArgs args = args_in;
  args.tiles = NK == 64 ? (units + 1) / 2 : NK == 256 && KIND != kStageLeft ? 2 * units : units;
  const long long total = (long long)args.tiles * g.E * g.H;
  if (total > 0x7fffffff) return cudaErrorInvalidValue;
  args.total = (int)total;
  const void* fn = (const void*)tile_kernel<T, NK, KIND, false>;
  if constexpr (is_right(KIND)) {
    if (hold) fn = (const void*)tile_kernel<T, NK, KIND, true>;
  }
  constexpr uint32_t smem = tile_smem(NK, KIND);
  if (const cudaError_t e = allow_dynamic_smem(fn, smem); e != cudaSuccess) return e;
  // one CTA for each place on the GPU; it takes tiles round-robin and loads the next one under the present one
  void* params[] = {(void*)&maps, (void*)&g, (void*)&args};
  return launch_kernel(fn, dim3(std::min(args.total, sm_count() * tile_ctas(NK))), dim3(kTileThreads), params, smem, stream);
}

template <typename T, int NK>
cudaError_t launch_tile_kind(const Geometry& g, StageKind kind, const TileMaps& maps, const TileArgs& args, bool hold, cudaStream_t stream) {
  switch (kind) {
    case kStageRight: return launch_tile_typed<T, NK, kStageRight>(g, maps, args, hold, stream);
    case kStageRightWithV: return launch_tile_typed<T, NK, kStageRightWithV>(g, maps, args, hold, stream);
    case kStageLeft: return launch_tile_typed<T, NK, kStageLeft>(g, maps, args, hold, stream);
    default: return launch_tile_typed<T, NK, kStageOutput>(g, maps, args, hold, stream);
  }
}

template <typename T>
cudaError_t launch_tile_dtype(const Geometry& g, int dtype, StageKind kind, bool first, int* host_status, bool wait_expiry, cudaStream_t stream) {
  const bool right = is_right(kind);
  const int keys = right ? g.B : g.M, nk = keys <= 64 ? 64 : keys <= 128 ? 128 : 256;
  const int a_rows = nk == 64 ? 64 : nk == 256 && kind == kStageLeft ? 256 : 128, b_rows = nk, s_rows = nk == 64 ? 64 : 128;
  TileMaps maps;
  bool ok;
  if (right) {
    ok = first ? token_map(&maps.a, dtype, g, g.q, a_rows) : state_map(&maps.a, dtype, g, g.ar, a_rows);
    ok = ok && token_map(&maps.b, dtype, g, g.k, b_rows) && strided_state_map(&maps.s0, dtype, g, g.al, g.M, g.B, s_rows);
    maps.v = maps.b;
    maps.s1 = maps.s0;
    if (kind == kStageRightWithV)
      ok = ok && token_map(&maps.v, dtype, g, g.v, b_rows) && strided_state_map(&maps.s1, dtype, g, g.y, g.M, g.B, s_rows);
  } else {
    ok = column_map(&maps.a, dtype, g, g.q, a_rows) && state_map(&maps.b, dtype, g, g.al, b_rows);
    maps.v = maps.b;
    if (kind == kStageOutput) ok = ok && state_map(&maps.v, dtype, g, g.y, b_rows) && column_map(&maps.s0, dtype, g, g.out, s_rows);
    else ok = ok && strided_state_map(&maps.s0, dtype, g, g.ar, g.B, g.M, s_rows);
    maps.s1 = maps.s0;
  }
  if (!ok) return cudaErrorInvalidValue;
  TileArgs args{};
  args.first = first ? 1 : 0;
  args.clear = right && first ? 1 : 0;
  args.host_status = host_status;
  if (nk == 64) return launch_tile_kind<T, 64>(g, kind, maps, args, wait_expiry, stream);
  if (nk == 128) return launch_tile_kind<T, 128>(g, kind, maps, args, wait_expiry, stream);
  return launch_tile_kind<T, 256>(g, kind, maps, args, wait_expiry, stream);
}

bool strides_ok(const View4& t, int E, int H, int D) {
  if (reinterpret_cast<uintptr_t>(t.ptr) % 16 != 0 || t.sn % 8 != 0 || t.sn < D) return false;
  if (H > 1 && (t.sh % 8 != 0 || t.sh == 0)) return false;
  if (E > 1 && (t.se % 8 != 0 || t.se == 0)) return false;
  return true;
}

}  // namespace

bool tile_supported(const Geometry& g, int qk_dtype, int v_dtype, const char** why) {
  auto no = [&](const char* w) { *why = w; return false; };
  if (qk_dtype != v_dtype || (qk_dtype != MA_B200_BF16 && qk_dtype != MA_B200_F16)) return no("needs bf16 or f16 for q, k and v");
  if (g.D != g.Dv || g.D % 8 != 0 || g.D > 64) return no("needs Dv = D, a multiple of 8, at most 64");
  if (g.B > 256 || g.M > 256) return no("needs block size and block count of at most 256");
  if (g.N < g.B) return no("needs at least one whole block");
  if ((long long)g.E * g.H > 65535) return no("E*H too large for the grid");
  if (g.q.ptr != nullptr) {
    if (!strides_ok(g.q, g.E, g.H, g.D) || !strides_ok(g.k, g.E, g.H, g.D) || !strides_ok(g.v, g.E, g.H, g.D) ||
        !strides_ok(g.out, g.E, g.H, g.D))
      return no("q, k, v, out need 16-byte aligned bases and strides that are non-zero multiples of 8 elements");
  }
  if (encode_fn() == nullptr) return no("driver entry point cuTensorMapEncodeTiled not available");
  return true;
}

cudaError_t launch_tile_stage(const Geometry& g, int dtype, StageKind kind, bool first, int* host_status, bool wait_expiry, cudaStream_t stream) {
  if (dtype == MA_B200_BF16) return launch_tile_dtype<__nv_bfloat16>(g, dtype, kind, first, host_status, wait_expiry, stream);
  return launch_tile_dtype<__half>(g, dtype, kind, first, host_status, wait_expiry, stream);
}

}  // namespace ma
