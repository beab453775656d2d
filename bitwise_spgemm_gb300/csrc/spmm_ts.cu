// spmm_ts.cu — persistent tensor-core bitmap SpMM for 16-bit B (tcgen05), the
// bit operand in tensor memory.
//
// C = A·B (or dX = Aᵀ·G) as a dense contraction over the occupied bit tiles:
// every 32-column word of A is expanded to 0 / 2.0 BF16 or FP16 values and
// multiplied by the matching 32 rows of B (the idea of the reference's tSparse
// kernel, source/src/mm.cu:123-145, which expanded 8x8 bitmap tiles into 0/1
// half wmma fragments).
//
// What bounds it: the tensor pipe and the producers that feed it.  With both
// operands in shared memory an MMA of 128x256x16 reads 12 KB in 128 cycles,
// and the producers' writes (16 KB a K tile) and B's arrival (16 KB) come on
// top: 180 bytes a cycle against 128.  Here the expanded bits go from the
// producers' registers straight into TMEM (tcgen05.st) and the MMA takes its A
// operand from there, so shared memory carries B alone: 64 bytes a cycle read,
// 32 written.  Measured with B's copy into tile order, against the kernel with
// both operands in shared memory and a CTA per 256x256 block: block-structured
// 16384x16384x2048 BF16 593 -> 556 us, 4096x4096x8192 at 10 % 207 -> 180
// (Aᵀ·G 209 -> 189), 8192x8192x512 63 -> 52, 1024x1024x256 17.8 -> 12.5.  A
// stage takes about 1210 cycles of which the MMAs need 1024; without MMAs it
// takes 1150, without the stores to TMEM 1050: expanding a tile (62
// instructions a warp and half), its store (440 cycles until it is visible)
// and the hand-offs make up the difference.  Stages of two tiles in four slots
// were slower (202 us at 4096x4096x8192), so were 20 and 24 producer warps.
//
// TMEM (512 columns): two accumulators of 128 rows x 128 columns (FP32), the
// halves of an item of 256 rows x 128 columns, and a ring of two stages of A
// (four K tiles x two halves x 16 columns).
//
// One CTA per SM.  The grid has a CTA per item; a resident CTA takes over the
// items of CTAs that have not started yet (cluster launch control), so items
// of unequal length balance without a queue in memory.  Roles:
//   warps 0-15  producers: four groups of four warps, group g expands every
//               fourth K tile into its slot (for Aᵀ·G the words of 32 rows are
//               transposed across the warp first), words loaded ahead;
//   warp 16     B by bulk copies (B in tile order) or TMA boxes;
//   warps 17-18 MMAs (128x128x16), one warp per half, by an elected lane; the
//               first also holds the CTA's TMEM;
//   warp 19     takes items and lists their occupied K tiles;
//   warps 20-27 epilogue: TMEM -> registers -> staging boxes -> C (TMA).
// Stage and item counters run over the whole launch, so every mbarrier phase
// follows from a counter.  Every wait is bounded: on timeout the role records
// error 5 in g_ts_error and stops; the others' bounded waits then end.
#include <cuda.h>

#include <cstring>
#include <type_traits>

#include "ptx.cuh"
#include "spmm_dev.cuh"
#include "tc_common.cuh"
#include "ts.cuh"

namespace bsp {

__device__ int g_ts_error;

namespace {

constexpr int kM = 128, kRows = 256, kN = 128, kK = 32;
constexpr int kTps = 4;                         // K tiles per stage, one per producer group
constexpr uint32_t kBox = 64 * kK * 2;          // 4 KB: 64 columns x 32 rows
constexpr uint32_t kBTile = 2 * kBox;           // 128 columns
constexpr uint32_t kBStage = kTps * kBTile;     // 32 KB
constexpr int kStages = 4;                      // of B, and of the barriers
constexpr int kAStages = 2;                     // of A, in TMEM
constexpr int kGroupWarps = 4, kProdWarps = kTps * kGroupWarps;
constexpr uint32_t kATmem = 2 * kN;             // first TMEM column of the A ring, behind the accumulators
constexpr uint32_t kATile = 32;                 // columns of a K tile: 16 per half
constexpr int kTmaWarp = kProdWarps, kMmaWarp = kProdWarps + 1, kSchedWarp = kProdWarps + 3;  // (two MMA warps)
constexpr int kEpiWarp0 = kProdWarps + 4, kEpiWarps = 8;
constexpr int kThreads = (kEpiWarp0 + kEpiWarps) * 32;
constexpr int kItems = 2;                       // items known ahead
constexpr int kItemUsers = kProdWarps + 3 + kEpiWarps;  // arrivals that free an item slot
constexpr int kAhead = 2;                       // tiles of its own a group loads A words ahead
constexpr int kListPad = kTps * (kAhead + 1);   // entries past the list that may be read
constexpr int kListMax = 4096;                  // K tiles of an item
constexpr int kSegMax = 32 / kTps;              // stages of a segment: a lane for each of its tiles
constexpr int kEpiCols = 64;                    // columns of an epilogue warp
constexpr int kEpiBox = 32 * 32 * 4;            // its staging: two boxes of 32 rows x 32 columns (128-byte swizzle)
constexpr int kErr = 5;
constexpr uint32_t kTmemCols = 512;
static_assert(kATmem + kAStages * kTps * kATile <= kTmemCols, "TMEM");

struct Item {
  int n;          // K tiles, -1 = no more items
  int x, y, z;    // row block, column block, split (batch: problem)
  int seen;       // halves with tiles
};

struct __align__(1024) Smem {
  uint8_t b[kStages * kBStage];
  uint8_t epi[kEpiWarps][2 * kEpiBox];
  __align__(16) uint16_t list[kItems][kListMax + kListPad];  // tile index | halves << 12, then zeros
  uint64_t full[kStages];   // the producers' warps and B's bytes
  uint64_t done[kStages];   // the stage's MMAs
  uint64_t tfull[2], tempty[2];
  uint64_t qfull[kItems], qempty[kItems];
  uint64_t clc;
  __align__(16) uint32_t clc_result[4];
  Item item[kItems];
  uint32_t tmem_addr;
  int gave_up;  // a role's wait expired
};
constexpr size_t kSmemAlign = 1024;
static_assert(sizeof(Smem) + kSmemAlign <= 232448, "shared memory");
static_assert(kListMax == 1 << 12, "tile index and halves in 16 bits");

__device__ __forceinline__ void fail() { atomicCAS(&g_ts_error, 0, kErr); }

// 32x32 bit transpose across the warp: afterwards bit j of lane i is what bit
// i of lane j was.  Five exchanges (Hacker's Delight 7-3); what each lane keeps
// and how it turns the other's word depend on the lane alone.
struct Transpose32 {
  uint32_t sel16, sel8, keep4, keep2, keep1;
  __device__ void init(int lane) {
    sel16 = (lane & 16) ? 0x3276u : 0x5410u;
    sel8 = (lane & 8) ? 0x3715u : 0x6240u;
    keep4 = (lane & 4) ? 0xf0f0f0f0u : 0x0f0f0f0fu;
    keep2 = (lane & 2) ? 0xccccccccu : 0x33333333u;
    keep1 = (lane & 1) ? 0xaaaaaaaau : 0x55555555u;
  }
  __device__ __forceinline__ uint32_t operator()(uint32_t x) const {
    const int lane = threadIdx.x & 31;
    x = __byte_perm(x, __shfl_xor_sync(kFull, x, 16), sel16);
    x = __byte_perm(x, __shfl_xor_sync(kFull, x, 8), sel8);
    uint32_t y = __shfl_xor_sync(kFull, x, 4);
    y = __funnelshift_l(y, y, (lane & 4) ? 28 : 4);
    x = (x & keep4) | (y & ~keep4);
    y = __shfl_xor_sync(kFull, x, 2);
    y = __funnelshift_l(y, y, (lane & 2) ? 30 : 2);
    x = (x & keep2) | (y & ~keep2);
    y = __shfl_xor_sync(kFull, x, 1);
    y = __funnelshift_l(y, y, (lane & 1) ? 31 : 1);
    return (x & keep1) | (y & ~keep1);
  }
};

constexpr int kModeBits = 0, kModeTrans = 1, kModeBatch = 2, kModeBatchTrans = 3, kModeI8 = 4, kModeBitsSeg = 5,
              kModeTransSeg = 6;

// Two FP32 sums rounded to the 16-bit type.
template <typename BT>
__device__ __forceinline__ uint32_t pack2(float lo, float hi) {
  if constexpr (std::is_same<BT, __nv_bfloat16>::value) {
    const __nv_bfloat162 p = __floats2bfloat162_rn(lo, hi);
    return *reinterpret_cast<const uint32_t*>(&p);
  } else {
    const __half2 p = __floats2half2_rn(lo, hi);
    return *reinterpret_cast<const uint32_t*>(&p);
  }
}

// The matrix of an item: the launch's, or its problem's.
struct Matrix {
  const uint32_t* A;
  int64_t M, K, Kw;
};

// int8 values as pairs of 16-bit floats (exact): 4 bytes of w -> 2 pairs.
// BF16: 128 + (low 7 bits) and 128 or 256 by the sign bit are bit patterns,
// their difference the value; FP16: 1024 + (value + 128) less 1152.
template <typename BT>
__device__ __forceinline__ uint32_t i8_pair(uint32_t p) {  // bytes 0 and 2 of p
  if constexpr (std::is_same<BT, __nv_bfloat16>::value) {
    const uint32_t a = (p & 0x007f007fu) | 0x43004300u, b = (p & 0x00800080u) | 0x43004300u;
    const __nv_bfloat162 d = __hsub2(*reinterpret_cast<const __nv_bfloat162*>(&a), *reinterpret_cast<const __nv_bfloat162*>(&b));
    return *reinterpret_cast<const uint32_t*>(&d);
  } else {
    const uint32_t a = (p ^ 0x00800080u) | 0x64006400u, b = 0x64806480u;
    const __half2 d = __hsub2(*reinterpret_cast<const __half2*>(&a), *reinterpret_cast<const __half2*>(&b));
    return *reinterpret_cast<const uint32_t*>(&d);
  }
}
template <typename BT>
__device__ __forceinline__ void i8_pairs(const uint4& q, uint32_t* v) {  // 16 values
  const uint32_t w[4] = {q.x, q.y, q.z, q.w};
#pragma unroll
  for (int i = 0; i < 4; i++) {
    v[2 * i] = i8_pair<BT>(__byte_perm(w[i], 0u, 0x4140));
    v[2 * i + 1] = i8_pair<BT>(__byte_perm(w[i], 0u, 0x4342));
  }
}

// I8: A is int8, [K tile][row][32] (bsp_i8_tiles), its values the MMA's operand
// (exact in 16 bits): one product over K where the planes' bits take eight,
// with weighted copies of B stacked first (4096x4096x256 BF16, 5 %: planes
// 29 us to stack B, 57 to multiply, 6 to reduce; values 19 in all, 32 with B in
// two parts, see k_split16_b).  Bound by the producers' loads and conversions
// (4096^3: 132 us, 1.04 PFLOP/s).
// TR: dX[K][N] = Aᵀ·G (output rows: columns of A, K tiles: 32 rows of A).
// kSeg: the accumulators are handed over every a.seg_stages stages (TsArgs);
// a kernel of its own, for the others' registers are full.
// BAT: CTA x of the grid is work item x of a batch (problem, 256-row block,
// 128-column block, K tiles), all of whose tiles are multiplied (a batch has
// no occupancy plan) and whose words come from A's rows.
template <typename BT, int MODE>
__global__ void __launch_bounds__(kThreads, 1) k_spmm_ts(TsArgs a, const __grid_constant__ CUtensorMap mapB,
                                                         const __grid_constant__ CUtensorMap mapC) {
  constexpr bool TR = MODE == kModeTrans || MODE == kModeBatchTrans || MODE == kModeTransSeg;
  constexpr bool BAT = MODE == kModeBatch || MODE == kModeBatchTrans;
  constexpr bool kSeg = MODE == kModeBitsSeg || MODE == kModeTransSeg;
  constexpr bool I8 = MODE == kModeI8;
  constexpr float kScale = I8 ? 1.f : tc::kTwoScale;  // a set bit is expanded to 2.0
  extern __shared__ __align__(1024) uint8_t smem_raw[];
  Smem& sm = *reinterpret_cast<Smem*>(
      smem_raw + ((kSmemAlign - (ptx::smem_addr(smem_raw) & (kSmemAlign - 1))) & (kSmemAlign - 1)));
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  auto matrix = [&](int z) -> Matrix {
    if (!BAT) return Matrix{a.A, a.M, a.K, a.Kw};
    const BatchProblemTc& p = a.probs[z];
    return Matrix{p.A, p.M, p.K, p.Kw};
  };
  ptx::griddep_launch_dependents();  // a batch's SDDMM may start on SMs this grid has left
  if (a.skip_if && __ldg(a.skip_if)) return;  // uniform over the grid
  if (tid == 0) {
    for (int s = 0; s < kStages; s++) {
      ptx::mbar_init(&sm.full[s], kProdWarps + 1);
      ptx::mbar_init(&sm.done[s], 2);
    }
    for (int h = 0; h < 2; h++) {
      ptx::mbar_init(&sm.tfull[h], 1);
      ptx::mbar_init(&sm.tempty[h], kEpiWarps);
    }
    for (int s = 0; s < kItems; s++) {
      ptx::mbar_init(&sm.qfull[s], 1);
      ptx::mbar_init(&sm.qempty[s], kItemUsers);
    }
    ptx::mbar_init(&sm.clc, 1);
    sm.gave_up = 0;
    ptx::fence_mbar_init();
  }
  if (warp == kMmaWarp) {
    ptx::tmem_alloc(&sm.tmem_addr, kTmemCols);
    ptx::tmem_relinquish();
  }
  ptx::tc_fence_before_sync();
  __syncthreads();
  ptx::tc_fence_after_sync();
  // Values that come from shared memory and steer a warp's loops go through a
  // warp reduction, whose result the compiler knows to be uniform: the issuing
  // warps then keep descriptors and addresses in uniform registers, without
  // which an MMA takes 54 cycles to issue.
  const uint32_t tmem = __reduce_max_sync(kFull, sm.tmem_addr);
  // 64-column boxes of an item's column block that hold output columns
  auto boxes = [&](int y) { return (int)min((int64_t)2, (a.N - (int64_t)y * kN + 63) / 64); };

  // Waits for a slot to be emptied use the parity of the phase before: a fresh
  // barrier passes it at once, so the first round needs no case of its own.
  if (warp < kProdWarps) {
    // ---------------- A producers ----------------
    // Group w/4 expands tile w/4 of every stage; a warp takes its 32 TMEM lanes
    // of both halves.  Rows past the matrix and
    // list entries past the item's repeat valid ones: their values meet output
    // rows that are not stored, rows of B that are zero, or no MMA.
    const int grp = warp / kGroupWarps, q = warp & 3;
    const uint32_t slot = tmem + ((uint32_t)(q * 32) << 16) + kATmem + (uint32_t)grp * kATile;
    Transpose32 transpose;
    if (TR) transpose.init(lane);
    // Aᵀ·G: lane p takes the A row that bit p of the transposed word stands for
    const uint32_t trow = (uint32_t)tc::unshuffled_column(lane);
    uint32_t g = 0, s2 = kStages - kAStages, p2 = 1u;  // stage, and the barrier and parity of the stage two before it
    for (int j = 0;; j++) {
      const int qs = j & (kItems - 1);
      if (!ptx::mbar_wait_warp(&sm.qfull[qs], (uint32_t)(j / kItems) & 1u)) {
        if (lane == 0) fail();
        break;
      }
      const int n = sm.item[qs].n;
      if (n < 0) break;
      const uint16_t* lst = sm.list[qs];
      const Matrix m = matrix(sm.item[qs].z);
      const uint32_t M = (uint32_t)m.M;
      // forward: the lane's row in each half; Aᵀ·G: the warp's word column in each half
      uint32_t at[2];
#pragma unroll
      for (int h = 0; h < 2; h++) {
        const int64_t r = (int64_t)sm.item[qs].x * kRows + h * kM + q * 32;
        at[h] = TR ? (uint32_t)min(r / 32, m.Kw - 1) : (uint32_t)min(r + lane, m.M - 1);
      }
      auto load_words = [&](int k, uint32_t (&w)[2]) {
        const uint32_t t = lst[k] & (kListMax - 1);
        const uint32_t r = TR ? min(t * kK + trow, M - 1) : 0u;
#pragma unroll
        for (int h = 0; h < 2; h++) {
          if (!BAT && a.At) w[h] = __ldg(a.At + (TR ? at[h] * M + r : t * M + at[h]));
          else w[h] = tc::unshuffle32(__ldg(m.A + (TR ? (int64_t)r * m.Kw + at[h] : (int64_t)at[h] * m.Kw + t)));
        }
      };
      uint32_t wq[kAhead][2];
      uint4 vq[2][2];  // int8: the coming tile's 32 bytes of each half
      auto load_bytes = [&](int k) {
        const uint32_t t = lst[k] & (kListMax - 1);
#pragma unroll
        for (int h = 0; h < 2; h++)
#pragma unroll
          for (int b = 0; b < 2; b++) vq[h][b] = __ldg(a.tiles + ((int64_t)t * m.M + at[h]) * 2 + b);
      };
      if (I8) {
        if (n > 0) load_bytes(grp);
      } else {
#pragma unroll
        for (int d = 0; d < kAhead; d++)
          if (n > 0) load_words(kTps * d + grp, wq[d]);
      }
      bool ok = true;
      for (int k = grp; k - grp < n; k += kTps, g++) {
        uint32_t e[32];
        if (I8) {
#pragma unroll
          for (int h = 0; h < 2; h++)
#pragma unroll
            for (int b = 0; b < 2; b++) i8_pairs<BT>(vq[h][b], e + 16 * h + 8 * b);
          load_bytes(min(k + kTps, n));
        } else {
#pragma unroll
          for (int h = 0; h < 2; h++) tc::expand_pairs(TR ? transpose(wq[0][h]) : wq[0][h], e + 16 * h);
#pragma unroll
          for (int d = 0; d + 1 < kAhead; d++)
#pragma unroll
            for (int h = 0; h < 2; h++) wq[d][h] = wq[d + 1][h];
          load_words(min(k + kTps * kAhead, n), wq[kAhead - 1]);
        }
        if (!ptx::mbar_wait_warp(&sm.done[s2], p2)) {
          ok = false;
          break;
        }
        ptx::tc_fence_after_sync();
        if (k < n) {
          ptx::tmem_st_32x32b_x32(slot + (g & (kAStages - 1)) * (kTps * kATile), e);
          ptx::tmem_wait_st();
        }
        ptx::tc_fence_before_sync();
        __syncwarp();
        const uint32_t s = s2 + kAStages < kStages ? s2 + kAStages : s2 + kAStages - kStages;
        if (lane == 0) ptx::mbar_arrive(&sm.full[s]);
        if (++s2 == kStages) {
          s2 = 0;
          p2 ^= 1u;
        }
      }
      if (!ok) {
        if (lane == 0) fail();
        break;
      }
      __syncwarp();
      if (lane == 0) ptx::mbar_arrive(&sm.qempty[qs]);
    }
  } else if (warp == kTmaWarp) {
    // ---------------- B ----------------
    const bool leader = ptx::elect_one();
    const uint32_t b0 = ptx::smem_addr(sm.b), f0 = ptx::smem_addr(&sm.full[0]);
    uint32_t s = 0, ph = 1;  // stage, and the parity that its emptying completes (the first round passes at once)
    for (int j = 0;; j++) {
      const int qs = j & (kItems - 1);
      if (!ptx::mbar_wait_warp<64>(&sm.qfull[qs], (uint32_t)(j / kItems) & 1u)) {
        if (leader) fail();
        break;
      }
      const int n = __reduce_max_sync(kFull, *(volatile int*)&sm.item[qs].n);
      if (n < 0) break;
      const uint16_t* lst = sm.list[qs];
      const int y = __reduce_max_sync(kFull, *(volatile int*)&sm.item[qs].y);
      const int nbox = boxes(y);
      const uint32_t tile_bytes = (uint32_t)nbox * kBox;
      // 256-column blocks of four 64-column atoms; this item's are two neighbours
      const uint8_t* bt = a.bt + (int64_t)(y >> 1) * (4 * (int)kBox) + (y & 1) * kBTile;
      const void* map = &mapB;
      if (BAT) {
        map = &a.probs[__reduce_max_sync(kFull, *(volatile int*)&sm.item[qs].z)].map;
        if (leader) ptx::tensormap_acquire(map);  // written by the host into global memory
        __syncwarp();
      }
      bool ok = true;
      for (int k0 = 0; k0 < n; k0 += kTps) {
        if (!ptx::mbar_wait_warp<64>(&sm.done[s], ph)) {
          ok = false;
          break;
        }
        if (leader) {
          const int cnt = min(kTps, n - k0);
          ptx::mbar_arrive_expect_tx(&sm.full[s], (uint32_t)cnt * tile_bytes);
#pragma unroll
          for (int u = 0; u < kTps; u++) {
            if (u >= cnt) break;
            const int t = lst[k0 + u] & (kListMax - 1);
            const uint32_t dst = b0 + s * kBStage + (uint32_t)u * kBTile;
            if (!BAT && a.bt) {
              ptx::bulk_g2s_u32(dst, bt + (int64_t)t * a.bt_cb * (4 * (int)kBox), tile_bytes, f0 + s * 8u);
            } else {
              for (int b = 0; b < nbox; b++)
                ptx::tma_load_2d_u32(dst + (uint32_t)b * kBox, map, y * kN + b * 64, t * kK, f0 + s * 8u);
            }
          }
        }
        __syncwarp();
        if (++s == kStages) {
          s = 0;
          ph ^= 1u;
        }
      }
      if (!ok) {
        if (leader) fail();
        break;
      }
      if (leader) ptx::mbar_arrive(&sm.qempty[qs]);
      __syncwarp();
    }
  } else if (warp == kMmaWarp || warp == kMmaWarp + 1) {
    // ---------------- MMA issuers ----------------
    // One warp per half: a stage is a wait, eight MMAs and a commit for each.
    const int h = warp - kMmaWarp;
    const bool leader = ptx::elect_one();
    const uint32_t ab = std::is_same<BT, __nv_bfloat16>::value ? 1u : 0u;
    const uint64_t bdesc = ptx::smem_desc_noswizzle_u32(ptx::smem_addr(sm.b), kBox, 1024) |
                           ((uint64_t)tc::kLayoutSw128 << 61);
    uint32_t g = 0, s = 0, ph = 0, tq = 0;  // tq: segments handed over
    for (int j = 0;; j++, tq++) {
      const int qs = j & (kItems - 1);
      if (!ptx::mbar_wait_warp(&sm.qfull[qs], (uint32_t)(j / kItems) & 1u)) {
        if (leader) fail();
        break;
      }
      const int n = __reduce_max_sync(kFull, *(volatile int*)&sm.item[qs].n);
      if (n < 0) break;
      const uint16_t* lst = sm.list[qs];
      const int nbox = boxes(__reduce_max_sync(kFull, *(volatile int*)&sm.item[qs].y));
      const uint32_t idesc = tc::idesc_f16(ab, 0u, 1u, (uint32_t)(nbox * 64), kM);
      // which of a stage's tiles have bits in this half, read before its wait
      const uint32_t bit = 0x1000u << h, bits = bit | (bit << 16);
      uint2 next = *reinterpret_cast<const uint2*>(lst);
      bool ok = ptx::mbar_wait_warp(&sm.tempty[h], (tq & 1u) ^ 1u);
      ptx::tc_fence_after_sync();
      int left = a.seg_stages;              // stages until the accumulator is handed over
      bool started = false, whole = false;  // whole: every tile of the stage has bits in this half
      bool ready = false;                   // the stage's barrier was seen complete
      for (int k0 = 0; ok && k0 < n; k0 += kTps, g++) {
        const uint2 cur = next;
        next = *reinterpret_cast<const uint2*>(lst + k0 + kTps);
        if (kSeg && left-- == 0) {  // a new segment, on an accumulator that the epilogue has read
          if (leader) ptx::tc_commit(&sm.tfull[h]);
          __syncwarp();
          tq++;
          ok = ptx::mbar_wait_warp(&sm.tempty[h], (tq & 1u) ^ 1u);
          if (!ok) break;
          started = whole = false;
          left = a.seg_stages - 1;
        }
        if (!ready) ok = ptx::mbar_wait_warp(&sm.full[s], ph);
        if (!ok) break;
        ptx::tc_fence_after_sync();
        const uint64_t bs = bdesc + (uint64_t)((s * kBStage) >> 4);
        const uint32_t as = tmem + kATmem + (g & (kAStages - 1)) * (kTps * kATile) + (uint32_t)(h * 16);
        const uint32_t d = tmem + (uint32_t)h * kN;
        const uint32_t s1 = s + 1 == kStages ? 0u : s + 1, ph1 = s + 1 == kStages ? ph ^ 1u : ph;
        uint32_t seen = 0;
        if (whole) {
          // The tensor pipe queues only a few MMAs: the coming stage's barrier
          // is asked before the last of this one's, so that the answer is
          // there when they are issued.
          if (leader) {
#pragma unroll
            for (int u = 0; u < kTps; u++)
#pragma unroll
              for (int k = 0; k < 2; k++) {  // K half k: A 8 columns on, B two 8-row groups on
                if (u == kTps - 1 && k == 0) seen = ptx::mbar_try_wait(&sm.full[s1], ph1);
                ptx::tc_mma_f16_ts(d, as + (uint32_t)(u * kATile + k * 8),
                                   bs + (uint64_t)((u * kBTile + k * 2048) >> 4), idesc, true);
              }
            ptx::tc_commit(&sm.done[s]);
          }
        } else {  // a tile without bits in this half, a short last stage, the item's first one
          if (leader) {
            bool on = started;
#pragma unroll
            for (int u = 0; u < kTps; u++) {
              if (!((u < 2 ? cur.x : cur.y) & (bit << (16 * (u & 1))))) continue;
#pragma unroll
              for (int k = 0; k < 2; k++)
                ptx::tc_mma_f16_ts(d, as + (uint32_t)(u * kATile + k * 8),
                                   bs + (uint64_t)((u * kBTile + k * 2048) >> 4), idesc, on || k > 0);
              on = true;
            }
            ptx::tc_commit(&sm.done[s]);
            seen = ptx::mbar_try_wait(&sm.full[s1], ph1);
          }
          started = started || ((cur.x | cur.y) & bits) != 0u;
        }
        whole = __all_sync(kFull, started && (next.x & next.y & bits) == bits);
        ready = __any_sync(kFull, seen);
        s = s1;
        ph = ph1;
      }
      if (!ok) {
        if (leader) fail();
        break;
      }
      if (leader) {
        if (n > 0) ptx::tc_commit(&sm.tfull[h]);
        else ptx::mbar_arrive(&sm.tfull[h]);
        ptx::mbar_arrive(&sm.qempty[qs]);
      }
      __syncwarp();
    }
  } else if (warp == kSchedWarp) {
    // ---------------- items and their lists ----------------
    uint32_t x = blockIdx.x, y = blockIdx.y, z = blockIdx.z;
    [[maybe_unused]] const uint32_t row_blocks = BAT ? 1u : (uint32_t)(((TR ? a.K : a.M) + kRows - 1) / kRows);
    // the grid's x runs over row blocks, then over column blocks (gridDim.y is 1)
    auto place = [&]() {
      if (BAT) return;
      y = x / row_blocks;
      x -= y * row_blocks;
    };
    place();
    const int nblk = BAT ? 0 : (int)(((TR ? a.K : a.M) + kM - 1) / kM);
    bool more = true;
    for (int j = 0;; j++) {
      if (lane == 0 && more) {  // ask for the next item while this one is listed
        ptx::mbar_arrive_expect_tx(&sm.clc, 16);
        ptx::clc_try_cancel(ptx::smem_addr(sm.clc_result), ptx::smem_addr(&sm.clc));
      }
      const int qs = j & (kItems - 1);
      if (!ptx::mbar_wait_warp<256>(&sm.qempty[qs], ((uint32_t)(j / kItems) & 1u) ^ 1u)) {
        if (lane == 0) fail();
        break;
      }
      if (!more) {
        if (lane == 0) {
          sm.item[qs].n = -1;
          ptx::mbar_arrive(&sm.qfull[qs]);
        }
        break;
      }
      if (BAT) {
        const int4 it = __ldg(a.items + x);
        const Matrix m = matrix(it.x);
        const uint32_t hv = (int64_t)it.y * kRows + kM < (TR ? m.K : m.M) ? 3u : 1u;
        const int n = it.w;
        // the item's first words, on their way to L2 before its producers ask
        if (n > 0) {
          const int64_t w0 = TR ? (int64_t)it.y * (kRows / 32) : 0;
          const int64_t r0 = TR ? 0 : (int64_t)it.y * kRows;
          for (int64_t r = r0 + lane; r < min(m.M, r0 + kRows); r += 32) ptx::prefetch_l2(m.A + r * m.Kw + w0);
        }
        for (int k = lane; k < n; k += 32) sm.list[qs][k] = (uint16_t)((uint32_t)k | (hv << 12));
        if (lane < kListPad) sm.list[qs][n + lane] = 0;
        __syncwarp();
        if (lane == 0) {
          sm.item[qs] = Item{n, it.y, it.z, it.x, n > 0 ? (int)hv : 0};
          ptx::mbar_arrive(&sm.qfull[qs]);
        }
      } else {
      // occupied tiles of the two 128-row blocks (ascending), this split's
      // share of them; the launcher guarantees that they fit
      const uint32_t* occ0 = a.occ + (int64_t)x * 2 * a.occ_words;
      const bool has1 = (int)x * 2 + 1 < nblk;
      int total = 0;
      if (gridDim.z > 1) {
        for (int w = lane; w < a.occ_words; w += 32)
          total += __popc(__ldg(occ0 + w) | (has1 ? __ldg(occ0 + a.occ_words + w) : 0u));
        total = (int)__reduce_add_sync(kFull, (unsigned)total);
      }
      const int lo = gridDim.z > 1 ? (int)((int64_t)total * z / gridDim.z) : 0;
      const int hi = gridDim.z > 1 ? (int)((int64_t)total * (z + 1) / gridDim.z) : kListMax;
      int n = 0;
      uint32_t hs = 0;
      for (int w0 = 0; w0 < a.occ_words; w0 += 32) {
        const int wl = w0 + lane;
        const uint32_t m0 = wl < a.occ_words ? __ldg(occ0 + wl) : 0u;
        const uint32_t m1 = (has1 && wl < a.occ_words) ? __ldg(occ0 + a.occ_words + wl) : 0u;
        const int nw = min(32, a.occ_words - w0);
        for (int i = 0; i < nw; i++) {  // lane b: tile b of word i
          const uint32_t b0 = __shfl_sync(kFull, m0, i), b1 = __shfl_sync(kFull, m1, i), bits = b0 | b1;
          const uint32_t hv = ((b0 >> lane) & 1u) | (((b1 >> lane) & 1u) << 1);
          const int pos = n + __popc(bits & ((1u << lane) - 1u));
          if (hv && pos >= lo && pos < hi) {
            sm.list[qs][pos - lo] = (uint16_t)((uint32_t)((w0 + i) * 32 + lane) | (hv << 12));
            hs |= hv;
          }
          n += __popc(bits);
        }
      }
      hs = __reduce_or_sync(kFull, hs);
      n = max(0, min(n, hi) - lo);
      if (lane < kListPad) sm.list[qs][n + lane] = 0;
      __syncwarp();
      if (lane == 0) {
        sm.item[qs] = Item{n, (int)x, (int)y, (int)z, (int)hs};
        ptx::mbar_arrive(&sm.qfull[qs]);
      }
      }
      // the answer
      if (!ptx::mbar_wait_warp<256>(&sm.clc, (uint32_t)j & 1u)) {
        if (lane == 0) fail();
        break;
      }
      more = ptx::clc_query(ptx::smem_addr(sm.clc_result), &x, &y, &z);
      place();
      __syncwarp();
      ptx::fence_proxy_async_smem();  // the answer is read before the next one is written
    }
  } else {
    // ---------------- epilogue ----------------
    // Every half is read back by all eight warps, a lane quarter and 64 columns
    // each, into two boxes of the warp's own, and handed back at once (590
    // cycles a half); the boxes leave by TMA while the next half is read.
    // Stores from registers took another 1700 cycles a half and kept the second
    // half's accumulator waiting (1024-column products 20.3 -> 18.6 us, a batch
    // of 128 problems of 64..2048 rows and columns with both gradients 114 ->
    // 111).
    const int ew = warp - kEpiWarp0, q = warp & 3;  // the TMEM lane quarter this warp may access
    const int cw = (ew >> 2) * kEpiCols;            // (ew & 3 runs over the quarters too)
    const bool leader = ptx::elect_one();
    uint8_t* box = sm.epi[ew];
    // the row of its 32 that a TMEM lane holds (Aᵀ·G: the column at the lane's
    // bit of an unshuffled word); 16-byte chunk u of row r sits at u ^ (r % 8)
    const uint32_t mr = (uint32_t)(TR ? tc::unshuffled_column(lane) : lane);
    uint8_t* mine = box + mr * 128;
    // one warp polls, the others wait for it at a hardware barrier
    auto epi_wait = [&](uint64_t* bar, uint32_t parity) -> bool {
      if (ew == 0 && !ptx::mbar_wait_warp(bar, parity) && lane == 0) *(volatile int*)&sm.gave_up = 1;
      ptx::bar_sync(1 + kTps, kEpiWarps * 32);
      return !*(volatile int*)&sm.gave_up;
    };
    uint32_t tq = 0;  // segments taken over
    for (int j = 0;; j++) {
      const int qs = j & (kItems - 1);
      if (!epi_wait(&sm.qfull[qs], (uint32_t)(j / kItems) & 1u)) {
        if (lane == 0) fail();
        break;
      }
      const Item it = sm.item[qs];
      if (it.n < 0) break;
      const Matrix m = matrix(it.z);
      const int64_t out_rows = TR ? m.K : m.M;
      const void* cmap = &mapC;
      if (BAT) {
        cmap = &a.probs[it.z].map2;
        if (leader) ptx::tensormap_acquire(cmap);  // written by the host into global memory
        __syncwarp();
      }
      const int64_t gcol = (int64_t)it.y * kN + cw;
      const int cols = (int)max((int64_t)0, min((int64_t)kEpiCols, a.N - gcol));  // live columns of this warp
      bool ok = true;
      int seg = 0, seen = it.seen;
      do {
        if (kSeg) {  // the halves with tiles in this segment
          const int k = seg * kTps * a.seg_stages + lane;
          if (it.n > 0)
            seen = __reduce_or_sync(kFull, lane < kTps * a.seg_stages && k < it.n ? sm.list[qs][k] >> 12 : 0);
        }
        const bool add = kSeg && seg > 0;  // to what the segments before left in the output
        for (int h = 0; h < 2; h++) {
          if (!epi_wait(&sm.tfull[h], tq & 1u)) {
            if (lane == 0) fail();
            ok = false;
            break;
          }
          ptx::tc_fence_after_sync();
          const int64_t rbase = (int64_t)it.x * kRows + h * kM + q * 32;  // the warp's first row
          const bool have = (seen >> h) & 1;
          const bool live = rbase < out_rows && cols > 0 && (have || !add);
          if (leader) {
            if (add) ptx::bulk_wait_all();  // the segment before is in the output
            else ptx::bulk_wait_read();     // the half before has left the boxes
          }
          __syncwarp();
          // FP32 rows of 32 columns, or 16-bit rows of 64: 128 bytes either way.
          // (dX in 16 bits from here instead of a pass that reads and casts it:
          // training step 4096x4096x8192 BF16 624 -> 594 us.)
          const bool half_out = MODE == kModeTrans && a.out16;
          if (live) {
            const uint32_t tb = tmem + ((uint32_t)(q * 32) << 16) + h * kN + (uint32_t)cw;
#pragma unroll
            for (int c = 0; c < 2; c++) {
              uint32_t v[32];
              if (have) {
                ptx::tmem_ld_32x32b_x32(tb + (uint32_t)(c * 32), v);
                ptx::tmem_wait_ld();
              }
              if (half_out) {
#pragma unroll
                for (int u = 0; u < 4; u++) {
                  uint32_t p[4];
#pragma unroll
                  for (int i = 0; i < 4; i++)
                    p[i] = have ? pack2<BT>(__uint_as_float(v[8 * u + 2 * i]) * kScale,
                                            __uint_as_float(v[8 * u + 2 * i + 1]) * kScale)
                                : 0u;
                  *reinterpret_cast<uint4*>(mine + (((c * 4 + u) ^ (mr & 7)) << 4)) = make_uint4(p[0], p[1], p[2], p[3]);
                }
                continue;
              }
#pragma unroll
              for (int u = 0; u < 8; u++)
                *reinterpret_cast<float4*>(mine + c * kEpiBox + ((u ^ (mr & 7)) << 4)) =
                    have ? make_float4(__uint_as_float(v[4 * u]) * kScale, __uint_as_float(v[4 * u + 1]) * kScale,
                                       __uint_as_float(v[4 * u + 2]) * kScale, __uint_as_float(v[4 * u + 3]) * kScale)
                         : make_float4(0.f, 0.f, 0.f, 0.f);
            }
          }
          ptx::tc_fence_before_sync();
          ptx::fence_proxy_async_smem();
          __syncwarp();
          if (lane == 0) ptx::mbar_arrive(&sm.tempty[h]);
          if (!live) continue;
          if (BAT || a.c_map) {  // rows and columns past the output are clipped
            if (leader) {
              for (int c = 0; c * (half_out ? 64 : 32) < cols; c++) {
                if (add) ptx::tma_add_3d(cmap, (int)gcol + c * 32, (int)rbase, it.z, box + c * kEpiBox);
                else ptx::tma_store_3d(cmap, (int)gcol + c * 32, (int)rbase, BAT ? 0 : it.z, box + c * kEpiBox);
              }
              ptx::bulk_commit();
            }
          } else {
            const int nr = (int)min((int64_t)32, out_rows - rbase);
            for (int r = 0; r < nr; r++)
              for (int c = lane; c < cols; c += 32) {
                const float x = *reinterpret_cast<const float*>(
                    box + (c >> 5) * kEpiBox + r * 128 + ((((c & 31) >> 2) ^ (r & 7)) << 4) + (c & 3) * 4);
                float* o = a.C + (rbase + r) * a.ldc + gcol + c;
                if (add) atomicAdd(o, x);  // (the thread that wrote it: in order)
                else *o = x;
              }
            __syncwarp();
          }
        }
        tq++;
        seg++;
      } while (ok && kSeg && seg * kTps * a.seg_stages < it.n);
      if (!ok) break;
      if (lane == 0) ptx::mbar_arrive(&sm.qempty[qs]);
    }
    if (leader) ptx::bulk_wait_all();
    __syncwarp();
  }
  ptx::tc_fence_before_sync();
  __syncthreads();
  if (warp == kMmaWarp) {
    ptx::tc_fence_after_sync();
    ptx::tmem_dealloc(tmem, kTmemCols);
  }
}

template <typename BT, int MODE>
int launch_t(const TsArgs& a, const CUtensorMap& map, const CUtensorMap& mapc, dim3 grid, cudaStream_t s) {
  constexpr size_t smem = sizeof(Smem) + kSmemAlign;
  auto kern = k_spmm_ts<BT, MODE>;
  static bool configured[64] = {};
  int dev = 0;
  BSP_CUDA(cudaGetDevice(&dev));
  if (dev >= 64 || !configured[dev]) {
    BSP_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    if (dev < 64) configured[dev] = true;
  }
  kern<<<grid, kThreads, smem, s>>>(a, map, mapc);
  BSP_LAUNCHED();
  return BSP_OK;
}

}  // namespace

int64_t ts_item_rows() { return kRows; }
int64_t ts_item_cols() { return kN; }
int64_t ts_max_cols() { return (int64_t)65535 * 256; }

int launch_ts(TsArgs a, const CUtensorMap& map, bool trans, int splits, cudaStream_t s) {
  const int64_t gx = ceil_div(trans ? a.K : a.M, kRows), gy = ceil_div(a.N, kN);
  if (a.N > ts_max_cols() || gx * gy > 0x7fffffff) return BSP_ERR_CAPACITY;
  const dim3 grid((unsigned)(gx * gy), 1, (unsigned)splits);
  // C (or the splits' partials) by TMA, where its rows start on 16 bytes
  CUtensorMap mapc;
  memset(&mapc, 0, sizeof(mapc));
  const int64_t rows = trans ? a.K : a.M;
  if (a.seg_stages < 0 || a.seg_stages > kSegMax) return BSP_ERR_INTERNAL;
  if (a.out16) {
    if (splits > 1 || !trans || a.tiles || a.seg_stages) return BSP_ERR_UNSUPPORTED;
    BSP_TRY(make_out_map16(&mapc, a.C, a.bdt, rows, a.N, a.ldc));
    a.c_map = true;
  } else if (a.part) {
    BSP_TRY(make_out_map(&mapc, a.part, rows, a.N, a.ldp, splits, a.part_stride));
    a.c_map = true;
  } else if (a.c_vec) {
    BSP_TRY(make_out_map(&mapc, a.C, rows, a.N, a.ldc, 1, rows * a.ldc));
    a.c_map = true;
  }
  if (a.tiles) {
    if (a.bdt == BSP_BF16) return launch_t<__nv_bfloat16, kModeI8>(a, map, mapc, grid, s);
    if (a.bdt == BSP_F16) return launch_t<__half, kModeI8>(a, map, mapc, grid, s);
    return BSP_ERR_UNSUPPORTED;
  }
  if (a.seg_stages) {
    if (a.bdt == BSP_BF16)
      return trans ? launch_t<__nv_bfloat16, kModeTransSeg>(a, map, mapc, grid, s)
                   : launch_t<__nv_bfloat16, kModeBitsSeg>(a, map, mapc, grid, s);
    if (a.bdt == BSP_F16 && !trans) return launch_t<__half, kModeBitsSeg>(a, map, mapc, grid, s);
    return BSP_ERR_UNSUPPORTED;
  }
  if (a.bdt == BSP_BF16)
    return trans ? launch_t<__nv_bfloat16, kModeTrans>(a, map, mapc, grid, s)
                 : launch_t<__nv_bfloat16, kModeBits>(a, map, mapc, grid, s);
  if (a.bdt == BSP_F16)
    return trans ? launch_t<__half, kModeTrans>(a, map, mapc, grid, s) : launch_t<__half, kModeBits>(a, map, mapc, grid, s);
  return BSP_ERR_UNSUPPORTED;
}

int launch_ts_batch(const BatchProblemTc* probs, const int4* items, int n_items, int64_t N, int bdt, bool trans,
                    cudaStream_t s) {
  if (n_items == 0 || N == 0) return BSP_OK;
  TsArgs a = {};
  a.N = N;
  a.bdt = bdt;
  a.c_vec = true;
  a.probs = probs;
  a.items = items;
  CUtensorMap unused;
  memset(&unused, 0, sizeof(unused));
  const dim3 grid((unsigned)n_items);
  if (bdt == BSP_BF16)
    return trans ? launch_t<__nv_bfloat16, kModeBatchTrans>(a, unused, unused, grid, s)
                 : launch_t<__nv_bfloat16, kModeBatch>(a, unused, unused, grid, s);
  if (bdt == BSP_F16)
    return trans ? launch_t<__half, kModeBatchTrans>(a, unused, unused, grid, s) : launch_t<__half, kModeBatch>(a, unused, unused, grid, s);
  return BSP_ERR_UNSUPPORTED;
}

int ts_device_error(int* out, bool clear) {
  BSP_CUDA(cudaMemcpyFromSymbol(out, g_ts_error, sizeof(int)));
  if (clear) {
    const int zero = 0;
    BSP_CUDA(cudaMemcpyToSymbol(g_ts_error, &zero, sizeof(int)));
  }
  return BSP_OK;
}

}  // namespace bsp
