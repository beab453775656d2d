// spmm_tc.cu — tensor-core kernels with both operands in shared memory
// (tcgen05, TMEM accumulators) and the host side of the tensor-core products.
//
// k_spmm_tc runs the SDDMM dA = (G·Xᵀ) ⊙ A, dense over N with a masked store,
// and the CTA-per-item forms of the batched products (forward, which wide
// batches take where it finishes first; Aᵀ·G and SDDMM on request).  The single forward product and Aᵀ·G run on the persistent kernel of
// spmm_ts.cu, launched from here.
//
// CTA tile: 256 rows x 256 columns of C as two 128-row halves, each with its
// FP32 accumulator in TMEM (2 x 256 columns); both halves multiply the same
// B stage, so every B byte brought into shared memory feeds 256 rows.  Per
// CTA:
//   256·TPS producer threads (one row of one tile each; batched bit operands):
//     load the tile's words, expand them into the A operand (K-major core
//     matrices, 2.0 per set bit; the idea of the reference's tSparse kernel,
//     source/src/mm.cu:123-145) and arrive on the stage's "full" mbarrier;
//     after the last stage 16 of these warps read the accumulators back
//     (tcgen05.ld), scale by 0.5 and store C through a 32x32 staging tile per
//     warp;
//   a TMA warp: the dense operands' boxes (128-byte swizzle);
//   an MMA warp: allocates TMEM; an elected lane issues two tcgen05.mma (K=16)
//     per occupied half per tile and commits the stage to its "empty" mbarrier.
// Every mbarrier wait is bounded (timeout -> error 3 in g_tc_error, the CTA
// skips its stores and frees its TMEM).
#include <cuda.h>
#include <cudaTypedefs.h>

#include <cstdlib>
#include <cstring>
#include <type_traits>

#include "ptx.cuh"
#include "spmm_dev.cuh"
#include "tc_common.cuh"
#include "ts.cuh"

namespace bsp {

__device__ int g_tc_error;

namespace {

constexpr int kTcM = 128;                 // rows of one MMA and of one occupancy block
constexpr int kHalves = 2;                // a CTA owns two 128-row halves ...
constexpr int kCtaM = kTcM * kHalves;     // ... 256 output rows, sharing every B tile
constexpr int kTcN = 256;
constexpr int kTcK = 32;                  // one packed word of A per row and K tile
constexpr int kATile = kCtaM * kTcK * 2;  // 16 KB: both halves of one K tile
constexpr int kAHalf = kTcM * kTcK * 2;   // 8 KB
constexpr int kBTile = kTcK * kTcN * 2;   // 16 KB
// Each operand has a 96 KB ring of stages.  A stage carries TPS K tiles (a
// kernel template parameter): 2 tiles in 3 stages of 32 KB.  The SDDMM runs 3
// stages of one 32 KB box per operand.
constexpr int kRingBytes = 96 * 1024;
constexpr int kMaxStages = 3;
// Producers: one group of 256 threads (one per row of the CTA tile) per tile
// of the stage, so a warp expands one tile per stage; then a TMA warp and an
// MMA warp (allocates TMEM, issues the MMAs).
constexpr int kGroupThreads = kCtaM;
constexpr __host__ __device__ int tc_threads(int tps) { return kGroupThreads * tps + 64; }
constexpr int kWordAhead = 4;                 // A words are loaded this many stages ahead
// Occupied K tiles of the CTA, listed once in shared memory: tile index in
// bits 0-27, which 128-row halves have bits in bits 28-29.
constexpr int kListMax = 4096;
constexpr uint32_t kTmemCols = 512;       // two 128x256 FP32 accumulators
// Epilogue staging: a warp's 32 rows x 32 columns of FP32 in the idle stage
// memory, rows 36 floats apart (16-byte aligned; the row-wise float4 writes
// and the column-block float4 reads are both free of bank conflicts).
constexpr int kEpiStride = 36;
constexpr int kEpiWarps = 16;  // 4 TMEM lane quarters x 2 accumulators x 2 column halves
using tc::kLbo;
using tc::kSbo;
using tc::kLayoutSw128;
constexpr int kSddmm = 2, kBatch = 3, kBatchT = 4, kBatchS = 5;
// kBatch / kBatchT / kBatchS: the forward product, Aᵀ·G and the SDDMM of a
// batch, CTA b running work item b with its problem's record
__host__ __device__ constexpr bool batched_mode(int m) { return m == kBatch || m == kBatchT || m == kBatchS; }
__host__ __device__ constexpr bool trans_mode(int m) { return m == kBatchT; }
__host__ __device__ constexpr bool sddmm_mode(int m) { return m == kSddmm || m == kBatchS; }
// B (fwd) / G (trans) tile: four TMA boxes of 64 columns x 32 reduction rows,
// 128-byte swizzle, kBox bytes apart (the LBO); 8-row groups 1 KB apart (SBO).
constexpr int kBoxCols = 64;
constexpr uint32_t kBox = kBoxCols * kTcK * 2;  // 4 KB
// SDDMM: a stage is 64 columns of N: the G tile (256 rows) and the X tile
// (256 rows) are one box each, K-major with 128-byte swizzle (rows 128 B,
// 8-row groups 1 KB apart); the four K=16 steps start 32 B apart.
constexpr int kSdK = 64;
constexpr int kSdTile = kCtaM * kSdK * 2;  // one G or X box of a stage: 32 KB
constexpr uint32_t kSdSbo = 1024;
// Shared memory is requested with this much slack so the stage buffers can
// be aligned to the 1 KB swizzle atom.
constexpr size_t kSmemAlign = 1024;

struct __align__(1024) TcSmem {
  uint8_t a[kRingBytes];  // stage s at s * stage bytes
  uint8_t b[kRingBytes];
  int list[kListMax];
  int nlist, seen, lo;
  uint64_t full[kMaxStages];   // producer warps + the TMA transaction arrival
  uint64_t empty[kMaxStages];  // tcgen05.commit of the stage's MMAs
  uint64_t done;
  uint32_t tmem_addr;
  int abort;
};


struct TcArgs {
  const uint32_t* A;  // bit matrix, packed rows [M][Kw]
  int64_t M, K, Kw;
  const void* B;      // fwd: B [K][ldb]; trans: G [M][ldb]; sddmm: X [K][ldb]
  int64_t ldb;
  const void* G;      // sddmm: G [M][ldg]
  int64_t ldg;
  int64_t N;
  float* C;           // fwd: C [M][ldc]; trans: dX [K][ldc]; sddmm: dA [M][ldc]
  int64_t ldc;
  int bdt;
  // batched form (kBatch): CTA b runs work item b of the batch
  const BatchProblemTc* bprobs;
  const int4* items;  // {problem, 256-row block, 256-column block, K tiles}
};

// MODE:
//   kSddmm   dA[M,K] = (G · Xᵀ) ⊙ A  G and X K-major (TMA, 128-byte swizzle),
//                                    dense over N, masked store
//   kBatch   C[M,N]  = A · B         A bits K-major from A's words, B MN-major
//   kBatchT  C[K,N]  = Aᵀ · G        Aᵀ MN-major built from A's row words (no
//                                    transposed copy), G MN-major
//   kBatchS  the SDDMM per problem
// The bit operands are expanded into core matrices (LBO = 128 B along the
// reduction, SBO = 512 B along M/N); the dense 16-bit operands come by TMA
// in swizzled layouts.  The modes differ only in the producers, the
// descriptors and the epilogue.
template <typename BT, int MODE, int TPS>
__global__ void __launch_bounds__(tc_threads(TPS), 1) k_spmm_tc(TcArgs a, const __grid_constant__ CUtensorMap mapA,
                                                               const __grid_constant__ CUtensorMap mapB) {
  constexpr int kTilesPerStage = TPS;
  constexpr bool kSd = sddmm_mode(MODE), kTr = trans_mode(MODE), kBat = batched_mode(MODE);
  constexpr int kStageBytes = kSd ? kSdTile : TPS * kATile;
  constexpr int kStages = kRingBytes / kStageBytes;
  constexpr int kProducerWarps = kGroupThreads * TPS / 32;
  constexpr int kTmaWarp = kProducerWarps;
  constexpr int kMmaWarp = kProducerWarps + 1;
  static_assert(kStages >= 2 && kStages <= kMaxStages, "stage ring");
  static_assert(kProducerWarps >= kEpiWarps, "the epilogue runs on producer warps");
  extern __shared__ __align__(1024) uint8_t smem_raw[];
  TcSmem& sm = *reinterpret_cast<TcSmem*>(
      smem_raw + ((kSmemAlign - (ptx::smem_addr(smem_raw) & (kSmemAlign - 1))) & (kSmemAlign - 1)));
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  constexpr bool kFwdLike = MODE == kBatch;
  // the CTA's problem: the launch's (fwd / trans / sddmm) or its work item's (batch)
  const uint32_t* gA = a.A;
  int64_t gM = a.M, gK = a.K, gKw = a.Kw, gldc = a.ldc;
  float* gC = a.C;
  const void* bmap = &mapB;
  const void* amap = &mapA;
  int64_t row0 = (int64_t)blockIdx.x * kCtaM;  // output rows: M (fwd, sddmm) or K (trans)
  int64_t col0 = (int64_t)blockIdx.y * kTcN;   // output columns: N (fwd, trans) or K (sddmm)
  if (kBat) {
    const int4 it = a.items[blockIdx.x];
    const BatchProblemTc& p = a.bprobs[it.x];
    gA = p.A;
    gM = p.M;
    gK = p.K;
    gKw = p.Kw;
    gC = p.C;
    gldc = p.ldc;
    bmap = kSd ? &p.map2 : &p.map;  // SDDMM: X [K][N] (the B side), G [M][N] (the A side)
    amap = &p.map;
    row0 = (int64_t)it.y * kCtaM;
    col0 = (int64_t)it.z * kTcN;
  }
  const int64_t out_rows = kTr ? gK : gM;
  const int64_t out_cols = kSd ? gK : a.N;
  // B boxes (64 columns) holding output columns of this CTA: a narrow last
  // column tile loads, multiplies and stores only those (MMA N = 64·nbox)
  const int nbox = kSd ? kTcN / kBoxCols
                                  : (int)min((int64_t)(kTcN / kBoxCols), (out_cols - col0 + kBoxCols - 1) / kBoxCols);
  const int dense_halves = __any_sync(kFull, row0 + kTcM < out_rows) ? 3 : 1;

  if (tid == 0) {
    for (int s = 0; s < kStages; s++) {
      // one arrival per producer warp + the TMA warp's (SDDMM: TMA only)
      ptx::mbar_init(&sm.full[s], kSd ? 1 : kProducerWarps + 1);
      ptx::mbar_init(&sm.empty[s], 1);
    }
    ptx::mbar_init(&sm.done, 1);
    sm.abort = 0;
    ptx::fence_mbar_init();
  }
  if (warp == kMmaWarp) {
    ptx::tmem_alloc(&sm.tmem_addr, kTmemCols);
    ptx::tmem_relinquish();
  }
  if ((MODE == kBatch || MODE == kBatchT) && warp == 0) {
    // every reduction tile (a batch has no occupancy plan): K tiles of the
    // forward product, 32-row tiles of A for Aᵀ·G; both halves that hold rows
    const int64_t red = MODE == kBatch ? gKw : (gM + kTcK - 1) / kTcK;
    const int ntot = (int)min(red, (int64_t)kListMax);
    for (int k = lane; k < ntot; k += 32) sm.list[k] = k | (dense_halves << 28);
    __syncwarp();
    if (lane == 0) {
      sm.lo = 0;
      sm.nlist = ntot;
      sm.seen = ntot > 0 ? dense_halves : 0;
    }
  }
  // SDDMM: a block of A without set bits needs no product at all
  if (kSd) {
    uint32_t acc = 0;
    if (tid < kCtaM && row0 + tid < gM) {
      const uint32_t* arow = gA + (row0 + tid) * gKw;
      for (int64_t w = col0 / 32; w < min(gKw, (col0 + kTcN) / 32); w++) acc |= __ldg(arow + w);
    }
    const int any = __syncthreads_or(acc != 0u);
    if (tid == 0) {
      sm.nlist = any ? (int)((a.N + kSdK - 1) / kSdK) : 0;  // steps of kSdK columns of N
      sm.seen = any ? dense_halves : 0;
      sm.lo = 0;
    }
  }
  ptx::tc_fence_before_sync();
  __syncthreads();
  ptx::tc_fence_after_sync();
  const uint32_t tmem = __reduce_max_sync(kFull, sm.tmem_addr);  // (uniform to the compiler, as is n)
  const int n = __reduce_max_sync(kFull, sm.nlist);
  const int* lst = sm.list + sm.lo;  // this CTA's occupied tiles (fwd / trans)
  // stage i: list entries 2i and 2i+1 (fwd / trans) or N columns [64i, 64i+64) (SDDMM)
  const int nstages = kSd ? n : (n + kTilesPerStage - 1) / kTilesPerStage;

  if (warp < kProducerWarps) {
    // ---------------- A producers (fwd / trans) ----------------
    // Group u (warps 8u..8u+7) expands tile u of every stage, one row (fwd)
    // or one (A row, word) pair (trans) per thread, from words loaded
    // kWordAhead stages ahead; each warp arrives once per stage after its
    // lanes' writes are fenced.  Lane 0 waits for the slot for the warp.
    if (!kSd) {
      const int u = warp / (kGroupThreads / 32);
      const int r = tid % kGroupThreads;
      auto load_word = [&](int k) -> uint32_t {
        if (k >= n) return 0u;
        const int t = lst[k] & 0x0fffffff;
        if (kFwdLike) {
          const int64_t arow = row0 + r;
          if (arow >= gM) return 0u;
          return __ldg(gA + arow * gKw + t);
        }
        const int64_t arow = (int64_t)t * kTcK + (r & 31);
        const int64_t wcol = row0 / 32 + (r >> 5);
        if (arow >= gM || wcol >= gKw) return 0u;
        return __ldg(gA + arow * gKw + wcol);
      };
      uint32_t wq[kWordAhead];
#pragma unroll
      for (int j = 0; j < kWordAhead; j++) wq[j] = load_word(kTilesPerStage * j + u);
      for (int i = 0; i < nstages; i++) {
        const int s = i % kStages;
        const uint32_t w0 = wq[0];
        const uint32_t wnew = load_word(kTilesPerStage * (i + kWordAhead) + u);
        // (no abort poll on this path: a role that gives up stops arriving,
        // and every other role's own bounded wait then ends its loop)
        int go = 1;
        if (lane == 0 && i >= kStages && !ptx::mbar_wait(&sm.empty[s], ((i / kStages) - 1) & 1)) {
          atomicCAS(&g_tc_error, 0, 3);
          sm.abort = 1;
          go = 0;
        }
        if (!__shfl_sync(kFull, go, 0)) break;
        if (kTilesPerStage * i + u < n) {
          uint8_t* at = sm.a + s * kStageBytes + u * kATile;
          uint4 e[4];
          tc::expand32_two(w0, e);
          if (kFwdLike) {
            // row r of the tile: half r/128 at 8 KB, then core matrices
            uint8_t* as = at + (r >> 3) * kSbo + (r & 7) * 16;
#pragma unroll
            for (int c = 0; c < 4; c++) *reinterpret_cast<uint4*>(as + c * kLbo) = e[c];
          } else {
            // A row j of the tile, word wk of the block: output rows wk*32 + 8c ..
            const int j = r & 31, wk = r >> 5;
            uint8_t* as = at + (j >> 3) * kLbo + (j & 7) * 16;
#pragma unroll
            for (int c = 0; c < 4; c++) *reinterpret_cast<uint4*>(as + (wk * 4 + c) * kSbo) = e[c];
          }
        }
        ptx::fence_proxy_async_smem();
        __syncwarp();
        if (lane == 0) ptx::mbar_arrive(&sm.full[s]);
#pragma unroll
        for (int j = 0; j < kWordAhead - 1; j++) wq[j] = wq[j + 1];
        wq[kWordAhead - 1] = wnew;
      }
    }
  } else if (warp == kTmaWarp) {
    // ---------------- TMA issuer ----------------
    // (this warp and the next run whole, with one elected lane to issue: see
    // ptx::mbar_wait_warp)
    const bool leader = ptx::elect_one();
    const uint32_t a0 = ptx::smem_addr(sm.a), b0 = ptx::smem_addr(sm.b), f0 = ptx::smem_addr(&sm.full[0]);
    if (kBat && leader) {  // written by the host into global memory
      ptx::tensormap_acquire(bmap);
      if (kSd) ptx::tensormap_acquire(amap);
    }
    __syncwarp();
    uint32_t s = 0, ph = 1;  // stage, and the parity its emptying completes (the first round passes at once)
    for (int i = 0; i < nstages; i++) {
      if (!ptx::mbar_wait_warp(&sm.empty[s], ph)) {
        if (leader) {
          atomicCAS(&g_tc_error, 0, 3);
          sm.abort = 1;
        }
        break;
      }
      if (leader) {
        const uint32_t fb = f0 + s * 8, as = a0 + s * kStageBytes, bs = b0 + s * kStageBytes;
        if (kSd) {
          // G rows row0.. and X rows col0.. (256 each), N columns i*64..
          ptx::mbar_arrive_expect_tx(&sm.full[s], 2 * kSdTile);
          ptx::tma_load_2d_u32(as, amap, i * kSdK, (int)row0, fb);
          ptx::tma_load_2d_u32(bs, bmap, i * kSdK, (int)col0, fb);
        } else {
          // B (fwd) / G (trans) rows t*32.. of the stage's tiles, columns col0 + 64*j
          const int k0 = kTilesPerStage * i;
          const int cnt = min(kTilesPerStage, n - k0);  // tiles in this stage
          ptx::mbar_arrive_expect_tx(&sm.full[s], cnt * nbox * kBox);
#pragma unroll
          for (int u = 0; u < kTilesPerStage; u++) {
            if (u >= cnt) break;
            const int t = lst[k0 + u] & 0x0fffffff;
#pragma unroll
            for (int j = 0; j < kTcN / kBoxCols; j++)
              if (j < nbox)
                ptx::tma_load_2d_u32(bs + u * kBTile + j * kBox, bmap, (int)col0 + j * kBoxCols, t * kTcK, fb);
          }
        }
      }
      __syncwarp();
      if (++s == kStages) {
        s = 0;
        ph ^= 1u;
      }
    }
  } else if (warp == kMmaWarp) {
    // ---------------- MMA issuer ----------------
    // Descriptors of stage 0 are built once; every MMA adds a compile-time
    // offset (plus the stage's) to the 14-bit start-address field (>> 4).
    const bool leader = ptx::elect_one();
    const uint32_t ab = std::is_same<BT, __nv_bfloat16>::value ? 1u : 0u;
    const uint32_t idesc = tc::idesc_f16(ab, kTr ? 1u : 0u, kSd ? 0u : 1u,
                                         (uint32_t)(nbox * kBoxCols), kTcM);
    const uint32_t a0 = ptx::smem_addr(sm.a), b0 = ptx::smem_addr(sm.b);
    const uint64_t adesc = kSd ? ptx::smem_desc_noswizzle_u32(a0, 16, kSdSbo) | ((uint64_t)kLayoutSw128 << 61)
                                          : ptx::smem_desc_noswizzle_u32(a0, kLbo, kSbo);
    const uint64_t bdesc = kSd ? ptx::smem_desc_noswizzle_u32(b0, 16, kSdSbo) | ((uint64_t)kLayoutSw128 << 61)
                                          : ptx::smem_desc_noswizzle_u32(b0, kBox, 1024) | ((uint64_t)kLayoutSw128 << 61);
    // (a batch's list names every tile of its rows, with the halves that hold rows)
    uint32_t s = 0, ph = 0;
    int i = 0;
    for (; i < nstages; i++) {
      if (!ptx::mbar_wait_warp(&sm.full[s], ph)) {
        if (leader) {
          atomicCAS(&g_tc_error, 0, 3);
          sm.abort = 1;
        }
        break;
      }
      ptx::tc_fence_after_sync();
      const uint64_t soff = (uint64_t)((s * kStageBytes) >> 4);
      const uint64_t as = adesc + soff, bs = bdesc + soff;
      if (leader) {
        if (kSd) {
#pragma unroll
          for (int h = 0; h < kHalves; h++) {
            if (!((dense_halves >> h) & 1)) break;
#pragma unroll
            for (int j = 0; j < kSdK / 16; j++)  // K step j starts 32 B into the 128-byte rows
              ptx::tc_mma_f16(tmem + (uint32_t)(h * kTcN), as + (uint64_t)((h * kTcM * 128 + j * 32) >> 4),
                              bs + (uint64_t)((j * 32) >> 4), idesc, i > 0 || j > 0);
          }
        } else {
#pragma unroll
          for (int u = 0; u < kTilesPerStage; u++) {
            if (kTilesPerStage * i + u >= n) break;
#pragma unroll
            for (int h = 0; h < kHalves; h++) {
              if (!((dense_halves >> h) & 1)) break;
#pragma unroll
              for (int j = 0; j < 2; j++)  // K half j: A two core-matrix columns on, B two 8-row groups on
                ptx::tc_mma_f16(tmem + (uint32_t)(h * kTcN),
                                as + (uint64_t)((u * kATile + h * kAHalf + j * 2 * kLbo) >> 4),
                                bs + (uint64_t)((u * kBTile + j * 2 * 1024) >> 4), idesc, i > 0 || u > 0 || j > 0);
            }
          }
        }
        ptx::tc_commit(&sm.empty[s]);
      }
      __syncwarp();
      if (++s == kStages) {
        s = 0;
        ph ^= 1u;
      }
    }
    if (leader) {
      if (i > 0) ptx::tc_commit(&sm.done);
      else ptx::mbar_arrive(&sm.done);
    }
    __syncwarp();
  }

  // ---------------- epilogue (producer warps) ----------------
  // Warp w reads TMEM lanes 32*(w%4).. (a warp may only touch its own
  // quarter of the lanes) of accumulator (w/4)%2, column half w/8 of the
  // tile's 64·nbox live columns (so a narrow tile keeps all 16 warps busy);
  // a thread holds 32 columns of one output row at a time and passes them
  // through a 32x32 tile of the (now idle) stage memory, so that each store
  // instruction writes four whole 128-byte rows of C instead of 16 bytes in
  // each of 32 rows.  The SDDMM first keeps only the set bits of A's row,
  // from the row's four words loaded once.
  if (warp < kEpiWarps) {
    const int h = (warp >> 2) & 1, q = warp & 3, cg = warp >> 3;
    const bool have = (sm.seen >> h) & 1;
    // warp-uniform flags: the TMEM loads and the tile hand-off below are
    // collective over the warp
    const bool ok = __all_sync(kFull, ptx::mbar_wait(&sm.done, 0));
    if (!ok && lane == 0) {
      atomicCAS(&g_tc_error, 0, 3);
      sm.abort = 1;
    }
    ptx::tc_fence_after_sync();
    const bool wlive = __all_sync(kFull, ok && !*(volatile int*)&sm.abort);
    const int64_t rbase = row0 + h * kTcM + q * 32;  // the warp's first row
    const int64_t row = rbase + lane;
    float* cbase = gC;
    const int64_t cld = gldc;
    const int cspan = nbox * (kBoxCols / 2);      // live columns per column half (a multiple of 32)
    const int64_t ccol = col0 + cg * cspan;         // the warp's first column
    const bool live = row < out_rows && wlive;
    const uint32_t* arow = gA + row * gKw;
    const uint32_t tbase = tmem + ((uint32_t)(q * 32) << 16) + (uint32_t)(h * kTcN + cg * cspan);
    float* tile = reinterpret_cast<float*>(sm.a) + warp * 32 * kEpiStride;
    const int c8_end = cspan / 8;
    // SDDMM: the row's A words of this warp's columns (cspan = 128: four
    // words), loaded once before the stores instead of once per 32 columns
    uint32_t aw[4] = {0u, 0u, 0u, 0u};
    if (kSd && live) {
#pragma unroll
      for (int i = 0; i < 4; i++) {
        const int64_t w = ccol / 32 + i;
        if (i * 32 < cspan && w < gKw) aw[i] = __ldg(arow + w);
      }
    }
    for (int c8 = 0; c8 < c8_end; c8 += 4) {
      uint32_t r[4][8];
      if (have && ok) {
#pragma unroll
        for (int u = 0; u < 4; u++) ptx::tmem_ld_32x32b_x8(tbase + (uint32_t)((c8 + u) * 8), r[u]);
        ptx::tmem_wait_ld();
      } else {
#pragma unroll
        for (int u = 0; u < 4; u++)
#pragma unroll
          for (int v = 0; v < 8; v++) r[u][v] = 0u;
      }
      if (kSd) {
        // keep the set bits of A's row only (the row's word of these 32 columns)
        const uint32_t wbits = aw[(c8 / 4) & 3];
#pragma unroll
        for (int u = 0; u < 4; u++)
#pragma unroll
          for (int v = 0; v < 8; v++)
            if (!((wbits >> (u * 8 + v)) & 1u)) r[u][v] = 0u;
      }
      if (!wlive) continue;
      // the bit operand held 2.0 per set bit (the SDDMM's operands are both
      // dense: no scale); row `lane` of the tile
      constexpr float kScale = kSd ? 1.0f : tc::kTwoScale;
#pragma unroll
      for (int u = 0; u < 4; u++) {
        float4* t4 = reinterpret_cast<float4*>(tile + lane * kEpiStride + u * 8);
        t4[0] = make_float4(__uint_as_float(r[u][0]) * kScale, __uint_as_float(r[u][1]) * kScale,
                            __uint_as_float(r[u][2]) * kScale, __uint_as_float(r[u][3]) * kScale);
        t4[1] = make_float4(__uint_as_float(r[u][4]) * kScale, __uint_as_float(r[u][5]) * kScale,
                            __uint_as_float(r[u][6]) * kScale, __uint_as_float(r[u][7]) * kScale);
      }
      __syncwarp();
      // 8 lanes per row: rows 4*it + lane/8, 16 bytes each
      const int c4 = (lane & 7) * 4;
      const int64_t gcol = ccol + c8 * 8 + c4;
#pragma unroll
      for (int it = 0; it < 8; it++) {
        const int j = it * 4 + (lane >> 3);
        const int64_t grow = rbase + j;
        if (grow < out_rows && gcol < out_cols)
          *reinterpret_cast<float4*>(cbase + grow * cld + gcol) =
              *reinterpret_cast<const float4*>(tile + j * kEpiStride + c4);
      }
      __syncwarp();
    }
  }
  ptx::tc_fence_before_sync();
  __syncthreads();
  if (warp == kMmaWarp) {
    ptx::tc_fence_after_sync();
    ptx::tmem_dealloc(tmem, kTmemCols);
  }
}

// B (fwd) or G (trans) [R][N] of 16-bit values -> the shared-memory order
// of the tensor-core kernel's B stage, so that a tile arrives by one
// contiguous bulk copy instead of four tensor boxes of 32 rows: block (t, cb)
// (16 KB, t = 32-row tile, cb = 256-column block) holds four 64-column atoms
// of 4 KB; in atom j, row r occupies 128 bytes whose 16-byte chunk c sits at
// position c ^ (r % 8) (the 128-byte swizzle, as a TMA load into a
// 1024-byte aligned stage writes it).  Rows past R and columns past N are
// zero.
// One thread per 16-byte chunk: a warp reads 512 contiguous bytes of one row
// and writes four 128-byte runs.  VEC: B's rows take 16-byte loads; otherwise
// the elements are read one by one, and `flag` is set if any of them is an
// infinity or a NaN (exp_mask: the type's exponent bits) or is nonzero with
// less than the exponent bits exp_min.
template <bool VEC>
__global__ void __launch_bounds__(256) k_tile_b(const uint8_t* __restrict__ B, int64_t R, int64_t N, int64_t ldb,
                                                int64_t ntiles, int64_t ncb, uint4* __restrict__ bt, uint32_t exp_mask,
                                                uint32_t exp_min, int* flag) {
  const int64_t total = ntiles * ncb * (kBTile / 16);
  bool bad = false;
  for (int64_t e = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; e < total; e += (int64_t)gridDim.x * blockDim.x) {
    const int64_t blk = e >> 10;
    const int in = (int)(e & 1023);
    const int r = in >> 5, j = (in >> 3) & 3, c = in & 7;
    const int64_t t = blk / ncb, cb = blk - t * ncb;
    const int64_t row = t * kTcK + r, col = cb * kTcN + j * kBoxCols + c * 8;
    uint4 v = make_uint4(0u, 0u, 0u, 0u);
    if (VEC) {
      if (row < R && col < N) v = __ldg(reinterpret_cast<const uint4*>(B + (row * ldb + col) * 2));
    } else if (row < R && col < N) {
      const uint16_t* p = reinterpret_cast<const uint16_t*>(B) + row * ldb + col;
      uint32_t w[8];
#pragma unroll
      for (int i = 0; i < 8; i++) {
        w[i] = col + i < N ? (uint32_t)__ldg(p + i) : 0u;
        const uint32_t e = w[i] & exp_mask;
        bad |= e == exp_mask || (e < exp_min && (w[i] & 0x7fffu) != 0u);
      }
      v = make_uint4(w[0] | (w[1] << 16), w[2] | (w[3] << 16), w[4] | (w[5] << 16), w[6] | (w[7] << 16));
    }
    bt[blk * 1024 + j * 256 + r * 8 + (c ^ (r & 7))] = v;
  }
  if (!VEC && bad) *flag = 1;
}

// FP32 B [R][N] as three BF16 parts in tile order: part p of column c is column
// p*Np + c of the tiles (Np = N rounded up to 8).  x = h + m + l exactly (the
// split of Henry, Tang and Heinecke, Leveraging the bfloat16 Artificial
// Intelligence Datatype For Higher-Precision Computations, ARITH 2019): each part
// takes the next 8 bits of the significand, rounded, and what is left of
// 24 bits after two of them fits the third, as long as no part leaves BF16's
// normal range: a column with an x that is not 0 or in [2^-100, 2^100), an infinity
// or a NaN does not pass (k_parts_stats).
//
// The tensor cores' sums are cut off towards zero at 24 bits, after every 16
// products.  That costs nothing while the first parts' 8 bits add up exactly,
// that is for values of at least 2^(E - 16), 2^E being where the sums are; each
// smaller one costs up to a unit of the last place, always towards zero, where
// the walk rounds every addend to nearest.  The walk's error grows with the square
// root of the addends, so the product keeps below it while a column has at most
// 0.7 of that root of such values in a sum; one column with more of them leaves
// the product to the walk.  (Values in [1,2), a fraction of them times 2^-9 to
// 2^-18, all positive, six sizes from 512x512 to 2048x4096 at 10 to 95 %: just
// inside the limit the errors against FP64 are 0.12 to 1.0 of the walk's, normal
// values 0.05 to 0.2.)
//
// Rows past R are zero; columns past 3 Np stay as they are (each column of a
// product depends on its own alone).  Bound by memory: 4 bytes in, 6 out per
// value.
template <bool VEC>
__global__ void __launch_bounds__(256) k_split_b(const float* __restrict__ B, int64_t R, int64_t N, int64_t ldb,
                                                 int64_t ntiles, int64_t ncb, uint4* __restrict__ bt,
                                                 PartsStats st) {
  const uint32_t q = (uint32_t)((N + 7) / 8);
  const int64_t rows = ntiles * kTcK;
  for (uint32_t c8 = blockIdx.x * blockDim.x + threadIdx.x; c8 < q; c8 += gridDim.x * blockDim.x) {
    const int64_t col = (int64_t)c8 * 8;
    if (__ldg(st.bad + c8)) {
      *st.flag = 1;
      return;
    }
    for (int64_t row = blockIdx.y; row < rows; row += gridDim.y) {
      float x[8];
#pragma unroll
      for (int i = 0; i < 8; i++) x[i] = 0.f;
      if (row < R) {
        const float* p = B + row * ldb + col;
        if (VEC && col + 8 <= N) {
          const float4 u = __ldg(reinterpret_cast<const float4*>(p)), v = __ldg(reinterpret_cast<const float4*>(p) + 1);
          x[0] = u.x, x[1] = u.y, x[2] = u.z, x[3] = u.w;
          x[4] = v.x, x[5] = v.y, x[6] = v.z, x[7] = v.w;
        } else {
#pragma unroll
          for (int i = 0; i < 8; i++)
            if (col + i < N) x[i] = __ldg(p + i);
        }
      }
#pragma unroll
      for (int part = 0; part < 3; part++) {
        uint32_t w[4];
#pragma unroll
        for (int i = 0; i < 4; i++) {
          const __nv_bfloat162 b = __floats2bfloat162_rn(x[2 * i], x[2 * i + 1]);
          w[i] = *reinterpret_cast<const uint32_t*>(&b);
          x[2 * i] -= __low2float(b);
          x[2 * i + 1] -= __high2float(b);
        }
        const int64_t c = ((int64_t)part * q + c8) * 8, cb = c / kTcN;
        const int in = (int)(c - cb * kTcN), j = in / kBoxCols, ch = (in % kBoxCols) / 8, r = (int)(row % kTcK);
        bt[((row / kTcK) * ncb + cb) * 1024 + j * 256 + r * 8 + (ch ^ (r & 7))] = make_uint4(w[0], w[1], w[2], w[3]);
      }
    }
  }
}

// 16-bit B [R][N] (16-byte rows, N a multiple of 8) as two parts in tile order,
// for int8 A: x = h + l exactly, h the leading bits of its significand (4 of
// BF16's 8, 6 of FP16's 11; keep: the mask of them), cut off, so that 7 bits of A
// and h's still add up exactly where the tensor cores' sums are cut off.  Part p
// of column c is column p*N + c of the tiles.  What is not finite is h alone.
// Errors against FP64 of 4096x4096x256 at 5 %, as planes, values as they are and
// values with two parts: BF16 3.5e-8, 4.0e-8, 2.9e-8, FP16 4.3e-8, 8.2e-8,
// 3.7e-8; 96, 23 and 38 us.  Bound by memory: 2 bytes in, 4 out per value.
template <typename T2>
__global__ void __launch_bounds__(256) k_split16_b(const uint16_t* __restrict__ B, int64_t R, int64_t N, int64_t ldb,
                                                   int64_t ntiles, int64_t ncb, uint4* __restrict__ bt, uint32_t keep,
                                                   uint32_t exp_mask) {
  const uint32_t q = (uint32_t)(N / 8);
  const int64_t rows = ntiles * kTcK;
  for (int64_t row = blockIdx.y; row < rows; row += gridDim.y) {
    for (uint32_t c8 = blockIdx.x * blockDim.x + threadIdx.x; c8 < q; c8 += gridDim.x * blockDim.x) {
      uint4 x = make_uint4(0u, 0u, 0u, 0u);
      if (row < R) x = __ldg(reinterpret_cast<const uint4*>(B + row * ldb + (int64_t)c8 * 8));
      const uint32_t in4[4] = {x.x, x.y, x.z, x.w};
      uint32_t w[2][4];
#pragma unroll
      for (int i = 0; i < 4; i++) {
        uint32_t mask = keep | (keep << 16);
        if ((in4[i] & exp_mask) == exp_mask) mask |= 0xffffu;
        if (((in4[i] >> 16) & exp_mask) == exp_mask) mask |= 0xffff0000u;
        w[0][i] = in4[i] & mask;
        const T2 l = __hsub2(*reinterpret_cast<const T2*>(&in4[i]), *reinterpret_cast<const T2*>(&w[0][i]));
        w[1][i] = *reinterpret_cast<const uint32_t*>(&l);
        if ((in4[i] & exp_mask) == exp_mask) w[1][i] &= 0xffff0000u;
        if (((in4[i] >> 16) & exp_mask) == exp_mask) w[1][i] &= 0xffffu;
      }
#pragma unroll
      for (int part = 0; part < 2; part++) {
        const int64_t c = ((int64_t)part * q + c8) * 8, cb = c / kTcN;
        const int in = (int)(c - cb * kTcN), j = in / kBoxCols, ch = (in % kBoxCols) / 8, r = (int)(row % kTcK);
        bt[((row / kTcK) * ncb + cb) * 1024 + j * 256 + r * 8 + (ch ^ (r & 7))] =
            make_uint4(w[part][0], w[part][1], w[part][2], w[part][3]);
      }
    }
  }
}

// C = (Σ_z l + Σ_z m) + Σ_z h over the splits z (ascending), from the parts'
// products side by side (rows of PARTS*Np floats); four columns per thread.
template <int PARTS>
__global__ void __launch_bounds__(256) k_join_parts(const float* __restrict__ part, int64_t Np, int64_t stride,
                                                    int splits, int64_t rows, int64_t cols, float* __restrict__ C,
                                                    int64_t ldc, bool c_vec, const int* __restrict__ skip_if) {
  if (skip_if && __ldg(skip_if)) return;
  const uint32_t q = (uint32_t)((cols + 3) / 4);
  for (int64_t r = blockIdx.y; r < rows; r += gridDim.y) {
    for (uint32_t c4 = blockIdx.x * blockDim.x + threadIdx.x; c4 < q; c4 += gridDim.x * blockDim.x) {
      const int64_t c = (int64_t)c4 * 4;
      float4 sum = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
      for (int p = PARTS - 1; p >= 0; p--) {
        const float* at = part + r * PARTS * Np + p * Np + c;
        float4 acc = __ldg(reinterpret_cast<const float4*>(at));
        for (int z = 1; z < splits; z++) {
          const float4 v = __ldg(reinterpret_cast<const float4*>(at + z * stride));
          acc.x += v.x;
          acc.y += v.y;
          acc.z += v.z;
          acc.w += v.w;
        }
        sum.x += acc.x;
        sum.y += acc.y;
        sum.z += acc.z;
        sum.w += acc.w;
      }
      float* o = C + r * ldc + c;
      if (c_vec) {
        *reinterpret_cast<float4*>(o) = sum;
      } else {
        o[0] = sum.x;
        if (c + 1 < cols) o[1] = sum.y;
        if (c + 2 < cols) o[2] = sum.z;
        if (c + 3 < cols) o[3] = sum.w;
      }
    }
  }
}

// Both occupancy bitmaps in one pass over A's words.  A block of 4 warps
// covers 128 rows x 32 word columns: thread (warp j, lane l) ORs the 32 rows
// of row tile 4·blockIdx.y + j in word column 32·blockIdx.x + l (coalesced
// across the lanes).  Forward: the OR of the 4 warps is the (128-row block,
// K tile) bit, and the 32 lanes' bits are one occupancy word (one ballot).
// Transposed: the OR of 4 neighbouring lanes is the (row tile, 128-column
// block) bit of Aᵀ's bitmap, set with atomicOr (the bitmap is zeroed first;
// a bit that was not yet set is counted).
__global__ void __launch_bounds__(128) k_occupancy_both(const uint32_t* __restrict__ A, int64_t M, int64_t Kw,
                                                        int ow, uint32_t* __restrict__ occ, int owt, int64_t nkb,
                                                        uint32_t* __restrict__ occT, unsigned long long* count,
                                                        unsigned long long* countT) {
  __shared__ uint32_t s_or[4][32];
  const int lane = threadIdx.x & 31, j = threadIdx.x >> 5;
  const int64_t w = (int64_t)blockIdx.x * 32 + lane;
  const int64_t rb = blockIdx.y, rt = rb * 4 + j;
  uint32_t acc = 0;
  if (w < Kw) {
    const int64_t r0 = rt * 32, r1 = min(M, r0 + 32);
    for (int64_t r = r0; r < r1; r++) acc |= __ldg(A + r * Kw + w);
  }
  s_or[j][lane] = acc;
  // transposed bitmap: 8 column blocks of 4 words per warp
  uint32_t g = acc | __shfl_xor_sync(kFull, acc, 1);
  g |= __shfl_xor_sync(kFull, g, 2);
  const int64_t kb = w >> 2;
  if ((lane & 3) == 0 && g != 0u && kb < nkb && rt * 32 < M) {
    const uint32_t bit = 1u << (rt & 31);
    const uint32_t old = atomicOr(occT + kb * owt + (rt >> 5), bit);
    if (countT && !(old & bit)) atomicAdd(countT, 1ull);
  }
  __syncthreads();
  if (j == 0) {
    const uint32_t v = s_or[0][lane] | s_or[1][lane] | s_or[2][lane] | s_or[3][lane];
    const uint32_t m = __ballot_sync(kFull, v != 0u);
    if (lane == 0) {
      occ[rb * ow + blockIdx.x] = m;
      if (count && m) atomicAdd(count, (unsigned long long)__popc(m));
    }
  }
}

}  // namespace

int tc_occupancy_words(int64_t K) { return (int)ceil_div(ceil_div(K, 32), 32); }
int64_t tc_max_reduction() { return (int64_t)kListMax * kTcK; }
int tc_occupancy_t_words(int64_t M) { return (int)ceil_div(ceil_div(M, 32), 32); }

// words [M][Kw] -> At [Kw][M] through 32x32 shared-memory tiles (coalesced
// on both sides), every word unshuffled (tc_common.cuh), as the persistent
// kernel's producers take it.
__global__ void __launch_bounds__(256) k_transpose_words(const uint32_t* __restrict__ w, int64_t M, int64_t Kw,
                                                         uint32_t* __restrict__ At) {
  __shared__ uint32_t tile[32][33];
  const int64_t c0 = (int64_t)blockIdx.x * 32, r0 = (int64_t)blockIdx.y * 32;
  const int tx = threadIdx.x & 31, ty = threadIdx.x >> 5;
  for (int k = ty; k < 32; k += 8) {
    const int64_t r = r0 + k, c = c0 + tx;
    tile[k][tx] = (r < M && c < Kw) ? __ldg(w + r * Kw + c) : 0u;
  }
  __syncthreads();
  for (int k = ty; k < 32; k += 8) {
    const int64_t c = c0 + k, r = r0 + tx;
    if (c < Kw && r < M) At[c * M + r] = tc::unshuffle32(tile[tx][k]);
  }
}

int launch_transpose_words(const uint32_t* words, int64_t M, int64_t Kw, uint32_t* At, cudaStream_t s) {
  if (M == 0 || Kw == 0) return BSP_OK;
  if (ceil_div(M, 32) > 65535) return BSP_ERR_CAPACITY;
  k_transpose_words<<<dim3((unsigned)ceil_div(Kw, 32), (unsigned)ceil_div(M, 32)), 256, 0, s>>>(words, M, Kw, At);
  BSP_LAUNCHED();
  return BSP_OK;
}

int launch_occupancy(const uint32_t* A, int64_t M, int64_t K, uint32_t* occ, uint32_t* occT,
                     unsigned long long* count, unsigned long long* countT, cudaStream_t s) {
  const int64_t Kw = ceil_div(K, 32);
  const int ow = tc_occupancy_words(K), owt = tc_occupancy_t_words(M);
  const int64_t nkb = ceil_div(K, kTcM), nrb = ceil_div(M, kTcM);
  if (M == 0 || K == 0) return BSP_OK;
  if (nrb > 65535) return BSP_ERR_CAPACITY;
  BSP_CUDA(cudaMemsetAsync(occT, 0, sizeof(uint32_t) * (size_t)nkb * owt, s));
  k_occupancy_both<<<dim3((unsigned)ow, (unsigned)nrb), 128, 0, s>>>(A, M, Kw, ow, occ, owt, nkb, occT, count,
                                                                      countT);
  BSP_LAUNCHED();
  return BSP_OK;
}

namespace {

// cuTensorMapEncodeTiled through the runtime's driver entry point (no
// link-time dependency on the driver library).
PFN_cuTensorMapEncodeTiled_v12000 encode_tiled() {
  static PFN_cuTensorMapEncodeTiled_v12000 fn = nullptr;
  if (!fn) {
    void* p = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPointByVersion("cuTensorMapEncodeTiled", &p, 12000, cudaEnableDefault, &q) ==
            cudaSuccess &&
        q == cudaDriverEntryPointSuccess)
      fn = reinterpret_cast<PFN_cuTensorMapEncodeTiled_v12000>(p);
  }
  return fn;
}

// 2-D map over a row-major [rows][cols] 16-bit matrix (row stride ld
// elements), box = box_cols x box_rows, out-of-range = zero.
int make_map(CUtensorMap* m, const void* base, int dt, int64_t rows, int64_t cols, int64_t ld, uint32_t box_cols,
             uint32_t box_rows, CUtensorMapSwizzle swz) {
  PFN_cuTensorMapEncodeTiled_v12000 enc = encode_tiled();
  if (!enc) return BSP_ERR_UNSUPPORTED;
  const cuuint64_t dims[2] = {(cuuint64_t)(cols > 0 ? cols : 1), (cuuint64_t)(rows > 0 ? rows : 1)};
  const cuuint64_t strides[1] = {(cuuint64_t)ld * 2};
  const cuuint32_t box[2] = {box_cols, box_rows};
  const cuuint32_t estr[2] = {1, 1};
  const CUresult r = enc(m, dt == BSP_BF16 ? CU_TENSOR_MAP_DATA_TYPE_BFLOAT16 : CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 2,
                         const_cast<void*>(base), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                         swz, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                         CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  return r == CUDA_SUCCESS ? BSP_OK : BSP_ERR_ALIGNMENT;
}

static_assert(sizeof(TcSmem) + kSmemAlign <= 232448, "stage ring exceeds the shared memory of a CTA");
static_assert(kEpiWarps * 32 * kEpiStride * (int)sizeof(float) <= kRingBytes,
              "epilogue tiles exceed the stage memory");

template <typename BT, int MODE, int TPS>
int launch_mode(const TcArgs& a, const CUtensorMap& ma, const CUtensorMap& mb, dim3 grid, cudaStream_t s) {
  const size_t smem = sizeof(TcSmem) + kSmemAlign;
  static bool configured[64] = {};
  int dev = 0;
  BSP_CUDA(cudaGetDevice(&dev));
  if (dev < 64 && !configured[dev]) {
    BSP_CUDA(cudaFuncSetAttribute(k_spmm_tc<BT, MODE, TPS>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    configured[dev] = true;
  }
  k_spmm_tc<BT, MODE, TPS><<<grid, tc_threads(TPS), smem, s>>>(a, ma, mb);
  BSP_LAUNCHED();
  return BSP_OK;
}

// C = Σ_z part[z] in ascending z (deterministic), four columns per thread
// (part's rows are a multiple of four floats; c_vec: C's take 16-byte stores).
__global__ void __launch_bounds__(256) k_split_reduce(const float* __restrict__ part, int64_t ldp, int64_t stride,
                                                      int splits, int64_t rows, int64_t cols, float* __restrict__ C,
                                                      int64_t ldc, bool c_vec) {
  const int64_t q = (cols + 3) / 4, total = rows * q;
  for (int64_t e = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; e < total; e += (int64_t)gridDim.x * blockDim.x) {
    const int64_t r = e / q, c = (e - r * q) * 4;
    float4 acc = __ldg(reinterpret_cast<const float4*>(part + r * ldp + c));
    for (int z = 1; z < splits; z++) {
      const float4 v = __ldg(reinterpret_cast<const float4*>(part + z * stride + r * ldp + c));
      acc.x += v.x;
      acc.y += v.y;
      acc.z += v.z;
      acc.w += v.w;
    }
    float* o = C + r * ldc + c;
    if (c_vec) {
      *reinterpret_cast<float4*>(o) = acc;
    } else {
      o[0] = acc.x;
      if (c + 1 < cols) o[1] = acc.y;
      if (c + 2 < cols) o[2] = acc.z;
      if (c + 3 < cols) o[3] = acc.w;
    }
  }
}

}  // namespace

// Split-K for the tensor-core products: when the output has fewer items
// than half the SMs, the reduction (list of occupied tiles) is cut into S
// slices, up to 8 and at least 16 reduction tiles each, so that about one CTA
// per SM runs; every slice's FP32 partial needs rows x round4(cols) floats.
int tc_split_count(int64_t out_rows, int64_t out_cols, int64_t red_tiles) {
  const int64_t tiles = ceil_div(out_rows, ts_item_rows()) * ceil_div(out_cols, ts_item_cols());
  const int64_t sms = num_sms();
  if (tiles == 0 || tiles * 2 > sms) return 1;
  int64_t S = sms / tiles;
  if (S > 8) S = 8;
  if (S > red_tiles / 16) S = red_tiles / 16;
  return S < 1 ? 1 : (int)S;
}

size_t tc_split_bytes(int64_t out_rows, int64_t out_cols, int64_t red_tiles) {
  const int S = tc_split_count(out_rows, out_cols, red_tiles);
  return S > 1 ? (size_t)S * (size_t)out_rows * (size_t)(ceil_div(out_cols, 4) * 4) * sizeof(float) + 256 : 0;
}

// B (or G) in tile order: every (32-row tile, 256-column block) is 16 KB.
size_t tc_tiled_b_bytes(int64_t red_rows, int64_t cols) {
  return (size_t)ceil_div(red_rows, kTcK) * (size_t)ceil_div(cols, kTcN) * kBTile + 2048;
}

// Tiling B costs a read and a write of it; it pays where many row blocks
// read every B tile.  Copy included, against boxes: 64 row blocks
// (16384x16384x2048) 556 and 652 us, 32 (8192x8192x512) 52 and 58, 16
// (4096x4096x8192) 180 and 186, 8 (2048x2048x1024) 20.3 and 18.6, 4 13.8 and
// 12.5.
constexpr int64_t kTiledMinRowBlocks = 16;

// Not of a small product, where the copy's launch costs more than it saves
// (10 % bits, BF16, tiled and not: 16384x1024x256 14.3 and 13.7 us,
// 4096x4096x256 18.5 and 17.5, x512 24.6 and 24.3, x1024 31.2 and 32.3), nor
// of int8 values, whose producers bound the kernel (4096x4096x256 20.8 and
// 18.7 us, x1024 41.3 and 37.6, x4096 144.9 and 131.7).
constexpr double kTiledMinWork = 6e9;  // rows x columns x reduction

// Stages (of four K tiles) between two additions in FP32 where a product that
// the walk would form, rounded to nearest, goes to the tensor cores, whose sums
// are cut off after every 16 products.  Errors against FP64 (Frobenius norm,
// FP16 normals; walk, no segments, segments by this rule) and times without and
// with segments: 16384x1024x1000 at 20 % 2.1e-8, 2.8e-8, 2.1e-8, 72 and 82 us;
// 4096x4096x512 at 24 % 5.5e-8, 6.1e-8, 4.7e-8, 42 and 44; 8192x8192x1000 7.9e-8,
// 2.1e-7, 6.0e-8, 123 and 154.  Four stages there 6.3e-8 and 193 us, eight at
// K = 1024 2.8e-8 (one segment): the short form up to 2048 only.
int seg_stages(int64_t red_tiles) { return red_tiles <= 64 ? 4 : 8; }

bool tc_tiles_b(int64_t out_rows) { return ceil_div(out_rows, ts_item_rows()) >= kTiledMinRowBlocks; }

// FP32 output with 16-byte rows.
static size_t one_part_bytes(int64_t rows, int64_t cols) {
  return (size_t)rows * (size_t)(ceil_div(cols, 4) * 4) * sizeof(float) + 256;
}

size_t tc_preferred_bytes(int64_t out_rows, int64_t out_cols, int64_t red_rows, bool any_layout) {
  size_t sums = tc_split_bytes(out_rows, out_cols, ceil_div(red_rows, kTcK));
  if (sums == 0 && any_layout && out_cols % 4 != 0) sums = one_part_bytes(out_rows, out_cols);
  return sums + (tc_tiles_b(out_rows) || out_cols % 8 != 0 ? tc_tiled_b_bytes(red_rows, out_cols) : 0);
}

size_t tc_unaligned_bytes(int64_t out_rows, int64_t out_cols, int64_t red_rows) {
  size_t sums = tc_split_bytes(out_rows, out_cols, ceil_div(red_rows, kTcK));
  if (sums == 0 && out_cols % 4 != 0) sums = one_part_bytes(out_rows, out_cols);
  return sums + tc_tiled_b_bytes(red_rows, out_cols);
}

namespace {

// BSP_TC_TILED_B=0 keeps B on tensor boxes even with room for the tiled copy.
bool tiled_b_enabled() {
  static const bool on = [] {
    const char* e = getenv("BSP_TC_TILED_B");
    return !(e && e[0] == '0');
  }();
  return on;
}

// C = A·B (trans: dX = Aᵀ·G) on the persistent kernel: split-K and B in tile
// order as far as the workspace goes.
int launch_product(TsArgs a, const void* B, int64_t ldb, bool vec, bool trans, cudaStream_t s, void* ws,
                   size_t ws_bytes, TcForm form, const int** skipped) {
  const int64_t rows = trans ? a.K : a.M, cols = a.N, red_rows = trans ? a.M : a.K;
  if (rows == 0 || cols == 0) return BSP_OK;
  if (a.bdt != BSP_BF16 && a.bdt != BSP_F16) return BSP_ERR_UNSUPPORTED;
  if (a.N > INT32_MAX || a.M > INT32_MAX || a.K > INT32_MAX) return BSP_ERR_CAPACITY;
  // an item's tile list holds every reduction tile (fwd: K, trans: M)
  if (ceil_div(red_rows, kTcK) > kListMax) return BSP_ERR_CAPACITY;
  const size_t tiled_bytes = tc_tiled_b_bytes(red_rows, cols);
  if (!vec && (!ws || ws_bytes < tiled_bytes)) return BSP_ERR_WORKSPACE;
  int splits = 1;
  size_t used = 0;
  if (ws && form.split != 0) {
    const int64_t red_tiles = ceil_div(red_rows, kTcK);
    const int S = tc_split_count(rows, cols, red_tiles);
    const size_t bytes = tc_split_bytes(rows, cols, red_tiles);
    if (S > 1 && ws_bytes >= bytes + (vec ? 0 : tiled_bytes)) {
      splits = S;
      a.part = reinterpret_cast<float*>((reinterpret_cast<uintptr_t>(ws) + 255) & ~(uintptr_t)255);
      a.ldp = ceil_div(cols, 4) * 4;
      a.part_stride = rows * a.ldp;
      used = bytes;
    }
  }
  if (!vec) {
    a.seg_stages = seg_stages(ceil_div(red_rows, kTcK));
    // Sums of segments leave by TMA, which adds 16 bytes at a time: where C's rows
    // do not start on 16 bytes, to a copy that does, as far as there is room
    // (8192x8192x1001: 338 us by single additions to C).
    const size_t bytes = one_part_bytes(rows, cols);
    if (splits == 1 && !a.c_vec && ws && ws_bytes >= bytes + tiled_bytes) {
      a.part = reinterpret_cast<float*>((reinterpret_cast<uintptr_t>(ws) + 255) & ~(uintptr_t)255);
      a.ldp = ceil_div(cols, 4) * 4;
      a.part_stride = rows * a.ldp;
      used = bytes;
    }
  }
  // B in tile order when the rest of the workspace holds it (else tensor boxes)
  const bool room = ws && ws_bytes >= used + tiled_bytes;
  const bool tiled = !vec || (room && (form.tiled >= 0 ? form.tiled == 1
                                                            : tc_tiles_b(rows) && tiled_b_enabled() &&
                                                                  !a.tiles &&
                                                                  (double)rows * (double)cols * (double)red_rows >= kTiledMinWork));
  CUtensorMap map;
  memset(&map, 0, sizeof(map));
  if (tiled) {
    // the blocks of tile order, behind a head that holds the flag
    const int64_t ntiles = ceil_div(red_rows, kTcK), ncb = ceil_div(cols, kTcN);
    uint8_t* bt = reinterpret_cast<uint8_t*>(
        (reinterpret_cast<uintptr_t>(static_cast<char*>(ws) + used) + 256 + 1023) & ~(uintptr_t)1023);
    int* flag = reinterpret_cast<int*>(bt - 256);
    const int64_t work = ntiles * ncb * (kBTile / 16);
    const int64_t cap = (int64_t)num_sms() * 16;
    const unsigned grid = (unsigned)(ceil_div(work, 256) < cap ? ceil_div(work, 256) : cap);
    if (vec) {
      k_tile_b<true><<<grid, 256, 0, s>>>(static_cast<const uint8_t*>(B), red_rows, cols, ldb, ntiles, ncb,
                                          reinterpret_cast<uint4*>(bt), 0u, 0u, nullptr);
    } else {
      BSP_CUDA(cudaMemsetAsync(flag, 0, sizeof(int), s));
      k_tile_b<false><<<grid, 256, 0, s>>>(static_cast<const uint8_t*>(B), red_rows, cols, ldb, ntiles, ncb,
                                           reinterpret_cast<uint4*>(bt), a.bdt == BSP_BF16 ? 0x7f80u : 0x7c00u,
                                           a.bdt == BSP_BF16 ? (127u - 100u) << 7 : 0u, flag);
      a.skip_if = flag;
      *skipped = flag;
    }
    BSP_LAUNCHED();
    a.bt = bt;
    a.bt_cb = ncb;
  } else {
    // B [K][N] (fwd) or G [M][N] (trans), 64 columns x 32 reduction rows per box
    BSP_TRY(make_map(&map, B, a.bdt, red_rows, a.N, ldb, kBoxCols, kTcK, CU_TENSOR_MAP_SWIZZLE_128B));
  }
  BSP_TRY(launch_ts(a, map, trans, splits, s));
  if (a.part) {
    const int64_t work = rows * ceil_div(cols, 4);
    const int64_t cap = (int64_t)num_sms() * 8;
    k_split_reduce<<<(unsigned)(ceil_div(work, 256) < cap ? ceil_div(work, 256) : cap), 256, 0, s>>>(
        a.part, a.ldp, a.part_stride, splits, rows, cols, a.C, a.ldc, a.c_vec);
    BSP_LAUNCHED();
  }
  return BSP_OK;
}
}  // namespace

// The room that an FP32 product on the tensor cores takes: the parts' products, B's parts in tile order.
static int64_t parts_cols(int64_t N) { return ceil_div(N, 8) * 8; }
size_t tc_parts_bytes(int64_t out_rows, int64_t N, int64_t red_rows) {
  const int64_t n3 = 3 * parts_cols(N);
  const int S = tc_split_count(out_rows, n3, ceil_div(red_rows, kTcK));
  return (size_t)S * (size_t)out_rows * (size_t)n3 * sizeof(float) + 256 + parts_stats_bytes(N) +
         tc_tiled_b_bytes(red_rows, n3);
}

template <int PARTS>
static int launch_join(const float* part, int64_t Np, int64_t stride, int splits, int64_t rows, int64_t N, float* C,
                       int64_t ldc, const int* skip_if, cudaStream_t s) {
  const int64_t q = ceil_div(N, 4);
  const unsigned t = q >= 256 ? 256 : (unsigned)(ceil_div(q, 32) * 32);
  const unsigned gx = (unsigned)(ceil_div(q, t) < 1024 ? ceil_div(q, t) : 1024);
  const bool c_vec = is_aligned(C, 16) && ldc % 4 == 0 && N % 4 == 0;
  k_join_parts<PARTS><<<dim3(gx, (unsigned)(rows < 65535 ? rows : 65535)), t, 0, s>>>(part, Np, stride, splits, rows, N,
                                                                                    C, ldc, c_vec, skip_if);
  BSP_LAUNCHED();
  return BSP_OK;
}

// C = A·B (trans: dX = Aᵀ·G) for FP32 B on the tensor cores, exact in B: its
// three BF16 parts are multiplied as 3N columns, each with accumulators of its
// own, and joined afterwards.  2048x2048x1024 at 10 %: walk 85 us, here 56, two
// of them to look at the columns.  Bound there by the tensor kernel's producers,
// below about 1024x1024x1024 by its launches.
// Errors against FP64, relative in the Frobenius norm, walk and here:
// normal values 2.6e-7 and 2.7e-8, their magnitudes 2.2e-7 and 3.5e-8
// (512x512x256 9.7e-8 and 2.5e-8, 1024x4096x512 3.7e-7 and 2.8e-8): the first
// part's 8 bits add up nearly exactly.
static int launch_parts(TsArgs a, int64_t nnz, const float* B, int64_t ldb, int64_t N, float* C, int64_t ldc, bool trans,
                        cudaStream_t s, void* ws, size_t ws_bytes, const int** skipped) {
  const int64_t rows = trans ? a.K : a.M, red_rows = trans ? a.M : a.K;
  if (a.M > INT32_MAX || a.K > INT32_MAX || N > INT32_MAX / 4) return BSP_ERR_CAPACITY;
  if (ceil_div(red_rows, kTcK) > kListMax) return BSP_ERR_CAPACITY;
  if (!ws || ws_bytes < tc_parts_bytes(rows, N, red_rows)) return BSP_ERR_WORKSPACE;
  const int64_t Np = parts_cols(N), n3 = 3 * Np, ntiles = ceil_div(red_rows, kTcK), ncb = ceil_div(n3, kTcN);
  const int splits = tc_split_count(rows, n3, ntiles);
  float* part = reinterpret_cast<float*>((reinterpret_cast<uintptr_t>(ws) + 255) & ~(uintptr_t)255);
  float* stats_ws = part + (int64_t)splits * rows * n3;
  uint8_t* bt = reinterpret_cast<uint8_t*>(
      (reinterpret_cast<uintptr_t>(stats_ws) + parts_stats_bytes(N) + 1023) & ~(uintptr_t)1023);
  // Segments only where sums are long: normal values pass the columns' limits up
  // to some 1500 addends.  A sum has an average row's bits of a slice or a segment,
  // and a quarter more.  (3000x4096x1000 at 50 %: 85 us and 3.3e-7 for magnitudes
  // of normals without segments, 120 and 5.5e-8 with them, the walk 990 and 6.5e-7.)
  const double bits = (double)nnz / (double)rows;
  a.seg_stages = bits <= 1024.0 ? 0 : bits > 0.55 * (double)red_rows ? 4 : 8;
  double slice = (double)red_rows / splits;
  if (a.seg_stages && slice > a.seg_stages * 4.0 * kTcK) slice = a.seg_stages * 4.0 * kTcK;
  const double addends = 1.25 * bits * slice / (double)red_rows;
  PartsStats stats = {};
  BSP_TRY(launch_parts_stats(B, red_rows, N, ldb, stats_ws, (float)(addends > 1.0 ? addends : 1.0), &stats, s));
  int* flag = stats.flag;
  const int64_t q = Np / 8;
  const unsigned t = q >= 256 ? 256 : (unsigned)(ceil_div(q, 32) * 32);
  const unsigned gx = (unsigned)(ceil_div(q, t) < 1024 ? ceil_div(q, t) : 1024);
  const int64_t blocks = ceil_div((int64_t)num_sms() * 8, gx);
  const int64_t gy = blocks < ntiles * kTcK ? blocks : ntiles * kTcK;
  const bool vec = is_aligned(B, 16) && ldb % 4 == 0;
  (vec ? k_split_b<true> : k_split_b<false>)<<<dim3(gx, (unsigned)(gy < 65535 ? gy : 65535)), t, 0, s>>>(
      B, red_rows, N, ldb, ntiles, ncb, reinterpret_cast<uint4*>(bt), stats);
  BSP_LAUNCHED();
  a.N = n3;
  a.bdt = BSP_BF16;
  a.bt = bt;
  a.bt_cb = ncb;
  a.C = part;
  a.ldc = n3;
  a.c_vec = true;
  a.part = part;
  a.ldp = n3;
  a.part_stride = rows * n3;
  a.skip_if = flag;
  CUtensorMap map;
  memset(&map, 0, sizeof(map));
  BSP_TRY(launch_ts(a, map, trans, splits, s));
  BSP_TRY(launch_join<3>(part, Np, rows * n3, splits, rows, N, C, ldc, flag, s));
  *skipped = flag;
  return BSP_OK;
}

int launch_spmm_parts(const uint32_t* A, int64_t M, int64_t K, const uint32_t* occ, const uint32_t* At, int64_t nnz,
                      const float* B, int64_t ldb, int64_t N, float* C, int64_t ldc, bool trans, cudaStream_t s,
                      void* ws, size_t ws_bytes, const int** skipped) {
  TsArgs a = {};
  a.At = At;
  a.A = A;
  a.M = M;
  a.K = K;
  a.Kw = ceil_div(K, 32);
  a.occ = occ;
  a.occ_words = trans ? tc_occupancy_t_words(M) : tc_occupancy_words(K);
  return launch_parts(a, nnz, B, ldb, N, C, ldc, trans, s, ws, ws_bytes, skipped);
}

int launch_spmm_tc(const SpmmArgs& sa, const uint32_t* occ, const uint32_t* At, bool vec, cudaStream_t s, void* ws,
                   size_t ws_bytes, TcForm form, const int** skipped) {
  TsArgs a = {};
  a.At = At;
  a.A = sa.A;
  a.M = sa.M;
  a.K = sa.K;
  a.Kw = sa.Kw;
  a.N = sa.N;
  a.C = sa.C;
  a.ldc = sa.ldc;
  a.c_vec = sa.c_vec;
  a.occ = occ;
  a.occ_words = tc_occupancy_words(sa.K);
  a.bdt = sa.bdt;
  return launch_product(a, sa.B, sa.ldb, vec, false, s, ws, ws_bytes, form, skipped);
}

int launch_spmm_t_tc(const uint32_t* A, int64_t M, int64_t K, const void* G, int gdt, int64_t ldg, int64_t N,
                     void* dX, bool out16, int64_t lddx, const uint32_t* occT, const uint32_t* At, cudaStream_t s,
                     void* ws, size_t ws_bytes) {
  TsArgs a = {};
  a.At = At;
  a.A = A;
  a.M = M;
  a.K = K;
  a.Kw = ceil_div(K, 32);
  a.N = N;
  a.C = static_cast<float*>(dX);
  a.ldc = lddx;
  a.out16 = out16;
  a.c_vec = is_aligned(dX, 16) && lddx % 4 == 0 && N % 4 == 0;
  a.occ = occT;
  a.occ_words = tc_occupancy_t_words(M);
  a.bdt = gdt;
  const int* skipped = nullptr;  // (only vector layouts come here)
  return launch_product(a, G, ldg, true, true, s, ws, ws_bytes, TcForm{}, &skipped);
}

size_t tc_i8_bytes(int64_t M, int64_t N, int64_t K) {
  const int S = tc_split_count(M, 2 * N, ceil_div(K, kTcK));
  return (size_t)S * (size_t)M * (size_t)(2 * N) * sizeof(float) + 256 + tc_tiled_b_bytes(K, 2 * N);
}

int launch_spmm_i8_tc(const void* tiles, int64_t M, int64_t K, const void* B, int bdt, int64_t ldb, int64_t N, float* C,
                      int64_t ldc, void* ws, size_t ws_bytes, cudaStream_t s) {
  TsArgs a = {};
  a.tiles = static_cast<const uint4*>(tiles);
  a.occ = reinterpret_cast<const uint32_t*>(static_cast<const uint8_t*>(tiles) + i8_values_bytes(M, K));
  a.occ_words = tc_occupancy_words(K);
  a.M = M;
  a.K = K;
  a.Kw = ceil_div(K, 32);
  a.N = N;
  a.C = C;
  a.ldc = ldc;
  a.c_vec = true;
  a.bdt = bdt;
  if (!ws || ws_bytes < tc_i8_bytes(M, N, K) || 2 * N > ts_max_cols()) {
    const int* skipped = nullptr;
    return launch_product(a, B, ldb, true, false, s, ws, ws_bytes, TcForm{}, &skipped);
  }
  if (ceil_div(K, kTcK) > kListMax) return BSP_ERR_CAPACITY;
  const int64_t n2 = 2 * N, ntiles = ceil_div(K, kTcK), ncb = ceil_div(n2, kTcN);
  const int splits = tc_split_count(M, n2, ntiles);
  float* part = reinterpret_cast<float*>((reinterpret_cast<uintptr_t>(ws) + 255) & ~(uintptr_t)255);
  uint8_t* bt = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(part + (int64_t)splits * M * n2) + 1023) &
                                           ~(uintptr_t)1023);
  const int64_t q = N / 8;
  const unsigned t = q >= 256 ? 256 : (unsigned)(ceil_div(q, 32) * 32);
  const unsigned gx = (unsigned)(ceil_div(q, t) < 1024 ? ceil_div(q, t) : 1024);
  const int64_t blocks = ceil_div((int64_t)num_sms() * 8 * 256 / t, gx), rows = ntiles * kTcK;
  const dim3 grid(gx, (unsigned)(blocks < rows ? blocks : rows));
  if (bdt == BSP_BF16)
    k_split16_b<__nv_bfloat162><<<grid, t, 0, s>>>(static_cast<const uint16_t*>(B), K, N, ldb, ntiles, ncb,
                                                   reinterpret_cast<uint4*>(bt), 0xfff0u, 0x7f80u);
  else
    k_split16_b<__half2><<<grid, t, 0, s>>>(static_cast<const uint16_t*>(B), K, N, ldb, ntiles, ncb,
                                            reinterpret_cast<uint4*>(bt), 0xffe0u, 0x7c00u);
  BSP_LAUNCHED();
  a.N = n2;
  a.bt = bt;
  a.bt_cb = ncb;
  a.C = part;
  a.ldc = n2;
  a.part = part;
  a.ldp = n2;
  a.part_stride = M * n2;
  CUtensorMap map;
  memset(&map, 0, sizeof(map));
  BSP_TRY(launch_ts(a, map, false, splits, s));
  return launch_join<2>(part, N, M * n2, splits, M, N, C, ldc, nullptr, s);
}

int launch_sddmm_tc(const uint32_t* A, int64_t M, int64_t K, const void* G, int64_t ldg, const void* X,
                    int64_t ldx, int dt, int64_t N, float* dA, int64_t ldda, cudaStream_t s) {
  TcArgs a = {};
  a.A = A;
  a.M = M;
  a.K = K;
  a.Kw = ceil_div(K, 32);
  a.B = X;
  a.ldb = ldx;
  a.G = G;
  a.ldg = ldg;
  a.N = N;
  a.C = dA;
  a.ldc = ldda;
  a.bdt = dt;
  if (M == 0 || K == 0) return BSP_OK;
  if (dt != BSP_BF16 && dt != BSP_F16) return BSP_ERR_UNSUPPORTED;
  const dim3 grid((unsigned)ceil_div(M, kCtaM), (unsigned)ceil_div(K, kTcN));
  if (ceil_div(K, kTcN) > 65535 || ceil_div(M, kCtaM) > 0x7fffffff) return BSP_ERR_CAPACITY;
  if (N > INT32_MAX || M > INT32_MAX || K > INT32_MAX) return BSP_ERR_CAPACITY;
  // Outputs of at most half as many 256x256 tiles as SMs: 128x256 items, so that
  // twice the SMs work (2048x2048x2048 26.7 us as tiles, 17.6 as items,
  // 1024x1024x1024 17.9 and 12.5, 512x512x512 13.0 and 9.9).  Beyond that the
  // larger tile wins, for it brings in two thirds of the bytes per product
  // (3072x3072x1024 19.4 and 21.7, 1024x8192x4096 48 and 72, 4096x4096x8192
  // 167 and 236).
  if ((int64_t)grid.x * grid.y * 2 <= num_sms()) return launch_sddmm_persist(A, M, K, G, ldg, X, ldx, dt, N, dA, ldda, s);
  CUtensorMap ma, mb;
  BSP_TRY(make_map(&ma, G, dt, M, N, ldg, kSdK, kCtaM, CU_TENSOR_MAP_SWIZZLE_128B));  // G [M][N]
  BSP_TRY(make_map(&mb, X, dt, K, N, ldx, kSdK, kTcN, CU_TENSOR_MAP_SWIZZLE_128B));   // X [K][N]
  return dt == BSP_BF16 ? launch_mode<__nv_bfloat16, kSddmm, 2>(a, ma, mb, grid, s)
                        : launch_mode<__half, kSddmm, 2>(a, ma, mb, grid, s);
}

int make_batch_map(CUtensorMap* m, const void* B, int bdt, int64_t K, int64_t N, int64_t ldb) {
  return make_map(m, B, bdt, K, N, ldb, kBoxCols, kTcK, CU_TENSOR_MAP_SWIZZLE_128B);
}

int make_batch_map_sddmm(CUtensorMap* m, const void* T, int bdt, int64_t rows, int64_t N, int64_t ld,
                         int box_rows) {
  return make_map(m, T, bdt, rows, N, ld, kSdK, (uint32_t)box_rows, CU_TENSOR_MAP_SWIZZLE_128B);
}

int make_out_map16(CUtensorMap* m, void* C, int dt, int64_t rows, int64_t cols, int64_t ld) {
  PFN_cuTensorMapEncodeTiled_v12000 enc = encode_tiled();
  if (!enc) return BSP_ERR_UNSUPPORTED;
  const cuuint64_t dims[3] = {(cuuint64_t)cols, (cuuint64_t)rows, 1};
  const cuuint64_t strides[2] = {(cuuint64_t)ld * 2, (cuuint64_t)ld * 2 * (cuuint64_t)rows};
  const cuuint32_t box[3] = {64, 32, 1};
  const cuuint32_t estr[3] = {1, 1, 1};
  const CUresult r = enc(m, dt == BSP_BF16 ? CU_TENSOR_MAP_DATA_TYPE_BFLOAT16 : CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 3, C,
                         dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
                         CU_TENSOR_MAP_L2_PROMOTION_NONE, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  return r == CUDA_SUCCESS ? BSP_OK : BSP_ERR_ALIGNMENT;
}

int make_rows_map_f32(CUtensorMap* m, const float* X, int64_t rows, int64_t cols, int64_t ld, int box_cols, int box_rows) {
  PFN_cuTensorMapEncodeTiled_v12000 enc = encode_tiled();
  if (!enc) return BSP_ERR_UNSUPPORTED;
  const cuuint64_t dims[2] = {(cuuint64_t)cols, (cuuint64_t)rows};
  const cuuint64_t strides[1] = {(cuuint64_t)ld * 4};
  const cuuint32_t box[2] = {(cuuint32_t)box_cols, (cuuint32_t)box_rows};
  const cuuint32_t estr[2] = {1, 1};
  const CUresult r = enc(m, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 2, const_cast<float*>(X), dims, strides, box, estr,
                         CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE,
                         CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  return r == CUDA_SUCCESS ? BSP_OK : BSP_ERR_ALIGNMENT;
}

int make_out_map(CUtensorMap* m, float* C, int64_t rows, int64_t cols, int64_t ld, int splits, int64_t split_stride) {
  PFN_cuTensorMapEncodeTiled_v12000 enc = encode_tiled();
  if (!enc) return BSP_ERR_UNSUPPORTED;
  const cuuint64_t dims[3] = {(cuuint64_t)cols, (cuuint64_t)rows, (cuuint64_t)splits};
  const cuuint64_t strides[2] = {(cuuint64_t)ld * 4, (cuuint64_t)split_stride * 4};
  const cuuint32_t box[3] = {32, 32, 1};
  const cuuint32_t estr[3] = {1, 1, 1};
  const CUresult r = enc(m, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 3, C, dims, strides, box, estr,
                         CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_NONE,
                         CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  return r == CUDA_SUCCESS ? BSP_OK : BSP_ERR_ALIGNMENT;
}

int launch_batched_tc(const BatchProblemTc* probs, const int4* items, int n_items, int64_t N, int bdt,
                      cudaStream_t s, int kind) {
  if (n_items == 0 || N == 0) return BSP_OK;
  TcArgs a = {};
  a.N = N;
  a.bdt = bdt;
  a.bprobs = probs;
  a.items = items;
  CUtensorMap unused;
  memset(&unused, 0, sizeof(unused));
  const dim3 grid((unsigned)n_items, 1, 1);
  if (bdt != BSP_BF16 && bdt != BSP_F16) return BSP_ERR_UNSUPPORTED;
  const bool bf = bdt == BSP_BF16;
  switch (kind) {
    case 0: return bf ? launch_mode<__nv_bfloat16, kBatch, 2>(a, unused, unused, grid, s)
                      : launch_mode<__half, kBatch, 2>(a, unused, unused, grid, s);
    case 1: return bf ? launch_mode<__nv_bfloat16, kBatchT, 2>(a, unused, unused, grid, s)
                      : launch_mode<__half, kBatchT, 2>(a, unused, unused, grid, s);
    case 2: return bf ? launch_mode<__nv_bfloat16, kBatchS, 2>(a, unused, unused, grid, s)
                      : launch_mode<__half, kBatchS, 2>(a, unused, unused, grid, s);
    default: return BSP_ERR_INVALID_ARG;
  }
}

int tc_device_error(int* out, bool clear) {
  BSP_CUDA(cudaMemcpyFromSymbol(out, g_tc_error, sizeof(int)));
  if (clear) {
    const int zero = 0;
    BSP_CUDA(cudaMemcpyToSymbol(g_tc_error, &zero, sizeof(int)));
  }
  return BSP_OK;
}

}  // namespace bsp
