// spmm_batched.cu — many independent bitmap SpMMs in one tensor-core launch.
//
// A batch (bsp_batch_create) holds, in device memory, one record per problem
// (B's tensor map, encoded once on the host, and A, C, sizes) and a work list
// with one item per (problem, 256-row block, 128-column block), sorted by
// reduction length, longest first.  bsp_batched_spmm runs the list in one
// launch of the persistent tensor-core kernel (spmm_ts.cu; batches wider than
// 128 columns as 256x256 blocks of spmm_tc.cu where that is faster), with no host
// synchronisation and no allocation; it reads the item's problem from its
// record, runs every K tile of its rows (a batch has no occupancy plan) and
// streams B by TMA through the problem's own tensor map.  dX of a gradient
// batch runs on the same kernel in its transposed form, dA on the persistent
// SDDMM below.  512 problems of 64..4096 rows and columns, N = 128: 150 us, where
// a persistent kernel with the expanded bits in shared memory and a queue in
// device memory took 170 (bound by shared-memory traffic; now by the words'
// loads and expansion, 1450 cycles per four K tiles, and 3000 to 4000 cycles
// from one item's last MMA to the next one's first).
#include <algorithm>
#include <new>
#include <type_traits>
#include <cstdlib>
#include <cstring>
#include <vector>

#include "bsp_internal.cuh"
#include "ptx.cuh"
#include "spmm.cuh"
#include "tc_common.cuh"
#include "ts.cuh"

namespace bsp {

// The SDDMM's waits that ran out (the products report their own).
__device__ int g_batch_error;

int batched_device_error(int* out, bool clear) {
  BSP_CUDA(cudaMemcpyFromSymbol(out, g_batch_error, sizeof(int)));
  if (clear) {
    const int zero = 0;
    BSP_CUDA(cudaMemcpyToSymbol(g_batch_error, &zero, sizeof(int)));
  }
  return BSP_OK;
}

namespace {
constexpr int64_t kItemRows = 256, kItemCols = 256;  // the tensor-core kernel's CTA tile

constexpr int kPQ = 4;                // items known ahead
constexpr int kPEpiStride = 36;       // staging rows 36 floats apart (16-byte aligned, conflict-free)
constexpr uint32_t kPTmemCols = 512;  // two sets x 256 columns
constexpr int kPErr = 4;
constexpr size_t kPSmemAlign = 1024;

__device__ __forceinline__ void persist_fail() { atomicCAS(&g_batch_error, 0, kPErr); }

// lane 0 waits on `bar` (bounded) and reads *val; the warp gets both
__device__ __forceinline__ bool warp_wait_read(uint64_t* bar, uint32_t parity, const int* val, int* out) {
  int ok = 1, v = 0;
  if ((threadIdx.x & 31) == 0) {
    ok = ptx::mbar_wait(bar, parity) ? 1 : 0;
    if (ok && val) v = *(volatile const int*)val;
  }
  ok = __shfl_sync(kFull, ok, 0);
  if (out) *out = __shfl_sync(kFull, v, 0);
  return ok != 0;
}

// ---- persistent batched SDDMM (dA = (G·Xᵀ) ⊙ A of a gradient batch) -----
// One CTA per SM takes items — (problem, 128 rows of dA, 256 columns of dA)
// — from the batch's work queue.  Both operands are dense 16-bit tiles, so
// there are no producers: the TMA warp loads, per 64 columns of N, G's box
// (128 rows, 16 KB) and X's box (256 rows, 32 KB), K-major with the 128-byte
// swizzle; the MMA warp issues four M128 N256 K16 MMAs per stage into
// accumulator set j % 2 of item j; 8 epilogue warps (two per TMEM lane
// quarter, one per 128-column half) keep the set bits of A's rows, pass 32
// columns at a time through a staging tile and store dA rows whole.  With
// two accumulator sets an item's epilogue — the store of 128 KB of dA, the
// bound of this write-heavy product — runs under the next item's loads and
// MMAs instead of after them.  Every wait is bounded (error 4 in
// g_batch_error).
constexpr int kSdRows = 128, kSdCols = 256, kSdStep = 64, kSdStages = 3;
constexpr int kSdGBox = kSdRows * kSdStep * 2;  // 16 KB
constexpr int kSdXBox = kSdCols * kSdStep * 2;  // 32 KB
constexpr int kSdEpiWarps = 8, kSdEpiWarp0 = 2;
constexpr int kSdThreads = (kSdEpiWarp0 + kSdEpiWarps) * 32;  // 320

struct __align__(1024) SddmmSmem {
  uint8_t g[kSdStages * kSdGBox];  // 1 KB-aligned boxes (128-byte swizzle atoms)
  uint8_t x[kSdStages * kSdXBox];
  float epi[kSdEpiWarps][32 * kPEpiStride];
  uint64_t full[kSdStages], empty[kSdStages];
  uint64_t tfull[2], tempty[2];
  uint64_t qfull[kPQ], qempty[kPQ];
  int qitem[kPQ];
  uint32_t tmem_addr;
};
static_assert(sizeof(SddmmSmem) + kPSmemAlign <= 232448, "persistent SDDMM: shared memory");

// SINGLE: one problem, whose record comes as an argument; its items are dealt
// to the CTAs in turn (rows fastest), and those without a bit in A are neither
// loaded nor multiplied.
constexpr int kSdSkip = 1 << 30;

template <typename BT, bool SINGLE>
__global__ void __launch_bounds__(kSdThreads, 1)
    k_batched_sddmm_persist(const BatchProblemTc* __restrict__ probs, const int4* __restrict__ items, int n_items,
                            int* next_item, int64_t N, const __grid_constant__ BatchProblemTc one) {
  extern __shared__ __align__(1024) uint8_t smem_raw[];
  SddmmSmem& sm = *reinterpret_cast<SddmmSmem*>(
      smem_raw + ((kPSmemAlign - (ptx::smem_addr(smem_raw) & (kPSmemAlign - 1))) & (kPSmemAlign - 1)));
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int nst = (int)((N + kSdStep - 1) / kSdStep);  // stages of an item (every item reduces all of N)
  auto item = [&](int it) -> int4 {
    if (!SINGLE) return __ldg(items + it);
    const int nrb = (int)((one.M + kSdRows - 1) / kSdRows);
    return make_int4(0, it % nrb, it / nrb, 0);
  };
  if (tid == 0) {
    for (int s = 0; s < kSdStages; s++) {
      ptx::mbar_init(&sm.full[s], 1);   // the TMA transaction arrival
      ptx::mbar_init(&sm.empty[s], 1);  // tcgen05.commit of the stage's MMAs
    }
    for (int b = 0; b < 2; b++) {
      ptx::mbar_init(&sm.tfull[b], 1);
      ptx::mbar_init(&sm.tempty[b], kSdEpiWarps);
    }
    for (int q = 0; q < kPQ; q++) {
      ptx::mbar_init(&sm.qfull[q], 1);
      ptx::mbar_init(&sm.qempty[q], kSdEpiWarps);
    }
    ptx::fence_mbar_init();
  }
  if (warp == 1) {
    ptx::tmem_alloc(&sm.tmem_addr, kPTmemCols);
    ptx::tmem_relinquish();
  }
  ptx::tc_fence_before_sync();
  __syncthreads();
  ptx::tc_fence_after_sync();
  const uint32_t tmem = __reduce_max_sync(kFull, sm.tmem_addr);  // (uniform to the compiler)

  if (warp == 0) {
    // ---------------- item queue + G and X by TMA ----------------
    const bool leader = ptx::elect_one();
    const uint32_t g0 = ptx::smem_addr(sm.g), x0 = ptx::smem_addr(sm.x), f0 = ptx::smem_addr(&sm.full[0]);
    uint32_t s = 0, ph = 1;
    for (int j = 0;; j++) {
      const int q = j % kPQ;
      if (!ptx::mbar_wait_warp(&sm.qempty[q], ((uint32_t)(j / kPQ) & 1u) ^ 1u)) {
        if (leader) persist_fail();
        break;
      }
      int it = 0;
      if (SINGLE) {
        it = (int)blockIdx.x + j * (int)gridDim.x;
        bool skip = false;
        if (it < n_items) {
          const int4 b = item(it);
          uint32_t any = 0u;
#pragma unroll
          for (int r = 0; r < kSdRows / 4; r++) {  // lanes 8 r' + w: word w of row 4 r + r'
            const int64_t row = (int64_t)b.y * kSdRows + r * 4 + (lane >> 3), w = (int64_t)b.z * (kSdCols / 32) + (lane & 7);
            if (row < one.M && w < one.Kw) any |= __ldg(one.A + row * one.Kw + w);
          }
          skip = !__any_sync(kFull, any != 0u);
        }
        if (leader) {
          sm.qitem[q] = it >= n_items ? -1 : (skip ? it | kSdSkip : it);
          ptx::mbar_arrive(&sm.qfull[q]);
        }
        __syncwarp();
        if (it >= n_items) break;
        if (skip) continue;
      } else {
        if (leader) {
          it = atomicAdd(next_item, 1);
          sm.qitem[q] = it < n_items ? it : -1;
          ptx::mbar_arrive(&sm.qfull[q]);
        }
        it = __reduce_max_sync(kFull, it);
        if (it >= n_items) break;
      }
      const int4 w4 = item(it);
      const BatchProblemTc* p = SINGLE ? &one : probs + w4.x;
      if (!SINGLE && leader) {
        ptx::tensormap_acquire(&p->map3);  // written by the host into global memory
        ptx::tensormap_acquire(&p->map2);
      }
      __syncwarp();
      bool ok = true;
      for (int i = 0; i < nst; i++) {
        if (!ptx::mbar_wait_warp(&sm.empty[s], ph)) {
          ok = false;
          break;
        }
        if (leader) {
          ptx::mbar_arrive_expect_tx(&sm.full[s], (uint32_t)(kSdGBox + kSdXBox));
          ptx::tma_load_2d_u32(g0 + (uint32_t)(s * kSdGBox), &p->map3, i * kSdStep, w4.y * kSdRows, f0 + (uint32_t)s * 8u);
          ptx::tma_load_2d_u32(x0 + (uint32_t)(s * kSdXBox), &p->map2, i * kSdStep, w4.z * kSdCols, f0 + (uint32_t)s * 8u);
        }
        __syncwarp();
        if (++s == kSdStages) {
          s = 0;
          ph ^= 1u;
        }
      }
      if (!ok) {
        if (leader) persist_fail();
        break;
      }
    }
  } else if (warp == 1) {
    // ---------------- MMA issuer ----------------
    const bool leader = ptx::elect_one();
    const uint32_t ab = std::is_same<BT, __nv_bfloat16>::value ? 1u : 0u;
    const uint32_t idesc = tc::idesc_f16(ab, 0u, 0u, (uint32_t)kSdCols, (uint32_t)kSdRows);
    const uint64_t gdesc = ptx::smem_desc_noswizzle_u32(ptx::smem_addr(sm.g), 16, 1024) |
                           ((uint64_t)tc::kLayoutSw128 << 61);
    const uint64_t xdesc = ptx::smem_desc_noswizzle_u32(ptx::smem_addr(sm.x), 16, 1024) |
                           ((uint64_t)tc::kLayoutSw128 << 61);
    uint32_t s = 0, ph = 0;
    for (int j = 0;; j++) {
      if (!ptx::mbar_wait_warp(&sm.qfull[j % kPQ], (uint32_t)(j / kPQ) & 1u)) {
        if (leader) persist_fail();
        break;
      }
      const int it = __reduce_max_sync(kFull, *(volatile const int*)&sm.qitem[j % kPQ]);
      if (it < 0) break;
      const int n = SINGLE && (it & kSdSkip) ? 0 : nst;
      const int set = j & 1;
      if (!ptx::mbar_wait_warp(&sm.tempty[set], ((uint32_t)(j >> 1) & 1u) ^ 1u)) {
        if (leader) persist_fail();
        break;
      }
      ptx::tc_fence_after_sync();
      const uint32_t dset = tmem + (uint32_t)(set * kSdCols);
      bool ok = true;
      for (int i = 0; i < n; i++) {
        if (!ptx::mbar_wait_warp(&sm.full[s], ph)) {
          ok = false;
          break;
        }
        ptx::tc_fence_after_sync();
        const uint64_t gs = gdesc + (uint64_t)((s * kSdGBox) >> 4), xs = xdesc + (uint64_t)((s * kSdXBox) >> 4);
        if (leader) {
#pragma unroll
          for (int k = 0; k < kSdStep / 16; k++)  // K step k starts 32 B into the 128-byte rows
            ptx::tc_mma_f16(dset, gs + (uint64_t)((k * 32) >> 4), xs + (uint64_t)((k * 32) >> 4), idesc, i > 0 || k > 0);
          ptx::tc_commit(&sm.empty[s]);
        }
        __syncwarp();
        if (++s == kSdStages) {
          s = 0;
          ph ^= 1u;
        }
      }
      if (!ok) {
        if (leader) persist_fail();
        break;
      }
      if (leader) {
        if (n > 0) ptx::tc_commit(&sm.tfull[set]);
        else ptx::mbar_arrive(&sm.tfull[set]);
      }
      __syncwarp();
    }
  } else {
    // ---------------- epilogue ----------------
    const int e = warp - kSdEpiWarp0;  // 0..7
    const int q4 = warp & 3;           // the TMEM lane quarter this warp may access
    const int ch = e >> 2;             // 128-column half of the item
    float* tile = sm.epi[e];
    for (int j = 0;; j++) {
      int it = -1;
      if (!warp_wait_read(&sm.qfull[j % kPQ], (uint32_t)(j / kPQ) & 1u, &sm.qitem[j % kPQ], &it)) {
        if (lane == 0) persist_fail();
        break;
      }
      if (it < 0) break;
      const int4 w4 = item(SINGLE ? it & (kSdSkip - 1) : it);
      const BatchProblemTc* p = SINGLE ? &one : probs + w4.x;
      const int64_t M = p->M, K = p->K, Kw = p->Kw, ldc = p->ldc;
      float* C = p->C;
      const int64_t rbase = (int64_t)w4.y * kSdRows + q4 * 32;  // the warp's first row
      const int64_t cbase = (int64_t)w4.z * kSdCols + ch * 128;  // its first column
      // the row's A words of these 128 columns
      uint32_t aw[4] = {0u, 0u, 0u, 0u};
      if (rbase + lane < M) {
        const uint32_t* arow = p->A + (rbase + lane) * Kw;
#pragma unroll
        for (int i = 0; i < 4; i++)
          if (cbase / 32 + i < Kw) aw[i] = __ldg(arow + cbase / 32 + i);
      }
      const int set = j & 1;
      if (!warp_wait_read(&sm.tfull[set], (uint32_t)(j >> 1) & 1u, nullptr, nullptr)) {
        if (lane == 0) persist_fail();
        break;
      }
      ptx::tc_fence_after_sync();
      const uint32_t tb = tmem + ((uint32_t)(q4 * 32) << 16) + (uint32_t)(set * kSdCols + ch * 128);
      for (int c32 = 0; c32 < 4; c32++) {
        uint32_t v[4][8];
#pragma unroll
        for (int u = 0; u < 4; u++) ptx::tmem_ld_32x32b_x8(tb + (uint32_t)(c32 * 32 + u * 8), v[u]);
        ptx::tmem_wait_ld();
        const uint32_t wbits = aw[c32];
#pragma unroll
        for (int u = 0; u < 4; u++) {
          float4* t4 = reinterpret_cast<float4*>(tile + lane * kPEpiStride + u * 8);
          float f[8];
#pragma unroll
          for (int x = 0; x < 8; x++) f[x] = ((wbits >> (u * 8 + x)) & 1u) ? __uint_as_float(v[u][x]) : 0.f;
          t4[0] = make_float4(f[0], f[1], f[2], f[3]);
          t4[1] = make_float4(f[4], f[5], f[6], f[7]);
        }
        __syncwarp();
        // 8 lanes per row: rows 4*k + lane/8, 16 bytes each
        const int c4 = (lane & 7) * 4;
        const int64_t gcol = cbase + c32 * 32 + c4;
#pragma unroll
        for (int k = 0; k < 8; k++) {
          const int jr = k * 4 + (lane >> 3);
          const int64_t grow = rbase + jr;
          if (grow < M && gcol < K)
            *reinterpret_cast<float4*>(C + grow * ldc + gcol) = *reinterpret_cast<const float4*>(tile + jr * kPEpiStride + c4);
        }
        __syncwarp();
      }
      ptx::tc_fence_before_sync();
      __syncwarp();
      if (lane == 0) {
        ptx::mbar_arrive(&sm.tempty[set]);
        ptx::mbar_arrive(&sm.qempty[j % kPQ]);
      }
    }
  }
  ptx::tc_fence_before_sync();
  __syncthreads();
  if (warp == 1) {
    ptx::tc_fence_after_sync();
    ptx::tmem_dealloc(tmem, kPTmemCols);
  }
  ptx::griddep_wait();  // this grid ends after the one it may have overlapped
}

template <typename BT>
int launch_sddmm_persist_t(const BatchProblemTc* probs, const int4* items, int n_items, int* counter, int64_t N,
                           bool overlap, cudaStream_t st) {
  constexpr size_t smem = sizeof(SddmmSmem) + kPSmemAlign;
  static bool configured[64] = {false};
  int dev = 0;
  BSP_CUDA(cudaGetDevice(&dev));
  if (dev >= 64 || !configured[dev]) {
    BSP_CUDA(cudaFuncSetAttribute(k_batched_sddmm_persist<BT, false>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    if (dev < 64) configured[dev] = true;
  }
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)std::min(num_sms(), n_items));
  cfg.blockDim = dim3(kSdThreads);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = overlap ? 1 : 0;
  BSP_CUDA(cudaLaunchKernelEx(&cfg, k_batched_sddmm_persist<BT, false>, probs, items, n_items, counter, N, BatchProblemTc{}));
  return BSP_OK;
}

template <typename BT>
int launch_sddmm_one_t(const BatchProblemTc& one, int n_items, int64_t N, cudaStream_t st) {
  constexpr size_t smem = sizeof(SddmmSmem) + kPSmemAlign;
  static bool configured[64] = {false};
  int dev = 0;
  BSP_CUDA(cudaGetDevice(&dev));
  if (dev >= 64 || !configured[dev]) {
    BSP_CUDA(cudaFuncSetAttribute(k_batched_sddmm_persist<BT, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    if (dev < 64) configured[dev] = true;
  }
  k_batched_sddmm_persist<BT, true><<<(unsigned)std::min(num_sms(), n_items), kSdThreads, smem, st>>>(
      nullptr, nullptr, n_items, nullptr, N, one);
  BSP_LAUNCHED();
  return BSP_OK;
}

}  // namespace

int launch_sddmm_persist(const uint32_t* A, int64_t M, int64_t K, const void* G, int64_t ldg, const void* X,
                         int64_t ldx, int dt, int64_t N, float* dA, int64_t ldda, cudaStream_t s) {
  const int64_t items = ceil_div(M, kSdRows) * ceil_div(K, kSdCols);
  if (items == 0) return BSP_OK;
  if (items >= kSdSkip - num_sms() || N > INT32_MAX || M > INT32_MAX || K > INT32_MAX) return BSP_ERR_CAPACITY;
  BatchProblemTc one = {};
  BSP_TRY(make_batch_map_sddmm(&one.map3, G, dt, M, N, ldg, kSdRows));
  BSP_TRY(make_batch_map_sddmm(&one.map2, X, dt, K, N, ldx, kSdCols));
  one.A = A;
  one.M = M;
  one.K = K;
  one.Kw = ceil_div(K, 32);
  one.C = dA;
  one.ldc = ldda;
  if (dt == BSP_BF16) return launch_sddmm_one_t<__nv_bfloat16>(one, (int)items, N, s);
  if (dt == BSP_F16) return launch_sddmm_one_t<__half>(one, (int)items, N, s);
  return BSP_ERR_UNSUPPORTED;
}


}  // namespace bsp

struct bsp_batch {
  int n = 0;
  int64_t N = 0;
  int bdt = BSP_BF16;
  int grad = 0;         // 0: forward batch (bsp_batch_create), 1: gradient batch (bsp_batch_grad_create)
  int n_items = 0;      // forward items, or the Aᵀ·G items of a gradient batch
  int n_items_s = 0;    // SDDMM items of a gradient batch
  int device = 0;
  void* dev = nullptr;  // records, items, the work-queue counter
  bsp::BatchProblemTc* probs = nullptr;    // forward, or Aᵀ·G (map = G)
  bsp::BatchProblemTc* probs_s = nullptr;  // SDDMM (map = G, map2 = X)
  int4* items = nullptr;     // 256x256 blocks (where they may run)
  bool blocks = false;       // a forward batch that is faster in these blocks
  int4* items_ts = nullptr;  // the same output in 256x128 blocks, for the persistent kernel
  int n_items_ts = 0;
  int4* items_s = nullptr;
  int4* items_sp = nullptr;  // SDDMM items of the persistent kernel: (problem, 128 rows, 256 columns)
  int n_items_sp = 0;
  int* counter = nullptr;  // next item of the persistent SDDMM (reset by every run)
};

namespace {

// Uploads records and items into one device block and fills the batch.
int batch_upload(bsp_batch* b, const std::vector<bsp::BatchProblemTc>& p1, const std::vector<int4>& i1,
                 const std::vector<bsp::BatchProblemTc>& p2, const std::vector<int4>& i2, cudaStream_t s,
                 const std::vector<int4>& it, const std::vector<int4>& i3 = {}) {
  using namespace bsp;
  auto up = [](size_t bytes) { return (std::max<size_t>(bytes, 1) + 255) & ~size_t(255); };
  const size_t o_p1 = 0, o_i1 = o_p1 + up(sizeof(BatchProblemTc) * p1.size());
  const size_t o_p2 = o_i1 + up(sizeof(int4) * i1.size()), o_i2 = o_p2 + up(sizeof(BatchProblemTc) * p2.size());
  const size_t o_i3 = o_i2 + up(sizeof(int4) * i2.size());
  const size_t o_it = o_i3 + up(sizeof(int4) * i3.size());
  const size_t o_c = o_it + up(sizeof(int4) * it.size()), total = o_c + 256;
  cudaError_t e = cudaMalloc(&b->dev, total);
  if (e != cudaSuccess) {
    cuda_status(e);
    b->dev = nullptr;
    return BSP_ERR_ALLOC;
  }
  char* base = static_cast<char*>(b->dev);
  b->probs = reinterpret_cast<BatchProblemTc*>(base + o_p1);
  b->items = reinterpret_cast<int4*>(base + o_i1);
  b->probs_s = reinterpret_cast<BatchProblemTc*>(base + o_p2);
  b->items_s = reinterpret_cast<int4*>(base + o_i2);
  b->items_sp = reinterpret_cast<int4*>(base + o_i3);
  b->items_ts = reinterpret_cast<int4*>(base + o_it);
  b->n_items_ts = (int)it.size();
  b->counter = reinterpret_cast<int*>(base + o_c);
  b->n_items = (int)i1.size();
  b->n_items_s = (int)i2.size();
  b->n_items_sp = (int)i3.size();
  struct Part { void* dst; const void* src; size_t bytes; };
  const Part parts[6] = {{b->items_ts, it.data(), sizeof(int4) * it.size()},
                         {b->probs, p1.data(), sizeof(BatchProblemTc) * p1.size()},
                         {b->items, i1.data(), sizeof(int4) * i1.size()},
                         {b->probs_s, p2.data(), sizeof(BatchProblemTc) * p2.size()},
                         {b->items_s, i2.data(), sizeof(int4) * i2.size()},
                         {b->items_sp, i3.data(), sizeof(int4) * i3.size()}};
  for (const Part& q : parts)
    if (q.bytes && (e = cudaMemcpyAsync(q.dst, q.src, q.bytes, cudaMemcpyHostToDevice, s)) != cudaSuccess)
      return cuda_status(e);
  if ((e = cudaStreamSynchronize(s)) != cudaSuccess) return cuda_status(e);
  return BSP_OK;
}

bool env_is(const char* name, char v) {
  const char* e = getenv(name);
  return e && e[0] == v;
}

// Time (us) until the last of `sms` SMs, each taking the next item when it is
// done, has finished a list of costs (of more than four rounds: what they add up
// to, and half an item).
double list_time(const std::vector<double>& cost, int sms) {
  if (cost.size() > 4 * (size_t)sms) {
    double sum = 0.0;
    for (const double c : cost) sum += c;
    return sum / sms + 0.5 * sum / (double)cost.size();
  }
  std::vector<double> busy((size_t)sms, 0.0);  // a heap, the first to be free on top
  double last = 0.0;
  for (const double c : cost) {
    const double t = busy[0] + c;
    last = std::max(last, t);
    size_t i = 0;
    for (size_t k = 1; k < busy.size(); k = 2 * i + 1) {
      if (k + 1 < busy.size() && busy[k + 1] < busy[k]) k++;
      if (busy[k] >= t) break;
      busy[i] = busy[k];
      i = k;
    }
    busy[i] = t;
  }
  return last;
}

// Forward batches wider than one 128-column item: a CTA per 256x256 block
// (k_spmm_tc, whose expanded A serves 256 columns) or the persistent kernel's
// 256x128 items, whichever finishes first by both lists' times; the figures are
// fitted to 54 batches of 3 to 512 problems, N = 136 to 1024, where the rule
// costs at most 1.13 of the better form and 1.01 on average (8 problems of 2048
// to 4096 rows and columns, N = 136: 46 us and 59 persistent, N = 1024: 129 and
// 163; 64 of 64 to 1024, N = 1024: 71 and 61; 3 of 4096, N = 256: 56 and 39).
bool blocks_are_faster(const std::vector<int4>& blocks, const std::vector<int4>& items, int64_t N) {
  std::vector<double> tb, ti;
  tb.reserve(blocks.size());
  ti.reserve(items.size());
  for (const int4& b : blocks) {
    const int64_t boxes = std::min<int64_t>(4, bsp::ceil_div(N - (int64_t)b.z * bsp::kItemCols, 64));
    tb.push_back(9.0 + (double)b.w * (0.27 + 0.025 * (double)boxes));
  }
  for (const int4& i : items) ti.push_back(1.9 + (double)i.w * 0.285);
  return list_time(tb, bsp::num_sms()) < 7.4 + list_time(ti, bsp::num_sms());
}

// longest reduction first (LPT), ties by problem order: stable
void sort_items(std::vector<int4>& items) {
  std::stable_sort(items.begin(), items.end(), [](const int4& x, const int4& y) { return x.w > y.w; });
}

}  // namespace

extern "C" {

int bsp_batch_create(const bsp_problem* problems, int n, int64_t N, int b_dtype, bsp_batch** batch,
                     bsp_stream_t stream) {
  using namespace bsp;
  if (!batch) return BSP_ERR_INVALID_ARG;
  *batch = nullptr;
  if (n < 0 || N < 0 || N > ((int64_t)1 << 30)) return BSP_ERR_INVALID_ARG;
  if (n > 0 && !problems) return BSP_ERR_INVALID_ARG;
  if (b_dtype != BSP_BF16 && b_dtype != BSP_F16) return BSP_ERR_UNSUPPORTED;
  if (N % 8 != 0) return BSP_ERR_ALIGNMENT;
  std::vector<BatchProblemTc> hp((size_t)n);
  std::vector<int4> items, ts;
  const bool blocks = N > ts_item_cols() || env_is("BSP_BATCH_PERSIST", '0');
  for (int i = 0; i < n; i++) {
    const bsp_problem& p = problems[i];
    if (p.M < 0 || p.K < 0 || p.M > INT32_MAX || p.K > ((int64_t)1 << 30)) return BSP_ERR_INVALID_ARG;
    if (p.K > tc_max_reduction()) return BSP_ERR_CAPACITY;
    if (p.ldb < N || p.ldc < N) return BSP_ERR_INVALID_ARG;
    if ((p.M > 0 && p.K > 0 && !p.A_words) || (p.K > 0 && N > 0 && !p.B) || (p.M > 0 && N > 0 && !p.C))
      return BSP_ERR_INVALID_ARG;
    if (!is_aligned(p.A_words, 4) || !is_aligned(p.B, 16) || (p.ldb * 2) % 16 != 0 || !is_aligned(p.C, 16) ||
        p.ldc % 4 != 0)
      return BSP_ERR_ALIGNMENT;
    const int64_t Kw = ceil_div(p.K, 32);
    BatchProblemTc& r = hp[(size_t)i];
    std::memset(&r, 0, sizeof(r));
    if (p.K > 0 && N > 0) BSP_TRY(make_batch_map(&r.map, p.B, b_dtype, p.K, N, p.ldb));
    r.A = p.A_words;
    r.M = p.M;
    r.K = p.K;
    r.Kw = Kw;
    r.C = p.C;
    r.ldc = p.ldc;
    if (p.M > 0 && N > 0) BSP_TRY(make_out_map(&r.map2, p.C, p.M, N, p.ldc, 1, p.M * p.ldc));
    for (int64_t rb = 0; blocks && rb < ceil_div(p.M, kItemRows); rb++)
      for (int64_t nb = 0; nb < ceil_div(N, kItemCols); nb++) items.push_back(make_int4(i, (int)rb, (int)nb, (int)Kw));
    for (int64_t rb = 0; rb < ceil_div(p.M, ts_item_rows()); rb++)
      for (int64_t nb = 0; nb < ceil_div(N, ts_item_cols()); nb++) ts.push_back(make_int4(i, (int)rb, (int)nb, (int)Kw));
  }
  if (ts.size() > (size_t)INT32_MAX) return BSP_ERR_CAPACITY;
  sort_items(items);
  sort_items(ts);
  bsp_batch* b = new (std::nothrow) bsp_batch();
  if (!b) return BSP_ERR_ALLOC;
  b->n = n;
  b->N = N;
  b->bdt = b_dtype;
  b->blocks = !items.empty() && blocks_are_faster(items, ts, N);
  cudaGetDevice(&b->device);
  const int st = batch_upload(b, hp, items, {}, {}, (cudaStream_t)stream, ts);
  if (st != BSP_OK) {
    if (b->dev) cudaFree(b->dev);
    delete b;
    return st;
  }
  *batch = b;
  return BSP_OK;
}

int bsp_batch_grad_create(const bsp_problem_grad* problems, int n, int64_t N, int dtype, bsp_batch** batch,
                          bsp_stream_t stream) {
  using namespace bsp;
  if (!batch) return BSP_ERR_INVALID_ARG;
  *batch = nullptr;
  if (n < 0 || N < 0 || N > ((int64_t)1 << 30)) return BSP_ERR_INVALID_ARG;
  if (n > 0 && !problems) return BSP_ERR_INVALID_ARG;
  if (dtype != BSP_BF16 && dtype != BSP_F16) return BSP_ERR_UNSUPPORTED;
  if (N % 8 != 0) return BSP_ERR_ALIGNMENT;
  std::vector<BatchProblemTc> pt, ps;
  std::vector<int4> it, is, isp, ts;
  const bool blocks = env_is("BSP_BATCH_PERSIST", '0'), blocks_s = env_is("BSP_BATCH_SDDMM_PERSIST", '0');
  for (int i = 0; i < n; i++) {
    const bsp_problem_grad& p = problems[i];
    if (p.M < 0 || p.K < 0 || p.M > INT32_MAX || p.K > INT32_MAX) return BSP_ERR_INVALID_ARG;
    if (p.ldx < N || p.ldg < N) return BSP_ERR_INVALID_ARG;
    if (p.dX && p.lddx < N) return BSP_ERR_INVALID_ARG;
    if (p.dA && p.ldda < p.K) return BSP_ERR_INVALID_ARG;
    const bool work = p.M > 0 && p.K > 0;
    if (work && (!p.A_words || (N > 0 && (!p.X || !p.G)))) return BSP_ERR_INVALID_ARG;
    if (!is_aligned(p.A_words, 4) || !is_aligned(p.X, 16) || !is_aligned(p.G, 16) || (p.ldx * 2) % 16 != 0 ||
        (p.ldg * 2) % 16 != 0)
      return BSP_ERR_ALIGNMENT;
    const int64_t Kw = ceil_div(p.K, 32);
    if (p.dX && p.K > 0) {  // dX = Aᵀ·G: output rows K, reduction over M in 32-row tiles
      if (ceil_div(p.M, 32) * 32 > tc_max_reduction()) return BSP_ERR_CAPACITY;
      if (!is_aligned(p.dX, 16) || p.lddx % 4 != 0) return BSP_ERR_ALIGNMENT;
      BatchProblemTc r;
      std::memset(&r, 0, sizeof(r));
      if (p.M > 0 && N > 0) BSP_TRY(make_batch_map(&r.map, p.G, dtype, p.M, N, p.ldg));
      r.A = p.A_words;
      r.M = p.M;
      r.K = p.K;
      r.Kw = Kw;
      r.C = p.dX;
      r.ldc = p.lddx;
      if (N > 0) BSP_TRY(make_out_map(&r.map2, p.dX, p.K, N, p.lddx, 1, p.K * p.lddx));
      const int idx = (int)pt.size();
      pt.push_back(r);
      for (int64_t rb = 0; blocks && rb < ceil_div(p.K, kItemRows); rb++)
        for (int64_t nb = 0; nb < ceil_div(N, kItemCols); nb++)
          it.push_back(make_int4(idx, (int)rb, (int)nb, (int)ceil_div(p.M, 32)));
      for (int64_t rb = 0; rb < ceil_div(p.K, ts_item_rows()); rb++)
        for (int64_t nb = 0; nb < ceil_div(N, ts_item_cols()); nb++)
          ts.push_back(make_int4(idx, (int)rb, (int)nb, (int)ceil_div(p.M, 32)));
    }
    if (p.dA && p.M > 0) {  // dA = (G·Xᵀ) ⊙ A: output [M][K], reduction over N in 64-column steps
      if (p.K % 8 != 0 || !is_aligned(p.dA, 16) || p.ldda % 4 != 0) return BSP_ERR_ALIGNMENT;
      if (ceil_div(p.K, kItemCols) > INT32_MAX) return BSP_ERR_CAPACITY;
      BatchProblemTc r;
      std::memset(&r, 0, sizeof(r));
      if (p.K > 0 && N > 0) {
        BSP_TRY(make_batch_map_sddmm(&r.map, p.G, dtype, p.M, N, p.ldg));
        BSP_TRY(make_batch_map_sddmm(&r.map2, p.X, dtype, p.K, N, p.ldx));
        BSP_TRY(make_batch_map_sddmm(&r.map3, p.G, dtype, p.M, N, p.ldg, 128));
      }
      r.A = p.A_words;
      r.M = p.M;
      r.K = p.K;
      r.Kw = Kw;
      r.C = p.dA;
      r.ldc = p.ldda;
      const int idx = (int)ps.size();
      ps.push_back(r);
      for (int64_t rb = 0; blocks_s && rb < ceil_div(p.M, kItemRows); rb++)
        for (int64_t kb = 0; kb < ceil_div(p.K, kItemCols); kb++)
          is.push_back(make_int4(idx, (int)rb, (int)kb, (int)ceil_div(N, 64)));
      for (int64_t rb = 0; rb < ceil_div(p.M, (int64_t)kSdRows); rb++)
        for (int64_t kb = 0; kb < ceil_div(p.K, (int64_t)kSdCols); kb++)
          isp.push_back(make_int4(idx, (int)rb, (int)kb, (int)ceil_div(N, 64)));
    }
  }
  if (ts.size() > (size_t)INT32_MAX || is.size() > (size_t)INT32_MAX || isp.size() > (size_t)INT32_MAX)
    return BSP_ERR_CAPACITY;
  sort_items(it);
  sort_items(is);
  sort_items(ts);
  bsp_batch* b = new (std::nothrow) bsp_batch();
  if (!b) return BSP_ERR_ALLOC;
  b->n = n;
  b->N = N;
  b->bdt = dtype;
  b->grad = 1;
  cudaGetDevice(&b->device);
  const int st = batch_upload(b, pt, it, ps, is, (cudaStream_t)stream, ts, isp);
  if (st != BSP_OK) {
    if (b->dev) cudaFree(b->dev);
    delete b;
    return st;
  }
  *batch = b;
  return BSP_OK;
}

int bsp_batch_destroy(bsp_batch* batch) {
  if (!batch) return BSP_OK;
  if (batch->dev) cudaFree(batch->dev);
  delete batch;
  return BSP_OK;
}

int bsp_batched_spmm(const bsp_batch* b, bsp_stream_t stream) {
  using namespace bsp;
  if (!b || b->grad) return BSP_ERR_INVALID_ARG;
  int dev = -1;
  cudaGetDevice(&dev);
  if (dev != b->device) return BSP_ERR_INVALID_ARG;
  if (b->n_items_ts == 0 || b->N == 0) return BSP_OK;
  const cudaStream_t s = (cudaStream_t)stream;
  // (BSP_BATCH_PERSIST, for comparisons: 1 = the persistent kernel, 0 = a CTA per
  // 256x256 block where the batch was created with it or is wider than 128)
  const bool blocks = b->n_items > 0 && !env_is("BSP_BATCH_PERSIST", '1') && (b->blocks || env_is("BSP_BATCH_PERSIST", '0'));
  if (!blocks) return launch_ts_batch(b->probs, b->items_ts, b->n_items_ts, b->N, b->bdt, false, s);
  return launch_batched_tc(b->probs, b->items, b->n_items, b->N, b->bdt, s);
}

int bsp_batch_tune(bsp_batch* b, bsp_stream_t stream, int* shape, float* ms) {
  using namespace bsp;
  if (!b || b->grad || !shape || !ms) return BSP_ERR_INVALID_ARG;
  int dev = -1;
  cudaGetDevice(&dev);
  if (dev != b->device) return BSP_ERR_INVALID_ARG;
  const cudaStream_t s = (cudaStream_t)stream;
  // one shape is built: its time is measured all the same
  cudaEvent_t e0 = nullptr, e1 = nullptr;
  float t = 0.f;
  auto measure = [&]() -> int {
    BSP_CUDA(cudaEventCreate(&e0));
    BSP_CUDA(cudaEventCreate(&e1));
    BSP_TRY(bsp_batched_spmm(b, stream));  // warm-up
    BSP_CUDA(cudaEventRecord(e0, s));
    for (int r = 0; r < 3; r++) BSP_TRY(bsp_batched_spmm(b, stream));
    BSP_CUDA(cudaEventRecord(e1, s));
    BSP_CUDA(cudaEventSynchronize(e1));
    BSP_CUDA(cudaEventElapsedTime(&t, e0, e1));
    return BSP_OK;
  };
  const int rc = measure();
  if (e0) cudaEventDestroy(e0);
  if (e1) cudaEventDestroy(e1);
  if (rc != BSP_OK) return rc;
  *shape = 0;
  *ms = t / 3.f;
  return BSP_OK;
}

int bsp_batched_spmm_grad(const bsp_batch* b, bsp_stream_t stream) {
  using namespace bsp;
  if (!b || !b->grad) return BSP_ERR_INVALID_ARG;
  int dev = -1;
  cudaGetDevice(&dev);
  if (dev != b->device) return BSP_ERR_INVALID_ARG;
  if (b->N == 0) return BSP_OK;
  const cudaStream_t s = (cudaStream_t)stream;
  // dX = Aᵀ·G: the persistent kernel in its transposed form.  dA neither reads nor
  // writes what dX does, and all that came before dX's launch is complete when
  // dX starts: as its programmatic dependent the persistent SDDMM takes the SMs
  // that dX's last items leave idle (128 problems of 64..2048 rows and columns, N
  // = 96, forward and both gradients: 111 -> 99 us).  Its counter is
  // reset before both, so that nothing stands between the two launches.
  // (BSP_BATCH_PERSIST=0, BSP_BATCH_SDDMM_PERSIST=0, set when the batch is created
  // and when it runs: a CTA per 256x256 block)
  const bool ts = b->n_items_ts > 0 && !(env_is("BSP_BATCH_PERSIST", '0') && b->n_items > 0);
  const bool blocks_s = env_is("BSP_BATCH_SDDMM_PERSIST", '0') && b->n_items_s > 0;
  const bool sd = !blocks_s && b->n_items_sp > 0;
  if (sd) BSP_CUDA(cudaMemsetAsync(b->counter, 0, sizeof(int), s));
  if (ts) BSP_TRY(launch_ts_batch(b->probs, b->items_ts, b->n_items_ts, b->N, b->bdt, true, s));
  else BSP_TRY(launch_batched_tc(b->probs, b->items, b->n_items, b->N, b->bdt, s, 1));
  if (!blocks_s) {
    if (!sd) return BSP_OK;
    if (b->bdt == BSP_BF16)
      return launch_sddmm_persist_t<__nv_bfloat16>(b->probs_s, b->items_sp, b->n_items_sp, b->counter, b->N, ts, s);
    return launch_sddmm_persist_t<__half>(b->probs_s, b->items_sp, b->n_items_sp, b->counter, b->N, ts, s);
  }
  return launch_batched_tc(b->probs_s, b->items_s, b->n_items_s, b->N, b->bdt, s, 2);
}

}  // extern "C"
