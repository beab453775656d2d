// sddmm_staged.cu — FP32 mask gradient for masks that are dense enough that
// neighbouring rows of A share rows of X.
//
// dA[i][k] = G[i]·X[k] at A's set bits, 0 elsewhere.  A CTA takes 32 rows of A;
// its 16 warps keep two rows of G each in registers (a slice of 128 VPL
// columns), and TMA brings the same slice of 32 rows of X at a time (one word
// of A's rows) into a ring of shared-memory stages.  A warp forms the products
// of its rows' set bits from there, up to four at a time: every lane sums its
// columns, exchanges of halves reduce the four sums together, and lane b ends
// with the product of bit b, so that dA leaves as whole 128-byte lines.
//
// Bound by shared memory, which reads 4 bytes of X a product and column at 128
// bytes a clock: 45 us of 95 at 2048x2048, N = 1024, 10 % set (its pipe 67 %
// busy; the rest waits for exchanges and the coming stage).  The walk
// (k_sddmm_rows) fetches X's row from L2 for every set bit, 1.7 GB there, in
// 206 us; here a CTA fetches each row once for 32 rows of A.  Columns in slices
// of 256 with four rows a warp took 174 us, for every slice reduces its
// products anew; two rows with 512 columns 95.
#include <type_traits>

#include "ptx.cuh"
#include "spmm.cuh"

namespace bsp {
namespace {

constexpr int kRowsCta = 32, kWarps = 16, kRowsWarp = kRowsCta / kWarps;
constexpr int kThreads = (kWarps + 1) * 32;
constexpr int kXRows = 32;    // rows of X per stage: the columns of one word of A
constexpr int kStageMax = 3;  // 64 KB each at VPL = 4
constexpr int kBoxCols = 128;
constexpr int kErr = 6;
constexpr uint32_t kFull = 0xffffffffu;

__device__ int g_staged_error;

template <int VPL>
struct Shared {
  float x[kStageMax][VPL][kXRows][kBoxCols];  // TMA boxes of 128 columns
  uint64_t full[kStageMax], empty[kStageMax];
};

template <int VPL>
__global__ void __launch_bounds__(kThreads, 1)
    k_sddmm_staged(const uint32_t* __restrict__ A, int64_t M, int64_t K, int64_t Kw, const float* __restrict__ G,
                   int64_t ldg, int64_t N, float* __restrict__ dA, int64_t ldda, int64_t part_words,
                   const __grid_constant__ CUtensorMap map) {
  constexpr int kCols = VPL * kBoxCols;
  extern __shared__ __align__(1024) uint8_t smem_raw[];
  Shared<VPL>& sm = *reinterpret_cast<Shared<VPL>*>(
      smem_raw + ((128 - (ptx::smem_addr(smem_raw) & 127)) & 127));
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (threadIdx.x == 0) {
    for (int s = 0; s < kStageMax; s++) {
      ptx::mbar_init(&sm.full[s], 1);
      ptx::mbar_init(&sm.empty[s], kWarps);
    }
    ptx::fence_mbar_init();
  }
  __syncthreads();
  const int64_t p0 = (int64_t)blockIdx.y * part_words, p1 = min(Kw, p0 + part_words);
  const int64_t slices = (N + kCols - 1) / kCols;
  if (warp == kWarps) {
    // X: slice by slice, word by word.  Rows past K and columns past N arrive
    // as zeros; a stage always takes its full size.
    const bool leader = ptx::elect_one();
    int64_t it = 0;
    bool ok = true;
    for (int64_t sl = 0; sl < slices && ok; sl++)
      for (int64_t w = p0; w < p1; w++, it++) {
        const int st = (int)(it % kStageMax);
        if (!ptx::mbar_wait_warp(&sm.empty[st], ((uint32_t)(it / kStageMax) & 1u) ^ 1u)) {
          if (leader) atomicCAS(&g_staged_error, 0, kErr);
          ok = false;
          break;
        }
        if (leader) {
          ptx::mbar_arrive_expect_tx(&sm.full[st], VPL * kXRows * kBoxCols * 4);
#pragma unroll
          for (int b = 0; b < VPL; b++)
            ptx::tma_load_2d(sm.x[st][b], &map, (int)(sl * kCols + b * kBoxCols), (int)(w * 32), &sm.full[st]);
        }
        __syncwarp();
      }
    // copies end before the CTA does, also those of a reader that gave up
    for (int64_t j = it > kStageMax ? it - kStageMax : 0; j < it; j++)
        ptx::mbar_wait_warp(&sm.full[j % kStageMax], (uint32_t)(j / kStageMax) & 1u);
    return;
  }
  int64_t row[kRowsWarp];
#pragma unroll
  for (int r = 0; r < kRowsWarp; r++) row[r] = (int64_t)blockIdx.x * kRowsCta + warp * kRowsWarp + r;
  float* out[kRowsWarp];
#pragma unroll
  for (int r = 0; r < kRowsWarp; r++) out[r] = dA + row[r] * ldda + lane;
  int64_t it = 0;
  for (int64_t sl = 0; sl < slices; sl++) {
    float4 g[kRowsWarp][VPL];
#pragma unroll
    for (int r = 0; r < kRowsWarp; r++)
#pragma unroll
      for (int v = 0; v < VPL; v++) {
        const int64_t c = sl * kCols + v * kBoxCols + lane * 4;
        const float* p = G + row[r] * ldg + c;
        g[r][v] = make_float4(0.f, 0.f, 0.f, 0.f);
        if (row[r] < M) {
          if (c + 4 <= N) {
            g[r][v] = __ldg(reinterpret_cast<const float4*>(p));
          } else {
            if (c < N) g[r][v].x = __ldg(p);
            if (c + 1 < N) g[r][v].y = __ldg(p + 1);
            if (c + 2 < N) g[r][v].z = __ldg(p + 2);
          }
        }
      }
    uint32_t held[kRowsWarp], ahead[kRowsWarp];  // lane l: word l of the current 32, of the next
    auto words = [&](int64_t w, uint32_t* out) {
#pragma unroll
      for (int r = 0; r < kRowsWarp; r++)
        out[r] = row[r] < M && w + lane < p1 ? __ldg(A + row[r] * Kw + w + lane) : 0u;
    };
    words(p0, ahead);
    for (int64_t w = p0; w < p1; w++, it++) {
      const int st = (int)(it % kStageMax);
      const int at = (int)(w - p0) & 31;
      if (at == 0) {
#pragma unroll
        for (int r = 0; r < kRowsWarp; r++) held[r] = ahead[r];
        words(w + 32, ahead);
      }
      const bool inside = w * 32 + lane < K;
      uint32_t word[kRowsWarp];
      float old[kRowsWarp];  // the same thread's sum over the slices before
#pragma unroll
      for (int r = 0; r < kRowsWarp; r++) {
        word[r] = __reduce_or_sync(kFull, lane == at ? held[r] : 0u);  // (the loops below are warp-uniform)
        old[r] = sl > 0 && inside && row[r] < M ? out[r][w * 32] : 0.f;
      }
      if (!ptx::mbar_wait_warp(&sm.full[st], (uint32_t)(it / kStageMax) & 1u)) {
        if (lane == 0) atomicCAS(&g_staged_error, 0, kErr);
        return;
      }
#pragma unroll
      for (int r = 0; r < kRowsWarp; r++) {
        const uint32_t all = word[r];
        // the place of this lane's bit among the word's set bits
        int place = ((all >> lane) & 1u) ? __popc(all & ((1u << lane) - 1u)) : 64;
        float mine = old[r];
        uint32_t rest = all;
        auto products = [&](auto count) {  // the next C set bits
          constexpr int C = decltype(count)::value;
          const float4* x[C];
#pragma unroll
          for (int s = 0; s < C; s++) {
            x[s] = reinterpret_cast<const float4*>(&sm.x[st][0][__ffs(rest) - 1][lane * 4]);
            rest &= rest - 1;
          }
          float acc[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
          for (int v = 0; v < VPL; v++) {
            float4 xv[C];
#pragma unroll
            for (int s = 0; s < C; s++) xv[s] = x[s][v * (kXRows * kBoxCols / 4)];
#pragma unroll
            for (int s = 0; s < C; s++) {
              acc[s] = fmaf(g[r][v].x, xv[s].x, acc[s]);
              acc[s] = fmaf(g[r][v].y, xv[s].y, acc[s]);
              acc[s] = fmaf(g[r][v].z, xv[s].z, acc[s]);
              acc[s] = fmaf(g[r][v].w, xv[s].w, acc[s]);
            }
          }
          // lanes of group s (all; halves; quarters of the warp) end with product s
          constexpr int kGroup = C == 1 ? 32 : (C == 2 ? 16 : 8);
          float t = acc[0];
          if (C == 2) {
            const bool up = (lane & 16) != 0;
            t = (up ? acc[1] : acc[0]) + __shfl_xor_sync(kFull, up ? acc[0] : acc[1], 16);
          } else if (C > 2) {
            const bool up = (lane & 16) != 0, up2 = (lane & 8) != 0;
            const float k0 = (up ? acc[2] : acc[0]) + __shfl_xor_sync(kFull, up ? acc[0] : acc[2], 16);
            const float k1 = (up ? acc[3] : acc[1]) + __shfl_xor_sync(kFull, up ? acc[1] : acc[3], 16);
            t = (up2 ? k1 : k0) + __shfl_xor_sync(kFull, up2 ? k0 : k1, 8);
          }
#pragma unroll
          for (int o = kGroup / 2; o > 0; o >>= 1) t += __shfl_xor_sync(kFull, t, o);
          if (C > 1) t = __shfl_sync(kFull, t, place * kGroup);  // (modulo 32 past the groups: not taken)
          if ((unsigned)place < (unsigned)C) mine += t;
          place -= C;
        };
        int left = __popc(all);
        for (; left >= 4; left -= 4) products(std::integral_constant<int, 4>());
        if (left == 3) products(std::integral_constant<int, 3>());
        else if (left == 2) products(std::integral_constant<int, 2>());
        else if (left == 1) products(std::integral_constant<int, 1>());
        if (inside && row[r] < M) out[r][w * 32] = mine;
      }
      __syncwarp();
      if (lane == 0) ptx::mbar_arrive(&sm.empty[st]);
    }
  }
}

template <int VPL>
int launch_t(const uint32_t* A, int64_t M, int64_t K, const float* G, int64_t ldg, int64_t N, float* dA, int64_t ldda,
             const CUtensorMap& map, cudaStream_t s) {
  constexpr size_t smem = sizeof(Shared<VPL>) + 128;
  auto kern = k_sddmm_staged<VPL>;
  static bool configured[64] = {};
  int dev = 0;
  BSP_CUDA(cudaGetDevice(&dev));
  if (dev >= 64 || !configured[dev]) {
    BSP_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    if (dev < 64) configured[dev] = true;
  }
  // Words cut into parts until whole rounds of one CTA an SM come out: the
  // fewest parts (of at least 8 words) whose last round is nearly full.
  const int64_t Kw = ceil_div(K, 32), blocks = ceil_div(M, kRowsCta), sms = num_sms();
  int64_t parts = 1;
  double best = 0.0;
  for (int64_t p = 1; p <= 512 && (p == 1 || Kw / p >= 8); p++) {
    const double eff = (double)(blocks * p) / (double)(ceil_div(blocks * p, sms) * sms);
    if (eff > best + 0.02) best = eff, parts = p;
  }
  const int64_t part_words = ceil_div(Kw, parts);
  const dim3 grid((unsigned)blocks, (unsigned)ceil_div(Kw, part_words));
  kern<<<grid, kThreads, smem, s>>>(A, M, K, Kw, G, ldg, N, dA, ldda, part_words, map);
  BSP_LAUNCHED();
  return BSP_OK;
}

}  // namespace

int launch_sddmm_staged(const uint32_t* A, int64_t M, int64_t K, const float* G, int64_t ldg, const float* X,
                        int64_t ldx, int64_t N, float* dA, int64_t ldda, cudaStream_t s) {
  if (M == 0 || K == 0) return BSP_OK;
  if (M > INT32_MAX || K > INT32_MAX - 32 || N > INT32_MAX / 2) return BSP_ERR_CAPACITY;
  CUtensorMap map;
  BSP_TRY(make_rows_map_f32(&map, X, K, N, ldx, kBoxCols, kXRows));
  if (N <= 128) return launch_t<1>(A, M, K, G, ldg, N, dA, ldda, map, s);
  if (N <= 256) return launch_t<2>(A, M, K, G, ldg, N, dA, ldda, map, s);
  return launch_t<4>(A, M, K, G, ldg, N, dA, ldda, map, s);
}

int sddmm_staged_device_error(int* out, bool clear) {
  BSP_CUDA(cudaMemcpyFromSymbol(out, g_staged_error, sizeof(int)));
  if (clear) {
    const int zero = 0;
    BSP_CUDA(cudaMemcpyToSymbol(g_staged_error, &zero, sizeof(int)));
  }
  return BSP_OK;
}

}  // namespace bsp
