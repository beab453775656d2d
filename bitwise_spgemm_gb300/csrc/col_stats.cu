// col_stats.cu — sizes of a dense operand's values, column by column.
//
// Routes that add a column's values in another order, or through sums that a
// row of A does not hold, are exact enough only while the values of a column
// are of about one size; this kernel says so on the device, without a host
// wait, to the kernels behind it.
#include "ptx.cuh"
#include "spmm_dev.cuh"

namespace bsp {
namespace {

// bad[b] = 1 if one of block b's columns holds a value that is not finite or at
// least 2^100, or has its largest exponent more than `octaves` above the mean one
// of its nonzeros.  A block takes all rows of a few columns, so that
// nothing is handed between blocks.  Bound by the latency of its rounds of loads.
// It is launched as a programmatic dependent: it reads B alone and runs beside
// the kernels before it, and ends after them.
constexpr int kWarps = 32;
template <typename T>
__global__ void __launch_bounds__(kWarps * 32) k_col_stats(const T* __restrict__ B, int64_t R, int64_t N, int64_t ldb,
                                                           int* __restrict__ bad, int octaves) {
  constexpr int COLS = kStatCols, LANES = 32 / COLS, ROWS = LANES * kWarps, U = 16;  // U loads of a lane in flight
  __shared__ int s_max[kWarps][COLS];
  __shared__ unsigned s_n[kWarps][COLS], s_sum[kWarps][COLS];
  ptx::griddep_launch_dependents();
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, c = lane % COLS;
  const int64_t col = (int64_t)blockIdx.x * COLS + c;
  int top = 0;
  unsigned n = 0, sum = 0;
  for (int64_t r0 = warp * LANES + lane / COLS; r0 < R; r0 += ROWS * U) {
    uint32_t x[U];
#pragma unroll
    for (int i = 0; i < U; i++) {
      const int64_t r = r0 + i * ROWS;
      x[i] = r < R && col < N ? __float_as_uint(to_f32(__ldg(B + r * ldb + col))) : 0u;
    }
#pragma unroll
    for (int i = 0; i < U; i++) {
      const int e = (int)((x[i] >> 23) & 255u);
      top = max(top, e);
      n += (x[i] << 1) != 0u;
      sum += (unsigned)e;
    }
  }
#pragma unroll
  for (int o = 16; o >= COLS; o >>= 1) {
    top = max(top, __shfl_xor_sync(kFull, top, o));
    n += __shfl_xor_sync(kFull, n, o);
    sum += __shfl_xor_sync(kFull, sum, o);
  }
  if (lane < COLS) {
    s_max[warp][c] = top;
    s_n[warp][c] = n;
    s_sum[warp][c] = sum;
  }
  __syncthreads();
  if (warp == 0) {
    bool out = false;
    if (lane < COLS) {
      for (int w = 1; w < kWarps; w++) {
        top = max(top, s_max[w][c]);
        n += s_n[w][c];
        sum += s_sum[w][c];
      }
      out = top >= kStatTop || (unsigned long long)top * n > sum + (unsigned long long)octaves * n;
    }
    out = __any_sync(kFull, out);
    if (lane == 0) bad[blockIdx.x] = out ? 1 : 0;
  }
  ptx::griddep_wait();
}

// *out = whether one of n flags is set.
__global__ void __launch_bounds__(1024) k_any(const int* __restrict__ flags, int64_t n, int* out) {
  int any = 0;
  for (int64_t i = threadIdx.x; i < n; i += blockDim.x) any |= __ldg(flags + i);
  any = __syncthreads_or(any);
  if (threadIdx.x == 0) *out = any ? 1 : 0;
}

// The values of a product in parts (see k_split_b), for sums of about `addends`
// values of a column: bad[b] = 1 if one of block b's columns does not pass.  A
// block takes all rows of 8 columns and keeps them in registers, U values a lane,
// for they are looked at twice; the sums' order is the same on every run.  Bound
// by latency: 2 us of the 56 of 2048x2048x1024 (values read again and counted by
// atomics in k_split_b: 4, and up to 120 where most of them are too small).
constexpr int kPartsRows = 32 / kStatCols * kWarps;  // rows of a block at a time
template <int U>
__global__ void __launch_bounds__(kWarps * 32) k_parts_stats(const float* __restrict__ B, int64_t R, int64_t N,
                                                             int64_t ldb, int* __restrict__ bad,
                                                             int* __restrict__ flag, float addends) {
  constexpr int COLS = kStatCols, LANES = 32 / COLS;
  __shared__ float s_abs[kWarps][COLS], s_n[kWarps][COLS];
  __shared__ int s_max[kWarps][COLS], s_low[COLS], s_cnt[kWarps][COLS];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, c = lane % COLS;
  const int64_t col = (int64_t)blockIdx.x * COLS + c;
  const int r0 = warp * LANES + lane / COLS;
  const float* p = B + (int64_t)r0 * ldb + col;
  float x[U];
#pragma unroll
  for (int i = 0; i < U; i++) {
    x[i] = r0 + i * kPartsRows < R && col < N ? __ldg(p) : 0.f;
    p += kPartsRows * ldb;
  }
  float mag = 0.f, n = 0.f;
  int top = 0, least = 255;  // largest and smallest exponent of a nonzero value
#pragma unroll
  for (int i = 0; i < U; i++) {
    const int e = (int)((__float_as_uint(x[i]) >> 23) & 255u);
    top = max(top, e);
    if (x[i] != 0.f) least = min(least, e);
    n += x[i] != 0.f ? 1.f : 0.f;
    mag += fabsf(x[i]);
  }
#pragma unroll
  for (int o = 16; o >= COLS; o >>= 1) {
    mag += __shfl_xor_sync(kFull, mag, o);
    n += __shfl_xor_sync(kFull, n, o);
    top = max(top, __shfl_xor_sync(kFull, top, o));
  }
  if (lane < COLS) {
    s_abs[warp][c] = mag;
    s_n[warp][c] = n;
    s_max[warp][c] = top;
  }
  const bool wrong = __syncthreads_or(least < kStatBottom || top >= kStatTop);
  float limit = 0.f;
  if (threadIdx.x < COLS) {
    for (int w = 1; w < kWarps; w++) {
      mag += s_abs[w][c];
      n += s_n[w][c];
      top = max(top, s_max[w][c]);
    }
    // |sums| stay below about `addends` mean magnitudes and the largest one
    const float bound = addends * mag / (float)R + __uint_as_float((uint32_t)min(top + 1, 254) << 23);
    s_low[c] = mag > 0.f ? (int)(__float_as_uint(bound) >> 23) - kPartsLow : 0;
    limit = kPartsLimit * sqrtf((float)R * n / addends);
  }
  __syncthreads();
  const int low = s_low[c];
  int few = 0;
#pragma unroll
  for (int i = 0; i < U; i++)
    few += x[i] != 0.f && (int)((__float_as_uint(x[i]) >> 23) & 255u) < low ? 1 : 0;
#pragma unroll
  for (int o = 16; o >= COLS; o >>= 1) few += __shfl_xor_sync(kFull, few, o);
  if (lane < COLS) s_cnt[warp][c] = few;
  __syncthreads();
  bool over = false;
  if (threadIdx.x < COLS) {
    for (int w = 1; w < kWarps; w++) few += s_cnt[w][c];
    over = (float)few > limit;
  }
  over = __syncthreads_or(over || wrong);
  if (threadIdx.x == 0) {
    bad[blockIdx.x] = over ? 1 : 0;
    if (blockIdx.x == 0) *flag = 0;  // (k_split_b sets it)
  }
}

template <typename T>
int launch_t(const void* B, int64_t R, int64_t N, int64_t ldb, int* bad, int octaves, int64_t blocks, cudaStream_t s) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)blocks);
  cfg.blockDim = dim3(kWarps * 32);
  cfg.stream = s;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  BSP_CUDA(cudaLaunchKernelEx(&cfg, k_col_stats<T>, static_cast<const T*>(B), R, N, ldb, bad, octaves));
  return BSP_OK;
}

}  // namespace

size_t col_stats_bytes(int64_t N) { return (size_t)ceil_div(N, kStatCols) * 4 + 1024; }

int launch_col_stats(const void* B, int bdt, int64_t R, int64_t N, int64_t ldb, void* ws, int octaves,
                     const int** flags, int* n_flags, cudaStream_t s) {
  if (R > kStatMaxRows || N > INT32_MAX || N == 0) return BSP_ERR_CAPACITY;
  int* p = reinterpret_cast<int*>((reinterpret_cast<uintptr_t>(ws) + 255) & ~uintptr_t(255));
  const int64_t blocks = ceil_div(N, kStatCols);
  int* bad = p + 64;
  switch (bdt) {
    case BSP_F32: BSP_TRY(launch_t<float>(B, R, N, ldb, bad, octaves, blocks, s)); break;
    case BSP_BF16: BSP_TRY(launch_t<__nv_bfloat16>(B, R, N, ldb, bad, octaves, blocks, s)); break;
    case BSP_F16: BSP_TRY(launch_t<__half>(B, R, N, ldb, bad, octaves, blocks, s)); break;
    default: return BSP_ERR_UNSUPPORTED;
  }
  *flags = bad;
  *n_flags = (int)blocks;
  if (blocks > 512) {
    k_any<<<1, 1024, 0, s>>>(bad, blocks, p);
    BSP_LAUNCHED();
    *flags = p;
    *n_flags = 1;
  }
  return BSP_OK;
}

size_t parts_stats_bytes(int64_t N) { return (size_t)ceil_div(N, kStatCols) * 4 + 1024; }

int launch_parts_stats(const float* B, int64_t R, int64_t N, int64_t ldb, void* ws, float addends, PartsStats* st,
                       cudaStream_t s) {
  if (N > INT32_MAX / 8 || R > 32 * kPartsRows) return BSP_ERR_CAPACITY;
  st->flag = reinterpret_cast<int*>((reinterpret_cast<uintptr_t>(ws) + 255) & ~uintptr_t(255));
  st->bad = st->flag + 64;
  const unsigned grid = (unsigned)ceil_div(N, kStatCols);
  if (R <= 8 * kPartsRows) k_parts_stats<8><<<grid, kWarps * 32, 0, s>>>(B, R, N, ldb, st->bad, st->flag, addends);
  else if (R <= 16 * kPartsRows) k_parts_stats<16><<<grid, kWarps * 32, 0, s>>>(B, R, N, ldb, st->bad, st->flag, addends);
  else k_parts_stats<32><<<grid, kWarps * 32, 0, s>>>(B, R, N, ldb, st->bad, st->flag, addends);
  BSP_LAUNCHED();
  return BSP_OK;
}

}  // namespace bsp
