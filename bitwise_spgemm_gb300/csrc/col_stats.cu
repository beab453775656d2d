// col_stats.cu — sizes of a dense operand's values, column by column.
//
// Routes that add a column's values in another order, or through sums that a
// row of A does not hold, are exact enough only while the values of a column
// are of about one size; this kernel says so on the device, without a host
// wait, to the kernels behind it.
#include "spmm_dev.cuh"

namespace bsp {
namespace {

constexpr int kChunkRows = 128, kWarps = 8;

// A block takes 32 columns (a lane each) of 128 rows at a time, 8 loads of a
// warp in flight; its figures join the columns' by integer atomics (the same
// on every run), and the last block of 32 columns gives the verdict.  Bound by
// the one read of B (2048x1024 FP32, 8 MB: 3 us).
template <typename T>
__global__ void __launch_bounds__(kWarps * 32) k_col_stats(const T* __restrict__ B, int64_t R, int64_t N, int64_t ldb,
                                                           ColStats st, int octaves) {
  __shared__ int s_max[kWarps][32];
  __shared__ unsigned s_n[kWarps][32], s_sum[kWarps][32];
  __shared__ bool s_last;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int64_t col = (int64_t)blockIdx.x * 32 + lane;
  int top = 0;
  unsigned n = 0, sum = 0;
  for (int64_t r0 = (int64_t)blockIdx.y * kChunkRows; r0 < R; r0 += (int64_t)gridDim.y * kChunkRows) {
    const int64_t r1 = min(R, r0 + kChunkRows);
    for (int64_t r = r0 + warp; r < r1; r += kWarps * 8) {
      uint32_t x[8];
#pragma unroll
      for (int i = 0; i < 8; i++)
        x[i] = col < N && r + i * kWarps < r1 ? __float_as_uint(to_f32(__ldg(B + (r + i * kWarps) * ldb + col))) : 0u;
#pragma unroll
      for (int i = 0; i < 8; i++) {
        const int e = (int)((x[i] >> 23) & 255u);
        top = max(top, e);
        n += (x[i] << 1) != 0u;
        sum += (unsigned)e;
      }
    }
  }
  s_max[warp][lane] = top;
  s_n[warp][lane] = n;
  s_sum[warp][lane] = sum;
  __syncthreads();
  if (warp == 0) {
    for (int w = 1; w < kWarps; w++) {
      top = max(top, s_max[w][lane]);
      n += s_n[w][lane];
      sum += s_sum[w][lane];
    }
    if (col < N) {
      atomicMax(st.max_exp + col, top);
      if (octaves >= 0) {
        atomicAdd(st.nonzeros + col, n);
        atomicAdd(st.exp_sum + col, sum);
      }
    }
    __threadfence();
    __syncwarp();
    if (lane == 0) s_last = atomicAdd(st.done + blockIdx.x, 1u) + 1u == gridDim.y;
    __syncwarp();
    if (s_last && col < N) {
      __threadfence();
      const int m = atomicMax(st.max_exp + col, 0);
      bool bad = m >= kStatTop;
      if (octaves >= 0) {
        const unsigned long long c = atomicAdd(st.nonzeros + col, 0u), e = atomicAdd(st.exp_sum + col, 0u);
        bad |= (unsigned long long)m * c > e + (unsigned long long)octaves * c;
      }
      if (bad) atomicExch(st.flag, 1);
    }
  }
}

// The limits of a product in parts (ColStats): a block takes all rows of 8
// columns (whole sectors), four rows a warp and 8 loads of a lane in flight, so
// that nothing is handed between blocks and the sums' order is the same on every
// run.  A column with a value that is not finite or too large gets a limit that
// its first value breaks.  Bound by the latency of its rounds of loads: 5.6 us at
// 2048x1024, 4 of them in the step; with chunks of rows in blocks of their own,
// joined by the last one, 8.
constexpr int kPartsCols = 8, kPartsWarps = 32, kPartsLanes = 32 / kPartsCols, kPartsRows = kPartsLanes * kPartsWarps;
__global__ void __launch_bounds__(kPartsWarps * 32) k_parts_stats(const float* __restrict__ B, int64_t R, int64_t N,
                                                                  int64_t ldb, ColStats st, float addends) {
  __shared__ float s_abs[kPartsWarps][kPartsCols], s_n[kPartsWarps][kPartsCols];
  __shared__ int s_max[kPartsWarps][kPartsCols];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, c = lane % kPartsCols;
  const int64_t col = (int64_t)blockIdx.x * kPartsCols + c;
  float mag = 0.f, n = 0.f;
  int top = 0;
  for (int64_t r0 = warp * kPartsLanes + lane / kPartsCols; r0 < R; r0 += kPartsRows * 8) {
    float x[8];
#pragma unroll
    for (int i = 0; i < 8; i++) {
      const int64_t r = r0 + i * kPartsRows;
      x[i] = r < R && col < N ? __ldg(B + r * ldb + col) : 0.f;
    }
#pragma unroll
    for (int i = 0; i < 8; i++) {
      top = max(top, (int)((__float_as_uint(x[i]) >> 23) & 255u));
      n += x[i] != 0.f ? 1.f : 0.f;
      mag += fabsf(x[i]);
    }
  }
#pragma unroll
  for (int o = 16; o >= kPartsCols; o >>= 1) {
    mag += __shfl_xor_sync(kFull, mag, o);
    n += __shfl_xor_sync(kFull, n, o);
    top = max(top, __shfl_xor_sync(kFull, top, o));
  }
  if (lane < kPartsCols) {
    s_abs[warp][c] = mag;
    s_n[warp][c] = n;
    s_max[warp][c] = top;
  }
  __syncthreads();
  if (threadIdx.x >= kPartsCols || col >= N) return;
  for (int w = 1; w < kPartsWarps; w++) {
    mag += s_abs[w][c];
    n += s_n[w][c];
    top = max(top, s_max[w][c]);
  }
  if (blockIdx.x == 0 && threadIdx.x == 0) *st.flag = 0;  // (k_split_b sets it)
  // |sums| stay below about `addends` mean magnitudes and the largest one
  const float bound = addends * mag / (float)R + __uint_as_float((uint32_t)min(top + 1, 254) << 23);
  const bool bad = top >= kStatTop;
  st.low[col] = bad ? 256 : mag > 0.f ? (int)(__float_as_uint(bound) >> 23) - kPartsLow : 0;
  st.limit[col] = bad ? 0u : (unsigned)(kPartsLimit * sqrtf((float)R * n / addends));
  st.count[col] = 0u;
}

template <typename T>
int launch_t(const void* B, int64_t R, int64_t N, int64_t ldb, const ColStats& st, int octaves, cudaStream_t s) {
  const int64_t chunks = ceil_div(R, kChunkRows);
  k_col_stats<T><<<dim3((unsigned)ceil_div(N, 32), (unsigned)(chunks < 65535 ? chunks : 65535)), kWarps * 32, 0, s>>>(
      static_cast<const T*>(B), R, N, ldb, st, octaves);
  BSP_LAUNCHED();
  return BSP_OK;
}

}  // namespace

size_t col_stats_bytes(int64_t N) { return (size_t)(3 * N + ceil_div(N, 32)) * 4 + 512; }

int launch_col_stats(const void* B, int bdt, int64_t R, int64_t N, int64_t ldb, void* ws, int octaves, ColStats* st,
                     cudaStream_t s) {
  if (R > kStatMaxRows || N > INT32_MAX) return BSP_ERR_CAPACITY;
  int* p = reinterpret_cast<int*>((reinterpret_cast<uintptr_t>(ws) + 255) & ~uintptr_t(255));
  st->flag = p;
  st->max_exp = p + 64;
  st->done = reinterpret_cast<unsigned*>(st->max_exp + N);
  st->nonzeros = st->done + ceil_div(N, 32);
  st->exp_sum = st->nonzeros + N;
  BSP_CUDA(cudaMemsetAsync(p, 0, (size_t)(64 + N + ceil_div(N, 32) + (octaves >= 0 ? 2 * N : 0)) * 4, s));
  if (R == 0 || N == 0) return BSP_OK;
  switch (bdt) {
    case BSP_F32: return launch_t<float>(B, R, N, ldb, *st, octaves, s);
    case BSP_BF16: return launch_t<__nv_bfloat16>(B, R, N, ldb, *st, octaves, s);
    case BSP_F16: return launch_t<__half>(B, R, N, ldb, *st, octaves, s);
    default: return BSP_ERR_UNSUPPORTED;
  }
}

size_t parts_stats_bytes(int64_t N) { return (size_t)(3 * N + 8) * 4 + 1024; }

int launch_parts_stats(const float* B, int64_t R, int64_t N, int64_t ldb, void* ws, float addends, ColStats* st,
                       cudaStream_t s) {
  if (N > INT32_MAX / 8) return BSP_ERR_CAPACITY;
  int* p = reinterpret_cast<int*>((reinterpret_cast<uintptr_t>(ws) + 255) & ~uintptr_t(255));
  st->flag = p;
  st->low = p + 64;  // (read 8 at a time)
  st->limit = reinterpret_cast<unsigned*>(st->low + N + 8);
  st->count = st->limit + N;
  k_parts_stats<<<(unsigned)ceil_div(N, kPartsCols), kPartsWarps * 32, 0, s>>>(B, R, N, ldb, *st, addends);
  BSP_LAUNCHED();
  return BSP_OK;
}

}  // namespace bsp
