// pack.cu — bit packing, transposition, unpacking and bit-plane split.
//
// All kernels are HBM-bound streaming passes.  A word of 32 columns is built
// by one warp ballot (lane i tests column 32w+i), which replaces the
// per-nonzero global atomicOr of dense2bitmask (reference
// source/src/main.cu:611-621) and the one-int-per-bit output of
// uint8_layout_trans (backup/layout_trans.cu:87-97).
#include "bsp_internal.cuh"

namespace bsp {
namespace {

// Nonzero test with the reference's `x != 0` semantics (main.cu:617):
// -0.0 is zero, NaN is nonzero.
template <int DT> struct Elem;
template <> struct Elem<BSP_F32> {
  using T = float;
  __device__ static bool nz(T x) { return x != 0.0f; }
};
template <> struct Elem<BSP_F16> {
  using T = uint16_t;
  __device__ static bool nz(T x) { return (x & 0x7fffu) != 0; }
};
template <> struct Elem<BSP_BF16> {
  using T = uint16_t;
  __device__ static bool nz(T x) { return (x & 0x7fffu) != 0; }
};
template <> struct Elem<BSP_I8> {
  using T = int8_t;
  __device__ static bool nz(T x) { return x != 0; }
};
template <> struct Elem<BSP_U8> {
  using T = uint8_t;
  __device__ static bool nz(T x) { return x != 0; }
};

// Rows that start 16-byte aligned.  A lane loads 16 bytes (VEC columns), makes
// their VEC bits, and the G = 32 / VEC lanes of a word OR theirs together; a
// warp takes U such loads (512 columns of FP32, 1024 of the narrower types)
// before it stores, so 2 KB a warp are in flight.  Bound by HBM: the form
// that built a word by one ballot of 32 scalar loads, with a 64-bit division
// per word, read 4096x4096 FP32 at 1.5 TB/s (45 us); this one takes 13 us.
template <int DT> struct PackVec;
template <> struct PackVec<BSP_F32> {
  static constexpr int VEC = 4, U = 4;
  __device__ static uint32_t bits(const uint4& q) {
    // x != 0 for -0.0 (no) and NaN (yes): any bit but the sign
    return ((q.x << 1) ? 1u : 0u) | ((q.y << 1) ? 2u : 0u) | ((q.z << 1) ? 4u : 0u) | ((q.w << 1) ? 8u : 0u);
  }
};
template <> struct PackVec<BSP_F16> {
  static constexpr int VEC = 8, U = 4;
  __device__ static uint32_t two(uint32_t x) { return ((x & 0x7fffu) ? 1u : 0u) | ((x & 0x7fff0000u) ? 2u : 0u); }
  __device__ static uint32_t bits(const uint4& q) {
    return two(q.x) | (two(q.y) << 2) | (two(q.z) << 4) | (two(q.w) << 6);
  }
};
template <> struct PackVec<BSP_BF16> : PackVec<BSP_F16> {};
template <> struct PackVec<BSP_U8> {
  static constexpr int VEC = 16, U = 2;
  // bytes 0..3 of x != 0 -> bits 0..3 (the multiply moves bit 8i to bit 24+i)
  __device__ static uint32_t four(uint32_t x) { return ((__vcmpne4(x, 0u) & 0x01010101u) * 0x01020408u) >> 24; }
  __device__ static uint32_t bits(const uint4& q) {
    return four(q.x) | (four(q.y) << 4) | (four(q.z) << 8) | (four(q.w) << 12);
  }
};
template <> struct PackVec<BSP_I8> : PackVec<BSP_U8> {};

template <int DT>
__global__ void __launch_bounds__(256) k_pack_rows_v16(const typename Elem<DT>::T* __restrict__ dense, int64_t M,
                                                       int64_t K, int64_t ld, uint32_t* __restrict__ words,
                                                       int64_t Kw, int msb) {
  using E = Elem<DT>;
  using V = PackVec<DT>;
  constexpr int G = 32 / V::VEC, WPL = 32 / G;  // lanes per word, words per load of the warp
  static_assert(V::U <= G, "a lane of every word's group for each load");
  const int lane = threadIdx.x & 31;
  const int64_t warp = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 5;
  const int64_t nwarps = ((int64_t)gridDim.x * blockDim.x) >> 5;
  const int64_t nch = (Kw + WPL * V::U - 1) / (WPL * V::U);
  const int64_t total = M * nch;
  for (int64_t t = warp; t < total; t += nwarps) {
    const int64_t r = total <= 0x7fffffff ? (int64_t)((uint32_t)t / (uint32_t)nch) : t / nch;
    const int64_t ch = t - r * nch;
    const typename E::T* row = dense + r * ld;
    const int64_t c0 = ch * (32 * WPL * V::U) + lane * V::VEC;
    uint4 q[V::U];
#pragma unroll
    for (int u = 0; u < V::U; u++) {
      const int64_t c = c0 + u * (32 * WPL);
      q[u] = make_uint4(0u, 0u, 0u, 0u);
      if (c + V::VEC <= K) q[u] = __ldg(reinterpret_cast<const uint4*>(row + c));
    }
    uint32_t mine = 0;
#pragma unroll
    for (int u = 0; u < V::U; u++) {
      const int64_t c = c0 + u * (32 * WPL);
      uint32_t b = V::bits(q[u]);
      if (c < K && c + V::VEC > K)  // the row's last columns
        for (int i = 0; i < V::VEC; i++)
          if (c + i < K && E::nz(row[c + i])) b |= 1u << i;
      b <<= V::VEC * (lane % G);
#pragma unroll
      for (int o = 1; o < G; o <<= 1) b |= __shfl_xor_sync(kFull, b, o);
      if (lane % G == u) mine = b;
    }
    const int64_t w = ch * (WPL * V::U) + (lane % G) * WPL + lane / G;
    if (lane % G < V::U && w < Kw) words[r * Kw + w] = msb ? __brev(mine) : mine;
  }
}

// Rows of up to kNarrowWords words: a warp takes 8 words one after the other,
// over the rows' ends, 8 loads in flight.  (A warp per row, as below, has one
// to three: 1048576x32 U8 194 us, here 45; 1048576x64 195 and 86.)
constexpr int64_t kNarrowWords = 3;
template <int DT>
__global__ void __launch_bounds__(256) k_pack_rows_narrow(const typename Elem<DT>::T* __restrict__ dense, int64_t M,
                                                          int64_t K, int64_t ld, uint32_t* __restrict__ words,
                                                          int64_t Kw, int msb) {
  using E = Elem<DT>;
  const int lane = threadIdx.x & 31;
  const int64_t warp = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 5;
  const int64_t nwarps = ((int64_t)gridDim.x * blockDim.x) >> 5;
  const int64_t total = M * Kw;
  for (int64_t base = warp * 8; base < total; base += nwarps * 8) {
    int64_t r = base / Kw;
    int w = (int)(base - r * Kw);
    bool nz[8];
#pragma unroll
    for (int j = 0; j < 8; j++) {
      const int64_t c = w * 32 + lane;
      nz[j] = r < M && c < K ? E::nz(dense[r * ld + c]) : false;
      if (++w == (int)Kw) w = 0, r++;
    }
    uint32_t mine = 0;
#pragma unroll
    for (int j = 0; j < 8; j++) {
      const uint32_t b = __ballot_sync(kFull, nz[j]);
      if (lane == j) mine = b;
    }
    if (lane < 8 && base + lane < total) words[base + lane] = msb ? __brev(mine) : mine;
  }
}

// Any alignment: a warp takes 32 words of a row, one coalesced load of 32
// columns and one ballot per word, 8 loads in flight; lane j keeps word j.
template <int DT>
__global__ void __launch_bounds__(256) k_pack_rows(const typename Elem<DT>::T* __restrict__ dense,
                                                   int64_t M, int64_t K, int64_t ld,
                                                   uint32_t* __restrict__ words, int64_t Kw,
                                                   int msb) {
  using E = Elem<DT>;
  const int lane = threadIdx.x & 31;
  const int64_t warp = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 5;
  const int64_t nwarps = ((int64_t)gridDim.x * blockDim.x) >> 5;
  const int64_t nch = (Kw + 31) / 32;
  const int64_t total = M * nch;
  for (int64_t t = warp; t < total; t += nwarps) {
    const int64_t r = total <= 0x7fffffff ? (int64_t)((uint32_t)t / (uint32_t)nch) : t / nch;
    const int64_t w0 = (t - r * nch) * 32;
    const typename E::T* row = dense + r * ld;
    const int nw = (int)(Kw - w0 < 32 ? Kw - w0 : 32);
    uint32_t mine = 0;
    for (int j0 = 0; j0 < nw; j0 += 8) {
      bool nz[8];
#pragma unroll
      for (int j = 0; j < 8; j++) {
        const int64_t c = (w0 + j0 + j) * 32 + lane;
        nz[j] = c < K ? E::nz(row[c]) : false;
      }
#pragma unroll
      for (int j = 0; j < 8; j++) {
        const uint32_t b = __ballot_sync(kFull, nz[j]);
        if (lane == j0 + j) mine = b;
      }
    }
    if (lane < nw) words[r * Kw + w0 + lane] = msb ? __brev(mine) : mine;
  }
}

// Column packing: a warp owns rows 32*mw .. 32*mw+31 (lane = row) and 32
// consecutive columns; ballot over lanes for column k yields words_t[k][mw].
template <int DT>
__global__ void __launch_bounds__(256) k_pack_cols(const typename Elem<DT>::T* __restrict__ dense,
                                                   int64_t M, int64_t K, int64_t ld,
                                                   uint32_t* __restrict__ words_t, int64_t Mw,
                                                   int msb) {
  using E = Elem<DT>;
  const int lane = threadIdx.x & 31;
  const int64_t warp = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 5;
  const int64_t nwarps = ((int64_t)gridDim.x * blockDim.x) >> 5;
  const int64_t Kc = (K + 31) / 32;
  const int64_t total = Mw * Kc;
  for (int64_t t = warp; t < total; t += nwarps) {
    const int64_t mw = t / Kc;
    const int64_t k0 = (t - mw * Kc) * 32;
    const int64_t r = mw * 32 + lane;
    uint32_t mine = 0;
#pragma unroll 8
    for (int j = 0; j < 32; j++) {
      const int64_t k = k0 + j;
      const bool nz = (r < M && k < K) ? E::nz(dense[r * ld + k]) : false;
      uint32_t b = __ballot_sync(kFull, nz);
      if (msb) b = __brev(b);
      if (lane == j) mine = b;
    }
    if (k0 + lane < K) words_t[(k0 + lane) * Mw + mw] = mine;
  }
}

// 32x32 bit-block transpose: lane i holds row 32*mw+i's word w; ballot of bit
// j across lanes is column 32w+j of the transpose.
__global__ void __launch_bounds__(256) k_transpose_bits(const uint32_t* __restrict__ words,
                                                        int64_t M, int64_t Kw, int64_t K,
                                                        uint32_t* __restrict__ words_t, int64_t Mw,
                                                        const int* __restrict__ run_if) {
  if (run_if && !__ldg(run_if)) return;
  const int lane = threadIdx.x & 31;
  const int64_t warp = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 5;
  const int64_t nwarps = ((int64_t)gridDim.x * blockDim.x) >> 5;
  const int64_t total = Mw * Kw;
  for (int64_t t = warp; t < total; t += nwarps) {
    const int64_t mw = t / Kw;
    const int64_t w = t - mw * Kw;
    const int64_t r = mw * 32 + lane;
    const uint32_t my = r < M ? words[r * Kw + w] : 0u;
    uint32_t mine = 0;
#pragma unroll
    for (int j = 0; j < 32; j++) {
      const uint32_t b = __ballot_sync(kFull, (my >> j) & 1u);
      if (lane == j) mine = b;
    }
    const int64_t k = w * 32 + lane;
    if (k < K) words_t[k * Mw + mw] = mine;
  }
}

// Thread per element; `one` is the dtype's bit pattern of 1.
template <typename T>
__global__ void __launch_bounds__(256) k_unpack_rows(const uint32_t* __restrict__ words, int64_t M,
                                                     int64_t K, int64_t Kw, T* __restrict__ dense,
                                                     int64_t ld, int msb, T one) {
  const int64_t n = M * K;
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n;
       i += (int64_t)gridDim.x * blockDim.x) {
    const int64_t r = i / K;
    const int64_t c = i - r * K;
    const uint32_t w = words[r * Kw + c / 32];
    const int bit = msb ? 31 - (int)(c & 31) : (int)(c & 31);
    dense[r * ld + c] = ((w >> bit) & 1u) ? one : T(0);
  }
}

// Warp per (row, word): lane c loads one byte, one ballot per plane.
__global__ void __launch_bounds__(256) k_bitplanes(const uint8_t* __restrict__ v, int64_t M,
                                                   int64_t K, int64_t ld, int planes,
                                                   uint32_t* __restrict__ words, int64_t Kw,
                                                   int msb, int rows_layout) {
  const int lane = threadIdx.x & 31;
  const int64_t warp = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 5;
  const int64_t nwarps = ((int64_t)gridDim.x * blockDim.x) >> 5;
  const int64_t total = M * Kw;
  for (int64_t t = warp; t < total; t += nwarps) {
    const int64_t r = t / Kw;
    const int64_t w = t - r * Kw;
    const int64_t c = w * 32 + lane;
    const uint32_t x = c < K ? v[r * ld + c] : 0u;
    uint32_t mine = 0;
#pragma unroll
    for (int b = 0; b < 8; b++) {
      if (b < planes) {
        uint32_t m = __ballot_sync(kFull, (x >> b) & 1u);
        if (msb) m = __brev(m);
        if (lane == b) mine = m;
      }
    }
    if (lane < planes)
      words[(rows_layout ? (r * planes + lane) : ((int64_t)lane * M + r)) * Kw + w] = mine;
  }
}

// 8x8 bit-matrix transpose of a uint64 (byte i = row i): afterwards byte b,
// bit i holds bit b of byte i (Hacker's Delight, section 7-3, transpose8).
__device__ __forceinline__ uint64_t transpose8x8(uint64_t x) {
  x = (x & 0xAA55AA55AA55AA55ull) | ((x & 0x00AA00AA00AA00AAull) << 7) | ((x >> 7) & 0x00AA00AA00AA00AAull);
  x = (x & 0xCCCC3333CCCC3333ull) | ((x & 0x0000CCCC0000CCCCull) << 14) | ((x >> 14) & 0x0000CCCC0000CCCCull);
  x = (x & 0xF0F0F0F00F0F0F0Full) | ((x & 0x00000000F0F0F0F0ull) << 28) | ((x >> 28) & 0x00000000F0F0F0F0ull);
  return x;
}

// Bit planes from 16-byte rows: a warp takes 512 columns of a row (lane l
// columns 16l..16l+15, one vector load), two 8x8 transposes give the lane's
// 16-bit mask of every plane, and the even lane of each pair joins its mask
// with its neighbour's into the 32-column word.  Rows must start 16-byte
// aligned (ld % 16 == 0); the ragged end of a row is read byte by byte.
__global__ void __launch_bounds__(256) k_bitplanes_v16(const uint8_t* __restrict__ v, int64_t M, int64_t K,
                                                       int64_t ld, int planes, uint32_t* __restrict__ words,
                                                       int64_t Kw, int msb, int rows_layout) {
  const int lane = threadIdx.x & 31;
  const int64_t warp = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 5;
  const int64_t nwarps = ((int64_t)gridDim.x * blockDim.x) >> 5;
  const int64_t nch = (K + 511) / 512;
  for (int64_t t = warp; t < M * nch; t += nwarps) {
    const int64_t r = t / nch, ch = t - r * nch;
    const int64_t c = ch * 512 + lane * 16;
    const uint8_t* p = v + r * ld + c;
    uint64_t x0 = 0, x1 = 0;
    if (c + 16 <= K) {
      const uint4 q = __ldg(reinterpret_cast<const uint4*>(p));
      x0 = (uint64_t)q.x | ((uint64_t)q.y << 32);
      x1 = (uint64_t)q.z | ((uint64_t)q.w << 32);
    } else {
      for (int i = 0; i < 16; i++)
        if (c + i < K) {
          const uint64_t b = p[i];
          if (i < 8) x0 |= b << (8 * i);
          else x1 |= b << (8 * (i - 8));
        }
    }
    x0 = transpose8x8(x0);
    x1 = transpose8x8(x1);
    // m[q] = 16-bit masks of planes 2q (low half) and 2q+1 (high half)
    uint32_t m[4], n[4];
#pragma unroll
    for (int q = 0; q < 4; q++) {
      m[q] = (uint32_t)((x0 >> (16 * q)) & 0xff) | ((uint32_t)((x1 >> (16 * q)) & 0xff) << 8) |
             ((uint32_t)((x0 >> (16 * q + 8)) & 0xff) << 16) | ((uint32_t)((x1 >> (16 * q + 8)) & 0xff) << 24);
      n[q] = __shfl_down_sync(kFull, m[q], 1);
    }
    const int64_t w = ch * 16 + (lane >> 1);
    if ((lane & 1) == 0 && w < Kw) {
#pragma unroll
      for (int b = 0; b < 8; b++) {
        if (b >= planes) break;
        const int sh = 16 * (b & 1);
        uint32_t word = ((m[b >> 1] >> sh) & 0xffffu) | (((n[b >> 1] >> sh) & 0xffffu) << 16);
        if (msb) word = __brev(word);
        words[(rows_layout ? (r * planes + b) : ((int64_t)b * M + r)) * Kw + w] = word;
      }
    }
  }
}

int grid_for(int64_t warps_needed) {
  const int64_t blocks = ceil_div(warps_needed, 8);
  const int64_t cap = (int64_t)num_sms() * 16;
  return (int)(blocks < 1 ? 1 : (blocks > cap ? cap : blocks));
}

}  // namespace

template <int DT>
static void pack_rows_t(const void* dense, int64_t M, int64_t K, int64_t ld, uint32_t* words, int64_t Kw, int msb,
                        cudaStream_t s) {
  using T = typename Elem<DT>::T;
  using V = PackVec<DT>;
  // 16-byte loads need every row to start on 16 bytes; a row narrower than
  // one load of the warp leaves most of its lanes idle there
  if (is_aligned(dense, 16) && (ld * (int64_t)sizeof(T)) % 16 == 0 && K >= 32 * V::VEC)
    k_pack_rows_v16<DT><<<grid_for(M * ceil_div(Kw, V::VEC * V::U)), 256, 0, s>>>((const T*)dense, M, K, ld, words, Kw,
                                                                               msb);
  else if (Kw <= kNarrowWords)
    k_pack_rows_narrow<DT><<<grid_for(ceil_div(M * Kw, 8)), 256, 0, s>>>((const T*)dense, M, K, ld, words, Kw, msb);
  else
    k_pack_rows<DT><<<grid_for(M * ceil_div(Kw, 32)), 256, 0, s>>>((const T*)dense, M, K, ld, words, Kw, msb);
}

int launch_pack_rows(const void* dense, int dtype, int64_t M, int64_t K, int64_t ld,
                     uint32_t* words, int msb, cudaStream_t s) {
  const int64_t Kw = ceil_div(K, 32);
  switch (dtype) {
    case BSP_F32: pack_rows_t<BSP_F32>(dense, M, K, ld, words, Kw, msb, s); break;
    case BSP_F16: pack_rows_t<BSP_F16>(dense, M, K, ld, words, Kw, msb, s); break;
    case BSP_BF16: pack_rows_t<BSP_BF16>(dense, M, K, ld, words, Kw, msb, s); break;
    case BSP_I8: pack_rows_t<BSP_I8>(dense, M, K, ld, words, Kw, msb, s); break;
    case BSP_U8: pack_rows_t<BSP_U8>(dense, M, K, ld, words, Kw, msb, s); break;
    default: return BSP_ERR_INVALID_ARG;
  }
  BSP_LAUNCHED();
  return BSP_OK;
}

int launch_pack_cols(const void* dense, int dtype, int64_t M, int64_t K, int64_t ld,
                     uint32_t* words_t, int msb, cudaStream_t s) {
  const int64_t Mw = ceil_div(M, 32);
  const int grid = grid_for(Mw * ceil_div(K, 32));
  switch (dtype) {
    case BSP_F32: k_pack_cols<BSP_F32><<<grid, 256, 0, s>>>((const float*)dense, M, K, ld, words_t, Mw, msb); break;
    case BSP_F16: k_pack_cols<BSP_F16><<<grid, 256, 0, s>>>((const uint16_t*)dense, M, K, ld, words_t, Mw, msb); break;
    case BSP_BF16: k_pack_cols<BSP_BF16><<<grid, 256, 0, s>>>((const uint16_t*)dense, M, K, ld, words_t, Mw, msb); break;
    case BSP_I8: k_pack_cols<BSP_I8><<<grid, 256, 0, s>>>((const int8_t*)dense, M, K, ld, words_t, Mw, msb); break;
    case BSP_U8: k_pack_cols<BSP_U8><<<grid, 256, 0, s>>>((const uint8_t*)dense, M, K, ld, words_t, Mw, msb); break;
    default: return BSP_ERR_INVALID_ARG;
  }
  BSP_LAUNCHED();
  return BSP_OK;
}

int launch_transpose_bits(const uint32_t* words, int64_t M, int64_t K, uint32_t* words_t,
                          cudaStream_t s, const int* run_if) {
  const int64_t Kw = ceil_div(K, 32), Mw = ceil_div(M, 32);
  k_transpose_bits<<<grid_for(Mw * Kw), 256, 0, s>>>(words, M, Kw, K, words_t, Mw, run_if);
  BSP_LAUNCHED();
  return BSP_OK;
}

int launch_unpack_rows(const uint32_t* words, int64_t M, int64_t K, void* dense, int dtype,
                       int64_t ld, int msb, cudaStream_t s) {
  const int64_t Kw = ceil_div(K, 32);
  const int grid = grid_for(ceil_div(M * K, 32));
  switch (dtype) {
    case BSP_F32: k_unpack_rows<float><<<grid, 256, 0, s>>>(words, M, K, Kw, (float*)dense, ld, msb, 1.0f); break;
    case BSP_F16: k_unpack_rows<uint16_t><<<grid, 256, 0, s>>>(words, M, K, Kw, (uint16_t*)dense, ld, msb, (uint16_t)0x3c00u); break;
    case BSP_BF16: k_unpack_rows<uint16_t><<<grid, 256, 0, s>>>(words, M, K, Kw, (uint16_t*)dense, ld, msb, (uint16_t)0x3f80u); break;
    case BSP_I8:
    case BSP_U8: k_unpack_rows<uint8_t><<<grid, 256, 0, s>>>(words, M, K, Kw, (uint8_t*)dense, ld, msb, (uint8_t)1u); break;
    default: return BSP_ERR_INVALID_ARG;
  }
  BSP_LAUNCHED();
  return BSP_OK;
}

int launch_bitplanes(const uint8_t* v, int64_t M, int64_t K, int64_t ld, int planes,
                     uint32_t* words, int msb, cudaStream_t s, int rows_layout) {
  const int64_t Kw = ceil_div(K, 32);
  if (is_aligned(v, 16) && ld % 16 == 0)
    k_bitplanes_v16<<<grid_for(M * ceil_div(K, 512)), 256, 0, s>>>(v, M, K, ld, planes, words, Kw, msb,
                                                                  rows_layout);
  else
    k_bitplanes<<<grid_for(M * Kw), 256, 0, s>>>(v, M, K, ld, planes, words, Kw, msb, rows_layout);
  BSP_LAUNCHED();
  return BSP_OK;
}

}  // namespace bsp
