// output.cu — the steps around the SpMM when the operands are themselves
// bitmaps or multi-bit values:
//
//  * symbolic output masks: for A (M×K) and B (K×N) both given as packed
//    bit rows, row i of C's mask is the OR of B's row masks at A's set bits
//    (the symbolic half of pre_spgemm, reference source/src/transform.cuh:
//    1028-1057, which walked a CSR copy of A one thread per row and kept the
//    mask in shared memory).  The first-fit grouping of the output rows that
//    follows it there is bsp_group_rows on the result.
//  * bit-plane products: C = Σ_b w_b · (P_b · B) for the 0/1 planes P_b of
//    an 8-bit matrix, w_b = 2^b and, for two's complement values, −2^7 for
//    the top plane — the recombination of spgemm_compute_1dthread_tcore_v3
//    (transform.cuh:2199-2246) with the weights of initialize_multiplicand
//    (main.cu:895-910).  There every plane went through a wmma tile of half
//    values and shared-memory atomics; here one warp walks the planes of a
//    row, sums each plane in FP32 (TwoSum compensated) and adds it, scaled by
//    its power-of-two weight (exact), to the row's total.
#include <climits>
#include <type_traits>

#include "ptx.cuh"
#include "spmm_dev.cuh"

namespace bsp {
namespace {

constexpr int kSymWords = 4;  // output words per lane (128 per warp)
constexpr int kSymDepth = 8;  // B row masks in flight per warp

// One warp per (row of C, 128-word chunk of its mask).  The walker yields
// A's set bits in ascending order; columns at or past K (stray bits in the
// padding of A's last word) are ignored.
__global__ void __launch_bounds__(256) k_symbolic_rows(const uint32_t* __restrict__ A, int64_t M, int64_t K,
                                                       int64_t Kw, const uint32_t* __restrict__ Bw, int64_t Nw,
                                                       uint32_t* __restrict__ Cw) {
  const int lane = threadIdx.x & 31;
  const int64_t row = (int64_t)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
  if (row >= M) return;
  const int64_t w0 = (int64_t)blockIdx.y * (32 * kSymWords);
  uint32_t acc[kSymWords] = {};
  BitWalker wk;
  wk.init(A + row * Kw, 0, (int)Kw, lane);
  while (true) {
    uint32_t idx[kSymDepth];
#pragma unroll
    for (int s = 0; s < kSymDepth; s++) idx[s] = wk.next();
    if (idx[0] == kEnd) break;
    uint32_t v[kSymDepth][kSymWords];
#pragma unroll
    for (int s = 0; s < kSymDepth; s++)
#pragma unroll
      for (int q = 0; q < kSymWords; q++) {
        const int64_t w = w0 + q * 32 + lane;
        v[s][q] = (idx[s] != kEnd && (int64_t)idx[s] < K && w < Nw) ? __ldg(Bw + (int64_t)idx[s] * Nw + w) : 0u;
      }
#pragma unroll
    for (int s = 0; s < kSymDepth; s++)
#pragma unroll
      for (int q = 0; q < kSymWords; q++) acc[q] |= v[s][q];
    if (idx[kSymDepth - 1] == kEnd) break;
  }
#pragma unroll
  for (int q = 0; q < kSymWords; q++) {
    const int64_t w = w0 + q * 32 + lane;
    if (w < Nw) Cw[row * Nw + w] = acc[q];
  }
}

// ---- symbolic masks through a prototype plan ------------------------------
// Row i of cluster c holds the cluster's consensus columns without those that
// it removes, and the columns that it adds.  Bit j of its mask is set if an
// added column's B mask has it, or if more of the consensus columns' masks
// have it than of the removed ones' (every removed column is in the
// consensus) — exact.  Counts are kept bit-sliced: plane p of a word holds
// bit p of its 32 columns' counts (16 planes: counts < 65536, which K < 65536
// guarantees).  Eight masks are counted at a time by full adders over whole
// words (two three-input operations each), and a count is compared with
// another by one such operation per plane.  A row then reads its cluster's
// planes in use and its delta rows' masks (≈16 for the clustered workload)
// instead of the mask of every set bit (≈425).
constexpr int kSymPlanes = 16;
constexpr int kSymCWords = 64;   // output words per CTA of the plane kernel
constexpr int kSymCGroups = 8;   // consensus parts per CTA of the plane kernel
constexpr int kSymRows = 8;      // rows per CTA of the planned row kernel
constexpr int kSymPWords = 2;    // output words per lane of the planned row kernel (64 per warp)

// a + b + c of every bit: the sum's low bit, the carry
__device__ __forceinline__ void full_add(uint32_t a, uint32_t b, uint32_t c, uint32_t* sum, uint32_t* carry) {
  *sum = a ^ b ^ c;
  *carry = (a & b) | (a & c) | (b & c);
}

// pl += the number of masks among x[0..8) that have the bit
template <int P>
__device__ __forceinline__ void planes_add8(uint32_t (&pl)[P], const uint32_t (&x)[8]) {
  uint32_t s1, s2, s3, c1, c2, c3, c4, t1, d1, d2, e;
  full_add(x[0], x[1], x[2], &s1, &c1);
  full_add(x[3], x[4], x[5], &s2, &c2);
  full_add(x[6], x[7], pl[0], &s3, &c3);
  full_add(s1, s2, s3, &pl[0], &c4);
  full_add(c1, c2, c3, &t1, &d1);
  full_add(t1, c4, pl[1], &pl[1], &d2);
  full_add(d1, d2, pl[2], &pl[2], &e);
#pragma unroll
  for (int p = 3; p < P; p++) {
    if (!e) break;
    const uint32_t carry = pl[p] & e;
    pl[p] ^= e;
    e = carry;
  }
}

// planes[c][p][w] for cluster c = blockIdx.x, words w of chunk blockIdx.y:
// thread (g, wl) counts its word's column bits over part g of the consensus
// columns (8 masks in flight), and the parts' planes are added up through
// shared memory.  Bound by the latency of the masks' gathers; one ripple of
// carries per mask, with the parts joined as counts of single columns by
// shared-memory atomics, took 27 us at 66 clusters x 8192 columns, this
// takes 17.
__global__ void __launch_bounds__(kSymCWords * kSymCGroups) k_sym_cluster_planes(
    const uint32_t* __restrict__ cons, int64_t Kw, int64_t K, const uint32_t* __restrict__ Bw, int64_t Nw,
    uint32_t* __restrict__ planes, int* __restrict__ top) {
  static_assert(kSymDepth == 8, "planes_add8");
  __shared__ uint32_t part[kSymCGroups][kSymPlanes][kSymCWords];
  const int lane = threadIdx.x & 31;
  const int g = threadIdx.x / kSymCWords, wl = threadIdx.x % kSymCWords;
  const int64_t c = blockIdx.x;
  const int64_t w = (int64_t)blockIdx.y * kSymCWords + wl;
  uint32_t pl[kSymPlanes];
#pragma unroll
  for (int p = 0; p < kSymPlanes; p++) pl[p] = 0u;
  BitWalker wk;
  wk.init(cons + c * Kw, (int)(Kw * g / kSymCGroups), (int)(Kw * (g + 1) / kSymCGroups), lane);
  while (true) {
    uint32_t idx[kSymDepth], v[kSymDepth];
#pragma unroll
    for (int s = 0; s < kSymDepth; s++) idx[s] = wk.next();
    if (idx[0] == kEnd) break;
#pragma unroll
    for (int s = 0; s < kSymDepth; s++)
      v[s] = (idx[s] != kEnd && (int64_t)idx[s] < K && w < Nw) ? __ldg(Bw + (int64_t)idx[s] * Nw + w) : 0u;
    planes_add8(pl, v);
    if (idx[kSymDepth - 1] == kEnd) break;
  }
#pragma unroll
  for (int p = 0; p < kSymPlanes; p++) part[g][p][wl] = pl[p];
  __syncthreads();
  // (whole warps: two of the first group)
  if (g == 0) {
    int used = 0;  // planes up to the highest nonzero one
    uint32_t carry[kSymCGroups - 1];
#pragma unroll
    for (int h = 0; h + 1 < kSymCGroups; h++) carry[h] = 0u;
#pragma unroll
    for (int p = 0; p < kSymPlanes; p++) {
      uint32_t sum = pl[p];
#pragma unroll
      for (int h = 1; h < kSymCGroups; h++) full_add(sum, part[h][p][wl], carry[h - 1], &sum, &carry[h - 1]);
      if (w < Nw) {
        planes[(c * kSymPlanes + p) * Nw + w] = sum;
        if (sum) used = p + 1;
      }
    }
    used = __reduce_max_sync(kFull, used);
    if (lane == 0 && used) atomicMax(top + c, used);
  }
}

// One warp per (row of C, 64-word chunk): clustered rows count their removed
// columns' masks, compare with their cluster's planes and OR their added
// columns'; a row without a cluster is the OR of its set bits' masks, by the
// whole block: one warp's chain of gathers for such a row, 433 bits long, made
// all of 8192x8192x8192 take 66 us (45 now; 53 with the words of a lane apart
// and a walker over the list).  Bound by the issue of the counting and by the
// latency of the gathers.
template <bool PAIR>
__global__ void __launch_bounds__(256, 4) k_sym_rows_planned(const uint32_t* __restrict__ A, int64_t M, int64_t K,
                                                          int64_t Kw, const uint32_t* __restrict__ Bw, int64_t Nw,
                                                          const int32_t* __restrict__ row_cluster,
                                                          const int32_t* __restrict__ delta_ptr,
                                                          const uint32_t* __restrict__ delta_idx,
                                                          const uint32_t* __restrict__ planes,
                                                          const int* __restrict__ top, uint32_t* __restrict__ Cw) {
  static_assert(kSymPWords == 2, "PAIR");
  const int lane = threadIdx.x & 31;
  const int warp = threadIdx.x >> 5;
  const int64_t row0 = (int64_t)blockIdx.x * kSymRows, row = row0 + warp;
  const int64_t w0 = (int64_t)blockIdx.y * (32 * kSymPWords);
  int64_t wq[kSymPWords];
  bool wv[kSymPWords];
#pragma unroll
  for (int q = 0; q < kSymPWords; q++) {
    wq[q] = w0 + (PAIR ? lane * 2 + q : q * 32 + lane);
    wv[q] = wq[q] < Nw;
  }
  const int cl = row < M ? __ldg(row_cluster + row) : 0;
  uint32_t out[kSymPWords];
#pragma unroll
  for (int q = 0; q < kSymPWords; q++) out[q] = 0u;
  // rows without a cluster: the whole block walks each, an eighth a warp
  if (__syncthreads_or(cl < 0)) {
    __shared__ uint32_t masks[kSymRows][32 * kSymPWords];
    for (int i = threadIdx.x; i < kSymRows * 32 * kSymPWords; i += blockDim.x) (&masks[0][0])[i] = 0u;
    __syncthreads();
    for (int r = 0; r < kSymRows; r++) {
      if (row0 + r >= M || __ldg(row_cluster + row0 + r) >= 0) continue;
      uint32_t got[kSymPWords];
#pragma unroll
      for (int q = 0; q < kSymPWords; q++) got[q] = 0u;
      BitWalker wk;
      wk.init(A + (row0 + r) * Kw, (int)(Kw * warp / kSymRows), (int)(Kw * (warp + 1) / kSymRows), lane);
      while (true) {
        uint32_t idx[kSymDepth];
#pragma unroll
        for (int s = 0; s < kSymDepth; s++) idx[s] = wk.next();
        if (idx[0] == kEnd) break;
#pragma unroll
        for (int s = 0; s < kSymDepth; s++)
#pragma unroll
          for (int q = 0; q < kSymPWords; q++)
            got[q] |= (idx[s] != kEnd && (int64_t)idx[s] < K && wv[q]) ? __ldg(Bw + (int64_t)idx[s] * Nw + wq[q]) : 0u;
        if (idx[kSymDepth - 1] == kEnd) break;
      }
#pragma unroll
      for (int q = 0; q < kSymPWords; q++)
        if (got[q]) atomicOr(&masks[r][q * 32 + lane], got[q]);
    }
    __syncthreads();
    if (cl < 0)
#pragma unroll
      for (int q = 0; q < kSymPWords; q++) out[q] = masks[warp][q * 32 + lane];
  }
  if (row >= M) return;
  if (cl >= 0) {
    const int d0 = __ldg(delta_ptr + row), d1 = __ldg(delta_ptr + row + 1);
    const int np = __ldg(top + cl);  // the removed ones' counts are within the cluster's
    const uint32_t nw = (uint32_t)Nw;
    const uint32_t* pc = planes + (int64_t)cl * kSymPlanes * Nw;
    // P planes of the removed columns' counts: five for lists below 32 entries
    // (16 of two words each cost the registers that keep four blocks on an SM)
    auto apply = [&](auto count) {
      constexpr int P = decltype(count)::value;
      uint32_t pl[kSymPWords][P];
#pragma unroll
      for (int q = 0; q < kSymPWords; q++)
#pragma unroll
        for (int p = 0; p < P; p++) pl[q][p] = 0u;
      for (int d = d0; d < d1; d += 32) {
        const int n = min(32, d1 - d);
        const uint32_t mine = lane < n ? __ldg(delta_idx + d + lane) : 0u;
        for (int e = 0; e < n; e += 8) {
          uint32_t idx[8], v[kSymPWords][8];
#pragma unroll
          for (int s = 0; s < 8; s++) idx[s] = __shfl_sync(kFull, mine, e + s);
#pragma unroll
          for (int s = 0; s < 8; s++) {
            const uint64_t at = (uint64_t)(idx[s] & 0x7fffffffu) * nw;
            if (PAIR) {
              uint2 x = make_uint2(0u, 0u);
              if (e + s < n && wv[0]) x = __ldg(reinterpret_cast<const uint2*>(Bw + wq[0] + at));
              v[0][s] = x.x;
              v[1][s] = x.y;
            } else {
#pragma unroll
              for (int q = 0; q < kSymPWords; q++) v[q][s] = (e + s < n && wv[q]) ? __ldg(Bw + wq[q] + at) : 0u;
            }
          }
#pragma unroll
          for (int s = 0; s < 8; s++) {
            const uint32_t sub = (uint32_t)((int32_t)idx[s] >> 31);  // all ones: removed
#pragma unroll
            for (int q = 0; q < kSymPWords; q++) {
              out[q] |= v[q][s] & ~sub;
              v[q][s] &= sub;
            }
          }
#pragma unroll
          for (int q = 0; q < kSymPWords; q++) planes_add8(pl[q], v[q]);
        }
      }
      // count of the cluster > count of the removed, from the lowest plane up
      uint32_t more[kSymPWords];
#pragma unroll
      for (int q = 0; q < kSymPWords; q++) more[q] = 0u;
#pragma unroll
      for (int p = 0; p < P; p++) {
        if (p >= np) break;
#pragma unroll
        for (int q = 0; q < kSymPWords; q++) {
          const uint32_t n = wv[q] ? __ldg(pc + (int64_t)p * Nw + wq[q]) : 0u, r = ~pl[q][p];
          more[q] = (n & r) | (n & more[q]) | (r & more[q]);
        }
      }
#pragma unroll 1
      for (int p = P; p < np; p++)  // (the removed ones' counts have none there)
#pragma unroll
        for (int q = 0; q < kSymPWords; q++) more[q] |= wv[q] ? __ldg(pc + (int64_t)p * Nw + wq[q]) : 0u;
#pragma unroll
      for (int q = 0; q < kSymPWords; q++) out[q] |= more[q];
    };
    if (d1 - d0 < 32) apply(std::integral_constant<int, 5>());
    else apply(std::integral_constant<int, kSymPlanes>());
  }
#pragma unroll
  for (int q = 0; q < kSymPWords; q++)
    if (wv[q]) Cw[row * Nw + wq[q]] = out[q];
}

struct PlaneArgs {
  const uint32_t* planes;  // [nplanes][M][Kw]
  int64_t M, K, Kw;
  int nplanes, signed_top;
  const void* B;
  int64_t ldb, N;
  float* C;
  int64_t ldc;
};

__device__ __forceinline__ float plane_weight(int b, int nplanes, int signed_top) {
  const float w = (float)(1u << b);
  return (signed_top && b == nplanes - 1) ? -w : w;
}

// One warp per (row, column chunk of 32*VPL*COLS), 16-byte vectors of B.
template <typename BT, int VPL, int D>
__global__ void __launch_bounds__(256) k_bitplane_rows(PlaneArgs a) {
  using V = Vec<BT>;
  constexpr int COLS = V::COLS;
  constexpr int CW = 32 * VPL * COLS;
  const int lane = threadIdx.x & 31;
  const int64_t row = (int64_t)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
  if (row >= a.M) return;
  const int n0 = (int)blockIdx.y * CW;
  const BT* __restrict__ B = static_cast<const BT*>(a.B);
  int col[VPL];
  bool cvalid[VPL];
#pragma unroll
  for (int v = 0; v < VPL; v++) {
    col[v] = n0 + (v * 32 + lane) * COLS;
    cvalid[v] = col[v] < a.N;
  }
  Acc<VPL, COLS, false> tot;
  tot.zero();
  for (int b = 0; b < a.nplanes; b++) {
    BitWalker wk;
    wk.init(a.planes + ((int64_t)b * a.M + row) * a.Kw, 0, (int)a.Kw, lane);
    Acc<VPL, COLS, true> acc;
    acc.zero();
    accumulate_walk<V, VPL, D, true>(wk, B, a.ldb, col, cvalid, acc);
    const float w = plane_weight(b, a.nplanes, a.signed_top);
#pragma unroll
    for (int v = 0; v < VPL; v++)
#pragma unroll
      for (int j = 0; j < COLS; j++) tot.s[v][j] += w * acc.result(v, j);
  }
  store_vecs<VPL, COLS, false>(a.C + row * a.ldc, col, cvalid, tot, nullptr, true, a.N);
}

// Any layout: one warp per (row, 32 columns), a lane per column.
template <typename BT>
__global__ void __launch_bounds__(256) k_bitplane_rows_scalar(PlaneArgs a) {
  const int lane = threadIdx.x & 31;
  const int64_t row = (int64_t)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
  if (row >= a.M) return;
  const BT* __restrict__ B = static_cast<const BT*>(a.B);
  for (int64_t c0 = (int64_t)blockIdx.y * 32; c0 < a.N; c0 += (int64_t)gridDim.y * 32) {
    const int64_t c = c0 + lane;
    float tot = 0.f;
    for (int b = 0; b < a.nplanes; b++) {
      BitWalker wk;
      wk.init(a.planes + ((int64_t)b * a.M + row) * a.Kw, 0, (int)a.Kw, lane);
      float s = 0.f, e = 0.f;
      for (uint32_t k = wk.next(); k != kEnd; k = wk.next()) {
        const float x = c < a.N ? to_f32(B[(int64_t)k * a.ldb + c]) : 0.f;
        const float t = s + x, bp = t - s;
        e += (s - (t - bp)) + (x - bp);
        s = t;
      }
      tot += plane_weight(b, a.nplanes, a.signed_top) * (s + e);
    }
    if (c < a.N) a.C[row * a.ldc + c] = tot;
  }
}

template <typename BT>
int launch_planes_t(const PlaneArgs& a, bool vec, cudaStream_t s) {
  const unsigned gx = (unsigned)ceil_div(a.M, 8);
  if (!vec) {
    const int64_t gy = ceil_div(a.N, 32) < 65535 ? ceil_div(a.N, 32) : 65535;
    k_bitplane_rows_scalar<BT><<<dim3(gx, (unsigned)gy), 256, 0, s>>>(a);
  } else {
    constexpr int COLS = Vec<BT>::COLS;
    constexpr int VPL = COLS == 4 ? 2 : 1;
    const int64_t gy = ceil_div(a.N, 32 * VPL * COLS);
    if (gy > 65535) return BSP_ERR_CAPACITY;
    k_bitplane_rows<BT, VPL, 8><<<dim3(gx, (unsigned)gy), 256, 0, s>>>(a);
  }
  BSP_LAUNCHED();
  return BSP_OK;
}

// B stacked for the planes-along-K form: row b*Kp + k of out is w_b·B[k]
// (k < K) or 0 (K ≤ k < Kp, Kp = 32·ceil(K/32)).  A power-of-two factor
// only changes the exponent, so the 16-bit values stay exact.  A CTA per
// output row (grid-stride), its threads along the columns.
template <typename BT>
__global__ void __launch_bounds__(256) k_stack_planes_b(const BT* __restrict__ B, int64_t ldb, int64_t K,
                                                        int64_t Kp, int64_t N, int nplanes, int signed_top,
                                                        BT* __restrict__ out, int64_t ldo) {
  const int64_t rows = (int64_t)nplanes * Kp;
  for (int64_t rr = blockIdx.x; rr < rows; rr += gridDim.x) {
    const int b = (int)(rr / Kp);
    const int64_t k = rr - (int64_t)b * Kp;
    const float w = plane_weight(b, nplanes, signed_top);
    BT* o = out + rr * ldo;
    if (k < K) {
      const BT* src = B + k * ldb;
      for (int64_t c = threadIdx.x; c < N; c += blockDim.x) o[c] = from_f32<BT>(to_f32(src[c]) * w);
    } else {
      for (int64_t c = threadIdx.x; c < N; c += blockDim.x) o[c] = from_f32<BT>(0.f);
    }
  }
}

// int8 A [M][K] -> [ceil(K/32)][M][32], zeros past K: the order in which the
// tensor-core product's producers read it (a lane's 32 bytes of a tile next to
// its neighbour row's), and behind it one bit per 128 x 32 tile that holds a
// nonzero.  A block takes 128 rows x 1024 columns, a thread 4 columns of every
// row, 8 rows in flight; its 32 tiles' bits are one word.  Runs once per weight
// matrix.  Bound by memory; with the bits set one by one by atomics, many
// threads on a word, the preparation of 4096x4096 took 535 us, now 180 (175
// without this order).
template <bool VEC>
__global__ void __launch_bounds__(256) k_i8_tiles(const int8_t* __restrict__ A, int64_t M, int64_t K, int64_t lda,
                                                  uint32_t* __restrict__ tiles, uint32_t* __restrict__ occ,
                                                  int occ_words) {
  __shared__ uint32_t s_bits[8];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int64_t c = ((int64_t)blockIdx.x * 256 + threadIdx.x) * 4, t = c >> 5;  // (a tile: 8 neighbouring threads)
  for (int64_t rb = blockIdx.y; rb * 128 < M; rb += gridDim.y) {
    const int64_t r0 = rb * 128, r1 = min(M, r0 + 128);
    uint32_t any = 0u;
    for (int64_t r = r0; r < r1; r += 8) {
      uint32_t w[8];
#pragma unroll
      for (int i = 0; i < 8; i++) {
        w[i] = 0u;
        if (r + i >= r1) continue;
        if (VEC && c + 4 <= K) {
          w[i] = __ldg(reinterpret_cast<const uint32_t*>(A + (r + i) * lda + c));
        } else {
#pragma unroll
          for (int j = 0; j < 4; j++)
            if (c + j < K) w[i] |= (uint32_t)(uint8_t)A[(r + i) * lda + c + j] << (8 * j);
        }
      }
#pragma unroll
      for (int i = 0; i < 8; i++) {
        any |= w[i];
        if (r + i < r1 && t * 32 < K) tiles[(t * M + r + i) * 8 + (threadIdx.x & 7)] = w[i];
      }
    }
    const uint32_t b = __ballot_sync(kFull, any != 0u);  // 8 lanes a tile
    if (lane == 0)
      s_bits[warp] = ((b & 0xffu) ? 1u : 0u) | ((b & 0xff00u) ? 2u : 0u) | ((b & 0xff0000u) ? 4u : 0u) |
                     ((b & 0xff000000u) ? 8u : 0u);
    __syncthreads();
    if (threadIdx.x == 0) {
      uint32_t word = 0u;
#pragma unroll
      for (int w = 0; w < 8; w++) word |= s_bits[w] << (4 * w);
      occ[rb * occ_words + blockIdx.x] = word;
    }
    __syncthreads();
  }
}

}  // namespace

size_t i8_values_bytes(int64_t M, int64_t K) { return (size_t)M * (size_t)ceil_div(K, 32) * 32; }

size_t i8_tiles_bytes(int64_t M, int64_t K) {
  return i8_values_bytes(M, K) + (size_t)ceil_div(M, 128) * tc_occupancy_words(K) * sizeof(uint32_t);
}

int launch_i8_tiles(const int8_t* A, int64_t M, int64_t K, int64_t lda, int8_t* tiles, cudaStream_t s) {
  const int64_t rb = ceil_div(M, 128);
  const dim3 grid((unsigned)tc_occupancy_words(K), (unsigned)(rb < 65535 ? rb : 65535));
  uint32_t* occ = reinterpret_cast<uint32_t*>(tiles + i8_values_bytes(M, K));
  const bool vec = lda % 4 == 0 && reinterpret_cast<uintptr_t>(A) % 4 == 0;
  (vec ? k_i8_tiles<true> : k_i8_tiles<false>)<<<grid, 256, 0, s>>>(A, M, K, lda, (uint32_t*)tiles, occ,
                                                                    tc_occupancy_words(K));
  BSP_LAUNCHED();
  return BSP_OK;
}

int launch_stack_planes_b(const void* B, int bdt, int64_t ldb, int64_t K, int64_t N, int nplanes, int signed_top,
                          void* out, int64_t ldo, cudaStream_t s) {
  const int64_t Kp = ceil_div(K, 32) * 32;
  const int64_t total = (int64_t)nplanes * Kp * N;
  if (total == 0) return BSP_OK;
  const int64_t rows = (int64_t)nplanes * Kp, cap = (int64_t)num_sms() * 32;
  const unsigned grid = (unsigned)(rows < cap ? rows : cap);
  if (bdt == BSP_F32)
    k_stack_planes_b<float><<<grid, 256, 0, s>>>((const float*)B, ldb, K, Kp, N, nplanes, signed_top, (float*)out, ldo);
  else if (bdt == BSP_BF16)
    k_stack_planes_b<__nv_bfloat16><<<grid, 256, 0, s>>>((const __nv_bfloat16*)B, ldb, K, Kp, N, nplanes, signed_top,
                                                         (__nv_bfloat16*)out, ldo);
  else if (bdt == BSP_F16)
    k_stack_planes_b<__half><<<grid, 256, 0, s>>>((const __half*)B, ldb, K, Kp, N, nplanes, signed_top, (__half*)out,
                                                  ldo);
  else
    return BSP_ERR_UNSUPPORTED;
  BSP_LAUNCHED();
  return BSP_OK;
}

int launch_symbolic_rows(const uint32_t* A, int64_t M, int64_t K, const uint32_t* Bw, int64_t N, uint32_t* Cw,
                         cudaStream_t s) {
  const int64_t Kw = ceil_div(K, 32), Nw = ceil_div(N, 32);
  const int64_t gy = ceil_div(Nw, 32 * kSymWords);
  if (M == 0 || Nw == 0) return BSP_OK;
  if (gy > 65535) return BSP_ERR_CAPACITY;
  k_symbolic_rows<<<dim3((unsigned)ceil_div(M, 8), (unsigned)gy), 256, 0, s>>>(A, M, K, Kw, Bw, Nw, Cw);
  BSP_LAUNCHED();
  return BSP_OK;
}

size_t symbolic_planes_bytes(int64_t n_proto, int64_t N) {
  // planes, then one int per cluster: the number of planes in use
  const size_t pb = sizeof(uint32_t) * (size_t)n_proto * kSymPlanes * (size_t)ceil_div(N, 32);
  return ((pb + 255) & ~size_t(255)) + sizeof(int) * (size_t)n_proto;
}

int launch_symbolic_planned(const uint32_t* A, int64_t M, int64_t K, const uint32_t* Bw, int64_t N, uint32_t* Cw,
                            const int32_t* row_cluster, const int32_t* delta_ptr, const uint32_t* delta_idx,
                            const uint32_t* cons, int64_t n_proto, uint32_t* planes, cudaStream_t s) {
  const int64_t Kw = ceil_div(K, 32), Nw = ceil_div(N, 32);
  if (M == 0 || Nw == 0) return BSP_OK;
  const int64_t gpy = ceil_div(Nw, kSymCWords), gry = ceil_div(Nw, 32 * kSymPWords);
  if (gpy > 65535 || gry > 65535 || n_proto > INT32_MAX) return BSP_ERR_CAPACITY;
  const size_t pb = sizeof(uint32_t) * (size_t)n_proto * kSymPlanes * (size_t)Nw;
  int* top = reinterpret_cast<int*>(reinterpret_cast<uint8_t*>(planes) + ((pb + 255) & ~size_t(255)));
  if (n_proto > 0) {
    BSP_CUDA(cudaMemsetAsync(top, 0, sizeof(int) * (size_t)n_proto, s));
    k_sym_cluster_planes<<<dim3((unsigned)n_proto, (unsigned)gpy), kSymCWords * kSymCGroups, 0, s>>>(cons, Kw, K, Bw,
                                                                                                    Nw, planes, top);
  }
  // a lane's two words side by side where every row starts on 8 bytes
  const bool pair = Nw % 2 == 0 && is_aligned(Bw, 8);
  auto rows = pair ? k_sym_rows_planned<true> : k_sym_rows_planned<false>;
  rows<<<dim3((unsigned)ceil_div(M, kSymRows), (unsigned)gry), kSymRows * 32, 0, s>>>(
      A, M, K, Kw, Bw, Nw, row_cluster, delta_ptr, delta_idx, planes, top, Cw);
  BSP_LAUNCHED();
  return BSP_OK;
}

int launch_bitplane_spmm(const uint32_t* planes, int nplanes, int signed_top, int64_t M, int64_t K,
                         const void* B, int bdt, int64_t ldb, int64_t N, float* C, int64_t ldc, bool vec,
                         cudaStream_t s) {
  if (M == 0 || N == 0) return BSP_OK;
  PlaneArgs a = {planes, M, K, ceil_div(K, 32), nplanes, signed_top, B, ldb, N, C, ldc};
  if (bdt == BSP_F32) return launch_planes_t<float>(a, vec, s);
  if (bdt == BSP_BF16) return launch_planes_t<__nv_bfloat16>(a, vec, s);
  if (bdt == BSP_F16) return launch_planes_t<__half>(a, vec, s);
  return BSP_ERR_UNSUPPORTED;
}

}  // namespace bsp
