// spmm.cu — CUDA-core bitmap SpMM kernels: C[M×N] = A·B, A packed LSB-first.
//
// "Multiply by one replaced by adds": row i of C is the sum of the rows k of
// B at A's set bits (reference backup/layout_trans.cu:158-171 did one global
// atomicAdd per set bit and column).  Here one warp owns a row and a chunk of
// columns, walks the row's set bits with __ffs in ascending column order,
// gathers D rows of B at a time with 16-byte vector loads (D gathers in
// flight per warp) and accumulates in FP32 registers in walk order.  Rows
// with more than 4096 set bits use a compensated two-term (TwoSum)
// accumulator.  Every output element is written once, without atomics, so
// results are deterministic run to run.
//
// Prototype mode (plans from plan.cu): a row i in cluster c is
//   C[i] = P[c] + Σ_{k ∈ A_i \ cons_c} B[k] − Σ_{k ∈ cons_c \ A_i} B[k],
// where P[c] = Σ_{k ∈ cons_c} B[k] is computed once per cluster by
// k_proto_sums (K split across the warps of a CTA, fixed-order reduction).
#include <cooperative_groups.h>

#include <type_traits>

#include "ptx.cuh"
#include "spmm_dev.cuh"

namespace cg = cooperative_groups;

namespace bsp {
namespace {

// A product that stands by for another one and is not asked for (whole block).
__device__ __forceinline__ bool stands_by(const SpmmArgs& a) {
  if (!a.run_if) return false;
  if (a.run_if_late) ptx::griddep_wait();
  if (a.run_if_n <= 1) return !__ldcg(a.run_if);
  int any = 0;
  for (int i = threadIdx.x; i < a.run_if_n; i += blockDim.x) any |= __ldcg(a.run_if + i);
  return !__syncthreads_or(any);
}

// Walking kernel: one warp per (row, column chunk of 32*VPL*COLS).  The warp
// first writes the columns of its row's set bits to a list in shared memory,
// 128 words at a time (a prefix sum of the lanes' bit counts gives every lane
// its place), and then gathers D rows of B per round, their indices read four
// to a shared load; sums run over the list in order, so a row is added in
// ascending column order whatever the shape.
//
// Bound by the L2 gather rate where there are enough warps, by the latency of
// a row's rounds of D gathers where there are few.  A walker that took one
// bit at a time from the words (find first set, shuffle, branch) between the
// gathers spent about twenty dependent instructions per bit and cut every
// round at a word: 1024x1024x256 FP32 at 10 %, 22.4 us against 9.7 now;
// 2048x2048x1024, 155 us against 85 (20 TB/s of gathers).  Rows with more than
// kCompThreshold set bits, where there can be any, are summed with TwoSum one
// vector at a time.
constexpr int kListStep = 128;                 // entries wanted before a round of gathers
constexpr int kListCap = kListStep + 32 * 32;  // one more group of 32 words

//
// FAST: no row has more than kCompThreshold set bits (K, or the plan, says so)
// and B's element offsets fit in 32 bits; without the TwoSum walk and the 64-bit
// row addresses, and with 4 gathers in flight, four blocks (MINB) run on an SM
// instead of two.
//
// LOOP: a walk that stands by; blocks for a few rounds go through all rows, so that
// the usual case, in which it is not asked for, does not start one for every
// eight rows (4096x4096x2048 BF16, single elements: 8192 blocks that end at once
// 22 us, now 4).
template <typename V, int VPL, int D, bool FAST, int MINB, bool LOOP>
__global__ void __launch_bounds__(256, MINB) k_spmm_list(SpmmArgs a) {
  using BT = typename V::T;
  using Off = typename std::conditional<FAST, uint32_t, int64_t>::type;
  constexpr int COLS = V::COLS;
  constexpr int CW = 32 * VPL * COLS;
  constexpr int GROUPS = 4;  // word groups (of 32) loaded at a time
  static_assert(kListStep % D == 0 && D % 4 == 0 && D <= 32, "whole rounds");
  __shared__ __align__(16) uint32_t lists[8][kListCap];
  const int lane = threadIdx.x & 31;
  uint32_t* list = lists[threadIdx.x >> 5];
  if (stands_by(a)) return;
  const int64_t rows = a.row_list ? a.n_list : a.M;
  int64_t at = (int64_t)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
  if (at >= rows) return;
  do {
    const int64_t row = a.row_list ? (int64_t)__ldg(a.row_list + at) : at;
    const BT* __restrict__ B = static_cast<const BT*>(a.B);
    const uint32_t* arow = a.A + row * a.Kw;
    const int Kw = (int)a.Kw;
    const bool comp = !FAST && a.K > kCompThreshold && row_popcount(arow, Kw, lane) > kCompThreshold;
    const Off ldb = (Off)a.ldb;
    for (int64_t n0 = (int64_t)blockIdx.y * CW; n0 < a.N; n0 += (int64_t)gridDim.y * CW) {
      int col[VPL];
      bool cvalid[VPL];
#pragma unroll
      for (int v = 0; v < VPL; v++) {
        const int64_t c = n0 + (v * 32 + lane) * COLS;
        cvalid[v] = c < a.Nb;
        col[v] = cvalid[v] ? (int)c : 0;
      }
      float* crow = a.C + row * a.ldc;
      if (!FAST && comp) {
        for (int v = 0; v < VPL; v++) {
          BitWalker wk;
          wk.init(arow, 0, Kw, lane);
          Acc<1, COLS, true> acc;
          acc.zero();
          int c1[1] = {col[v]};
          bool ok[1] = {cvalid[v]};
          accumulate_walk<V, 1, 4, true>(wk, B, a.ldb, c1, ok, acc);
          store_vecs<1, COLS, true>(crow, c1, ok, acc, nullptr, a.c_vec, a.N);
        }
        continue;
      }
      Acc<VPL, COLS, false> acc;
      acc.zero();
      auto gather = [&](int i, int n) {  // list entries [i, i + n), n <= D (uniform)
        uint32_t idx[D];
#pragma unroll
        for (int s = 0; s < D; s += 4) {
          const uint4 q = *reinterpret_cast<const uint4*>(list + i + s);
          idx[s] = q.x;
          idx[s + 1] = q.y;
          idx[s + 2] = q.z;
          idx[s + 3] = q.w;
        }
        typename V::Raw raw[D][VPL];
#pragma unroll
        for (int s = 0; s < D; s++) {
          const BT* brow = B + (Off)idx[s] * ldb;
#pragma unroll
          for (int v = 0; v < VPL; v++)
            if (s < n && cvalid[v]) raw[s][v] = V::load(brow + col[v]);
        }
#pragma unroll
        for (int s = 0; s < D; s++) {
          if (s >= n) break;
#pragma unroll
          for (int v = 0; v < VPL; v++) {
            if (!cvalid[v]) continue;
            float f[COLS];
            V::cvt(raw[s][v], f);
#pragma unroll
            for (int j = 0; j < COLS; j++) acc.add(v, j, f[j]);
          }
        }
      };
      uint32_t wx[GROUPS];
#pragma unroll
      for (int g = 0; g < GROUPS; g++) wx[g] = g * 32 + lane < Kw ? __ldg(arow + g * 32 + lane) : 0u;
      int n = 0;  // entries in the list
      for (int w0 = 0; w0 < Kw; w0 += GROUPS * 32) {
        uint32_t wn[GROUPS];
#pragma unroll
        for (int g = 0; g < GROUPS; g++) {
          const int w = w0 + (GROUPS + g) * 32 + lane;
          wn[g] = w < Kw ? __ldg(arow + w) : 0u;
        }
#pragma unroll
        for (int g = 0; g < GROUPS; g++) {
          if (w0 + g * 32 >= Kw) break;
          uint32_t x = wx[g];
          const int c = __popc(x);
          int incl = c;
#pragma unroll
          for (int o = 1; o < 32; o <<= 1) {
            const int y = __shfl_up_sync(kFull, incl, o);
            if (lane >= o) incl += y;
          }
          int pos = n + incl - c;
          const uint32_t k0 = (uint32_t)(w0 + g * 32 + lane) * 32u;
          while (x) {
            list[pos++] = k0 + (uint32_t)(__ffs(x) - 1);
            x &= x - 1;
          }
          n += __shfl_sync(kFull, incl, 31);
          const bool last = w0 + (g + 1) * 32 >= Kw;
          if (n < kListStep && !last) continue;
          __syncwarp();
          int i = 0;
          for (; i + D <= n; i += D) gather(i, D);
          n -= i;
          if (last) {
            if (n > 0) gather(i, n);
          } else if (i > 0) {  // the rest (less than D entries) starts the next round
            const uint32_t rest = lane < n ? list[i + lane] : 0u;
            __syncwarp();
            if (lane < n) list[lane] = rest;
          }
          __syncwarp();
        }
#pragma unroll
        for (int g = 0; g < GROUPS; g++) wx[g] = wn[g];
      }
      store_vecs<VPL, COLS, false>(crow, col, cvalid, acc, nullptr, a.c_vec, a.N);
      __syncwarp();
    }
    at += (int64_t)gridDim.x * (blockDim.x >> 5);
  } while (LOOP && at < rows);
}

// A few long rows: a CTA per (row, column chunk).  Its 8 warps write the row's
// column list (8192 columns at a time), gather 16 rows of B each into shared
// memory, and then every thread adds its own column over the 128 staged rows
// in list order — the sum the walking kernel forms.  One row of 427 bits cost
// the walking kernel a chain of gathers of 115 us behind the clustered 8192x8192x512
// product, more than the product; here it has 4 rounds and adds 3 us.
constexpr int kCoopSlots = 16;                  // rows in flight per warp
constexpr int kCoopBatch = 8 * kCoopSlots;
constexpr int kCoopWords = 256;                 // words listed at a time, one per thread

template <typename V, int VPL>
struct CoopSmem {
  static constexpr int CW = 32 * VPL * V::COLS;
  typename V::Raw stage[kCoopBatch][VPL][32];
  uint16_t list[kCoopWords * 32];
  int scan[32];
};

template <typename V, int VPL>
__global__ void __launch_bounds__(256) k_spmm_coop(SpmmArgs a) {
  using BT = typename V::T;
  using Smem = CoopSmem<V, VPL>;
  constexpr int COLS = V::COLS, CW = Smem::CW;
  static_assert(CW <= 256, "one thread per column");
  extern __shared__ __align__(16) uint8_t coop_raw[];
  Smem& sm = *reinterpret_cast<Smem*>(coop_raw);
  ptx::griddep_launch_dependents();
  if (stands_by(a)) return;  // (never with a row list)
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int64_t row = a.row_list ? (int64_t)__ldg(a.row_list + blockIdx.x) : (int64_t)blockIdx.x;
  const BT* __restrict__ B = static_cast<const BT*>(a.B);
  const uint32_t* arow = a.A + row * a.Kw;
  const int Kw = (int)a.Kw;
  const int64_t n0 = (int64_t)blockIdx.y * CW;
  const BT* bcol[VPL];
  bool cvalid[VPL];
#pragma unroll
  for (int v = 0; v < VPL; v++) {
    const int64_t c = n0 + (v * 32 + lane) * COLS;
    cvalid[v] = c < a.Nb;
    bcol[v] = B + (cvalid[v] ? c : 0);
  }
  bool comp = false;
  if (a.K > kCompThreshold) {
    int c = 0;
    for (int w = tid; w < Kw; w += 256) c += __popc(__ldg(arow + w));
    int total;
    block_exclusive_scan(c, sm.scan, &total);
    comp = total > kCompThreshold;
  }
  float s = 0.f, e = 0.f;
  const BT* mine = reinterpret_cast<const BT*>(&sm.stage[0][0][0]) + tid;  // column tid of slot 0
  for (int w0 = 0; w0 < Kw; w0 += kCoopWords) {
    uint32_t x = w0 + tid < Kw ? __ldg(arow + w0 + tid) : 0u;
    int total;
    int pos = block_exclusive_scan(__popc(x), sm.scan, &total);
    while (x) {
      sm.list[pos++] = (uint16_t)(tid * 32 + __ffs(x) - 1);
      x &= x - 1;
    }
    __syncthreads();
    typename V::Raw raw[kCoopSlots][VPL];
    auto load = [&](int b0) {
#pragma unroll
      for (int u = 0; u < kCoopSlots; u++) {
        const int i = b0 + warp * kCoopSlots + u;
        if (i >= total) break;
        const int64_t k = (int64_t)w0 * 32 + sm.list[i];
#pragma unroll
        for (int v = 0; v < VPL; v++)
          if (cvalid[v]) raw[u][v] = V::load(bcol[v] + k * a.ldb);
      }
    };
    load(0);
    for (int b0 = 0; b0 < total; b0 += kCoopBatch) {
      const int cnt = min(kCoopBatch, total - b0);
#pragma unroll
      for (int u = 0; u < kCoopSlots; u++)
#pragma unroll
        for (int v = 0; v < VPL; v++) sm.stage[warp * kCoopSlots + u][v][lane] = raw[u][v];
      __syncthreads();
      load(b0 + kCoopBatch);
      if (tid < CW) {
        if (comp) {
          for (int i = 0; i < cnt; i++) {
            const float f = to_f32(mine[i * CW]);
            const float t = s + f, bp = t - s;
            e += (s - (t - bp)) + (f - bp);
            s = t;
          }
        } else {
#pragma unroll 8
          for (int i = 0; i < cnt; i++) s += to_f32(mine[i * CW]);
        }
      }
      __syncthreads();
    }
  }
  if (tid < CW && n0 + tid < a.N) a.C[row * a.ldc + n0 + tid] = comp ? s + e : s;
  ptx::griddep_wait();  // this grid ends after the one it may overlap
}

// Plans of A with 2^30 or more columns: one warp per (row, column chunk).
// Rows with a cluster walk their delta list and add P[c]; every other row
// walks A's words.
template <typename BT, int VPL, int D>
__global__ void __launch_bounds__(256) k_spmm_rows_wide(SpmmArgs a) {
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
  float* crow = a.C + row * a.ldc;
  const int cl = __ldg(a.row_cluster + row);
  if (cl >= 0) {
    ListWalker wk;
    wk.init(a.delta_idx, __ldg(a.delta_ptr + row), __ldg(a.delta_ptr + row + 1), lane);
    Acc<VPL, COLS, false> acc;
    acc.zero();
    accumulate_walk<V, VPL, D, false>(wk, B, a.ldb, col, cvalid, acc);
    store_vecs<VPL, COLS, false>(crow, col, cvalid, acc, a.P + (int64_t)cl * a.ldp, a.c_vec, a.N);
    return;
  }
  const uint32_t* arow = a.A + row * a.Kw;
  const bool comp = row_popcount(arow, (int)a.Kw, lane) > kCompThreshold;
  for (int v = 0; v < VPL; v++) {
    BitWalker wk;
    wk.init(arow, 0, (int)a.Kw, lane);
    int c1[1] = {col[v]};
    bool ok[1] = {cvalid[v]};
    if (comp) {
      Acc<1, COLS, true> acc;
      acc.zero();
      accumulate_walk<V, 1, 4, true>(wk, B, a.ldb, c1, ok, acc);
      store_vecs<1, COLS, true>(crow, c1, ok, acc, nullptr, a.c_vec, a.N);
    } else {
      Acc<1, COLS, false> acc;
      acc.zero();
      accumulate_walk<V, 1, 4, false>(wk, B, a.ldb, c1, ok, acc);
      store_vecs<1, COLS, false>(crow, c1, ok, acc, nullptr, a.c_vec, a.N);
    }
  }
}

// Prototype rows, register path: one warp per (clustered row, column chunk).
// The delta gathers are issued first; P[c] is read after griddep_wait(), so
// with programmatic dependent launch the whole gather phase overlaps the
// prototype-sum kernel.  MINB caps registers (occupancy sweep).  OFF32 = B's
// element offsets fit in 32 bits (K·ldb < 2^31) and FULL = every column
// chunk is whole (N a multiple of the chunk width); with 32-bit row
// arithmetic (M < 2^31, checked on the host) they keep the 8-blocks-per-SM
// shape within its 32 registers without spilling (a 12-byte spill cost the
// clustered 8192²×512 step 3 µs).
template <typename V, int VPL, int D, int MINB, bool OFF32, bool FULL, bool SLOT>
__global__ void __launch_bounds__(256, MINB) k_spmm_proto_regs(SpmmArgs a) {
  using BT = typename V::T;
  constexpr int COLS = V::COLS;
  constexpr int CW = 32 * VPL * COLS;
  const int lane = threadIdx.x & 31;
  ptx::griddep_launch_dependents();  // the direct rows' kernel, if there is one
  int row, cl;
  uint32_t slot = 0u;
  if (SLOT) {
    // warp p takes the p-th row slot (rows by descending delta count): row,
    // cluster and list in one load whose address depends on p alone
    const int p = (int)blockIdx.x * 8 + (threadIdx.x >> 5);
    if (p < (int)a.n_slot) slot = __ldg(a.delta_pad + (int64_t)p * 32 + lane);
    row = (int)__shfl_sync(kFull, slot, 0);
    cl = p < (int)a.n_slot ? (int)__shfl_sync(kFull, slot, 1) : -1;
  } else {
    row = (int)blockIdx.x * 8 + (threadIdx.x >> 5);
    cl = row < (int)a.M ? __ldg(a.row_cluster + row) : -1;
  }
  if (cl >= 0) {
    const int n0 = (int)blockIdx.y * CW;
    const BT* __restrict__ B = static_cast<const BT*>(a.B);
    int col[VPL];
    bool cvalid[VPL];
#pragma unroll
    for (int v = 0; v < VPL; v++) {
      col[v] = n0 + (v * 32 + lane) * COLS;
      cvalid[v] = FULL || col[v] < (int)a.Nb;
    }
    Acc<VPL, COLS, false> acc;
    acc.zero();
    if (SLOT) {
      SlotWalker wk;
      wk.init(slot, a.delta_idx, lane);
      if (OFF32) accumulate_walk<V, VPL, D, false>(wk, B, (uint32_t)a.ldb, col, cvalid, acc);
      else accumulate_walk<V, VPL, D, false>(wk, B, a.ldb, col, cvalid, acc);
    } else {
      ListWalker wk;
      wk.init(a.delta_idx, __ldg(a.delta_ptr + row), __ldg(a.delta_ptr + row + 1), lane);
      if (OFF32) accumulate_walk<V, VPL, D, false>(wk, B, (uint32_t)a.ldb, col, cvalid, acc);
      else accumulate_walk<V, VPL, D, false>(wk, B, a.ldb, col, cvalid, acc);
    }
    ptx::griddep_wait();
    store_vecs<VPL, COLS, false>(a.C + (int64_t)row * a.ldc, col, cvalid, acc, a.P + (int64_t)cl * a.ldp, a.c_vec, a.N);
  } else {
    ptx::griddep_wait();
  }
}

// P[c][n0 .. n0+32*COLS) for one prototype per CTA row: warp w walks the
// prototype's words [w*Kw/W, (w+1)*Kw/W), partial sums meet in shared memory
// and are added in warp order.  COMP (the densest prototype has more than
// 4096 set bits): each warp keeps a TwoSum pair (sum, error) and the pairs
// are added with TwoSum too; P = sum + error.
template <typename V, int D, bool COMP, bool OFF32>
__global__ void __launch_bounds__(512) k_proto_sums(SpmmArgs a) {
  using BT = typename V::T;
  constexpr int COLS = V::COLS;
  constexpr int CW = 32 * COLS;
  extern __shared__ float part[];  // [W][CW] sums, then (COMP) [W][CW] errors
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5, W = blockDim.x >> 5;
  const int64_t c = blockIdx.x;
  const int64_t n0 = (int64_t)blockIdx.y * CW;
  const BT* __restrict__ B = static_cast<const BT*>(a.B);
  int col[1] = {(int)n0 + lane * COLS};
  bool cvalid[1] = {col[0] < a.Nb};
  ptx::griddep_launch_dependents();
  const uint32_t* cw = a.cons + c * a.Kw;
  const int w0 = (int)(a.Kw * wid / W), w1 = (int)(a.Kw * (wid + 1) / W);
  BitWalker wk;
  wk.init(cw, w0, w1, lane);
  Acc<1, COLS, COMP> acc;
  acc.zero();
  if (OFF32) accumulate_walk<V, 1, D, COMP>(wk, B, (uint32_t)a.ldb, col, cvalid, acc);
  else accumulate_walk<V, 1, D, COMP>(wk, B, a.ldb, col, cvalid, acc);
#pragma unroll
  for (int j = 0; j < COLS; j++) {
    part[wid * CW + lane * COLS + j] = acc.s[0][j];
    if (COMP) part[(W + wid) * CW + lane * COLS + j] = acc.c[0][COMP ? j : 0];
  }
  __syncthreads();
  for (int j = threadIdx.x; j < CW; j += blockDim.x) {
    float s = 0.f, e = 0.f;
    for (int w = 0; w < W; w++) {
      const float x = part[w * CW + j];
      if (COMP) {
        const float t = s + x, bp = t - s;
        e += ((s - (t - bp)) + (x - bp)) + part[(W + w) * CW + j];
        s = t;
      } else {
        s += x;
      }
    }
    if (n0 + j < a.N) a.P[c * a.ldp + n0 + j] = COMP ? s + e : s;
  }
}

// P[c] over one chunk of CW = 32·VPL·COLS columns from the prototype's
// column list, by a cluster of 8 CTAs × 8 warps: warp p = rank·8 + w sums
// list entries [len·p/64, len·(p+1)/64) with one B slice in flight.  With 64
// short chains instead of 16 long ones the sums finish sooner (each gather
// waits out the L2 latency of a loaded GPU), and 256-thread CTAs at 32
// registers leave the SMs to the row kernel that runs beside them under
// programmatic dependent launch.  Each CTA adds its warps' partials in warp
// order; rank 0 adds the 8 CTA partials in rank order through distributed
// shared memory (all loads issued first), so P is the same on every run.
constexpr int kSumCluster = 8;
template <typename V, int VPL, bool OFF32>
__global__ void __cluster_dims__(kSumCluster, 1, 1) __launch_bounds__(256) k_proto_sums_list(SpmmArgs a) {
  using BT = typename V::T;
  constexpr int COLS = V::COLS;
  constexpr int CW = 32 * VPL * COLS;
  constexpr int PARTS = kSumCluster * 8;
  __shared__ float4 wp[8][CW / 4];
  __shared__ float4 cp[CW / 4];
  cg::cluster_group cluster = cg::this_cluster();
  const int rank = (int)cluster.block_rank();
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  const int n0 = (int)(blockIdx.x / kSumCluster) * CW;
  const int64_t c = blockIdx.y;
  ptx::griddep_launch_dependents();
  int col[VPL];
  bool cvalid[VPL];
#pragma unroll
  for (int v = 0; v < VPL; v++) {
    col[v] = n0 + (v * 32 + lane) * COLS;
    cvalid[v] = col[v] < (int)a.Nb;
  }
  const int s0 = __ldg(a.cons_ptr + c), len = __ldg(a.cons_ptr + c + 1) - s0;
  const int p = rank * 8 + wid;
  ListWalker wk;
  wk.init(a.cons_idx, s0 + (int)((int64_t)len * p / PARTS), s0 + (int)((int64_t)len * (p + 1) / PARTS), lane);
  Acc<VPL, COLS, false> acc;
  acc.zero();
  const BT* __restrict__ B = static_cast<const BT*>(a.B);
  if (OFF32) accumulate_walk<V, VPL, 1, false>(wk, B, (uint32_t)a.ldb, col, cvalid, acc);
  else accumulate_walk<V, VPL, 1, false>(wk, B, a.ldb, col, cvalid, acc);
  float* w = reinterpret_cast<float*>(&wp[wid][0]);
#pragma unroll
  for (int v = 0; v < VPL; v++)
#pragma unroll
    for (int j = 0; j < COLS; j++) w[(v * 32 + lane) * COLS + j] = acc.result(v, j);
  __syncthreads();
  if (threadIdx.x < CW / 4) {
    float4 t = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
    for (int u = 0; u < 8; u++) {
      const float4 x = wp[u][threadIdx.x];
      t.x += x.x;
      t.y += x.y;
      t.z += x.z;
      t.w += x.w;
    }
    cp[threadIdx.x] = t;
  }
  cluster.sync();
  if (rank == 0 && threadIdx.x < CW / 4) {
    float4 x[kSumCluster];
#pragma unroll
    for (int r = 0; r < kSumCluster; r++) x[r] = cluster.map_shared_rank(cp, r)[threadIdx.x];
    float4 t = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
    for (int r = 0; r < kSumCluster; r++) {
      t.x += x[r].x;
      t.y += x[r].y;
      t.z += x[r].z;
      t.w += x[r].w;
    }
    // P rows are ldp = ceil8(N) floats: a float4 starting below N stays in the row
    if (n0 + 4 * (int)threadIdx.x < (int)a.N) reinterpret_cast<float4*>(a.P + c * a.ldp + n0)[threadIdx.x] = t;
  }
  cluster.sync();
}

bool list_fast(const SpmmArgs& a) {
  return (a.K <= kCompThreshold || a.no_long_rows) && a.K * a.ldb < ((int64_t)1 << 31);
}

template <typename V, int VPL, int D, bool FAST = false, int MINB = 0>
int launch_list_s(const SpmmArgs& a, int64_t rows, cudaStream_t s) {
  const int64_t gy = ceil_div(a.N, 32 * VPL * V::COLS);
  k_spmm_list<V, VPL, D, FAST, MINB, false>
      <<<dim3((unsigned)ceil_div(rows, 8), (unsigned)(gy < 65535 ? gy : 65535)), 256, 0, s>>>(a);
  BSP_LAUNCHED();
  return BSP_OK;
}

// ... of a walk that stands by: 4 blocks an SM at most.
template <typename V, int VPL, int D, bool FAST, int MINB>
int launch_standby_s(const SpmmArgs& a, int64_t rows, cudaStream_t s) {
  const int64_t most = (int64_t)num_sms() * 4;
  int64_t gy = ceil_div(a.N, 32 * VPL * V::COLS), gx = ceil_div(rows, 8);
  if (gy > most) gy = most;
  if (gx * gy > most) gx = most / gy > 0 ? most / gy : 1;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)gx, (unsigned)gy);
  cfg.blockDim = dim3(256);
  cfg.stream = s;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = a.run_if_late ? 1 : 0;
  BSP_CUDA(cudaLaunchKernelEx(&cfg, k_spmm_list<V, VPL, D, FAST, MINB, true>, a));
  return BSP_OK;
}

template <typename V, int VPL>
int launch_coop_s(const SpmmArgs& a, int64_t rows, cudaStream_t s) {
  constexpr int smem = (int)sizeof(CoopSmem<V, VPL>);
  auto kern = k_spmm_coop<V, VPL>;
  static bool configured[64] = {};
  int dev = 0;
  BSP_CUDA(cudaGetDevice(&dev));
  if (dev >= 64 || !configured[dev]) {
    BSP_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
    if (dev < 64) configured[dev] = true;
  }
  // A programmatic dependent of the prototype rows' kernel: it reads only A
  // and B and writes its own rows of C, so it may run beside that kernel's
  // last CTAs (alone in its stream the attribute changes nothing).
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)rows, (unsigned)ceil_div(a.N, CoopSmem<V, VPL>::CW));
  cfg.blockDim = dim3(256);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = s;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = a.row_list || a.run_if_late ? 1 : 0;
  BSP_CUDA(cudaLaunchKernelEx(&cfg, kern, a));
  return BSP_OK;
}

template <typename V>
int launch_rows_t(const SpmmArgs& a, cudaStream_t s) {
  constexpr int VPL = V::COLS == 1 ? 4 : 1;
  const int64_t rows = a.row_list ? a.n_list : a.M;
  if (rows == 0) return BSP_OK;
  const int64_t sms = num_sms(), chunks = ceil_div(a.N, 32 * VPL * V::COLS), tasks = rows * chunks;
  // One (row, chunk) per SM at most: a chain of gathers per row would be all
  // that runs (one row, 8192 columns at 5 %, N = 512: 9.1 us against 15.2;
  // from a few hundred tasks on the two are equal, 117 rows 21.5 and 20.0).
  if (tasks <= sms && a.K >= 1024 && chunks <= 65535) return launch_coop_s<V, VPL>(a, rows, s);
  if (a.run_if) {
    if constexpr (V::COLS != 1) {  // (as below)
      if (tasks >= 32 * sms && list_fast(a)) return launch_standby_s<V, VPL, 4, true, 4>(a, rows, s);
    }
    return launch_standby_s<V, VPL, 8, false, 0>(a, rows, s);
  }
  if constexpr (V::COLS == 1) {
    // No more columns a lane than there are: 100000x32x8 FP32 170 us with four a
    // lane, 29 with one; 4096x4096x12 BF16 at 5 % 107 and 23.
    if (a.N <= 32) return list_fast(a) ? launch_list_s<V, 1, 4, true, 6>(a, rows, s) : launch_list_s<V, 1, 8>(a, rows, s);
    if (a.N <= 64) return list_fast(a) ? launch_list_s<V, 2, 8, true>(a, rows, s) : launch_list_s<V, 2, 8>(a, rows, s);
    return launch_list_s<V, VPL, 8>(a, rows, s);
  } else {
    // Many more warps than run at once: 4 gathers in flight each, four blocks an SM
    // (2048x2048x1024 FP32 at 10 % 86 us, 8 in flight and two blocks 99;
    // 4096x4096x512 BF16 at 5 % 67 and 76; 4000x400x2000 FP32 at 10 % 85 and 107),
    // of FP32 two vectors a lane where they are nearly filled (one vector, two, 8 in
    // flight: 4000x100x2000 at 10 % 45, 37, 56; 4096x4096x256 at 0.1 % 10.5, 8.4,
    // 11.6; 2048x2048x1024 86, 85, 99; but 2000x3001x336 36, 38, 37).
    // Not for FP16, whose conversions take the place (4096x4096x512 at 5 % 81 and 77).
    if (!std::is_same<typename V::T, __half>::value && tasks >= 32 * sms && list_fast(a)) {
      if (V::COLS == 4 && ceil_div(a.N, 256) * 256 * 10 <= a.N * 11) return launch_list_s<V, 2, 4, true>(a, rows, s);
      return launch_list_s<V, 1, 4, true, 4>(a, rows, s);
    }
    // With 12 or more warps an SM, 8 gathers in flight each (1024x1024x256: 9.7 us,
    // 16 in flight 11.2, 4 11.7; 2048x2048x1024: 96 and 123); with fewer, 16
    // (300x4000x512 at 2 %: 6.7 us, 8 in flight 7.7; 512x512x64: 4.3 and 5.2).
    if (tasks >= 12 * sms) return launch_list_s<V, VPL, 8>(a, rows, s);
    return launch_list_s<V, VPL, 16>(a, rows, s);
  }
}

template <typename BT>
int launch_rows_wide_t(const SpmmArgs& a, cudaStream_t s) {
  const dim3 g((unsigned)ceil_div(a.M, 8), (unsigned)ceil_div(a.N, 32 * Vec<BT>::COLS));
  k_spmm_rows_wide<BT, 1, 8><<<g, 256, 0, s>>>(a);
  BSP_LAUNCHED();
  return BSP_OK;
}

// BSP_SLOT_LISTS=0: rows in index order, each list read through its bounds
// (for comparisons).
bool slot_lists_enabled() {
  static const bool on = [] {
    const char* e = getenv("BSP_SLOT_LISTS");
    return !(e && e[0] == '0');
  }();
  return on;
}

template <typename V, int VPL, int D, int MINB>
int launch_proto_regs_t(const SpmmArgs& a, cudaStream_t s) {
  constexpr int CW = 32 * VPL * V::COLS;
  cudaLaunchConfig_t cfg = {};
  const bool off32 = a.K * a.ldb < ((int64_t)1 << 31), full = a.Nb % CW == 0;
  const bool slot = off32 && a.delta_pad && a.n_slot > 0 && slot_lists_enabled();
  cfg.gridDim = dim3((unsigned)ceil_div(slot ? a.n_slot : a.M, 8), (unsigned)ceil_div(a.N, CW));
  cfg.blockDim = dim3(256);
  cfg.dynamicSmemBytes = 0;
  cfg.stream = s;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  if (slot && full)
    BSP_CUDA(cudaLaunchKernelEx(&cfg, k_spmm_proto_regs<V, VPL, D, MINB, true, true, true>, a));
  else if (slot)
    BSP_CUDA(cudaLaunchKernelEx(&cfg, k_spmm_proto_regs<V, VPL, D, MINB, true, false, true>, a));
  else if (off32 && full)
    BSP_CUDA(cudaLaunchKernelEx(&cfg, k_spmm_proto_regs<V, VPL, D, MINB, true, true, false>, a));
  else if (off32)
    BSP_CUDA(cudaLaunchKernelEx(&cfg, k_spmm_proto_regs<V, VPL, D, MINB, true, false, false>, a));
  else
    BSP_CUDA(cudaLaunchKernelEx(&cfg, k_spmm_proto_regs<V, VPL, D, MINB, false, false, false>, a));
  return BSP_OK;
}

template <typename BT>
int launch_proto_regs_v(const SpmmArgs& a, int variant, bool vec, cudaStream_t s) {
  if (!vec) return launch_proto_regs_t<Elem1<BT>, 4, 4, 4>(a, s);
  constexpr bool F32 = Vec<BT>::COLS == 4;
  // variants: columns per warp (VPL vectors per lane), gathers in flight (D), min blocks/SM
  if (a.N <= 32 * Vec<BT>::COLS) return launch_proto_regs_t<Vec<BT>, 1, 16, 3>(a, s);
  switch (variant) {
    case 1: return launch_proto_regs_t<Vec<BT>, 2, 4, 4>(a, s);
    case 2: return launch_proto_regs_t<Vec<BT>, (F32 ? 4 : 2), 1, 5>(a, s);
    case 3: return launch_proto_regs_t<Vec<BT>, 2, 2, 6>(a, s);
    case 4: return launch_proto_regs_t<Vec<BT>, 2, 1, 8>(a, s);
    case 5: return launch_proto_regs_t<Vec<BT>, 1, 4, 8>(a, s);
    case 6: return launch_proto_regs_t<Vec<BT>, 2, 2, 5>(a, s);
    case 7: return launch_proto_regs_t<Vec<BT>, (F32 ? 4 : 2), 1, 6>(a, s);
    case 8: return launch_proto_regs_t<Vec<BT>, (F32 ? 4 : 2), 3, 3>(a, s);
    default: return launch_proto_regs_t<Vec<BT>, (F32 ? 4 : 2), 2, 4>(a, s);
  }
}

template <typename V>
int launch_proto_t(const SpmmArgs& a, cudaStream_t s) {
  using BT = typename V::T;
  constexpr int VPL = V::COLS == 1 ? 8 : V::COLS == 4 ? 2 : 1;
  constexpr int CWL = 32 * VPL * V::COLS;
  const bool comp = a.proto_max_nnz > kCompThreshold;
  // From the column lists, B slices staged by bulk copies when B's rows are
  // 16-byte aligned (BSP_SUMS_BULK = -1 selects the cluster form below, n >=
  // 0 a staging shape; defaults measured at 8192x8192x512: FP32 23.4 -> 22.8
  // us a step, BF16 20.1 -> 16.9 us)
  static const int sv = getenv("BSP_SUMS_BULK") ? atoi(getenv("BSP_SUMS_BULK")) : (sizeof(BT) == 4 ? 1 : 8);
  const int esz = (int)sizeof(BT);
  if (sv >= 0 && a.cons_idx && !comp && a.n_proto <= 65535 && reinterpret_cast<uintptr_t>(a.B) % 16 == 0 &&
      (a.ldb * esz) % 16 == 0 && (a.Nb * esz) % 16 == 0) {
    const int rc = launch_proto_sums_bulk(a, sv, s);
    if (rc != BSP_ERR_UNSUPPORTED) return rc;  // a shape too large for this B type: the cluster form
  }
  if (a.cons_idx && !comp && a.n_proto <= 65535 && ceil_div(a.N, CWL) * kSumCluster <= 0x7fffffff) {
    const dim3 g((unsigned)(ceil_div(a.N, CWL) * kSumCluster), (unsigned)a.n_proto);
    if (a.K * a.ldb < ((int64_t)1 << 31)) k_proto_sums_list<V, VPL, true><<<g, 256, 0, s>>>(a);
    else k_proto_sums_list<V, VPL, false><<<g, 256, 0, s>>>(a);
    BSP_LAUNCHED();
    return BSP_OK;
  }
  constexpr int CW = 32 * V::COLS;
  const int threads = 512;
  const size_t smem = (size_t)(threads / 32) * CW * sizeof(float) * (comp ? 2 : 1);
  const dim3 g((unsigned)a.n_proto, (unsigned)ceil_div(a.N, CW));
  const bool off32 = a.K * a.ldb < ((int64_t)1 << 31);
  if (comp && off32) k_proto_sums<V, 8, true, true><<<g, threads, smem, s>>>(a);
  else if (comp) k_proto_sums<V, 8, true, false><<<g, threads, smem, s>>>(a);
  else if (off32) k_proto_sums<V, 8, false, true><<<g, threads, smem, s>>>(a);
  else k_proto_sums<V, 8, false, false><<<g, threads, smem, s>>>(a);
  BSP_LAUNCHED();
  return BSP_OK;
}

// An aligned copy of B for layouts without 16-byte access: a warp takes 256
// columns of a row, 8 loads in flight.
template <typename T>
__global__ void __launch_bounds__(256) k_align_b(const T* __restrict__ B, int64_t K, int64_t N, int64_t ldb,
                                                 T* __restrict__ out, int64_t Nb) {
  const int lane = threadIdx.x & 31;
  const int64_t nch = (Nb + 255) / 256, total = K * nch;
  const int64_t nwarps = ((int64_t)gridDim.x * blockDim.x) >> 5;
  for (int64_t t = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 5; t < total; t += nwarps) {
    const int64_t k = total <= 0x7fffffff ? (int64_t)((uint32_t)t / (uint32_t)nch) : t / nch;
    const int64_t c0 = (t - k * nch) * 256 + lane;
    const T* src = B + k * ldb;
    T* dst = out + k * Nb;
    T v[8];
#pragma unroll
    for (int u = 0; u < 8; u++) v[u] = c0 + 32 * u < N ? __ldg(src + c0 + 32 * u) : T(0);
#pragma unroll
    for (int u = 0; u < 8; u++)
      if (c0 + 32 * u < Nb) dst[c0 + 32 * u] = v[u];
  }
}

// SDDMM on CUDA cores: a warp takes a row i of A, or a part of its words (so
// that few rows still fill the GPU).  It zeroes its part of dA's row, lists
// the set bits' columns in shared memory and forms 8 dot products
// G[i]·X[k] at a time: every lane keeps 8 FP32 sums over its columns of N, a
// vector of G serves 8 vectors of X, and one exchange of halves reduces all 8
// sums over the warp.  Bound by the L2 gather rate of X's rows.  One product
// at a time, with two scalar loads per lane in flight and a full reduction
// each, took 1246 us at 2048x2048, N = 1024 FP32, 10 % set; this takes 209 (8.4
// TB/s of gathered rows).
constexpr int kSdDots = 8;
template <typename V>
__global__ void __launch_bounds__(256) k_sddmm_rows(const uint32_t* __restrict__ A, int64_t M, int64_t K, int64_t Kw,
                                                    const typename V::T* __restrict__ G, int64_t ldg,
                                                    const typename V::T* __restrict__ X, int64_t ldx, int64_t N,
                                                    float* __restrict__ dA, int64_t ldda, int64_t part_words) {
  using T = typename V::T;
  constexpr int COLS = V::COLS, D = kSdDots;
  static_assert(D == 8, "the reduction below");
  __shared__ __align__(16) uint32_t lists[8][kListCap];
  const int lane = threadIdx.x & 31;
  uint32_t* list = lists[threadIdx.x >> 5];
  const int64_t row = (int64_t)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
  if (row >= M) return;
  float* out = dA + row * ldda;
  const T* g = G + row * ldg;
  const uint32_t* arow = A + row * Kw;
  for (int64_t p0 = (int64_t)blockIdx.y * part_words; p0 < Kw; p0 += (int64_t)gridDim.y * part_words) {
    const int64_t p1 = min(Kw, p0 + part_words);
    for (int64_t k = p0 * 32 + lane; k < min(K, p1 * 32); k += 32) out[k] = 0.f;
    __syncwarp();
    auto dots = [&](int i, int n) {  // list entries [i, i + n), n <= D (uniform)
      const T* x[D];
#pragma unroll
      for (int s = 0; s < D; s++) x[s] = X + (int64_t)list[i + (s < n ? s : 0)] * ldx;
      float acc[D];
#pragma unroll
      for (int s = 0; s < D; s++) acc[s] = 0.f;
      int64_t j = (int64_t)lane * COLS;
#pragma unroll 2
      for (; j + COLS <= N; j += 32 * COLS) {
        const typename V::Raw gr = V::load(g + j);
        typename V::Raw xr[D];
#pragma unroll
        for (int s = 0; s < D; s++) xr[s] = V::load(x[s] + j);
        float gf[COLS];
        V::cvt(gr, gf);
#pragma unroll
        for (int s = 0; s < D; s++) {
          float xf[COLS];
          V::cvt(xr[s], xf);
#pragma unroll
          for (int c = 0; c < COLS; c++) acc[s] = fmaf(gf[c], xf[c], acc[s]);
        }
      }
      for (int c = 0; COLS > 1 && c < COLS && j + c < N; c++)  // a last partial vector
#pragma unroll
        for (int s = 0; s < D; s++) acc[s] = fmaf(to_f32(g[j + c]), to_f32(x[s][j + c]), acc[s]);
      // the halves of the warp keep half of the sums each, three times over
#pragma unroll
      for (int o = 16, h = D / 2; o >= 4; o >>= 1, h >>= 1)
#pragma unroll
        for (int s = 0; s < D / 2; s++) {
          if (s >= h) break;
          const bool up = (lane & o) != 0;
          const float send = up ? acc[s] : acc[s + h];
          const float keep = up ? acc[s + h] : acc[s];
          acc[s] = keep + __shfl_xor_sync(kFull, send, o);
        }
      acc[0] += __shfl_xor_sync(kFull, acc[0], 2);
      acc[0] += __shfl_xor_sync(kFull, acc[0], 1);
      const int s = ((lane >> 4) & 1) * 4 + ((lane >> 3) & 1) * 2 + ((lane >> 2) & 1);
      if ((lane & 3) == 0 && s < n) out[list[i + s]] = acc[0];
    };
    int n = 0;
    uint32_t next = p0 + lane < p1 ? __ldg(arow + p0 + lane) : 0u;
    for (int64_t w0 = p0; w0 < p1; w0 += 32) {
      uint32_t w = next;
      next = w0 + 32 + lane < p1 ? __ldg(arow + w0 + 32 + lane) : 0u;
      const int c = __popc(w);
      int incl = c;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const int y = __shfl_up_sync(kFull, incl, o);
        if (lane >= o) incl += y;
      }
      int pos = n + incl - c;
      while (w) {
        list[pos++] = (uint32_t)(w0 + lane) * 32u + (uint32_t)(__ffs(w) - 1);
        w &= w - 1;
      }
      n += __shfl_sync(kFull, incl, 31);
      const bool last = w0 + 32 >= p1;
      if (n < kListStep && !last) continue;
      __syncwarp();
      int i = 0;
      for (; i + D <= n; i += D) dots(i, D);
      n -= i;
      if (last) {
        if (n > 0) dots(i, n);
      } else if (i > 0) {
        const uint32_t rest = lane < n ? list[i + lane] : 0u;
        __syncwarp();
        if (lane < n) list[lane] = rest;
      }
      __syncwarp();
    }
  }
}

template <typename T>
int launch_sddmm_t(const uint32_t* A, int64_t M, int64_t K, const T* G, int64_t ldg, const T* X, int64_t ldx, int64_t N,
                   float* dA, int64_t ldda, cudaStream_t s) {
  const int64_t Kw = ceil_div(K, 32);
  // rows cut into parts of whole 32-word groups until 16 warps an SM run
  const int64_t groups = ceil_div(Kw, 32);
  int64_t parts = ceil_div((int64_t)num_sms() * 16, M);
  if (parts > groups) parts = groups;
  if (parts > 65535) parts = 65535;
  const int64_t part_words = ceil_div(groups, parts) * 32;
  const dim3 grid((unsigned)ceil_div(M, 8), (unsigned)ceil_div(Kw, part_words));
  constexpr int esz = (int)sizeof(T);
  const bool vec = is_aligned(G, 16) && is_aligned(X, 16) && (ldg * esz) % 16 == 0 && (ldx * esz) % 16 == 0;
  if (vec) k_sddmm_rows<Vec<T>><<<grid, 256, 0, s>>>(A, M, K, Kw, G, ldg, X, ldx, N, dA, ldda, part_words);
  else k_sddmm_rows<Elem1<T>><<<grid, 256, 0, s>>>(A, M, K, Kw, G, ldg, X, ldx, N, dA, ldda, part_words);
  BSP_LAUNCHED();
  return BSP_OK;
}

}  // namespace

int launch_align_b(const void* B, int bdt, int64_t K, int64_t N, int64_t ldb, void* out, int64_t Nb, cudaStream_t s) {
  if (K == 0 || Nb == 0) return BSP_OK;
  const int64_t blocks = ceil_div(K * ceil_div(Nb, 256), 8), cap = (int64_t)num_sms() * 8;
  const unsigned grid = (unsigned)(blocks < cap ? blocks : cap);
  if (dtype_size(bdt) == 4) k_align_b<<<grid, 256, 0, s>>>((const uint32_t*)B, K, N, ldb, (uint32_t*)out, Nb);
  else k_align_b<<<grid, 256, 0, s>>>((const uint16_t*)B, K, N, ldb, (uint16_t*)out, Nb);
  BSP_LAUNCHED();
  return BSP_OK;
}

int launch_sddmm_rows(const uint32_t* A, int64_t M, int64_t K, const void* G, int64_t ldg, const void* X,
                      int64_t ldx, int dt, int64_t N, float* dA, int64_t ldda, cudaStream_t s) {
  if (M == 0 || K == 0) return BSP_OK;
  switch (dt) {
    case BSP_F32: return launch_sddmm_t(A, M, K, (const float*)G, ldg, (const float*)X, ldx, N, dA, ldda, s);
    case BSP_BF16:
      return launch_sddmm_t(A, M, K, (const __nv_bfloat16*)G, ldg, (const __nv_bfloat16*)X, ldx, N, dA, ldda, s);
    case BSP_F16: return launch_sddmm_t(A, M, K, (const __half*)G, ldg, (const __half*)X, ldx, N, dA, ldda, s);
    default: return BSP_ERR_UNSUPPORTED;
  }
}

int launch_spmm_rows(const SpmmArgs& a, bool vec, cudaStream_t s) {
  if (a.M == 0 || a.N == 0) return BSP_OK;
  switch (a.bdt) {
    case BSP_F32: return vec ? launch_rows_t<Vec<float>>(a, s) : launch_rows_t<Elem1<float>>(a, s);
    case BSP_BF16: return vec ? launch_rows_t<Vec<__nv_bfloat16>>(a, s) : launch_rows_t<Elem1<__nv_bfloat16>>(a, s);
    case BSP_F16: return vec ? launch_rows_t<Vec<__half>>(a, s) : launch_rows_t<Elem1<__half>>(a, s);
    default: return BSP_ERR_UNSUPPORTED;
  }
}

int launch_spmm_rows_wide(const SpmmArgs& a, cudaStream_t s) {
  if (a.M == 0 || a.N == 0) return BSP_OK;
  switch (a.bdt) {
    case BSP_F32: return launch_rows_wide_t<float>(a, s);
    case BSP_BF16: return launch_rows_wide_t<__nv_bfloat16>(a, s);
    case BSP_F16: return launch_rows_wide_t<__half>(a, s);
    default: return BSP_ERR_UNSUPPORTED;
  }
}

int launch_spmm_proto_regs(const SpmmArgs& a, int variant, bool vec, cudaStream_t s) {
  if (a.M == 0 || a.N == 0) return BSP_OK;
  switch (a.bdt) {
    case BSP_F32: return launch_proto_regs_v<float>(a, variant, vec, s);
    case BSP_BF16: return launch_proto_regs_v<__nv_bfloat16>(a, variant, vec, s);
    case BSP_F16: return launch_proto_regs_v<__half>(a, variant, vec, s);
    default: return BSP_ERR_UNSUPPORTED;
  }
}

int launch_proto_sums(const SpmmArgs& a, bool vec, cudaStream_t s) {
  if (a.n_proto == 0 || a.N == 0) return BSP_OK;
  switch (a.bdt) {
    case BSP_F32: return vec ? launch_proto_t<Vec<float>>(a, s) : launch_proto_t<Elem1<float>>(a, s);
    case BSP_BF16: return vec ? launch_proto_t<Vec<__nv_bfloat16>>(a, s) : launch_proto_t<Elem1<__nv_bfloat16>>(a, s);
    case BSP_F16: return vec ? launch_proto_t<Vec<__half>>(a, s) : launch_proto_t<Elem1<__half>>(a, s);
    default: return BSP_ERR_UNSUPPORTED;
  }
}

}  // namespace bsp
