// ts.cuh — the persistent tensor-core kernel's launcher (spmm_ts.cu).
#pragma once
#include <cuda.h>

#include "bsp_internal.cuh"
#include "spmm.cuh"

namespace bsp {

struct TsArgs {
  const uint32_t* A;   // packed rows [M][Kw]
  const uint32_t* At;  // A's words column by column ([Kw][M], launch_transpose_words), or null
  int64_t M, K, Kw;
  int64_t N;
  float* C;            // [M][ldc]; trans: dX [K][ldc]
  int64_t ldc;
  bool c_vec;          // C's rows start on 16 bytes
  bool out16;          // trans: dX in G's 16-bit type (C and ldc in its elements, 16-byte rows, no splits)
  bool c_map;          // (set by the launcher) the output leaves by TMA
  const uint32_t* occ; // occupancy bitmap of 128-row blocks (trans: of 128-column blocks)
  int occ_words;
  int bdt;
  // split-K: slice z of an item's tile list goes to part + z*part_stride (row stride ldp, 16-byte rows); null
  // = one slice, to C
  float* part;
  int64_t ldp, part_stride;
  // B (or G) in tile order, bt_cb blocks of 256 columns per 32-row tile; null = TMA boxes through the map
  const uint8_t* bt;
  int64_t bt_cb;
  const uint4* tiles;  // int8 A in [K tile][row][32] order instead of words; null = words
  // batch: work items (problem, 256-row block, 128-column block, K tiles) and the problems' records
  const BatchProblemTc* probs;
  const int4* items;
  const int* skip_if;  // device flag: nonzero = leave C alone; null = run
  // Every seg_stages stages (of four K tiles; 0 = never) the accumulators are
  // cleared and their sums added to the output in FP32, rounded to nearest (by
  // the memory system, one warp's additions in order; subnormal sums may become
  // zero there, so values below 2^-100 are not for this form): the tensor cores
  // cut their own sums off towards zero after every 16 products.
  int seg_stages;
};

// rows and columns of the output per work item
int64_t ts_item_rows();
int64_t ts_item_cols();
int64_t ts_max_cols();  // widest output that launch_ts takes
int launch_ts(TsArgs a, const CUtensorMap& map, bool trans, int splits, cudaStream_t s);
// Every item of a batch: C = A·B of its problem (trans: dX = Aᵀ·G), longest items first.
int launch_ts_batch(const BatchProblemTc* probs, const int4* items, int n_items, int64_t N, int bdt, bool trans,
                    cudaStream_t s);
int ts_device_error(int* out, bool clear);

}  // namespace bsp
