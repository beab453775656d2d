// spmm.cuh — argument block and launchers of the CUDA-core SpMM kernels.
#pragma once
#include <cuda.h>

#include "bsp_internal.cuh"

namespace bsp {

constexpr int kCompThreshold = 4096;  // set bits above which rows use TwoSum

// One problem of the batched form on the tensor cores: B's tensor map (64x32
// boxes, 128-byte swizzle; first, so the record keeps the map's alignment), A
// and C.
struct BatchProblemTc {
  CUtensorMap map;   // forward: B [K][N]; Aᵀ·G: G [M][N] (64x32 boxes); SDDMM: G [M][N] (64x256 boxes)
  CUtensorMap map2;  // SDDMM: X [K][N] (64x256 boxes); forward, Aᵀ·G: C, dX (make_out_map)
  CUtensorMap map3;  // SDDMM: G [M][N] in 64x128 boxes (the persistent batched SDDMM); otherwise unused
  const uint32_t* A;
  int64_t M, K, Kw;
  float* C;          // forward: C [M][N]; Aᵀ·G: dX [K][N]; SDDMM: dA [M][K]
  int64_t ldc;
};
// Tensor map of a batch problem's B [K][N] (row stride ldb elements), or of
// G [M][N] for the batched Aᵀ·G: 64-column x 32-row boxes.
int make_batch_map(CUtensorMap* m, const void* B, int bdt, int64_t K, int64_t N, int64_t ldb);
// Tensor map of G [M][N] or X [K][N] for the batched SDDMM: 64-column x
// 256-row boxes.
int make_batch_map_sddmm(CUtensorMap* m, const void* T, int bdt, int64_t rows, int64_t N, int64_t ld,
                         int box_rows = 256);
// Tensor map of an FP32 output [rows][cols] (row stride ld floats, 16-byte
// aligned), `splits` of them split_stride floats apart: 32x32 boxes, 128-byte
// swizzle.
int make_out_map(CUtensorMap* m, float* C, int64_t rows, int64_t cols, int64_t ld, int splits, int64_t split_stride);
// The same of a 16-bit output: 64 x 32 boxes.
int make_out_map16(CUtensorMap* m, void* C, int dt, int64_t rows, int64_t cols, int64_t ld);
// Rows of FP32 X in plain boxes (16-byte rows): zeros past the matrix.
int make_rows_map_f32(CUtensorMap* m, const float* X, int64_t rows, int64_t cols, int64_t ld, int box_cols, int box_rows);
// Work item b = {problem, 256-row block, 256-column block, reduction tiles}:
// one CTA each.  kind 0 = forward C = A·B, 1 = dX = Aᵀ·G (rows: K),
// 2 = dA = (G·Xᵀ) ⊙ A (columns: K).
int launch_batched_tc(const BatchProblemTc* probs, const int4* items, int n_items, int64_t N, int bdt,
                      cudaStream_t s, int kind = 0);

struct SpmmArgs {
  const uint32_t* A;  // packed rows [M][Kw], LSB-first
  int64_t M, K, Kw;
  const void* B;      // [K][ldb] of bdt
  int bdt;
  int64_t ldb, N;
  int64_t Nb;         // columns of B that may be read: N, or N rounded up to a vector in an aligned copy of B
  float* C;           // [M][ldc]
  int64_t ldc;
  bool c_vec;         // C's rows take 16-byte stores (else element by element)
  bool no_long_rows;  // a plan says that no row has more than kCompThreshold set bits
  const int* run_if;  // device flags: all zero = do nothing (walking kernels only); null = run
  int run_if_n;       // how many (0 = one)
  bool run_if_late;   // the kernel before sets them: launched as its programmatic dependent
  // prototype mode (plan)
  const int32_t* row_cluster;  // [M], -1 = walk A's row
  const int32_t* delta_ptr;    // [M+1]
  const uint32_t* delta_idx;   // column | 0x80000000 for "subtract"
  int64_t n_delta;             // entries in delta_idx
  const uint32_t* cons;        // [n_proto][Kw] prototype masks
  int64_t n_proto;
  int64_t proto_max_nnz;       // set bits of the densest prototype (TwoSum above 4096)
  const uint32_t* delta_pad;   // [n_slot][32] row slots (row, cluster, count, start, 28 entries), or null
  int64_t n_slot;              // clustered rows, in slot order
  const int32_t* cons_ptr;     // [n_proto + 1] prototype column lists, or null
  const uint32_t* cons_idx;
  float* P;                    // [n_proto][ldp] prototype sums (workspace)
  int64_t ldp;
  // optional row subset for the walking kernel (rows of A without a cluster)
  const int32_t* row_list;     // [n_list] or nullptr = rows 0..M-1
  int64_t n_list;
};

// Sizes of the values of B [R][N] by column (col_stats.cu).
constexpr int kStatTop = 127 + 100;
constexpr int64_t kStatMaxRows = 65536;  // (a block reads all of them)
constexpr int kStatCols = 8;             // columns of a block
// n_flags device flags, at most 512, one of them nonzero if a value is not finite
// or at least 2^100, or if a column's largest exponent is more than `octaves`
// above the mean one of its nonzeros; runs beside the kernels before it.  In
// col_stats_bytes(N) of workspace.
size_t col_stats_bytes(int64_t N);
int launch_col_stats(const void* B, int bdt, int64_t R, int64_t N, int64_t ldb, void* ws, int octaves,
                     const int** flags, int* n_flags, cudaStream_t s);
// The values of a product in parts (spmm_tc.cu), R up to 4096: bad[b] = 1 if
// columns 8b to 8b+7 do not pass (see k_split_b, which sets flag then).
constexpr int kStatBottom = 127 - 100;
constexpr int kPartsLow = 16;
constexpr float kPartsLimit = 0.7f;
struct PartsStats {
  int* flag;
  int* bad;
};
size_t parts_stats_bytes(int64_t N);
int launch_parts_stats(const float* B, int64_t R, int64_t N, int64_t ldb, void* ws, float addends, PartsStats* st,
                       cudaStream_t s);
// B [K][N] (row stride ldb, any alignment) -> out [K][Nb], columns N..Nb-1 zero
int launch_align_b(const void* B, int bdt, int64_t K, int64_t N, int64_t ldb, void* out, int64_t Nb, cudaStream_t s);
// vec = B's layout allows 16-byte vector access (else lane-per-column path)
int launch_spmm_rows(const SpmmArgs& a, bool vec, cudaStream_t s);
// prototype plans of A with 2^30 or more columns (vec layouts only)
int launch_spmm_rows_wide(const SpmmArgs& a, cudaStream_t s);
int launch_proto_sums(const SpmmArgs& a, bool vec, cudaStream_t s);
// Clustered rows through registers, launched as a programmatic dependent of
// the prototype-sum kernel; rows without a cluster are left to the walker.
int launch_spmm_proto_regs(const SpmmArgs& a, int variant, bool vec, cudaStream_t s);

// Prototype rows through TMA bulk copies staged in shared memory
// (spmm_bulk.cu).  Needs the vector layout; rows without a cluster are
// skipped (walk them with launch_spmm_rows over the plan's direct-row list).
int launch_spmm_proto_bulk(const SpmmArgs& a, int variant, cudaStream_t s);
// Device-side error word of the bulk kernels (0 = none); clear resets it.
int bulk_device_error(int* out, bool clear);
// Prototype sums from the column lists with B slices staged by bulk copies
// (B 16-byte aligned, ldb·esize and N·esize multiples of 16).
int launch_proto_sums_bulk(const SpmmArgs& a, int variant, cudaStream_t s);

// Tensor-core path (spmm_tc.cu) for 16-bit B: occupancy bitmap of 32-column
// K tiles per 128-row block ([ceil(M/128)][tc_occupancy_words(K)]), then the
// tcgen05 kernel over the occupied tiles.
int tc_occupancy_words(int64_t K);
// Longest reduction (K forward, M transposed) the tensor-core kernels take:
// a CTA lists its occupied 32-column tiles in shared memory.
int64_t tc_max_reduction();
int tc_occupancy_t_words(int64_t M);
int launch_occupancy(const uint32_t* A, int64_t M, int64_t K, uint32_t* occ, uint32_t* occT,
                     unsigned long long* count, unsigned long long* countT, cudaStream_t s);
// ws (optional): room for split-K partials (used when the output grid is
// small and ws_bytes ≥ tc_split_bytes(...)) and, after them, for B in tile
// order (used when the rest holds tc_tiled_b_bytes(...)); else ignored.
// At (optional): A's words column by column ([Kw][M], launch_transpose_words)
// for coalesced word loads; null = loads from the rows.
// form: the tile form a tuned schedule fixes (-1 = the rule): B pre-tiled (1)
// or by TMA boxes (0), split-K allowed (-1) or not (0).  tps, once the K tiles
// of a stage, chooses nothing: one stage form is built.
struct TcForm {
  int tps = 0, tiled = -1, split = -1;
};
// vec = false (layouts without 16-byte access): B has to fit the workspace in
// tile order, and *skipped becomes a device flag that is nonzero when the
// product was left to the walking kernels (infinities or NaN in B, which a
// dense product would spread over rows that do not hold their column).
int launch_spmm_tc(const SpmmArgs& a, const uint32_t* occ, const uint32_t* At, bool vec, cudaStream_t s, void* ws,
                   size_t ws_bytes, TcForm form, const int** skipped);
int launch_transpose_words(const uint32_t* words, int64_t M, int64_t Kw, uint32_t* At, cudaStream_t s);
int tc_split_count(int64_t out_rows, int64_t out_cols, int64_t red_tiles);
size_t tc_split_bytes(int64_t out_rows, int64_t out_cols, int64_t red_tiles);
// B (fwd) / G (trans) copied into tile order for one bulk copy per tile: the
// workspace it takes, and the workspace with which the tensor-core launch
// both splits the reduction (when it would) and tiles B; any_layout: and, where
// the output's rows cannot start on 16 bytes, keeps its sums in rows that do.
size_t tc_tiled_b_bytes(int64_t red_rows, int64_t cols);
size_t tc_preferred_bytes(int64_t out_rows, int64_t out_cols, int64_t red_rows, bool any_layout = false);
// ... of a 16-bit B without 16-byte rows: in tile order always
size_t tc_unaligned_bytes(int64_t out_rows, int64_t out_cols, int64_t red_rows);
// FP32 B (any layout) on the tensor cores as three exact BF16 parts: C = A·B, or
// dX = Aᵀ·G with occT; the workspace must hold tc_parts_bytes(output rows, N,
// reduction rows), nnz are A's set bits.  *skipped: a device flag, nonzero when C was left to the
// walking kernels (values outside the parts' range, or too unequal for exact sums).
size_t tc_parts_bytes(int64_t out_rows, int64_t N, int64_t red_rows);
int launch_spmm_parts(const uint32_t* A, int64_t M, int64_t K, const uint32_t* occ, const uint32_t* At, int64_t nnz,
                      const float* B, int64_t ldb, int64_t N, float* C, int64_t ldc, bool trans, cudaStream_t s,
                      void* ws, size_t ws_bytes, const int** skipped);
// dX[K][N] = Aᵀ·G on the tensor cores, Aᵀ read from A's row words
int launch_spmm_t_tc(const uint32_t* A, int64_t M, int64_t K, const void* G, int gdt, int64_t ldg, int64_t N,
                     void* dX, bool out16, int64_t lddx, const uint32_t* occT, const uint32_t* At, cudaStream_t s,
                     void* ws, size_t ws_bytes);
// C = A·B for int8 A in the order of launch_i8_tiles (values [ceil(K/32)][M][32], then a bit per 128 x 32
// tile with a nonzero), 16-bit B, vector layouts; with tc_i8_bytes of workspace B goes there in two parts
// (k_split16_b), with less as it is
size_t tc_i8_bytes(int64_t M, int64_t N, int64_t K);
size_t i8_values_bytes(int64_t M, int64_t K);
size_t i8_tiles_bytes(int64_t M, int64_t K);
int launch_spmm_i8_tc(const void* tiles, int64_t M, int64_t K, const void* B, int bdt, int64_t ldb, int64_t N, float* C,
                      int64_t ldc, void* ws, size_t ws_bytes, cudaStream_t s);
int launch_i8_tiles(const int8_t* A, int64_t M, int64_t K, int64_t lda, int8_t* tiles, cudaStream_t s);
// dA[M][K] = (G·Xᵀ) at A's set bits, 0 elsewhere, on the tensor cores
int launch_sddmm_tc(const uint32_t* A, int64_t M, int64_t K, const void* G, int64_t ldg, const void* X,
                    int64_t ldx, int dt, int64_t N, float* dA, int64_t ldda, cudaStream_t s);
// same on CUDA cores (any dtype / layout): warp per row, one dot product per set bit
// 16-bit dA = (G·Xᵀ) ⊙ A on the persistent batched kernel: one problem, layouts as for launch_sddmm_tc, which
// calls it for outputs of few tiles
int launch_sddmm_persist(const uint32_t* A, int64_t M, int64_t K, const void* G, int64_t ldg, const void* X,
                         int64_t ldx, int dt, int64_t N, float* dA, int64_t ldda, cudaStream_t s);
// FP32, 16-byte rows of G and X: X staged in shared memory for 32 rows of A at a time.
int launch_sddmm_staged(const uint32_t* A, int64_t M, int64_t K, const float* G, int64_t ldg, const float* X,
                        int64_t ldx, int64_t N, float* dA, int64_t ldda, cudaStream_t s);
int sddmm_staged_device_error(int* out, bool clear);
int launch_sddmm_rows(const uint32_t* A, int64_t M, int64_t K, const void* G, int64_t ldg, const void* X,
                      int64_t ldx, int dt, int64_t N, float* dA, int64_t ldda, cudaStream_t s);
int tc_device_error(int* out, bool clear);
int batched_device_error(int* out, bool clear);



}  // namespace bsp
