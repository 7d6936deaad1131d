// Host-side helpers shared by the GEMM translation units: the tensor-map cache, tiling defaults
// and the operand set-up of C[M,N] = A[M,K] * Bt[N,K]^T. Defined in gemm.cu.
#pragma once
#include <algorithm>
#include <cmath>
#include "kraken/driver_api.h"
#include "kraken/gemm_core.cuh"

namespace kraken {

// Tensor map of a row-major bf16 (elt 2) or fp32 (elt 4) matrix [rows, cols] (cols contiguous, `ld`
// elements per row), box = box_bytes (128 or 64) of columns x box_rows rows, swizzled by as much, out-of-range
// elements read as zero. narrow_rows > 0: *narrow is the same with boxes of so many rows. Cached.
int get_tmap(const void* ptr, unsigned long long rows, unsigned long long cols, unsigned long long ld,
             unsigned box_rows, CUtensorMap* out, int elt = 2, unsigned box_bytes = 128, bool promote_256 = true,
             unsigned narrow_rows = 0, CUtensorMap* narrow = nullptr);
// Tensor map for TMA stores of bf16 tiles (box of 32 rows); false when the matrix cannot be
// described to TMA or TMA stores are switched off.
bool store_tmap(const void* ptr, long long rows, long long cols, long long ld, CUtensorMap* m);
bool tma_store_enabled();       // KRAKEN_TMA_STORE
int default_group_r();
bool pair_enabled();
unsigned grid_cap(const DeviceState* d);
int setup_problem(GemmParams& p, const void* a, long long lda, const void* bt, long long ldb, int M, int N, int K,
                  bool swap, int bn_override, int* bn_out, int elt = 2, int c_box_rows = 0, bool promote_256 = true, int narrow_rows = 0,
                  CUtensorMap* narrow = nullptr);
// Single-CTA kernels for fp32 operands multiplied as tf32 (GEMM -> all-reduce; column tiles of 16, 64 or 256). Defined in gemm_tf32.cu.
int launch_gemm_tf32(int bn, const GemmParams& p, unsigned nb, cudaStream_t stream);
// Single-CTA kernels of the decode GEMM -> all-reduce. Defined in gemm_ar.cu.
int launch_gemm_ar(int bn, const GemmParams& p, unsigned nb, cudaStream_t stream);
// Routes a parameter block to the kernel family of its mode and operand type (gemm.cu).
int launch_gemm(int bn, const GemmParams& p, unsigned nb, cudaStream_t stream);
// Fewer SMs busy run faster (power), up to full clock.
constexpr double kBusyFloor = 0.79;
inline double busy_factor(double busy) { return std::max(kBusyFloor, std::pow(busy, 0.24)); }
// What planning cost this thread: plans worked out, kernels whose time was worked out for them.
struct PlanStats {
  unsigned long long plans, timed;
};
// One-wave GEMM (gemm_tile.cu): the K splits with which `tiles` tiles of this kernel run at once in less than *us, and that
// time in *us; 0 when there are none (kb_us: one K block of a tile, hbm_us: the operands' time out of HBM); and its launch.
constexpr double kTilePairUs = 5.5, kTileSingleUs = 4.6;       // its start and end
int tile_gemm_splits(const DeviceState* d, int tiles, int num_kb, int bn, bool pair, int elt, double kb_us, double hbm_us, double* us, PlanStats* stats);
int launch_tile_gemm(const GemmParams& g, int bn, bool pair, int splits, cudaStream_t stream);
// Persistent pairs that draw their tiles in order (gemm_flow.cu); sched: two zero words, zero again afterwards.
// last_cols: columns of the last column tile, in 16s; below bn with a tensor map of half as many rows of the column operand.
int launch_flow_gemm(const GemmParams& g, int bn, int rb, int pairs, int last_cols, const CUtensorMap& tmap_last, uint32_t* sched,
                     cudaStream_t stream);
int pick_bn(int rows_c);      // column-tile width for `rows_c` rows of the column operand
int tf32_bn(int rows_c);      // the same among the widths the tf32 kernels exist for

}  // namespace kraken
