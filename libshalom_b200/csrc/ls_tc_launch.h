// ls_tc_launch.h -- host-side entry points of the split-BF16 tcgen05 kernels.
#pragma once

#include "../../include/LibShalom.h"
#include "ls_simt.cuh"

namespace ls {

// Single (irregular) SGEMM on the tensor cores; `mode` is a
// LIBSHALOM_PREC_BF16X* value, `splits` as LibShalom_set_splitk.
// splits: 0 = chosen here, s > 0 = about s slices; *used (if given) gets the
// factor launched
int tc_sgemm_single(const GemmArgs<float> &g, int mode, int splits, int *used = nullptr);

// Uniform batch on the tensor cores.
int tc_sgemm_strided(const GemmArgs<float> &g, long sA, long sB, long sC, long count, int mode);

// Grouped batch (entries in device memory) on the tensor cores.
int tc_sgemm_grouped(const LibShalom_sgemm_entry *entries, long count, int mode);

// Tiles of the small-product kernel (ls_tc_small.cu): C rows and columns.
constexpr int SM_SMALL_TM = 64, SM_SMALL_TN = 128;
// Its K chunks, and the rows of a tile whose chunk sums fit beside the
// accumulators (tiles of its HOLD loop, for products of several chunks that
// read C).
constexpr int SM_SMALL_CHUNK = 128, SM_SUM_ROWS = 32;

// Work of the small-product kernel.  Grouped: items {first entry of the run,
// products << 5 | hold << 4 | tile} in device memory, n_items_dev[0] upwards from
// items[0] and, of the HOLD loop, n_items_dev[1] downwards from items[n_slots - 1].
// Uniform: GEMM g of the batch at A + g * sA etc., `tiles` tiles each.
struct TcSmallArgs {
  const LibShalom_sgemm_entry *entries;
  const uint2 *items;
  long n_slots;
  const unsigned *n_items_dev;
  unsigned *counter;  // zeroed before the launch
  const float *A, *B;
  float *C;
  long sA, sB, sC, lda, ldb, ldc, n_items;
  int M, N, K, transb, tiles, tiles_n;
  float alpha, beta;
  unsigned *err;  // device status word (bounded waits)
};
// hold: of a uniform batch
int tc_small_launch(const TcSmallArgs &a, bool uniform, bool hold, int mode);

// Runs the bounded-wait self-check kernel (an mbarrier nothing arrives at);
// returns LIBSHALOM_ERR_DEVICE_TIMEOUT when its waits expired and reported.
int tc_wait_expiry_selftest(int iterations);

}  // namespace ls
