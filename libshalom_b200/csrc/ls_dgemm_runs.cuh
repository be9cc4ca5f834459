// ls_dgemm_runs.cuh -- the run list of a grouped FP64 batch: maximal groups of
// consecutive entries naming the same C, found and ordered on the device.
#pragma once

#include "ls_common.cuh"

namespace ls {

constexpr int DM_CLASSES = 64;  // run cost classes of the heaviest-first order; the
                                // first is that of the deep runs
// Shapes of a run's C block, each with its own code in the kernels: 0 both
// edges above 16, 1 at most 16 columns, 2 at most 16 rows
constexpr int DM_SHAPES = 3;
constexpr int DM_BINS = DM_SHAPES * DM_CLASSES;

// Runs with a C block of at most 32 x 32 (small), by shape and then heaviest
// first, and the others (large).
struct RunPlan {
  unsigned few;                  // deep small runs are large ones where there are no
                                 // more small runs than this
  unsigned *n_large;
  unsigned *n_shape;             // [DM_SHAPES] runs
  unsigned *bin_runs, *bin_fill; // [DM_BINS] each
  unsigned *small_first, *small_len;
  unsigned *large_first, *large_len;
  // from the first pass for the second: an entry's bin (DM_BINS: not the start
  // of a small run) and its run's length
  unsigned *entry_len;
  unsigned char *entry_bin;
};

// word `lane` of an entry: loaded a product ahead and broadcast when it is
// needed, so that no product waits for its entry
__device__ __forceinline__ uint32_t entry_word(const LibShalom_dgemm_entry *e, int lane) {
  return lane < 18 ? reinterpret_cast<const uint32_t *>(e)[lane] : 0u;
}
static_assert(sizeof(LibShalom_dgemm_entry) == 72, "entry words");

// lists the runs on the library's stream (scratch: 2 KB + 21 bytes an entry)
int plan_dgemm_runs(const LibShalom_dgemm_entry *entries, long count, unsigned few, RunPlan *pl);

}  // namespace ls
