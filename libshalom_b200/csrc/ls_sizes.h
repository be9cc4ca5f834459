// ls_sizes.h -- counts of tiles and slabs from sizes that may lie anywhere in
// int: grouped entries are read on the device, where no call refuses them.
#pragma once

#ifdef __CUDACC__
#define LS_HOST_DEVICE __host__ __device__ __forceinline__
#else
#define LS_HOST_DEVICE inline
#endif

namespace ls {

// ceil(n / d), 0 for n <= 0 (n + d - 1 does not fit an int for n near its end)
LS_HOST_DEVICE int ceil_div(int n, int d) { return n > 0 ? (n - 1) / d + 1 : 0; }
// the same, at least 1: slabs of a product (one of K = 0 still updates C)
LS_HOST_DEVICE int slabs(int n, int d) { return n > 0 ? (n - 1) / d + 1 : 1; }

}  // namespace ls
