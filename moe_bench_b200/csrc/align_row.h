// Row arithmetic of the sort-and-pad step, apart from its kernels so that the host can check it.
#pragma once

#include <cstdint>

#ifdef __CUDACC__
#define MB200_HOST_DEVICE __host__ __device__ __forceinline__
#else
#define MB200_HOST_DEVICE inline
#endif

namespace mb200 {

// Row of an assignment: its expert's segment starts at row block `first_block`, and `before` of the
// expert's assignments come ahead of it.  Both fit 32 bits; the row need not: 2^31 - 4097 assignments
// (the most the sort accepts) plus up to pad - 1 padding rows per expert pass 2^31, and a wrapped row
// would be negative, below any capacity, and stored in front of the buffer.
MB200_HOST_DEVICE int64_t sorted_row(int first_block, int pad, int before) {
  return int64_t(first_block) * pad + before;
}

}  // namespace mb200
