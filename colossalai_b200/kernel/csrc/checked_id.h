// The row of a table that an id names.  An id outside the table ends the kernel in an assertion, as in torch's index kernels: no row
// is made up for it.  Plain C++ beside CUDA, so that the rule can be run on the host.
#pragma once
#include <assert.h>
#include <stdint.h>

#ifdef __CUDACC__
#define CB_CHECKED_ID __host__ __device__ __forceinline__
#else
#define CB_CHECKED_ID inline
#endif

CB_CHECKED_ID int64_t cb_checked_id(int64_t id, int64_t entries) {
  assert(id >= 0 && id < entries && "an embedding id is outside the table");
  return id;
}
