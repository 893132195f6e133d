// Which part of a pooling window one of several warps adds up.  Plain C++ so that the arithmetic can be checked on the host.
#pragma once

#ifdef __CUDACC__
#define FDNN_HOST_DEVICE __host__ __device__ __forceinline__
#else
#define FDNN_HOST_DEVICE inline
#endif

namespace fdnn {

// First element of stretch `slice` of `slices` nearly equal stretches of `count` elements; stretch `slice` ends where the
// next one starts.  64 bits: a window is a whole plane at most, H * W below 2^62, and the product is with `slices`.
FDNN_HOST_DEVICE long long stretch_begin(long long count, int slice, int slices) {
  return count / slices * slice + count % slices * slice / slices;
}

}  // namespace fdnn
