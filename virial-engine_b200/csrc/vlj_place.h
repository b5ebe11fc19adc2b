// Where the stand-alone grid's scatter puts a particle, in plain C++ so that
// the host can check it too.
#pragma once

#include <stdint.h>

#ifdef __CUDACC__
#define VLJ_HOST_DEVICE __host__ __device__ __forceinline__
#else
#define VLJ_HOST_DEVICE inline
#endif

namespace vlj {

// The place in the order of n particles for one whose cell begins at `start`
// and whose cell's counter held `left` before it took one off. False where
// there is none. That happens only when overlapping calls share a scratch:
// one call clears counters that another still runs down, so a counter can be
// seen at zero, and after that as wrapped below zero. The order is then
// undefined, but every place written lies in the buffer.
VLJ_HOST_DEVICE bool scatter_place(uint32_t start, uint32_t left, uint32_t n, uint32_t* at) {
    *at = start + left - 1u;
    return left != 0u && *at < n;
}

}  // namespace vlj
