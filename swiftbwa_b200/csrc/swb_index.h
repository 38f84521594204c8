// swb_index.h -- index arithmetic of kernels that give several threads to one
// item.  Plain C++, so that a host compiler checks it too.
#pragma once

#include <cstddef>

#ifdef __CUDACC__
#define SWB_HD __host__ __device__
#else
#define SWB_HD
#endif

namespace swb {

// The item of a thread when `per` consecutive threads share one.  The thread
// number passes 32 bits long before the item does (2^29 items of eight threads).
SWB_HD inline size_t group_item(unsigned block, unsigned block_threads, unsigned thread, unsigned per) {
    return ((size_t)block * block_threads + thread) / per;
}

}  // namespace swb
