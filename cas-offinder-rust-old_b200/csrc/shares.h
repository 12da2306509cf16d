// shares.h -- a whole split into consecutive shares, on the host and on the device.
#pragma once

#include <cstdint>

#ifdef __CUDACC__
#define COF_HOST_DEVICE __host__ __device__
#else
#define COF_HOST_DEVICE
#endif

namespace cof {

// First element of share i of n (i = n: the end).  The shares cover [0, total)
// in order and differ by one element at most; no product passes `total`, which
// may be any 32-bit number.
COF_HOST_DEVICE inline uint32_t share_begin(uint32_t total, uint32_t i, uint32_t n) {
    const uint32_t rest = total % n;
    return total / n * i + (i < rest ? i : rest);
}

}  // namespace cof
