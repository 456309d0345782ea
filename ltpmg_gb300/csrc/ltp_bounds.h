// ltp_bounds.h -- bounds predicates on numbers that a caller supplies.
#pragma once
#include <stdint.h>

#ifdef __CUDACC__
#define LTP_HOST_DEVICE __host__ __device__ __forceinline__
#else
#define LTP_HOST_DEVICE inline
#endif

namespace ltp {

// Does a row of `slots` payload slots that starts at slot `key` lie inside a
// payload of `len` slots?  An insert's key may be any 64-bit number, so the
// row's end is not computed: key + slots wraps for keys near 2^64.
LTP_HOST_DEVICE bool payload_row_fits(uint64_t key, uint64_t slots, uint64_t len) {
    return slots <= len && key <= len - slots;
}

}  // namespace ltp
