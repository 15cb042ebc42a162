// The common case of reducing a difference to [0, p), p = 2^255 - 19.
// Plain C++ with one macro, so that a CPU build of the same code can be
// checked against integers.
#pragma once
#include <cstdint>

#ifdef __CUDACC__
#define FEF_FN __device__ __forceinline__
#else
#define FEF_FN static inline
#endif

// d = (a - b) mod 2^256 with borrow 0 or all ones (a < b): folds bit 255 (19)
// and the borrow (-38) into limb 0 and returns true when that gives the
// canonical a - b.  Only a limb 0 within 64 of its ends can carry on or leave
// a negative value, and only a top limb of all ones can reach p: false (for
// random inputs below 2^-24), and d is of no use.
FEF_FN bool fef_fold(uint32_t d[8], uint32_t borrow) {
    const uint32_t top = d[7] >> 31;
    d[7] &= 0x7fffffffu;
    const bool rare = d[0] + 64u < 128u || d[7] == 0x7fffffffu;
    d[0] += top * 19u + borrow * 38u;
    return !rare;
}
