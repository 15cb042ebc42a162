// Batch inversion by Montgomery's trick, a group per one or several threads
// (the array entry points; the walks have their own).
#pragma once
#include <cstdint>

#include "fe25519.cuh"

namespace lxk {

// 8 words with bit 255 dropped, as the reference's fe_from_words reads them
// (common.h:131-142).
__device__ __forceinline__ fe load_words_drop255(const uint32_t* p) {
    fe r;
    const uint4* p4 = reinterpret_cast<const uint4*>(p);
    const uint4 lo = p4[0], hi = p4[1];
    r.v[0] = lo.x; r.v[1] = lo.y; r.v[2] = lo.z; r.v[3] = lo.w;
    r.v[4] = hi.x; r.v[5] = hi.y; r.v[6] = hi.z; r.v[7] = hi.w & 0x7fffffffu;
    return r;
}

__device__ __forceinline__ void store_words(uint32_t* p, const fe& x) {
    uint4* p4 = reinterpret_cast<uint4*>(p);
    p4[0] = make_uint4(x.v[0], x.v[1], x.v[2], x.v[3]);
    p4[1] = make_uint4(x.v[4], x.v[5], x.v[6], x.v[7]);
}

__device__ __forceinline__ fe shfl_up_fe(const fe& x, int d, int width) {
    fe r;
#pragma unroll
    for (int i = 0; i < 8; i++) r.v[i] = __shfl_up_sync(0xffffffffu, x.v[i], d, width);
    return r;
}

__device__ __forceinline__ fe shfl_down_fe(const fe& x, int d, int width) {
    fe r;
#pragma unroll
    for (int i = 0; i < 8; i++) r.v[i] = __shfl_down_sync(0xffffffffu, x.v[i], d, width);
    return r;
}

constexpr int kInvertThreads = 128;

// Threads per group: a power of two up to 32 and the group, as long as the
// device has an idle SM sub-partition for the next doubling.  An inversion
// takes 15 us however long the groups are, so more warps than one per
// sub-partition would only repeat it (a second one makes it 23 us).
inline uint32_t invert_threads(uint64_t groups, uint32_t group, uint32_t sms) {
    uint32_t t = 1;
    while (t < 32 && 2 * t <= group && groups * (2 * t) <= (uint64_t)sms * 128) t *= 2;
    return t;
}

// The inverse of every element of `a`, in groups of `group` consecutive ones
// that share an inversion (so a zero makes its whole group zero).  T threads
// (a power of two up to 32) take a group's elements in runs: each multiplies
// its run up, prefix and suffix products over the T lanes give every thread
// the product of the others, and the group's inverse times that is its run's.
// Prefix products go to `scratch`; it may be `out` unless `out` is `a`.  A
// thread touches its own run only, and reads an element before its inverse is
// stored, so `out` may be `a`.
// 131,072 elements in groups of 64 on B200: 33 us with 8 threads per group, 113
// with one, whose 192 multiplies in a row outlast the inversion.
static __global__ void __launch_bounds__(kInvertThreads) batch_invert_kernel(const uint32_t* a, uint32_t* out,
                                                                             uint32_t* scratch, uint64_t count,
                                                                             uint32_t group, uint32_t threads) {
    const uint64_t id = blockIdx.x * (uint64_t)kInvertThreads + threadIdx.x;
    const uint64_t base = id / threads * group;  // past the last group: an empty run, for the shuffles
    const uint32_t t = (uint32_t)(id % threads);
    const uint32_t len = base >= count ? 0 : count - base < group ? (uint32_t)(count - base) : group;
    const uint32_t lo = len * t / threads, hi = len * (t + 1) / threads;
    fe acc = fe_one();
#pragma unroll 1
    for (uint32_t i = lo; i < hi; i++) {
        store_words(scratch + 8 * (base + i), acc);
        acc = fe_mul(acc, load_words_drop255(a + 8 * (base + i)));
    }
    // Products of the runs before (and with) this one, and from this one on.
    fe before = acc, after = acc;
#pragma unroll 1
    for (uint32_t d = 1; d < threads; d *= 2) {
        const fe x = fe_mul(before, shfl_up_fe(before, d, threads));
        const fe y = fe_mul(after, shfl_down_fe(after, d, threads));
        if (t >= d) before = x;
        if (t + d < threads) after = y;
    }
    fe total;
#pragma unroll
    for (int i = 0; i < 8; i++) total.v[i] = __shfl_sync(0xffffffffu, before.v[i], threads - 1, threads);
    fe inv = fe_invert(total);
    if (threads > 1) {
        const fe x = shfl_up_fe(before, 1, threads), y = shfl_down_fe(after, 1, threads);
        if (t > 0) inv = fe_mul(inv, x);
        if (t + 1 < threads) inv = fe_mul(inv, y);
    }
#pragma unroll 1
    for (uint32_t i = hi; i-- > lo;) {
        const fe x = load_words_drop255(a + 8 * (base + i));
        const uint4* p4 = reinterpret_cast<const uint4*>(scratch + 8 * (base + i));
        const uint4 l = p4[0], h = p4[1];
        const fe pre{{l.x, l.y, l.z, l.w, h.x, h.y, h.z, h.w}};
        store_words(out + 8 * (base + i), fe_canon(fe_mul(inv, pre)));
        inv = fe_mul(inv, x);
    }
}

}  // namespace lxk
