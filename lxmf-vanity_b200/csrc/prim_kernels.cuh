// Primitive kernels: the field and hash microbench, and the integer-pipe
// throughput probes that give the roofline its denominators.
#pragma once
#include <cstdint>

#include "batch_invert.cuh"
#include "fe25519.cuh"
#include "sha256_lxmf.cuh"

namespace lxk {

static __global__ void fe_op_kernel(int op, const uint32_t* __restrict__ a, const uint32_t* __restrict__ b,
                             uint32_t* __restrict__ out, uint64_t count) {
    for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < count; i += (uint64_t)gridDim.x * blockDim.x) {
        const fe x = load_words_drop255(a + 8 * i);
        fe r;
        if (op == 0) r = fe_mul(x, load_words_drop255(b + 8 * i));
        else if (op == 1) r = fe_sqr(x);
        else r = fe_invert(x);
        store_words(out + 8 * i, fe_canon(r));
    }
}

// Destination hashes of whole 64-byte public keys (both halves per element).
static __global__ void address_chain_kernel(const uint32_t* __restrict__ pk, lxsha::AddrConsts ac, uint32_t* __restrict__ out,
                                     uint64_t count) {
    for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < count; i += (uint64_t)gridDim.x * blockDim.x) {
        uint32_t u[8], hi[8], d[4];
#pragma unroll
        for (int w = 0; w < 8; w++) {
            u[w] = pk[16 * i + w];
            hi[w] = __byte_perm(pk[16 * i + 8 + w], 0, 0x0123);
        }
        lxsha::dest_hash(u, hi, ac, d);
        // Back to bytes in hash order: big-endian words.
#pragma unroll
        for (int w = 0; w < 4; w++) out[4 * i + w] = __byte_perm(d[w], 0, 0x0123);
    }
}

// Each thread runs 8 independent dependency chains of one instruction class
// so that issue, not latency, is the limit; `sink` keeps the work alive.
// Operations counted per step and chain: kinds 2 and 5 issue two.
//   0 mad.lo.u32   1 mad.hi.u32   2 xor + shf   3 mad.wide.u32 (64-bit addend)
//   4 add.u32      5 mad.lo + xor (two pipes)   6 shf only   7 xor only
static __global__ void __launch_bounds__(256) probe_kernel(int kind, uint32_t iters, uint32_t seed, uint32_t* sink) {
    uint32_t x[8], y[8];
#pragma unroll
    for (int j = 0; j < 8; j++) {
        x[j] = seed + threadIdx.x * 8 + j;
        y[j] = x[j] ^ 0x55555555u;
    }
    const uint32_t m = seed | 1u, c = seed ^ 0x9e3779b9u;
#define LXK_PROBE(BODY)                                   \
    _Pragma("unroll 1") for (uint32_t i = 0; i < iters; i++) { \
        _Pragma("unroll") for (int r = 0; r < 16; r++) {   \
            _Pragma("unroll") for (int j = 0; j < 8; j++) { BODY; } \
        }                                                  \
    }
    switch (kind) {
        case 0: LXK_PROBE(asm volatile("mad.lo.u32 %0, %0, %1, %2;" : "+r"(x[j]) : "r"(m), "r"(c))) break;
        case 1: LXK_PROBE(asm volatile("mad.hi.u32 %0, %0, %1, %2;" : "+r"(x[j]) : "r"(m), "r"(c))) break;
        case 2:
            LXK_PROBE(asm volatile("xor.b32 %0, %0, %1;" : "+r"(x[j]) : "r"(c));
                      asm volatile("shf.r.wrap.b32 %0, %0, %0, 7;" : "+r"(x[j])))
            break;
        case 3:
            LXK_PROBE(asm volatile("{.reg .u64 t; mov.b64 t, {%0, %1}; mad.wide.u32 t, %0, %2, t; mov.b64 {%0, %1}, t;}"
                                   : "+r"(x[j]), "+r"(y[j]) : "r"(m)))
            break;
        // The neighbour operand keeps ptxas from folding repeated ops on one constant.
        case 4: LXK_PROBE(asm volatile("add.u32 %0, %0, %1;" : "+r"(x[j]) : "r"(x[(j + 1) & 7]))) break;
        case 5:
            LXK_PROBE(asm volatile("mad.lo.u32 %0, %0, %1, %2;" : "+r"(x[j]) : "r"(m), "r"(c));
                      asm volatile("xor.b32 %0, %0, %1;" : "+r"(y[j]) : "r"(y[(j + 1) & 7])))
            break;
        case 6: LXK_PROBE(asm volatile("shf.r.wrap.b32 %0, %0, %0, 7;" : "+r"(x[j]))) break;
        default: LXK_PROBE(asm volatile("xor.b32 %0, %0, %1;" : "+r"(x[j]) : "r"(x[(j + 1) & 7]))) break;
    }
#undef LXK_PROBE
    uint32_t acc = 0;
#pragma unroll
    for (int j = 0; j < 8; j++) acc ^= x[j] ^ y[j];
    if (acc == 0x12345678u) sink[0] = acc;
}

}  // namespace lxk
