// Inversion mod p = 2^255 - 19 by divsteps (Bernstein and Yang, "Fast
// constant-time gcd computation and modular inversion", CHES 2019), in the
// half-delta variant: zeta = -(delta + 1/2) from -1, for which 588 steps
// bring every 0 <= g < f < 2^255 to g = 0.  20 batches of 30 steps run
// always, so the time depends on no input.
//
// A batch runs 30 divsteps on the low 32 bits of f and g and collects them in
// a 2 x 2 matrix scaled by 2^30; the matrix is then applied to f, g (exact
// division by 2^30) and to d, e mod p, where d z = f and e z = g (mod p).
// Values are 9 signed limbs of 30 bits, so that a row of a product is a chain
// of 32 x 32 + 64 multiply-adds without carries.
//
// Fermat's chain (254 squares and 11 multiplies) takes about 63,000 cycles of
// an SM sub-partition per warp with four warps on it, and 42 us in a lone warp;
// this takes 24,000 cycles and 16 us on B200.  A step is seven multiply-adds and
// eight ALU operations, a batch's updates 76 wide multiply-adds.  The grouped
// walk at G = 64 goes from 4.53 to 4.91 G keys/s, the x-only walk at B = 64 from
// 3.71 to 3.94.  Unrolled 15 steps (3: 24,900 cycles; 6: 24,400; 30: 23,700, for
// twice the code).
//
// Plain C++ with one macro, so that a CPU build of the same code can be
// checked against integers.
#pragma once
#include <cstdint>

#ifdef __CUDACC__
#define FED_FN __device__ __forceinline__
#define FED_UNROLL _Pragma("unroll")
#define FED_NO_UNROLL _Pragma("unroll 1")
// x * y + z, kept a multiply-add: the compiler would turn factors of 0 and 1
// into selects on the ALU pipe.
FED_FN uint32_t fed_mad(uint32_t x, uint32_t y, uint32_t z) {
    uint32_t r;
    asm("mad.lo.u32 %0, %1, %2, %3;" : "=r"(r) : "r"(x), "r"(y), "r"(z));
    return r;
}
// -(x & 1)
FED_FN uint32_t fed_low_bit_mask(uint32_t x) {
    int32_t r;
    asm("bfe.s32 %0, %1, 0, 1;" : "=r"(r) : "r"(x));
    return (uint32_t)r;
}
#else
#define FED_FN static inline
#define FED_UNROLL
#define FED_NO_UNROLL
FED_FN uint32_t fed_mad(uint32_t x, uint32_t y, uint32_t z) { return x * y + z; }
FED_FN uint32_t fed_low_bit_mask(uint32_t x) { return 0u - (x & 1u); }
#endif

constexpr int kFedLimbs = 9;
constexpr uint32_t kFedMask = (1u << 30) - 1;
constexpr uint32_t kFedPInv = 0x179435e5u;  // p^-1 mod 2^30
constexpr int kFedBatches = 20;

// 30 divsteps on the low words of f and g: the matrix (u v; q r) and the new
// zeta.  The first row (nf, nu, nv) is kept negated, so that both updates
// multiply by a mask or a sum of masks.
FED_FN int32_t fed_steps(int32_t zeta, uint32_t f, uint32_t g, int32_t m[4]) {
    uint32_t nf = 0u - f, nu = 0xffffffffu, nv = 0, q = 0, r = 1;
    FED_NO_UNROLL
    for (int i = 0; i < 2; i++) {
        FED_UNROLL
        for (int j = 0; j < 15; j++) {
            // g odd: add f, or subtract it when delta > 0 and then swap.
            const uint32_t odd = fed_low_bit_mask(g);                // 0 or -1
            const uint32_t swap = odd & (uint32_t)(zeta >> 31);      // 0 or -1
            const uint32_t sign = fed_mad(swap, 0xfffffffeu, odd);   // 0, -1 (add f) or 1 (subtract f)
            g = fed_mad(nf, sign, g);
            q = fed_mad(nu, sign, q);
            r = fed_mad(nv, sign, r);
            zeta = (int32_t)(((uint32_t)zeta ^ swap) - 1u);
            nf = fed_mad(g, swap, nf);
            nu = fed_mad(q, swap, nu);
            nv = fed_mad(r, swap, nv);
            g >>= 1;
            nu += nu;
            nv += nv;
        }
    }
    m[0] = (int32_t)(0u - nu);
    m[1] = (int32_t)(0u - nv);
    m[2] = (int32_t)q;
    m[3] = (int32_t)r;
    return zeta;
}

// f, g <- (u f + v g) / 2^30, (q f + r g) / 2^30, both exact.
FED_FN void fed_update_fg(int32_t f[9], int32_t g[9], const int32_t m[4]) {
    int64_t cf = (int64_t)m[0] * f[0] + (int64_t)m[1] * g[0];
    int64_t cg = (int64_t)m[2] * f[0] + (int64_t)m[3] * g[0];
    cf >>= 30;
    cg >>= 30;
    FED_UNROLL
    for (int i = 1; i < kFedLimbs; i++) {
        cf += (int64_t)m[0] * f[i] + (int64_t)m[1] * g[i];
        cg += (int64_t)m[2] * f[i] + (int64_t)m[3] * g[i];
        f[i - 1] = (int32_t)((uint32_t)cf & kFedMask);
        g[i - 1] = (int32_t)((uint32_t)cg & kFedMask);
        cf >>= 30;
        cg >>= 30;
    }
    f[8] = (int32_t)cf;
    g[8] = (int32_t)cg;
}

// d, e <- (u d + v e) / 2^30, (q d + r e) / 2^30 mod p, kept in (-2p, p): a
// multiple of p (limbs -19, 0, ..., 0, 2^15) makes the low 30 bits zero.
FED_FN void fed_update_de(int32_t d[9], int32_t e[9], const int32_t m[4]) {
    const int32_t sd = d[8] >> 31, se = e[8] >> 31;
    int32_t md = (m[0] & sd) + (m[1] & se), me = (m[2] & sd) + (m[3] & se);
    int64_t cd = (int64_t)m[0] * d[0] + (int64_t)m[1] * e[0];
    int64_t ce = (int64_t)m[2] * d[0] + (int64_t)m[3] * e[0];
    md -= (int32_t)((kFedPInv * (uint32_t)cd + (uint32_t)md) & kFedMask);
    me -= (int32_t)((kFedPInv * (uint32_t)ce + (uint32_t)me) & kFedMask);
    cd += (int64_t)md * -19;
    ce += (int64_t)me * -19;
    cd >>= 30;
    ce >>= 30;
    FED_UNROLL
    for (int i = 1; i < kFedLimbs; i++) {
        cd += (int64_t)m[0] * d[i] + (int64_t)m[1] * e[i];
        ce += (int64_t)m[2] * d[i] + (int64_t)m[3] * e[i];
        if (i == 8) {
            cd += (int64_t)md * 32768;
            ce += (int64_t)me * 32768;
        }
        d[i - 1] = (int32_t)((uint32_t)cd & kFedMask);
        e[i - 1] = (int32_t)((uint32_t)ce & kFedMask);
        cd >>= 30;
        ce >>= 30;
    }
    d[8] = (int32_t)cd;
    e[8] = (int32_t)ce;
}

// d += p where d is negative, with the limbs carried.
FED_FN void fed_add_p_if_negative(int32_t d[9]) {
    const int32_t neg = d[8] >> 31;
    d[0] += neg & -19;
    d[8] += neg & 32768;
    FED_UNROLL
    for (int i = 0; i < 8; i++) {
        d[i + 1] += d[i] >> 30;
        d[i] &= (int32_t)kFedMask;
    }
}

// z^-1 mod p of a canonical z (8 little-endian words), canonical; 0 for 0.
FED_FN void fed_invert(const uint32_t z[8], uint32_t out[8]) {
    int32_t f[9], g[9], d[9], e[9];
    FED_UNROLL
    for (int i = 0; i < kFedLimbs; i++) {
        const int w = 30 * i / 32, s = 30 * i % 32;
        uint32_t x = z[w] >> s;
        if (s > 2 && w < 7) x |= z[w + 1] << (32 - s);
        g[i] = (int32_t)(x & kFedMask);
        f[i] = i == 0 ? -19 : i == 8 ? 32768 : 0;
        d[i] = 0;
        e[i] = i == 0 ? 1 : 0;
    }
    int32_t zeta = -1;
    FED_NO_UNROLL
    for (int b = 0; b < kFedBatches; b++) {
        int32_t m[4];
        // Step j reads bits 0..j of f and g, so limb 0 (30 bits) is enough.
        zeta = fed_steps(zeta, (uint32_t)f[0], (uint32_t)g[0], m);
        fed_update_de(d, e, m);
        fed_update_fg(f, g, m);
    }
    // f = +-1 (or p, with d = 0, for z = 0): z^-1 = d f.
    fed_add_p_if_negative(d);
    const int32_t flip = f[8] >> 31;
    FED_UNROLL
    for (int i = 0; i < kFedLimbs; i++) d[i] = (d[i] ^ flip) - flip;
    FED_UNROLL
    for (int i = 0; i < 8; i++) {
        d[i + 1] += d[i] >> 30;
        d[i] &= (int32_t)kFedMask;
    }
    fed_add_p_if_negative(d);
    FED_UNROLL
    for (int w = 0; w < 8; w++) {
        const int i = 32 * w / 30, s = 32 * w % 30;
        out[w] = (uint32_t)d[i] >> s | (uint32_t)d[i + 1] << (30 - s);
    }
}
