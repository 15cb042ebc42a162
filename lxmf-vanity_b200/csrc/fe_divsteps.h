// Inversion mod p = 2^255 - 19 by divsteps (Bernstein and Yang, "Fast
// constant-time gcd computation and modular inversion", CHES 2019): steps on
// the low words of f = p and g = z, collected in 2 x 2 matrices that are then
// applied to f, g and, mod p, to d, e.  The paper starts at delta = 1; from
// delta = 1/2 (Pieter Wuille's variant; zeta = -(delta + 1/2) here) 590 steps
// bring 256-bit inputs to g = 0.  20 batches of 30 run always.
//
// A batch runs 30 divsteps on the low 32 bits of f and g and collects them in
// a matrix scaled by 2^30.  f and g are two's complement numbers of 8 words,
// divided exactly by 2^30 after each batch; d and e are residues in the
// field's own form, 8 words with 2^256 = 38, never divided: the power of two
// that they gather is known beforehand and taken out of e's first value.
//
// Fermat's chain (254 squares and 11 multiplies) takes about 63,000 cycles of
// an SM sub-partition per warp with four warps on it, and 42 us in a lone warp;
// this takes 22,100 cycles and 15 us on B200.  A step is seven multiply-adds and
// eight ALU operations, a batch's updates 64 wide multiply-adds.  The grouped
// walk at G = 64 goes from 4.53 to 4.96 G keys/s, the x-only walk at B = 64 from
// 3.71 to 3.96.  All four values on 30-bit limbs, d and e divided by 2^30 too
// (76 wide multiply-adds, masks and 64-bit shifts for every limb): 24,200 cycles
// and 16.3 us, 4.92 and 3.93 G keys/s.  Unrolled 15 steps; with 30-bit limbs 3 took
// 24,900 cycles, 6 24,400 and 30 23,700, for twice the code.
//
// Plain C++ with a few macros, so that a CPU build of the same code can be
// checked against integers.
#pragma once
#include <cstdint>

#ifdef __CUDACC__
#define FED_FN __device__ __forceinline__
#define FED_MEMBER __device__ __forceinline__
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
#define FED_MEMBER
#define FED_UNROLL
#define FED_NO_UNROLL
FED_FN uint32_t fed_mad(uint32_t x, uint32_t y, uint32_t z) { return x * y + z; }
FED_FN uint32_t fed_low_bit_mask(uint32_t x) { return 0u - (x & 1u); }
#endif

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

// A row of the matrix, a x + b y with |a| + |b| <= 2^30: the magnitudes, and
// all ones where a factor is negative and its operand is complemented.  With
// that every product of two words is below 2^62 and a word's sum stays in 63
// bits, and nothing is negated: what a complement is off by is a constant
// times its factor, added at the bottom word.
struct FedRow {
    uint32_t a, b, ma, mb;
    FED_MEMBER uint64_t at(uint32_t x, uint32_t y) const { return (uint64_t)a * (x ^ ma) + (uint64_t)b * (y ^ mb); }
    FED_MEMBER int64_t at_top(uint32_t x, uint32_t y) const {
        return (int64_t)(int32_t)a * (int32_t)(x ^ ma) + (int64_t)(int32_t)b * (int32_t)(y ^ mb);
    }
    FED_MEMBER uint32_t complements() const { return (a & ma) + (b & mb); }
};
FED_FN FedRow fed_row(int32_t a, int32_t b) {
    const uint32_t ma = (uint32_t)(a >> 31), mb = (uint32_t)(b >> 31);
    return FedRow{((uint32_t)a ^ ma) - ma, ((uint32_t)b ^ mb) - mb, ma, mb};
}

// f, g <- both rows of (f, g) / 2^30, exact divisions of 256-bit two's
// complement numbers: -x = ~x + 1, so a complement adds its factor once.  The
// top words carry the signs.  |f|, |g| < 2^255 hold through every step.
FED_FN void fed_apply_fg(uint32_t f[8], uint32_t g[8], const FedRow& up, const FedRow& down) {
    uint64_t sf = up.complements(), sg = down.complements();
    uint32_t pf = 0, pg = 0;  // the words before this one, not yet shifted
    FED_UNROLL
    for (int k = 0; k < 7; k++) {
        sf += up.at(f[k], g[k]);
        sg += down.at(f[k], g[k]);
        if (k) {
            f[k - 1] = pf >> 30 | (uint32_t)sf << 2;
            g[k - 1] = pg >> 30 | (uint32_t)sg << 2;
        }
        pf = (uint32_t)sf;
        pg = (uint32_t)sg;
        sf >>= 32;
        sg >>= 32;
    }
    const int64_t tf = (int64_t)sf + up.at_top(f[7], g[7]), tg = (int64_t)sg + down.at_top(f[7], g[7]);
    f[6] = pf >> 30 | (uint32_t)tf << 2;
    g[6] = pg >> 30 | (uint32_t)tg << 2;
    f[7] = (uint32_t)(tf >> 30);
    g[7] = (uint32_t)(tg >> 30);
}

// A residue mod p: 256 bits and a carry of -1, 0 or 1 at 2^64 that the next
// row takes in, in place of a chain through six more words.
struct FedResidue {
    uint32_t w[8];
    int32_t c;
};

// x's words are in place and `above` is what is left at 2^256 = 38: it goes
// into the lowest two words and the pending carry.
FED_FN void fed_fold(FedResidue& x, int64_t above) {
    const uint64_t low = (uint64_t)x.w[1] << 32 | x.w[0], sum = low + (uint64_t)(38 * above);
    x.w[0] = (uint32_t)sum;
    x.w[1] = (uint32_t)(sum >> 32);
    x.c = (int32_t)(sum < low) + (int32_t)(above >> 63);
}

// d, e <- both rows of (d, e) mod p; m: the rows' signed factors.  2^256 = 38,
// so ~x = 37 - x (mod p), and a complement takes 37 times its factor back.
FED_FN void fed_apply_de(FedResidue& d, FedResidue& e, const FedRow& up, const FedRow& down, const int32_t m[4]) {
    int64_t sd = -37 * (int64_t)up.complements(), se = -37 * (int64_t)down.complements();
    FED_UNROLL
    for (int k = 0; k < 8; k++) {
        sd += (int64_t)up.at(d.w[k], e.w[k]);
        se += (int64_t)down.at(d.w[k], e.w[k]);
        if (k == 2) {
            sd += m[0] * d.c + m[1] * e.c;
            se += m[2] * d.c + m[3] * e.c;
        }
        d.w[k] = (uint32_t)sd;
        e.w[k] = (uint32_t)se;
        sd >>= 32;
        se >>= 32;
    }
    fed_fold(d, sd);
    fed_fold(e, se);
}

// x + add + c2 2^64 in place; the carry out of 2^256.
FED_FN int32_t fed_carry(uint32_t x[8], int32_t add, int32_t c2) {
    int64_t acc = add;
    FED_UNROLL
    for (int k = 0; k < 8; k++) {
        acc += (int64_t)x[k] + (k == 2 ? c2 : 0);
        x[k] = (uint32_t)acc;
        acc >>= 32;
    }
    return (int32_t)acc;
}

// z^-1 mod p of a canonical z (8 little-endian words), canonical; 0 for 0.
// d z = f and e z = g (mod p) up to the power of two that the divisions of f
// and g take out; e starts at 2^-600, so that none is left at the end.
FED_FN void fed_invert(const uint32_t z[8], uint32_t out[8]) {
    constexpr uint32_t kStart[8] = {0x88dd407eu, 0x65683e67u, 0xcfc744c9u, 0x90aa31a3u,
                                    0x4e016b14u, 0x855b1b22u, 0x2c905dc1u, 0x4469d942u};  // 2^-600 mod p
    uint32_t f[8], g[8];
    FedResidue d, e;
    FED_UNROLL
    for (int k = 0; k < 8; k++) {
        f[k] = k == 0 ? 0xffffffedu : k == 7 ? 0x7fffffffu : 0xffffffffu;
        g[k] = z[k];
        d.w[k] = 0;
        e.w[k] = kStart[k];
    }
    d.c = e.c = 0;
    int32_t zeta = -1;
    FED_NO_UNROLL
    for (int i = 0; i < kFedBatches; i++) {
        int32_t m[4];
        zeta = fed_steps(zeta, f[0], g[0], m);  // step j reads bits 0..j of f and g
        const FedRow up = fed_row(m[0], m[1]), down = fed_row(m[2], m[3]);
        fed_apply_de(d, e, up, down, m);
        fed_apply_fg(f, g, up, down);
    }
    // f = 1 or -1 (or p, with d = 0, for z = 0): z^-1 = d f, by ~d - 37 = -d.
    const int32_t neg = (int32_t)f[7] >> 31;
    FED_UNROLL
    for (int k = 0; k < 8; k++) d.w[k] ^= (uint32_t)neg;
    int32_t c = fed_carry(d.w, neg & -37, (d.c ^ neg) - neg);
    // d + 2^256 c, c in -1..1: all above 2^255 folds in (2^255 = 19), which
    // leaves -38 < d < 2^255 + 57; then p is added once where d < 0 and taken
    // off where d + 19 reaches 2^255.
    const int32_t high = (int32_t)(d.w[7] >> 31) + 2 * c;
    d.w[7] &= 0x7fffffffu;
    c = fed_carry(d.w, 19 * high, 0);
    d.w[7] += (uint32_t)c & 0x80000000u;
    fed_carry(d.w, c & -19, 0);
    uint32_t less[8];
    FED_UNROLL
    for (int k = 0; k < 8; k++) less[k] = d.w[k];
    fed_carry(less, 19, 0);
    const uint32_t keep = (less[7] >> 31) - 1u;  // all ones where d < p
    less[7] &= 0x7fffffffu;
    FED_UNROLL
    for (int k = 0; k < 8; k++) out[k] = less[k] ^ ((less[k] ^ d.w[k]) & keep);
}
