// Start points: multiples s Q of the fixed point Q = 8B (sm_100a).
//
// Q never changes, so s Q is a sum of 64 table entries, one per signed 4-bit
// digit of s, on the twisted Edwards form: a mixed addition takes 7 M, and its
// formulas hold for every pair of points.  The table (comb_table.cuh) has the
// multiples 1..8 of 256^i Q; the digits of odd weight are added first and
// raised by four doublings.  64 x 7 M + 16 M + 16 S + one inversion per start
// point, where a Montgomery ladder takes 253 x (5 M + 4 S) and its inversion.
//
// No address and no choice of an entry depends on a scalar: every digit reads
// all eight entries of its window, at one address per warp, from shared memory,
// and keeps one by selects (about a fifth of the addition's time).  What is
// left, as in a ladder on the same field functions, are their branches on a
// last carry, taken below 2^-21 of the time.
#pragma once
#include <cstdint>

#include "comb_table.cuh"
#include "walk_kernels.cuh"

namespace lxk {

constexpr int kCombThreads = 128;
constexpr int kCombVecs = 32 * 8 * 24 / 4;  // uint4 of the table (24 KB)
// A window's 48 uint4 at a stride of 49, so that threads at different windows
// read different banks.
constexpr int kCombStride = 49;
constexpr int kCombShared = 32 * kCombStride;

// Threads per scalar: one scalar's 64 additions and its inversion are a serial
// chain of 0.18 ms, so few scalars are split over up to 16 threads, which take
// every 16th window and add their sums up by shuffles, as long as every SM
// sub-partition has a warp at most (more would only repeat the inversion).
// 128 scalars on B200: 0.06 ms against 0.18; a serving turn that admits two
// searches 4.63 -> 4.51 ms.
inline uint32_t comb_threads(uint64_t scalars, uint32_t sms) {
    uint32_t t = 1;
    while (t < 16 && scalars * (2 * t) <= (uint64_t)sms * 128) t *= 2;
    return t;
}
inline unsigned comb_blocks(uint64_t scalars, uint32_t threads) {
    return (unsigned)((scalars * threads + kCombThreads - 1) / kCombThreads);
}

struct EdPoint {
    fe x, y, z, t;  // extended coordinates: x = X/Z, y = Y/Z, T = X Y / Z
};

// The table into shared memory; every thread of the block calls this.
__device__ __forceinline__ void comb_stage(uint4* table) {
    const uint4* src = reinterpret_cast<const uint4*>(kCombTable);
    for (int i = threadIdx.x; i < kCombVecs; i += blockDim.x) table[i / 48 * kCombStride + i % 48] = src[i];
    __syncthreads();
}

__device__ __forceinline__ fe comb_fe(const uint4* p) {
    const uint4 a = p[0], b = p[1];
    fe r;
    r.v[0] = a.x; r.v[1] = a.y; r.v[2] = a.z; r.v[3] = a.w;
    r.v[4] = b.x; r.v[5] = b.y; r.v[6] = b.z; r.v[7] = b.w;
    return r;
}

__device__ __forceinline__ fe fe_select(bool c, const fe& a, const fe& b) {
    fe r;
#pragma unroll
    for (int i = 0; i < 8; i++) r.v[i] = c ? a.v[i] : b.v[i];
    return r;
}

// p + digit * 256^i Q, -8 <= digit <= 7; window: the entries of 256^i.
__device__ __forceinline__ void comb_add(EdPoint& p, const uint4* window, int digit) {
    const bool neg = digit < 0;
    const int mag = neg ? -digit : digit;
    fe yx = fe_one(), xy = fe_one(), td = fe_zero();  // the neutral element
#pragma unroll 2
    for (int j = 1; j <= 8; j++) {
        const uint4* e = window + (j - 1) * 6;
        yx = fe_select(mag == j, comb_fe(e), yx);
        xy = fe_select(mag == j, comb_fe(e + 2), xy);
        td = fe_select(mag == j, comb_fe(e + 4), td);
    }
    // The negative of a point has y + x and y - x exchanged and -2 d x y,
    // which exchanges F and G.
    const fe A = fe_mul(fe_sub(p.y, p.x), fe_select(neg, yx, xy));
    const fe B = fe_mul(fe_add(p.y, p.x), fe_select(neg, xy, yx));
    const fe C = fe_mul(p.t, td);
    const fe D2 = fe_add(p.z, p.z);
    const fe f = fe_sub(D2, C), g = fe_add(D2, C);
    const fe E = fe_sub(B, A), H = fe_add(B, A);
    const fe F = fe_select(neg, g, f), G = fe_select(neg, f, g);
    p.x = fe_mul(E, F);
    p.y = fe_mul(G, H);
    p.t = fe_mul(E, H);
    p.z = fe_mul(F, G);
}

__device__ __forceinline__ void ed_double(EdPoint& p) {
    const fe a = fe_sqr(p.x), b = fe_sqr(p.y), zz = fe_sqr(p.z);
    const fe e = fe_sub(fe_sub(fe_sqr(fe_add(p.x, p.y)), a), b);
    const fe g = fe_sub(b, a);
    const fe f = fe_sub(g, fe_add(zz, zz));
    const fe h = fe_sub(fe_zero(), fe_add(a, b));
    p.x = fe_mul(e, f);
    p.y = fe_mul(g, h);
    p.t = fe_mul(e, h);
    p.z = fe_mul(f, g);
}

// p + q, both in extended coordinates (9 M).
__device__ __forceinline__ EdPoint ed_add(const EdPoint& p, const EdPoint& q) {
    constexpr uint32_t k2d[8] = LXK_COMB_2D;
    fe d2;
#pragma unroll
    for (int i = 0; i < 8; i++) d2.v[i] = k2d[i];
    const fe A = fe_mul(fe_sub(p.y, p.x), fe_sub(q.y, q.x));
    const fe B = fe_mul(fe_add(p.y, p.x), fe_add(q.y, q.x));
    const fe C = fe_mul(fe_mul(p.t, q.t), d2);
    const fe zz = fe_mul(p.z, q.z), D = fe_add(zz, zz);
    const fe E = fe_sub(B, A), F = fe_sub(D, C), G = fe_add(D, C), H = fe_add(B, A);
    return EdPoint{fe_mul(E, F), fe_mul(G, H), fe_mul(F, G), fe_mul(E, H)};
}

__device__ __forceinline__ fe shfl_xor_fe(const fe& x, int m) {
    fe r;
#pragma unroll
    for (int i = 0; i < 8; i++) r.v[i] = __shfl_xor_sync(0xffffffffu, x.v[i], m);
    return r;
}

// s Q for s <= 0x77...7, 64 sevens (8 little-endian words; above that the sum
// below leaves 256 bits; a clamped scalar over 8 and the group's half are below
// 2^252 + 2^10), by `threads` threads (a power of two; thread t takes the windows
// t, t + threads, ...): every one gets it.
__device__ __forceinline__ EdPoint comb_mul(const uint32_t s[8], const uint4* table, uint32_t t, uint32_t threads) {
    // s + 8 (1 + 16 + ... + 16^63): its nibbles less 8 are signed digits of s.
    uint32_t n[8], carry = 0;
#pragma unroll
    for (int w = 0; w < 8; w++) {
        const uint64_t x = (uint64_t)s[w] + 0x88888888u + carry;
        n[w] = (uint32_t)x;
        carry = (uint32_t)(x >> 32);
    }
    EdPoint p{fe_zero(), fe_one(), fe_one(), fe_zero()};
#pragma unroll 1
    for (int odd = 1; odd >= 0; odd--) {
#pragma unroll 1
        for (uint32_t i = t; i < 32; i += threads)
            comb_add(p, table + i * kCombStride, (int)(n[i >> 2] >> (8 * (i & 3) + 4 * odd) & 15u) - 8);
        if (odd) {
#pragma unroll 1
            for (int i = 0; i < 4; i++) ed_double(p);
        }
    }
#pragma unroll 1
    for (uint32_t m = 1; m < threads; m *= 2)
        p = ed_add(p, EdPoint{shfl_xor_fe(p.x, m), shfl_xor_fe(p.y, m), shfl_xor_fe(p.z, m), shfl_xor_fe(p.t, m)});
    return p;
}

// u = (Z + Y) / (Z - Y), v = c u / x = c (Z + Y) Z / ((Z - Y) X), affine and canonical.
__device__ __forceinline__ void ed_to_affine_uv(const EdPoint& p, fe& u, fe& v) {
    constexpr uint32_t kC[8] = LXK_COMB_C;
    fe c;
#pragma unroll
    for (int i = 0; i < 8; i++) c.v[i] = kC[i];
    const fe den = fe_sub(p.z, p.y);
    const fe t = fe_mul(fe_add(p.z, p.y), fe_invert(fe_mul(den, p.x)));
    u = fe_canon(fe_mul(t, p.x));
    v = fe_canon(fe_mul(fe_mul(t, p.z), c));
}

// The centre C = (k/8 + m) Q of lane k's first group (walk indices 0 .. 2m-1).
__device__ __forceinline__ void start_centre(const uint32_t* __restrict__ scalars, uint32_t i, uint32_t m,
                                             const uint4* table, uint32_t t, uint32_t threads, fe& u, fe& v) {
    uint32_t s[8];
    scalar_over_8(scalars, i, (int)m, s);
    ed_to_affine_uv(comb_mul(s, table, t, threads), u, v);
}

// The scalar of a thread and its place among the scalar's threads; the last
// block's spare threads repeat the last scalar (they take part in shuffles)
// and store nothing.
struct CombLane {
    uint32_t i, t;
    bool stores;
};
__device__ __forceinline__ CombLane comb_lane(uint32_t count, uint32_t threads) {
    const uint64_t id = blockIdx.x * (uint64_t)kCombThreads + threadIdx.x;
    const uint64_t i = id / threads;
    const uint32_t t = (uint32_t)(id % threads);
    return CombLane{i < count ? (uint32_t)i : count - 1, t, i < count && t == 0};
}

// Grouped walk from scalars.  75,776 lanes on B200: 0.47 ms, by the ladder 2.73; 128 lanes: 0.18 and 1.06.
static __global__ void __launch_bounds__(kCombThreads) group_start_kernel(uint32_t* state, uint64_t* ns,
                                                                          const uint32_t* __restrict__ scalars,
                                                                          uint32_t lanes, uint32_t m,
                                                                          uint32_t threads) {
    __shared__ uint4 table[kCombShared];
    comb_stage(table);
    const CombLane c = comb_lane(lanes, threads);
    const uint32_t lane = c.i;
    fe u, v;
    start_centre(scalars, lane, m, table, c.t, threads, u, v);
    if (!c.stores) return;
    store_fe(state, 0, lane, lanes, u);
    store_fe(state, 1, lane, lanes, v);
    ns[lane] = 0;
}

// P(-1) and P(0) of lane k, ((k - 8)B, kB), as u = X : Z.
__device__ __forceinline__ void start_pair(const uint32_t* __restrict__ scalars, uint32_t lane, const uint4* table,
                                           uint32_t t, uint32_t threads, fe& x0, fe& z0, fe& x1, fe& z1) {
    uint32_t s[8];
    scalar_over_8(scalars, lane, -1, s);
    EdPoint p = comb_mul(s, table, t, threads);
    x0 = fe_add(p.z, p.y);
    z0 = fe_sub(p.z, p.y);
    comb_add(p, table, 1);  // + Q
    x1 = fe_add(p.z, p.y);
    z1 = fe_sub(p.z, p.y);
}

// x-only walk from scalars, left projective (replacing the CPU start points
// of first_public_keys, mod.rs:212-228, for the walk).
static __global__ void __launch_bounds__(kCombThreads) xonly_start_kernel(uint32_t* state, uint64_t* ns,
                                                                          const uint32_t* __restrict__ scalars,
                                                                          uint32_t lanes, uint32_t threads) {
    __shared__ uint4 table[kCombShared];
    comb_stage(table);
    const CombLane c = comb_lane(lanes, threads);
    const uint32_t lane = c.i;
    fe x0, z0, x1, z1;
    start_pair(scalars, lane, table, c.t, threads, x0, z0, x1, z1);
    if (!c.stores) return;
    store_fe(state, 0, lane, lanes, x0);
    store_fe(state, 1, lane, lanes, z0);
    store_fe(state, 2, lane, lanes, x1);
    store_fe(state, 3, lane, lanes, z1);
    ns[lane] = 0;
}

// first_public_keys (mod.rs:212-228) on the GPU: u(k-8) and u(k) as 16
// canonical little-endian words per lane, the input of Backend::init.  One
// inversion of Z0 * Z1 serves both coordinates.  75,776 scalars: 0.47 ms, by
// the ladder 2.62.
static __global__ void __launch_bounds__(kCombThreads) first_keys_kernel(uint4* __restrict__ upc,
                                                                         const uint32_t* __restrict__ scalars,
                                                                         uint32_t lanes, uint32_t threads) {
    __shared__ uint4 table[kCombShared];
    comb_stage(table);
    const CombLane c = comb_lane(lanes, threads);
    const uint32_t lane = c.i;
    fe x0, z0, x1, z1;
    start_pair(scalars, lane, table, c.t, threads, x0, z0, x1, z1);
    if (!c.stores) return;
    const fe inv = fe_invert(fe_mul(z0, z1));
    const fe u_prev = fe_canon(fe_mul(x0, fe_mul(inv, z1)));
    const fe u_cur = fe_canon(fe_mul(x1, fe_mul(inv, z0)));
    uint4* out = upc + (size_t)lane * 4;
    out[0] = make_uint4(u_prev.v[0], u_prev.v[1], u_prev.v[2], u_prev.v[3]);
    out[1] = make_uint4(u_prev.v[4], u_prev.v[5], u_prev.v[6], u_prev.v[7]);
    out[2] = make_uint4(u_cur.v[0], u_cur.v[1], u_cur.v[2], u_cur.v[3]);
    out[3] = make_uint4(u_cur.v[4], u_cur.v[5], u_cur.v[6], u_cur.v[7]);
}

}  // namespace lxk
