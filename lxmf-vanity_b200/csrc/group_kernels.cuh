// The grouped affine walk (sm_100a): the same keys as the x-only walk, with
// about half the field work per key.
//
// Curve25519 in Montgomery form, v^2 = u^3 + A u^2 + u, A = 486662.  Every
// point here is a multiple of Q = 8B, with v(Q) fixed to the even square
// root, so a lane's key with walk index n is the point (k/8 + n) Q and its
// public key is that point's u.  A group is G = 2M keys: walk indices
// c-M .. c+M-1 around a centre C = (k/8 + c) Q kept affine (u_C, v_C):
//
//   key c +- i  =  C +- T_i,  T_i = i Q from a table (i = 1..M),
//   affine addition:  l = (v_T -+ v_C) / (u_T - u_C),  u = l^2 - A - u_C - u_T.
//
// C + T_i and C - T_i share the denominator u_T - u_C, so one batch inversion
// (Montgomery's trick) over the M denominators and the step to the next
// centre, C' = C + J with J = 2M Q, serves all 2M keys.  Per group:
// (5M + 2) M + (2M + 1) S and one inversion, about 2.5 M + 1 S per key,
// against 8 M + 4 S for the x-only walk (G = B = 128).  The lane's local
// buffer holds only the M prefix products (the denominators are recomputed
// from the table on the way back).
//
// Lane state in HBM: u_C, v_C (2 x 32 bytes, word-major) and the walk index
// of the group's first key.
#pragma once
#include <cstdint>
#include <type_traits>

#include "walk_kernels.cuh"

namespace lxk {

// 2A, for the y-coordinate recovery.
#define LXK_TWO_A 973324u
#define LXK_A 486662u

template <int M>
struct GroupTable {
    fe u[M + 1];  // [0]: J = 2M Q; [i]: i Q
    fe v[M + 1];
};

template <int M>
struct GroupArgs {
    uint32_t* state;  // [16][lanes]: u_C, v_C
    uint64_t* ns;     // [lanes]: walk index of the first key of the lane's next group (centre - M)
    uint32_t lanes;
    uint32_t iters;   // groups per lane in this launch
    uint32_t parts;   // warps per 32 lanes (group_parts_kernel)
    uint32_t* done;   // [lanes / 32]: warps that have finished their part; zero between launches
    const uint4* first_words;  // [M / 4]: the first words of u of 1Q .. MQ (walks in parts from any start points)
    EmitArgs em;
    GroupTable<M> t;
};

// G = 1024 (M = 512): the table (2 x 513 points, 33 KB) no longer fits the
// kernel parameter block (32 KB), so it lives in constant memory, where the
// warps read it through the same constant cache.  It depends on nothing but
// M, so every handle on a device shares it; lxmfv_open writes it there.
constexpr int kConstTableM = 512;
static __device__ __constant__ fe c_group_u[kConstTableM + 1];
static __device__ __constant__ fe c_group_v[kConstTableM + 1];
struct ConstTableU {
    __device__ __forceinline__ fe operator[](int i) const { return c_group_u[i]; }
};
struct ConstTableV {
    __device__ __forceinline__ fe operator[](int i) const { return c_group_v[i]; }
};
struct ConstGroupTable {
    ConstTableU u;
    ConstTableV v;
};
struct GroupArgsConst {
    uint32_t* state;
    uint64_t* ns;
    uint32_t lanes;
    uint32_t iters;
    uint32_t parts;
    uint32_t* done;
    const uint4* first_words;
    EmitArgs em;
};
template <int M>
__device__ __forceinline__ const GroupTable<M>& table_of(const GroupArgs<M>& a) { return a.t; }
__device__ __forceinline__ ConstGroupTable table_of(const GroupArgsConst&) { return ConstGroupTable{}; }
// The launch parameters of the grouped walk at M: the table travels in them
// up to M = 256, and sits in constant memory above.
template <int M>
using GroupArgsFor = typename std::conditional<(M > 256), GroupArgsConst, GroupArgs<M>>::type;

// y-coordinate recovery on a Montgomery curve (Okeya and Sakurai, CHES 2001;
// the form of Costello and Smith, "Montgomery curves and their arithmetic",
// Algorithm 5): from P = (xp, yp) affine, (X1:Z1) = sP and (X2:Z2) = (s+1)P,
// the projective (X:Y:Z) of sP.
__device__ __forceinline__ void recover_y(const fe& xp, const fe& yp, const fe& X1, const fe& Z1, const fe& X2,
                                          const fe& Z2, fe& X, fe& Y, fe& Z) {
    fe v1 = fe_mul(xp, Z1);
    fe v2 = fe_add(X1, v1);
    fe v3 = fe_sub(X1, v1);
    v3 = fe_mul(fe_sqr(v3), X2);
    v1 = fe_mul_small(Z1, LXK_TWO_A);
    v2 = fe_add(v2, v1);
    const fe v4 = fe_add(fe_mul(xp, X1), Z1);
    v2 = fe_mul(v2, v4);
    v1 = fe_mul(v1, Z1);
    v2 = fe_mul(fe_sub(v2, v1), Z2);
    Y = fe_sub(v2, v3);
    v1 = fe_mul(fe_mul(fe_add(yp, yp), Z1), Z2);
    X = fe_mul(v1, X1);
    Z = fe_mul(v1, Z1);
}

__device__ __forceinline__ void to_affine(const fe& X, const fe& Y, const fe& Z, fe& u, fe& v) {
    const fe zi = fe_invert(Z);
    u = fe_canon(fe_mul(X, zi));
    v = fe_canon(fe_mul(Y, zi));
}

// The table: thread i computes i Q (i = 1..M) and thread 0 computes J = 2M Q,
// affine and canonical, into tu / tv ([M + 1] each).
static __global__ void __launch_bounds__(32) group_table_kernel(fe* tu, fe* tv, uint32_t m, fe q, fe vq) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i > m) return;
    uint32_t s[8] = {i == 0 ? 2 * m : i, 0, 0, 0, 0, 0, 0, 0};
    fe x2, z2, x3, z3, X, Y, Z;
    ladder(s, 11, q, x2, z2, x3, z3);  // 2M <= 1024
    recover_y(q, vq, x2, z2, x3, z3, X, Y, Z);
    to_affine(X, Y, Z, tu[i], tv[i]);
}

// Start from Backend::init's u(k-8), u(k): y of P = kB = (k/8) Q is recovered
// with -Q (P - Q is known, not P + Q), then C = P + T_M (tm = M Q).
static __global__ void __launch_bounds__(128) group_init_kernel(uint32_t* state, uint64_t* ns,
                                                         const uint32_t* __restrict__ upc, uint32_t lanes, fe q,
                                                         fe vq_neg, fe tmu, fe tmv) {
    const uint32_t lane = blockIdx.x * blockDim.x + threadIdx.x;
    if (lane >= lanes) return;
    fe um8, uk;
#pragma unroll
    for (int w = 0; w < 8; w++) {
        um8.v[w] = upc[(size_t)lane * 16 + w];
        uk.v[w] = upc[(size_t)lane * 16 + 8 + w];
    }
    um8.v[7] &= 0x7fffffffu;
    uk.v[7] &= 0x7fffffffu;
    fe X, Y, Z, pu, pv;
    recover_y(q, vq_neg, uk, fe_one(), um8, fe_one(), X, Y, Z);
    to_affine(X, Y, Z, pu, pv);
    fe cA = fe_zero();
    cA.v[0] = LXK_A;
    const fe l = fe_mul(fe_sub(tmv, pv), fe_invert(fe_sub(tmu, pu)));
    const fe u = fe_canon(fe_sub(fe_sqr(l), fe_add(fe_add(pu, tmu), cA)));
    const fe v = fe_canon(fe_sub(fe_mul(l, fe_sub(pu, u)), pv));
    store_fe(state, 0, lane, lanes, u);
    store_fe(state, 1, lane, lanes, v);
    ns[lane] = 0;
}

// One field element per thread in shared memory, out of the registers' way.
// The load is volatile: it stays where it is used.
template <int BLOCK>
__device__ __forceinline__ void park_fe(uint4* at, const fe& x) {
    at[0] = make_uint4(x.v[0], x.v[1], x.v[2], x.v[3]);
    at[BLOCK] = make_uint4(x.v[4], x.v[5], x.v[6], x.v[7]);
}
template <int BLOCK>
__device__ __forceinline__ fe parked_fe(const uint4* at) {
    const uint32_t p = (uint32_t)__cvta_generic_to_shared(at);
    fe r;
    asm volatile("ld.shared.v4.u32 {%0, %1, %2, %3}, [%4];"
                 : "=r"(r.v[0]), "=r"(r.v[1]), "=r"(r.v[2]), "=r"(r.v[3])
                 : "r"(p)
                 : "memory");
    asm volatile("ld.shared.v4.u32 {%0, %1, %2, %3}, [%4];"
                 : "=r"(r.v[4]), "=r"(r.v[5]), "=r"(r.v[6]), "=r"(r.v[7])
                 : "r"(p + 16 * BLOCK)
                 : "memory");
    return r;
}

// Whether a canonical u is that of a point 1Q .. MQ: by the first words, four
// to a load, then by all (the whole table through the constant cache takes
// 18 us at M = 512, a line's latency for every two entries; this 1.2 us: one
// lane 0.130 -> 0.134 ms for four groups, 2,048 lanes 1.83 -> 1.86).
template <int M, class Table>
__device__ __forceinline__ bool table_holds(const Table& t, const uint4* __restrict__ first_words, const fe& u) {
    bool near = false;
#pragma unroll 8
    for (int i = 0; i < M / 4; ++i) {
        const uint4 w = first_words[i];
        near |= (w.x == u.v[0]) | (w.y == u.v[0]) | (w.z == u.v[0]) | (w.w == u.v[0]);
    }
    bool held = false;
    if (near) {
#pragma unroll 1
        for (int i = 1; i <= M; ++i) {
            const fe x = t.u[i];
            uint32_t d = 0;
#pragma unroll
            for (int w = 0; w < 8; w++) d |= x.v[w] ^ u.v[w];
            held |= d == 0;
        }
    }
    return held;
}

// `groups` groups of one lane's walk from centre (uc, vc) at walk index n
// (the first key of the next group); emit(u, key) receives every key's
// canonical u.  Shared by the plain walk and the pool's persistent kernel.
// SYNC: a block barrier after each group keeps the block's warps in the same
// phase of the walk, so that they share the instruction cache's working set
// (one phase's code instead of all of it); every thread of the block must
// then call this with the same `groups`.
// lo, hi: the part of each group to walk, the keys c +- i with lo < i <= hi
// (and the centre where lo is 0); 0 and M: all of it.  Every part steps to
// the next centre by itself.
// ANY: start points of any kind (Backend::init).  A centre may then be a table
// point up to sign, whose denominator of zero makes every inverse of its group
// zero; so that all parts agree, each looks for its centre among all table
// points.  Walks from clamped scalars never get there: their centres are
// s Q with 2^251 < s, and the order of Q is above s by 2^124 keys at least.
// The loop takes 126 to 128 registers, the cap, in all its kernels; with the
// sum u_C + A among them, and -u_C or -v_C, ptxas schedules around the cap and
// the parts kernel loses 7% (4.71-4.77 against 5.12-5.14 G keys/s at 37,888
// lanes).  So the sum, used once per pair, waits in shared memory, 32 bytes per
// thread of the block.
template <int M, int BLOCK, bool SYNC, bool ANY = false, class Table, class Emit>
__device__ __forceinline__ void walk_groups(fe& uc, fe& vc, uint64_t& n, uint32_t groups, const Table& t,
                                            const Emit& emit, const int lo = 0, const int hi = M,
                                            const uint4* first_words = nullptr) {
    __shared__ uint4 s_sum[2 * BLOCK];
    uint4* const sum = s_sum + threadIdx.x;
    fe pre[M + 1];
    fe cA = fe_zero();
    cA.v[0] = LXK_A;
#pragma unroll 1
    for (uint32_t it = 0; it < groups; ++it) {
        // With canonical coordinates (as the table's are), sums of two need no reduction.
        uc = fe_canon(uc);
        vc = fe_canon(vc);
        const fe nu = fe_neg_raw(uc);
        // Denominators e_0 = u_J - u_C, e_i = u_{T_i} - u_C; pre[i] = e_0 e_{lo+1} ... e_{i-1}.
        fe acc = fe_add_raw(t.u[0], nu);
#pragma unroll 1
        for (int i = lo + 1; i <= hi; ++i) {
            pre[i] = acc;
            acc = fe_mul(acc, fe_add_raw(t.u[i], nu));
        }
        if (ANY && table_holds<M>(t, first_words, uc)) acc = fe_zero();
        fe inv = fe_invert(acc);
        const uint64_t c = n + M;
        park_fe<BLOCK>(sum, fe_canon(fe_add(uc, cA)));
        fe vnext = vc;
#pragma unroll 1
        for (int k = hi; k >= lo; --k) {
            const int i = k > lo ? k : 0;  // last, the step to the next centre
            const fe tu = t.u[i], tv = t.v[i];
            fe invi = inv;  // 1 / e_i
            if (i > 0) {
                invi = fe_mul(inv, pre[i]);
                inv = fe_mul(inv, fe_add_raw(tu, nu));
            }
            const fe s = fe_add_raw(parked_fe<BLOCK>(sum), tu);
            const fe lp = fe_mul(fe_sub(tv, vc), invi);
            const fe up = fe_sub_canon(fe_sqr(lp), s);  // C + T_i (for i = 0: the next centre C + J)
            fe um;
            if (i > 0) {
                const fe lm = fe_mul(fe_add_raw(tv, vc), invi);
                um = fe_sub_canon(fe_sqr(lm), s);       // C - T_i
            } else {
                um = uc;                                // C itself
                vnext = fe_sub(fe_mul(lp, fe_sub(uc, up)), vc);
            }
#pragma unroll 1
            for (int side = 0; side < 2; ++side) {
                // side 0: key c + i (only 0 < i < M: c + M is the next group's);
                // side 1: key c - i (i = 0: the centre, walked by the part that starts at 0).
                if (side == 1 ? (i > 0 || lo == 0) : (i > 0 && i < M))
                    emit(side ? um : up, side ? c - (uint64_t)i : c + (uint64_t)i);
            }
            if (i == 0) {
                uc = up;
                vc = vnext;
            }
        }
        n += 2 * M;
        if (SYNC) __syncthreads();
    }
}

// ---- Parts: each group split over several warps.
//
// A lane's groups are a serial chain, so a walk of few lanes leaves most of
// the device idle, and one whose lanes are no multiple of a wave leaves its
// last wave nearly empty.  The parts of a group are independent: 32 lanes are
// walked by S warps, warp j the keys c +- i with floor(j M/S) < i <=
// floor((j+1) M/S), each with its own batch inversion and its own step to the next centre.  Every
// key, hash and hit is the one that a single warp finds.
constexpr int kPartsWarps = 16;  // warps per block (512 threads, one block per SM)

// S for `chunks` chunks of 32 lanes on `sms` SMs: the one with the smallest
// predicted time, (ceil(M/S) + 1.8) x (full rounds of 16 warps per SM + the
// last round's share).  Measured on B200: an inversion with the step to
// the next centre takes as long as 1.8 pairs of keys at any occupancy (on 30-bit
// limbs; 8% less now, and the rule not refitted), and a
// round of 1, 2, 3 or 4 warps per SM sub-partition takes 10.2, 16.7, 23.9 or
// 31.1 us per pair (a lone warp issues at three quarters of the full rate).
// So few lanes split until every sub-partition has a warp and the inversions
// (15 us at least) weigh as much as the keys; full waves stay whole.
inline uint32_t group_parts(uint64_t chunks, uint32_t m, uint32_t sms) {
    static const uint32_t kRound[5] = {0, 21, 34, 49, 64};
    const uint64_t slots = (uint64_t)sms * kPartsWarps;
    if (slots == 0) return 1;  // a handle that failed to open
    uint32_t best = 1;
    uint64_t best_cost = ~0ull;
    for (uint32_t s = 1; s <= m; s++) {
        const uint64_t units = chunks * s, rest = units % slots;
        const uint64_t rounds = units / slots * kRound[4] + kRound[(rest + 4 * sms - 1) / (4 * sms)];
        const uint64_t cost = (10 * ((m + s - 1) / s) + 18) * rounds;
        if (cost <= best_cost) {  // of equals the larger: some of its parts have a pair less
            best_cost = cost;
            best = s;
        }
    }
    return best;
}

// Part j's first i, exclusive, and the next part's.
__device__ __forceinline__ int part_begin(uint32_t m, uint32_t j, uint32_t parts) { return (int)(j * m / parts); }

// A warp has walked its part of a chunk.  True for the last of the S
// warps to come here, the one that stores the chunk's new state: by then the
// others have read the old one.  The count orders those reads before the
// store: released by each warp, acquired by the last, and passed on to and from
// the other lanes by the warp barriers.
__device__ __forceinline__ bool part_done(uint32_t* done, uint32_t parts) {
    if (parts == 1) return true;
    uint32_t before = 0;
    __syncwarp();
    if ((threadIdx.x & 31) == 0) {
        asm volatile("atom.acq_rel.gpu.global.add.u32 %0, [%1], 1;" : "=r"(before) : "l"(__cvta_generic_to_global(done)) : "memory");
        if (before == parts - 1) *done = 0;  // for the next launch
    }
    __syncwarp();
    return __shfl_sync(0xffffffffu, before, 0) == parts - 1;
}

// The plain search's emission: one prefix for every lane of the launch.
template <bool DUMP>
struct LaneEmit {
    const EmitArgs& em;
    uint32_t lane;
    uint64_t key0;
    bool active;
    __device__ __forceinline__ void operator()(const fe& u, uint64_t key) const {
        if (active) emit_key<DUMP>(em, lane, key, key0, u);
    }
};

// Threads past the last lane walk a copy of the last lane and neither emit
// nor store (with SYNC they must still reach every barrier).
template <int M, int BLOCK, int MINB, bool SYNC, bool DUMP, class Args = GroupArgsFor<M>>
static __global__ void __launch_bounds__(BLOCK, MINB) group_walk_kernel(const __grid_constant__ Args a) {
    const uint32_t tid = blockIdx.x * BLOCK + threadIdx.x;
    if (!SYNC && tid >= a.lanes) return;
    const bool active = tid < a.lanes;
    const uint32_t lane = active ? tid : a.lanes - 1;
    fe uc = load_fe(a.state, 0, lane, a.lanes);
    fe vc = load_fe(a.state, 1, lane, a.lanes);
    const uint64_t key0 = a.ns[lane];
    uint64_t n = key0;
    const LaneEmit<DUMP> emit{a.em, lane, key0, active};
    walk_groups<M, BLOCK, SYNC>(uc, vc, n, a.iters, table_of(a), emit);
    if (active) {
        store_fe(a.state, 0, lane, a.lanes, uc);
        store_fe(a.state, 1, lane, a.lanes, vc);
        a.ns[lane] = n;
    }
}

// The plain walk in parts: one block per SM, whose warps take units of (32
// lanes, part) a grid apart, so that the units of a short last round spread
// over all SMs and their sub-partitions.  Lanes past the last one walk a copy
// of it.  At G = 1024 on B200, one group: 32 lanes 0.04 ms, 2,048 lanes
// 0.46, 100,003 lanes 19.9 (5.15 G keys/s; a whole wave 5.26); one warp per
// chunk in blocks of 512: 15, 15 and 30 ms.
template <int M, bool DUMP, bool ANY, class Args = GroupArgsFor<M>>
static __global__ void __launch_bounds__(32 * kPartsWarps, 1) group_parts_kernel(const __grid_constant__ Args a) {
    const uint32_t lid = threadIdx.x & 31;
    const uint32_t chunks = (a.lanes + 31) / 32, parts = a.parts;
    const uint64_t units = (uint64_t)chunks * parts;
#pragma unroll 1
    for (uint64_t unit = blockIdx.x + (uint64_t)gridDim.x * (threadIdx.x >> 5); unit < units;
         unit += (uint64_t)gridDim.x * kPartsWarps) {
        const uint32_t chunk = (uint32_t)(unit / parts);
        const uint32_t j = (uint32_t)(unit - (uint64_t)chunk * parts);
        const bool active = chunk * 32 + lid < a.lanes;
        const uint32_t lane = active ? chunk * 32 + lid : a.lanes - 1;
        fe uc = load_fe(a.state, 0, lane, a.lanes);
        fe vc = load_fe(a.state, 1, lane, a.lanes);
        const uint64_t key0 = a.ns[lane];
        uint64_t n = key0;
        const LaneEmit<DUMP> emit{a.em, lane, key0, active};
        walk_groups<M, 32 * kPartsWarps, false, ANY>(uc, vc, n, a.iters, table_of(a), emit, part_begin(M, j, parts),
                                                      part_begin(M, j + 1, parts), a.first_words);
        if (part_done(a.done + chunk, parts) && active) {
            store_fe(a.state, 0, lane, a.lanes, uc);
            store_fe(a.state, 1, lane, a.lanes, vc);
            a.ns[lane] = n;
        }
    }
}

}  // namespace lxk
