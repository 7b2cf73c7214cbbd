// Point arithmetic by groups of lanes, for the bucket reduction.
//
// A point operation is ten to fourteen products deep when one thread runs it,
// and a warp takes 845 cycles for a dependent product whether one of its lanes
// works or all 32: 528 to issue its multiply-adds (128 wide at 8 lanes a clock,
// 8 low halves at 16) and about 320 of latency that nothing covers.  The
// reduction's last steps have few points left, so here every point is spread
// over a group of lanes, one coordinate each (X, Y, ZZ, ZZZ), and the
// independent products of a formula run side by side: an addition is four
// products deep and a doubling three.  The 14 products of an addition fill 16
// slots, so a group's addition costs a full device about a sixth more than a
// thread's, and a third of the time where warps are few.  A lane holds a quarter
// of each point: blocks of 256 threads at 95 to 106 registers over G1 and 100 to
// 122 over G2, two blocks an SM and no spills, where a thread's version needed 250.
//
// A G1 point takes 4 lanes; a G2 point 8, lane 2k + i holding component i of
// coordinate k.  A group's lanes are consecutive and aligned, and lane q's
// element is the q-th 32 bytes of the point in memory, so loads and stores
// are contiguous.  Every function here is called by whole warps (the groups of
// a warp run together and exchange values by shuffles); a group without work
// adds the identity.
#pragma once
#include "curve.cuh"

namespace g16d {

template <class F>
struct Lanes;
template <>
struct Lanes<Fq> {
    static constexpr int C = 1, N = 4;   // lanes per coordinate and per point
};
template <>
struct Lanes<Fq2> {
    static constexpr int C = 2, N = 8;
};

constexpr unsigned FULL_WARP = 0xffffffffu;

__device__ __forceinline__ Fq shfl_xor(const Fq& a, int m) {
    Fq r;
#pragma unroll
    for (int i = 0; i < 8; i++) r.v[i] = __shfl_xor_sync(FULL_WARP, a.v[i], m);
    return r;
}
__device__ __forceinline__ Fq shfl_from(const Fq& a, int lane) {
    Fq r;
#pragma unroll
    for (int i = 0; i < 8; i++) r.v[i] = __shfl_sync(FULL_WARP, a.v[i], lane);
    return r;
}
__device__ __forceinline__ Fq pick(bool c, const Fq& a, const Fq& b) {
    Fq r;
#pragma unroll
    for (int i = 0; i < 8; i++) r.v[i] = c ? a.v[i] : b.v[i];
    return r;
}

// The lane's component of the product of two coordinates.  Over Fq2 the two
// lanes of a coordinate exchange their components and each forms its own with
// one reduction: a0 b0 + (q - a1) b1 and a1 b0 + a0 b1.
template <class F>
__device__ __forceinline__ Fq lane_mul(const Fq& a, const Fq& b) {
    if constexpr (Lanes<F>::C == 1) {
        return mul(a, b);
    } else {
        const bool odd = threadIdx.x & 1;
        const Fq ax = shfl_xor(a, 1), bx = shfl_xor(b, 1);
        const Modulus<FqParams> q;
        Fq n, r;
        sub_words<8>(n.v, q.v, ax.v);   // q - a1
        const Fq y = pick(odd, bx, b), z = pick(odd, ax, n), w = pick(odd, b, bx);
        mul_add_redc<FqParams>(a.v, y.v, z.v, w.v, r.v);
        reduce_once<FqParams>(r.v);
        return r;
    }
}

// Where a lane stands in its group.
template <class F>
struct Place {
    int base;    // the group's first lane
    int k;       // coordinate: 0 X, 1 Y, 2 ZZ, 3 ZZZ
    int i;       // component
    __device__ __forceinline__ Place() {
        const int lane = threadIdx.x & 31;
        base = lane & ~(Lanes<F>::N - 1);
        k = (lane & (Lanes<F>::N - 1)) / Lanes<F>::C;
        i = lane & (Lanes<F>::C - 1);
    }
    // the lane of coordinate c with this lane's component
    __device__ __forceinline__ int at(int c) const { return base + c * Lanes<F>::C + i; }
    // is coordinate c zero, from a warp's ballot of zero elements
    __device__ __forceinline__ bool zero(unsigned ballot, int c) const {
        constexpr unsigned m = (1u << Lanes<F>::C) - 1u;
        return ((ballot >> (base + c * Lanes<F>::C)) & m) == m;
    }
};

// Bit 2 C of each group of a warp (the lane of ZZ's first component), and those
// bits where the group's point is the identity, from a warp's ballot of zero
// elements: the same value in every lane.
template <class F>
constexpr unsigned ZZ_LANES = Lanes<F>::C == 1 ? 0x44444444u : 0x10101010u;
template <class F>
__device__ __forceinline__ unsigned identities(unsigned ballot) {
    return (Lanes<F>::C == 1 ? ballot : ballot & (ballot >> 1)) & ZZ_LANES<F>;
}

// 2 p (dbl-2008-s-1): V = (2Y)^2 and X^2; then W = 2Y V, S = X V, ZZ3 = V ZZ and
// M^2; then M (S - X3), W Y and ZZZ3 = W ZZZ.  The identity stays itself; a warp
// of identities returns at once.
template <class F>
__device__ __forceinline__ Fq lanes_dbl(const Fq& p) {
    if (identities<F>(__ballot_sync(FULL_WARP, p.is_zero())) == ZZ_LANES<F>) return p;
    const Place<F> g;
    const Fq u = pick(g.k == 1, dbl(p), p);
    const Fq s1 = lane_mul<F>(u, u);                     // k 0: X^2, 1: V
    const Fq v = shfl_from(s1, g.at(1)), xx = shfl_from(s1, g.at(0));
    const Fq m = add(dbl(xx), xx);
    const Fq s2 = lane_mul<F>(pick(g.k == 3, m, u), pick(g.k == 3, m, v));   // S, W, ZZ3, M^2
    const Fq w = shfl_from(s2, g.at(1)), mm = shfl_from(s2, g.at(3));
    const Fq x3 = sub(mm, dbl(s2));                      // k 0
    const Fq s3 = lane_mul<F>(pick(g.k == 0, m, w), pick(g.k == 0, sub(s2, x3), p));
    const Fq o = shfl_from(s3, g.at(0));
    Fq r = pick(g.k == 0, x3, s3);
    r = pick(g.k == 1, sub(o, s3), r);
    return pick(g.k == 2, s2, r);
}

// p + q (add-2008-s), the identity and equal operands included: U1, S1, U2, S2;
// then P^2, R^2, ZZ1 ZZ2, ZZZ1 ZZZ2; then Q, PPP, ZZ3; then R (Q - X3), S1 PPP
// and ZZZ3.  p + (-p) comes out with ZZ3 = ZZZ3 = 0, the identity.  A warp whose
// groups each have an identity operand forms no product: the reduction of few or
// no full buckets costs little (MSMs with every scalar zero, G1 2^20 638 us with
// the products and 217 without, G2 2^18 880 and 167; every scalar one, 899 and
// 479, 1207 and 502; uniform ones level).
template <class F>
__device__ __forceinline__ Fq lanes_add(const Fq& p, const Fq& q) {
    constexpr int C = Lanes<F>::C;
    const Place<F> g;
    const unsigned pz = __ballot_sync(FULL_WARP, p.is_zero()), qz = __ballot_sync(FULL_WARP, q.is_zero());
    const bool p_inf = g.zero(pz, 2);
    if ((identities<F>(pz) | identities<F>(qz)) == ZZ_LANES<F>) return pick(p_inf, q, p);
    const bool q_inf = g.zero(qz, 2);
    const Fq t = lane_mul<F>(p, shfl_xor(q, 2 * C));     // U1, S1, U2, S2
    const Fq tx = shfl_xor(t, 2 * C);
    const bool low = g.k < 2;
    const Fq d = sub(pick(low, tx, t), pick(low, t, tx));   // k 0, 2: P; 1, 3: R
    const unsigned dz = __ballot_sync(FULL_WARP, d.is_zero());
    const bool twice = !p_inf && !q_inf && g.zero(dz, 0) && g.zero(dz, 1);
    const Fq u = lane_mul<F>(pick(low, d, p), pick(low, d, q));   // P^2, R^2, ZZ1 ZZ2, ZZZ1 ZZZ2
    const Fq pp = shfl_from(u, g.at(0)), dp = shfl_from(d, g.at(0));
    Fq a = pick(g.k == 0, t, u);
    a = pick(g.k == 1, dp, a);
    const Fq w = lane_mul<F>(a, pp);                     // Q, PPP, ZZ3, -
    const Fq ppp = shfl_from(w, g.at(1));
    const Fq e = shfl_from(sub(u, w), g.at(1));          // R^2 - PPP
    const Fq r = shfl_from(d, g.at(1));
    const Fq x3 = sub(e, dbl(w));                        // k 0
    a = pick(g.k == 0, sub(w, x3), pick(g.k == 1, t, u));
    const Fq v = lane_mul<F>(a, pick(g.k == 0, r, ppp)); // R (Q - X3), S1 PPP, -, ZZZ3
    const Fq o = shfl_from(v, g.at(0));
    Fq s = pick(g.k == 0, x3, v);
    s = pick(g.k == 1, sub(o, v), s);
    s = pick(g.k == 2, w, s);
    if (__any_sync(FULL_WARP, twice)) {   // equal operands are rare
        const Fq s2 = lanes_dbl<F>(p);
        s = pick(twice, s2, s);
    }
    s = pick(q_inf, p, s);
    return pick(p_inf, q, s);
}

// The lane's element of point i.
template <class F>
__device__ __forceinline__ Fq ld_lane(const uint4* base, size_t i) {
    return ld_fq_rw(base + (i * Lanes<F>::N + (threadIdx.x & (Lanes<F>::N - 1))) * 2);
}
template <class F>
__device__ __forceinline__ void st_lane(uint4* base, size_t i, const Fq& x) {
    st_fq(base + (i * Lanes<F>::N + (threadIdx.x & (Lanes<F>::N - 1))) * 2, x);
}

// The sum of one point per group over the block (groups a power of two of
// them); the result is valid in group 0.  smem holds groups points.
template <class F>
__device__ __forceinline__ Fq block_sum_lanes(Fq acc, uint4* smem, uint32_t groups) {
    const uint32_t t = threadIdx.x / Lanes<F>::N, warp_first = (threadIdx.x & ~31u) / Lanes<F>::N;
    st_lane<F>(smem, t, acc);
    __syncthreads();
    for (uint32_t s = groups / 2; s > 0; s >>= 1) {
        if (warp_first < s) {   // a whole warp at a time
            const Fq o = t < s ? ld_lane<F>(smem, t + s) : Fq::zero();
            acc = lanes_add<F>(acc, o);
            if (t < s) st_lane<F>(smem, t, acc);
        }
        __syncthreads();
    }
    return acc;
}

}  // namespace g16d
