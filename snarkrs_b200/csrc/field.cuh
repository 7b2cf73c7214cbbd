// BN254 Fr / Fq / Fq2 arithmetic for sm_100a.
//
// Eight 32-bit little-endian limbs, Montgomery form with R = 2^256: the same
// bits as arkworks' in-memory Fp and snarkrs' PackedFr / PackedFq
// (crates/gpu-layout/src/lib.rs:30-46, 75-113).  Every value leaving a
// function is fully reduced into [0, p), so device results compare bit for
// bit with the CPU prover.
//
// The Montgomery product is CIOS (Koc, Acar and Kaliski, "Analyzing and
// comparing Montgomery multiplication algorithms", 1996) with the running sum
// held as two vectors of 64-bit lanes, one over the even limb positions and
// one over the odd ones (the column split that Emmart, Zheng and Weems use on
// GPUs).  Within a vector the partial products a[j] b do not overlap, so a row
// is one carry chain of 32x32+64-bit multiply-adds and no other instruction;
// the carry between the vectors rides into the next row's chain.  What bounds
// it is the issue rate of multiply-adds: 128 wide ones at 32 a clock on an SM
// and 8 low halves (the quotient digits) at 64 a clock are 4.125 clocks a
// product, 70.5 G products/s on 148 SMs at 1965 MHz.  It measured 66.5 G/s, 0.94
// of that (one product per thread and step, 1024 threads an SM), and 845 cycles
// for one warp's dependent product, against 44.0 G/s and 1127 cycles for the
// form it replaced, a single vector whose carries were 64-bit sums on the ALU
// pipe.
// BN254's moduli are below 2^254, so the running sum stays below 2^287 and
// fits nine limbs; the carry out of the ninth is provably zero.
#pragma once
#include <cstdint>

namespace g16d {

// Limb tables as constexpr functions: every use sits in a fully unrolled loop
// or an "n" asm operand, so each call folds to an immediate.
struct FrParams {
    __host__ __device__ static constexpr uint32_t P(int i) {
        constexpr uint32_t v[8] = {0xf0000001u, 0x43e1f593u, 0x79b97091u, 0x2833e848u,
                                   0x8181585du, 0xb85045b6u, 0xe131a029u, 0x30644e72u};
        return v[i];
    }
    static constexpr uint32_t N0 = 0xefffffffu;
    // R mod r, the Montgomery form of one
    __host__ __device__ static constexpr uint32_t ONE(int i) {
        constexpr uint32_t v[8] = {0x4ffffffbu, 0xac96341cu, 0x9f60cd29u, 0x36fc7695u,
                                   0x7879462eu, 0x666ea36fu, 0x9a07df2fu, 0x0e0a77c1u};
        return v[i];
    }
};

struct FqParams {
    __host__ __device__ static constexpr uint32_t P(int i) {
        constexpr uint32_t v[8] = {0xd87cfd47u, 0x3c208c16u, 0x6871ca8du, 0x97816a91u,
                                   0x8181585du, 0xb85045b6u, 0xe131a029u, 0x30644e72u};
        return v[i];
    }
    static constexpr uint32_t N0 = 0xe4866389u;
    __host__ __device__ static constexpr uint32_t ONE(int i) {
        constexpr uint32_t v[8] = {0xc58f0d9du, 0xd35d438du, 0xf5c70b3du, 0x0a78eb28u,
                                   0x7879462cu, 0x666ea36fu, 0x9a07df2fu, 0x0e0a77c1u};
        return v[i];
    }
    // q^2 as 16 limbs (the Fq2 product's offset that keeps a0 b0 - a1 b1 positive)
    __host__ __device__ static constexpr uint32_t P2W(int i) {
        constexpr uint32_t v[16] = {0x275d69b1u, 0x3b5458a2u, 0x09eac101u, 0xa602072du, 0x6d96cadcu, 0x4a50189cu,
                                    0x7a1242c8u, 0x04689e95u, 0x34c6b38du, 0x26edfa5cu, 0x16375606u, 0xb00b8551u,
                                    0x0348d21cu, 0x599a6f7cu, 0x763cbf9cu, 0x0925c4b8u};
        return v[i];
    }
};

template <class Params>
struct __align__(16) Fp {
    uint32_t v[8];

    __device__ __forceinline__ static Fp zero() {
        Fp r;
#pragma unroll
        for (int i = 0; i < 8; i++) r.v[i] = 0;
        return r;
    }
    __device__ __forceinline__ static Fp one() {
        Fp r;
#pragma unroll
        for (int i = 0; i < 8; i++) r.v[i] = Params::ONE(i);
        return r;
    }
    __device__ __forceinline__ bool is_zero() const {
        uint32_t acc = v[0];
#pragma unroll
        for (int i = 1; i < 8; i++) acc |= v[i];
        return acc == 0;
    }
    __device__ __forceinline__ bool eq(const Fp& o) const {
        uint32_t acc = 0;
#pragma unroll
        for (int i = 0; i < 8; i++) acc |= v[i] ^ o.v[i];
        return acc == 0;
    }
    __device__ __forceinline__ bool is_one() const { return eq(one()); }
};

// r = a - p if a >= p (a < 2p), in registers
template <class Params>
__device__ __forceinline__ void reduce_once(uint32_t* a) {
    uint32_t d[8], borrow;
    asm("sub.cc.u32  %0, %9, %17;\n\t"
        "subc.cc.u32 %1, %10, %18;\n\t"
        "subc.cc.u32 %2, %11, %19;\n\t"
        "subc.cc.u32 %3, %12, %20;\n\t"
        "subc.cc.u32 %4, %13, %21;\n\t"
        "subc.cc.u32 %5, %14, %22;\n\t"
        "subc.cc.u32 %6, %15, %23;\n\t"
        "subc.cc.u32 %7, %16, %24;\n\t"
        "subc.u32    %8, 0, 0;"
        : "=r"(d[0]), "=r"(d[1]), "=r"(d[2]), "=r"(d[3]), "=r"(d[4]), "=r"(d[5]), "=r"(d[6]), "=r"(d[7]),
          "=r"(borrow)
        : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(a[4]), "r"(a[5]), "r"(a[6]), "r"(a[7]),
          "n"(Params::P(0)), "n"(Params::P(1)), "n"(Params::P(2)), "n"(Params::P(3)), "n"(Params::P(4)),
          "n"(Params::P(5)), "n"(Params::P(6)), "n"(Params::P(7)));
    // borrow == 0xffffffff when a < p: keep a
#pragma unroll
    for (int i = 0; i < 8; i++) a[i] = borrow ? a[i] : d[i];
}

template <class Params>
__device__ __forceinline__ Fp<Params> add(const Fp<Params>& a, const Fp<Params>& b) {
    Fp<Params> r;
    asm("add.cc.u32  %0, %8, %16;\n\t"
        "addc.cc.u32 %1, %9, %17;\n\t"
        "addc.cc.u32 %2, %10, %18;\n\t"
        "addc.cc.u32 %3, %11, %19;\n\t"
        "addc.cc.u32 %4, %12, %20;\n\t"
        "addc.cc.u32 %5, %13, %21;\n\t"
        "addc.cc.u32 %6, %14, %22;\n\t"
        "addc.u32    %7, %15, %23;"
        : "=r"(r.v[0]), "=r"(r.v[1]), "=r"(r.v[2]), "=r"(r.v[3]), "=r"(r.v[4]), "=r"(r.v[5]), "=r"(r.v[6]),
          "=r"(r.v[7])
        : "r"(a.v[0]), "r"(a.v[1]), "r"(a.v[2]), "r"(a.v[3]), "r"(a.v[4]), "r"(a.v[5]), "r"(a.v[6]), "r"(a.v[7]),
          "r"(b.v[0]), "r"(b.v[1]), "r"(b.v[2]), "r"(b.v[3]), "r"(b.v[4]), "r"(b.v[5]), "r"(b.v[6]), "r"(b.v[7]));
    reduce_once<Params>(r.v);
    return r;
}

template <class Params>
__device__ __forceinline__ Fp<Params> sub(const Fp<Params>& a, const Fp<Params>& b) {
    Fp<Params> r;
    uint32_t borrow;
    asm("sub.cc.u32  %0, %9, %17;\n\t"
        "subc.cc.u32 %1, %10, %18;\n\t"
        "subc.cc.u32 %2, %11, %19;\n\t"
        "subc.cc.u32 %3, %12, %20;\n\t"
        "subc.cc.u32 %4, %13, %21;\n\t"
        "subc.cc.u32 %5, %14, %22;\n\t"
        "subc.cc.u32 %6, %15, %23;\n\t"
        "subc.cc.u32 %7, %16, %24;\n\t"
        "subc.u32    %8, 0, 0;"
        : "=r"(r.v[0]), "=r"(r.v[1]), "=r"(r.v[2]), "=r"(r.v[3]), "=r"(r.v[4]), "=r"(r.v[5]), "=r"(r.v[6]),
          "=r"(r.v[7]), "=r"(borrow)
        : "r"(a.v[0]), "r"(a.v[1]), "r"(a.v[2]), "r"(a.v[3]), "r"(a.v[4]), "r"(a.v[5]), "r"(a.v[6]), "r"(a.v[7]),
          "r"(b.v[0]), "r"(b.v[1]), "r"(b.v[2]), "r"(b.v[3]), "r"(b.v[4]), "r"(b.v[5]), "r"(b.v[6]), "r"(b.v[7]));
    // add p back when the subtraction borrowed (p & mask)
    uint32_t m = borrow;
    asm("add.cc.u32  %0, %0, %8;\n\t"
        "addc.cc.u32 %1, %1, %9;\n\t"
        "addc.cc.u32 %2, %2, %10;\n\t"
        "addc.cc.u32 %3, %3, %11;\n\t"
        "addc.cc.u32 %4, %4, %12;\n\t"
        "addc.cc.u32 %5, %5, %13;\n\t"
        "addc.cc.u32 %6, %6, %14;\n\t"
        "addc.u32    %7, %7, %15;"
        : "+r"(r.v[0]), "+r"(r.v[1]), "+r"(r.v[2]), "+r"(r.v[3]), "+r"(r.v[4]), "+r"(r.v[5]), "+r"(r.v[6]),
          "+r"(r.v[7])
        : "r"(Params::P(0) & m), "r"(Params::P(1) & m), "r"(Params::P(2) & m), "r"(Params::P(3) & m),
          "r"(Params::P(4) & m), "r"(Params::P(5) & m), "r"(Params::P(6) & m), "r"(Params::P(7) & m));
    return r;
}

template <class Params>
__device__ __forceinline__ Fp<Params> neg(const Fp<Params>& a) {
    return a.is_zero() ? a : sub(Fp<Params>::zero(), a);
}

template <class Params>
__device__ __forceinline__ Fp<Params> dbl(const Fp<Params>& a) {
    return add(a, a);
}

// ---- r = a + b, r = a - b over 8 or 16 words, the last carry or borrow dropped ----
// (early-clobber outputs: a word of r is written before the later words of a
// and b are read)
template <int N>
__host__ __device__ __forceinline__ void add_words(uint32_t* r, const uint32_t* a, const uint32_t* b) {
    static_assert(N == 8 || N == 16, "word count");
#ifdef __CUDA_ARCH__
    if constexpr (N == 8)
        asm("add.cc.u32 %0, %8, %16;\n\t"
            "addc.cc.u32 %1, %9, %17;\n\t"
            "addc.cc.u32 %2, %10, %18;\n\t"
            "addc.cc.u32 %3, %11, %19;\n\t"
            "addc.cc.u32 %4, %12, %20;\n\t"
            "addc.cc.u32 %5, %13, %21;\n\t"
            "addc.cc.u32 %6, %14, %22;\n\t"
            "addc.u32  %7, %15, %23;"
            : "=&r"(r[0]), "=&r"(r[1]), "=&r"(r[2]), "=&r"(r[3]), "=&r"(r[4]), "=&r"(r[5]), "=&r"(r[6]), "=&r"(r[7])
            : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(a[4]), "r"(a[5]), "r"(a[6]), "r"(a[7]),
              "r"(b[0]), "r"(b[1]), "r"(b[2]), "r"(b[3]), "r"(b[4]), "r"(b[5]), "r"(b[6]), "r"(b[7]));
    else
        asm("add.cc.u32 %0, %16, %32;\n\t"
            "addc.cc.u32 %1, %17, %33;\n\t"
            "addc.cc.u32 %2, %18, %34;\n\t"
            "addc.cc.u32 %3, %19, %35;\n\t"
            "addc.cc.u32 %4, %20, %36;\n\t"
            "addc.cc.u32 %5, %21, %37;\n\t"
            "addc.cc.u32 %6, %22, %38;\n\t"
            "addc.cc.u32 %7, %23, %39;\n\t"
            "addc.cc.u32 %8, %24, %40;\n\t"
            "addc.cc.u32 %9, %25, %41;\n\t"
            "addc.cc.u32 %10, %26, %42;\n\t"
            "addc.cc.u32 %11, %27, %43;\n\t"
            "addc.cc.u32 %12, %28, %44;\n\t"
            "addc.cc.u32 %13, %29, %45;\n\t"
            "addc.cc.u32 %14, %30, %46;\n\t"
            "addc.u32  %15, %31, %47;"
            : "=&r"(r[0]), "=&r"(r[1]), "=&r"(r[2]), "=&r"(r[3]), "=&r"(r[4]), "=&r"(r[5]), "=&r"(r[6]), "=&r"(r[7]),
          "=&r"(r[8]), "=&r"(r[9]), "=&r"(r[10]), "=&r"(r[11]), "=&r"(r[12]), "=&r"(r[13]), "=&r"(r[14]), "=&r"(r[15])
            : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(a[4]), "r"(a[5]), "r"(a[6]), "r"(a[7]), "r"(a[8]),
          "r"(a[9]), "r"(a[10]), "r"(a[11]), "r"(a[12]), "r"(a[13]), "r"(a[14]), "r"(a[15]),
              "r"(b[0]), "r"(b[1]), "r"(b[2]), "r"(b[3]), "r"(b[4]), "r"(b[5]), "r"(b[6]), "r"(b[7]), "r"(b[8]),
          "r"(b[9]), "r"(b[10]), "r"(b[11]), "r"(b[12]), "r"(b[13]), "r"(b[14]), "r"(b[15]));
#else
    uint64_t c = 0;
    for (int k = 0; k < N; k++) {
        c += (uint64_t)a[k] + b[k];
        r[k] = (uint32_t)c;
        c >>= 32;
    }
#endif
}
template <int N>
__host__ __device__ __forceinline__ void sub_words(uint32_t* r, const uint32_t* a, const uint32_t* b) {
    static_assert(N == 8 || N == 16, "word count");
#ifdef __CUDA_ARCH__
    if constexpr (N == 8)
        asm("sub.cc.u32 %0, %8, %16;\n\t"
            "subc.cc.u32 %1, %9, %17;\n\t"
            "subc.cc.u32 %2, %10, %18;\n\t"
            "subc.cc.u32 %3, %11, %19;\n\t"
            "subc.cc.u32 %4, %12, %20;\n\t"
            "subc.cc.u32 %5, %13, %21;\n\t"
            "subc.cc.u32 %6, %14, %22;\n\t"
            "subc.u32  %7, %15, %23;"
            : "=&r"(r[0]), "=&r"(r[1]), "=&r"(r[2]), "=&r"(r[3]), "=&r"(r[4]), "=&r"(r[5]), "=&r"(r[6]), "=&r"(r[7])
            : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(a[4]), "r"(a[5]), "r"(a[6]), "r"(a[7]),
              "r"(b[0]), "r"(b[1]), "r"(b[2]), "r"(b[3]), "r"(b[4]), "r"(b[5]), "r"(b[6]), "r"(b[7]));
    else
        asm("sub.cc.u32 %0, %16, %32;\n\t"
            "subc.cc.u32 %1, %17, %33;\n\t"
            "subc.cc.u32 %2, %18, %34;\n\t"
            "subc.cc.u32 %3, %19, %35;\n\t"
            "subc.cc.u32 %4, %20, %36;\n\t"
            "subc.cc.u32 %5, %21, %37;\n\t"
            "subc.cc.u32 %6, %22, %38;\n\t"
            "subc.cc.u32 %7, %23, %39;\n\t"
            "subc.cc.u32 %8, %24, %40;\n\t"
            "subc.cc.u32 %9, %25, %41;\n\t"
            "subc.cc.u32 %10, %26, %42;\n\t"
            "subc.cc.u32 %11, %27, %43;\n\t"
            "subc.cc.u32 %12, %28, %44;\n\t"
            "subc.cc.u32 %13, %29, %45;\n\t"
            "subc.cc.u32 %14, %30, %46;\n\t"
            "subc.u32  %15, %31, %47;"
            : "=&r"(r[0]), "=&r"(r[1]), "=&r"(r[2]), "=&r"(r[3]), "=&r"(r[4]), "=&r"(r[5]), "=&r"(r[6]), "=&r"(r[7]),
          "=&r"(r[8]), "=&r"(r[9]), "=&r"(r[10]), "=&r"(r[11]), "=&r"(r[12]), "=&r"(r[13]), "=&r"(r[14]), "=&r"(r[15])
            : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(a[4]), "r"(a[5]), "r"(a[6]), "r"(a[7]), "r"(a[8]),
          "r"(a[9]), "r"(a[10]), "r"(a[11]), "r"(a[12]), "r"(a[13]), "r"(a[14]), "r"(a[15]),
              "r"(b[0]), "r"(b[1]), "r"(b[2]), "r"(b[3]), "r"(b[4]), "r"(b[5]), "r"(b[6]), "r"(b[7]), "r"(b[8]),
          "r"(b[9]), "r"(b[10]), "r"(b[11]), "r"(b[12]), "r"(b[13]), "r"(b[14]), "r"(b[15]));
#else
    int64_t c = 0;
    for (int k = 0; k < N; k++) {
        c += (int64_t)a[k] - b[k];
        r[k] = (uint32_t)c;
        c >>= 32;
    }
#endif
}

// ---- rows: N partial products on the 64-bit lanes of x (x[2k], x[2k + 1]) ----
// A row takes the N words a[0], a[2], .. of its multiplicand (every second
// one, those that fall on this vector's lanes) times b.  On the device each is
// one asm statement, since the carry flag does not outlive a statement; the
// host forms give the same words, for the unit checks of the limbs.

// x = a b
template <int N>
__host__ __device__ __forceinline__ void row_mul(uint32_t* x, const uint32_t* a, uint32_t b) {
#pragma unroll
    for (int k = 0; k < N; k++) {
        const uint64_t p = (uint64_t)a[2 * k] * b;
        x[2 * k] = (uint32_t)p;
        x[2 * k + 1] = (uint32_t)(p >> 32);
    }
}

#ifndef __CUDA_ARCH__
// the chain shared by the host forms: x + a b + carry, the carry out returned
template <int N>
inline uint32_t row_mad_host(uint32_t* x, const uint32_t* a, uint32_t b, uint32_t carry) {
    for (int k = 0; k < N; k++) {
        const uint64_t t = (uint64_t)x[2 * k + 1] << 32 | x[2 * k];
        const uint64_t p = (uint64_t)a[2 * k] * b, s = t + p, r = s + carry;
        carry = (uint32_t)(s < t) + (uint32_t)(r < s);
        x[2 * k] = (uint32_t)r;
        x[2 * k + 1] = (uint32_t)(r >> 32);
    }
    return carry;
}
#endif

// x += a b; the caller knows that nothing is carried out of the last lane
template <int N>
__host__ __device__ __forceinline__ void row_mad(uint32_t* x, const uint32_t* a, uint32_t b) {
    static_assert(N >= 1 && N <= 4, "row length");
#ifdef __CUDA_ARCH__
    if constexpr (N == 4)
        asm("mad.lo.cc.u32  %0, %8, %12, %0;\n\t"
            "madc.hi.cc.u32 %1, %8, %12, %1;\n\t"
            "madc.lo.cc.u32 %2, %9, %12, %2;\n\t"
            "madc.hi.cc.u32 %3, %9, %12, %3;\n\t"
            "madc.lo.cc.u32 %4, %10, %12, %4;\n\t"
            "madc.hi.cc.u32 %5, %10, %12, %5;\n\t"
            "madc.lo.cc.u32 %6, %11, %12, %6;\n\t"
            "madc.hi.u32    %7, %11, %12, %7;"
            : "+r"(x[0]), "+r"(x[1]), "+r"(x[2]), "+r"(x[3]), "+r"(x[4]), "+r"(x[5]), "+r"(x[6]), "+r"(x[7])
            : "r"(a[0]), "r"(a[2]), "r"(a[4]), "r"(a[6]), "r"(b));
    else if constexpr (N == 3)
        asm("mad.lo.cc.u32  %0, %6, %9, %0;\n\t"
            "madc.hi.cc.u32 %1, %6, %9, %1;\n\t"
            "madc.lo.cc.u32 %2, %7, %9, %2;\n\t"
            "madc.hi.cc.u32 %3, %7, %9, %3;\n\t"
            "madc.lo.cc.u32 %4, %8, %9, %4;\n\t"
            "madc.hi.u32    %5, %8, %9, %5;"
            : "+r"(x[0]), "+r"(x[1]), "+r"(x[2]), "+r"(x[3]), "+r"(x[4]), "+r"(x[5])
            : "r"(a[0]), "r"(a[2]), "r"(a[4]), "r"(b));
    else if constexpr (N == 2)
        asm("mad.lo.cc.u32  %0, %4, %6, %0;\n\t"
            "madc.hi.cc.u32 %1, %4, %6, %1;\n\t"
            "madc.lo.cc.u32 %2, %5, %6, %2;\n\t"
            "madc.hi.u32    %3, %5, %6, %3;"
            : "+r"(x[0]), "+r"(x[1]), "+r"(x[2]), "+r"(x[3])
            : "r"(a[0]), "r"(a[2]), "r"(b));
    else
        asm("mad.lo.cc.u32  %0, %2, %3, %0;\n\t"
            "madc.hi.u32    %1, %2, %3, %1;"
            : "+r"(x[0]), "+r"(x[1])
            : "r"(a[0]), "r"(b));
#else
    row_mad_host<N>(x, a, b, 0);
#endif
}

// x += a b, the carry out of the last lane added to c
template <int N>
__host__ __device__ __forceinline__ void row_mad_c(uint32_t* x, const uint32_t* a, uint32_t b, uint32_t& c) {
    static_assert(N >= 1 && N <= 4, "row length");
#ifdef __CUDA_ARCH__
    if constexpr (N == 4)
        asm("mad.lo.cc.u32  %0, %9, %13, %0;\n\t"
            "madc.hi.cc.u32 %1, %9, %13, %1;\n\t"
            "madc.lo.cc.u32 %2, %10, %13, %2;\n\t"
            "madc.hi.cc.u32 %3, %10, %13, %3;\n\t"
            "madc.lo.cc.u32 %4, %11, %13, %4;\n\t"
            "madc.hi.cc.u32 %5, %11, %13, %5;\n\t"
            "madc.lo.cc.u32 %6, %12, %13, %6;\n\t"
            "madc.hi.cc.u32 %7, %12, %13, %7;\n\t"
            "addc.u32       %8, %8, 0;"
            : "+r"(x[0]), "+r"(x[1]), "+r"(x[2]), "+r"(x[3]), "+r"(x[4]), "+r"(x[5]), "+r"(x[6]), "+r"(x[7]),
              "+r"(c)
            : "r"(a[0]), "r"(a[2]), "r"(a[4]), "r"(a[6]), "r"(b));
    else if constexpr (N == 3)
        asm("mad.lo.cc.u32  %0, %7, %10, %0;\n\t"
            "madc.hi.cc.u32 %1, %7, %10, %1;\n\t"
            "madc.lo.cc.u32 %2, %8, %10, %2;\n\t"
            "madc.hi.cc.u32 %3, %8, %10, %3;\n\t"
            "madc.lo.cc.u32 %4, %9, %10, %4;\n\t"
            "madc.hi.cc.u32 %5, %9, %10, %5;\n\t"
            "addc.u32       %6, %6, 0;"
            : "+r"(x[0]), "+r"(x[1]), "+r"(x[2]), "+r"(x[3]), "+r"(x[4]), "+r"(x[5]), "+r"(c)
            : "r"(a[0]), "r"(a[2]), "r"(a[4]), "r"(b));
    else if constexpr (N == 2)
        asm("mad.lo.cc.u32  %0, %5, %7, %0;\n\t"
            "madc.hi.cc.u32 %1, %5, %7, %1;\n\t"
            "madc.lo.cc.u32 %2, %6, %7, %2;\n\t"
            "madc.hi.cc.u32 %3, %6, %7, %3;\n\t"
            "addc.u32       %4, %4, 0;"
            : "+r"(x[0]), "+r"(x[1]), "+r"(x[2]), "+r"(x[3]), "+r"(c)
            : "r"(a[0]), "r"(a[2]), "r"(b));
    else
        asm("mad.lo.cc.u32  %0, %3, %4, %0;\n\t"
            "madc.hi.cc.u32 %1, %3, %4, %1;\n\t"
            "addc.u32       %2, %2, 0;"
            : "+r"(x[0]), "+r"(x[1]), "+r"(c)
            : "r"(a[0]), "r"(b));
#else
    c += row_mad_host<N>(x, a, b, 0);
#endif
}

// One limb down and the next row: e0 += x[1], and x = (x >> 64) + a b + the
// carry of that sum.  x holds the even positions of a sum whose lowest limb is
// zero and e0 is the first odd position; afterwards x holds the odd positions
// of the sum one limb lower (four lanes) and e0 starts the even ones.
__host__ __device__ __forceinline__ void row_shift_mad(uint32_t* x, uint32_t& e0, const uint32_t* a, uint32_t b) {
#ifdef __CUDA_ARCH__
    asm("add.cc.u32     %8, %8, %1;\n\t"
        "madc.lo.cc.u32 %0, %9, %13, %2;\n\t"
        "madc.hi.cc.u32 %1, %9, %13, %3;\n\t"
        "madc.lo.cc.u32 %2, %10, %13, %4;\n\t"
        "madc.hi.cc.u32 %3, %10, %13, %5;\n\t"
        "madc.lo.cc.u32 %4, %11, %13, %6;\n\t"
        "madc.hi.cc.u32 %5, %11, %13, %7;\n\t"
        "madc.lo.cc.u32 %6, %12, %13, 0;\n\t"
        "madc.hi.u32    %7, %12, %13, 0;"
        : "+r"(x[0]), "+r"(x[1]), "+r"(x[2]), "+r"(x[3]), "+r"(x[4]), "+r"(x[5]), "+r"(x[6]), "+r"(x[7]), "+r"(e0)
        : "r"(a[0]), "r"(a[2]), "r"(a[4]), "r"(a[6]), "r"(b));
#else
    const uint64_t s = (uint64_t)e0 + x[1];
    e0 = (uint32_t)s;
    for (int k = 0; k < 6; k++) x[k] = x[k + 2];
    x[6] = x[7] = 0;
    row_mad_host<4>(x, a, b, (uint32_t)(s >> 32));
#endif
}

// r = x + y[1..7]: the odd positions of a sum plus its even ones one limb
// lower (y[0] is zero)
__host__ __device__ __forceinline__ void merge_odd_even(uint32_t* r, const uint32_t* x, const uint32_t* y) {
    const uint32_t lower[8] = {y[1], y[2], y[3], y[4], y[5], y[6], y[7], 0};
    add_words<8>(r, x, lower);
}

// the modulus' limbs from position i on, as a row's multiplicand
template <class Params>
struct Modulus {
    uint32_t v[8];
    __host__ __device__ __forceinline__ Modulus() {
#pragma unroll
        for (int i = 0; i < 8; i++) v[i] = Params::P(i);
    }
};

// even += m p (even limbs), odd += m p (odd limbs), with m chosen so that
// even[0] becomes zero
template <class Params>
__host__ __device__ __forceinline__ void reduce_row(uint32_t* even, uint32_t* odd) {
    const Modulus<Params> p;
    const uint32_t m = even[0] * Params::N0;
    row_mad<4>(odd, p.v + 1, m);
    row_mad_c<4>(even, p.v, m, odd[7]);
}

// a b R^-1 mod p in [0, 2p)
template <class Params>
__host__ __device__ __forceinline__ void mul_redc(const uint32_t* a, const uint32_t* b, uint32_t* r) {
    uint32_t x[8], y[8];
    row_mul<4>(x, a, b[0]);
    row_mul<4>(y, a + 1, b[0]);
    reduce_row<Params>(x, y);
#pragma unroll
    for (int i = 1; i < 8; i += 2) {   // the vectors trade places with every limb
        row_shift_mad(x, y[0], a + 1, b[i]);
        row_mad_c<4>(y, a, b[i], x[7]);
        reduce_row<Params>(y, x);
        if (i + 1 < 8) {
            row_shift_mad(y, x[0], a + 1, b[i + 1]);
            row_mad_c<4>(x, a, b[i + 1], y[7]);
            reduce_row<Params>(x, y);
        }
    }
    merge_odd_even(r, x, y);
}

template <class Params>
__device__ __forceinline__ Fp<Params> mul(const Fp<Params>& a, const Fp<Params>& b) {
    Fp<Params> r;
    mul_redc<Params>(a.v, b.v, r.v);
    reduce_once<Params>(r.v);
    return r;
}

// Montgomery reduction of a 16-limb t < p R: t R^-1 mod p, left in [0, 2p)
// in r[0..7].  The low half is reduced as in mul_redc, the high half added at
// the end: (t + M p) / R < 2p < 2^255, so no carry is left.
template <class Params>
__host__ __device__ __forceinline__ void redc_wide(const uint32_t* t, uint32_t* r) {
    const Modulus<Params> p;
    uint32_t x[8], y[8];
#pragma unroll
    for (int k = 0; k < 8; k++) x[k] = t[k];
    uint32_t m = x[0] * Params::N0;
    row_mul<4>(y, p.v + 1, m);
    row_mad_c<4>(x, p.v, m, y[7]);
#pragma unroll
    for (int i = 1; i < 8; i += 2) {
        m = (y[0] + x[1]) * Params::N0;
        row_shift_mad(x, y[0], p.v + 1, m);
        row_mad_c<4>(y, p.v, m, x[7]);
        if (i + 1 < 8) {
            m = (x[0] + y[1]) * Params::N0;
            row_shift_mad(y, x[0], p.v + 1, m);
            row_mad_c<4>(x, p.v, m, y[7]);
        }
    }
    merge_odd_even(r, x, y);
    add_words<8>(r, r, t + 8);
}

// t = e + o 2^32, the even and odd positions of a product below 2^512
__host__ __device__ __forceinline__ void merge_wide(uint32_t* t, const uint32_t* e, const uint32_t* o) {
    const uint32_t up[16] = {0, o[0], o[1], o[2], o[3], o[4], o[5], o[6], o[7], o[8], o[9], o[10], o[11], o[12],
                             o[13], o[14]};
    add_words<16>(t, e, up);
}

// a b as a 16-limb integer.  A row reaches at most two limbs that no row
// before it wrote, so one of its two chains ends in a fresh lane and the other
// carries into a fresh limb.
__host__ __device__ __forceinline__ void mul_wide(const uint32_t* a, const uint32_t* b, uint32_t* t) {
    uint32_t e[16], o[16];
#pragma unroll
    for (int k = 8; k < 16; k++) e[k] = o[k] = 0;
    row_mul<4>(e, a, b[0]);
    row_mul<4>(o, a + 1, b[0]);
#pragma unroll
    for (int i = 1; i < 8; i++) {
        if (i & 1) {   // a's even words fall on odd positions
            row_mad_c<4>(o + i - 1, a, b[i], o[i + 7]);
            row_mad<4>(e + i + 1, a + 1, b[i]);
        } else {
            row_mad_c<4>(e + i, a, b[i], e[i + 8]);
            row_mad<4>(o + i, a + 1, b[i]);
        }
    }
    merge_wide(t, e, o);
}

// t += sum a_i^2 2^(64 i), nothing carried out of limb 15
__host__ __device__ __forceinline__ void sqr_diagonal(uint32_t* t, const uint32_t* a) {
#ifdef __CUDA_ARCH__
    asm("mad.lo.cc.u32  %0, %16, %16, %0;\n\t"
        "madc.hi.cc.u32 %1, %16, %16, %1;\n\t"
        "madc.lo.cc.u32 %2, %17, %17, %2;\n\t"
        "madc.hi.cc.u32 %3, %17, %17, %3;\n\t"
        "madc.lo.cc.u32 %4, %18, %18, %4;\n\t"
        "madc.hi.cc.u32 %5, %18, %18, %5;\n\t"
        "madc.lo.cc.u32 %6, %19, %19, %6;\n\t"
        "madc.hi.cc.u32 %7, %19, %19, %7;\n\t"
        "madc.lo.cc.u32 %8, %20, %20, %8;\n\t"
        "madc.hi.cc.u32 %9, %20, %20, %9;\n\t"
        "madc.lo.cc.u32 %10, %21, %21, %10;\n\t"
        "madc.hi.cc.u32 %11, %21, %21, %11;\n\t"
        "madc.lo.cc.u32 %12, %22, %22, %12;\n\t"
        "madc.hi.cc.u32 %13, %22, %22, %13;\n\t"
        "madc.lo.cc.u32 %14, %23, %23, %14;\n\t"
        "madc.hi.u32    %15, %23, %23, %15;"
        : "+r"(t[0]), "+r"(t[1]), "+r"(t[2]), "+r"(t[3]), "+r"(t[4]), "+r"(t[5]), "+r"(t[6]), "+r"(t[7]),
          "+r"(t[8]), "+r"(t[9]), "+r"(t[10]), "+r"(t[11]), "+r"(t[12]), "+r"(t[13]), "+r"(t[14]), "+r"(t[15])
        : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(a[4]), "r"(a[5]), "r"(a[6]), "r"(a[7]));
#else
    uint32_t carry = 0;
    for (int i = 0; i < 8; i++) {
        const uint64_t x = (uint64_t)t[2 * i + 1] << 32 | t[2 * i], p = (uint64_t)a[i] * a[i], s = x + p, r = s + carry;
        carry = (uint32_t)(s < x) + (uint32_t)(r < s);
        t[2 * i] = (uint32_t)r;
        t[2 * i + 1] = (uint32_t)(r >> 32);
    }
#endif
}

// a^2 R^-1 mod p, left in [0, 2p) in r[0..7] (separated operand scanning):
// the 28 cross products a_i a_j (i < j) once, doubled, plus the 8 squares
// a_i^2, then a Montgomery reduction of the 16-limb square.  36 limb products
// and 64 for the reduction against 128: the same REDC value (a^2 + M p) / R, M
// being the unique multiple in [0, R), so the result is identical to
// mul(a, a).
template <class Params>
__host__ __device__ __forceinline__ void sqr_redc(const uint32_t* a, uint32_t* r) {
    // a_i a_j at position i + j; o[k] is position k + 1
    uint32_t e[16], o[16], t[16];
#pragma unroll
    for (int k = 0; k < 16; k++) e[k] = o[k] = 0;
    row_mul<4>(o, a + 1, a[0]);                // 1, 3, 5, 7
    row_mul<3>(e + 2, a + 2, a[0]);            // 2, 4, 6
    row_mad_c<3>(o + 2, a + 2, a[1], o[8]);    // 3, 5, 7
    row_mad<3>(e + 4, a + 3, a[1]);            // 4, 6, 8
    row_mad<3>(o + 4, a + 3, a[2]);            // 5, 7, 9
    row_mad_c<2>(e + 6, a + 4, a[2], e[10]);   // 6, 8
    row_mad_c<2>(o + 6, a + 4, a[3], o[10]);   // 7, 9
    row_mad<2>(e + 8, a + 5, a[3]);            // 8, 10
    row_mad<2>(o + 8, a + 5, a[4]);            // 9, 11
    row_mad_c<1>(e + 10, a + 6, a[4], e[12]);  // 10
    row_mad_c<1>(o + 10, a + 6, a[5], o[12]);  // 11
    row_mad<1>(e + 12, a + 7, a[5]);           // 12
    row_mad<1>(o + 12, a + 7, a[6]);           // 13
    merge_wide(t, e, o);
    // double (the cross sum is below 2^511, so the shift loses nothing)
#pragma unroll
    for (int k = 15; k >= 1; k--) t[k] = (t[k] << 1) | (t[k - 1] >> 31);
    // t[0] is zero: no cross product lands on limb 0
    sqr_diagonal(t, a);
    redc_wide<Params>(t, r);
}

template <class Params>
__device__ __forceinline__ Fp<Params> sqr(const Fp<Params>& a) {
    Fp<Params> r;
    sqr_redc<Params>(a.v, r.v);
    reduce_once<Params>(r.v);
    return r;
}

// Montgomery -> standard form: a R^-1, the reduction alone
template <class Params>
__device__ __forceinline__ Fp<Params> from_mont(const Fp<Params>& a) {
    uint32_t t[16];
#pragma unroll
    for (int i = 0; i < 8; i++) {
        t[i] = a.v[i];
        t[i + 8] = 0;
    }
    Fp<Params> r;
    redc_wide<Params>(t, r.v);
    reduce_once<Params>(r.v);
    return r;
}

typedef Fp<FrParams> Fr;
typedef Fp<FqParams> Fq;

// ---- Fq2 = Fq[u]/(u^2 + 1) ----
struct __align__(16) Fq2 {
    Fq c0, c1;
    __device__ __forceinline__ static Fq2 zero() { return {Fq::zero(), Fq::zero()}; }
    __device__ __forceinline__ static Fq2 one() { return {Fq::one(), Fq::zero()}; }
    __device__ __forceinline__ bool is_zero() const { return c0.is_zero() && c1.is_zero(); }
};

__device__ __forceinline__ Fq2 add(const Fq2& a, const Fq2& b) { return {add(a.c0, b.c0), add(a.c1, b.c1)}; }
__device__ __forceinline__ Fq2 sub(const Fq2& a, const Fq2& b) { return {sub(a.c0, b.c0), sub(a.c1, b.c1)}; }
__device__ __forceinline__ Fq2 neg(const Fq2& a) { return {neg(a.c0), neg(a.c1)}; }
__device__ __forceinline__ Fq2 dbl(const Fq2& a) { return {dbl(a.c0), dbl(a.c1)}; }
// (a b + c d) R^-1 mod p, left in [0, 2p), with one Montgomery reduction
// instead of two, row by row as in mul_redc with two products a row.  Operands
// up to p: the running value stays below 3 p 2^32 < 2^288 and the result below
// 2p.
template <class Params>
__host__ __device__ __forceinline__ void mul_add_redc(const uint32_t* a, const uint32_t* b, const uint32_t* c,
                                                      const uint32_t* d, uint32_t* r) {
    uint32_t x[8], y[8];
    row_mul<4>(x, a, b[0]);
    row_mul<4>(y, a + 1, b[0]);
    row_mad<4>(y, c + 1, d[0]);
    row_mad_c<4>(x, c, d[0], y[7]);
    reduce_row<Params>(x, y);
#pragma unroll
    for (int i = 1; i < 8; i += 2) {
        row_shift_mad(x, y[0], a + 1, b[i]);
        row_mad_c<4>(y, a, b[i], x[7]);
        row_mad<4>(x, c + 1, d[i]);
        row_mad_c<4>(y, c, d[i], x[7]);
        reduce_row<Params>(y, x);
        if (i + 1 < 8) {
            row_shift_mad(y, x[0], a + 1, b[i + 1]);
            row_mad_c<4>(x, a, b[i + 1], y[7]);
            row_mad<4>(y, c + 1, d[i + 1]);
            row_mad_c<4>(x, c, d[i + 1], y[7]);
            reduce_row<Params>(x, y);
        }
    }
    merge_odd_even(r, x, y);
}

// (a b - c d) R^-1 mod p, left in [0, 2p): a b + (p - c) d
template <class Params>
__host__ __device__ __forceinline__ void mul_sub_redc(const uint32_t* a, const uint32_t* b, const uint32_t* c,
                                                      const uint32_t* d, uint32_t* r) {
    const Modulus<Params> p;
    uint32_t n[8];
    sub_words<8>(n, p.v, c);
    mul_add_redc<Params>(a, b, n, d, r);
}

// a b - c d in Fq with one reduction (mul_sub_redc)
__device__ __forceinline__ Fq mul_sub(const Fq& a, const Fq& b, const Fq& c, const Fq& d) {
    Fq r;
    mul_sub_redc<FqParams>(a.v, b.v, c.v, d.v, r.v);
    reduce_once<FqParams>(r.v);
    return r;
}

// (a0 + a1 u)(b0 + b1 u) with two Montgomery reductions instead of three
// (Karatsuba with the reduction deferred, as in Aranha et al., "Faster explicit
// formulas for computing pairings over ordinary curves", 2011): the three
// 512-bit products t0 = a0 b0, t1 = a1 b1, m = (a0 + a1)(b0 + b1) with the
// sums taken as integers (below 2q), then
//   c1 = m - t0 - t1 = a0 b1 + a1 b0          (exact, below 2 q^2)
//   c0 = t0 + q^2 - t1 = a0 b0 - a1 b1 mod q  (positive, below 2 q^2),
// and one reduction each (inputs below q R give results below 2q).  The
// coordinates equal those of three reduced products once brought below q.
// Inputs below q.  Host-callable for the unit check of the limbs.
__host__ __device__ __forceinline__ void fq2_mul_redc(const uint32_t* a0, const uint32_t* a1, const uint32_t* b0,
                                                      const uint32_t* b1, uint32_t* r0, uint32_t* r1) {
    uint32_t t0[16], t1[16], m[16], sa[8], sb[8], q2[16];
    add_words<8>(sa, a0, a1);
    add_words<8>(sb, b0, b1);
    mul_wide(a0, b0, t0);
    mul_wide(a1, b1, t1);
    mul_wide(sa, sb, m);
    sub_words<16>(m, m, t0);
    sub_words<16>(m, m, t1);
#pragma unroll
    for (int i = 0; i < 16; i++) q2[i] = FqParams::P2W(i);
    add_words<16>(t0, t0, q2);
    sub_words<16>(t0, t0, t1);
    redc_wide<FqParams>(t0, r0);
    redc_wide<FqParams>(m, r1);
}

__device__ __forceinline__ Fq2 mul(const Fq2& a, const Fq2& b) {
    Fq2 r;
    fq2_mul_redc(a.c0.v, a.c1.v, b.c0.v, b.c1.v, r.c0.v, r.c1.v);
    reduce_once<FqParams>(r.c0.v);
    reduce_once<FqParams>(r.c1.v);
    return r;
}
// a b - c d in Fq2: two products and a difference
__device__ __forceinline__ Fq2 mul_sub(const Fq2& a, const Fq2& b, const Fq2& c, const Fq2& d) {
    return sub(mul(a, b), mul(c, d));
}
// (a0 + a1 u)^2 = (a0 + a1)(a0 - a1) + 2 a0 a1 u
__device__ __forceinline__ Fq2 sqr(const Fq2& a) {
    Fq p = mul(add(a.c0, a.c1), sub(a.c0, a.c1));
    Fq q = mul(a.c0, a.c1);
    return {p, dbl(q)};
}

// ---- product policy: inlined, or one out-of-line copy ----
// The G1 accumulate, the NTT and the groups of lanes (lanes.cuh) keep every
// product inlined.  The G2 accumulate calls one out-of-line Fq2 product
// (operands by value, so they stay in registers): ten inlined ones overflow the
// instruction cache (2.44 against 2.18 ms for a 2^18 MSM).  So do the
// window tables, the key generator and the rare doubling inside an addition,
// where code size counts and speed does not.
template <class Params>
__device__ __noinline__ Fp<Params> mul_ool(Fp<Params> a, Fp<Params> b) {
    return mul(a, b);
}

template <bool INL, class Params>
__device__ __forceinline__ Fp<Params> fmul(const Fp<Params>& a, const Fp<Params>& b) {
    if constexpr (INL) return mul(a, b);
    else return mul_ool(a, b);
}
template <bool INL, class Params>
__device__ __forceinline__ Fp<Params> fsqr(const Fp<Params>& a) {
    if constexpr (INL) return sqr(a);
    else return mul_ool(a, a);
}

// Out-of-line copies that hold several independent products.  A warp issues
// in order and a CIOS product is one long carry chain, so a lone out-of-line
// product leaves the pipe idle for part of its latency; two or three chains in
// one body are scheduled side by side.  The point formulas over G1 that run out
// of line (window tables, rare doublings) group their independent products this way.
template <class F>
struct Two {
    F a, b;
};
template <class F>
struct Three {
    F a, b, c;
};

template <class Params>
__device__ __noinline__ Two<Fp<Params>> mul2_ool(Fp<Params> a0, Fp<Params> b0, Fp<Params> a1, Fp<Params> b1) {
    return {mul(a0, b0), mul(a1, b1)};
}
template <class Params>
__device__ __noinline__ Three<Fp<Params>> mul3_ool(Fp<Params> a0, Fp<Params> b0, Fp<Params> a1, Fp<Params> b1,
                                                   Fp<Params> a2, Fp<Params> b2) {
    return {mul(a0, b0), mul(a1, b1), mul(a2, b2)};
}
// an Fq2 product is already three independent Fq products (Karatsuba)
static __device__ __noinline__ Fq2 fq2_mul_ool(Fq2 a, Fq2 b) { return mul(a, b); }
static __device__ __noinline__ Fq2 fq2_sqr_ool(Fq2 a) { return sqr(a); }

template <bool INL>
__device__ __forceinline__ Fq2 fmul(const Fq2& a, const Fq2& b) {
    if constexpr (INL) return mul(a, b);
    else return fq2_mul_ool(a, b);
}
template <bool INL>
__device__ __forceinline__ Fq2 fsqr(const Fq2& a) {
    if constexpr (INL) return sqr(a);
    else return fq2_sqr_ool(a);
}

// r0 = a0 b0, r1 = a1 b1 (and r2 = a2 b2), independent products side by side
template <bool INL, class Params>
__device__ __forceinline__ void fmul2(const Fp<Params>& a0, const Fp<Params>& b0, const Fp<Params>& a1,
                                      const Fp<Params>& b1, Fp<Params>& r0, Fp<Params>& r1) {
    if constexpr (INL) {
        r0 = mul(a0, b0);
        r1 = mul(a1, b1);
    } else {
        Two<Fp<Params>> t = mul2_ool(a0, b0, a1, b1);
        r0 = t.a;
        r1 = t.b;
    }
}
template <bool INL, class Params>
__device__ __forceinline__ void fmul3(const Fp<Params>& a0, const Fp<Params>& b0, const Fp<Params>& a1,
                                      const Fp<Params>& b1, const Fp<Params>& a2, const Fp<Params>& b2,
                                      Fp<Params>& r0, Fp<Params>& r1, Fp<Params>& r2) {
    if constexpr (INL) {
        r0 = mul(a0, b0);
        r1 = mul(a1, b1);
        r2 = mul(a2, b2);
    } else {
        Three<Fp<Params>> t = mul3_ool(a0, b0, a1, b1, a2, b2);
        r0 = t.a;
        r1 = t.b;
        r2 = t.c;
    }
}
template <bool INL>
__device__ __forceinline__ void fmul2(const Fq2& a0, const Fq2& b0, const Fq2& a1, const Fq2& b1, Fq2& r0, Fq2& r1) {
    r0 = fmul<INL>(a0, b0);
    r1 = fmul<INL>(a1, b1);
}
template <bool INL>
__device__ __forceinline__ void fmul3(const Fq2& a0, const Fq2& b0, const Fq2& a1, const Fq2& b1, const Fq2& a2,
                                      const Fq2& b2, Fq2& r0, Fq2& r1, Fq2& r2) {
    r0 = fmul<INL>(a0, b0);
    r1 = fmul<INL>(a1, b1);
    r2 = fmul<INL>(a2, b2);
}

// a^(p-2) by right-to-left square-and-multiply (Fermat); 0 maps to 0.  Used
// off the hot path (table building), so it calls the out-of-line product.
template <class Params>
__device__ Fp<Params> inv(const Fp<Params>& a) {
    Fp<Params> r = Fp<Params>::one(), b = a;
#pragma unroll
    for (int limb = 0; limb < 8; limb++) {
        uint32_t e = Params::P(limb) - (limb == 0 ? 2u : 0u);
        for (int bit = 0; bit < 32; bit++) {
            if (e & 1u) r = mul_ool(r, b);
            b = mul_ool(b, b);
            e >>= 1;
        }
    }
    return r;
}

// 1/(c0 + c1 u) = (c0 - c1 u) / (c0^2 + c1^2)
__device__ __forceinline__ Fq2 inv(const Fq2& a) {
    Fq n = inv(add(mul_ool(a.c0, a.c0), mul_ool(a.c1, a.c1)));
    return {mul_ool(a.c0, n), neg(mul_ool(a.c1, n))};
}

// ---- 128-bit vector loads / stores of 32-byte elements ----
template <class T>
__device__ __forceinline__ T load32(const T* p) {
    static_assert(sizeof(T) == 32, "32-byte element");
    const uint4* q = reinterpret_cast<const uint4*>(p);
    uint4 lo = q[0], hi = q[1];
    T r;
    r.v[0] = lo.x; r.v[1] = lo.y; r.v[2] = lo.z; r.v[3] = lo.w;
    r.v[4] = hi.x; r.v[5] = hi.y; r.v[6] = hi.z; r.v[7] = hi.w;
    return r;
}
template <class T>
__device__ __forceinline__ void store32(T* p, const T& x) {
    uint4* q = reinterpret_cast<uint4*>(p);
    q[0] = make_uint4(x.v[0], x.v[1], x.v[2], x.v[3]);
    q[1] = make_uint4(x.v[4], x.v[5], x.v[6], x.v[7]);
}

}  // namespace g16d
