// pair_math.h -- paired single-precision sums for the 8x8 transforms.
//
// sm_100a adds two f32 pairs in one instruction (add.rn.f32x2); each half
// is the IEEE round-to-nearest sum of its own operands, the value
// __fadd_rn gives. The transforms add their terms in pairs and keep every
// product scalar (__fmul_rn, mul.rn.f32), which is never contracted into a
// multiply-add: the crate's two roundings per term stay, with three
// instructions for two terms instead of four.
//
// Paired products (mul.rn.f32x2) are not used: measured on a B200, a
// paired product feeding a paired sum was at times fused into a paired
// multiply-add by the code generator, even with contraction turned off,
// which changes the last bit of the sum.
// A pair is a 64-bit value, low half first.
#pragma once

#include <cstdint>

namespace prores {

__device__ __forceinline__ uint64_t pair_of(float lo, float hi) {
    uint64_t r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
    return r;
}

__device__ __forceinline__ void pair_split(uint64_t v, float &lo, float &hi) {
    asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(v));
}

__device__ __forceinline__ uint64_t pair_add(uint64_t a, uint64_t b) {
    uint64_t r;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}

// a - b: each half the sum of a and the exact negative of b.
__device__ __forceinline__ uint64_t pair_sub(uint64_t a, uint64_t b) {
    uint64_t r;
    asm("sub.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}

// The 8-point basis T[x][u] (dct_basis) in single precision has the cosine's
// symmetries bit for bit (every context checks it: dct_basis_mirrors):
// T[7 - x][u] = (-1)^u T[x][u], and for even u T[3 - x][u] = T[x][u] (u = 0, 4)
// or -T[x][u] (u = 2, 6). So in out[x] = sum_u F[u] T[x][u] the eight products
// of one u are two (u even) or four (u odd) products and their exact negatives,
// and with the outputs paired as (0, 1), (7, 6), (3, 2), (4, 5) every pair adds
// or subtracts one of two product pairs: 24 products and 32 paired sums for 8
// outputs, each output's terms in the same order and rounded alike.
struct Pairs8 {
    uint64_t o01, o76, o32, o45;
};

// Adds term u of value f; `T` is the basis in constant memory, [8 x + u].
template <int u, bool first>
__device__ __forceinline__ void pairs_term(Pairs8 &o, float f, const float *T) {
    const uint64_t p01 = pair_of(__fmul_rn(f, T[u]), __fmul_rn(f, T[8 + u]));
    if constexpr (first) {
        // 0 + p is p (but for the sign of a zero, which no later step sees).
        static_assert(u == 0);
        o.o01 = o.o76 = o.o32 = o.o45 = p01;
    } else if constexpr (u % 2 == 0) {
        o.o01 = pair_add(o.o01, p01);
        o.o76 = pair_add(o.o76, p01);
        o.o32 = u == 4 ? pair_add(o.o32, p01) : pair_sub(o.o32, p01);
        o.o45 = u == 4 ? pair_add(o.o45, p01) : pair_sub(o.o45, p01);
    } else {
        const uint64_t p32 = pair_of(__fmul_rn(f, T[24 + u]), __fmul_rn(f, T[16 + u]));
        o.o01 = pair_add(o.o01, p01);
        o.o76 = pair_sub(o.o76, p01);
        o.o32 = pair_add(o.o32, p32);
        o.o45 = pair_sub(o.o45, p32);
    }
}

}  // namespace prores
