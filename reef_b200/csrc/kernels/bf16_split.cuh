// fp32 products on the tensor cores without giving up a bit of the operands: an fp32 value is the exact sum of three bf16
// values (8 + 8 + 8 significand bits), a product of two values the sum of nine bf16 products, each of them exact in fp32.
// Six of the nine are computed; the three left out together stay below 2^-26 of |a b|, under half of what one fp32
// rounding loses.
//
// That holds for the values that three bf16 values can carry.  bf16 has the exponents of fp32, but from 3.3962e38 on a
// finite value (up to 3.4028e38) rounds to infinity, and the remainders of an infinity are NaN, also where fp32 instructions
// would give infinity.  A sum with such an operand always ends as infinity or NaN: whoever computes sums this way looks at
// each result once and repeats it with fp32 instructions where it is not finite (split_sum_lost).  At the other end, of
// |x| below 2^-110 what lies under 2^-134 is dropped.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

namespace reef {

// an operand was beyond what bf16 carries, or the sum itself is not finite
__device__ __forceinline__ bool split_sum_lost(float x) { return !(fabsf(x) <= 3.402823466e38f); }

// x = the exact sum of three bf16 values, two values of x at a time (first in the lower half)
struct Bf16Triple {
    uint32_t h, m, l;
};
__device__ __forceinline__ Bf16Triple bf16_split(float x, float y) {
    Bf16Triple r;
    // x - h as h * -1 + x with a bf16 operand: no unpacking (two instructions a value less), and exact, as the subtraction is
    // (a loop of splits alone 389 -> 319 cycles a slice of 16 x 32)
    asm("{\n\t.reg .b16 p, q, n;\n\tmov.b16 n, 0xBF80;\n\tcvt.rn.bf16x2.f32 %0, %2, %1;\n\tmov.b32 {p, q}, %0;\n\t"
        "fma.rn.f32.bf16 %1, p, n, %1;\n\tfma.rn.f32.bf16 %2, q, n, %2;\n\t}"
        : "=&r"(r.h), "+f"(x), "+f"(y));
    asm("{\n\t.reg .b16 p, q, n;\n\tmov.b16 n, 0xBF80;\n\tcvt.rn.bf16x2.f32 %0, %2, %1;\n\tmov.b32 {p, q}, %0;\n\t"
        "fma.rn.f32.bf16 %1, p, n, %1;\n\tfma.rn.f32.bf16 %2, q, n, %2;\n\t}"
        : "=&r"(r.m), "+f"(x), "+f"(y));
    asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(r.l) : "f"(y), "f"(x));
    return r;
}
__device__ __forceinline__ void mma_bf16(float (&d)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
    asm("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"
        : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
        : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}
// the same from zero: no registers to clear
__device__ __forceinline__ void mma_bf16_zero(float (&d)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
    asm("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%10, %10, %10, %10};"
        : "=f"(d[0]), "=f"(d[1]), "=f"(d[2]), "=f"(d[3])
        : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1), "f"(0.f));
}

// d[i] = the product of fragments a and b[i], N of them side by side (the multiplications into one accumulator depend on one
// another).  The five small products come first, the large one on top: the tensor core truncates what it adds, at the
// size of the sum so far, so the order leaves one truncation at full size.
template <int N>
__device__ __forceinline__ void mma_split(float (&d)[N][4], const Bf16Triple (&a)[4], const Bf16Triple (&b0)[N], const Bf16Triple (&b1)[N]) {
#pragma unroll
    for (int i = 0; i < N; i++) {
        d[i][0] = d[i][1] = d[i][2] = d[i][3] = 0.f;
        mma_bf16(d[i], a[0].l, a[1].l, a[2].l, a[3].l, b0[i].h, b1[i].h);
    }
#pragma unroll
    for (int i = 0; i < N; i++) mma_bf16(d[i], a[0].h, a[1].h, a[2].h, a[3].h, b0[i].l, b1[i].l);
#pragma unroll
    for (int i = 0; i < N; i++) mma_bf16(d[i], a[0].m, a[1].m, a[2].m, a[3].m, b0[i].m, b1[i].m);
#pragma unroll
    for (int i = 0; i < N; i++) mma_bf16(d[i], a[0].m, a[1].m, a[2].m, a[3].m, b0[i].h, b1[i].h);
#pragma unroll
    for (int i = 0; i < N; i++) mma_bf16(d[i], a[0].h, a[1].h, a[2].h, a[3].h, b0[i].m, b1[i].m);
#pragma unroll
    for (int i = 0; i < N; i++) mma_bf16(d[i], a[0].h, a[1].h, a[2].h, a[3].h, b0[i].h, b1[i].h);
}

}  // namespace reef
