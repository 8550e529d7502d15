// mul_int.cuh -- an FP64 multiply on the integer pipes.
#pragma once
#include <cstdint>

namespace magpy {

// a * b rounded to nearest even by integer multiplies: the same bits as the
// FP64 multiply for operands that are zero or normal with exponents such that
// a non-zero product is at least 2^-766 and at most 2^1000, and a product with
// a zero operand has the other one below 2^255.  (Zero has exponent field 0: its
// product's field comes out below 256, which no non-zero product's does.)
// The FP64 pipe takes 19 cycles of an SM per warp instruction on two different
// registers (16 on one, as in a conversion or a square), this takes 14 of the
// integer pipes, so beside FP64 additions it is free: multiply and add 19 cycles
// the pair, 38 with both on the FP64 pipe.
__device__ __forceinline__ double mul_int(double a, double b)
{
    const uint32_t ah = __double2hiint(a), a0 = __double2loint(a);
    const uint32_t bh = __double2hiint(b), bl = __double2loint(b);
    // mantissas: a as 21 + 32 bits, b shifted to 32 + 32; the product's top
    // bit is bit 116 or 115
    const uint32_t a1 = (ah & 0x000fffffu) | 0x00100000u;
    const uint32_t b1 = __funnelshift_l(bl, bh, 11) | 0x80000000u, b0 = bl << 11;
    const uint64_t ll = (uint64_t)a0 * b0;
    const uint64_t m1 = (uint64_t)a0 * b1 + (ll >> 32);
    const uint64_t m2 = (uint64_t)a1 * b0 + (uint32_t)m1;
    const uint64_t hi = (uint64_t)a1 * b1 + ((m1 >> 32) + (m2 >> 32));
    const uint32_t hh = (uint32_t)(hi >> 32), hl = (uint32_t)hi, lh = (uint32_t)m2,
                   l0 = (uint32_t)ll;
    const uint32_t sh = (hh >> 20) ^ 1u;  // normalise
    const uint32_t mh = __funnelshift_l(hl, hh, sh), ml = __funnelshift_l(lh, hl, sh);
    const uint32_t rest = __funnelshift_l(l0, lh, sh) | (l0 ? 1u : 0u);
    // the implicit bit adds one to the exponent field
    const uint32_t e = (ah & 0x7ff00000u) + (bh & 0x7ff00000u) - (1023u << 20) - (sh << 20);
    // half the last place rounds up with an odd mantissa: carry of the rest
    const uint32_t half = (ml & 1u) + 0x7fffffffu;
    uint32_t rl, rh;
    asm("{\n\t.reg .u32 t;\n\tadd.cc.u32 t, %2, %3;\n\taddc.cc.u32 %0, %4, 0;\n\t"
        "addc.u32 %1, %5, %6;\n\t}"
        : "=r"(rl), "=r"(rh)
        : "r"(rest), "r"(half), "r"(ml), "r"(mh), "r"(e));
    const bool zero = (int)e < (256 << 20);
    rl = zero ? 0u : rl;
    rh = zero ? 0u : rh;
    return __hiloint2double(rh | ((ah ^ bh) & 0x80000000u), rl);
}

}  // namespace magpy
