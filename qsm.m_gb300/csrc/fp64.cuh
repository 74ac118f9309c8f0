// FP64 multiplication beside the FP64 pipe.
//
// This GPU has one FP64 unit per SM, which takes ~19 cycles per warp
// instruction whatever its active lanes (0.50 T operations/s measured, 1/74 of
// FP32), so an FP64 kernel leaves the integer pipes idle nearly all the time.
// The functions here compute the IEEE 754 binary64 product (round to nearest,
// ties to even) from the operands' encodings in integer arithmetic: the bits of
// the hardware instruction, from the other pipes.  Zeros are handled too;
// subnormals, infinities, NaNs and values near the ends of the exponent range
// take the hardware instruction.  Measured on full SMs (cycles per warp
// operation and scheduler): a hardware add or multiply 81, an integer multiply
// 68, an integer multiply feeding a hardware add 83 for the pair against 162 for
// two hardware instructions: the multiply is free.  Its latency is longer than
// the instruction's 64 cycles, so kernels with a warp or two per scheduler keep
// the hardware multiply.  qsm_fp_convert_check compares both forms.
#pragma once
#include <stdint.h>
#include <string.h>

namespace qsm {

// A constant factor (uniform over a kernel).  For FP32 the factor itself.
template <typename T>
struct KMul {
    T w;
};

// For FP64 also its significand left-justified in 64 bits (wh:wl), its sign and
// exponent as the word k to add to a product's high word, its sign s; span is
// the width of the exponent window of the integer way (0: always the hardware
// multiply).
template <>
struct KMul<double> {
    double w;
    uint32_t wl, wh, k, s, span;
};

inline KMul<float> make_kmul(float w) { return KMul<float>{w}; }
inline KMul<double> make_kmul(double w)
{
    uint64_t b;
    memcpy(&b, &w, sizeof b);
    const int e = (int)((b >> 52) & 0x7ff) - 1023;
    const uint64_t m = ((b & 0xfffffffffffffull) | (1ull << 52)) << 11;
    KMul<double> c;
    c.w = w;
    c.wl = (uint32_t)m;
    c.wh = (uint32_t)(m >> 32);
    c.k = ((uint32_t)e << 20) + ((uint32_t)(b >> 32) & 0x80000000u);
    c.s = (uint32_t)(b >> 32) & 0x80000000u;
    c.span = e > -100 && e < 100 ? 1792u : 0u;
    return c;
}

#ifdef __CUDACC__

// The rest of the range, out of line: as an inlined alternative the compiler
// predicates the hardware instruction, and an FP64 instruction takes its slot in
// the pipe with every lane off (256^3 FP64 solve: 40.2 ms inlined, 35.6 so).
static __device__ __noinline__ double fp64_mul_hw(double a, double b) { return __dmul_rn(a, b); }

__device__ __forceinline__ uint64_t mad_wide(uint32_t a, uint32_t b, uint64_t c)
{
    uint64_t r;
    asm("mad.wide.u32 %0, %1, %2, %3;" : "=l"(r) : "r"(a), "r"(b), "l"(c));
    return r;
}

// Rounds the 117-bit product of two significands (W in [2^63, 2^64) times M in
// [2^52, 2^53)), given as hi:l1:l0, and assembles it with the sign and exponent
// word base (the exponent of a product in [1, 2), less one, since the leading
// bit of the significand adds one).
__device__ __forceinline__ double fp64_round_product(uint64_t hi, uint32_t l1, uint32_t l0, uint32_t base)
{
    const uint32_t h0 = (uint32_t)hi, h1 = (uint32_t)(hi >> 32);
    const uint32_t s = (h1 >> 20) ^ 1u;  // significands' product below 2: one place left
    const uint32_t g1 = __funnelshift_l(h0, h1, s), g0 = __funnelshift_l(l1, h0, s), r1 = __funnelshift_l(l0, l1, s),
                   r0 = l0 << s;
    const uint32_t odd = (r0 != 0u ? 1u : 0u) | (g0 & 1u);  // breaks a tie upwards
    const uint32_t b = base - (s << 20);
    uint32_t o0, o1;
    asm("{\n\t.reg .u32 d;\n\tadd.cc.u32 d, %2, %3;\n\taddc.cc.u32 %0, %4, 0;\n\taddc.u32 %1, %5, %6;\n\t}"
        : "=r"(o0), "=r"(o1)
        : "r"(r1), "r"(0x7fffffffu + odd), "r"(g0), "r"(g1), "r"(b));
    return __hiloint2double((int)o1, (int)o0);
}

__device__ __forceinline__ float operator*(const KMul<float> &c, float b) { return c.w * b; }

__device__ __forceinline__ double operator*(const KMul<double> &c, double b)
{
    const uint32_t bh = (uint32_t)__double2hiint(b), bl = (uint32_t)__double2loint(b);
    if (((bh >> 20) & 0x7ffu) - 128u >= c.span) {
        if (((bh << 1) | bl) == 0u && c.span) return __hiloint2double((int)((bh ^ c.s) & 0x80000000u), 0);
        return fp64_mul_hw(c.w, b);
    }
    const uint32_t mh = (bh & 0xfffffu) | 0x100000u;
    const uint64_t ll = (uint64_t)c.wl * bl;
    const uint64_t t = mad_wide(c.wh, bl, ll >> 32);
    const uint64_t u = mad_wide(c.wl, mh, (uint64_t)(uint32_t)t);
    const uint64_t hi = mad_wide(c.wh, mh, t >> 32) + (u >> 32);
    return fp64_round_product(hi, (uint32_t)u, (uint32_t)ll, (bh & 0xfff00000u) + c.k);
}

// a * b of two variables
__device__ __forceinline__ float xmul(float a, float b) { return a * b; }

__device__ __forceinline__ double xmul(double a, double b)
{
    const uint32_t ah = (uint32_t)__double2hiint(a), al = (uint32_t)__double2loint(a);
    const uint32_t bh = (uint32_t)__double2hiint(b), bl = (uint32_t)__double2loint(b);
    const uint32_t ea = (ah >> 20) & 0x7ffu, eb = (bh >> 20) & 0x7ffu;
    // both exponents within 2^+-480: no product near the range's ends
    if (ea - 543u >= 960u || eb - 543u >= 960u) {
        const bool za = ((ah << 1) | al) == 0u, zb = ((bh << 1) | bl) == 0u;
        if ((za && eb < 0x7ffu) || (zb && ea < 0x7ffu)) return __hiloint2double((int)((ah ^ bh) & 0x80000000u), 0);
        return fp64_mul_hw(a, b);
    }
    const uint32_t wh = 0x80000000u | __funnelshift_l(al, ah & 0xfffffu, 11), wl = al << 11;
    const uint32_t mh = (bh & 0xfffffu) | 0x100000u;
    const uint64_t ll = (uint64_t)wl * bl;
    const uint64_t t = mad_wide(wh, bl, ll >> 32);
    const uint64_t u = mad_wide(wl, mh, (uint64_t)(uint32_t)t);
    const uint64_t hi = mad_wide(wh, mh, t >> 32) + (u >> 32);
    return fp64_round_product(hi, (uint32_t)u, (uint32_t)ll,
                              (ah & 0xfff00000u) + (bh & 0xfff00000u) - 0x3ff00000u);
}

// a * 2^E, E small: the exponent field plus E
template <int E>
__device__ __forceinline__ float scale2(float a)
{
    return a * (E < 0 ? 1.0f / (float)(1 << (E < 0 ? -E : 0)) : (float)(1 << (E < 0 ? 0 : E)));
}
template <int E>
__device__ __forceinline__ double scale2(double a)
{
    const uint32_t h = (uint32_t)__double2hiint(a), l = (uint32_t)__double2loint(a);
    if (((h >> 20) & 0x7ffu) - 128u >= 1792u) {
        if (((h << 1) | l) == 0u) return a;
        return fp64_mul_hw(a, E < 0 ? 1.0 / (double)(1 << (E < 0 ? -E : 0)) : (double)(1 << (E < 0 ? 0 : E)));
    }
    return __hiloint2double((int)(h + ((uint32_t)E << 20)), (int)l);
}

#endif  // __CUDACC__

}  // namespace qsm
