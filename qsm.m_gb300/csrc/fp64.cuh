// FP64 multiplication, and the quotient of a constant and a square root, beside
// the FP64 pipe.
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

// x > b for b >= 0 and x not negative (a sum of squares), on the encodings
__device__ __forceinline__ bool above(float x, float b) { return x > b; }
__device__ __forceinline__ bool above(double x, double b)
{
    const long long m = __double_as_longlong(x);
    return m > __double_as_longlong(b) && m <= 0x7ff0000000000000ll;  // (no NaN is above)
}

// c / sqrt(x), each correctly rounded (x > 0): the projections' factor.
__device__ __forceinline__ float over_sqrt(const KMul<float> &c, float x) { return c.w / sqrtf(x); }

static __device__ __noinline__ double fp64_over_sqrt_hw(double c, double x) { return c / sqrt(x); }

// High 128-bit difference (ah:al) - (bh:bl), arithmetically shifted right by 54.
__device__ __forceinline__ int64_t sub128_hi(uint64_t ah, uint64_t al, uint64_t bh, uint64_t bl)
{
    const uint64_t l = al - bl, h = ah - bh - (al < bl ? 1u : 0u);
    return (int64_t)((h << 10) | (l >> 54));
}

// In integers, by Newton's iteration on the residual (Markstein's scheme: an
// approximation from a short reciprocal, corrected by its exact remainder):
// r ~ 1/sqrt to 22 bits from rsqrtf; s0 = x r; s1 = s0 + (x - s0^2) r / 2 to ~43
// bits; s2 = s1 + (x - s1^2) r / 2 to four units in 2^-62, x - s1^2 being exact.
// A square root is never midway between two doubles, so s2 decides the rounding
// except within those units of a midpoint m, where m^2 is compared with x
// exactly.  The quotient c / s follows in the same way from r ~ 1/s.  ~230 cycles
// per warp and scheduler against ~1200 for the hardware division and square
// root, which are sequences on the FP64 pipe.
__device__ __forceinline__ double over_sqrt(const KMul<double> &c, double x)
{
    const uint64_t b = (uint64_t)__double_as_longlong(x), ab = (uint64_t)__double_as_longlong(c.w);
    const uint32_t e = (uint32_t)(b >> 52);
    if (e - 128u >= 1792u || !c.span || c.s) return fp64_over_sqrt_hw(c.w, x);
    // x = X 2^-62 4^k, X 2^-62 in [1, 4)
    const uint32_t odd = (e & 1u) ^ 1u;
    const uint64_t X = ((b & 0xfffffffffffffull) | (1ull << 52)) << (10 + odd);
    const float rf = fminf(rsqrtf((float)(uint32_t)(X >> 40) * (1.0f / 4194304.0f)), 1.0f);
    const uint32_t R = (uint32_t)(rf * 2147483648.0f);  // 2^31 r
    const uint64_t t0 = ((uint64_t)(uint32_t)(X >> 32) * R) >> 30;
    const uint32_t S0 = t0 > 0xffffffffull ? 0xffffffffu : (uint32_t)t0;  // 2^31 s0
    const int64_t D = (int64_t)(X - (uint64_t)S0 * S0);                   // 2^62 (x - s0^2)
    const uint64_t S1 = ((uint64_t)S0 << 31) + (uint64_t)(((D >> 13) * (int64_t)R) >> 19);  // 2^62 s1
    const uint64_t S2 = S1 + (uint64_t)((sub128_hi(X >> 2, X << 62, __umul64hi(S1, S1), S1 * S1) * (int64_t)R) >> 40);
    uint64_t h = S2 >> 10, q = h + (((uint32_t)S2 >> 9) & 1u);
    if (((uint32_t)S2 & 1023u) - 507u <= 10u) {
        const uint64_t M = 2 * h + 1, mh = __umul64hi(M, M), ml = M * M, xh = X >> 20, xl = X << 44;
        q = h + (xh > mh || (xh == mh && xl > ml) ? 1u : 0u);
    }
    const uint32_t es = (e + 1023u - odd) >> 1;  // exponent field of s, whose significand is q
    if (q >> 53) return fp64_over_sqrt_hw(c.w, x);
    const uint64_t B = q << 11, A = (uint64_t)c.wh << 32 | c.wl;  // significands, 2^63
    const uint64_t P = (B >> 32) * R + (((uint64_t)(uint32_t)B * R) >> 32);  // 2^62 s r
    const int64_t E = (int64_t)((1ull << 62) - P);
    const uint64_t r1 = ((uint64_t)R << 31) + (uint64_t)(((E >> 11) * (int64_t)R) >> 20);  // 2^62 / s to ~42 bits
    const uint64_t q1 = __umul64hi(A, r1);                                                 // 2^61 c / s
    const uint64_t q2 = q1 + (uint64_t)((sub128_hi(A >> 3, A << 61, __umul64hi(q1, B), q1 * B) * (int64_t)R) >> 40);
    const uint32_t ge = (uint32_t)(q2 >> 61), sh = 8 + ge, half = 1u << (sh - 1);
    h = q2 >> sh;
    uint64_t m = h + (((uint32_t)q2 >> (sh - 1)) & 1u);
    if (((uint32_t)q2 & (2 * half - 1)) - (half - 4u) <= 8u) {
        const uint64_t M = 2 * h + 1, mh = __umul64hi(M, q), ml = M * q, a = A >> 11;
        const uint64_t xh = a >> (2 + sh), xl = a << (62 - sh);
        m = h + (xh > mh || (xh == mh && xl > ml) ? 1u : 0u);
    }
    const uint64_t er = (ab >> 52) - es + 1022u + ge;
    return __longlong_as_double((long long)((er << 52) + (m - (1ull << 52))));
}

#endif  // __CUDACC__

}  // namespace qsm
