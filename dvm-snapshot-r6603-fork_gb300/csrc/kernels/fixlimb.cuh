// Chains of FP64 additions of non-negative values, bit-exact with the FP64 unit in round-to-nearest-even, on the
// FP32 pipe.
//
// Why: a GB300 SM does 2 FP64 operations per clock and 128 FP32 ones, and a Blackwell FP32 instruction may do two
// (add / mul / fma.f32x2).  The same sums on the integer pipes (softfp64.cuh, q61) cost about 11 instructions per
// addition and cell -- a leading-bit count, a table lookup, 64-bit carries.  Here an addition with its rounding is 10
// instructions for two cells.
//
// Form.  With E the exponent field of the smallest value allowed, a double x = +0 or 2^(E-1023) <= x < 2^(E-1014) (nine
// binades) is an integer multiple q of u = 2^(E-1075) below 2^61.  q is held as three limbs
//     q = H 2^40 + M 2^20 + L,     h = H 2^11, m = M, l = L as floats   (H < 2^21, M, L < 2^20 for one value),
// and a sum of up to six values adds the limbs without carries: H, M, L stay below 6 * 2^21 < 2^24, exact in FP32.
//
// Rounding.  The sum S = RN of the exact sum keeps 53 significant bits: with p its leading bit, its last k = p - 52
// bits go (k <= 11 for S < 2^64), and S is a multiple of 2^k for k <= 0 anyway.  All of them lie in l.
//   t = fma.rz(fma.rz(l, 2^-20, m), 2^-9, h) is S 2^-29 rounded down (a rounding towards zero of a rounding towards
//   zero): for a power of two 2^e >= 2^40, and for 3 * 2^e, S >= 2^e exactly when t >= 2^(e-29), because both sides
//   compare integers that FP32 holds.  So t's exponent is p - 29, and B = t with its significand cleared = 2^(23+k).
//   (l + B) - B then rounds l to a multiple of 2^k, ties to even, by the FP32 unit's own rounding: 0 <= l < 2^23 <=
//   2^(23+k), so l + B stays in [B, 2B), where FP32 numbers are 2^k apart, and l / 2^k has the parity of S / 2^k since
//   k < 20.  For k < 0 the sum is below 2^24 and exact.
// (The rounding of a sum by adding and subtracting a large constant is the classic technique of, e.g., Dekker 1971 and
// Muller et al., Handbook of Floating-Point Arithmetic, ch. 4.)
//
// Division by 6 is long division of the limbs: quotient digits floor(h / 6) and floor((rest) / 6) as products by
// RN(1/6) rounded towards zero onto the integers (the product exceeds the quotient by less than 0.1 and a fraction of
// a sixth is at most 5/6), the last digit rounded to the quotient's 53 bits by one fma: l2 / 6 + B', B' = 2^(23+k').
// RN(1/6) is off by 2^-25 relatively, so l2 * RN(1/6) is within 0.06 of l2 / 6, while l2 / 6 is at least 1/6 away from
// every rounding boundary (a multiple of 1/2): at a boundary the quotient would have 54 significant bits, and six
// times such a number has at least 55, more than the sum's 53.  This needs k' >= 0, a quotient of at least 2^52 u.
//
// V: float (host checks) or f32x2 (device, two cells).
#pragma once

#include "softfp64.cuh"

#ifndef __CUDA_ARCH__
#include <cfenv>
#endif

namespace fx {

constexpr uint32_t EXPMASK = 0x7F800000u;
constexpr float C6 = 0x1.555556p-3f;  // RN(1/6)
constexpr int E_DEFAULT = 1014;       // values in [2^-9, 1)
constexpr int E_MIN = 64, E_MAX = 1980;

SF_HD uint32_t fbits(float x) {
#ifdef __CUDA_ARCH__
    return __float_as_uint(x);
#else
    uint32_t b;
    memcpy(&b, &x, 4);
    return b;
#endif
}
SF_HD float ffrom(uint32_t b) {
#ifdef __CUDA_ARCH__
    return __uint_as_float(b);
#else
    float x;
    memcpy(&x, &b, 4);
    return x;
#endif
}

// ---- one value
#ifndef __CUDA_ARCH__
struct Rz {  // rounding towards zero for a scope
    Rz() { fesetround(FE_TOWARDZERO); }
    ~Rz() { fesetround(FE_TONEAREST); }
};
static inline float vadd(float a, float b) { return a + b; }
static inline float vfma(float a, float b, float c) { return std::fma(a, b, c); }
static inline float vfma_rz(float a, float b, float c) {
    Rz rz;
    volatile float r = std::fma(a, b, c);
    return r;
}
static inline float vmul_rz(float a, float b) {
    Rz rz;
    volatile float x = a, y = b, r = x * y;
    return r;
}
#else
__device__ __forceinline__ float vadd(float a, float b) { return __fadd_rn(a, b); }
__device__ __forceinline__ float vfma(float a, float b, float c) { return __fmaf_rn(a, b, c); }
__device__ __forceinline__ float vfma_rz(float a, float b, float c) { return __fmaf_rz(a, b, c); }
__device__ __forceinline__ float vmul_rz(float a, float b) { return __fmul_rz(a, b); }
#endif
SF_HD float vpow2(float a) { return ffrom(fbits(a) & EXPMASK); }
template <typename V>
struct Const;
template <>
struct Const<float> {
#ifdef __CUDACC__
    static __host__ __device__ __forceinline__ float of(float c) { return c; }
#else
    static float of(float c) { return c; }
#endif
};

// ---- two values in one 64-bit register (device)
#ifdef __CUDACC__
struct f32x2 {
    unsigned long long v;
};
__device__ __forceinline__ f32x2 pack(float x, float y) {
    f32x2 r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r.v) : "f"(x), "f"(y));
    return r;
}
__device__ __forceinline__ float lo(f32x2 a) {
    float x, y;
    asm("mov.b64 {%0, %1}, %2;" : "=f"(x), "=f"(y) : "l"(a.v));
    return x;
}
__device__ __forceinline__ float hi(f32x2 a) {
    float x, y;
    asm("mov.b64 {%0, %1}, %2;" : "=f"(x), "=f"(y) : "l"(a.v));
    return y;
}
template <>
struct Const<f32x2> {
    static __device__ __forceinline__ f32x2 of(float c) { return pack(c, c); }
};
__device__ __forceinline__ f32x2 vadd(f32x2 a, f32x2 b) {
    f32x2 r;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r.v) : "l"(a.v), "l"(b.v));
    return r;
}
__device__ __forceinline__ f32x2 vmul(f32x2 a, f32x2 b) {
    f32x2 r;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r.v) : "l"(a.v), "l"(b.v));
    return r;
}
__device__ __forceinline__ f32x2 vfma(f32x2 a, f32x2 b, f32x2 c) {
    f32x2 r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r.v) : "l"(a.v), "l"(b.v), "l"(c.v));
    return r;
}
__device__ __forceinline__ f32x2 vfma_rz(f32x2 a, f32x2 b, f32x2 c) {
    f32x2 r;
    asm("fma.rz.f32x2 %0, %1, %2, %3;" : "=l"(r.v) : "l"(a.v), "l"(b.v), "l"(c.v));
    return r;
}
__device__ __forceinline__ f32x2 vmul_rz(f32x2 a, f32x2 b) {
    f32x2 r;
    asm("mul.rz.f32x2 %0, %1, %2;" : "=l"(r.v) : "l"(a.v), "l"(b.v));
    return r;
}
__device__ __forceinline__ f32x2 vpow2(f32x2 a) {
    return pack(ffrom(fbits(lo(a)) & EXPMASK), ffrom(fbits(hi(a)) & EXPMASK));
}
#endif

template <typename V>
struct Limbs {
    V h, m, l;
};

#ifdef __CUDACC__
#define FX_FN template <typename V> __host__ __device__ __forceinline__
#else
#define FX_FN template <typename V> static inline
#endif

FX_FN V vsub(V a, V b) { return vfma(b, Const<V>::of(-1.0f), a); }

FX_FN Limbs<V> plus(const Limbs<V> &a, const Limbs<V> &b) { return {vadd(a.h, b.h), vadd(a.m, b.m), vadd(a.l, b.l)}; }

// S 2^-29 rounded down
FX_FN V magnitude(const Limbs<V> &s) {
    return vfma_rz(vfma_rz(s.l, Const<V>::of(0x1p-20f), s.m), Const<V>::of(0x1p-9f), s.h);
}

// s rounded to 53 significant bits; t = magnitude(s)
FX_FN Limbs<V> rounded(const Limbs<V> &s, V t) {
    const V b = vpow2(t);
    return {s.h, s.m, vsub(vadd(s.l, b), b)};
}

// RN(a + b)
FX_FN Limbs<V> add(const Limbs<V> &a, const Limbs<V> &b) {
    const Limbs<V> s = plus(a, b);
    return rounded(s, magnitude(s));
}

// a quotient, with what its assembly to a double takes: hm, mm = 2^23 + H and 2^23 + M as floats (their low bits are
// the integers), b = 2^(23+k'); l is rounded
template <typename V>
struct Quotient {
    V hm, mm, l, b;
};

// magnitude(s) below this: the quotient by 6 is below 2^52 u
constexpr float SMALL6 = 3.0f * 0x1p24f;

// RN(s / 6) for s rounded, magnitude(s) >= SMALL6
FX_FN Quotient<V> div6(const Limbs<V> &s) {
    const V c6 = Const<V>::of(C6), two23 = Const<V>::of(0x1p23f), mtwo23 = Const<V>::of(-0x1p23f);
    Quotient<V> q;
    q.b = vpow2(vmul_rz(magnitude(s), c6));
    q.hm = vfma_rz(s.h, Const<V>::of(C6 * 0x1p-11f), two23);
    const V rh = vfma(vadd(q.hm, mtwo23), Const<V>::of(-6.0f * 0x1p11f), s.h);  // 2^11 (H - 6 floor(H / 6))
    const V m2 = vfma(rh, Const<V>::of(0x1p9f), s.m);
    q.mm = vfma_rz(m2, c6, two23);
    const V rm = vfma(vadd(q.mm, mtwo23), Const<V>::of(-6.0f), m2);
    const V l2 = vfma(rm, Const<V>::of(0x1p20f), s.l);
    q.l = vsub(vfma(l2, c6, q.b), q.b);
    return q;
}

// the sum itself in that form, times 2^-shift (an exact division by a power of two)
// (H and M are below 2^23: at most four values were added)
FX_FN Quotient<V> whole(const Limbs<V> &s) {
    Quotient<V> q;
    q.b = vpow2(magnitude(s));
    q.hm = vfma(s.h, Const<V>::of(0x1p-11f), Const<V>::of(0x1p23f));
    q.mm = vadd(s.m, Const<V>::of(0x1p23f));
    q.l = s.l;
    return q;
}

// x's limbs (of one cell), biased: h a float 2^33 + 2^10 H, m and l floats 2^23 + M, 2^23 + L
struct Raw {
    uint32_t h, m, l;
};
// the position of x's exponent in the range, 0..8 for a normal value inside it
SF_HD uint32_t place(uint32_t xh, int E) { return (xh >> 20) - (uint32_t)E; }
// limbs of the significand mh:xl at place sh (its low five bits count)
SF_HD Raw limbsOf(uint32_t mh, uint32_t xl, uint32_t sh) {
#ifdef __CUDA_ARCH__
    const uint32_t qh = __funnelshift_l(xl, mh, sh), ql = __funnelshift_l(0u, xl, sh);
    const uint32_t h = __byte_perm(qh, 0x50u, 0x4321);
#else
    sh &= 31u;
    const uint32_t qh = sf::fshl(xl, mh, sh), ql = xl << sh;
    const uint32_t h = (qh >> 8) | 0x50000000u;
#endif
    return {h, (sf::fshl(ql, qh, 12) & 0xFFFFFu) | 0x4B000000u, (ql & 0xFFFFFu) | 0x4B000000u};
}
// a value whose place is in range
SF_HD Raw split(uint32_t xh, uint32_t xl, uint32_t sh) { return limbsOf((xh & 0xFFFFFu) | 0x100000u, xl, sh); }
// any value: +0 has zero limbs, a value outside the range clears ok (its limbs are arbitrary)
SF_HD Raw splitAny(uint32_t xh, uint32_t xl, uint32_t sh, bool &ok) {
    const bool zero = (xh | xl) == 0;
    ok &= zero || sh <= 8u;
    return limbsOf(zero ? 0u : (xh & 0xFFFFFu) | 0x100000u, xl, sh);
}
// the limbs proper
FX_FN Limbs<V> unbias(V h, V m, V l) {
    const V c = Const<V>::of(-0x1p23f);
    return {vfma(h, Const<V>::of(2.0f), Const<V>::of(-0x1p34f)), vadd(m, c), vadd(l, c)};
}

// a double from h's part of its high word, 2^23 + M, l and b, times 2^-shift
SF_HD double assembleAt(uint32_t hw, float mm, float l, float b, int E, int shift) {
    const uint32_t il = fbits(l + 0x1p23f) & 0x7FFFFFu;
    // M 2^20 + L; the float's exponent bits (0x4B0 << 20) leave with the addend
    const uint64_t u = (uint64_t)fbits(mm) * (1u << 20) + (((uint64_t)(0u - 0x4B000u) << 32) | il);
    const uint32_t uh = hw + sf::hi32(u);
    const uint32_t f = (fbits(b) >> 23) + 10u;  // p - 52 modulo 32: the zero bits below the significand
#ifdef __CUDA_ARCH__
    const uint32_t lo = __funnelshift_r((uint32_t)u, uh, f), hi = __funnelshift_r(uh, 0u, f);
#else
    const uint32_t lo = sf::fshr((uint32_t)u, uh, f & 31u), hi = uh >> (f & 31u);
#endif
    // the significand's leading one adds 1 to the exponent field (2 where the rounding of l carried out of it)
    const uint32_t res = f * (1u << 20) + hi + ((uint32_t)(E - 161 - shift) << 20);
    return sf::from(((uint64_t)res << 32) | lo);
}

// the double of a quotient's (or sum's) limbs, times 2^-shift: hm, mm, l and b of one cell; the value is at least 2^52 u
SF_HD double assemble(float hm, float mm, float l, float b, int E, int shift = 0) {
    return assembleAt(fbits(hm) * 256u, mm, l, b, E, shift);
}

// RN(s) of one cell's sum of up to six values, not rounded yet (H may exceed 2^23: its low bit goes to M); s >= 2^52 u
SF_HD double sumDouble(const Limbs<float> &s, int E) {
    const float b = vpow2(magnitude(s));
    const float h2 = vfma_rz(s.h, 0x1p-12f, 0x1p23f);                             // 2^23 + floor(H / 2)
    const float odd = vfma(vadd(h2, -0x1p23f), -0x1p12f, s.h);                    // 2^11 (H mod 2)
    const float mm = vadd(vfma(odd, 0x1p9f, s.m), 0x1p23f);
    return assembleAt(fbits(h2) * 512u, mm, vsub(vadd(s.l, b), b), b, E, 0);
}
// magnitude(s) below this: s is below 2^52 u
constexpr float SMALL1 = 0x1p23f;

// RN(i u) for an integer |i| < 2^63: normalised to bit 62, its last ten bits rounded to nearest even, +0 for 0
SF_HD double round63(int64_t i, int E) {
    const uint32_t sign = (uint32_t)((uint64_t)i >> 32) & 0x80000000u;
    const uint64_t a = i < 0 ? 0 - (uint64_t)i : (uint64_t)i;
    const int p = sf::msb32(sf::hi32(a));  // the leading one is bit 32 + p
    if (p < 0) {                           // below 2^32: exact
        const uint64_t X = sf::bits((double)i);
        return sf::from(X == 0 ? 0 : X + ((uint64_t)(int64_t)(E - 1075) << 52));
    }
    const uint32_t c = 30u - (uint32_t)p;
    const uint32_t nh = sf::fshl((uint32_t)a, sf::hi32(a), c), nl = (uint32_t)a << c;
    const uint64_t n = (((uint64_t)nh << 32) | nl) + (0x1FFu + ((nl >> 10) & 1u));
    // the significand's leading one adds 1 to the exponent field, a carry out of it 2
    const uint32_t hi = (sf::hi32(n) >> 10) + ((uint32_t)(p + E - 21) << 20);
    return sf::from(((uint64_t)(hi | sign) << 32) | sf::fshr((uint32_t)n, sf::hi32(n), 10));
}

// a double in the range of E (or a sum or quotient of at least 2^52 u) as an integer of u
SF_HD uint64_t integer(double x, int E) {
    const uint64_t X = sf::bits(x);
    return X == 0 ? 0 : ((X & sf::MANT) | sf::HID) << (((uint32_t)(X >> 52) - (uint32_t)E) & 63u);
}

}  // namespace fx
