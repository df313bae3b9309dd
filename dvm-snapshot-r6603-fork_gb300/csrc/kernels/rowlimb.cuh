// Rows of a 2-D field walked by a warp in 64-wide chunks (lane l holds the pair of
// columns base + 2l, base + 2l + 1), split into FP32 limbs (fixlimb.cuh): what the
// heat and the Jacobi 2-D kernels share.
#pragma once

#include "fixlimb.cuh"

namespace rows {

using fx::f32x2;

// a row of the strip: the lane's pair, lane 0's left and lane 31's right edge value, and their limbs
struct Row {
    double2 d;
    double e;
    fx::Limbs<f32x2> v;
    float eh, em, el;
    bool ok;  // its values fit the range (the same on every lane)
    int top;  // when they do not: the largest exponent field among them (with the sign bit above it)
};

// the row's limbs in the range E
__device__ __forceinline__ void split(Row &r, int E) {
    const uint64_t x = sf::bits(r.d.x), y = sf::bits(r.d.y), z = sf::bits(r.e);
    const uint32_t sx = fx::place(sf::hi32(x), E), sy = fx::place(sf::hi32(y), E), sz = fx::place(sf::hi32(z), E);
    fx::Raw rx = fx::split(sf::hi32(x), (uint32_t)x, sx), ry = fx::split(sf::hi32(y), (uint32_t)y, sy);
    fx::Raw rz = fx::split(sf::hi32(z), (uint32_t)z, sz);
    r.ok = true;
    if (__any_sync(0xffffffffu, max(max(sx, sy), sz) > 8u)) {
        bool ok = true;
        rx = fx::splitAny(sf::hi32(x), (uint32_t)x, sx, ok);
        ry = fx::splitAny(sf::hi32(y), (uint32_t)y, sy, ok);
        rz = fx::splitAny(sf::hi32(z), (uint32_t)z, sz, ok);
        r.ok = __all_sync(0xffffffffu, ok);
        r.top = (int)(__reduce_max_sync(0xffffffffu, max(max(sf::hi32(x), sf::hi32(y)), sf::hi32(z))) >> 20);
    }
    r.v = fx::unbias(fx::pack(fx::ffrom(rx.h), fx::ffrom(ry.h)), fx::pack(fx::ffrom(rx.m), fx::ffrom(ry.m)),
                     fx::pack(fx::ffrom(rx.l), fx::ffrom(ry.l)));
    r.eh = __fmaf_rn(fx::ffrom(rz.h), 2.0f, -0x1p34f);
    r.em = fx::ffrom(rz.m) - 0x1p23f;
    r.el = fx::ffrom(rz.l) - 0x1p23f;
}

// the limbs' k - 1 and k + 1 neighbours: (left of x, x), (y, right of y)
__device__ __forceinline__ void sides(f32x2 v, float edge, int lane, f32x2 &left, f32x2 &right) {
    const float up = __shfl_up_sync(0xffffffffu, fx::hi(v), 1), dn = __shfl_down_sync(0xffffffffu, fx::lo(v), 1);
    left = fx::pack(lane == 0 ? edge : up, fx::lo(v));
    right = fx::pack(fx::hi(v), lane == 31 ? edge : dn);
}

// volatile: the next row's loads stay where they are, a step ahead of their use
__device__ __forceinline__ double2 ldGlobal2(const double *p) {
    double2 v;
    asm volatile("ld.global.nc.v2.f64 {%0, %1}, [%2];" : "=d"(v.x), "=d"(v.y) : "l"(p));
    return v;
}
__device__ __forceinline__ double ldGlobal(const double *p) {
    double v;
    asm volatile("ld.global.nc.f64 %0, [%1];" : "=d"(v) : "l"(p));
    return v;
}

// A warp's rows on their way: asynchronous copies into a ring of DEPTH rows in shared memory, DEPTH - 1 rows ahead of
// the one taken.  (With one row in registers ahead, 16 warps an SM had 8 KB in flight, a quarter of what HBM's latency
// takes at its rate.)  A lane reads back only what it copied itself.
constexpr int DEPTH = 8;
struct Ring {
    double2 pair[DEPTH][32];
    double edge[DEPTH][2];
};
__device__ __forceinline__ uint32_t shared(const void *p) { return (uint32_t)__cvta_generic_to_shared(p); }
// 16 (or 8) bytes; zeros where `in` is false (nothing is read then)
__device__ __forceinline__ void copy16(void *dst, const double *src, bool in = true) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(shared(dst)), "l"(src), "r"(in ? 16 : 0) : "memory");
}
__device__ __forceinline__ void copy8(void *dst, const double *src, bool in = true) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;" ::"r"(shared(dst)), "l"(src), "r"(in ? 8 : 0) : "memory");
}
__device__ __forceinline__ void commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
// the oldest of DEPTH - 1 committed rows has landed
__device__ __forceinline__ void landed() { asm volatile("cp.async.wait_group %0;" ::"n"(DEPTH - 2) : "memory"); }
__device__ __forceinline__ void allLanded() { asm volatile("cp.async.wait_group 0;" ::: "memory"); }

__device__ __forceinline__ void stGlobal(double *p, double v) { asm volatile("st.global.f64 [%0], %1;" ::"l"(p), "d"(v) : "memory"); }
__device__ __forceinline__ void stGlobal(double *p, double2 v) {
    asm volatile("st.global.v2.f64 [%0], {%1, %2};" ::"l"(p), "d"(v.x), "d"(v.y) : "memory");
}
__device__ __forceinline__ void stGlobal(int *p, int v) { asm volatile("st.global.s32 [%0], %1;" ::"l"(p), "r"(v) : "memory"); }

// the range for three rows of which one does not fit E: the one that ends with their largest value, a row that fits
// reaching up to E's end; E itself when that is no other or cannot be
__device__ __forceinline__ int rangeOf(const Row &a, const Row &b, const Row &c, int E) {
    const int top = max(max(a.ok ? E + 8 : a.top, b.ok ? E + 8 : b.top), c.ok ? E + 8 : c.top);
    return top - 8 >= fx::E_MIN && top - 8 <= fx::E_MAX ? top - 8 : E;
}

}  // namespace rows
