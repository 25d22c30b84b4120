/*
 * Two neighbouring columns in one operation: packed float arithmetic
 * (add / sub / mul .f32x2, each half rounded separately) and the four-column
 * values the register-tile step kernels work on.
 */
#ifndef GC_PACKED_CUH
#define GC_PACKED_CUH

#include "open_bd.cuh"

namespace gcpacked {

constexpr unsigned FULL = 0xffffffffu;

/* ---- two floats in one register pair ---- */
typedef unsigned long long u64;
static __constant__ u64 c_minus_zero2 = 0x8000000080000000ull;
__device__ __forceinline__ u64 pk(float2 a) {
    u64 r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a.x), "f"(a.y));
    return r;
}
__device__ __forceinline__ float2 upk(u64 a) {
    float2 r;
    asm("mov.b64 {%0, %1}, %2;" : "=f"(r.x), "=f"(r.y) : "l"(a));
    return r;
}
__device__ __forceinline__ float2 add2(float2 a, float2 b) {
    u64 r;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(pk(a)), "l"(pk(b)));
    return upk(r);
}
__device__ __forceinline__ float2 sub2(float2 a, float2 b) {
    u64 r;
    asm("sub.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(pk(a)), "l"(pk(b)));
    return upk(r);
}
__device__ __forceinline__ float2 mul2(float2 a, float2 b) {
    /* a*b + (-0) is a*b rounded once, whatever its sign.  The addend comes
     * from constant memory, where the compiler cannot see its value: a plain
     * mul.rn.f32x2, or this with an immediate -0, was merged with the addition
     * that follows and rounded once where the Fortran rounds twice. */
    u64 r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(pk(a)), "l"(pk(b)), "l"(c_minus_zero2));
    return upk(r);
}
/* a lane's four columns as two pairs */
struct V4 {
    float2 a, b;
};
__device__ __forceinline__ V4 v4(float4 v) { return {make_float2(v.x, v.y), make_float2(v.z, v.w)}; }
__device__ __forceinline__ float4 f4(const V4 &v) { return make_float4(v.a.x, v.a.y, v.b.x, v.b.y); }
__device__ __forceinline__ V4 v4(float x, float y, float z, float w) { return {make_float2(x, y), make_float2(z, w)}; }
__device__ __forceinline__ V4 operator+(const V4 &p, const V4 &q) { return {add2(p.a, q.a), add2(p.b, q.b)}; }
__device__ __forceinline__ V4 operator-(const V4 &p, const V4 &q) { return {sub2(p.a, q.a), sub2(p.b, q.b)}; }
__device__ __forceinline__ V4 operator*(const V4 &p, const V4 &q) { return {mul2(p.a, q.a), mul2(p.b, q.b)}; }
__device__ __forceinline__ V4 operator*(float2 k, const V4 &q) { return {mul2(k, q.a), mul2(k, q.b)}; }

/* min / max of three numbers (a NaN operand is passed over) */
__device__ __forceinline__ float min3(float a, float b, float c) {
    float r;
    asm("min.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(a), "f"(b), "f"(c));
    return r;
}
__device__ __forceinline__ float max3(float a, float b, float c) {
    float r;
    asm("max.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(a), "f"(b), "f"(c));
    return r;
}
__device__ __forceinline__ float min4(float m, const V4 &v) { return min3(min3(m, v.a.x, v.a.y), v.b.x, v.b.y); }
/* the same, NaN when an operand is */
__device__ __forceinline__ float min3nan(float a, float b, float c) {
    float r;
    asm("min.NaN.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(a), "f"(b), "f"(c));
    return r;
}
__device__ __forceinline__ float min4nan(float m, const V4 &v) {
    return min3nan(min3nan(m, v.a.x, v.a.y), v.b.x, v.b.y);
}
__device__ __forceinline__ float max4(float m, const V4 &v) { return max3(max3(m, v.a.x, v.a.y), v.b.x, v.b.y); }
__device__ __forceinline__ float minabs4(float m, const V4 &v) {
    return min3(min3(m, fabsf(v.a.x), fabsf(v.a.y)), fabsf(v.b.x), fabsf(v.b.y));
}
__device__ __forceinline__ V4 lds4(const float *p) { return v4(*reinterpret_cast<const float4 *>(p)); }
__device__ __forceinline__ void sts4(float *p, const V4 &v) { *reinterpret_cast<float4 *>(p) = f4(v); }
__device__ __forceinline__ float shw(float v) { return __shfl_up_sync(FULL, v, 1); }   /* lane - 1 */
__device__ __forceinline__ float she(float v) { return __shfl_down_sync(FULL, v, 1); } /* lane + 1 */

/* the bits of four values that are not +0 */
__device__ __forceinline__ unsigned bits4(const V4 &v) {
    return __float_as_uint(v.a.x) | __float_as_uint(v.a.y) | __float_as_uint(v.b.x) | __float_as_uint(v.b.y);
}
/* |x| < EPS flushed to 0 */
__device__ __forceinline__ float flush(float x) { return (fabsf(x) < CC_EPS) ? 0.0f : x; }
__device__ __forceinline__ V4 flush4(const V4 &v) { return v4(flush(v.a.x), flush(v.a.y), flush(v.b.x), flush(v.b.y)); }
/* the land clamp of MASS_S: Z + H <= EPS becomes -H */
__device__ __forceinline__ V4 clamp4(const V4 &z, const V4 &h) {
    const V4 s = z + h;
    return v4(s.a.x <= CC_EPS ? -h.a.x : z.a.x, s.a.y <= CC_EPS ? -h.a.y : z.a.y, s.b.x <= CC_EPS ? -h.b.x : z.b.x,
              s.b.y <= CC_EPS ? -h.b.y : z.b.y);
}
__device__ __forceinline__ float comp(const V4 &v, int q) { return q == 0 ? v.a.x : q == 1 ? v.a.y : q == 2 ? v.b.x : v.b.y; }

/* |OPEN| of the fluxes along (a) and across (b) the boundary, c = sqrt(g h)
 * (boundaries.f90:42-200, open_bd.cuh), with its sign and bound */
__device__ __forceinline__ float open_value(float a, float b, float c, bool neg, bool wet) {
    float zz = gcopen::div_nz(gcopen::sqrt_nz(a * a + b * b), c);
    if (neg) zz = -zz;
    if (fabsf(zz) > CC_UB) zz = 0.0f;
    return wet ? zz : 0.0f;
}

} // namespace gcpacked

#endif
