// Multiplications and additions whose fusing is written down.
//
// With -fmad=true the compiler chooses which product of a sum to fuse, and
// chooses differently in two instantiations of one body (a kernel and its
// batched twin, a column walked whole and in blocks of rows), which then
// differ in the last bit.  The bodies that have to agree bit for bit use
// these: a product is kept as its two factors until it meets a sum, which
// fuses it (of two products the left one); anything else rounds it.
#pragma once

namespace cf {

__device__ __forceinline__ double mul(double a, double b) { return __dmul_rn(a, b); }
__device__ __forceinline__ double add(double a, double b) { return a + b; }   // no product to fuse: mul is opaque to the compiler
__device__ __forceinline__ double mad(double a, double b, double c) { return __fma_rn(a, b, c); }    // c + a b
__device__ __forceinline__ double msub(double a, double b, double c) { return __fma_rn(-a, b, c); }  // c - a b
// a x + b y (+ c z + ...)
__device__ __forceinline__ double dot(double a, double x, double b, double y) { return mad(b, y, mul(a, x)); }
template <class... T>
__device__ __forceinline__ double dot_onto(double s, double a, double x, T... t)
{
    s = mad(a, x, s);
    if constexpr (sizeof...(t) > 0) return dot_onto(s, t...);
    else return s;
}
template <class... T>
__device__ __forceinline__ double dot(double a, double x, double b, double y, T... t)
{
    return dot_onto(dot(a, x, b, y), t...);
}

// pairs of points
struct Product2 {
    double2 a, b;
    __device__ __forceinline__ operator double2() const { return make_double2(mul(a.x, b.x), mul(a.y, b.y)); }
};
__device__ __forceinline__ double2 mad(Product2 p, double2 c)
{
    return make_double2(mad(p.a.x, p.b.x, c.x), mad(p.a.y, p.b.y, c.y));
}
__device__ __forceinline__ double2 neg(double2 a) { return make_double2(-a.x, -a.y); }
__device__ __forceinline__ Product2 operator*(double2 a, double2 b) { return {a, b}; }
__device__ __forceinline__ Product2 operator*(double a, double2 b) { return {make_double2(a, a), b}; }
__device__ __forceinline__ double2 operator+(double2 a, double2 b)
{
    return make_double2(add(a.x, b.x), add(a.y, b.y));
}
__device__ __forceinline__ double2 operator-(double2 a, double2 b)
{
    return make_double2(add(a.x, -b.x), add(a.y, -b.y));
}
__device__ __forceinline__ double2 operator+(Product2 p, double2 c) { return mad(p, c); }
__device__ __forceinline__ double2 operator+(double2 c, Product2 p) { return mad(p, c); }
__device__ __forceinline__ double2 operator+(Product2 p, Product2 q) { return mad(p, (double2) q); }
__device__ __forceinline__ double2 operator-(Product2 p, double2 c) { return mad(p, neg(c)); }
__device__ __forceinline__ double2 operator-(double2 c, Product2 p) { return mad(Product2{neg(p.a), p.b}, c); }
__device__ __forceinline__ double2 operator-(Product2 p, Product2 q) { return mad(p, neg(q)); }

}  // namespace cf
