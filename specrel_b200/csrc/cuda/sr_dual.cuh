// Forward-mode dual numbers for the gradient kernel: a float value and its derivatives with respect
// to the observer parameters (rapidity x, y, z, event t, x, y, z). The value parts are computed with
// exactly the operations, in exactly the order, of the forward shading code they mirror, so they
// reproduce the forward frame's values bit for bit; the derivative parts follow the chain rule.
// Min/max/clamp select by value and carry the selected operand's derivatives (zero for a constant).
// Templated on the number of tangents: all seven in one thread, or one per thread (a group of threads then holds
// a number's tangents, each computing the value too), with the same operations per tangent either way.
// The types live in their own namespace so that their overloads never hide the float ones.
#pragma once
#include "sr_device.cuh"

namespace srg {

using srd::F3;

constexpr int NT = 7;  // tangents

template <int N>
struct DFT {
    float v;
    float d[N];
};
using DF = DFT<NT>;

template <int N = NT>
__device__ __forceinline__ DFT<N> dconst(float v) {
    DFT<N> r;
    r.v = v;
#pragma unroll
    for (int i = 0; i < N; ++i) r.d[i] = 0.0f;
    return r;
}
template <int N>
__device__ __forceinline__ DFT<N> operator+(const DFT<N>& a, const DFT<N>& b) {
    DFT<N> r;
    r.v = a.v + b.v;
#pragma unroll
    for (int i = 0; i < N; ++i) r.d[i] = a.d[i] + b.d[i];
    return r;
}
template <int N>
__device__ __forceinline__ DFT<N> operator-(const DFT<N>& a, const DFT<N>& b) {
    DFT<N> r;
    r.v = a.v - b.v;
#pragma unroll
    for (int i = 0; i < N; ++i) r.d[i] = a.d[i] - b.d[i];
    return r;
}
template <int N>
__device__ __forceinline__ DFT<N> operator-(const DFT<N>& a) {
    DFT<N> r;
    r.v = -a.v;
#pragma unroll
    for (int i = 0; i < N; ++i) r.d[i] = -a.d[i];
    return r;
}
template <int N>
__device__ __forceinline__ DFT<N> operator*(const DFT<N>& a, const DFT<N>& b) {
    DFT<N> r;
    r.v = a.v * b.v;
#pragma unroll
    for (int i = 0; i < N; ++i) r.d[i] = a.d[i] * b.v + a.v * b.d[i];
    return r;
}
template <int N>
__device__ __forceinline__ DFT<N> operator/(const DFT<N>& a, const DFT<N>& b) {
    DFT<N> r;
    r.v = a.v / b.v;
    const float ib = 1.0f / b.v;
#pragma unroll
    for (int i = 0; i < N; ++i) r.d[i] = (a.d[i] - r.v * b.d[i]) * ib;
    return r;
}
template <int N>
__device__ __forceinline__ DFT<N> operator+(const DFT<N>& a, float b) {
    DFT<N> r = a;
    r.v = a.v + b;
    return r;
}
template <int N>
__device__ __forceinline__ DFT<N> operator+(float a, const DFT<N>& b) {
    DFT<N> r = b;
    r.v = a + b.v;
    return r;
}
template <int N>
__device__ __forceinline__ DFT<N> operator-(const DFT<N>& a, float b) {
    DFT<N> r = a;
    r.v = a.v - b;
    return r;
}
template <int N>
__device__ __forceinline__ DFT<N> operator-(float a, const DFT<N>& b) {
    DFT<N> r;
    r.v = a - b.v;
#pragma unroll
    for (int i = 0; i < N; ++i) r.d[i] = -b.d[i];
    return r;
}
template <int N>
__device__ __forceinline__ DFT<N> operator*(const DFT<N>& a, float s) {
    DFT<N> r;
    r.v = a.v * s;
#pragma unroll
    for (int i = 0; i < N; ++i) r.d[i] = a.d[i] * s;
    return r;
}
template <int N>
__device__ __forceinline__ DFT<N> operator*(float s, const DFT<N>& a) {
    DFT<N> r;
    r.v = s * a.v;
#pragma unroll
    for (int i = 0; i < N; ++i) r.d[i] = s * a.d[i];
    return r;
}
template <int N>
__device__ __forceinline__ DFT<N> operator/(const DFT<N>& a, float b) {
    DFT<N> r;
    r.v = a.v / b;
#pragma unroll
    for (int i = 0; i < N; ++i) r.d[i] = a.d[i] / b;
    return r;
}
template <int N>
__device__ __forceinline__ DFT<N> operator/(float a, const DFT<N>& b) {
    DFT<N> r;
    r.v = a / b.v;
    const float ib = 1.0f / b.v;
#pragma unroll
    for (int i = 0; i < N; ++i) r.d[i] = -r.v * b.d[i] * ib;
    return r;
}
template <int N>
__device__ __forceinline__ DFT<N> dsqrt(const DFT<N>& a) {
    DFT<N> r;
    r.v = sqrtf(a.v);
    const float k = r.v > 0.0f ? 0.5f / r.v : 0.0f;
#pragma unroll
    for (int i = 0; i < N; ++i) r.d[i] = a.d[i] * k;
    return r;
}
template <int N>
__device__ __forceinline__ DFT<N> dexp(const DFT<N>& a) {
    DFT<N> r;
    r.v = expf(a.v);
#pragma unroll
    for (int i = 0; i < N; ++i) r.d[i] = a.d[i] * r.v;
    return r;
}
// fmaxf(a, b) / fminf(a, b) with a constant b.
template <int N>
__device__ __forceinline__ DFT<N> dmaxc(const DFT<N>& a, float b) { return fmaxf(a.v, b) == a.v && a.v >= b ? a : dconst<N>(fmaxf(a.v, b)); }
template <int N>
__device__ __forceinline__ DFT<N> dminc(const DFT<N>& a, float b) { return fminf(a.v, b) == a.v && a.v <= b ? a : dconst<N>(fminf(a.v, b)); }
template <int N>
__device__ __forceinline__ DFT<N> dclamp(const DFT<N>& x, float lo, float hi) {  // clampf_
    if (x.v < lo) return dconst<N>(lo);
    if (x.v > hi) return dconst<N>(hi);
    return x;
}

template <int N>
struct DF3T {
    DFT<N> x, y, z;
};
template <int N>
struct DF4T {
    DFT<N> x, y, z, w;  // (t, x, y, z)
};
using DF3 = DF3T<NT>;
using DF4 = DF4T<NT>;

template <int N = NT>
__device__ __forceinline__ DF4T<N> dconst4(float4 a) { return DF4T<N>{dconst<N>(a.x), dconst<N>(a.y), dconst<N>(a.z), dconst<N>(a.w)}; }
template <int N>
__device__ __forceinline__ float4 val4(const DF4T<N>& a) { return make_float4(a.x.v, a.y.v, a.z.v, a.w.v); }
template <int N>
__device__ __forceinline__ DF4T<N> add4(const DF4T<N>& a, const DF4T<N>& b) { return DF4T<N>{a.x + b.x, a.y + b.y, a.z + b.z, a.w + b.w}; }
template <int N>
__device__ __forceinline__ DF4T<N> sub4(const DF4T<N>& a, const DF4T<N>& b) { return DF4T<N>{a.x - b.x, a.y - b.y, a.z - b.z, a.w - b.w}; }
template <int N>
__device__ __forceinline__ DF4T<N> sub4(float4 a, const DF4T<N>& b) { return DF4T<N>{a.x - b.x, a.y - b.y, a.z - b.z, a.w - b.w}; }
template <int N>
__device__ __forceinline__ DF4T<N> mul4(const DF4T<N>& a, const DFT<N>& s) { return DF4T<N>{a.x * s, a.y * s, a.z * s, a.w * s}; }
template <int N>
__device__ __forceinline__ DF4T<N> mul4(const DF4T<N>& a, float s) { return DF4T<N>{a.x * s, a.y * s, a.z * s, a.w * s}; }
template <int N>
__device__ __forceinline__ DF4T<N> mul4(float4 a, const DFT<N>& s) { return DF4T<N>{a.x * s, a.y * s, a.z * s, a.w * s}; }
template <int N>
__device__ __forceinline__ DF4T<N> neg4(const DF4T<N>& a) { return DF4T<N>{-a.x, -a.y, -a.z, -a.w}; }
// mdot / edot in the forward code's order.
template <int N>
__device__ __forceinline__ DFT<N> mdot(const DF4T<N>& a, const DF4T<N>& b) { return -a.x * b.x + a.y * b.y + a.z * b.z + a.w * b.w; }
template <int N>
__device__ __forceinline__ DFT<N> mdot(const DF4T<N>& a, float4 b) { return -a.x * b.x + a.y * b.y + a.z * b.z + a.w * b.w; }
template <int N>
__device__ __forceinline__ DFT<N> edot(float4 a, const DF4T<N>& b) { return a.x * b.x + a.y * b.y + a.z * b.z + a.w * b.w; }
template <int N>
__device__ __forceinline__ DF3T<N> spatial(const DF4T<N>& a) { return DF3T<N>{a.y, a.z, a.w}; }
template <int N>
__device__ __forceinline__ DFT<N> dot3(const DF3T<N>& a, const DF3T<N>& b) { return a.x * b.x + a.y * b.y + a.z * b.z; }
template <int N>
__device__ __forceinline__ DF3T<N> add(const DF3T<N>& a, const DF3T<N>& b) { return DF3T<N>{a.x + b.x, a.y + b.y, a.z + b.z}; }
template <int N>
__device__ __forceinline__ DF3T<N> mul(const DF3T<N>& a, const DFT<N>& s) { return DF3T<N>{a.x * s, a.y * s, a.z * s}; }
template <int N>
__device__ __forceinline__ DF3T<N> mul(F3 a, const DFT<N>& s) { return DF3T<N>{a.x * s, a.y * s, a.z * s}; }
template <int N>
__device__ __forceinline__ DF3T<N> mulv(const DF3T<N>& a, F3 b) { return DF3T<N>{a.x * b.x, a.y * b.y, a.z * b.z}; }
template <int N = NT>
__device__ __forceinline__ DF3T<N> dconst3(F3 a) { return DF3T<N>{dconst<N>(a.x), dconst<N>(a.y), dconst<N>(a.z)}; }
template <int N>
__device__ __forceinline__ DFT<N> len3(const DF3T<N>& a) { return dsqrt(dot3(a, a)); }
template <int N>
__device__ __forceinline__ DF3T<N> normalized3(const DF3T<N>& a) {
    DFT<N> l = len3(a);
    if (l.v > 1e-12f) {
        DFT<N> il = 1.0f / l;
        return DF3T<N>{a.x * il, a.y * il, a.z * il};
    }
    return DF3T<N>{dconst<N>(0.0f), dconst<N>(0.0f), dconst<N>(0.0f)};
}

// A double with its derivatives with respect to the three rapidity components, for the FP64
// tetrad (TetradT<DD3> in sr_camera.cuh).
struct DD3 {
    double v, d[3];
    __device__ DD3(double x = 0.0) : v(x), d{0.0, 0.0, 0.0} {}
};
__device__ __forceinline__ DD3 operator+(const DD3& a, const DD3& b) {
    DD3 r(a.v + b.v);
    for (int i = 0; i < 3; ++i) r.d[i] = a.d[i] + b.d[i];
    return r;
}
__device__ __forceinline__ DD3 operator-(const DD3& a, const DD3& b) {
    DD3 r(a.v - b.v);
    for (int i = 0; i < 3; ++i) r.d[i] = a.d[i] - b.d[i];
    return r;
}
__device__ __forceinline__ DD3 operator-(const DD3& a) {
    DD3 r(-a.v);
    for (int i = 0; i < 3; ++i) r.d[i] = -a.d[i];
    return r;
}
__device__ __forceinline__ DD3 operator*(const DD3& a, const DD3& b) {
    DD3 r(a.v * b.v);
    for (int i = 0; i < 3; ++i) r.d[i] = a.d[i] * b.v + a.v * b.d[i];
    return r;
}
__device__ __forceinline__ DD3 operator/(const DD3& a, const DD3& b) {
    DD3 r(a.v / b.v);
    for (int i = 0; i < 3; ++i) r.d[i] = (a.d[i] - r.v * b.d[i]) / b.v;
    return r;
}
__device__ __forceinline__ DD3 operator+(double a, const DD3& b) { return DD3(a) + b; }
__device__ __forceinline__ DD3 operator-(double a, const DD3& b) { return DD3(a) - b; }
__device__ __forceinline__ DD3 operator*(double a, const DD3& b) { return DD3(a) * b; }
__device__ __forceinline__ DD3 operator*(const DD3& a, double b) { return a * DD3(b); }
__device__ __forceinline__ DD3 operator/(double a, const DD3& b) { return DD3(a) / b; }
__device__ __forceinline__ bool operator<(const DD3& a, double b) { return a.v < b; }
__device__ __forceinline__ bool operator>=(const DD3& a, double b) { return a.v >= b; }
__device__ __forceinline__ DD3 sqrt(const DD3& a) {
    DD3 r(::sqrt(a.v));
    for (int i = 0; i < 3; ++i) r.d[i] = r.v > 0.0 ? a.d[i] * (0.5 / r.v) : 0.0;
    return r;
}
__device__ __forceinline__ DD3 fmax(const DD3& a, double b) { return ::fmax(a.v, b) == a.v && a.v >= b ? a : DD3(::fmax(a.v, b)); }
__device__ __forceinline__ DD3 cosh(const DD3& a) {
    DD3 r(::cosh(a.v));
    const double s = ::sinh(a.v);
    for (int i = 0; i < 3; ++i) r.d[i] = a.d[i] * s;
    return r;
}
__device__ __forceinline__ DD3 sinh(const DD3& a) {
    DD3 r(::sinh(a.v));
    const double c = ::cosh(a.v);
    for (int i = 0; i < 3; ++i) r.d[i] = a.d[i] * c;
    return r;
}

}  // namespace srg
