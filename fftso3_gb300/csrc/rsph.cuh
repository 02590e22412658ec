// The real-harmonic basis change matrix2rsph (fdcl_FFTSO3.cpp:1107-1139) as
// device helpers shared by the basis conversions and the Clebsch-Gordan tables.
#pragma once
#include <cuda_runtime.h>

namespace fftso3 {

// matrix2rsph T(l; a, c) (fdcl_FFTSO3.cpp:1107-1139), row a, column c, in the
// arithmetic type A (double for the FP64 path, float for the tensor-core path).
template <typename A> struct c2t { A x, y; };

// 1/sqrt(2): the FP64 path forms it as the reference does, 1./sqrt(2.).
template <typename A> __device__ __forceinline__ A inv_sqrt2();
template <> __device__ __forceinline__ double inv_sqrt2<double>() { return 1. / sqrt(2.); }
template <> __device__ __forceinline__ float inv_sqrt2<float>() { return 0.70710678118654752440f; }

template <typename A>
__device__ __forceinline__ c2t<A> tmat_t(int a, int c)
{
    const A s = inv_sqrt2<A>();
    if (a < 0) {
        if (c == a) return {(A)0, s};
        if (c == -a) return {(A)0, -s * ((a & 1) ? (A)-1 : (A)1)};
    } else if (a == 0) {
        if (c == 0) return {(A)1, (A)0};
    } else {
        if (c == -a) return {s, (A)0};
        if (c == a) return {((a & 1) ? (A)-1 : (A)1) * s, (A)0};
    }
    return {(A)0, (A)0};
}

template <typename A>
__device__ __forceinline__ c2t<A> cmul_t(c2t<A> a, c2t<A> b)
{
    return {a.x * b.x - a.y * b.y, a.x * b.y + a.y * b.x};
}
template <typename A>
__device__ __forceinline__ c2t<A> conj_t(c2t<A> a) { return {a.x, -a.y}; }

// The basis change of one coefficient with T's entries (0, +-s, +-i s, 1) multiplied out: each of the four (two, one) terms
// is a signed real or imaginary part, so a value costs additions only (as complex products of T's entries it took about
// 40 operations, FP64 ones in the FP64 path).
//
// F_r(m, n) = Re sum_{a = +-m, b = +-n} T[m][a] F(a, b) conj(T[n][b]); f(a, b) returns F(a, b).
// HERM: F(-a, -b) = (-1)^(a+b) conj F(a, b) holds exactly, so half of the terms are read.
template <typename A, bool HERM, typename FN>
__device__ __forceinline__ A real_coefficient(int m, int n, FN&& f)
{
    const int mu = m < 0 ? -m : m, nu = n < 0 ? -n : n;
    const bool ui = m < 0, wi = n < 0, mixed = ui != wi;
    const A sm = (m & 1) ? (A)-1 : (A)1, sn = (n & 1) ? (A)-1 : (A)1;
    const A sq = (ui && wi) ? (A)-1 : (A)1;
    // Re(conj(u) w F), Re(conj(u) conj(w) F), Re(u conj(w) F), Re(u w F) with u, w = 1 or i
    auto t4 = [&](c2t<A> v) { return !mixed ? v.x : ui ? v.y : -v.y; };
    auto t3 = [&](c2t<A> v) { return !mixed ? sq * v.x : v.y; };
    auto t1 = [&](c2t<A> v) { return !mixed ? v.x : ui ? -v.y : v.y; };
    auto t2 = [&](c2t<A> v) { return !mixed ? sq * v.x : -v.y; };
    const A p = sm * sn * t4(f(mu, nu));
    if (mu == 0 && nu == 0) return p;
    const A h = (A)0.70710678118654752440;
    if (HERM) {
        if (mu == 0 || nu == 0) return ((A)2 * h) * p;
        return p + sm * t3(f(mu, -nu));
    }
    if (mu == 0) return h * (p + sm * t3(f(0, -nu)));
    if (nu == 0) return h * (p + t1(f(-mu, 0)));
    return (A)0.5 * ((t1(f(-mu, -nu)) + p) + (sn * t2(f(-mu, nu)) + sm * t3(f(mu, -nu))));
}

// F(m, n) = sum_{a = +-m, b = +-n} conj(T[a][m]) F_r(a, b) T[b][n]; f(a, b) returns F_r(a, b).
template <typename A, typename FN>
__device__ __forceinline__ c2t<A> complex_coefficient(int m, int n, FN&& f)
{
    const int mu = m < 0 ? -m : m, nu = n < 0 ? -n : n;
    const A tm = m < 0 ? (A)-1 : (A)1, tn = n < 0 ? (A)-1 : (A)1;
    const A sg = ((m > 0 && (m & 1)) != (n > 0 && (n & 1))) ? (A)-1 : (A)1;
    const A h = (A)0.70710678118654752440;
    const A pp = f(mu, nu);
    if (mu == 0 && nu == 0) return {pp, (A)0};
    if (mu == 0) return {h * sg * pp, -(h * sg * tn) * f(0, -nu)};
    if (nu == 0) return {h * sg * pp, (h * sg * tm) * f(-mu, 0)};
    const A k = (A)0.5 * sg;
    return {k * (pp + (tm * tn) * f(-mu, -nu)), k * (tm * f(-mu, nu) - tn * f(mu, -nu))};
}

// The packed offset of degree l (< 2^31 for l <= 511), and the degree of packed place r.
__device__ __forceinline__ int off32(int l) { return l * (4 * l * l - 1) / 3; }
__device__ __forceinline__ int degree_of(int r)
{
    int l = (int)cbrtf(0.75f * (float)r);
    while (l > 0 && off32(l) > r) --l;
    while (off32(l + 1) <= r) ++l;
    return l;
}

}  // namespace fftso3
