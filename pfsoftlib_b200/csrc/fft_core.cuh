// Device building blocks of the DFT kernels: register butterflies (radix 2 .. 32), the
// twiddle table access, and the padded shared-memory position of an element. Shared by the grid's FFT
// passes (fft.cu, fft_two_kind.cu, fft_matrix.cu) and the beta transforms of the discrete Wigner transform (dwt_fixed.cu).
#pragma once

#include "common.cuh"
#include "fft_roots.cuh"

namespace pfsoft_dev {
namespace fftk {

constexpr double kSqrtHalf = 0.70710678118654752440084436210485;
constexpr double kCosPi8 = 0.92387953251128675612818318939679;   // cos(pi/8)
constexpr double kSinPi8 = 0.38268343236508977172845998403040;   // sin(pi/8)
constexpr double kSin60 = 0.86602540378443864676372317075294;    // sin(pi/3)
constexpr double kC5_1 = 0.30901699437494742410229341718282;     // cos(2pi/5)
constexpr double kC5_2 = -0.80901699437494742410229341718282;    // cos(4pi/5)
constexpr double kS5_1 = 0.95105651629515357211643933337938;     // sin(2pi/5)
constexpr double kS5_2 = 0.58778525229247312916870595463907;     // sin(4pi/5)

template <int SIGN>
__device__ __forceinline__ void dft2(double2* v)
{
    double2 a = v[0], b = v[1];
    v[0] = cadd(a, b);
    v[1] = csub(a, b);
}

template <int SIGN>
__device__ __forceinline__ void dft4(double2& v0, double2& v1, double2& v2, double2& v3)
{
    double2 a0 = cadd(v0, v2), a1 = csub(v0, v2);
    double2 b0 = cadd(v1, v3), b1 = cmul_i<SIGN>(csub(v1, v3));
    v0 = cadd(a0, b0);
    v2 = csub(a0, b0);
    v1 = cadd(a1, b1);
    v3 = csub(a1, b1);
}

// w8^q = exp(SIGN*2*pi*i*q/8)
template <int SIGN, int Q>
__device__ __forceinline__ double2 rot8(double2 a)
{
    if (Q == 0) return a;
    if (Q == 2) return cmul_i<SIGN>(a);
    if (Q == 1) return make_double2(kSqrtHalf * (a.x - SIGN * a.y), kSqrtHalf * (a.y + SIGN * a.x));
    // Q == 3: (-1 + SIGN i)/sqrt2
    return make_double2(kSqrtHalf * (-a.x - SIGN * a.y), kSqrtHalf * (-a.y + SIGN * a.x));
}

template <int SIGN>
__device__ __forceinline__ void dft8(double2* v)
{
    // even/odd split: E = DFT4(v0 v2 v4 v6), O = DFT4(v1 v3 v5 v7)
    dft4<SIGN>(v[0], v[2], v[4], v[6]);
    dft4<SIGN>(v[1], v[3], v[5], v[7]);
    double2 o1 = rot8<SIGN, 1>(v[3]), o2 = rot8<SIGN, 2>(v[5]), o3 = rot8<SIGN, 3>(v[7]);
    double2 e0 = v[0], e1 = v[2], e2 = v[4], e3 = v[6], o0 = v[1];
    v[0] = cadd(e0, o0);
    v[4] = csub(e0, o0);
    v[1] = cadd(e1, o1);
    v[5] = csub(e1, o1);
    v[2] = cadd(e2, o2);
    v[6] = csub(e2, o2);
    v[3] = cadd(e3, o3);
    v[7] = csub(e3, o3);
}

template <int SIGN>
__device__ __forceinline__ void dft16(double2* v)
{
    double2 e[8], o[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        e[i] = v[2 * i];
        o[i] = v[2 * i + 1];
    }
    dft8<SIGN>(e);
    dft8<SIGN>(o);
    // w16^q = (cos(pi q/8), SIGN sin(pi q/8))
    const double cq[8] = {1.0, kCosPi8, kSqrtHalf, kSinPi8, 0.0, -kSinPi8, -kSqrtHalf, -kCosPi8};
    const double sq[8] = {0.0, kSinPi8, kSqrtHalf, kCosPi8, 1.0, kCosPi8, kSqrtHalf, kSinPi8};
#pragma unroll
    for (int q = 0; q < 8; ++q) {
        double2 t = (q == 0) ? o[0] : make_double2(cq[q] * o[q].x - SIGN * sq[q] * o[q].y,
                                                    cq[q] * o[q].y + SIGN * sq[q] * o[q].x);
        v[q] = cadd(e[q], t);
        v[q + 8] = csub(e[q], t);
    }
}

template <int SIGN>
__device__ __forceinline__ void dft3(double2* v)
{
    double2 t1 = cadd(v[1], v[2]);
    double2 t2 = csub(v[1], v[2]);
    double2 a = make_double2(v[0].x - 0.5 * t1.x, v[0].y - 0.5 * t1.y);
    double2 b = cmul_i<SIGN>(cscale(t2, kSin60));
    v[0] = cadd(v[0], t1);
    v[1] = cadd(a, b);
    v[2] = csub(a, b);
}

template <int SIGN>
__device__ __forceinline__ void dft5(double2* v)
{
    double2 t1 = cadd(v[1], v[4]), t2 = cadd(v[2], v[3]);
    double2 t3 = csub(v[1], v[4]), t4 = csub(v[2], v[3]);
    double2 a1 = make_double2(v[0].x + kC5_1 * t1.x + kC5_2 * t2.x, v[0].y + kC5_1 * t1.y + kC5_2 * t2.y);
    double2 a2 = make_double2(v[0].x + kC5_2 * t1.x + kC5_1 * t2.x, v[0].y + kC5_2 * t1.y + kC5_1 * t2.y);
    double2 b1 = cmul_i<SIGN>(make_double2(kS5_1 * t3.x + kS5_2 * t4.x, kS5_1 * t3.y + kS5_2 * t4.y));
    double2 b2 = cmul_i<SIGN>(make_double2(kS5_2 * t3.x - kS5_1 * t4.x, kS5_2 * t3.y - kS5_1 * t4.y));
    v[0] = cadd(v[0], cadd(t1, t2));
    v[1] = cadd(a1, b1);
    v[4] = csub(a1, b1);
    v[2] = cadd(a2, b2);
    v[3] = csub(a2, b2);
}

__device__ __forceinline__ double2 twiddle(const double2* __restrict__ tw, int t, int sign)
{
    double2 w = __ldg(tw + t);
    return sign < 0 ? w : make_double2(w.x, -w.y);
}

// smem position of element i of a vector (one pad slot every 16 elements)
__device__ __forceinline__ int spos(int i) { return i + (i >> 4); }

__host__ __device__ __forceinline__ int padded_len(int n) { return n + (n >> 4) + 1; }

template <int SIGN, int R>
__device__ __forceinline__ void butterfly(double2* v);

// An odd prime R: the inputs k and R - k enter by their sum and difference.
template <int SIGN, int R>
__device__ __forceinline__ void dft_prime(double2* v)
{
    constexpr int h = (R - 1) / 2;
    double2 t[h], d[h];
#pragma unroll
    for (int k = 1; k <= h; ++k) {
        t[k - 1] = cadd(v[k], v[R - k]);
        d[k - 1] = csub(v[k], v[R - k]);
    }
    double2 sum = v[0];
#pragma unroll
    for (int q = 1; q <= h; ++q) {
        double2 a = v[0], b = make_double2(0.0, 0.0);
#pragma unroll
        for (int k = 1; k <= h; ++k) {
            const double c = root<R>(k * q % R).x, s = root<R>(k * q % R).y;
            a = make_double2(fma(c, t[k - 1].x, a.x), fma(c, t[k - 1].y, a.y));
            b = k == 1 ? cscale(d[0], s) : make_double2(fma(s, d[k - 1].x, b.x), fma(s, d[k - 1].y, b.y));
        }
        b = cmul_i<SIGN>(b);
        v[q] = cadd(a, b);
        v[R - q] = csub(a, b);
        sum = cadd(sum, t[q - 1]);
    }
    v[0] = sum;
}

// R = P Q: P-point DFTs of every Q-th input, the roots between, Q-point DFTs.
template <int SIGN, int P, int Q>
__device__ __forceinline__ void dft_product(double2* v)
{
    constexpr int R = P * Q;
    double2 u[Q][P];
#pragma unroll
    for (int j = 0; j < Q; ++j) {
#pragma unroll
        for (int i = 0; i < P; ++i) u[j][i] = v[i * Q + j];
        butterfly<SIGN, P>(u[j]);
    }
#pragma unroll
    for (int i = 0; i < P; ++i) {
        double2 w[Q];
#pragma unroll
        for (int j = 0; j < Q; ++j) {
            const int e = i * j % R;
            w[j] = e == 0 ? u[j][i] : cmul(u[j][i], make_double2(root<R>(e).x, SIGN * root<R>(e).y));
        }
        butterfly<SIGN, Q>(w);
#pragma unroll
        for (int j = 0; j < Q; ++j) v[i + P * j] = w[j];
    }
}

// Radix-R butterfly in registers (R = 1: a copy).
template <int SIGN, int R>
__device__ __forceinline__ void butterfly(double2* v)
{
    if constexpr (R == 2) dft2<SIGN>(v);
    else if constexpr (R == 3) dft3<SIGN>(v);
    else if constexpr (R == 4) dft4<SIGN>(v[0], v[1], v[2], v[3]);
    else if constexpr (R == 5) dft5<SIGN>(v);
    else if constexpr (R == 8) dft8<SIGN>(v);
    else if constexpr (R == 16) dft16<SIGN>(v);
    else if constexpr (R == 7 || R == 11 || R == 13 || R == 17 || R == 19 || R == 23 || R == 29 || R == 31) dft_prime<SIGN, R>(v);
    else if constexpr (R == 32) dft_product<SIGN, 4, 8>(v);
    else if constexpr (R == 24) dft_product<SIGN, 3, 8>(v);
    else if constexpr (R == 25) dft_product<SIGN, 5, 5>(v);
    else if constexpr (R == 30) dft_product<SIGN, 5, 6>(v);
    else if constexpr (R % 4 == 0) dft_product<SIGN, R / 4, 4>(v);       // 12, 20, 28
    else if constexpr (R % 3 == 0) dft_product<SIGN, R / 3, 3>(v);       // 6, 9, 15, 18, 21
    else if constexpr (R % 2 == 0) dft_product<SIGN, R / 2, 2>(v);       // 10, 14, 22, 26
    else static_assert(R == 1, "no butterfly for this radix");
}

}  // namespace fftk
}  // namespace pfsoft_dev
