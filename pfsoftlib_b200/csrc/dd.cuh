// Double-double arithmetic (Dekker 1971, Knuth; products by FMA) and the seeds of the Wigner rows at beta = pi/2
// that need it. Host and device, so that the seeds can be checked without a GPU.
#pragma once

#include <cuda_runtime.h>
#include <math.h>

namespace pfsoft_dev {

struct dd {
    double h, l;
};
__host__ __device__ __forceinline__ dd quick_sum(double a, double b)   // |a| >= |b|
{
    const double s = a + b;
    return {s, b - (s - a)};
}
__host__ __device__ __forceinline__ dd dd_add(dd a, dd b)
{
    const double s = a.h + b.h, v = s - a.h;
    const double e = (a.h - (s - v)) + (b.h - v);
    return quick_sum(s, e + a.l + b.l);
}
__host__ __device__ __forceinline__ dd dd_mul(dd a, dd b)
{
    const double p = a.h * b.h;
    return quick_sum(p, fma(a.h, b.h, -p) + (a.h * b.l + a.l * b.h));
}
__host__ __device__ __forceinline__ dd dd_scale(dd a, double b)
{
    const double p = a.h * b;
    return quick_sum(p, fma(a.h, b, -p) + a.l * b);
}
__host__ __device__ __forceinline__ dd dd_div(dd a, dd b)
{
    const double q = a.h / b.h;
    const dd r = dd_add(a, dd_scale(b, -q));
    return quick_sum(q, (r.h + r.l) / b.h);
}
__host__ __device__ __forceinline__ dd dd_sqrt(dd a)
{
    if (a.h == 0.0) return {0.0, 0.0};
    const double r = sqrt(a.h);
    return quick_sum(r, (fma(-r, r, a.h) + a.l) / (2.0 * r));
}

// P[a][a][b] = sqrt(binomial(2a, a - b)) 2^-a, a >= b >= 0. The binomial passes the double range from a = 511
// on (its largest, times the next factor, 2^1025.7); an even power of two taken out on the way keeps every step
// in range and the digits as they are.
__host__ __device__ __forceinline__ dd delta_seed(int a, int b)
{
    dd c = {1.0, 0.0};
    int e = 0;
    for (int q = 0; q < a - b; ++q) {
        c = dd_div(dd_scale(c, (double)(2 * a - q)), dd{(double)(q + 1), 0.0});
        if (c.h >= 0x1p600) {
            c.h *= 0x1p-600;
            c.l *= 0x1p-600;
            e += 300;   // of the square root
        }
    }
    c = dd_sqrt(c);
    return {ldexp(c.h, e - a), ldexp(c.l, e - a)};
}

}  // namespace pfsoft_dev
