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

// P[a][a][b] = sqrt(binomial(2a, a - b)) 2^-a, a >= b >= 0, the binomial as eight partial products of every
// eighth factor (2a - q) / (q + 1), q < a - b, which are all at least 1: no product in between passes the
// whole, 2^1016.7 at a = 511 (one long product, multiplied before it is divided, passes the double range
// there).
constexpr int kSeedParts = 8;
__host__ __device__ __forceinline__ dd seed_part(int a, int b, int first)
{
    dd c = {1.0, 0.0};
    for (int q = first; q < a - b; q += kSeedParts) c = dd_div(dd_scale(c, (double)(2 * a - q)), dd{(double)(q + 1), 0.0});
    return c;
}
__host__ __device__ __forceinline__ dd seed_of(dd binomial, int a)
{
    const dd r = dd_sqrt(binomial);
    return {ldexp(r.h, -a), ldexp(r.l, -a)};
}
inline dd delta_seed(int a, int b)   // as eight lanes compute it
{
    dd c[kSeedParts];
    for (int i = 0; i < kSeedParts; ++i) c[i] = seed_part(a, b, i);
    for (int s = kSeedParts / 2; s > 0; s /= 2)
        for (int i = 0; i < s; ++i) c[i] = dd_mul(c[i], c[i + s]);
    return seed_of(c[0], a);
}

}  // namespace pfsoft_dev
