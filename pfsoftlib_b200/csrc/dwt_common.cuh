// Device helpers of the discrete Wigner transform kernels (dwt.cu, dwt_split.cu): recurrence
// coefficients, table seeds, the FP64 MMA and the class lists.
#pragma once

#include "common.cuh"
#include "dwt.cuh"

namespace pfsoft_dev {
namespace dwtk {

constexpr double kPi = 3.141592653589793;

// Recurrence step degree l -> l+1 for orders (M, Mp) (fn_dwt.hpp:167-192):
//   d(l+1) = c1 d(l-1) + d(l) f1 (f2 + cos beta)
__device__ __forceinline__ void rec_coef(int l, int M, int Mp, double& c1, double& f1, double& f2)
{
    const double idx = (double)l;
    const double nrm = sqrt((2.0 * idx + 3.0) / (2.0 * idx + 1.0));
    const double nom = (idx + 1.0) * (2.0 * idx + 1.0);
    const double a1 = (idx + 1.0) * (idx + 1.0) - (double)M * M;   // exact integers
    const double a2 = (idx + 1.0) * (idx + 1.0) - (double)Mp * Mp;
    const double den = 1.0 / sqrt(a1 * a2);
    f1 = nrm * nom * den;
    c1 = 0.0;
    f2 = 0.0;
    if (l != 0) {
        const double t1 = sqrt((2.0 * idx + 3.0) / (2.0 * idx - 1.0)) * (idx + 1.0) / idx;
        const double t2 = sqrt((idx * idx - (double)M * M) * (idx * idx - (double)Mp * Mp));
        c1 = -t1 * t2 * den;
        f2 = -(double)M * Mp / (idx * (idx + 1.0));
    }
}

// Seed of one beta column with its scale count (see the header comment): nf_w * s * c where s
// and c are table powers {mantissa, exponent}.
__device__ __forceinline__ double seed_value(double nf_w, double2 s, double2 c, int& sc)
{
    int ev;
    const double v = frexp(nf_w * s.x * c.x, &ev);
    const int E = ev + (int)s.y + (int)c.y;
    if (E >= -900) {
        sc = 0;
        return -ldexp(v, E);
    }
    sc = (-900 - E + 599) / 600;
    return -ldexp(v, E + 600 * sc);
}

__device__ __forceinline__ double case_sign(const PairCase& p, int l, int M)
{
    return (p.rev && ((l - M) & 1)) ? -p.s0 : p.s0;
}

// One FP64 MMA: C(8x8) += A(8x4, row) * B(4x8, col). Fragments per lane (g = lane/4, t = lane%4):
// A[g][t], B[t][g], C[g][2t], C[g][2t+1].
__device__ __forceinline__ void dmma(double& c0, double& c1, double a, double b)
{
    asm("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0,%1}, {%2}, {%3}, {%0,%1};"
        : "+d"(c0), "+d"(c1)
        : "d"(a), "d"(b));
}

// The i-th class of the launch (all classes in order when no subset is given).
__device__ __forceinline__ int list_class(const DwtArgs& a, int i) { return a.classes ? __ldg(a.classes + i) : i; }

}  // namespace dwtk
}  // namespace pfsoft_dev
