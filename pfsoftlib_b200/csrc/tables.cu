// Per-bandwidth constant tables, computed on the device in FP64 once per bandwidth.
//
//   cos(beta_k), sin(beta_k/2), cos(beta_k/2)  beta_k = pi(2k+1)/(4B)     fn_dwt.hpp:155-159
//   w_B(j) = 2/B sin(pi(2j+1)/(4B)) sum_{k<B} sin((2j+1)(2k+1)pi/(4B))/(2k+1)   fn_dwt.hpp:62-83
//   twiddle[t] = exp(-2 pi i t/N), ht[n] = {cos, sin}(pi n/(2N))
//   delta: the Wigner rows at beta = pi/2, whose products are the rows' Fourier coefficients in beta
// and for the split-precision DWT alone
//   normf(M,M') = sqrt((2M+1)/2) prod_{i<M-M'} sqrt((2M-i)/(i+1))              fn_dwt.hpp:117-121
//   rc_cf / rc_f1: the recurrence coefficients c1, f1 f2 and f1 of every class and degree
//       (fn_dwt.hpp:167-199), so that the kernel loads them instead of recomputing them
//   pw_sin[p][k], pw_cos[p][k] = sin(beta_k/2)^p, cos(beta_k/2)^p, p < 2B, as an exact binary
//       exponent and a mantissa in [0.5, 1) (exponentiation by squaring, renormalised each
//       product), so that Wigner seeds far below the FP64 range keep full relative precision
// The sine arguments are reduced exactly in integers before sinpi/cospi, and the weight sum
// is compensated (Neumaier), so each entry is within a few ulp of the exact value.

#include <algorithm>

#include "common.cuh"
#include "dd.cuh"
#include "dwt.cuh"
#include "dwt_common.cuh"
#include "fft.cuh"

namespace pfsoft_dev {

namespace {

__host__ __device__ inline size_t align256(size_t x) { return (x + 255) & ~size_t(255); }

// x^p as {m, e}: x^p = m 2^e, m in [0.5, 1); x > 0
__device__ double2 ext_pow_tab(double x, int p)
{
    int xe;
    double xm = frexp(x, &xe);
    double rm = 1.0;
    int re = 0;
    while (p) {
        if (p & 1) {
            int t;
            rm = frexp(rm * xm, &t);
            re += xe + t;
        }
        p >>= 1;
        if (p) {
            int t;
            xm = frexp(xm * xm, &t);
            xe = 2 * xe + t;
        }
    }
    int t;
    rm = frexp(rm, &t);
    return make_double2(rm, (double)(re + t));
}

__global__ void powers_kernel(int B, const double* sinh, const double* cosh, double2* pw_sin, double2* pw_cos)
{
    const int N = 2 * B;
    const long long total = (long long)2 * B * N;
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < total; i += (long long)gridDim.x * blockDim.x) {
        const int p = (int)(i / N), k = (int)(i - (long long)p * N);
        pw_sin[i] = ext_pow_tab(sinh[k], p);
        pw_cos[i] = ext_pow_tab(cosh[k], p);
    }
}

__global__ void tables_kernel(int B, double* cosb, double* sinh, double* cosh, double* w,
                              double2* tw, double2* ht, int ra)
{
    const int N = 2 * B;
    const int tid = blockIdx.x * blockDim.x + threadIdx.x;
    const int nthr = gridDim.x * blockDim.x;
    for (int k = tid; k < N; k += nthr) {
        const double x = (double)(2 * k + 1) / (double)(4 * B);
        cosb[k] = cospi(x);
        double s, c;
        sincospi(0.5 * x, &s, &c);
        sinh[k] = s;
        cosh[k] = c;
        // twiddles of the length-N DFT
        double ts, tc;
        sincospi(2.0 * (double)k / (double)N, &ts, &tc);
        tw[k] = make_double2(tc, -ts);
        // the two-stage kernel's copy: exp(-2 pi i (r j mod N) / N), r = k / ra + 1, j = k mod ra
        if (ra) {
            sincospi(2.0 * (double)((k / ra + 1) * (k % ra) % N) / (double)N, &ts, &tc);
            tw[N + k] = make_double2(tc, -ts);
        }
        if (k < B) {
            sincospi((double)k / (double)(2 * N), &ts, &tc);
            ht[k] = make_double2(tc, ts);
        }
        // weights are symmetric, w(N-1-k) = w(k) (fn_dwt.hpp:80-81): compute k < B, mirror
        if (k >= B) continue;
        // exact integer reduction of (2k+1)(2q+1) modulo 8B (period of sin(pi p/(4B)))
        double sum = 0.0, comp = 0.0;
        const long long a = 2 * k + 1;
        for (int q = 0; q < B; ++q) {
            const long long p = (a * (2 * q + 1)) % (8LL * B);
            const double term = sinpi((double)p / (double)(4 * B)) / (double)(2 * q + 1);
            const double t = sum + term;
            comp += (fabs(sum) >= fabs(term)) ? (sum - t) + term : (term - t) + sum;
            sum = t;
        }
        const double wk = 2.0 / B * sinpi(x) * (sum + comp);
        w[k] = wk;
        w[N - 1 - k] = wk;
    }
}

// Seed norms of the order classes.
__global__ void normf_kernel(int B, double* normf)
{
    const int tid = blockIdx.x * blockDim.x + threadIdx.x;
    const int nthr = gridDim.x * blockDim.x;
    const int ncls = num_classes(B);
    for (int i = tid; i < ncls; i += nthr) {
        int M, Mp;
        class_orders(i, M, Mp);
        double nf = sqrt((2.0 * M + 1.0) / 2.0);
        for (int q = 0; q < M - Mp; ++q) nf *= sqrt((2.0 * M - q) / (q + 1.0));
        normf[i] = nf;
    }
}

// One CTA per order class: c1, f1 f2, f1 of the steps l -> l+1, l = M .. B-1.
__global__ void rc_kernel(int B, double2* rc_cf, double* rc_f1)
{
    int M, Mp;
    class_orders(blockIdx.x, M, Mp);
    const long long base = rc_offset(B, M, Mp);
    for (int l = M + threadIdx.x; l < B; l += blockDim.x) {
        double c1, f1, f2;
        dwtk::rec_coef(l, M, Mp, c1, f1, f2);
        rc_cf[base + (l - M)] = make_double2(c1, f1 * f2);
        rc_f1[base + (l - M)] = f1;
    }
}

// The cosines and sines of the beta sums (BandTables::trig); n (2k+1) is reduced modulo 8B, the period of
// the angle pi n (2k+1) / (4B).
__global__ void trig_kernel(int B, double* trig)
{
    const int nb = (B + 7) / 8, mb = (nb + 1) / 2;
    const long long total = trig_entries(B);
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < total; i += (long long)gridDim.x * blockDim.x) {
        const int tile = (int)(i / 64), kt = tile % nb, mt = tile / nb % mb, q = tile / (nb * mb) & 1, sine = tile / (2 * nb * mb);
        const int n = 2 * (8 * mt + (int)(i >> 3 & 7)) + q, k = 8 * kt + (int)(i & 7);
        double v = 0.0;
        if (n < B && k < B) {
            const double x = (double)(((long long)n * (2 * k + 1)) % (8LL * B)) / (double)(4 * B);
            v = (n == 0 ? 1.0 : 2.0) * (sine ? sinpi(x) : cospi(x));
        }
        trig[i] = v;
    }
}

// P[l][a][b] for one pair a >= b per eight lanes, l = a .. B-1, and its mirror image: the recurrence of
// fn_dwt.hpp:167-199 at cos beta = 0 without its normalisation,
//   P(l+1) = -((2l+1) a b P(l) + (l+1) sqrt(q(l)) P(l-1)) / (l sqrt(q(l+1))),  q(l) = (l^2-a^2)(l^2-b^2),
// from the seed, in double-double arithmetic (dd.cuh), which keeps the products of two entries within
// two ulp over any number of steps. The table starts zeroed.
// What bounds it: the chain over l. A lane takes one of a tile's eight degrees for what does not depend on
// the chain (the two factors with their roots and quotients, the norm), all eight run the chain, two products
// and a sum a step. One thread per pair, roots and quotients in the chain, against this, us, cold: B = 8
// 14.6 / 7.0, 32 43 / 15, 64 80 / 24, 128 150 / 50, 256 294 / 136, 384 466 / 399.
__global__ void delta_kernel(int B, double* delta)
{
    const int i = (blockIdx.x * blockDim.x + threadIdx.x) >> 3, lane = threadIdx.x & 7;
    if (i >= num_classes(B)) return;
    const unsigned group = 0xffu << (threadIdx.x & 24);
    auto from = [&](dd v, int src) { return dd{__shfl_sync(group, v.h, src, 8), __shfl_sync(group, v.l, src, 8)}; };
    int a, b;
    class_orders(i, a, b);
    dd cur = seed_part(a, b, lane), prev = {0.0, 0.0};
    for (int s = kSeedParts / 2; s > 0; s /= 2)
        cur = dd_mul(cur, dd{__shfl_xor_sync(group, cur.h, s, 8), __shfl_xor_sync(group, cur.l, s, 8)});
    cur = seed_of(from(cur, 0), a);
    auto at = [&](int M, int n, int l) {
        const int lb = l >> 3, b0 = M >> 3;
        return delta_offset(B, M) + 64 * (long long)(lb * (lb + 1) / 2 - b0 * (b0 + 1) / 2 + (n >> 3)) + (l & 7) * 8 + (n & 7);
    };
    auto root = [&](int l) {   // sqrt(q(l)), q an exact integer
        const double k2 = (double)l * l;
        return dd_sqrt(dd{(k2 - (double)a * a) * (k2 - (double)b * b), 0.0});
    };
    for (int l0 = a & ~7; l0 < B; l0 += 8) {
        const int l = l0 + lane;
        dd f1 = {0.0, 0.0}, f2 = {0.0, 0.0}, mine = {0.0, 0.0};
        if (l >= a && l > 0) {
            const dd inv = dd_div(dd{1.0, 0.0}, dd_scale(root(l + 1), (double)l));
            f1 = dd_scale(inv, -(double)(2 * l + 1) * a * b);
            f2 = dd_mul(dd_scale(root(l), -(double)(l + 1)), inv);
        }
#pragma unroll
        for (int j = 0; j < 8; ++j) {
            const dd g1 = from(f1, j), g2 = from(f2, j);
            if (l0 + j < a) continue;
            if (lane == j) mine = cur;
            const dd next = dd_add(dd_mul(g1, cur), dd_mul(g2, prev));
            prev = cur;
            cur = next;
        }
        if (l < a || l >= B) continue;
        // with a fourth root of the rows' squared norm, so that a product of two has its square root
        const dd x = dd_mul(mine, dd_sqrt(dd_sqrt(dd{l + 0.5, 0.0})));
        const double v = x.h + x.l;
        delta[at(a, b, l)] = v;
        if (a != b) delta[at(b, a, l)] = ((a - b) & 1) ? -v : v;
    }
}

}  // namespace

size_t tables_bytes(int B)
{
    const size_t N = 2 * (size_t)B;
    return 4 * align256(N * sizeof(double)) + align256(fft_twiddle_elems((int)N) * sizeof(double2)) +
           align256(B * sizeof(double2));
}

cudaError_t tables_build(int B, void* mem, BandTables* t, cudaStream_t stream)
{
    const size_t N = 2 * (size_t)B;
    char* p = static_cast<char*>(mem);
    *t = BandTables();
    t->B = B;
    t->N = (int)N;
    t->block = mem;
    auto take = [&](size_t bytes) {
        char* q = p;
        p += align256(bytes);
        return q;
    };
    t->cosb = reinterpret_cast<double*>(take(N * sizeof(double)));
    t->sinh = reinterpret_cast<double*>(take(N * sizeof(double)));
    t->cosh = reinterpret_cast<double*>(take(N * sizeof(double)));
    t->w = reinterpret_cast<double*>(take(N * sizeof(double)));
    t->twiddle = reinterpret_cast<double2*>(take(fft_twiddle_elems((int)N) * sizeof(double2)));
    t->ht = reinterpret_cast<double2*>(take(B * sizeof(double2)));
    const int threads = 64;
    int ra = 0, rb = 0;
    if (!fft_two_radices((int)N, &ra, &rb)) ra = 0;
    tables_kernel<<<((int)N + threads - 1) / threads, threads, 0, stream>>>(B, t->cosb, t->sinh, t->cosh, t->w,
                                                                             t->twiddle, t->ht, ra);
    return cudaGetLastError();
}

size_t series_tables_bytes(int B)
{
    return align256((size_t)delta_entries(B) * sizeof(double)) + align256((size_t)trig_entries(B) * sizeof(double));
}

cudaError_t series_tables_build(int B, void* mem, BandTables* t, cudaStream_t stream)
{
    const size_t dbytes = (size_t)delta_entries(B) * sizeof(double);
    double* delta = static_cast<double*>(mem);
    double* trig = reinterpret_cast<double*>(static_cast<char*>(mem) + align256(dbytes));
    const int threads = 64;
    cudaError_t e = cudaMemsetAsync(delta, 0, dbytes, stream);
    if (e != cudaSuccess) return e;
    delta_kernel<<<(8 * num_classes(B) + threads - 1) / threads, threads, 0, stream>>>(B, delta);
    e = cudaGetLastError();
    if (e != cudaSuccess) return e;
    trig_kernel<<<(int)std::min<long long>((trig_entries(B) + 255) / 256, 1024), 256, 0, stream>>>(B, trig);
    t->delta = delta;
    t->trig = trig;
    return cudaGetLastError();
}

size_t split_tables_bytes(int B)
{
    const size_t N = 2 * (size_t)B, R = (size_t)rc_entries(B);
    return align256(num_classes(B) * sizeof(double)) + 2 * align256(N * N * sizeof(double2)) +
           align256(R * sizeof(double2)) + align256(R * sizeof(double));
}

cudaError_t split_tables_build(int B, void* mem, BandTables* t, cudaStream_t stream)
{
    const size_t N = 2 * (size_t)B;
    char* p = static_cast<char*>(mem);
    t->normf = reinterpret_cast<double*>(p);
    p += align256(num_classes(B) * sizeof(double));
    t->pw_sin = reinterpret_cast<double2*>(p);
    p += align256(N * N * sizeof(double2));
    t->pw_cos = reinterpret_cast<double2*>(p);
    p += align256(N * N * sizeof(double2));
    t->rc_cf = reinterpret_cast<double2*>(p);
    p += align256((size_t)rc_entries(B) * sizeof(double2));
    t->rc_f1 = reinterpret_cast<double*>(p);
    const int threads = 128;
    normf_kernel<<<(num_classes(B) + threads - 1) / threads, threads, 0, stream>>>(B, t->normf);
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return e;
    const long long total = (long long)N * N;
    int pblocks = (int)((total + 255) / 256);
    if (pblocks > 4096) pblocks = 4096;
    powers_kernel<<<pblocks, 256, 0, stream>>>(B, t->sinh, t->cosh, t->pw_sin, t->pw_cos);
    e = cudaGetLastError();
    if (e != cudaSuccess) return e;
    rc_kernel<<<num_classes(B), 128, 0, stream>>>(B, t->rc_cf, t->rc_f1);
    return cudaGetLastError();
}

}  // namespace pfsoft_dev
