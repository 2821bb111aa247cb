// DFT passes of lengths n = R p with an odd p, mostly a large prime, on the FP64 MMA (sm_100a).
//
// With u_q[j] = w_n^(j q) sum_s x[j + s p] w_R^(s q) (a radix-R butterfly per j < p), output q + R k is the
// p-point DFT of u_q at k. Its inputs j and p - j enter by their sum t_j and difference d_j, and outputs k
// and p - k share both halves:
//
//   X[q + R k], X[q + R (p - k)] = C_k +- i sign S_k,  C_k = sum_j cos(2 pi j k / p) t_j,
//                                                      S_k = sum_j sin(2 pi j k / p) d_j,  j, k <= (p-1)/2
//
// two real matrix products of ((p+1)/2)^2 with a table of tiles (a.bluestein), p multiply-adds per point in
// all. A CTA takes 8 vectors: its columns of t and d lie in shared memory as B fragments, each warp takes
// up to MT row tiles of one q at a time, real and imaginary parts with the same table values.
//
// What bounds it: the FP64 unit from p of about 60 on (the multiply-adds that fit the HBM time number 90
// per point): 70 % busy at n = 274, with the shared-memory pipe at 73 %. Against the chirp pass, us per
// pass: n = 34 8.7 / 11, 74 11 / 19, 148 38 / 75, 222 136 / 240, 274 285 / 464, 346 621 / 1000, 370 563 /
// 1150, 444 1030 / 1800, 478 1957 / 2120, 502 2405 / 2370: the cost grows with p, which ends at 249.

#include <algorithm>
#include <cmath>
#include <vector>

#include "common.cuh"
#include "dwt.cuh"
#include "dwt_common.cuh"
#include "fft.cuh"
#include "fft_core.cuh"

namespace pfsoft_dev {

namespace {

using namespace fftk;
using dwtk::dmma;

constexpr int kMaxR = 12, kMaxP = 249;
constexpr int kMaxTiles = 64;   // shared memory of a CTA, 2 KB each: 128 KB

// Row k of a block of B fragments: vector kk at column 2 (kk & 3) + kk / 4, so that the accumulators' columns
// 2 t + u of a warp's four t are neighbours in HBM; the columns are swizzled by the row so that rows
// k = t, t < 4 (or 4 + t) and columns of a fragment read, eight rows of one vector, and eight vectors of
// one row all meet distinct 16-byte banks.
__device__ __forceinline__ int swizzle(int k) { return ((k & 3) << 1) | ((k >> 2) & 1); }
__device__ __forceinline__ int place(int k, int kk) { return 8 * k + ((2 * (kk & 3) + (kk >> 2)) ^ swizzle(k)); }

// The radix-R butterflies of j and p - j, and their sums and differences into the blocks of every q.
template <int SIGN, int R>
__device__ __forceinline__ void load_tile(const FftPassArgs& a, const double2* src, double2* smem, int nv, int p)
{
    const int h1 = (p + 1) / 2, rows = (h1 + 7) & ~7;
    const bool across = a.src.se != 1;
    const unsigned inv = 0xffffffffu / (unsigned)h1 + 1u;
    for (int t = threadIdx.x; t < 8 * h1; t += blockDim.x) {
        const int kk = across ? t & 7 : (int)__umulhi((unsigned)t, inv);   // t / h1
        const int j = across ? t >> 3 : t - kk * h1;
        if (kk >= nv) continue;   // a column that is not there touches no other
        const double2* x = src + (long long)kk * a.src.sv;
        const int j2 = j ? p - j : 0;
        double2 u[R], v[R];
#pragma unroll
        for (int s = 0; s < R; ++s) {
            u[s] = __ldg(x + (long long)(j + s * p) * a.src.se);
            v[s] = __ldg(x + (long long)(j2 + s * p) * a.src.se);
        }
        butterfly<SIGN, R>(u);
        butterfly<SIGN, R>(v);
        double2* o = smem + place(j, kk);
#pragma unroll
        for (int q = 0; q < R; ++q) {
            if (q > 0) {
                u[q] = cmul(u[q], twiddle(a.twiddle, j * q, SIGN));
                v[q] = cmul(v[q], twiddle(a.twiddle, j2 * q, SIGN));
            }
            o[16 * q * rows] = j ? cadd(u[q], v[q]) : u[q];
            o[16 * q * rows + 8 * rows] = csub(u[q], v[q]);   // j = 0: zero
        }
    }
    // rows past the last: zeros meet the table's zeros
    const int pad = 8 * (rows - h1);
    for (int t = threadIdx.x; t < 2 * R * pad; t += blockDim.x)
        smem[(t / pad) * 8 * rows + 8 * h1 + t % pad] = make_double2(0.0, 0.0);
}

template <int SIGN, int R, int RMAX>
__device__ __forceinline__ void load_any(const FftPassArgs& a, const double2* src, double2* smem, int nv, int p)
{
    if (a.radix[0] == R) load_tile<SIGN, R>(a, src, smem, nv, p);
    else if constexpr (R < RMAX) load_any<SIGN, R + 1, RMAX>(a, src, smem, nv, p);
}

// Row tiles m0 .. m0 + MT - 1 of outputs q + R k and q + R (p - k).
template <int SIGN, int MT>
__device__ __forceinline__ void product(const FftPassArgs& a, double2* dst, const double2* smem, int nv, int p, int q, int m0)
{
    const int lane = threadIdx.x & 31, g = lane >> 2, t4 = lane & 3;
    const int h1 = (p + 1) / 2, nt = (h1 + 7) >> 3, R = a.radix[0];
    const double2* A = a.bluestein + (size_t)64 * m0 * nt + lane;
    const double2* b0 = smem + 128 * nt * q + 8 * t4 + (g ^ (2 * t4));
    const double2* b1 = smem + 128 * nt * q + 8 * (4 + t4) + (g ^ (2 * t4 + 1));
    double acc[MT][2][2][2];
#pragma unroll
    for (int m = 0; m < MT; ++m)
#pragma unroll
        for (int i = 0; i < 8; ++i) acc[m][i >> 2][(i >> 1) & 1][i & 1] = 0.0;
    const int half = (h1 + 3) >> 2;   // steps of four rows
#pragma unroll 2
    for (int kt = 0; kt < half >> 1; ++kt) {
        double2 c[MT], s[MT];
#pragma unroll
        for (int m = 0; m < MT; ++m) {
            c[m] = __ldg(A + 64 * m * nt);
            s[m] = __ldg(A + 64 * m * nt + 32);
        }
        const double2 t0 = b0[0], d0 = b0[64 * nt], t1 = b1[0], d1 = b1[64 * nt];
        A += 64;
        b0 += 64;
        b1 += 64;
#pragma unroll
        for (int m = 0; m < MT; ++m) {
            dmma(acc[m][0][0][0], acc[m][0][0][1], c[m].x, t0.x);
            dmma(acc[m][0][1][0], acc[m][0][1][1], c[m].x, t0.y);
            dmma(acc[m][1][0][0], acc[m][1][0][1], s[m].x, d0.x);
            dmma(acc[m][1][1][0], acc[m][1][1][1], s[m].x, d0.y);
        }
#pragma unroll
        for (int m = 0; m < MT; ++m) {
            dmma(acc[m][0][0][0], acc[m][0][0][1], c[m].y, t1.x);
            dmma(acc[m][0][1][0], acc[m][0][1][1], c[m].y, t1.y);
            dmma(acc[m][1][0][0], acc[m][1][0][1], s[m].y, d1.x);
            dmma(acc[m][1][1][0], acc[m][1][1][1], s[m].y, d1.y);
        }
    }
    if (half & 1) {
        const double2 t0 = b0[0], d0 = b0[64 * nt];
#pragma unroll
        for (int m = 0; m < MT; ++m) {
            const double c = __ldg(A + 64 * m * nt).x, s = __ldg(A + 64 * m * nt + 32).x;
            dmma(acc[m][0][0][0], acc[m][0][0][1], c, t0.x);
            dmma(acc[m][0][1][0], acc[m][0][1][1], c, t0.y);
            dmma(acc[m][1][0][0], acc[m][1][0][1], s, d0.x);
            dmma(acc[m][1][1][0], acc[m][1][1][1], s, d0.y);
        }
    }
#pragma unroll
    for (int u = 0; u < 2; ++u) {
        const int kk = t4 + 4 * u;
        if (kk >= nv) continue;
        double2* y = dst + (long long)kk * a.dst.sv;
#pragma unroll
        for (int m = 0; m < MT; ++m) {
            const int k = 8 * (m0 + m) + g;
            if (k >= h1) continue;
            const double2 c = make_double2(acc[m][0][0][u], acc[m][0][1][u]);
            const double2 is = cmul_i<SIGN>(make_double2(acc[m][1][0][u], acc[m][1][1][u]));
            y[(long long)(q + R * k) * a.dst.se] = cscale(cadd(c, is), a.scale);
            if (k > 0) y[(long long)(q + R * (p - k)) * a.dst.se] = cscale(csub(c, is), a.scale);
        }
    }
}

template <int SIGN, int RMAX, int THREADS, int BLOCKS, int MT>
__global__ void __launch_bounds__(THREADS, BLOCKS)
    fft_matrix_kernel(const double2* src, double2* dst, const __grid_constant__ FftPassArgs a)
{
    extern __shared__ double2 smem[];
    if (a.srcs) {
        src = a.srcs[blockIdx.z];
        dst = a.dsts[blockIdx.z];
    }
    const int v0 = blockIdx.x * 8, nv = min(8, a.nvec - v0), R = a.radix[0], p = a.radix[1];
    src += (long long)v0 * a.src.sv + (long long)blockIdx.y * a.src.sb;
    dst += (long long)v0 * a.dst.sv + (long long)blockIdx.y * a.dst.sb;
    load_any<SIGN, 1, RMAX>(a, src, smem, nv, p);
    __syncthreads();   // in place: every input of the tile has been read
    // a q's row tiles in groups of at most MT, as even as they come; the warp that has one item more
    // changes from CTA to CTA
    const int nt = ((p + 1) / 2 + 7) >> 3, groups = (nt + MT - 1) / MT, low = nt / groups, more = nt - low * groups;
    for (int i = ((threadIdx.x >> 5) + blockIdx.x) % (THREADS / 32); i < R * groups; i += THREADS / 32) {
        const int q = i % R, gr = i / R, m0 = low * gr + min(gr, more), count = low + (gr < more);
        if (count == MT) product<SIGN, MT>(a, dst, smem, nv, p, q, m0);
        else product<SIGN, 1>(a, dst, smem, nv, p, q, m0);
    }
}

}  // namespace

bool fft_matrix_radices(int n, int* r, int* p)
{
    // the smallest odd factor that leaves a butterfly of at most kMaxR points
    for (int m = 17; m <= kMaxP && m <= n; m += 2)
        if (n % m == 0 && n / m <= kMaxR) {
            *r = n / m;
            *p = m;
            return n / m * (((m + 1) / 2 + 7) / 8) <= kMaxTiles;
        }
    return false;
}

size_t fft_matrix_elems(int p)
{
    const size_t nt = ((p + 1) / 2 + 7) / 8;
    return 64 * nt * nt;
}

void fft_matrix_fill(int p, double2* out)
{
    typedef long double ld;
    const ld pi = 3.14159265358979323846264338327950288L;
    const int h1 = (p + 1) / 2, nt = (h1 + 7) / 8;
    std::vector<double> c(p), s(p);
    for (int t = 0; t < p; ++t) {
        c[t] = (double)cosl(2 * pi * (ld)t / (ld)p);
        s[t] = (double)sinl(2 * pi * (ld)t / (ld)p);
    }
    // tile (row, column): lane 4 g + t holds the cosines, then the sines, of row g, columns t and 4 + t
    for (int m = 0; m < nt; ++m)
        for (int k = 0; k < nt; ++k)
            for (int lane = 0; lane < 32; ++lane) {
                const int row = 8 * m + lane / 4, j0 = 8 * k + lane % 4, j1 = j0 + 4;
                const int e0 = row * j0 % p, e1 = row * j1 % p;
                const bool in0 = row < h1 && j0 < h1, in1 = row < h1 && j1 < h1;
                double2* o = out + (size_t)64 * (m * nt + k) + lane;
                o[0] = make_double2(in0 ? c[e0] : 0.0, in1 ? c[e1] : 0.0);
                o[32] = make_double2(in0 ? s[e0] : 0.0, in1 ? s[e1] : 0.0);
            }
}

cudaError_t fft_matrix_launch(const double2* src, double2* dst, const FftPassArgs& a0, int ntiles, int sign, cudaStream_t stream,
                              int nz)
{
    FftPassArgs a = a0;
    if (!fft_matrix_radices(a.n, &a.radix[0], &a.radix[1])) return cudaErrorInvalidValue;
    const int R = a.radix[0], nt = ((a.radix[1] + 1) / 2 + 7) / 8;
    const size_t smem = (size_t)R * 128 * nt * sizeof(double2);
    auto go = [&](auto k, int threads) -> cudaError_t {
        const cudaError_t e = allow_shared(k, smem, (size_t)kMaxTiles * 128 * sizeof(double2));
        if (e != cudaSuccess) return e;
        k<<<dim3((a.nvec + 7) / 8, ntiles, nz), threads, smem, stream>>>(src, dst, a);
        return cudaGetLastError();
    };
    // Two row tiles at a time halve the shared-memory reads, single ones spread better over the warps where
    // there are few (us per pass: n = 274 285 single, 304 in pairs; 478 2220 and 1957). The butterflies of
    // radices 5 .. 12 take 168 registers; 12 warps of them hide more than 9 (n = 370 563 against 590, 444
    // 1030 against 1230).
    if (R > 4) return sign < 0 ? go(fft_matrix_kernel<-1, kMaxR, 192, 2, 1>, 192) : go(fft_matrix_kernel<1, kMaxR, 192, 2, 1>, 192);
    if (nt <= 9) return sign < 0 ? go(fft_matrix_kernel<-1, 4, 128, 4, 1>, 128) : go(fft_matrix_kernel<1, 4, 128, 4, 1>, 128);
    return sign < 0 ? go(fft_matrix_kernel<-1, 4, 192, 3, 2>, 192) : go(fft_matrix_kernel<1, 4, 192, 3, 2>, 192);
}

}  // namespace pfsoft_dev
