// What the kernels of the FP64 discrete Wigner transform share (dwt.cu: the design; the matrix form; dwt_fixed.cu: the
// form with a compile-time DFT over beta): an item's description, the sums over the series on the FP64 MMA in
// both directions, the Nyquist bins, the launch.
#pragma once

#include <algorithm>

#include "common.cuh"
#include "dwt.cuh"
#include "dwt_common.cuh"

namespace pfsoft_dev {
namespace dwtk {

struct CaseInfo {
    long long col;   // the case's beta column in X (double2 elements)
    int i1, i2;      // its place in degree l's block: i2 (2l+1) + i1, plus (2l+1) to each that is negative
    double s0;       // sign with the series' own sign
};

__device__ __forceinline__ void copy_async16(double2* dst, const double2* src)
{
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((unsigned)__cvta_generic_to_shared(dst)), "l"(src)
                 : "memory");
}
__device__ __forceinline__ void copy_async_wait() { asm volatile("cp.async.wait_all;" ::: "memory"); }

__device__ __forceinline__ int tri(int x) { return x * (x + 1) / 2; }

// Where the series table's tiles of order M count from: tile (lb, jb) -- degrees 8 lb .. 8 lb + 7,
// coefficients 8 jb .. 8 jb + 7, row-major -- is at tiles_at + 64 (tri(lb) + jb) doubles (32 bits: B <= 512).
__device__ __forceinline__ int tiles_at(int B, int M) { return (int)delta_offset(B, M) - 64 * tri(M >> 3); }

// Packed index of degree l's coefficient of the case (coef_index in 32 bits: B <= 512).
__device__ __forceinline__ int case_index(int i1, int i2, int l)
{
    const int L = 2 * l + 1;
    return (int)((unsigned)(l * (4 * l * l - 1)) / 3u) + (i2 < 0 ? i2 + L : i2) * L + (i1 < 0 ? i1 + L : i1);
}

// The launch's items, one per CTA: every class (of the list) of every transform, a class's transforms side by
// side, longest classes first.
struct Item {
    int M, Mp, nc, odd, tr;
    int rev;           // bit c: case c is read at pi - beta
    int offM, offP;    // both orders' tiles in the series table (tiles_at)
};

// Item i and its cases into shared memory (threads 0..7); the caller's barrier follows.
__device__ __forceinline__ void fill_item(const DwtArgs& a, int i, int N, Item* item, CaseInfo* cases)
{
    if (threadIdx.x < 8) {
        const int c = threadIdx.x;
        Item it;
        it.tr = a.T > 1 ? i % a.T : 0;
        class_orders(list_class(a, a.T > 1 ? i / a.T : i), it.M, it.Mp);
        it.nc = class_case_count(it.M, it.Mp);
        it.odd = (it.M - it.Mp) & 1;
        const PairCase p = class_case(it.M, it.Mp, c < it.nc ? c : 0, N);
        const int q = (it.M - it.Mp) & 3;
        CaseInfo ci;
        ci.col = ((long long)p.row * N + p.col) * N;
        ci.i1 = p.m1;
        ci.i2 = p.m2;
        ci.s0 = (q == 1 || q == 2) ? p.s0 : -p.s0;   // p.s0 carries the rows' seed sign -1
        cases[c] = ci;
        it.rev = (int)(__ballot_sync(0xffu, p.rev) & 0xffu);
        it.offM = tiles_at(a.B, it.M);
        it.offP = tiles_at(a.B, it.Mp);
        if (c == 0) *item = it;
    }
}

// Place of T[n][case c] (double2) in the forward's B-fragment order: tiles of 8 n; lane (c, t) of a warp
// reads n = 2 t and 2 t + 1 in two conflict-free accesses.
__device__ __forceinline__ int frag_pos(int n, int c)
{
    return (n >> 3) * 64 + c * 8 + ((((n & 1) << 2) | ((n >> 1) & 3)) ^ ((c & 1) << 2));
}

// An item's sums over n. A warp takes every NW-th block of 8 degrees, in snake order from the last block
// down, all of them along the tile columns so that they share the B fragments (those of columns >= nc
// are never stored); tile column jb is in the blocks from jb on: `COUNT` of the warp's.
template <int NW, int KP>
struct ForwardSums {
    double acc[KP][2][2];
    const double2 *x[KP], *y[KP];   // tile column jb of the blocks, both orders, the lane's element
    const double2 *f0, *f1;         // the column's fragments

    template <int COUNT>
    __device__ __forceinline__ void column()
    {
        double2 d[COUNT];
#pragma unroll
        for (int p = 0; p < COUNT; ++p) {
            const double2 u = __ldg(x[p]), v = __ldg(y[p]);
            d[p] = make_double2(u.x * v.x, u.y * v.y);
            x[p] += 32;
            y[p] += 32;
        }
        const double2 t0 = *f0, t1 = *f1;
        f0 += 64;
        f1 += 64;
#pragma unroll
        for (int p = 0; p < COUNT; ++p) {
            dmma(acc[p][0][0], acc[p][0][1], d[p].x, t0.x);
            dmma(acc[p][1][0], acc[p][1][1], d[p].x, t0.y);
        }
#pragma unroll
        for (int p = 0; p < COUNT; ++p) {
            dmma(acc[p][0][0], acc[p][0][1], d[p].y, t1.x);
            dmma(acc[p][1][0], acc[p][1][1], d[p].y, t1.y);
        }
    }
    template <int COUNT>
    __device__ __forceinline__ void columns(int& jb, const int (&lb)[KP])
    {
#pragma unroll 2
        for (; jb <= lb[COUNT - 1]; ++jb) column<COUNT>();
        if constexpr (COUNT > 1) columns<COUNT - 1>(jb, lb);
    }
};

template <int NW, int KP>
__device__ __forceinline__ void forward_sums(const double* tM, const double* tP, const double2* frag, int B, const Item& it,
                                             const CaseInfo* cases, double2* out)
{
    // which warp takes the last block changes from CTA to CTA: short classes leave warps without one
    const int lane = threadIdx.x & 31, warp = ((threadIdx.x >> 5) + blockIdx.x) & (NW - 1), g = lane >> 2, t4 = lane & 3;
    const int nb = (B + 7) >> 3, lbM = it.M >> 3;
    const double norm = kPi / (double)(B * 2 * B);   // src/fn_dsoft.cpp:119
    ForwardSums<NW, KP> s;
    int lb[KP];
#pragma unroll
    for (int p = 0; p < KP; ++p) {
        const int b = nb - 1 - (p * NW + ((p & 1) ? NW - 1 - warp : warp));
        lb[p] = b >= lbM ? b : -1;
        s.x[p] = reinterpret_cast<const double2*>(tM) + 32 * tri(b) + lane;
        s.y[p] = reinterpret_cast<const double2*>(tP) + 32 * tri(b) + lane;
        s.acc[p][0][0] = s.acc[p][0][1] = s.acc[p][1][0] = s.acc[p][1][1] = 0.0;
    }
    s.f0 = frag + frag_pos(2 * t4, g);
    s.f1 = frag + frag_pos(2 * t4 + 1, g);
    int jb = 0;
    s.template columns<KP>(jb, lb);
    // lane holds F[8 lb + g][cases 2 t4, 2 t4 + 1]
#pragma unroll
    for (int u = 0; u < 2; ++u) {
        const int c = 2 * t4 + u;
        if (c < it.nc) {
            const int i1 = cases[c].i1, i2 = cases[c].i2;
            const double f = norm * cases[c].s0;
#pragma unroll
            for (int p = 0; p < KP; ++p) {
                const int l = 8 * lb[p] + g;
                if (lb[p] >= 0 && l >= it.M && l < B) {
                    const double fs = (it.rev >> c) & (l ^ it.M) & 1 ? -f : f;
                    out[case_index(i1, i2, l)] = make_double2(fs * s.acc[p][0][u], fs * s.acc[p][1][u]);
                }
            }
        }
    }
}

// The Nyquist bins of X (row B with every column, column B with every other row; every beta),
// which no order class writes: set to zero, element i = first, first + stride, ...
__device__ __forceinline__ void nyquist_zero(double2* X, int B, long long first, long long stride)
{
    const int N = 2 * B;
    const long long total = (long long)(2 * N - 1) * N;
    for (long long i = first; i < total; i += stride) {
        const long long v = i / N;
        const int k = (int)(i - v * N);
        int row, col;
        if (v < N) {
            row = B;
            col = (int)v;
        } else {
            col = B;
            row = (int)(v - N);
            if (row >= B) ++row;   // skip (B, B), covered above
        }
        X[((size_t)row * N + col) * N + k] = make_double2(0.0, 0.0);
    }
}

constexpr int kGS = 10;   // row stride of the staged coefficients (double2): conflict-free B fragments

// An item's coefficients of the degrees 8 (M/8) .. 8 nb - 1 into s_g, asynchronously; zeros where there
// are none.
template <int NW>
__device__ __forceinline__ void load_coefficients(int B, const Item& it, const CaseInfo* cases, const double2* coeffs, double2* s_g)
{
    const int c = threadIdx.x & 7;   // a thread keeps its case: 32 NW is a multiple of 8
    const int i1 = cases[c].i1, i2 = cases[c].i2;
    const int lo = it.M & ~7, rows = ((B + 7) & ~7) - lo;
#pragma unroll 2
    for (int row = threadIdx.x >> 3; row < rows; row += 4 * NW) {
        const int l = lo + row;
        if (c < it.nc && l >= it.M && l < B) copy_async16(s_g + row * kGS + c, coeffs + case_index(i1, i2, l));
        else s_g[row * kGS + c] = make_double2(0.0, 0.0);
    }
}

// An item's sums over l. Warp w takes the tile columns w + NW p of 8 n, all of them along the blocks of
// degrees, and puts their T into the two ends of each case's column of DFT input. In block lb the
// columns up to lb are there: `count` of the warp's.
template <int NW, int KP>
struct InverseSums {
    double acc[KP][2][2];
    const double *x, *y;        // block lb's tiles of both orders at the warp's first column, the lane's element
    const double2* gb;          // block lb's coefficients, the lane's element
    bool flip;

    __device__ __forceinline__ double2 fragment(int row) const
    {
        const double2 v = gb[row * kGS];
        return flip ? make_double2(-v.x, -v.y) : v;
    }
    template <int COUNT>
    __device__ __forceinline__ void block(int lb)
    {
        double d[COUNT][2];
#pragma unroll
        for (int p = 0; p < COUNT; ++p) {
            d[p][0] = __ldg(x + 64 * NW * p) * __ldg(y + 64 * NW * p);
            d[p][1] = __ldg(x + 64 * NW * p + 32) * __ldg(y + 64 * NW * p + 32);
        }
        const double2 b0 = fragment(0), b1 = fragment(4);
#pragma unroll
        for (int p = 0; p < COUNT; ++p) {
            dmma(acc[p][0][0], acc[p][0][1], d[p][0], b0.x);
            dmma(acc[p][1][0], acc[p][1][1], d[p][0], b0.y);
        }
#pragma unroll
        for (int p = 0; p < COUNT; ++p) {
            dmma(acc[p][0][0], acc[p][0][1], d[p][1], b1.x);
            dmma(acc[p][1][0], acc[p][1][1], d[p][1], b1.y);
        }
        x += 64 * (lb + 1);
        y += 64 * (lb + 1);
        gb += 8 * kGS;
    }
    // blocks lb .. nb - 1 in runs of equal column count
    template <int COUNT>
    __device__ __forceinline__ void blocks(int& lb, int nb, int warp)
    {
        const int end = COUNT == KP ? nb : min(nb, warp + NW * COUNT);
#pragma unroll 2
        for (; lb < end; ++lb) block<COUNT>(lb);
        if constexpr (COUNT < KP) blocks<COUNT + 1>(lb, nb, warp);
    }
};

// put(n, case, T): the scaled sums of the item's cases, for n < B (all of them between two of the
// caller's barriers).
template <int NW, int KP, class Put>
__device__ __forceinline__ void inverse_sums(const double* tM, const double* tP, const double2* s_g, int B, const Item& it,
                                             const CaseInfo* cases, const Put& put)
{
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, g = lane >> 2, t4 = lane & 3;
    const int nb = (B + 7) >> 3, lbM = it.M >> 3;
    const double norm = (double)(B * 2 * B) / kPi;   // src/fn_idsoft.cpp:109
    InverseSums<NW, KP> s;
#pragma unroll
    for (int p = 0; p < KP; ++p) s.acc[p][0][0] = s.acc[p][0][1] = s.acc[p][1][0] = s.acc[p][1][1] = 0.0;
    // (-1)^(l - M) of a reversed case: l has the parity of t4, so it is the lane's own
    s.flip = (it.rev >> g) & (t4 ^ it.M) & 1;
    int lb = max(lbM, warp);
    s.x = tM + 64 * (tri(lb) + warp) + 8 * t4 + g;
    s.y = tP + 64 * (tri(lb) + warp) + 8 * t4 + g;
    s.gb = s_g + (8 * (lb - lbM) + t4) * kGS + g;
    s.template blocks<1>(lb, nb, warp);
    // lane holds T[8 (warp + NW p) + g][cases 2 t4, 2 t4 + 1]
#pragma unroll
    for (int u = 0; u < 2; ++u) {
        const int c = 2 * t4 + u;
        if (c < it.nc) {
            const double f = norm * cases[c].s0;
            const int rev = it.rev >> c;
#pragma unroll
            for (int p = 0; p < KP; ++p) {
                const int n = 8 * (warp + NW * p) + g;
                if (n >= B) break;
                const double fs = rev & (n ^ it.odd) & 1 ? -f : f;
                put(n, c, make_double2(fs * s.acc[p][0][u], fs * s.acc[p][1][u]));
            }
        }
    }
}

// The kernel's tail: the bins that no class writes, for every transform of the launch.
__device__ __forceinline__ void zero_nyquist_of(const DwtArgs& a, double2* X0, int B)
{
    if (!a.zero_nyquist) return;
    for (int t = 0; t < a.T; ++t)
        nyquist_zero(a.Xs ? a.Xs[t] : X0, B, (long long)blockIdx.x * blockDim.x + threadIdx.x, (long long)gridDim.x * blockDim.x);
}

template <class K, class In, class Out>
cudaError_t launch(K kernel, In in, Out out, int threads, size_t smem, size_t largest, const DwtArgs& a, int T, cudaStream_t s)
{
    DwtArgs b = a;
    b.T = T;
    const int items = (a.classes ? a.n_classes : num_classes(a.B)) * T;
    const cudaError_t e = allow_shared(kernel, smem, largest);
    if (e != cudaSuccess) return e;
    kernel<<<items, threads, smem, s>>>(in, out, b);
    return cudaGetLastError();
}

}  // namespace dwtk
}  // namespace pfsoft_dev
