// Discrete Wigner transform (DWT) over beta for every order class, FP64 (sm_100a).
//
// For the class (M, M'), M >= M' >= 0, the reference applies the Wigner rows d_{M,M'}(l, beta_k),
// l = M..B-1 (include/PFSOFTlib_headers/fn_dwt.hpp:105-200), to the up to eight beta columns that
// it serves from one matrix (src/fn_dsoft.cpp:137-283, src/fn_idsoft.cpp:127-283). Here a row is
// written as its Fourier series in beta,
//
//   d_{M,M'}(l, beta) = -kappa sqrt((2l+1)/2) sum_{n=0..l} (2 - [n=0]) P[l][n][M] P[l][n][M'] t(n beta),
//   t = cos for even M - M', sin for odd,  kappa = -1 for (M - M') mod 4 in {1, 2}, else 1,
//
// P[l][n][M] the rows at beta = pi/2 (tables.cu; Risbo 1996, Trapani & Navaza 2006). So
//
//   forward  T[n][v] = sum_k w_k t(n beta_k) S[k][v]      a length-N DFT per column (N = 2B), then
//            F[l][v] = sum_{n<=l} P[l][n][M] P[l][n][M'] T[n][v]       on the FP64 MMA
//   inverse  T[n][v] = sum_{l>=n} P[l][n][M] P[l][n][M'] G[l][v]       on the FP64 MMA, then
//            S[k][v] = sum_n t(n beta_k) T[n][v]          a length-N DFT per column
//
// with v = 2*case + (re, im), S[k][v] the beta column of the case's FFT bin, G the scaled, signed
// coefficients. A column that the reference reads at pi - beta only turns signs of T.
//
// Why the series: the rows' own recurrence in l needs three FP64 operations and a shared-memory
// store for each of the (B - M) 2B values of a class, B^4/3 over all classes, and 16 MMA
// multiply-adds for each; the series has l + 1 coefficients per degree, B^4/8 over all classes, each
// one product of two table values, and the beta sums add either a DFT or a matrix product per column.
// Against the recurrence kernels that this replaces (us per launch on B200, forward / inverse):
// B = 64 29 / 29 (31 / 46), 100 98 / 103 (131 / 138), 128 180 / 177 (263 / 265), 137 457 / 450
// (610 / 605), 200 888 / 904 (1810 / 1793), 251 3182 / 3085 (3911 / 3705), 256 1879 / 1932
// (4092 / 3903); the error against 64 bits falls four- to twelvefold (B = 256 DSOFT 1.4e-14 to 1.1e-15).
//
// What bounds it at B = 128: the shared-memory pipe (65 % of its cycles) and latency at 16 warps per
// SM; the MMA takes 34 of the 180 us, the other FP64 work 30.
//
// The beta sums: a DFT of compile-time radices (fixed_plan) where N = 98 .. 512 is a product of two or
// three of at most 20, else the MMA form. The DFT costs N log N per column but passes the columns
// through shared memory once per stage between barriers; the matrix product costs B^2 per column and has
// one barrier. Measured, MMA form against DFT, us forward / inverse: N = 96 17 / 18 against 19 / 19,
// 98 25 / 26 against 20 / 22, 128 33 / 33 against 29 / 29, 168 70 / 77 against 60 / 64, 224 168 / 168
// against 126 / 123, 272 428 / 434 against 309 / 300, 360 956 / 1007 against 699 / 664, 480 2699 / 2658
// against 1602 / 1628; the radices 17 and 19 at N = 114 and 152 break even, 23 spills. The register caps cost some
// kernels a little too: 8 to 80 bytes of spills in the forward sums at four tile columns per warp (60 at N = 256, 64 at
// 512, 80 in the MMA form up to B = 256). Two large
// radices beat three small ones (N = 240 16.15 152 / 152 against 16.3.5 160 / 168).
//
// One CTA per item, a class of one transform; longest classes first.

#include <algorithm>

#include "common.cuh"
#include "dwt.cuh"
#include "dwt_common.cuh"
#include "fft_core.cuh"

namespace pfsoft_dev {

namespace {

using namespace dwtk;
using namespace fftk;

// ---- the beta DFT of a class's columns -------------------------------------------------------
// The columns lie in shared memory with an odd pitch, and consecutive threads take consecutive
// columns: then every access of eight columns meets eight distinct 16-byte banks whatever the
// element, and the eight share each twiddle. HBM is read and written in contiguous rows, the
// reordering of the samples happens on the shared-memory side.

struct CaseInfo {
    long long col;   // the case's beta column in X (double2 elements)
    int i1, i2;      // its place in degree l's block: i2 (2l+1) + i1, plus (2l+1) to each that is negative
    double s0;       // sign with the series' own sign
};

__host__ __device__ __forceinline__ int col_pitch(int N) { return N | 1; }

// Element e of a column's DFT is the sample k: even samples ascending, then odd ones descending, so
// that the length-N DFT gives the cosine sums (Makhoul 1980).
__device__ __forceinline__ int sample_of(int e, int B, int N) { return e < B ? 2 * e : 2 * (N - 1 - e) + 1; }

__device__ __forceinline__ void copy_async16(double2* dst, const double2* src)
{
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((unsigned)__cvta_generic_to_shared(dst)), "l"(src)
                 : "memory");
}
__device__ __forceinline__ void copy_async_wait() { asm volatile("cp.async.wait_all;" ::: "memory"); }

// An item's columns into dst, asynchronously.
template <int N, int NT>
__device__ __forceinline__ void load_columns(const double2* X, const CaseInfo* cases, int count, double2* dst)
{
#pragma unroll 4
    for (int c = 0; c < count; ++c) {
        const double2* src = X + cases[c].col;
#pragma unroll
        for (int k = threadIdx.x; k < N; k += NT) copy_async16(dst + c * col_pitch(N) + k, src + k);
    }
}

// The same columns from shared memory to X.
template <int N, int NT>
__device__ __forceinline__ void store_columns(double2* X, const CaseInfo* cases, int count, const double2* src)
{
#pragma unroll 4
    for (int c = 0; c < count; ++c) {
        double2* dst = X + cases[c].col;
#pragma unroll
        for (int k = threadIdx.x; k < N; k += NT) dst[k] = src[c * col_pitch(N) + k];
    }
}

// One Stockham stage (fft.cu) of up to eight columns of a compile-time length, P butterflies per
// thread held in registers between the loads and the stores, so that a stage can work in place.
template <int SIGN, int R, int NS, int N, int NT, class Ld, class St>
__device__ __forceinline__ void fixed_stage(const double2* __restrict__ tw, int nv, const Ld& ld, const St& st)
{
    constexpr int m = N / R, step = N / (NS * R), P = (8 * m + NT - 1) / NT;
    const int lg = nv == 8 ? 3 : (nv == 4 ? 2 : 0);
    // threads past the last butterfly repeat it and store nothing (guarded loads would put v in local memory)
    double2 v[P][R];
#pragma unroll
    for (int p = 0; p < P; ++p) {
        const int t = threadIdx.x + p * NT, kk = t & (nv - 1), j = min(t >> lg, m - 1);
#pragma unroll
        for (int r = 0; r < R; ++r) v[p][r] = ld(kk, j, r);
    }
    __syncthreads();
#pragma unroll
    for (int p = 0; p < P; ++p) {
        const int t = threadIdx.x + p * NT, kk = t & (nv - 1), j = min(t >> lg, m - 1);
        const int k = j % NS;
        if (NS > 1) {
#pragma unroll
            for (int r = 1; r < R; ++r) v[p][r] = cmul(v[p][r], twiddle(tw, r * k * step, SIGN));
        }
        butterfly<SIGN, R>(v[p]);
        const int ob = (j / NS) * NS * R + k;
        if ((t >> lg) < m) {
#pragma unroll
            for (int q = 0; q < R; ++q) st(kk, ob + q * NS, v[p][q]);
        }
    }
}

// A length known at compile time, two or three radices (R2 = 1: two), in place.
template <int N_, int NW_, int R0, int R1, int R2>
struct FixedFft {
    static constexpr int N = N_, NW = NW_, NT = 32 * NW_, PL = N_ | 1, B = N_ / 2;
    static constexpr int kMinBlocks = NW_ == 8 ? 2 : (N_ <= 128 ? 5 : 4);
    static_assert(R0 * R1 * R2 == N_, "radices");
    static constexpr int kElems = 8 * PL;
    static __device__ __forceinline__ void forward(const double2* tw, const double* w, int nv, int odd, double2* smem)
    {
        // element j + r m of the first stage: the first half of the r are even samples
        auto in = [&](int kk, int j, int r) {
            constexpr int m = N_ / R0;
            const int k = r < R0 / 2 ? 2 * j + 2 * m * r : (2 * N_ - 1 - 2 * m * r) - 2 * j;
            const double f = __ldg(w + k);
            return cscale(smem[kk * PL + k], odd && r >= R0 / 2 ? -f : f);
        };
        auto ld1 = [&](int kk, int j, int r) { return smem[kk * PL + j + r * (N_ / R1)]; };
        auto ld2 = [&](int kk, int j, int r) { return smem[kk * PL + j + r * (N_ / R2)]; };
        auto st = [&](int kk, int e, double2 x) { smem[kk * PL + e] = x; };
        fixed_stage<-1, R0, 1, N_, NT>(tw, nv, in, st);
        __syncthreads();
        fixed_stage<-1, R1, R0, N_, NT>(tw, nv, ld1, st);
        if (R2 > 1) {
            __syncthreads();
            fixed_stage<-1, R2, R0 * R1, N_, NT>(tw, nv, ld2, st);
        }
        __syncthreads();
    }
    static __device__ __forceinline__ void inverse(const double2* tw, int nv, int odd, double2* X, const CaseInfo* cases, double2* smem)
    {
        auto ld0 = [&](int kk, int j, int r) { return smem[kk * PL + j + r * (N_ / R0)]; };
        auto ld1 = [&](int kk, int j, int r) { return smem[kk * PL + j + r * (N_ / R1)]; };
        auto ld2 = [&](int kk, int j, int r) { return smem[kk * PL + j + r * (N_ / R2)]; };
        auto st = [&](int kk, int e, double2 x) { smem[kk * PL + e] = x; };
        auto out = [&](int kk, int e, double2 x) {
            smem[kk * PL + sample_of(e, B, N_)] = odd && e >= B ? make_double2(-x.x, -x.y) : x;
        };
        fixed_stage<+1, R0, 1, N_, NT>(tw, nv, ld0, st);
        __syncthreads();
        if (R2 > 1) {
            fixed_stage<+1, R1, R0, N_, NT>(tw, nv, ld1, st);
            __syncthreads();
            fixed_stage<+1, R2, R0 * R1, N_, NT>(tw, nv, ld2, out);
        } else {
            fixed_stage<+1, R1, R0, N_, NT>(tw, nv, ld1, out);
        }
        __syncthreads();
        store_columns<N_, NT>(X, cases, nv, smem);
    }
};

// ---- the kernels -------------------------------------------------------------------------------

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

// B fragments of an item from its columns' DFTs: the cosine (odd: sine) sums T[n][case], zeros up to the
// last tile's end.
template <int N, int NT>
__device__ __forceinline__ void fill_fragments(const double2* ht, int nc, int odd, int rev, const double2* v, double2* frag)
{
    constexpr int B = N >> 1, nb = (B + 7) >> 3, pl = N | 1;
    for (int n = threadIdx.x; n < 8 * nb; n += NT) {
        double ca = 0.0, cb = 0.0;
        if (n < B) {
            const double2 cs = __ldg(ht + n);
            ca = odd ? cs.y : cs.x;
            cb = odd ? -cs.x : cs.y;
            if (n == 0) {
                ca = odd ? 0.0 : 0.5;
                cb = 0.0;
            }
        }
        const int n1 = n < B ? n : 0, n2 = n1 ? N - n1 : 0;
#pragma unroll
        for (int c = 0; c < 8; ++c) {
            if (c >= nc) break;
            const double2 p = v[c * pl + n1], q = v[c * pl + n2];
            const bool turn = (rev >> c) & (n ^ odd) & 1;
            const double fa = turn ? -ca : ca, fb = turn ? -cb : cb;
            frag[frag_pos(n, c)] = n < B ? make_double2(fa * (p.x + q.x) + fb * (p.y - q.y), fa * (p.y + q.y) - fb * (p.x - q.x))
                                         : make_double2(0.0, 0.0);
        }
    }
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

template <class F, int KP>
__global__ void __launch_bounds__(32 * F::NW, F::kMinBlocks)
    dwt_forward_fft_kernel(const double2* X0, double2* out0, const __grid_constant__ DwtArgs a)
{
    constexpr int NT = 32 * F::NW, N = F::N;
    extern __shared__ double2 smem[];
    __shared__ CaseInfo s_cases[8];
    __shared__ Item s_item;
    double2* frag = smem + F::kElems;
    fill_item(a, blockIdx.x, N, &s_item, s_cases);
    __syncthreads();
    const Item it = s_item;
    load_columns<N, NT>(a.Xs ? a.Xs[it.tr] : X0, s_cases, it.nc, smem);
    copy_async_wait();
    __syncthreads();
    F::forward(a.tw, a.w, it.nc, it.odd, smem);
    fill_fragments<N, NT>(a.ht, it.nc, it.odd, it.rev, smem, frag);
    __syncthreads();
    forward_sums<F::NW, KP>(a.delta + it.offM, a.delta + it.offP, frag, N / 2, it, s_cases, a.Xs ? a.coefs[it.tr] : out0);
}

// The same with the cosine or sine sums as a matrix product on the FP64 MMA, for any N: the columns are
// folded at beta = pi/2 (even n need the sum of the halves, odd n the difference, for sines the other
// way round), then T[2m + q] = sum_{k<B} C[m][k] S_q[k] with the table's tiles of t((2m+q) beta_k).
template <int NW, int KP, int MB>
__global__ void __launch_bounds__(32 * NW, MB)
    dwt_forward_mma_kernel(const double2* X0, double2* out0, const __grid_constant__ DwtArgs a)
{
    extern __shared__ double2 smem[];
    __shared__ CaseInfo s_cases[8];
    __shared__ Item s_item;
    const int N = a.N, B = N >> 1, nb = (B + 7) >> 3;
    double2* fold = smem;               // [2][nb] fragment tiles of k
    double2* frag = smem + 128 * nb;    // [nb] fragment tiles of n
    fill_item(a, blockIdx.x, N, &s_item, s_cases);
    __syncthreads();
    const Item it = s_item;
    const double2* X = a.Xs ? a.Xs[it.tr] : X0;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, g = lane >> 2, t4 = lane & 3;
    for (int k = threadIdx.x; k < 8 * nb; k += 32 * NW) {
        const bool in = k < B;
        const double w = in ? __ldg(a.w + k) : 0.0;
        double2 p[8], q[8];
#pragma unroll
        for (int c = 0; c < 8; ++c) {
            p[c] = q[c] = make_double2(0.0, 0.0);
            if (c < it.nc && in) {
                const double2* col = X + s_cases[c].col;
                p[c] = __ldg(col + k);
                q[c] = __ldg(col + (N - 1 - k));
            }
        }
#pragma unroll
        for (int c = 0; c < 8; ++c) {
            if (c < it.nc) {
                const double2 sum = cscale(cadd(p[c], q[c]), w), diff = cscale(csub(p[c], q[c]), w);
                const int o = frag_pos(k, c);
                fold[o] = it.odd ? diff : sum;
                fold[64 * nb + o] = it.odd ? sum : diff;
            }
        }
    }
    __syncthreads();
    {
        // warp w: n of parity w & 1, tiles of m = n / 2 from w / 2 in steps of NW / 2
        const int q = warp & 1, mb = (nb + 1) >> 1;
        const double2* f0 = fold + 64 * nb * q + frag_pos(2 * t4, g);
        const double2* f1 = fold + 64 * nb * q + frag_pos(2 * t4 + 1, g);
        const double2* tg = reinterpret_cast<const double2*>(a.trig) + (size_t)32 * ((2 * it.odd + q) * mb + (warp >> 1)) * nb + lane;
        double acc[KP][2][2];
#pragma unroll
        for (int p = 0; p < KP; ++p) acc[p][0][0] = acc[p][0][1] = acc[p][1][0] = acc[p][1][1] = 0.0;
#pragma unroll 2
        for (int kt = 0; kt < nb; ++kt) {
            double2 d[KP];
#pragma unroll
            for (int p = 0; p < KP; ++p)
                d[p] = (warp >> 1) + p * (NW / 2) < mb ? __ldg(tg + 32 * (NW / 2) * p * nb) : make_double2(0.0, 0.0);
            const double2 t0 = f0[64 * kt], t1 = f1[64 * kt];
            tg += 32;
#pragma unroll
            for (int p = 0; p < KP; ++p) {
                dmma(acc[p][0][0], acc[p][0][1], d[p].x, t0.x);
                dmma(acc[p][1][0], acc[p][1][1], d[p].x, t0.y);
            }
#pragma unroll
            for (int p = 0; p < KP; ++p) {
                dmma(acc[p][0][0], acc[p][0][1], d[p].y, t1.x);
                dmma(acc[p][1][0], acc[p][1][1], d[p].y, t1.y);
            }
        }
        // lane holds T[2 m + q][cases 2 t4, 2 t4 + 1]
#pragma unroll
        for (int p = 0; p < KP; ++p) {
            const int n = 2 * (8 * ((warp >> 1) + p * (NW / 2)) + g) + q;
            if (n < 8 * nb) {
#pragma unroll
                for (int u = 0; u < 2; ++u) {
                    const int c = 2 * t4 + u;
                    const double sg = (it.rev >> c) & (n ^ it.odd) & 1 ? -1.0 : 1.0;
                    frag[frag_pos(n, c)] = make_double2(sg * acc[p][0][u], sg * acc[p][1][u]);
                }
            }
        }
    }
    __syncthreads();
    forward_sums<NW, KP>(a.delta + it.offM, a.delta + it.offP, frag, B, it, s_cases, a.Xs ? a.coefs[it.tr] : out0);
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

template <class F, int KP>
__global__ void __launch_bounds__(32 * F::NW, F::kMinBlocks)
    dwt_inverse_fft_kernel(const double2* coeffs0, double2* X0, const __grid_constant__ DwtArgs a)
{
    constexpr int N = F::N, B = N / 2, PL = F::PL;
    extern __shared__ double2 smem[];
    __shared__ CaseInfo s_cases[8];
    __shared__ Item s_item;
    double2* s_g = smem + F::kElems;
    fill_item(a, blockIdx.x, N, &s_item, s_cases);
    __syncthreads();
    const Item it = s_item;
    load_coefficients<F::NW>(B, it, s_cases, a.Xs ? a.coefs[it.tr] : coeffs0, s_g);
    copy_async_wait();
    __syncthreads();
    // T into the two ends of each column's DFT input
    inverse_sums<F::NW, KP>(a.delta + it.offM, a.delta + it.offP, s_g, B, it, s_cases, [&](int n, int c, double2 t) {
        const double2 cs = __ldg(a.ht + n);
        const double ca = it.odd ? cs.y : cs.x, cb = it.odd ? -cs.x : cs.y;
        double2* v = smem + c * PL;
        if (n == 0) {
            v[0] = it.odd ? make_double2(0.0, 0.0) : t;
            v[B] = make_double2(0.0, 0.0);
        } else {
            v[n] = make_double2(ca * t.x - cb * t.y, ca * t.y + cb * t.x);
            v[N - n] = make_double2(ca * t.x + cb * t.y, ca * t.y - cb * t.x);
        }
    });
    __syncthreads();
    F::inverse(a.tw, it.nc, it.odd, a.Xs ? a.Xs[it.tr] : X0, s_cases, smem);
    zero_nyquist_of(a, X0, B);
}

// The same for any N: the matrix products of dwt_forward_mma_kernel, transposed, and the halves unfolded.
template <int NW, int KP, int MB>
__global__ void __launch_bounds__(32 * NW, MB)
    dwt_inverse_mma_kernel(const double2* coeffs0, double2* X0, const __grid_constant__ DwtArgs a)
{
    extern __shared__ double2 smem[];
    __shared__ CaseInfo s_cases[8];
    __shared__ Item s_item;
    const int N = a.N, B = N >> 1, nb = (B + 7) >> 3, mb = (nb + 1) >> 1;
    double2* frag = smem;               // [2][mb] fragment tiles of m, n = 2 m + parity
    double2* s_g = smem + 128 * mb;
    fill_item(a, blockIdx.x, N, &s_item, s_cases);
    __syncthreads();
    const Item it = s_item;
    load_coefficients<NW>(B, it, s_cases, a.Xs ? a.coefs[it.tr] : coeffs0, s_g);
    for (int e = threadIdx.x; e < 8 * (16 * mb - B); e += 32 * NW) {   // n past the last
        const int n = B + (e >> 3), c = e & 7;
        frag[64 * mb * (n & 1) + frag_pos(n >> 1, c)] = make_double2(0.0, 0.0);
    }
    copy_async_wait();
    __syncthreads();
    inverse_sums<NW, KP>(a.delta + it.offM, a.delta + it.offP, s_g, B, it, s_cases,
                         [&](int n, int c, double2 t) { frag[64 * mb * (n & 1) + frag_pos(n >> 1, c)] = t; });
    __syncthreads();
    {
        // warp w: tiles of k from w in steps of NW, both parities
        const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, g = lane >> 2, t4 = lane & 3;
        // fragment k-steps: lane needs m = 4 s + t4 of a tile, case g
        const double2* f0 = frag + frag_pos(t4, g);
        const double2* f1 = frag + frag_pos(4 + t4, g);
        double2* X = a.Xs ? a.Xs[it.tr] : X0;
        double acc[KP][2][2][2];   // [tile][parity][re, im][case 2 t4 + u]
#pragma unroll
        for (int p = 0; p < KP; ++p)
#pragma unroll
            for (int i = 0; i < 8; ++i) acc[p][i >> 2][(i >> 1) & 1][i & 1] = 0.0;
#pragma unroll
        for (int q = 0; q < 2; ++q) {
            const double* tg = a.trig + (size_t)64 * ((2 * it.odd + q) * mb * nb + warp) + 8 * t4 + g;
#pragma unroll 2
            for (int mt = 0; mt < mb; ++mt) {
                double d[KP][2];
#pragma unroll
                for (int p = 0; p < KP; ++p) {
                    const bool in = warp + NW * p < nb;
                    d[p][0] = in ? __ldg(tg + 64 * NW * p) : 0.0;
                    d[p][1] = in ? __ldg(tg + 64 * NW * p + 32) : 0.0;
                }
                tg += 64 * nb;
                const double2 t0 = f0[64 * (mb * q + mt)], t1 = f1[64 * (mb * q + mt)];
#pragma unroll
                for (int p = 0; p < KP; ++p) {
                    dmma(acc[p][q][0][0], acc[p][q][0][1], d[p][0], t0.x);
                    dmma(acc[p][q][1][0], acc[p][q][1][1], d[p][0], t0.y);
                }
#pragma unroll
                for (int p = 0; p < KP; ++p) {
                    dmma(acc[p][q][0][0], acc[p][q][0][1], d[p][1], t1.x);
                    dmma(acc[p][q][1][0], acc[p][q][1][1], d[p][1], t1.y);
                }
            }
        }
#pragma unroll
        for (int u = 0; u < 2; ++u) {
            const int c = 2 * t4 + u;
            if (c < it.nc) {
                double2* col = X + s_cases[c].col;
#pragma unroll
                for (int p = 0; p < KP; ++p) {
                    const int k = 8 * (warp + NW * p) + g;
                    if (k < B) {
                        const double2 ev = make_double2(acc[p][0][0][u], acc[p][0][1][u]), od = make_double2(acc[p][1][0][u], acc[p][1][1][u]);
                        col[k] = cadd(ev, od);
                        col[N - 1 - k] = it.odd ? csub(od, ev) : csub(ev, od);
                    }
                }
            }
        }
    }
    zero_nyquist_of(a, X0, B);
}

__global__ void zero_nyquist_kernel(double2* X, int B)
{
    nyquist_zero(X, B, blockIdx.x * (long long)blockDim.x + threadIdx.x, (long long)gridDim.x * blockDim.x);
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

template <class F, int KP>
cudaError_t launch_fft(int dir, const double2* X, double2* coeffs, const DwtArgs& a, int T, cudaStream_t s)
{
    // the columns' DFT, and behind it the forward's B fragments or the inverse's coefficients
    const size_t smem = (F::kElems + ((F::B + 7) / 8) * (dir == 0 ? 64 : 8 * kGS)) * sizeof(double2);
    return dir == 0 ? launch(dwt_forward_fft_kernel<F, KP>, X, coeffs, F::NT, smem, smem, a, T, s)
                    : launch(dwt_inverse_fft_kernel<F, KP>, (const double2*)coeffs, const_cast<double2*>(X), F::NT, smem, smem, a, T, s);
}

template <int NW, int KP, int MB>
cudaError_t launch_mma(int dir, const double2* X, double2* coeffs, const DwtArgs& a, int T, cudaStream_t s)
{
    auto bytes = [&](int nb) { return (dir == 0 ? 192 * nb : 128 * ((nb + 1) / 2) + 8 * kGS * nb) * sizeof(double2); };
    const size_t smem = bytes((a.B + 7) / 8), largest = bytes(NW * KP);   // the warps' accumulators hold NW KP tiles
    return dir == 0 ? launch(dwt_forward_mma_kernel<NW, KP, MB>, X, coeffs, 32 * NW, smem, largest, a, T, s)
                    : launch(dwt_inverse_mma_kernel<NW, KP, MB>, (const double2*)coeffs, const_cast<double2*>(X), 32 * NW, smem, largest, a, T, s);
}

// The radices of a DFT length N: of the products of two or three of at most 20, the first even, the one
// whose stages hold the fewest points in the block's registers, a stage's last butterflies rounded up to
// a whole one per thread, and a stage's two barriers counted as 4 points; r0 = 0 if there is none that
// fits the registers (24 points).
struct FixedPlan {
    int r0, r1, r2;
};

constexpr FixedPlan fixed_plan(int N, int NT)
{
    FixedPlan best = {0, 0, 0};
    int least = 0, widest = 0;
    for (int r0 = 20; r0 >= 2; r0 -= 2)
        for (int r1 = 20; r1 >= 2; --r1) {
            if (N % (r0 * r1) || N / (r0 * r1) > 20) continue;
            const int r[3] = {r0, r1, N / (r0 * r1)};
            int sum = 0, wide = 0;
            bool fits = true;
            for (int i = 0; i < 3; ++i) {
                const int points = r[i] > 1 ? (8 * (N / r[i]) + NT - 1) / NT * r[i] : 0;
                sum += points + (points ? 4 : 0);
                fits = fits && points <= 24;
                wide = r[i] > wide ? r[i] : wide;
            }
            if (fits && (best.r0 == 0 || sum < least || (sum == least && wide < widest))) {
                best = {r[0], r[1], r[2]};
                least = sum;
                widest = wide;
            }
        }
    return best;
}

typedef cudaError_t (*LaunchFn)(int, const double2*, double2*, const DwtArgs&, int, cudaStream_t);

template <int N>
constexpr LaunchFn fixed_launch()
{
    constexpr int NW = N <= 256 ? 4 : 8;
    constexpr FixedPlan p = fixed_plan(N, 32 * NW);
    if constexpr (p.r0 > 0) return launch_fft<FixedFft<N, NW, p.r0, p.r1, p.r2>, ((N + 15) / 16 + NW - 1) / NW>;
    else return nullptr;
}

constexpr int kFixedFirst = 98, kFixedLast = 512;

template <int... I>
LaunchFn fixed_launch_of(int N, std::integer_sequence<int, I...>)
{
    static constexpr LaunchFn table[] = {fixed_launch<kFixedFirst + 2 * I>()...};
    return N < kFixedFirst || N > kFixedLast ? nullptr : table[(N - kFixedFirst) / 2];
}

LaunchFn fixed_launch_for(int N)
{
    return fixed_launch_of(N, std::make_integer_sequence<int, (kFixedLast - kFixedFirst) / 2 + 1>());
}

cudaError_t dispatch(int dir, const double2* X, double2* coeffs, const DwtArgs& a, int T, cudaStream_t s)
{
    if (const LaunchFn fixed = fixed_launch_for(a.N)) return fixed(dir, X, coeffs, a, T, s);
    // The MMA form: warps, tile columns per warp (NW KP blocks of 8 in all: the bandwidth's), CTAs per SM. Few
    // warps keep short classes' warps busy, eight hide more where the CTA's shared memory allows two only. Measured, us
    // forward / inverse, this against the best other: B = 16 8.5 / 8.6 (all shapes), 32 10.6 / 10.6 (4 warps the same), 33
    // 11.3 / 12.6 (2 warps of 3, 12.6 / 12.6), 40 15.4 / 17.0 (the same, 12.7 / 12.8), 48 16.7 / 16.8 (the same, 14.7 / 16.7), 64
    // 31 / 31 (4 of 2, 29 / 33), 67 41 / 44 (six CTAs, 39 / 41), 96 93 / 97 (six, 100 / 97), 127 260 / 233 (8 of 2, 242 / 249), 137
    // 453 / 443 (three CTAs, 387 / 397), 191 1113 / 1127 (three, 1080 / 1058), 193 1457 / 1437 (three, 1477 / 1455), 251
    // 3183 / 3086 (three, 3327 / 3166). So the lines at 40 and 192 are not the best there are.
    if (a.B <= 16) return launch_mma<2, 1, 12>(dir, X, coeffs, a, T, s);
    if (a.B <= 32) return launch_mma<2, 2, 12>(dir, X, coeffs, a, T, s);
    if (a.B <= 40) return launch_mma<4, 2, 5>(dir, X, coeffs, a, T, s);
    if (a.B <= 64) return launch_mma<2, 4, 8>(dir, X, coeffs, a, T, s);
    if (a.B <= 96) return launch_mma<4, 3, 5>(dir, X, coeffs, a, T, s);
    if (a.B <= 128) return launch_mma<4, 4, 5>(dir, X, coeffs, a, T, s);
    if (a.B <= 192) return launch_mma<8, 3, 2>(dir, X, coeffs, a, T, s);
    if (a.B <= 256) return launch_mma<8, 4, 2>(dir, X, coeffs, a, T, s);
    if (a.B <= 512) return launch_mma<8, 8, 1>(dir, X, coeffs, a, T, s);
    return cudaErrorInvalidValue;
}

}  // namespace

DwtArgs dwt_args_for(const BandTables& t)
{
    DwtArgs a = {};
    a.B = t.B;
    a.N = t.N;
    a.w = t.w;
    a.ht = t.ht;
    a.tw = t.twiddle;
    a.delta = t.delta;
    a.trig = t.trig;
    return a;
}

bool dwt_has_dft(int N) { return fixed_launch_for(N) != nullptr; }

cudaError_t dwt_forward_launch(const double2* X, double2* coeffs, const DwtArgs& a, int T, cudaStream_t s)
{
    return dispatch(0, X, coeffs, a, T, s);
}

cudaError_t dwt_inverse_launch(const double2* coeffs, double2* X, const DwtArgs& a, int T, cudaStream_t s)
{
    return dispatch(1, X, const_cast<double2*>(coeffs), a, T, s);
}

cudaError_t zero_nyquist_launch(double2* X, int B, cudaStream_t s)
{
    const int N = 2 * B;
    const long long total = (long long)(2 * N - 1) * N;
    int blocks = (int)((total + 255) / 256);
    if (blocks > 4096) blocks = 4096;
    zero_nyquist_kernel<<<blocks, 256, 0, s>>>(X, B);
    return cudaGetLastError();
}

}  // namespace pfsoft_dev
