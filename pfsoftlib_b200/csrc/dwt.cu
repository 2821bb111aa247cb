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
// The beta sums: a DFT of compile-time radices (fixed_plan, dwt_fixed.cu) where N = 98 .. 512 is a product of two or
// three of at most 20, else the MMA form (here). The DFT costs N log N per column but passes the columns
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

#include <utility>

#include "dwt_sums.cuh"

namespace pfsoft_dev {

namespace {

using namespace dwtk;

// The forward kernel with the cosine or sine sums as a matrix product on the FP64 MMA, for any N: the columns are
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

// The inverse: the matrix products of dwt_forward_mma_kernel, transposed, and the halves unfolded.
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

template <int NW, int KP, int MB>
cudaError_t launch_mma(int dir, const double2* X, double2* coeffs, const DwtArgs& a, int T, cudaStream_t s)
{
    auto bytes = [&](int nb) { return (dir == 0 ? 192 * nb : 128 * ((nb + 1) / 2) + 8 * kGS * nb) * sizeof(double2); };
    const size_t smem = bytes((a.B + 7) / 8), largest = bytes(NW * KP);   // the warps' accumulators hold NW KP tiles
    return dir == 0 ? launch(dwt_forward_mma_kernel<NW, KP, MB>, X, coeffs, 32 * NW, smem, largest, a, T, s)
                    : launch(dwt_inverse_mma_kernel<NW, KP, MB>, (const double2*)coeffs, const_cast<double2*>(X), 32 * NW, smem, largest, a, T, s);
}

// The launch of a length's compile-time DFT form, null if it has none.
template <int... P>
DwtLaunch fixed_launch_of(int N, std::integer_sequence<int, P...>)
{
    static constexpr DwtLaunch (*parts[])(int) = {DwtFixedPart<P>::launch...};
    return N < kFixedFirst || N > kFixedLast ? nullptr : parts[(N - kFixedFirst) / kFixedSpan](N);
}

DwtLaunch fixed_launch_for(int N) { return fixed_launch_of(N, std::make_integer_sequence<int, kFixedParts>()); }

cudaError_t dispatch(int dir, const double2* X, double2* coeffs, const DwtArgs& a, int T, cudaStream_t s)
{
    if (const DwtLaunch fixed = fixed_launch_for(a.N)) return fixed(dir, X, coeffs, a, T, s);
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
