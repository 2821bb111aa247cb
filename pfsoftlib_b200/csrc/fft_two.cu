// DFT passes of lengths n = ra rb with ra, rb <= 32, each factor one register butterfly: one exchange
// through shared memory between the load from HBM and the store to HBM (sm_100a).
//
// Stage 1 takes butterfly j < rb of a vector, inputs x[j + r rb], r < ra, and leaves its outputs as row j
// (pitch ra | 1) of the vector's block in shared memory. Stage 2 takes column j < ra, inputs
// row r times w_n^(r j), and stores outputs j + q ra. With two stages no index needs a division, the
// twiddles of a stage-2 load lie side by side (a.twiddle + n, fft_two_twiddle), and the rows' and
// vectors' odd pitches keep both thread maps (along the vector, or across the tile's vectors: the side
// that is contiguous in HBM) clear of bank conflicts.
//
// What bounds it: HBM. Against the ping-pong and in-place kernels of three or four stages that ran these
// lengths before, us per pass (of the 32 N^3 bytes at the measured copy rate): N = 112 17 against
// 31 .. 62, 200 66 against 108 (0.60), 256 89 against 98 (0.93), 320 199 against about 290 (0.82), 384 345
// against 553 (0.82), 400 390 against 760 (0.81), 512 853 against 1210 (0.78). The primes 17 .. 31 cost R
// multiply-adds per point, under the 90 that fit the HBM time; against the chirp pass, us per pass: N =
// 136 32 / 64, 184 81 / 145, 248 179 / 292, 272 131 / 449, 304 183 / 571, 408 426 / 1480, 496 970 / 2274.
//
// Tiles of 8 vectors move 128-byte runs on the transposed side; at radices 18 .. 26 four vectors and four
// CTAs per SM measured faster (N = 320 199 us against 230), from 28 on eight (N = 512 885 against 1000).

#include <algorithm>

#include "common.cuh"
#include "fft.cuh"
#include "fft_core.cuh"
#include "fft_two.cuh"

namespace pfsoft_dev {

namespace {

using namespace fftk;

// ---- both passes of small planes ------------------------------------------------------------------
// One CTA transforms a whole beta layer, N x N points in shared memory: four stages in place between
// three barriers, with the butterflies, twiddles and order of the two passes, so with their results bit
// for bit. A stage leaves output q of butterfly j in the slot it read input q from; the order that
// leaves (slot j rb + q holds element j + q ra) is undone in the next addresses. Rows (index c) have an
// odd pitch and runs of rb slots the pitch rb | 1: threads across c, across the slots, or across the j of
// the contiguous side meet distinct 16-byte banks.
//
// What bounds it: the latency of the four stages; the strided side moves single 16-byte values, which
// costs twice the sectors but stays in L2 at these sizes. One launch and one round trip through L2 less:
// a whole transform, us, two passes against this: N = 8 6.7 / 5.5 in a graph, 16 7.5 / 6.0, 32 9.2 / 7.7 (called
// from Python 15.5 / 13.0), 40 10.8 / 10.0, 48 10.9 / 11.0 (16.4 / 14.4), 56 11.8 / 13.0. Where several
// transforms fill the SMs the passes' better sectors win from N = 40 on (T = 4 19.2 / 19.4, 16 37 / 41).

struct Plane {
    int n, ra, rb, pr, pl;   // pr: pitch of a run of rb slots, pl: of a row
    unsigned inv_n, inv_ra, inv_rb;
    __host__ __device__ Plane(int n_, int ra_, int rb_) : n(n_), ra(ra_), rb(rb_), pr(rb_ | 1), pl((ra_ * (rb_ | 1)) | 1)
    {
        inv_n = 0xffffffffu / (unsigned)n + 1u;
        inv_ra = 0xffffffffu / (unsigned)ra + 1u;
        inv_rb = 0xffffffffu / (unsigned)rb + 1u;
    }
    __device__ int div_rb(int x) const { return (int)__umulhi((unsigned)x, inv_rb); }
    __device__ int slot(int s) const { return s + div_rb(s) * (pr - rb); }
    __device__ int element(int s) const { return div_rb(s) + (s - div_rb(s) * rb) * ra; }   // in slot s
};

// Butterflies of one stage over the plane's n vectors: consecutive threads take consecutive vectors, or
// (along) the consecutive butterflies of a vector.
template <int SIGN, int R, class Ld, class St>
__device__ __forceinline__ void plane_stage(int n, int m, unsigned inv, bool along, const double2* tw, const Ld& ld, const St& st)
{
    for (int t = threadIdx.x; t < n * m; t += blockDim.x) {
        const int hi = (int)__umulhi((unsigned)t, inv), lo = t - hi * (along ? m : n);
        const int v = along ? hi : lo, j = along ? lo : hi;
        double2 x[R];
#pragma unroll
        for (int r = 0; r < R; ++r) {
            x[r] = ld(v, j, r);
            if (tw && r > 0) {
                double2 w = __ldg(tw + (r - 1) * m + j);
                if (SIGN > 0) w.y = -w.y;
                x[r] = cmul(x[r], w);
            }
        }
        butterfly<SIGN, R>(x);
#pragma unroll
        for (int q = 0; q < R; ++q) st(v, j, q, x[q]);
    }
}

template <int SIGN>
__global__ void __launch_bounds__(512, 1)
    fft_plane_kernel(const double2* src, double2* dst, const __grid_constant__ FftPlaneArgs a)
{
    extern __shared__ double2 smem[];
    if (a.srcs) {
        src = a.srcs[blockIdx.z];
        dst = a.dsts[blockIdx.z];
    }
    const Plane p(a.n, a.ra, a.rb);
    const int n = a.n, k = blockIdx.x;
    const double2* tw = a.twiddle + n;
    if (SIGN < 0) {
        // over r, then over c: G[k][c][r] to X[r][c][k]
        src += (long long)k * n * n;
        dst += k;
        with_radix<0, 2>(p.ra, [&](auto R) {
            plane_stage<SIGN, decltype(R)::value>(n, p.rb, p.inv_rb, true, nullptr,
                [&](int c, int j, int r) { return __ldg(src + c * n + j + r * p.rb); },
                [&](int c, int j, int q, double2 x) { smem[c * p.pl + q * p.pr + j] = x; });
        });
        __syncthreads();
        with_radix<0, 2>(p.rb, [&](auto R) {
            plane_stage<SIGN, decltype(R)::value>(n, p.ra, p.inv_n, false, tw,
                [&](int c, int j, int r) { return smem[c * p.pl + j * p.pr + r]; },
                [&](int c, int j, int q, double2 x) { smem[c * p.pl + j * p.pr + q] = x; });
        });
        __syncthreads();
        with_radix<0, 2>(p.ra, [&](auto R) {
            plane_stage<SIGN, decltype(R)::value>(n, p.rb, p.inv_n, false, nullptr,
                [&](int s, int j, int r) { return smem[(j + r * p.rb) * p.pl + p.slot(s)]; },
                [&](int s, int j, int q, double2 x) { smem[(j + q * p.rb) * p.pl + p.slot(s)] = x; });
        });
        __syncthreads();
        with_radix<0, 2>(p.rb, [&](auto R) {
            plane_stage<SIGN, decltype(R)::value>(n, p.ra, p.inv_n, false, tw,
                [&](int s, int j, int r) { return smem[(j * p.rb + r) * p.pl + p.slot(s)]; },
                [&](int s, int j, int q, double2 x) { dst[(long long)(p.element(s) * n + j + q * p.ra) * n] = x; });
        });
    } else {
        // over c, then over r: X[r][c][k] to G[k][c][r]
        src += k;
        dst += (long long)k * n * n;
        with_radix<0, 2>(p.ra, [&](auto R) {
            plane_stage<SIGN, decltype(R)::value>(n, p.rb, p.inv_n, false, nullptr,
                [&](int v, int j, int r) { return __ldg(src + (long long)(v * n + j + r * p.rb) * n); },
                [&](int v, int j, int q, double2 x) { smem[(j + q * p.rb) * p.pl + p.slot(v)] = x; });
        });
        __syncthreads();
        with_radix<0, 2>(p.rb, [&](auto R) {
            plane_stage<SIGN, decltype(R)::value>(n, p.ra, p.inv_n, false, tw,
                [&](int v, int j, int r) { return smem[(j * p.rb + r) * p.pl + p.slot(v)]; },
                [&](int v, int j, int q, double2 x) { smem[(j * p.rb + q) * p.pl + p.slot(v)] = x; });
        });
        __syncthreads();
        with_radix<0, 2>(p.ra, [&](auto R) {
            plane_stage<SIGN, decltype(R)::value>(n, p.rb, p.inv_n, false, nullptr,
                [&](int s, int j, int r) { return smem[s * p.pl + r * p.pr + j]; },
                [&](int s, int j, int q, double2 x) { smem[s * p.pl + q * p.pr + j] = x; });
        });
        __syncthreads();
        with_radix<0, 2>(p.rb, [&](auto R) {
            plane_stage<SIGN, decltype(R)::value>(n, p.ra, p.inv_ra, true, tw,
                [&](int s, int j, int r) { return smem[s * p.pl + j * p.pr + r]; },
                [&](int s, int j, int q, double2 x) { dst[p.element(s) * n + j + q * p.ra] = cscale(x, a.scale); });
        });
    }
}

}  // namespace

namespace {

// The two radices of every length up to 32 x 32, zero for those without: a pass asks several times.
struct TwoPlans {
    static constexpr int kLast = 32 * 32;
    unsigned char ra[kLast + 1] = {}, rb[kLast + 1] = {};
    TwoPlans()
    {
        // of a length's pairs the one with the smallest larger factor, the larger one last
        for (int hi = 32; hi >= 4; --hi)
            for (int lo = 2; lo <= hi; ++lo) {
                const int kind = kind_of(lo, hi);
                // 2 x 17 .. 2 x 31 fill too few threads (n = 58, us per pass: 19, the chirp pass 13)
                if (kind < 0 || ((kind == 4 || kind == 5) && lo < (is_prime17(lo) || is_prime17(hi) ? 3 : 14))) continue;
                ra[lo * hi] = (unsigned char)lo;
                rb[lo * hi] = (unsigned char)hi;
            }
    }
};

}  // namespace

bool fft_two_radices(int n, int* ra, int* rb)
{
    static const TwoPlans plans;
    if (n < 0 || n > TwoPlans::kLast || plans.ra[n] == 0) return false;
    *ra = plans.ra[n];
    *rb = plans.rb[n];
    return true;
}

int fft_two_vectors(int n)
{
    int ra, rb;
    return fft_two_radices(n, &ra, &rb) && (kind_of(ra, rb) == 1 || kind_of(ra, rb) == 4) ? 4 : 8;
}

cudaError_t fft_two_launch(const double2* src, double2* dst, const FftPassArgs& a, int ntiles, int sign, cudaStream_t stream, int nz)
{
    switch (kind_of(a.radix[0], a.radix[1])) {
        case 0: return FftTwoKind<0>::launch(src, dst, a, ntiles, sign, stream, nz);
        case 1: return FftTwoKind<1>::launch(src, dst, a, ntiles, sign, stream, nz);
        case 2: return FftTwoKind<2>::launch(src, dst, a, ntiles, sign, stream, nz);
        case 3: return FftTwoKind<3>::launch(src, dst, a, ntiles, sign, stream, nz);
        case 4: return FftTwoKind<4>::launch(src, dst, a, ntiles, sign, stream, nz);
        case 5: return FftTwoKind<5>::launch(src, dst, a, ntiles, sign, stream, nz);
        case 6: return FftTwoKind<6>::launch(src, dst, a, ntiles, sign, stream, nz);
        default: return cudaErrorInvalidValue;
    }
}

bool fft_plane_supported(int n, int nz)
{
    int ra, rb;
    return n <= (nz == 1 ? 48 : 32) && fft_two_radices(n, &ra, &rb) && kind_of(ra, rb) == 0;
}

cudaError_t fft_plane_launch(const double2* src, double2* dst, const FftPlaneArgs& a0, int sign, cudaStream_t stream, int nz)
{
    FftPlaneArgs a = a0;
    if (!fft_plane_supported(a.n, nz) || !fft_two_radices(a.n, &a.ra, &a.rb)) return cudaErrorInvalidValue;
    const size_t smem = (size_t)a.n * Plane(a.n, a.ra, a.rb).pl * sizeof(double2);
    const int threads = std::min(512, (a.n * a.rb + 31) / 32 * 32);
    auto go = [&](auto k) -> cudaError_t {   // 42 KB of shared memory at most
        k<<<dim3(a.n, 1, nz), threads, smem, stream>>>(src, dst, a);
        return cudaGetLastError();
    };
    return sign < 0 ? go(fft_plane_kernel<-1>) : go(fft_plane_kernel<1>);
}

}  // namespace pfsoft_dev
