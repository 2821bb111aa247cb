// The FP64 discrete Wigner transform with a compile-time DFT over beta, for the lengths N = 98 .. 512 that are a product
// of two or three radices of at most 20 (dwt.cu says why, and what it measures against the matrix form).
//
// Compiled once for each part DWT_PART of the range, into a module of its own: a process loads a module whole
// when it first launches from it. With the 97 lengths in one module (43 MB) and the FFT kinds in another
// (21 MB) a process's first transform took 68 ms, of whatever length; so 4 to 5.

#include <utility>

#include "dwt_sums.cuh"
#include "fft_core.cuh"

#ifndef DWT_PART
#define DWT_PART 0
#endif

namespace pfsoft_dev {

namespace {

using namespace dwtk;
using namespace fftk;

// ---- the beta DFT of a class's columns -------------------------------------------------------
// The columns lie in shared memory with an odd pitch, and consecutive threads take consecutive
// columns: then every access of eight columns meets eight distinct 16-byte banks whatever the
// element, and the eight share each twiddle. HBM is read and written in contiguous rows, the
// reordering of the samples happens on the shared-memory side.

__host__ __device__ __forceinline__ int col_pitch(int N) { return N | 1; }

// Element e of a column's DFT is the sample k: even samples ascending, then odd ones descending, so
// that the length-N DFT gives the cosine sums (Makhoul 1980).
__device__ __forceinline__ int sample_of(int e, int B, int N) { return e < B ? 2 * e : 2 * (N - 1 - e) + 1; }

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

template <class F, int KP>
cudaError_t launch_fft(int dir, const double2* X, double2* coeffs, const DwtArgs& a, int T, cudaStream_t s)
{
    // the columns' DFT, and behind it the forward's B fragments or the inverse's coefficients
    const size_t smem = (F::kElems + ((F::B + 7) / 8) * (dir == 0 ? 64 : 8 * kGS)) * sizeof(double2);
    return dir == 0 ? launch(dwt_forward_fft_kernel<F, KP>, X, coeffs, F::NT, smem, smem, a, T, s)
                    : launch(dwt_inverse_fft_kernel<F, KP>, (const double2*)coeffs, const_cast<double2*>(X), F::NT, smem, smem, a, T, s);
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

template <int N>
constexpr DwtLaunch fixed_launch()
{
    constexpr int NW = N <= 256 ? 4 : 8;
    constexpr FixedPlan p = fixed_plan(N, 32 * NW);
    if constexpr (p.r0 > 0) return launch_fft<FixedFft<N, NW, p.r0, p.r1, p.r2>, ((N + 15) / 16 + NW - 1) / NW>;
    else return nullptr;
}

// Length first + 2 i of the part's; those past the range's end have no launch.
template <int... I>
DwtLaunch part_launch_of(int i, std::integer_sequence<int, I...>)
{
    constexpr int first = kFixedFirst + kFixedSpan * DWT_PART;
    static constexpr DwtLaunch table[] = {first + 2 * I <= kFixedLast ? fixed_launch<(first + 2 * I <= kFixedLast ? first + 2 * I : kFixedFirst)>()
                                                                      : nullptr...};
    return table[i];
}

}  // namespace

template <int PART>
DwtLaunch DwtFixedPart<PART>::launch(int N)
{
    return part_launch_of((N - kFixedFirst - kFixedSpan * PART) / 2, std::make_integer_sequence<int, kFixedSpan / 2>());
}

template struct DwtFixedPart<DWT_PART>;

}  // namespace pfsoft_dev
