// A kind of two-stage FFT pass (fft_two.cu has the design and what it measures). Compiled once for each FFT_KIND, into a
// module of its own: a process loads a module whole when it first launches from it, and the seven kinds in one
// (21 MB) took 20 ms of a process's first transform.

#include <algorithm>

#include "fft_core.cuh"
#include "fft_two.cuh"

#ifndef FFT_KIND
#define FFT_KIND 0
#endif

namespace pfsoft_dev {
namespace fftk {

namespace {

// butterfly t of a stage with m butterflies per vector: its vector and index
__device__ __forceinline__ void place(bool across, int t, int lg, int m, unsigned inv, int& kk, int& j)
{
    if (across) {
        kk = t & ((1 << lg) - 1);
        j = t >> lg;
    } else {
        kk = m == 1 ? t : (int)__umulhi((unsigned)t, inv);   // t / m
        j = t - kk * m;
    }
}

template <int SIGN, int R>
__device__ __forceinline__ void stage_one(const FftPassArgs& a, const double2* src, double2* smem, int nv, int lg, int vp)
{
    const int m = a.n / R, pitch = R | 1;
    const bool across = a.src.se != 1;
    const unsigned inv = 0xffffffffu / (unsigned)m + 1u;
    for (int t = threadIdx.x; t < m << lg; t += blockDim.x) {
        int kk, j;
        place(across, t, lg, m, inv, kk, j);
        if (kk >= nv) continue;
        const double2* p = src + (long long)kk * a.src.sv + (long long)j * a.src.se;
        const long long step = (long long)m * a.src.se;
        double2 v[R];
#pragma unroll
        for (int r = 0; r < R; ++r) v[r] = __ldg(p + r * step);
        butterfly<SIGN, R>(v);
        double2* o = smem + kk * vp + j * pitch;
#pragma unroll
        for (int q = 0; q < R; ++q) o[q] = v[q];
    }
}

template <int SIGN, int R>
__device__ __forceinline__ void stage_two(const FftPassArgs& a, double2* dst, const double2* smem, int nv, int lg, int vp)
{
    const int m = a.n / R, pitch = m | 1;
    const bool across = a.dst.se != 1;
    const unsigned inv = 0xffffffffu / (unsigned)m + 1u;
    const double2* tw = a.twiddle + a.n;
    for (int t = threadIdx.x; t < m << lg; t += blockDim.x) {
        int kk, j;
        place(across, t, lg, m, inv, kk, j);
        if (kk >= nv) continue;
        const double2* o = smem + kk * vp + j;
        double2 v[R];
        v[0] = o[0];
#pragma unroll
        for (int r = 1; r < R; ++r) {
            double2 w = __ldg(tw + (r - 1) * m + j);
            if (SIGN > 0) w.y = -w.y;
            v[r] = cmul(o[r * pitch], w);
        }
        butterfly<SIGN, R>(v);
        double2* p = dst + (long long)kk * a.dst.sv + (long long)j * a.dst.se;
        const long long step = (long long)m * a.dst.se;
#pragma unroll
        for (int q = 0; q < R; ++q) __stcs(p + q * step, cscale(v[q], a.scale));   // evict-first: next read from HBM
    }
}

template <int SIGN, int KIND>
__global__ void __launch_bounds__(128, kBlocks[KIND])
    fft_two_kernel(const double2* src, double2* dst, const __grid_constant__ FftPassArgs a)
{
    extern __shared__ double2 smem[];
    if (a.srcs) {
        src = a.srcs[blockIdx.z];
        dst = a.dsts[blockIdx.z];
    }
    const int v0 = blockIdx.x * a.kb;
    const int nv = min(a.kb, a.nvec - v0), lg = a.kb == 8 ? 3 : 2;
    const int vp = block_pitch(a.radix[0], a.radix[1], a.kb);
    src += (long long)v0 * a.src.sv + (long long)blockIdx.y * a.src.sb;
    dst += (long long)v0 * a.dst.sv + (long long)blockIdx.y * a.dst.sb;
    with_radix<KIND, 2>(a.radix[0], [&](auto R) { stage_one<SIGN, decltype(R)::value>(a, src, smem, nv, lg, vp); });
    __syncthreads();   // in place: every input of the tile has been read
    with_radix<KIND, 2>(a.radix[1], [&](auto R) { stage_two<SIGN, decltype(R)::value>(a, dst, smem, nv, lg, vp); });
}

}  // namespace

template <int KIND>
cudaError_t FftTwoKind<KIND>::launch(const double2* src, double2* dst, const FftPassArgs& a0, int ntiles, int sign, cudaStream_t stream, int nz)
{
    FftPassArgs a = a0;
    const int ra = a.radix[0], rb = a.radix[1], top = kMaxRadix[KIND];
    // Where tiles of eight vectors leave SMs idle, tiles of four: a thread then has one butterfly of a stage, not two
    // or more. Us per layer-wise call of two passes, the kernels before these / eight / four: 640 x 24 x 9 14.4 / 17.5 /
    // 15.4, 768 16.4 / 17.6 / 16.1, 960 18.5 / 20.5 / 18.5, 512 14.4 / 11.3 / 10.6, 1024 16.4 / 15.4 / 12.4, with 24 layers
    // (72 tiles) 640 17.5 / 18.5 / 17.5, 1024 21.6 / 18.5 / 16.4.
    if (a.kb == 8 && 8 * rb > 128 && (long long)((a.nvec + 7) / 8) * ntiles * nz <= 148) a.kb = 4;
    const size_t smem = (size_t)a.kb * block_pitch(ra, rb, a.kb) * sizeof(double2);
    const size_t largest = (size_t)8 * block_pitch(top, top, 8) * sizeof(double2);   // the kind's largest radices
    const int threads = std::min(128, (a.kb * rb + 31) / 32 * 32);
    auto go = [&](auto k) -> cudaError_t {
        const cudaError_t e = allow_shared(k, smem, largest);
        if (e != cudaSuccess) return e;
        k<<<dim3((a.nvec + a.kb - 1) / a.kb, ntiles, nz), threads, smem, stream>>>(src, dst, a);
        return cudaGetLastError();
    };
    return sign < 0 ? go(fft_two_kernel<-1, KIND>) : go(fft_two_kernel<1, KIND>);
}

template struct FftTwoKind<FFT_KIND>;

}  // namespace fftk
}  // namespace pfsoft_dev
