// Batched layer-wise 2D DFT passes (the reference's uzl_fftw_layer_wise_{DFT2,IDFT2}_grid3D,
// src/fftw_wrapper.cpp:47-173, re-designed for HBM): each pass is one 1D DFT direction over
// every beta layer, tiled so that one CTA transforms KB vectors, with the transpose to or from
// the beta-innermost spectrum layout fused into the load or store.
#pragma once

#include <cuda_runtime.h>

namespace pfsoft_dev {

constexpr int kFftMaxStages = 12;

// Element e of vector v in tile b lives at  base + v*sv + b*sb + e*se  (units of double2).
struct FftStrides {
    long long sv, sb, se;
};

struct FftPassArgs {
    int n;                       // transform length
    int nvec;                    // total vectors along the tiled index (k)
    int kb;                      // vectors per CTA
    int nstages;
    int radix[kFftMaxStages];
    int ns[kFftMaxStages];       // product of the radices of the earlier stages
    FftStrides src, dst;
    double scale;                // applied to the stored values (1 = none)
    // twiddle[t] = exp(-2*pi*i*t/n), t < n; behind them, for two-stage plans, exp(-2*pi*i*r*j/n) at
    // n + (r - 1) ra + j, 1 <= r < rb, j < ra (fft_twiddle_elems entries in all)
    const double2* twiddle;
    // batched passes: when set, transform z = blockIdx.z reads srcs[z] and writes dsts[z]
    const double2* const* srcs;
    double2* const* dsts;
    // lengths that fft_needs_bluestein names: the table of the matrix or the chirp kernel
    // (fft_bluestein_fill); null keeps direct O(R^2) stages for their prime factors
    const double2* bluestein;
};

// Lengths with a prime factor too large for a direct stage whose passes need a table: the matrix kernel's
// (fft_matrix.cu), or the chirps of Bluestein's algorithm (fft_chirp_kernel) for n <= 512, or even and
// <= 1024.
bool fft_needs_bluestein(int n);
size_t fft_bluestein_elems(int n);   // double2 entries of the table
// The table, computed on the host in long double (layout: fft_matrix_fill, fft_chirp_kernel).
void fft_bluestein_fill(int n, double2* out);

// Lengths n = ra rb that the two-stage kernel takes (fft_two.cu), its tile vectors, and its launch.
bool fft_two_radices(int n, int* ra, int* rb);
int fft_two_vectors(int n);
cudaError_t fft_two_launch(const double2* src, double2* dst, const FftPassArgs& a, int ntiles, int sign, cudaStream_t stream, int nz);

// Both passes of a transform in one launch, for small even N = n (fft_two.cu): forward G[k][c][r] to X[r][c][k],
// backward X to G scaled; for nz > 1 transforms the device tables srcs and dsts.
struct FftPlaneArgs {
    int n, ra, rb;
    double scale;
    const double2* twiddle;
    const double2* const* srcs;
    double2* const* dsts;
};
bool fft_plane_supported(int n, int nz);
cudaError_t fft_plane_launch(const double2* src, double2* dst, const FftPlaneArgs& a, int sign, cudaStream_t stream, int nz);

// Lengths n = r p that the matrix kernel takes (fft_matrix.cu), its table for p (double2 entries, contents)
// and its launch.
bool fft_matrix_radices(int n, int* r, int* p);
size_t fft_matrix_elems(int p);
void fft_matrix_fill(int p, double2* out);
cudaError_t fft_matrix_launch(const double2* src, double2* dst, const FftPassArgs& a, int ntiles, int sign, cudaStream_t stream,
                              int nz);

// Entries of a length's twiddle table (FftPassArgs::twiddle).
__host__ __device__ __forceinline__ size_t fft_twiddle_elems(int n) { return 2 * (size_t)n; }

// Radix plan for length n; returns the number of stages (0 if n cannot be planned).
int fft_plan_radices(int n, int* radix, int* ns);

// Launch one pass over a grid of (ceil(nvec/kb), ntiles, nz) CTAs. sign = -1 forward, +1 inverse.
// nz > 1 requires a.srcs / a.dsts (one base pointer per transform).
cudaError_t fft_pass_launch(const double2* src, double2* dst, const FftPassArgs& a, int ntiles, int sign,
                            cudaStream_t stream, int nz = 1);

size_t fft_pass_smem_bytes(const FftPassArgs& a);

// Bytes past a transform's spectrum that its workspace size has always included (they held the counters
// of a launch of both passes at once).
constexpr int kFftSyncBytes = 4096;

// Vectors per tile for length n: 8 (128 contiguous bytes on the transposed side), or 4 where the buffers
// of 8 vectors would leave a single CTA per SM, or the radices few.
int fft_tile_vectors(int n);

}  // namespace pfsoft_dev
