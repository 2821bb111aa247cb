// What the two-stage FFT kernels (fft_two_kind.cu) and their choice and launch (fft_two.cu, which has the design) share:
// the kinds, their radices, and the shared-memory pitch of a vector.
#pragma once

#include <type_traits>

#include "common.cuh"
#include "fft.cuh"

namespace pfsoft_dev {
namespace fftk {

// Vectors of a tile are this far apart in shared memory: 8 vectors (or 4 vectors x 2 butterflies) of one
// access meet distinct 16-byte banks.
__host__ __device__ __forceinline__ int block_pitch(int ra, int rb, int kb)
{
    const int len = rb * (ra | 1);
    return kb == 8 ? (len | 1) : len + (10 - len % 8) % 8;
}

// The kernels: 0 for radices up to 16, 1 up to 26, 2 up to 30, 4 and 5 up to 26 and 32 with the primes from
// 17 on (23 only in 5: its sums would spill in 4), 3 and 6 for 16.32, 32.32 and 16.16 alone, so that no length
// pays the registers or the code of a radix that it does not need (us per pass: N = 256 in kernel 0 93.2,
// alone 88.9; 512 with the primes 913, without 885, alone 853). CTAs per SM: up to 16 five are faster than four (N =
// 128 21.2 against 23.1, 192 44.8 against 47.3, 240 78.2 against 80.7; not for 16.16), up to 30 three
// faster than two (N = 448 545 against 653), at 32 two (N = 512 885 against 947).
constexpr int kKinds = 7;
constexpr int kMaxRadix[kKinds] = {16, 26, 30, 32, 26, 32, 16}, kBlocks[kKinds] = {5, 4, 3, 2, 4, 2, 4};
constexpr bool is_prime17(int r) { return r == 17 || r == 19 || r == 23 || r == 29 || r == 31; }
constexpr bool has_radix(int kind, int r)
{
    if (kind == 3 || kind == 6) return r == 16 || (kind == 3 && r == 32);
    return r >= (kind == 1 ? 7 : (kind == 2 ? 14 : 2)) && r <= kMaxRadix[kind] && r != 27 &&
           (kind == 4 || kind == 5 || !is_prime17(r)) && (kind != 4 || r != 23);
}
constexpr int kind_of(int ra, int rb)
{
    if (ra == 16 && rb == 16) return 6;
    for (int kind = 0; kind < kKinds; ++kind)
        if (has_radix(kind, ra) && has_radix(kind, rb)) return kind;
    return -1;
}

// f.template run<R>() for the kernel's radix R == r
template <int KIND, int R, class Fn>
__device__ __forceinline__ void with_radix(int r, const Fn& f)
{
    if constexpr (R <= kMaxRadix[KIND]) {
        if constexpr (has_radix(KIND, R)) {
            if (r == R) {
                f(std::integral_constant<int, R>());
                return;
            }
        }
        with_radix<KIND, R + 1>(r, f);
    }
}

// A launch of a kind's kernel (fft_two_kind.cu, compiled once for each kind).
template <int KIND>
struct FftTwoKind {
    static cudaError_t launch(const double2* src, double2* dst, const FftPassArgs& a, int ntiles, int sign, cudaStream_t stream, int nz);
};

}  // namespace fftk
}  // namespace pfsoft_dev
