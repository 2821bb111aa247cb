// Discrete Wigner transform over beta (the DWT stage of DSOFT / iDSOFT) and its tables.
#pragma once

#include <cuda_runtime.h>

#include <vector>

namespace pfsoft_dev {

// Per-bandwidth constant tables, built once on the device (tables_build) and cached.
// All doubles; N = 2B, beta_k = pi(2k+1)/(4B) (include/PFSOFTlib_headers/fn_dwt.hpp:155-159).
struct BandTables {
    int B = 0, N = 0;
    double* cosb = nullptr;     // cos(beta_k)                    [N]
    double* sinh = nullptr;     // sin(beta_k / 2)                [N]
    double* cosh = nullptr;     // cos(beta_k / 2)                [N]
    double* w = nullptr;        // quadrature weights w_B(k)      [N]   (fn_dwt.hpp:62-83)
    double2* twiddle = nullptr; // exp(-2 pi i t / N) and the FFT's second copy (fft_twiddle_elems)
    double2* ht = nullptr;      // {cos, sin}(pi n / (2N))        [B]
    void* block = nullptr;      // single allocation holding all of the above
    double2* bluestein = nullptr;   // fft_needs_bluestein(N): the FFT pass's table (own allocation)
    // only for the FP64 DWT (series_tables_build; null until a caller asks for them)
    // the Wigner rows at beta = pi/2, ((2l+1)/2)^(1/4) P[l][n][M] (-1)^(n-M) for n > M, tiles of 8 degrees x 8 n per
    // order M (delta_offset); zero for l < M, n > l and l >= B          [delta_entries(B)]
    double* delta = nullptr;
    // (2 - [n = 0]) cos(n beta_k) and sin, n = 2 m + q < B, k < B, tiles of 8 m x 8 k in the order
    // [cos, sin][q][m / 8][k / 8], row-major, zero past either end            [trig_entries(B)]
    double* trig = nullptr;
    // only for the split-precision DWT (split_tables_build; null until a caller asks for them)
    double* normf = nullptr;    // seed norm per order class      [B(B+1)/2] (fn_dwt.hpp:117-121)
    double2* pw_sin = nullptr;  // sin(beta_k/2)^p as {mantissa, exponent}  [2B][N], p < 2B
    double2* pw_cos = nullptr;  // cos(beta_k/2)^p as {mantissa, exponent}  [2B][N]
    // recurrence coefficients of the step l -> l+1 for every order class and degree M <= l < B,
    // class (M, M') from rc_offset(B, M, M'): {c1, f1 f2} and f1      [rc_entries(B)]
    double2* rc_cf = nullptr;
    double* rc_f1 = nullptr;
};

// Entries of the recurrence-coefficient table before class (M, M'): classes run M = 0, 1, ...
// and M' = 0..M within M, each with B - M degrees.
__host__ __device__ __forceinline__ long long rc_offset(int B, int M, int Mp)
{
    const long long m = M;
    return (long long)(B + 1) * m * (m + 1) / 2 - m * (m + 1) * (2 * m + 1) / 6 + (long long)Mp * (B - M);
}
__host__ __device__ __forceinline__ long long rc_entries(int B) { return rc_offset(B, B, 0); }

// Doubles before order M's tiles in BandTables::delta: order m has tri(nb) - tri(m/8) tiles of 64 (nb = ceil(B/8)
// blocks of degrees, block lb with lb + 1 tiles).
__host__ __device__ __forceinline__ long long delta_offset(int B, int M)
{
    const long long nb = (B + 7) / 8, T = nb * (nb + 1), b = M >> 3, r = M & 7;
    return 256 * (b * T - (b - 1) * b * (b + 1) / 3) + r * 32 * (T - b * (b + 1));
}
__host__ __device__ __forceinline__ long long delta_entries(int B) { return delta_offset(B, B); }

__host__ __device__ __forceinline__ long long trig_entries(int B)
{
    const long long nb = (B + 7) / 8;
    return 4 * ((nb + 1) / 2) * nb * 64;
}

size_t tables_bytes(int B);
// Carve the tables out of `mem` (tables_bytes(B) bytes, 256-byte aligned) and fill them.
cudaError_t tables_build(int B, void* mem, BandTables* t, cudaStream_t stream);
// The FP64 DWT's own tables, and the split-precision DWT's, after tables_build, each from another block.
size_t series_tables_bytes(int B);
cudaError_t series_tables_build(int B, void* mem, BandTables* t, cudaStream_t stream);
size_t split_tables_bytes(int B);
cudaError_t split_tables_build(int B, void* mem, BandTables* t, cudaStream_t stream);

// The cached tables of a bandwidth on the current device (api.cu), with the DWTs' named by `sets` built on
// first use: what a process keeps is what its calls need.
constexpr int kSeriesTables = 1, kSplitTables = 2;
int tables_for(int B, BandTables* out, int sets = kSeriesTables);

struct DwtArgs {
    int B, N;
    const double* w;
    const double2* ht;
    const double2* tw;
    const double* delta;
    const double* trig;
    // Optional subset of order classes (ascending, so longest first): when set, the kernels run
    // classes[0 .. n_classes-1] only and leave every other class's outputs untouched.
    const int* classes;
    int n_classes;
    // Several transforms of one bandwidth: device tables of their spectra and coefficients
    double2* const* Xs;
    double2* const* coefs;
    int T;   // set by the launch
    // Inverse only: also zero the Nyquist bins (row B or column B of X, which no order class
    // writes) in the kernel's tail, instead of a separate launch.
    int zero_nyquist;
};

// Arguments of the DWT launches over every order class of a bandwidth's tables.
DwtArgs dwt_args_for(const BandTables& t);

// A launch of direction 0 (forward) or 1: of T transforms of one length.
typedef cudaError_t (*DwtLaunch)(int dir, const double2* X, double2* coeffs, const DwtArgs& a, int T, cudaStream_t stream);

// The even lengths that may have a compile-time DFT over beta (dwt_fixed.cu), in parts of kFixedSpan that are
// compiled by themselves, part by part; null for a length without one.
constexpr int kFixedFirst = 98, kFixedLast = 512, kFixedSpan = 32;
constexpr int kFixedParts = (kFixedLast - kFixedFirst) / kFixedSpan + 1;
template <int PART>
struct DwtFixedPart {
    static DwtLaunch launch(int N);
};

// T transforms (T > 1: a.Xs and a.coefs; X and coeffs are then unused).
// Forward: X (beta-innermost spectrum, N^3) -> packed coefficients, scale pi/(2B^2).
// Whether the columns of length N have a compile-time DFT over beta (dwt.cu) instead of a matrix product.
bool dwt_has_dft(int N);

cudaError_t dwt_forward_launch(const double2* X, double2* coeffs, const DwtArgs& a, int T, cudaStream_t stream);
// Inverse: packed coefficients -> X (all non-Nyquist beta columns), scale 2B^2/pi.
cudaError_t dwt_inverse_launch(const double2* coeffs, double2* X, const DwtArgs& a, int T, cudaStream_t stream);
// Zero the beta columns of the Nyquist bins (row == B or col == B) of X.
cudaError_t zero_nyquist_launch(double2* X, int B, cudaStream_t stream);

// ---- split-precision DWT over many transforms and bandwidths (dwt_split.cu) ------------------
// A group holds T transforms of one bandwidth; X[t] is transform t's beta-innermost spectrum
// (N^3) and coeffs[t] its packed coefficients. Forward reads X and writes coeffs, inverse the
// other way.
struct DwtGroup {
    int B, N, T;
    const double* cosb;
    const double* w;
    const double* normf;
    const double2* pw_sin;
    const double2* pw_cos;
    const double2* rc_cf;   // recurrence coefficients (BandTables::rc_cf / rc_f1)
    const double* rc_f1;
    double2* const* X;
    double2* const* coeffs;
};

// Split-precision DWT on the tensor cores (dwt_split.cu) for groups whose bandwidth passes
// dwt_split_supported. A launch covers several groups of d_groups, described by segments
// (dwt_split_segments: group index, bandwidth and transform count of each); one persistent
// launch per direction; a bounded wait that ran out sets *d_status to 1.
bool dwt_split_supported(int B);
int dwt_split_segments(int direction, const std::vector<int>& group, const std::vector<int>& B,
                       const std::vector<int>& T, std::vector<unsigned char>& out);   // returns the item count
size_t dwt_split_seg_bytes();
cudaError_t dwt_split_prepare();   // kernel attributes; call once per device before any capture
// The split kernels read operand scales from a table of dwt_split_aux_elems(B) double2 that
// follows each transform's spectrum (N^3 double2) in its workspace; dwt_split_scales fills it
// (forward: from the spectra, after the FFT passes; inverse: from the coefficients), and the
// row scales of the generated operand. w: the group's quadrature weights.
size_t dwt_split_aux_elems(int B);
cudaError_t dwt_split_scales(int direction, int B, int T, double2* const* d_ws, const double2* const* d_coeffs,
                             const double* w, cudaStream_t stream);
cudaError_t dwt_split_launch(int direction, const DwtGroup* d_groups, const void* d_segs, int nseg, int n_items,
                             int* d_status, cudaStream_t stream);
// Test knob: when nonzero, every later split launch first waits up to `ns` nanoseconds on a
// barrier that nothing signals, before any MMA is issued, so that its bounded-wait exit runs.
void dwt_split_set_fail_ns(unsigned long long ns);

// Sets the detail string returned by pfsoft_last_error() on the calling thread.
void set_last_error(const char* msg);

}  // namespace pfsoft_dev
