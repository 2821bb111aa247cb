// Batched 1D DFT passes over the (alpha, gamma) plane of every beta layer (sm_100a): the choice of a
// pass's kernel, and two of the four.
//
//   fft_two.cu         n = ra rb with register butterflies up to 32: one shared-memory exchange
//   fft_matrix.cu      n = R p, p odd and 17 .. 249: a matrix product on the FP64 MMA
//   fft_chirp_kernel   n with a larger prime, or one with too many other factors: Bluestein's convolution
//   fft_pass_kernel    what is left: n up to 7, 9, 11 and 13; products of 2, 3, 5, 7, 11 and 13 that no two factors
//                      up to 32 make, such as 243, 343, 486 and 648; odd n of 513 and more with a prime that the
//                      matrix pass does not take (521: direct O(R^2) stages, no table is kept for odd lengths
//                      and the chirp pass ends at 512); such n above 1024. Mixed-radix Stockham autosort
//                      (Govindaraju et al., SC'08 formulation). A stage of
//     radix R over n points with Ns = product of the earlier radices maps butterfly j to
//       inputs  x[j + r*n/R] * w_n^(r * (j mod Ns) * n/(Ns R)),   r < R
//       outputs y[(j/Ns)*Ns*R + (j mod Ns) + q*Ns],              q < R
//     and the last stage leaves the result in natural order.
//
// In each, the first stage reads HBM into registers and the last one stores to HBM from registers,
// the exchanges between go through shared memory, and the butterfly -> thread map of a stage that
// touches HBM follows the stride there: along the vector where its elements are contiguous (se == 1),
// else across the tile's vectors, whose values are contiguous (sv == 1). That is how the
// beta <-> (alpha, gamma) transpose rides inside the first and last stage at no extra HBM traffic.
// Stores are evict-first: a pass's output is next read from HBM (measured at B = 128: -1.0 % iDSOFT,
// -0.5 % DSOFT; neutral at B = 256).

#include <algorithm>
#include <cmath>
#include <cstring>
#include <vector>

#include "common.cuh"
#include "fft.cuh"
#include "fft_core.cuh"

namespace pfsoft_dev {

namespace {

using namespace fftk;

template <int SIGN, int R>
__device__ __forceinline__ void run_stage_fixed(const FftPassArgs& a, int s, const double2* gsrc,
                                                double2* gdst, const double2* sin_, double2* sout,
                                                int nv, long long src_base, long long dst_base)
{
    const int n = a.n;
    const int m = n / R;
    const int Ns = a.ns[s];
    const int step = n / (Ns * R);
    const bool first = (s == 0), last = (s == a.nstages - 1);
    const int pl = padded_len(n);
    // thread map: along the vector (j fastest) unless this stage touches HBM with a non-unit
    // element stride, in which case across vectors (kk fastest)
    const bool kk_fast = (first && a.src.se != 1) || (last && a.dst.se != 1);
    const int total = nv * m;
    for (int t = threadIdx.x; t < total; t += blockDim.x) {
        int j, kk;
        if (kk_fast) {
            kk = t % nv;
            j = t / nv;
        } else {
            j = t % m;
            kk = t / m;
        }
        double2 v[R];
        if (first) {
            const double2* p = gsrc + src_base + (long long)kk * a.src.sv;
#pragma unroll
            for (int r = 0; r < R; ++r) v[r] = __ldg(p + (long long)(j + r * m) * a.src.se);
        } else {
            const double2* p = sin_ + kk * pl;
#pragma unroll
            for (int r = 0; r < R; ++r) v[r] = p[spos(j + r * m)];
        }
        const int k = j % Ns;
        if (Ns > 1) {
#pragma unroll
            for (int r = 1; r < R; ++r) v[r] = cmul(v[r], twiddle(a.twiddle, r * k * step, SIGN));
        }
        butterfly<SIGN, R>(v);
        const int ob = (j / Ns) * Ns * R + k;
        if (last) {
            double2* p = gdst + dst_base + (long long)kk * a.dst.sv;
#pragma unroll
            for (int q = 0; q < R; ++q) __stcs(p + (long long)(ob + q * Ns) * a.dst.se, cscale(v[q], a.scale));
        } else {
            double2* p = sout + kk * pl;
#pragma unroll
            for (int q = 0; q < R; ++q) p[spos(ob + q * Ns)] = v[q];
        }
    }
}

// Direct O(R^2) butterfly for any other radix (lengths with a prime factor above 5). The stage's
// outputs, not its butterflies, are spread over the threads: a large prime leaves few butterflies
// per tile (m = n / R of them per vector), while each of the R outputs of a butterfly is an
// independent R-term sum. A stage never writes the buffer it reads.
template <int SIGN>
__device__ void run_stage_generic(const FftPassArgs& a, int s, const double2* gsrc,
                                  double2* gdst, const double2* sin_, double2* sout, int nv,
                                  long long src_base, long long dst_base)
{
    const int n = a.n, R = a.radix[s];
    const int m = n / R;
    const int Ns = a.ns[s];
    const int step = n / (Ns * R);
    const int rstep = n / R;   // exp(SIGN 2 pi i rq/R) = twiddle[(rq mod R) * n/R]
    const bool first = (s == 0), last = (s == a.nstages - 1);
    const int pl = padded_len(n);
    const bool kk_fast = (first && a.src.se != 1) || (last && a.dst.se != 1);
    const int total = nv * m * R;
    for (int t = threadIdx.x; t < total; t += blockDim.x) {
        int j, kk, q;
        if (kk_fast) {   // consecutive threads: consecutive vectors (contiguous in HBM)
            kk = t % nv;
            const int u = t / nv;
            q = u % R;
            j = u / R;
        } else {
            q = t % R;
            const int u = t / R;
            j = u % m;
            kk = u / m;
        }
        const int k = j % Ns;
        const int ob = (j / Ns) * Ns * R + k;
        // input r carries the stage twiddle w_n^(r k step) and the DFT twiddle w_R^(r q) =
        // w_n^(r q rstep): one table entry w_n^(r cq mod n), its index advanced by cq per input
        const int cq = (int)(((long long)k * step + (long long)q * rstep) % n);
        double2 acc = first ? __ldg(gsrc + src_base + (long long)kk * a.src.sv + (long long)j * a.src.se)
                            : sin_[kk * pl + spos(j)];
        int e = 0;
        for (int r = 1; r < R; ++r) {
            double2 x = first ? __ldg(gsrc + src_base + (long long)kk * a.src.sv + (long long)(j + r * m) * a.src.se)
                              : sin_[kk * pl + spos(j + r * m)];
            e += cq;
            if (e >= n) e -= n;
            if (e) x = cmul(x, twiddle(a.twiddle, e, SIGN));
            acc = cadd(acc, x);
        }
        if (last) gdst[dst_base + (long long)kk * a.dst.sv + (long long)(ob + q * Ns) * a.dst.se] = cscale(acc, a.scale);
        else sout[kk * pl + spos(ob + q * Ns)] = acc;
    }
}

template <int SIGN>
__global__ void __launch_bounds__(256, 2) fft_pass_kernel(const double2* src, double2* dst, const FftPassArgs a)
{
    extern __shared__ double2 smem[];
    if (a.srcs) {
        src = a.srcs[blockIdx.z];
        dst = a.dsts[blockIdx.z];
    }
    const int v0 = blockIdx.x * a.kb;
    const int nv = min(a.kb, a.nvec - v0);
    const long long src_base = (long long)v0 * a.src.sv + (long long)blockIdx.y * a.src.sb;
    const long long dst_base = (long long)v0 * a.dst.sv + (long long)blockIdx.y * a.dst.sb;
    const int pl = padded_len(a.n);
    double2* buf[2] = {smem, smem + a.kb * pl};
    // In-place passes (src == dst) are safe: every CTA reads its whole tile in stage 0 and
    // writes it only in the last stage, after at least one __syncthreads (nstages >= 2), or in
    // the same thread's registers when there is a single stage.
    for (int s = 0; s < a.nstages; ++s) {
        const double2* sin_ = buf[(s + 1) & 1];
        double2* sout = buf[s & 1];
        switch (a.radix[s]) {
            case 16: run_stage_fixed<SIGN, 16>(a, s, src, dst, sin_, sout, nv, src_base, dst_base); break;
            case 8: run_stage_fixed<SIGN, 8>(a, s, src, dst, sin_, sout, nv, src_base, dst_base); break;
            case 4: run_stage_fixed<SIGN, 4>(a, s, src, dst, sin_, sout, nv, src_base, dst_base); break;
            case 2: run_stage_fixed<SIGN, 2>(a, s, src, dst, sin_, sout, nv, src_base, dst_base); break;
            case 1: run_stage_fixed<SIGN, 1>(a, s, src, dst, sin_, sout, nv, src_base, dst_base); break;
            case 3: run_stage_fixed<SIGN, 3>(a, s, src, dst, sin_, sout, nv, src_base, dst_base); break;
            case 5: run_stage_fixed<SIGN, 5>(a, s, src, dst, sin_, sout, nv, src_base, dst_base); break;
            default: run_stage_generic<SIGN>(a, s, src, dst, sin_, sout, nv, src_base, dst_base); break;
        }
        if (s + 1 < a.nstages) __syncthreads();
    }
}

// Bluestein pass for a length n with a large prime factor. An even n is first split in two (decimation
// in frequency): outputs 2k + s are the length n/2 DFT of (x_j + x_(j+n/2)) or (x_j - x_(j+n/2))
// w_n^j. Each length-m DFT (m = n/2, or n when odd) is the chirp-z convolution
//   X_k = w_k sum_j (x_j w_j) conj(w_(k-j)),  w_j = exp(-pi i j^2 / m),
// by two transforms of the smallest planned length M >= 2m - 1: decimation in frequency with radices
// R0, R1, R2 (natural order in, digit-reversed out), a product with the chirp's transform stored in
// that order, and decimation in time back. The first stage reads HBM into registers (its upper half
// of inputs is zero), the last forward stage, the product and the first backward stage work on one
// thread's registers, and the last stage stores to HBM (its upper half of outputs is not needed), so
// that a sequence crosses shared memory four times. A backward DFT is the forward one of the conjugate.
// What bounds it: FP64 arithmetic and the shared-memory pipe, about 4 M (M/m) log2 M multiply-adds a
// value. Measured on B200 at n = 502, per pass: 2.37 ms, radix-4 stages in shared memory at M >= 2n - 1
// 9.15 ms, the matrix pass 2.41 ms: the larger primes stay here.
template <int R0_, int R1_, int R2_, int V_>
struct ChirpPlan {
    static constexpr int R0 = R0_, R1 = R1_, R2 = R2_, V = V_;   // V vectors per CTA
    static constexpr int M = R0 * R1 * R2, h0 = M / R0, h1 = h0 / R1;
    static constexpr int RL = R2;                                // the last radix, on contiguous elements
    // one pad slot per RL elements when RL is even: the threads' runs then start in distinct banks
    static constexpr int kPad = RL == 16 ? 4 : (RL == 8 ? 3 : (RL == 4 ? 2 : 31));
    static __device__ __forceinline__ int pos(int i) { return kPad < 31 ? i + (i >> (kPad & 15)) : i; }
    static constexpr int kLen = kPad < 31 ? M + (M >> (kPad & 15)) : M;
    // pitch of a sequence: consecutive vectors' elements in distinct banks
    static constexpr int PM = V == 4 ? kLen + ((10 - kLen % 8) % 8) : (kLen | 1);
    static constexpr size_t kSmem = (size_t)2 * V * PM * sizeof(double2);
    static constexpr int kMinBlocks = kSmem <= 50 * 1024 ? 3 : 2;
};

// The radix-R0 = 8 butterfly of a first stage whose inputs 4..7 are zero.
template <int SIGN>
__device__ __forceinline__ void dft8_half(double2* v)
{
    const double2 r2 = cmul_i<SIGN>(v[2]), r3 = cmul_i<SIGN>(v[3]);
    const double2 e0 = cadd(v[0], v[2]), e2 = csub(v[0], v[2]), e1 = cadd(v[0], r2), e3 = csub(v[0], r2);
    const double2 o0 = cadd(v[1], v[3]);
    const double2 o1 = rot8<SIGN, 1>(cadd(v[1], r3)), o2 = rot8<SIGN, 2>(csub(v[1], v[3])), o3 = rot8<SIGN, 3>(csub(v[1], r3));
    v[0] = cadd(e0, o0);
    v[4] = csub(e0, o0);
    v[1] = cadd(e1, o1);
    v[5] = csub(e1, o1);
    v[2] = cadd(e2, o2);
    v[6] = csub(e2, o2);
    v[3] = cadd(e3, o3);
    v[7] = csub(e3, o3);
}

template <class P>
__global__ void __launch_bounds__(256, P::kMinBlocks)
    fft_chirp_kernel(const double2* src, double2* dst, const __grid_constant__ FftPassArgs a, int sign)
{
    constexpr int R0 = P::R0, R1 = P::R1, RL = P::RL, V = P::V, M = P::M, h0 = P::h0, h1 = P::h1, PM = P::PM;
    static_assert(R0 == 8, "the first stage's butterfly");
    extern __shared__ double2 smem[];   // [2][V][PM]
    if (a.srcs) {
        src = a.srcs[blockIdx.z];
        dst = a.dsts[blockIdx.z];
    }
    const int n = a.n;
    const bool split = (n & 1) == 0;
    const int m = split ? n >> 1 : n, S = split ? 2 * V : V;
    const double2* wtab = a.bluestein;               // w_j
    const double2* ctab = wtab + m;                  // w_j w_n^j
    const double2* fh = ctab + m;                    // the chirp's transform, digit-reversed, 1/M included
    const double2* tw1 = fh + M;                     // w_M^(i q), [q - 1][i]
    const double2* tw2 = tw1 + (R0 - 1) * h0;        // w_h0^(i q), [q - 1][i]
    const int v0 = blockIdx.x * V;
    const int nv = min(V, a.nvec - v0);
    const long long sbase = (long long)v0 * a.src.sv + (long long)blockIdx.y * a.src.sb;
    const long long dbase = (long long)v0 * a.dst.sv + (long long)blockIdx.y * a.dst.sb;
    const bool vfast_in = a.src.se != 1, vfast_out = a.dst.se != 1;   // vectors contiguous in HBM
    const double cj = sign < 0 ? 1.0 : -1.0;
    for (int t = threadIdx.x; t < V * h0; t += 256) {
        const int v = vfast_in ? t % V : t / h0, i = vfast_in ? t / V : t % h0;
        const double2* p = src + sbase + (long long)v * a.src.sv;
        double2 u[R0], z[R0], x[R0 / 2], y[R0 / 2];
#pragma unroll
        for (int q = 0; q < R0 / 2; ++q) {
            const int j = i + q * h0;
            const bool in = v < nv && j < m;
            x[q] = y[q] = make_double2(0.0, 0.0);
            if (in) x[q] = __ldg(p + (long long)j * a.src.se);
            if (in && split) y[q] = __ldg(p + (long long)(j + m) * a.src.se);
        }
#pragma unroll
        for (int q = 0; q < R0 / 2; ++q) {
            const int j = min(i + q * h0, m - 1);
            x[q].y *= cj;
            y[q].y *= cj;
            u[q] = cmul(cadd(x[q], y[q]), __ldg(wtab + j));
            z[q] = cmul(csub(x[q], y[q]), __ldg(ctab + j));
        }
        dft8_half<-1>(u);
        double2* o = smem + v * PM;
        o[P::pos(i)] = u[0];
#pragma unroll
        for (int q = 1; q < R0; ++q) o[P::pos(i + q * h0)] = cmul(u[q], __ldg(tw1 + (q - 1) * h0 + i));
        if (split) {
            dft8_half<-1>(z);
            o += V * PM;
            o[P::pos(i)] = z[0];
#pragma unroll
            for (int q = 1; q < R0; ++q) o[P::pos(i + q * h0)] = cmul(z[q], __ldg(tw1 + (q - 1) * h0 + i));
        }
    }
    __syncthreads();
    for (int t = threadIdx.x; t < S * (M / R1); t += 256) {
        const int i = t % h1, blk = t / h1 % R0, sq = t / (M / R1);
        double2* o = smem + sq * PM;
        double2 u[R1];
#pragma unroll
        for (int q = 0; q < R1; ++q) u[q] = o[P::pos(blk * h0 + i + q * h1)];
        butterfly<-1, R1>(u);
        o[P::pos(blk * h0 + i)] = u[0];
#pragma unroll
        for (int q = 1; q < R1; ++q) o[P::pos(blk * h0 + i + q * h1)] = cmul(u[q], __ldg(tw2 + (q - 1) * h1 + i));
    }
    __syncthreads();
    for (int t = threadIdx.x; t < S * (M / RL); t += 256) {
        const int e = t % (M / RL) * RL;
        double2* o = smem + t / (M / RL) * PM;
        double2 u[RL];
#pragma unroll
        for (int q = 0; q < RL; ++q) u[q] = o[P::pos(e + q)];
        butterfly<-1, RL>(u);
#pragma unroll
        for (int q = 0; q < RL; ++q) u[q] = cmul(u[q], __ldg(fh + e + q));
        butterfly<+1, RL>(u);
#pragma unroll
        for (int q = 0; q < RL; ++q) o[P::pos(e + q)] = u[q];
    }
    __syncthreads();
    for (int t = threadIdx.x; t < S * (M / R1); t += 256) {
        const int i = t % h1, blk = t / h1 % R0, sq = t / (M / R1);
        double2* o = smem + sq * PM;
        double2 u[R1];
        u[0] = o[P::pos(blk * h0 + i)];
#pragma unroll
        for (int q = 1; q < R1; ++q) {
            double2 w = __ldg(tw2 + (q - 1) * h1 + i);
            w.y = -w.y;
            u[q] = cmul(o[P::pos(blk * h0 + i + q * h1)], w);
        }
        butterfly<+1, R1>(u);
#pragma unroll
        for (int q = 0; q < R1; ++q) o[P::pos(blk * h0 + i + q * h1)] = u[q];
    }
    __syncthreads();
    for (int t = threadIdx.x; t < V * h0; t += 256) {
        const int v = vfast_out ? t % V : t / h0, i = vfast_out ? t / V : t % h0;
        if (v >= nv) continue;
        double2* p = dst + dbase + (long long)v * a.dst.sv;
#pragma unroll
        for (int s = 0; s < 2; ++s) {
            if (s == 1 && !split) break;
            const double2* o = smem + (s * V + v) * PM;
            double2 u[R0];
            u[0] = o[P::pos(i)];
#pragma unroll
            for (int q = 1; q < R0; ++q) {
                double2 w = __ldg(tw1 + (q - 1) * h0 + i);
                w.y = -w.y;
                u[q] = cmul(o[P::pos(i + q * h0)], w);
            }
            butterfly<+1, R0>(u);
#pragma unroll
            for (int q = 0; q < R0 / 2; ++q) {
                const int k = i + q * h0;
                if (k < m) {
                    double2 r = cscale(cmul(u[q], __ldg(wtab + k)), a.scale);
                    r.y *= cj;
                    __stcs(p + (long long)(split ? 2 * k + s : k) * a.dst.se, r);
                }
            }
        }
    }
}

// Planned convolution lengths: the radices and a launch of each.
struct ChirpEntry {
    int r0, r1, r2, v;
    cudaError_t (*launch)(const double2*, double2*, const FftPassArgs&, int, int, cudaStream_t, int);
};

template <class P>
cudaError_t chirp_launch(const double2* src, double2* dst, const FftPassArgs& a, int ntiles, int sign, cudaStream_t stream, int nz)
{
    const cudaError_t e = allow_shared(fft_chirp_kernel<P>, P::kSmem, P::kSmem);
    if (e != cudaSuccess) return e;
    fft_chirp_kernel<P><<<dim3((a.nvec + P::V - 1) / P::V, ntiles, nz), 256, P::kSmem, stream>>>(src, dst, a, sign);
    return cudaGetLastError();
}

template <int R0, int R1, int R2, int V>
constexpr ChirpEntry chirp_entry()
{
    return {R0, R1, R2, V, chirp_launch<ChirpPlan<R0, R1, R2, V>>};
}

const ChirpEntry kChirps[] = {
    chirp_entry<8, 8, 8, 4>(),    // 512
    chirp_entry<8, 16, 5, 4>(),   // 640
    chirp_entry<8, 8, 16, 2>(),   // 1024
};

// The plan for length n: the smallest M >= 2m - 1.
const ChirpEntry& chirp_for(int n)
{
    const int m = n % 2 ? n : n / 2;
    for (const ChirpEntry& c : kChirps)
        if (c.r0 * c.r1 * c.r2 >= 2 * m - 1) return c;
    return kChirps[sizeof(kChirps) / sizeof(kChirps[0]) - 1];
}

// The largest prime factor that does not go to the chirp pass, for what the other kernels leave: even
// lengths (tables kept) such as 686, direct stages of 7, 11 and 13 measured slower at every length
// from 28 to 448 (N = 308 597 us against 2014); odd ones (table made on the host for each call) such as 343.
int largest_direct_radix(int n) { return n % 2 ? 16 : 5; }

// Whether passes of length n run the two-stage kernel.
bool two_stage(int n)
{
    int ra, rb;
    return fft_two_radices(n, &ra, &rb);
}

int largest_prime(int n)
{
    int big = 1;
    for (int p = 2; p * p <= n; ++p)
        while (n % p == 0) {
            big = p;
            n /= p;
        }
    return std::max(big, n);
}

// The odd factor p of a length n = R p that passes on the matrix kernel, or 0.
int matrix_factor(int n)
{
    int r, p;
    return !two_stage(n) && largest_prime(n) > largest_direct_radix(n) && fft_matrix_radices(n, &r, &p) ? p : 0;
}

}  // namespace

int fft_plan_radices(int n, int* radix, int* ns)
{
    if (n < 1) return 0;
    if (two_stage(n)) {
        fft_two_radices(n, &radix[0], &radix[1]);
        ns[0] = 1;
        ns[1] = radix[0];
        return 2;
    }
    int r[64];
    int cnt = 0, rem = n;
    int p2 = 0;
    while (rem % 2 == 0) {
        rem /= 2;
        ++p2;
    }
    // power-of-two part: as few stages as radix 16 allows, bits spread evenly (8.8.8, 16.8)
    if (p2 > 0) {
        const int st = (p2 + 3) / 4;
        for (int i = 0; i < st; ++i) {
            const int bits = p2 / st + (i < p2 % st ? 1 : 0);
            r[cnt++] = 1 << bits;
        }
    }
    while (rem % 3 == 0) { r[cnt++] = 3; rem /= 3; }
    while (rem % 5 == 0) { r[cnt++] = 5; rem /= 5; }
    for (int p = 7; rem > 1; p += 2) {
        while (rem % p == 0) { r[cnt++] = p; rem /= p; }
    }
    if (cnt == 0) r[cnt++] = 1;
    // A lone direct (O(R^2)) stage would read and write the same HBM vector when the pass
    // is in place; a leading radix-1 stage (a plain copy into shared memory) separates them.
    const bool direct = !(r[0] == 1 || r[0] == 2 || r[0] == 3 || r[0] == 4 || r[0] == 5 || r[0] == 8 || r[0] == 16);
    if (cnt == 1 && direct) {
        r[1] = r[0];
        r[0] = 1;
        cnt = 2;
    }
    if (cnt > kFftMaxStages) return 0;
    int nsv = 1;
    for (int i = 0; i < cnt; ++i) {
        radix[i] = r[i];
        ns[i] = nsv;
        nsv *= r[i];
    }
    return cnt;
}

bool fft_needs_bluestein(int n)
{
    if (matrix_factor(n)) return true;
    return n >= 2 && (n % 2 ? n : n / 2) <= 512 && !two_stage(n) && largest_prime(n) > largest_direct_radix(n);
}

size_t fft_bluestein_elems(int n)
{
    if (const int p = matrix_factor(n)) return fft_matrix_elems(p);
    const ChirpEntry& c = chirp_for(n);
    const int M = c.r0 * c.r1 * c.r2, m = n % 2 ? n : n / 2, h0 = M / c.r0;
    return 2 * (size_t)m + M + (size_t)(c.r0 - 1) * h0 + (size_t)(c.r1 - 1) * (h0 / c.r1);
}

void fft_bluestein_fill(int n, double2* out)
{
    if (const int p = matrix_factor(n)) return fft_matrix_fill(p, out);
    typedef long double ld;
    const ld pi = 3.14159265358979323846264338327950288L;
    const ChirpEntry& c = chirp_for(n);
    const int M = c.r0 * c.r1 * c.r2, m = n % 2 ? n : n / 2, h0 = M / c.r0, h1 = h0 / c.r1;
    // w_j = exp(-pi i j^2 / m), the exponent reduced mod 2m first, and w_j exp(-2 pi i j / (2m))
    std::vector<ld> wr(m), wi(m);
    for (int j = 0; j < m; ++j) {
        const ld ang = pi * (ld)(((long long)j * j) % (2ll * m)) / (ld)m;
        wr[j] = cosl(ang);
        wi[j] = -sinl(ang);
        out[j] = make_double2((double)wr[j], (double)wi[j]);
        const ld both = pi * (ld)(((long long)j * j + j) % (2ll * m)) / (ld)m;
        out[m + j] = make_double2((double)cosl(both), (double)-sinl(both));
    }
    std::vector<ld> cr(M), ci(M);   // exp(-2 pi i t / M)
    for (int t = 0; t < M; ++t) {
        cr[t] = cosl(2 * pi * (ld)t / (ld)M);
        ci[t] = -sinl(2 * pi * (ld)t / (ld)M);
    }
    // the convolution kernel conj(w_d) at d and M - d, its DFT / M in the order the forward stages leave:
    // index k = k0 + R0 (k1 + R1 k2) at k0 h0 + k1 h1 + k2
    std::vector<ld> hr(M, 0), hi(M, 0);
    for (int d = 0; d < m; ++d) {
        hr[d] = wr[d];
        hi[d] = -wi[d];
        if (d > 0) {
            hr[M - d] = wr[d];
            hi[M - d] = -wi[d];
        }
    }
    double2* fh = out + 2 * m;
    for (int k = 0; k < M; ++k) {
        ld sr = 0, si = 0;
        for (int j = 0; j < M; ++j) {
            const int t = (int)(((long long)j * k) % M);
            sr += hr[j] * cr[t] - hi[j] * ci[t];
            si += hr[j] * ci[t] + hi[j] * cr[t];
        }
        const int k0 = k % c.r0, k1 = k / c.r0 % c.r1, k2 = k / (c.r0 * c.r1);
        fh[k0 * h0 + k1 * h1 + k2] = make_double2((double)(sr / M), (double)(si / M));
    }
    double2* tw = fh + M;
    for (int q = 1; q < c.r0; ++q)
        for (int i = 0; i < h0; ++i) *tw++ = make_double2((double)cr[q * i % M], (double)ci[q * i % M]);
    for (int q = 1; q < c.r1; ++q)
        for (int i = 0; i < h1; ++i) *tw++ = make_double2((double)cr[c.r0 * q * i % M], (double)ci[c.r0 * q * i % M]);
}

int fft_tile_vectors(int n)
{
    if (two_stage(n)) return fft_two_vectors(n);
    if (matrix_factor(n)) return 8;
    const size_t two_buffers = 2 * (size_t)8 * padded_len(n) * sizeof(double2);
    return two_buffers > (size_t)110 * 1024 ? 4 : 8;
}

size_t fft_pass_smem_bytes(const FftPassArgs& a)
{
    const int buffers = a.nstages >= 3 ? 2 : (a.nstages == 2 ? 1 : 0);
    return (size_t)buffers * a.kb * padded_len(a.n) * sizeof(double2);
}

cudaError_t fft_pass_launch(const double2* src, double2* dst, const FftPassArgs& a, int ntiles, int sign,
                            cudaStream_t stream, int nz)
{
    if (a.bluestein && fft_needs_bluestein(a.n)) {
        if (matrix_factor(a.n)) return fft_matrix_launch(src, dst, a, ntiles, sign, stream, nz);
        return chirp_for(a.n).launch(src, dst, a, ntiles, sign, stream, nz);
    }
    if (two_stage(a.n)) return fft_two_launch(src, dst, a, ntiles, sign, stream, nz);
    // one butterfly per thread in the widest stage, up to 256 threads
    int widest = 1;
    for (int s = 0; s < a.nstages; ++s) widest = std::max(widest, a.n / a.radix[s]);
    const int nthreads = std::min(256, ((a.kb * widest + 31) / 32) * 32);
    dim3 grid((a.nvec + a.kb - 1) / a.kb, ntiles, nz);
    const size_t smem = fft_pass_smem_bytes(a);
    auto go = [&](auto kern) -> cudaError_t {
        const cudaError_t e = allow_shared(kern, smem, kMaxShared);
        if (e != cudaSuccess) return e;
        kern<<<grid, nthreads, smem, stream>>>(src, dst, a);
        return cudaGetLastError();
    };
    // the kernel indexes two buffers; with a single buffer the second is never used
    return sign < 0 ? go(fft_pass_kernel<-1>) : go(fft_pass_kernel<1>);
}

}  // namespace pfsoft_dev
