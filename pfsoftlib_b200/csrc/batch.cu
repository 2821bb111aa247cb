// Batched SO(3) transforms over many bandwidths (C ABI: pfsoft_batch_*).
//
// A batch plan groups its transforms by bandwidth. One forward execution is
//   per group:  F1 (gamma DFT -> beta-innermost spectrum), F2 (alpha DFT)   [one launch each,
//               gridDim.z = transforms of the group]
//               then one DWT launch over every (order class, transform) of the group (dwt.cu)
// and the inverse runs the mirror image. With PFSOFT_BATCH_SPLIT every group up to B = 256 shares
// one split-precision DWT launch.
// The whole sequence is captured once into a CUDA graph; the device tables of grid and
// coefficient pointers that the kernels read are refreshed before each replay, so one graph
// serves any buffers.

#include <cuda_runtime.h>

#include <algorithm>
#include <cstring>
#include <map>
#include <mutex>
#include <string>
#include <vector>

#include "../../include/pfsoft_b200.h"
#include "common.cuh"
#include "dwt.cuh"
#include "fft.cuh"

using namespace pfsoft_dev;

namespace {

// The split-precision choice per bandwidth (0 that of the rest, 1 split, -1 FP64) and of the rest (0 FP64, 1 the
// faster form, 2 split), read when a PFSOFT_BATCH_SPLIT plan is created.
signed char g_split_choice[513] = {};
int g_split_rest = 1;

// Default: the faster DWT for T transforms of bandwidth B. The FP64 kernels' sums over the series take
// fewer steps than the split kernel's digit products; only without a DFT over beta, whose matrix product
// grows as B^4, and with pairs of transforms to share the split kernel's Wigner tiles, the split kernel
// is ahead from about B = 140 on. Whole plans, split over FP64, iDSOFT / DSOFT: B = 32 (T = 4) 2.0 / 2.5, 64 1.4 /
// 1.6, 128 1.3 / 1.3, 256 1.1 / 1.2; without DFT and T >= 2: 116 1.1, 137 1.0, 166 0.98, 184 0.94, 251
// 0.92, T = 1: 1.1 and more. Up to B = 16, where calls of a few transforms are bound by their launches, the rule
// does not follow the times (FP64 is 5 to 15 us ahead): split plans run there what they always ran, and with
// it the bounded waits whose failure pfsoft_batch_status reports in plans made without a tuning call.
bool split_faster(int B, int T) { return B <= 16 || (B >= 140 && T >= 2 && !dwt_has_dft(2 * B)); }

bool split_wanted(int B, int T)
{
    if (B >= 1 && B <= 512 && g_split_choice[B]) return g_split_choice[B] > 0;
    return g_split_rest == 2 || (g_split_rest == 1 && split_faster(B, T));
}

__global__ void zero_nyquist_batched(double2* const* X, int B)
{
    double2* x = X[blockIdx.z];
    const int N = 2 * B;
    const long long total = (long long)(2 * N - 1) * N;
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < total; i += (long long)gridDim.x * blockDim.x) {
        const long long v = i / N;
        const int k = (int)(i - v * N);
        int row, col;
        if (v < N) {
            row = B;
            col = (int)v;
        } else {
            col = B;
            row = (int)(v - N);
            if (row >= B) ++row;
        }
        x[((size_t)row * N + col) * N + k] = make_double2(0.0, 0.0);
    }
}

int fail(int status, const std::string& msg)
{
    set_last_error(msg.c_str());
    return status;
}

}  // namespace


namespace pfsoft_dev {

// FFT pass of one same-bandwidth group: forward F1 (gamma DFT, grid -> beta-innermost spectrum)
// and F2 (alpha DFT in place), inverse I2 (alpha, in place) and I1 (gamma, spectrum -> grid,
// scaled 1/(4B^2)). grids / ws are device tables with one pointer per transform.
FftPassArgs group_pass_args(int dir, bool first, const BandTables& t, double2** grids, double2** ws)
{
    const long long n = t.N, n2 = n * n;
    FftPassArgs a;
    memset(&a, 0, sizeof(a));
    a.n = t.N;
    a.nvec = t.N;
    a.kb = fft_tile_vectors(t.N);
    a.nstages = fft_plan_radices(t.N, a.radix, a.ns);
    a.twiddle = t.twiddle;
    a.bluestein = t.bluestein;
    a.scale = 1.0;
    if (dir == 0 && first) {          // F1
        a.src = FftStrides{n2, n, 1};
        a.dst = FftStrides{1, n, n2};
        a.srcs = grids;
        a.dsts = ws;
    } else if (dir == 0 || first) {   // F2 / I2, in place
        a.src = a.dst = FftStrides{1, n2, n};
        a.srcs = ws;
        a.dsts = ws;
    } else {                          // I1
        a.src = FftStrides{1, n, n2};
        a.dst = FftStrides{n2, n, 1};
        a.srcs = ws;
        a.dsts = grids;
        a.scale = 1.0 / (4.0 * t.B * t.B);
    }
    return a;
}

cudaError_t zero_nyquist_launch(double2** ws, int B, int T, cudaStream_t s)
{
    const int N = 2 * B;
    const long long total = (long long)(2 * N - 1) * N;
    dim3 grid((unsigned)std::min<long long>((total + 255) / 256, 1024), 1, (unsigned)T);
    zero_nyquist_batched<<<grid, 256, 0, s>>>(ws, B);
    return cudaGetLastError();
}

// The FP64 DWT of a group's T transforms in one launch; ws / coefs are device pointer tables.
// The inverse also zeroes the Nyquist bins.
cudaError_t group_dwt_launch(int dir, const BandTables& t, int T, double2** ws, double2** coefs, cudaStream_t s)
{
    DwtArgs a = dwt_args_for(t);
    a.Xs = ws;
    a.coefs = coefs;
    a.zero_nyquist = dir;
    return dir == 0 ? dwt_forward_launch(nullptr, nullptr, a, T, s) : dwt_inverse_launch(nullptr, nullptr, a, T, s);
}

// Both FFT passes of a group.
cudaError_t group_fft_launch(int dir, const BandTables& t, int T, double2** grids, double2** ws, cudaStream_t s)
{
    const int sign = dir == 0 ? -1 : +1;
    if (fft_plane_supported(t.N, T)) {
        const double scale = dir == 0 ? 1.0 : 1.0 / (4.0 * t.B * t.B);
        return fft_plane_launch(nullptr, nullptr, FftPlaneArgs{t.N, 0, 0, scale, t.twiddle, dir == 0 ? grids : ws, dir == 0 ? ws : grids},
                                sign, s, T);
    }
    cudaError_t e = fft_pass_launch(nullptr, nullptr, group_pass_args(dir, true, t, grids, ws), t.N, sign, s, T);
    return e == cudaSuccess ? fft_pass_launch(nullptr, nullptr, group_pass_args(dir, false, t, grids, ws), t.N, sign, s, T) : e;
}

// One same-bandwidth group of T transforms in direction dir (0 forward, 1 inverse) on stream s;
// d_grids / d_coefs / d_ws are device tables of T pointers.
int launch_group(int dir, const BandTables& t, int T, double2** d_grids, double2** d_coefs, double2** d_ws, cudaStream_t s)
{
    cudaError_t e = dir == 0 ? group_fft_launch(dir, t, T, d_grids, d_ws, s) : group_dwt_launch(dir, t, T, d_ws, d_coefs, s);
    if (e == cudaSuccess)
        e = dir == 0 ? group_dwt_launch(dir, t, T, d_ws, d_coefs, s) : group_fft_launch(dir, t, T, d_grids, d_ws, s);
    if (e != cudaSuccess) return fail(PFSOFT_ECUDA, std::string("group launch: ") + cudaGetErrorString(e));
    return PFSOFT_OK;
}

}  // namespace pfsoft_dev

struct pfsoft_batch {
    struct Group {
        int B = 0, N = 0;
        std::vector<int> members;   // transform indices in the caller's order
        BandTables tables;
        size_t ptr_base = 0;        // offset of this group's entries in the pointer tables
        bool split = false;         // DWT on the split-precision tensor-core kernel
    };
    int count = 0;
    int tpc = 1;
    bool use_graph = true;
    std::vector<Group> groups;
    // device: pointer tables [3][count] (grid, coeffs, workspace) in group order
    double2** d_ptr = nullptr;
    double2** h_ptr = nullptr;   // pinned staging of the same
    DwtGroup* d_groups = nullptr;   // the split groups
    // split-precision DWT (PFSOFT_BATCH_SPLIT): segments of the groups it takes (one per group),
    // their item counts, and the sticky status of its bounded waits
    void* d_split_fwd = nullptr;
    void* d_split_inv = nullptr;
    int n_split_fwd = 0, n_split_inv = 0;
    int n_split_seg = 0;
    int* d_split = nullptr;   // [0] counter, [1] status
    void* ws = nullptr;
    size_t ws_bytes = 0;
    cudaGraphExec_t graph[2] = {nullptr, nullptr};
    cudaEvent_t uploaded = nullptr;   // the last pointer upload has read h_ptr
    std::mutex mu;

    double2** grid_ptrs() const { return d_ptr; }
    double2** coef_ptrs() const { return d_ptr + count; }
    double2** ws_ptrs() const { return d_ptr + 2 * (size_t)count; }
};

namespace {

// Sequence of one direction on stream s (captured into a graph, or run directly).
int enqueue(pfsoft_batch* b, int dir, cudaStream_t s)
{
    typedef pfsoft_batch::Group Group;
    auto T = [](const Group& g) { return (int)g.members.size(); };
    auto fft = [&](const Group& g) {
        return group_fft_launch(dir, g.tables, T(g), b->grid_ptrs() + g.ptr_base, b->ws_ptrs() + g.ptr_base, s);
    };
    cudaError_t e = cudaSuccess;
    if (dir == 0)
        for (const auto& g : b->groups)
            if (e == cudaSuccess) e = fft(g);
    for (const auto& g : b->groups) {
        double2** ws = b->ws_ptrs() + g.ptr_base;
        double2** coefs = b->coef_ptrs() + g.ptr_base;
        if (e == cudaSuccess && !g.split) e = group_dwt_launch(dir, g.tables, T(g), ws, coefs, s);
        if (e == cudaSuccess && g.split && dir == 1) e = zero_nyquist_launch(ws, g.B, T(g), s);
        if (e == cudaSuccess && g.split) e = dwt_split_scales(dir, g.B, T(g), ws, coefs, g.tables.w, s);
    }
    const int n_split = dir == 0 ? b->n_split_fwd : b->n_split_inv;
    if (e == cudaSuccess && n_split > 0) {
        e = cudaMemsetAsync(b->d_split, 0, sizeof(int), s);
        if (e == cudaSuccess)
            e = dwt_split_launch(dir, b->d_groups, dir == 0 ? b->d_split_fwd : b->d_split_inv, b->n_split_seg, n_split,
                                 b->d_split + 1, s);
    }
    if (dir == 1)
        for (const auto& g : b->groups)
            if (e == cudaSuccess) e = fft(g);
    if (e != cudaSuccess) return fail(PFSOFT_ECUDA, std::string("batch launch: ") + cudaGetErrorString(e));
    return PFSOFT_OK;
}

void free_batch(pfsoft_batch* b)
{
    for (auto& g : b->graph)
        if (g) cudaGraphExecDestroy(g);
    if (b->uploaded) cudaEventDestroy(b->uploaded);
    cudaFree(b->d_ptr);
    cudaFreeHost(b->h_ptr);
    cudaFree(b->d_groups);
    cudaFree(b->d_split_fwd);
    cudaFree(b->d_split_inv);
    cudaFree(b->d_split);
    cudaFree(b->ws);
    delete b;
}

}  // namespace

extern "C" {

int pfsoft_batch_create(const int* bandwidths, int count, int transforms_per_cta, int flags, pfsoft_batch** out)
{
    set_last_error("");
    if (!out) return fail(PFSOFT_EINVAL, "null output handle");
    *out = nullptr;
    if (!bandwidths || count < 1) return fail(PFSOFT_EINVAL, "batch needs at least one bandwidth");
    if (transforms_per_cta != 0 && transforms_per_cta != 1 && transforms_per_cta != 2 && transforms_per_cta != 4)
        return fail(PFSOFT_EINVAL, "transforms_per_cta must be 0 (auto), 1, 2 or 4");
    for (int i = 0; i < count; ++i)
        if (bandwidths[i] < 1 || bandwidths[i] > 512) return fail(PFSOFT_EINVAL, "bandwidth must be in [1, 512]");
    pfsoft_batch* b = new pfsoft_batch();
    b->count = count;
    b->use_graph = (flags & 1) == 0;
    std::map<int, std::vector<int> > by_b;
    for (int i = 0; i < count; ++i) by_b[bandwidths[i]].push_back(i);
    size_t base = 0, ws_total = 0;
    std::vector<size_t> ws_off(count);
    for (auto& kv : by_b) {
        pfsoft_batch::Group g;
        g.B = kv.first;
        g.N = 2 * kv.first;
        g.members = kv.second;
        g.ptr_base = base;
        base += g.members.size();
        g.split = (flags & PFSOFT_BATCH_SPLIT) && dwt_split_supported(g.B) && split_wanted(g.B, (int)g.members.size());
        for (int t : g.members) {
            ws_off[t] = ws_total;
            ws_total += ((((size_t)g.N * g.N * g.N + (g.split ? dwt_split_aux_elems(g.B) : 0)) * sizeof(double2) + kFftSyncBytes
                          + 255) & ~(size_t)255);   // each workspace 256-byte aligned
        }
        int rc = tables_for(g.B, &g.tables, g.split ? kSplitTables : kSeriesTables);
        if (rc) {
            free_batch(b);
            return rc;
        }
        b->groups.push_back(g);
    }
    // reported as asked for (0: 4 up to B = 64, 2 above); the DWT kernels take one transform per CTA
    b->tpc = transforms_per_cta ? transforms_per_cta : (std::min(by_b.rbegin()->first, 128) <= 64 ? 4 : 2);
    std::vector<int> split_group, split_B, split_T;   // the split groups: index in d_groups, B, T
    for (const auto& g : b->groups) {
        if (!g.split) continue;
        split_group.push_back((int)split_group.size());
        split_B.push_back(g.B);
        split_T.push_back((int)g.members.size());
    }
    std::vector<unsigned char> split_f, split_i;   // forward / inverse segments
    const int n_split_f = dwt_split_segments(0, split_group, split_B, split_T, split_f);
    const int n_split_i = dwt_split_segments(1, split_group, split_B, split_T, split_i);
    cudaError_t e = cudaMalloc(&b->d_ptr, 3 * (size_t)count * sizeof(double2*));
    if (e == cudaSuccess) e = cudaHostAlloc(&b->h_ptr, 3 * (size_t)count * sizeof(double2*), cudaHostAllocDefault);
    if (e == cudaSuccess) e = cudaMalloc(&b->ws, ws_total);
    if (e == cudaSuccess) e = cudaEventCreateWithFlags(&b->uploaded, cudaEventDisableTiming);
    if (e == cudaSuccess) e = cudaMalloc(&b->d_split, 2 * sizeof(int));
    if (e == cudaSuccess && n_split_f > 0) e = cudaMalloc(&b->d_split_fwd, split_f.size());
    if (e == cudaSuccess && n_split_i > 0) e = cudaMalloc(&b->d_split_inv, split_i.size());
    if (e != cudaSuccess) {
        free_batch(b);
        return fail(PFSOFT_ENOMEM, std::string("batch allocation: ") + cudaGetErrorString(e));
    }
    b->n_split_fwd = n_split_f;
    b->n_split_inv = n_split_i;
    b->n_split_seg = (int)split_group.size();
    e = cudaMemset(b->d_split, 0, 2 * sizeof(int));
    if (e == cudaSuccess && (n_split_f > 0 || n_split_i > 0)) e = dwt_split_prepare();
    if (e == cudaSuccess && n_split_f > 0) e = cudaMemcpy(b->d_split_fwd, split_f.data(), split_f.size(), cudaMemcpyHostToDevice);
    if (e == cudaSuccess && n_split_i > 0) e = cudaMemcpy(b->d_split_inv, split_i.data(), split_i.size(), cudaMemcpyHostToDevice);
    if (e != cudaSuccess) {
        free_batch(b);
        return fail(PFSOFT_ECUDA, std::string("batch setup: ") + cudaGetErrorString(e));
    }
    b->ws_bytes = ws_total;
    std::memset(b->h_ptr, 0, 3 * (size_t)count * sizeof(double2*));
    for (const auto& g : b->groups)
        for (size_t i = 0; i < g.members.size(); ++i)
            b->h_ptr[2 * (size_t)count + g.ptr_base + i] =
                reinterpret_cast<double2*>(static_cast<char*>(b->ws) + ws_off[g.members[i]]);
    // group descriptors of the split-precision DWT (pointer tables inside the device array)
    std::vector<DwtGroup> dg;
    for (const auto& g : b->groups) {
        if (!g.split) continue;
        DwtGroup d;
        d.B = g.B;
        d.N = g.N;
        d.T = (int)g.members.size();
        d.cosb = g.tables.cosb;
        d.w = g.tables.w;
        d.normf = g.tables.normf;
        d.pw_sin = g.tables.pw_sin;
        d.pw_cos = g.tables.pw_cos;
        d.rc_cf = g.tables.rc_cf;
        d.rc_f1 = g.tables.rc_f1;
        d.X = b->ws_ptrs() + g.ptr_base;
        d.coeffs = b->coef_ptrs() + g.ptr_base;
        dg.push_back(d);
    }
    if (!dg.empty()) {
        e = cudaMalloc(&b->d_groups, dg.size() * sizeof(DwtGroup));
        if (e == cudaSuccess) e = cudaMemcpy(b->d_groups, dg.data(), dg.size() * sizeof(DwtGroup), cudaMemcpyHostToDevice);
    }
    if (e == cudaSuccess) e = cudaMemcpy(b->d_ptr, b->h_ptr, 3 * (size_t)count * sizeof(double2*), cudaMemcpyHostToDevice);
    if (e != cudaSuccess) {
        free_batch(b);
        return fail(PFSOFT_ECUDA, std::string("batch setup: ") + cudaGetErrorString(e));
    }
    *out = b;
    return PFSOFT_OK;
}

int pfsoft_batch_destroy(pfsoft_batch* b)
{
    if (!b) return PFSOFT_OK;
    cudaDeviceSynchronize();
    free_batch(b);
    return PFSOFT_OK;
}

size_t pfsoft_batch_workspace_bytes(const pfsoft_batch* b) { return b ? b->ws_bytes : 0; }

int pfsoft_batch_transforms_per_cta(const pfsoft_batch* b) { return b ? b->tpc : 0; }

int pfsoft_split_supported(int B) { return dwt_split_supported(B) ? 1 : 0; }

int pfsoft_tune_split_bandwidth(int B, int use_split)
{
    if (B > 512) return fail(PFSOFT_EINVAL, "bandwidth must be at most 512");
    if (B <= 0) {
        g_split_rest = use_split == 2 ? 2 : use_split != 0;
        for (auto& v : g_split_choice) v = 0;
    } else {
        g_split_choice[B] = use_split ? 1 : -1;
    }
    return PFSOFT_OK;
}

int pfsoft_test_split_wait_ns(unsigned long long wait_ns)
{
    dwt_split_set_fail_ns(wait_ns);
    return PFSOFT_OK;
}

int pfsoft_batch_status(pfsoft_batch* b)
{
    if (!b) return fail(PFSOFT_EINVAL, "null batch");
    int st[2] = {0, 0};
    cudaError_t e = cudaDeviceSynchronize();
    if (e == cudaSuccess) e = cudaMemcpy(st, b->d_split, sizeof(st), cudaMemcpyDeviceToHost);
    if (e != cudaSuccess) return fail(PFSOFT_ECUDA, std::string("batch status: ") + cudaGetErrorString(e));
    if (st[1]) return fail(PFSOFT_ETIMEOUT, "a bounded wait in the split-precision DWT ran out");
    return PFSOFT_OK;
}

static int batch_run(pfsoft_batch* b, int dir, const double* const* in, double* const* out, void* stream)
{
    set_last_error("");
    if (!b) return fail(PFSOFT_EINVAL, "null batch");
    if (!in || !out) return fail(PFSOFT_EINVAL, "null pointer table");
    std::lock_guard<std::mutex> lk(b->mu);
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    // the previous call's upload must have read the staging table before it is rewritten
    cudaError_t e = cudaEventSynchronize(b->uploaded);
    if (e != cudaSuccess) return fail(PFSOFT_ECUDA, std::string("pointer upload wait: ") + cudaGetErrorString(e));
    // pointer tables in group order (forward: in = grids, out = coeffs; inverse: swapped)
    for (const auto& g : b->groups)
        for (size_t i = 0; i < g.members.size(); ++i) {
            const int t = g.members[i];
            if (!in[t] || !out[t]) return fail(PFSOFT_EINVAL, "null buffer in the pointer table");
            double2* grid = reinterpret_cast<double2*>(const_cast<double*>(dir == 0 ? in[t] : out[t]));
            double2* coef = reinterpret_cast<double2*>(const_cast<double*>(dir == 0 ? out[t] : in[t]));
            b->h_ptr[g.ptr_base + i] = grid;
            b->h_ptr[b->count + g.ptr_base + i] = coef;
        }
    e = cudaMemcpyAsync(b->d_ptr, b->h_ptr, 2 * (size_t)b->count * sizeof(double2*), cudaMemcpyHostToDevice, s);
    if (e == cudaSuccess) e = cudaEventRecord(b->uploaded, s);
    if (e != cudaSuccess) return fail(PFSOFT_ECUDA, std::string("pointer upload: ") + cudaGetErrorString(e));
    if (!b->use_graph) return enqueue(b, dir, s);
    if (!b->graph[dir]) {
        cudaStream_t cs;
        e = cudaStreamCreateWithFlags(&cs, cudaStreamNonBlocking);
        if (e != cudaSuccess) return fail(PFSOFT_ECUDA, "capture stream");
        cudaGraph_t graph = nullptr;
        e = cudaStreamBeginCapture(cs, cudaStreamCaptureModeThreadLocal);
        int rc = PFSOFT_OK;
        if (e == cudaSuccess) rc = enqueue(b, dir, cs);
        cudaError_t e2 = cudaStreamEndCapture(cs, &graph);
        if (e == cudaSuccess) e = e2;
        if (e == cudaSuccess && rc == PFSOFT_OK) e = cudaGraphInstantiate(&b->graph[dir], graph, 0);
        if (graph) cudaGraphDestroy(graph);
        cudaStreamDestroy(cs);
        if (rc != PFSOFT_OK) return rc;
        if (e != cudaSuccess) return fail(PFSOFT_ECUDA, std::string("graph capture: ") + cudaGetErrorString(e));
    }
    e = cudaGraphLaunch(b->graph[dir], s);
    if (e != cudaSuccess) return fail(PFSOFT_ECUDA, std::string("graph launch: ") + cudaGetErrorString(e));
    return PFSOFT_OK;
}

int pfsoft_batch_dsoft(pfsoft_batch* b, const double* const* d_grids, double* const* d_coeffs, void* stream)
{
    return batch_run(b, 0, d_grids, d_coeffs, stream);
}

int pfsoft_batch_idsoft(pfsoft_batch* b, const double* const* d_coeffs, double* const* d_grids, void* stream)
{
    return batch_run(b, 1, d_coeffs, d_grids, stream);
}

}  // extern "C"
