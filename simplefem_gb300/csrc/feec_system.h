// The device-resident system object and small host helpers shared by the
// C ABI translation units (capi.cu, batched.cu).
#pragma once

#include <cstddef>
#include <vector>

#include <cuda_runtime.h>

#include "feec_batched.h"
#include "feec_internal.h"

namespace feec {

inline int cuda_status(cudaError_t e) {
    if (e == cudaSuccess) return FEEC_OK;
    if (e == cudaErrorMemoryAllocation) return FEEC_OOM;
    return FEEC_CUDA_ERROR;
}

// Stream-ordered device allocations owned by one object.
struct DevArena {
    std::vector<void*> ptrs;
    size_t bytes = 0;
    cudaStream_t stream = nullptr;
    template <typename T>
    cudaError_t alloc(T*& p, size_t count) {
        p = nullptr;
        if (count == 0) count = 1;
        void* q = nullptr;
        cudaError_t e = cudaMallocAsync(&q, count * sizeof(T), stream);
        if (e != cudaSuccess) return e;
        ptrs.push_back(q);
        bytes += count * sizeof(T);
        p = (T*)q;
        return cudaSuccess;
    }
    void release() {
        for (void* p : ptrs) cudaFreeAsync(p, stream);
        ptrs.clear();
        bytes = 0;
    }
};

#define FEEC_TRY(expr)                                        \
    do {                                                      \
        cudaError_t _e = (expr);                              \
        if (_e != cudaSuccess) return ::feec::cuda_status(_e); \
    } while (0)

int init_device(int& dev, cudaStream_t& stream);

// While alive, routes a system's work to its creation ("home") stream, after the
// stream of the current call has drained; used for one-time set-up whose
// allocations outlive the call (their frees are ordered on the home stream).
struct HomeStreamScope;

// A SELL-32 copy of a system's matrix (see SellView).
struct SellData {
    DevArena mem;
    bool ready = false;
    int nslices = 0, ncolors = 0;
    int* slice_row0 = nullptr; int* slice_nrow = nullptr; int4* slice_len = nullptr; long long* slice_off = nullptr;
    int* color_slice = nullptr; int* ci = nullptr; float* val32 = nullptr; double* val64 = nullptr;
    int* ident = nullptr;
    long long entries = 0;
};

// The multicolor layout cut into row slices for the dataflow solvers (kernels_flow.cu).
struct FlowData {
    DevArena mem;
    bool ready = false;
    int nslices = 0;
    long long units = 0;                 // 32-entry columns over all slices
    int4* meta = nullptr; int* ci = nullptr; double* val64 = nullptr; float* val32 = nullptr;
    double* pub[4] = {nullptr, nullptr, nullptr, nullptr};   // published vectors (n values of either precision)
    // plain CG (kernels_flow_cg.cu): rows in its own order, work vectors in that order
    int longest = 0;                     // entries per lane of the longest slice
    int* perm = nullptr; int* iperm = nullptr;
    double* own[5] = {nullptr, nullptr, nullptr, nullptr, nullptr};
};

// D's published vectors. Large ones start at 2 MB boundaries: gathers all over a vector that lies
// across one page more cost 1 to 3 % (3D P2 refined 5 times, two sweeps, 170 iterations: 16.18 ms at
// boundaries, 16.29 to 16.65 by where the allocator had put them).
inline cudaError_t alloc_published(FlowData& D, int vectors, int n) {
    constexpr size_t kPage = 2 << 20;
    const size_t bytes = sizeof(double) * (size_t)n;
    if (bytes < kPage / 2) {
        cudaError_t e = cudaSuccess;
        for (int k = 0; k < vectors && e == cudaSuccess; k++) e = D.mem.alloc(D.pub[k], (size_t)n);
        return e;
    }
    const size_t stride = (bytes + kPage - 1) / kPage * kPage;
    char* raw = nullptr;
    const cudaError_t e = D.mem.alloc(raw, stride * (size_t)vectors + kPage);
    if (e != cudaSuccess) return e;
    char* const first = reinterpret_cast<char*>((reinterpret_cast<size_t>(raw) + kPage - 1) / kPage * kPage);
    for (int k = 0; k < vectors; k++) D.pub[k] = reinterpret_cast<double*>(first + stride * (size_t)k);
    return cudaSuccess;
}

// Slices (kernels_slices.cu): the rows of colors ranges[c] .. ranges[c + 1] of a split layout, or a
// matrix's rows sorted by length within windows of kSortWindow (perm, iperm). They set D's slices,
// units and longest part; scratch and tables are allocated on st.
constexpr int kSortWindow = 2048;
int cut_colors(FlowData& D, cudaStream_t st, int sms, const std::vector<int>& ranges, const int* rp, const int* lsplit,
               const int* usplit);
int cut_natural(FlowData& D, cudaStream_t st, int sms, int n, const int* rp);

struct SmallData;   // one-block solver's slices and sweep schedules (kernels_small.cu)

}  // namespace feec

struct feec_system {
    int dev = 0;
    int n = 0;
    int nnz = 0;
    cudaStream_t stream = nullptr;         // stream of the current call
    cudaStream_t home_stream = nullptr;    // stream given at creation: owns every persistent allocation
    feec::DevArena mem;      // matrix + layouts
    feec::DevArena work;     // Krylov workspace
    int* A = nullptr; int* C = nullptr; double* V = nullptr;   // original CSR
    float* V32 = nullptr;                                        // FP32 copy for mixed CG
    int lanes = 4;
    // preconditioner layout (valid if prepared >= 0)
    int prepared = -1;
    int* perm = nullptr; int* iperm = nullptr;
    int* rp = nullptr; int* ci = nullptr; double* val = nullptr; float* val32 = nullptr;
    int* lsplit = nullptr; int* usplit = nullptr;
    double* diag = nullptr; float* diag32 = nullptr;
    double* wd = nullptr; double* sd = nullptr; float* wd32 = nullptr; float* sd32 = nullptr;
    int nf = 0; int* fptr = nullptr;
    int nbw = 0; int* bptr = nullptr; int* brows = nullptr;
    int* fsplit = nullptr; int* bsplit = nullptr;   // multicolor: end of each phase's long rows
    double omega = 1.0;
    int num_levels = 0;
    // workspace (FP64 permuted vectors + FP32 inner vectors)
    bool work_ready = false;
    double *x = nullptr, *r = nullptr, *d = nullptr, *z = nullptr, *m = nullptr, *q = nullptr, *b = nullptr;
    double* w = nullptr;               // Eisenstat solvers only: auxiliary + technical
    float* w32 = nullptr;              // ... FP32 copy for the mixed-precision inner solves
    feec::SmallData* small = nullptr;  // one-block solver, built on its first solve
    // MIXED on the whole GPU, per method slot (0: plain CG, 1: preconditioned): 0 = not yet
    // measured, 1 = FP32 inner iterations, 2 = FP64; device ms per decade of residual fall
    int mixed_pick[2] = {0, 0};
    double mixed_rate[2][2] = {{0.0, 0.0}, {0.0, 0.0}};
    int zero_diag_rows = 0;            // rows with D == 0 in the prepared layout (the sweeps skip them)
    double* precon = nullptr;          // diagonal preconditioner of FEEC_METHOD_DIAGONAL (original numbering)
    float *x32 = nullptr, *r32 = nullptr, *d32 = nullptr, *z32 = nullptr, *m32 = nullptr, *q32 = nullptr, *b32 = nullptr;
    double* partials = nullptr;
    double* scal = nullptr;   // device scalars
    feec::DeviceStatus* st = nullptr;
    int max_blocks = 0;
    int max_phase_rows = 0;     // largest sweep phase (rows)
    int user_blocks = 0;        // launch-shape overrides (0 = automatic)
    int user_lanes = 0;
    cudaEvent_t ev0 = nullptr, ev1 = nullptr;
    // SELL-32 layouts: [0] natural row order (SpMV, batched plain CG), [1] Rainbow order
    feec::SellData sell[2];
    feec::FlowData flow;               // multicolor layout
    std::vector<int> color_ranges;     // rows of each color, host copy of fptr (multicolor layouts)
    feec::FlowData flow_cg;            // natural layout, plain CG
    // batched-engine launch choice made by the autotuner, per [method][mode] (0 = not tuned)
    int tuned_k[3][3] = {};
    int tuned_threads[3][3] = {};
    int tuned_blocks[3][3] = {};       // blocks per team: 1 = block team, 2..16 = cluster team
    double tuned_rate[3][3] = {};
};

namespace feec {
// Doubles of partial sums per block of a dataflow solver (two sets of four).
constexpr size_t kFlowPartials = 8;
// Dataflow solvers over the Rainbow layout (kernels_flow.cu): flow_build prepares the slices
// and values of one precision; the launchers enqueue one solve. feec_status results.
int flow_build(feec_system* s, bool f32);
int launch_flow_eisenstat(feec_system* s, const PcgArgs<double>& a, LaunchShape& shape);
int launch_flow_eisenstat(feec_system* s, const PcgArgs<float>& a, LaunchShape& shape);
int launch_flow_pcg(feec_system* s, const PcgArgs<double>& a, LaunchShape& shape);
// Fills slices (columns where ci is not null, values of either precision) from a split layout.
cudaError_t flow_fill(int nslices, const int4* meta, const int* rp, const int* lsplit, const int* usplit, const int* ci_in,
                      const double* val_in, int* ci, double* val64, float* val32, cudaStream_t st);
// One-block FP64 SSOR / multicolor SSOR PCG for small systems (kernels_small.cu), reference rule.
bool small_pcg_fits(const feec_system* s);
int small_pcg_prepare(feec_system* s);
int launch_small_pcg(feec_system* s, const PcgArgs<double>& a, LaunchShape& shape);
void small_release(feec_system* s);
cudaError_t launch_missing_copy(DeviceStatus* st, cudaStream_t s);   // self-test of the staging wait
size_t small_bytes(const feec_system* s);
// Natural-order slices of a matrix (kernels_flow_cg.cu), and the form that a solver over them runs
// in: every vector in registers, vectors in memory with the gathered one published, or (neither) too
// large for publishing to pay.
constexpr int kFlowPublishedRows = 80000, kFlowPublishedEntries = 8000000;   // measured in kernels_flow_cg.cu
struct FlowForm {
    int blocks, threads;
    bool registers, published;
};
int flow_natural_build(FlowData& D, cudaStream_t st, int dev, int n, const int* A, const int* C, const double* V, bool f32);
FlowForm flow_natural_form(const FlowData& D, int n, int sms);
cudaError_t flow_permute(int n, const int* perm, const double* src, double* dst, bool back, cudaStream_t st);
// Plain CG (kernels_flow_cg.cu).
int flow_cg_build(feec_system* s, bool f32);
int launch_flow_cg(feec_system* s, const CgArgs<double>& a, LaunchShape& shape);
int launch_flow_cg(feec_system* s, const CgArgs<float>& a, LaunchShape& shape);

struct HomeStreamScope {
    feec_system* s;
    cudaStream_t saved;
    explicit HomeStreamScope(feec_system* sys) : s(sys), saved(sys->stream) {
        if (saved != s->home_stream) {
            cudaStreamSynchronize(saved);
            s->stream = s->home_stream;
        }
    }
    ~HomeStreamScope() {
        if (saved != s->home_stream) {
            cudaStreamSynchronize(s->home_stream);
            s->stream = saved;
        }
    }
};
}  // namespace feec
