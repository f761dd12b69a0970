// Self-test of the bounded device waits. Every wait in the solver kernels (the grid
// barrier of the persistent solvers) gives up after a time limit, records
// FEEC_TIMEOUT and the wait site in the status block, and lets every thread leave, so
// the host gets an error status with the GPU context still usable. This entry point
// exercises that path on purpose and safely, for each kind of wait: one thread waits,
// through the same wait_counter the grid barrier uses, for a counter value that nothing ever
// writes, with a short limit chosen by the caller; a warp gathers a value that nobody publishes, as
// the dataflow solvers do, and a warp waits for a staged copy that nobody starts, as the one-block
// solver does, both with the solvers' own limit (4 s, fixed in their code). Each then returns like a
// solver that gave up.
#include <chrono>

#include "feec_device.cuh"
#include "feec_internal.h"
#include "feec_system.h"
#include "flow_device.cuh"
#include "persistent_common.cuh"

namespace feec {
namespace {

__global__ void unset_flag_wait_kernel(DeviceStatus* st, unsigned long long limit_ns) {
    if (threadIdx.x != 0 || blockIdx.x != 0) return;
    // the counter starts at 0 and no thread increments it: the wait can only run out
    wait_counter(st, 1ull, 77, limit_ns);
}

// A warp gathers a published value whose slot keeps the sentinel; the sum's block leaves by the
// reduction that every dataflow solver leaves by.
__global__ void unpublished_value_kernel(DeviceStatus* st, const double* X, double* part) {
    __shared__ FlowShared sh;
    FlowGather<double> in;
    FlowCols cols;
    for (int u = 0; u < kFlowChunk; u++) {
        cols.c[u] = u == 2 && (threadIdx.x & 31) == 5 ? 0 : -1;     // one slot of one lane
        in.v[u] = 1.0;
        in.g[u] = cols.c[u] >= 0 ? ld_flow(X) : 0.0;
    }
    bool live = true;
    double acc[1] = {in.wait(cols, kFlowChunk, X, 0.0, st, 78, live)}, sum[1];
    unsigned long long epoch = 0;
    if (!flow_reduce<double, 1>(acc, part, st, epoch, 79, live, sh, sum)) return;
    finish(st, FEEC_OK, 1, sum[0], 0.0);       // not reached: live is false
}

}  // namespace
}  // namespace feec

using namespace feec;

namespace {

// One run of kind 0 (with a limit), 1 or 2 (with the solvers' own).
int run_wait(int kind, unsigned long long limit_ns, int* status, int* site, double* elapsed_ms) {
    int dev = 0;
    cudaStream_t lib = nullptr;
    int st = init_device(dev, lib);
    if (st != FEEC_OK) return st;
    DevArena mem;
    mem.stream = lib;
    struct Release { DevArena& m; ~Release() { m.release(); } } rel{mem};
    DeviceStatus* d = nullptr;
    double* slot = nullptr;
    FEEC_TRY(mem.alloc(d, 1));
    FEEC_TRY(mem.alloc(slot, 8));
    FEEC_TRY(cudaMemsetAsync(d, 0, sizeof(DeviceStatus), lib));
    FEEC_TRY(cudaMemsetAsync(slot, 0xFF, 8 * sizeof(double), lib));
    const auto t0 = std::chrono::steady_clock::now();
    if (kind == 2) {
        FEEC_TRY(launch_missing_copy(d, lib));
    } else {
        note_launch();
        if (kind == 0) unset_flag_wait_kernel<<<1, 32, 0, lib>>>(d, limit_ns);
        else unpublished_value_kernel<<<1, 64, 0, lib>>>(d, slot, slot + 4);
        FEEC_TRY(cudaGetLastError());
    }
    DeviceStatus h{};
    FEEC_TRY(cudaMemcpyAsync(&h, d, sizeof(h), cudaMemcpyDeviceToHost, lib));
    FEEC_TRY(cudaStreamSynchronize(lib));
    if (elapsed_ms) *elapsed_ms = std::chrono::duration<double, std::milli>(std::chrono::steady_clock::now() - t0).count();
    if (status) *status = h.status;
    if (site) *site = h.timeout_site;
    return FEEC_OK;
}

}  // namespace

extern "C" int feec_selftest_solver_wait(int kind, int* status, int* site, double* elapsed_ms) {
    if (kind != 1 && kind != 2) return FEEC_BADARG;
    return run_wait(kind, 0, status, site, elapsed_ms);
}

extern "C" int feec_selftest_wait_timeout(double limit_s, int* status, int* site, double* elapsed_ms) {
    if (!(limit_s > 0.0) || limit_s > 10.0) return FEEC_BADARG;
    return run_wait(0, (unsigned long long)(limit_s * 1e9), status, site, elapsed_ms);
}
