// Plain CG (ConjugateGradientSolverCSR, solver/sparsesolver.cpp:26-201) with one grid-wide sum
// per iteration, one cooperative launch per solve.
//
// The barrier-phase kernel (cg_persistent) spends three grid barriers and two block-wide FP64
// reductions on an iteration: 12 us on 2D P1 refined 6 times (N = 4,225), where the product
// itself is 1 us. Here the direction d is published row by row and gathered as it arrives
// (flow_device.cuh), and the sum that gives alpha also gives beta: with r.r, d.q, r.q and q.q
// of the same r, alpha = r.r / d.q and r'.r' = r.r - 2 alpha r.q + alpha^2 q.q, the square of
// r' = r - alpha q expanded. The next iteration sums r'.r' itself, for its alpha and for the
// stopping rule, so the expansion's rounding (a few units of r.r in r'.r') only enters beta; a solve that ends
// at the iteration cap sums its last residual once more for the reported norm.
//
// Rows are cut into slices as for the multicolor solvers, rows of equal length next to each
// other (sorted within windows of kSortWindow, so that gathers stay local). When every warp
// has at most one slice of at most kFlowChunk entries per lane, the matrix, x, r, d and q stay
// in registers for the whole solve (kCgRegisters). Measured against cg_persistent, FP64 us per
// iteration: 2D P1 refined 6 times (4,225 rows) 12.1 -> 4.6, 8 times (66,049) 16.5 -> 6.9; 3D P2
// refined 4 times (35,937) 17.9 -> 10.0; 3D P1 refined 6 times (274,625) 28.4 -> 20.3, 7 times
// (2,146,689) 130 -> 102.
#include <algorithm>
#include <cmath>
#include <cstdio>

#include "flow_device.cuh"
#include "feec_system.h"
#include "persistent_common.cuh"

namespace feec {
namespace {

template <typename T>
struct FlowCgArgs {
    int n, nslices;
    const int4* meta; const int* ci; const T* val;
    const T* b;
    T *x, *r, *d, *q;
    T* pub[2];
    double tol2;
    int max_iter, print_modulo;
    double print_tol;
    double* partials;
    DeviceStatus* st;
};

struct CgControl {
    double alpha, beta;
    int status;          // -1: go on
};

// Control of one iteration, from the sums [r.r, d.q, r.q, q.q], by warp 0 of every block. The
// two divisions run in two lanes at once: a division is some ten dependent FP64 operations of
// 64 cycles each.
__device__ __forceinline__ void cg_control(const double (&tot)[4], int K, int n, double tol2, int print_modulo,
                                           double print_tol, CgControl& c) {
    const int lane = threadIdx.x & 31;
    const double rr = tot[0], dq = tot[1];
    const double div = (lane == 0 ? rr : 1.0) / (lane == 0 ? dq : rr);      // alpha, 1 / r.r
    const double inv = __shfl_sync(0xffffffffu, div, 1);
    if (lane == 0) {
        int status = -1;
        if (print_modulo > 0 && K % print_modulo == 0 && blockIdx.x == 0)
            printf("(%d/%d)   INTERIM: Residual norm is %.9le < %.9le\n", K, n, sqrt(rr), print_tol);
        if (abs_below(rr, tol2)) status = FEEC_OK;                                                          // :116-119
        else if (!isfinite(rr) || below_zero(rr) || !isfinite(dq) || below_zero(dq)) status = FEEC_BREAKDOWN;   // :142-151
        else if (energy_small(dq)) status = FEEC_SMALL_ENERGY;                                             // :153-157
        c.status = status;
        c.alpha = div;
        c.beta = fma(div, fma(div, tot[3], -2.0 * tot[2]), rr) * inv;                                      // :175-183
    }
}

// kCgRegisters as above. Otherwise the vectors are in memory: up to kFlowPublishedRows rows
// and kFlowPublishedEntries entries d is published (kCgPublished; 9.2 us per iteration against 10.8 on
// 60,000 rows of 3D P1, equal at 100,000; a solve of 44 iterations, 201 entries per row, 20,000 rows 1.19
// ms here, 40,000 rows 1.87 against 1.71, 80,000 rows 3.53 against 2.67); above, publishing costs a
// sentinel store per row and gathers that skip L1, and a second grid barrier before the product costs
// less (kCgBarrier; compiled for 64 registers, it spills 128 bytes a thread). There the product is bound by
// the FP64 rate (a warp's FP64 instruction takes an SM 19 - 20 cycles: 78 us of the 102 on 3D P1
// refined 7 times) and wants 32 warps with 4 entries in flight each: 102 us against 111 for 16
// warps with 8, 107 for 24 with 4, 125 for 32 with 2, and 130 for cg_persistent.
enum { kCgPublished = 0, kCgRegisters = 1, kCgBarrier = 2 };
constexpr int kCgBarrierThreads = 1024;
constexpr int kCgBarrierChunk = 4;

template <typename T, int MODE>
__global__ void __launch_bounds__(MODE == kCgBarrier ? kCgBarrierThreads : kFlowThreads, 1) flow_cg(FlowCgArgs<T> a) {
    constexpr bool REG = MODE == kCgRegisters;
    using AT = AccT<T>;
    using Acc = typename AT::type;
    __shared__ FlowShared sh;
    __shared__ CgControl ctl;
    FlowWarp w;
    w.init(a.meta, a.nslices);
    const int lane = w.lane;
    unsigned long long epoch = 0;
    bool live = true;
    DeviceStatus* st = a.st;
    int K = 0, status = FEEC_MAXITER;
    double tot[4] = {0.0, 0.0, 0.0, 0.0};

    // One-slice state (REG)
    FlowSlice s0{};
    FlowRow row0{0, false};
    FlowCols cols0;
    T v0[kFlowChunk], x0 = T(0), r0 = T(0), d0 = T(0), q0 = T(0);

    // restart (:76-104): r = b - A x, d = r
    if constexpr (REG) {
        s0 = flow_slice(w.raw(0));
        row0 = flow_row(s0, lane);
        cols0.load(a.ci, s0.off, s0.len_u, lane);
        #pragma unroll
        for (int u = 0; u < kFlowChunk; u++) v0[u] = u < s0.len_u ? __ldg(a.val + s0.off + 32 * u + lane) : T(0);
        T acc = T(0);
        if (row0.own) acc = __ldg(&a.b[row0.i]);
        acc = direct_minus<T>(a.ci, a.val, s0.off, s0.len_u, lane, a.x, acc);
        acc = row_sum<T>(acc, s0.shift);
        // every lane of a row carries the row's state
        if ((lane >> s0.shift) < s0.nrow) { r0 = d0 = acc; x0 = a.x[row0.i]; }
    } else {
        for (int j = 0; j < w.mine; j++) {
            const FlowSlice s = flow_slice(w.raw(j));
            const FlowRow row = flow_row(s, lane);
            T acc = row.own ? __ldg(&a.b[row.i]) : T(0);
            acc = direct_minus<T>(a.ci, a.val, s.off, s.len_u, lane, a.x, acc);
            acc = row_sum<T>(acc, s.shift);
            if (row.own) { a.r[row.i] = acc; a.d[row.i] = acc; }
        }
        // the row loop below is not cut into slices: other threads read these rows
        if (MODE == kCgBarrier && !grid_barrier(st, epoch, 95)) return;
    }
    T alpha = T(0), beta = T(0);
    for (;;) {
        T* const pub = a.pub[K & 1];
        T* const old = a.pub[(K & 1) ^ 1];
        Acc sums[4] = {AT::zero(), AT::zero(), AT::zero(), AT::zero()};
        if constexpr (REG) {
            if (row0.own) {
                st_flow(pub + row0.i, d0);
                reset_flow(old + row0.i);
            }
            if (w.mine > 0) {
                // the cols and values stay in registers: only the gathers move
                FlowGather<T> in;
                #pragma unroll
                for (int u = 0; u < kFlowChunk; u++) {
                    in.g[u] = T(0);
                    if (cols0.c[u] >= 0) in.g[u] = ld_flow(pub + cols0.c[u]);
                    in.v[u] = v0[u];
                }
                T acc = in.wait(cols0, s0.len_u, pub, T(0), st, 90, live);
                acc = row_sum<T>(acc, s0.shift);
                q0 = -acc;
            }
            // the four sums of a row on four of its lanes, or two each on two, before the warp adds
            // lanes: 4 FP64 operations instead of 10 (6 for two lanes per row)
            const int t = lane & ((1 << s0.shift) - 1);
            const bool row = (lane >> s0.shift) < s0.nrow;
            if (s0.shift >= 2) {
                Acc k = AT::zero();
                if (row && t < 4) k = acc_product(k, t == 1 ? d0 : t == 3 ? q0 : r0, t == 0 ? r0 : q0);
                for (int off = 4; off < 32; off <<= 1) k = AT::merge(k, AT::shfl_xor(k, off));
                if (lane < 4) sh.warp_sum[threadIdx.x >> 5][lane] = AT::value(k);
            } else if (s0.shift == 1) {
                Acc k0 = AT::zero(), k1 = AT::zero();
                if (row) {
                    k0 = acc_product(k0, r0, t ? q0 : r0);      // r.r | r.q
                    k1 = acc_product(k1, t ? q0 : d0, q0);      // d.q | q.q
                }
                const bool hi = lane & 16;
                Acc k = AT::merge(hi ? k1 : k0, AT::shfl_xor(hi ? k0 : k1, 16));
                for (int off = 2; off < 16; off <<= 1) k = AT::merge(k, AT::shfl_xor(k, off));
                if ((lane & 14) == 0) sh.warp_sum[threadIdx.x >> 5][2 * t + (hi ? 1 : 0)] = AT::value(k);
            } else {
                if (row) {
                    sums[0] = acc_product(sums[0], r0, r0);
                    sums[1] = acc_product(sums[1], d0, q0);
                    sums[2] = acc_product(sums[2], r0, q0);
                    sums[3] = acc_product(sums[3], q0, q0);
                }
                flow_warp_sums<T, 4>(sums, sh);
            }
            // one call for all warps: those of a block may have taken different branches above
            if (!flow_reduce_warps<4>(a.partials + (K & 1) * 4 * gridDim.x, st, epoch, 92, live, sh, tot)) return;
        } else {
            // x += alpha d, r -= alpha q, d = r + beta d of the last iteration (:158-183)
            if constexpr (MODE == kCgPublished) {
                for (int j = 0; j < w.mine; j++) {
                    const FlowSlice s = flow_slice(w.raw(j));
                    const FlowRow row = flow_row(s, lane);
                    if (row.own) {
                        const int i = row.i;
                        T d = a.d[i], r = a.r[i];
                        if (K > 0) {
                            a.x[i] = fma(alpha, d, a.x[i]);
                            r = fma(-alpha, a.q[i], r);
                            a.r[i] = r;
                            d = fma(beta, d, r);
                            a.d[i] = d;
                        }
                        st_flow(pub + i, d);
                        reset_flow(old + i);
                        sums[0] = acc_product(sums[0], r, r);
                    }
                }
            } else {
                const int threads = gridDim.x * blockDim.x;
                #pragma unroll 4
                for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < a.n; i += threads) {
                    T d = a.d[i], r = a.r[i];
                    if (K > 0) {
                        a.x[i] = fma(alpha, d, a.x[i]);
                        r = fma(-alpha, a.q[i], r);
                        a.r[i] = r;
                        d = fma(beta, d, r);
                        a.d[i] = d;
                    }
                    sums[0] = acc_product(sums[0], r, r);
                }
            }
            if constexpr (MODE == kCgPublished) {
            flow_sweep<kFlowU, false>(w, a.ci, [&](const FlowSlice& s, FlowCols& cols, long long noff, int nlen) {
                const FlowRow row = flow_row(s, lane);
                FlowGather<T> in;
                in.begin(a.ci, a.val, s.off, s.len_u, cols, noff, nlen, lane, pub);
                T d = T(0), r = T(0);
                if (row.own) { d = a.d[row.i]; r = a.r[row.i]; }
                T acc = in.finish(a.ci, a.val, s.off, s.len_u, cols, noff, nlen, lane, pub, T(0), st, 91, live);
                acc = row_sum<T>(acc, s.shift);
                if (row.own) {
                    const T q = -acc;
                    a.q[row.i] = q;
                    sums[1] = acc_product(sums[1], d, q);
                    sums[2] = acc_product(sums[2], r, q);
                    sums[3] = acc_product(sums[3], q, q);
                }
            });
            } else {
                if (!grid_barrier(st, epoch, 93)) return;
                // d does not change during this product: plain gathers, and the next entries
                // requested with the gathers of the current ones
                int4 raw = w.raw(0);
                for (int j = 0; j < w.mine; j++) {
                    const FlowSlice s = flow_slice(raw);
                    raw = w.raw(j + 1);
                    const FlowRow row = flow_row(s, lane);
                    const int* cp = a.ci + s.off + lane;
                    const T* vp = a.val + s.off + lane;
                    T d = T(0), r = T(0), acc = T(0);
                    if (row.own) { d = a.d[row.i]; r = a.r[row.i]; }
                    int c[kCgBarrierChunk];
                    T v[kCgBarrierChunk];
                    #pragma unroll
                    for (int u = 0; u < kCgBarrierChunk; u++) {
                        c[u] = u < s.len_u ? __ldcs(cp + 32 * u) : -1;
                        v[u] = u < s.len_u ? __ldcs(vp + 32 * u) : T(0);
                    }
                    for (int k = 0; k < s.len_u; k += kCgBarrierChunk) {
                        T g[kCgBarrierChunk];
                        #pragma unroll
                        for (int u = 0; u < kCgBarrierChunk; u++) g[u] = c[u] >= 0 ? a.d[c[u]] : T(0);
                        int cn[kCgBarrierChunk];
                        T vn[kCgBarrierChunk];
                        #pragma unroll
                        for (int u = 0; u < kCgBarrierChunk; u++) {
                            const bool ok = k + kCgBarrierChunk + u < s.len_u;
                            cn[u] = ok ? __ldcs(cp + 32 * (k + kCgBarrierChunk + u)) : -1;
                            vn[u] = ok ? __ldcs(vp + 32 * (k + kCgBarrierChunk + u)) : T(0);
                        }
                        #pragma unroll
                        for (int u = 0; u < kCgBarrierChunk; u++)
                            if (k + u < s.len_u) acc = fma(v[u], g[u], acc);
                        #pragma unroll
                        for (int u = 0; u < kCgBarrierChunk; u++) { c[u] = cn[u]; v[u] = vn[u]; }
                    }
                    acc = row_sum<T>(acc, s.shift);
                    if (row.own) {
                        a.q[row.i] = acc;
                        sums[1] = acc_product(sums[1], d, acc);
                        sums[2] = acc_product(sums[2], r, acc);
                        sums[3] = acc_product(sums[3], acc, acc);
                    }
                }
            }
        }
        if constexpr (!REG)
            if (!flow_reduce<T, 4>(sums, a.partials + (K & 1) * 4 * gridDim.x, st, epoch, 94, live, sh, tot)) return;
        if (threadIdx.x < 32) cg_control(tot, K, a.n, a.tol2, a.print_modulo, a.print_tol, ctl);
        __syncthreads();
        status = ctl.status;
        if (status >= 0) break;
        alpha = (T)ctl.alpha;
        beta = (T)ctl.beta;
        K++;
        if constexpr (REG) {
            x0 = fma(alpha, d0, x0);
            r0 = fma(-alpha, q0, r0);
            d0 = fma(beta, d0, r0);
        }
        if (K >= a.max_iter) { status = FEEC_MAXITER; break; }
    }
    Acc last[1] = {AT::zero()};
    if constexpr (REG) {
        if (row0.own) {
            a.x[row0.i] = x0;
            a.r[row0.i] = r0;
            last[0] = acc_product(last[0], r0, r0);
        }
    } else if (status == FEEC_MAXITER) {
        for (int j = 0; j < w.mine; j++) {
            const FlowSlice s = flow_slice(w.raw(j));
            const FlowRow row = flow_row(s, lane);
            if (row.own) {
                const int i = row.i;
                const T r = fma(-alpha, a.q[i], a.r[i]);
                a.x[i] = fma(alpha, a.d[i], a.x[i]);
                a.r[i] = r;
                last[0] = acc_product(last[0], r, r);
            }
        }
    }
    // at the cap no iteration follows that would sum the last residual: it is summed here
    double rr[1] = {tot[0]};
    if (status == FEEC_MAXITER &&
        !flow_reduce<T, 1>(last, a.partials + (K & 1) * 4 * gridDim.x, st, epoch, 89, live, sh, rr))
        return;
    finish(st, status, K, rr[0], tot[1]);
    if (blockIdx.x == 0 && threadIdx.x == 0) st->extra[0] = tot[0];
}

// Fills the slices of the permuted rows: entry p of row perm[i] at lane r << shift | (p mod
// 2^shift), column p >> shift, in the matrix's order, columns renumbered.
__global__ void flow_cg_fill_kernel(int nslices, const int4* __restrict__ meta, const int* __restrict__ perm,
                                    const int* __restrict__ iperm, const int* __restrict__ A, const int* __restrict__ C,
                                    const double* __restrict__ V, int* __restrict__ ci, double* __restrict__ val64,
                                    float* __restrict__ val32) {
    const int sl = blockIdx.x * (blockDim.x / 32) + threadIdx.x / 32;
    const int lane = threadIdx.x & 31;
    if (sl >= nslices) return;
    const FlowSlice s = flow_slice(__ldg(&meta[sl]));
    const int r = lane >> s.shift, t = lane & ((1 << s.shift) - 1);
    const int i = r < s.nrow ? perm[s.row0 + r] : -1;
    const int lo = i >= 0 ? A[i] : 0, hi = i >= 0 ? A[i + 1] : 0;
    for (int k = 0; k < s.len_u; k++) {
        const int j = lo + (k << s.shift) + t;
        const bool real = j < hi;
        const long long o = s.off + 32ll * k + lane;
        if (ci) ci[o] = real ? iperm[C[j]] : -1;
        const double v = real ? V[j] : 0.0;
        if (val64) val64[o] = v;
        if (val32) val32[o] = (float)v;
    }
}

}  // namespace

// The form a natural-order solver runs in: vectors in registers, published, or neither.
FlowForm flow_natural_form(const FlowData& D, int n, int sms) {
    FlowForm f;
    // one warp per scheduler and block before more blocks are added: fewer partial sums to add
    f.blocks = std::max(1, std::min(sms, (D.nslices + 3) / 4));
    const int warps = (D.nslices + f.blocks - 1) / f.blocks;
    f.threads = 32 * std::min(warps, kFlowWarps);
    f.registers = warps <= kFlowWarps && D.longest <= kFlowChunk;
    f.published = n <= kFlowPublishedRows && 32 * D.units <= kFlowPublishedEntries;
    return f;
}

// Rows sorted by length (longest first, stable) within windows of kSortWindow, slices, columns
// and the values of the wanted precision, from the device CSR (A, C, V).
int flow_natural_build(FlowData& D, cudaStream_t st, int dev, int n, const int* A, const int* C, const double* V, bool f32) {
    const bool first = !D.ready;
    if (first) {
        D.mem.release();
        D = FlowData{};
        D.mem.stream = st;
        int sms = 0;
        FEEC_TRY(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
        const int e = cut_natural(D, st, sms, n, A);
        if (e != FEEC_OK) return e;
        FEEC_TRY(D.mem.alloc(D.ci, (size_t)D.units * 32));
        FEEC_TRY(alloc_published(D, 2, n));
        for (int k = 0; k < 5; k++) FEEC_TRY(D.mem.alloc(D.own[k], (size_t)n));
    }
    if (f32) FEEC_TRY(D.mem.alloc(D.val32, (size_t)D.units * 32));
    else FEEC_TRY(D.mem.alloc(D.val64, (size_t)D.units * 32));
    note_launch();
    flow_cg_fill_kernel<<<(D.nslices + 7) / 8, 256, 0, st>>>(D.nslices, D.meta, D.perm, D.iperm, A, C, V,
                                                            first ? D.ci : nullptr, f32 ? nullptr : D.val64,
                                                            f32 ? D.val32 : nullptr);
    FEEC_TRY(cudaGetLastError());
    D.ready = true;
    return FEEC_OK;
}

// A system's slices for plain CG, kept with the system.
int flow_cg_build(feec_system* s, bool f32) {
    FlowData& D = s->flow_cg;
    if (D.ready && (f32 ? (void*)D.val32 : (void*)D.val64)) return FEEC_OK;
    HomeStreamScope home(s);
    return flow_natural_build(D, s->stream, s->dev, s->n, s->A, s->C, s->V, f32);
}

namespace {

template <typename T>
__global__ void permute_kernel(int n, const int* __restrict__ perm, const T* __restrict__ src, T* __restrict__ dst, bool back) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    if (back) dst[perm[i]] = src[i];
    else dst[i] = src[perm[i]];
}

template <typename T>
cudaError_t permute(int n, const int* perm, const T* src, T* dst, bool back, cudaStream_t st) {
    note_launch();
    permute_kernel<T><<<(n + 255) / 256, 256, 0, st>>>(n, perm, src, dst, back);
    return cudaGetLastError();
}

template <typename T>
int flow_cg_launch(feec_system* s, const CgArgs<T>& p, LaunchShape& shape) {
    const FlowData& D = s->flow_cg;
    cudaStream_t st = s->stream;
    FlowCgArgs<T> a{};
    a.n = p.n; a.nslices = D.nslices; a.meta = D.meta; a.ci = D.ci;
    if constexpr (sizeof(T) == 8) a.val = D.val64;
    else a.val = D.val32;
    T* own[5];
    for (int k = 0; k < 5; k++) own[k] = reinterpret_cast<T*>(D.own[k]);
    a.b = own[0]; a.x = own[1]; a.r = own[2]; a.d = own[3]; a.q = own[4];
    for (int k = 0; k < 2; k++) {
        a.pub[k] = reinterpret_cast<T*>(D.pub[k]);
        FEEC_TRY(cudaMemsetAsync(a.pub[k], 0xFF, sizeof(T) * (size_t)p.n, st));
    }
    a.tol2 = p.tol2; a.max_iter = p.max_iter; a.print_modulo = p.print_modulo; a.print_tol = p.print_tol;
    a.partials = p.partials; a.st = p.st;
    int sms = 0;
    FEEC_TRY(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, s->dev));
    const FlowForm form = flow_natural_form(D, p.n, sms);
    const int mode = form.registers ? kCgRegisters : form.published ? kCgPublished : kCgBarrier;
    shape.blocks = form.blocks;
    shape.threads = mode == kCgBarrier ? kCgBarrierThreads : form.threads;
    shape.lanes = 1;
    FEEC_TRY(permute<T>(p.n, D.perm, p.b, own[0], false, st));
    FEEC_TRY(permute<T>(p.n, D.perm, p.x, own[1], false, st));
    const void* fn = mode == kCgRegisters ? (const void*)flow_cg<T, kCgRegisters>
                     : mode == kCgPublished ? (const void*)flow_cg<T, kCgPublished> : (const void*)flow_cg<T, kCgBarrier>;
    void* args[] = {&a};
    note_launch();
    FEEC_TRY(cudaLaunchCooperativeKernel(fn, dim3(shape.blocks), dim3(shape.threads), args, 0, st));
    FEEC_TRY(permute<T>(p.n, D.perm, own[1], p.x, true, st));
    FEEC_TRY(permute<T>(p.n, D.perm, own[2], p.r, true, st));
    return FEEC_OK;
}

}  // namespace

int launch_flow_cg(feec_system* s, const CgArgs<double>& a, LaunchShape& shape) { return flow_cg_launch<double>(s, a, shape); }
int launch_flow_cg(feec_system* s, const CgArgs<float>& a, LaunchShape& shape) { return flow_cg_launch<float>(s, a, shape); }

cudaError_t flow_permute(int n, const int* perm, const double* src, double* dst, bool back, cudaStream_t st) {
    return permute<double>(n, perm, src, dst, back, st);
}

}  // namespace feec
