// SSOR / multicolor SSOR preconditioned CG for small systems in one thread block, with the
// gathered vectors in shared memory.
//
// ConjugateGradientSolverCSR_SSOR (solver/sparsesolver.cpp:446-724) sweeps its rows in index
// order: over a dependency-level schedule that is 2 x (number of levels) dependent phases per
// iteration (129 levels on the 2D P1 operator refined 6 times) of a few dozen rows each, so a
// phase costs its latency. What that latency is made of on GB300: a warp's FP64 instruction
// holds its scheduler 64 cycles whatever its active lanes, a shared-memory access takes 30, a
// barrier of a few warps 20. So a phase's rows get a lane each (or several for long rows)
// on as many warps as they fill; a row's factor omega / D is multiplied into its entries and,
// before the sweep, into its right-hand side; and the phase's entries are staged in shared memory
// by a warp that does nothing else. Behind a phase's barrier stand one gather and the row's
// products. Colors (multicolor schedules) hold hundreds of rows and are bound by the one SM's
// FP64 units instead (19 cycles per warp instruction).
//
// The block leaves the other SMs free: small solves on several streams run side by side.
// Index-order systems come here up to
// 13,569 rows, where their two vectors leave a ring of eight slices (us per iteration here and in
// pcg_persistent: 2D P1, 9,000 rows 156 / 495, 12,000 rows 182 / 900, 13,569 rows 285 / 972; 3D P2, 9,000
// rows 515 / 808, 13,500 rows 657 / 1224); multicolor ones up to kSmallColorRows, beyond which
// the dataflow solver takes them (alone on the GPU it is the faster one here too: 18 us).
//
// Measured per iteration, 2D P1 refined 6 times (4,225 rows): index order 228 us (one warp walking
// the levels over records, up to three rows a lane) -> 93; multicolor 70 -> 47. 3D P1, 4,913 rows,
// 49 levels: 221 -> 114; 3D P2, 4,913 rows, 113 levels: 1793 -> 284.
#include <algorithm>
#include <cmath>
#include <cstdio>
#include <cstring>
#include <vector>

#include "flow_device.cuh"
#include "feec_system.h"
#include "persistent_common.cuh"

namespace feec {
namespace {

constexpr int kSmallColorRows = 4608;   // multicolor systems
// 512: 93 / 47 us per iteration (index order / colors, 4,225 rows); 768: 96 / 48; 1024: 100 / 50
constexpr int kSmallThreads = 512;
constexpr int kSmallWarps = kSmallThreads / 32;
constexpr int kSweepEntries = 4;    // entries of a row part per lane and chunk
constexpr int kMaxSweepDepth = 8;   // phases staged ahead (at least 3)
constexpr int kMaxPadding = 4;      // staged slices to slices with rows, at most

// What a warp needs for its slice of a phase: per lane 4 columns, 4 values times the row's factor
// omega / D, and the row (n, the slot past the vector, where the lane has none). Rows are
// numbered in 16 bits: a system that fits here has fewer.
struct __align__(16) SweepSlice {
    double v[32][kSweepEntries];
    unsigned short c[32][kSweepEntries];
    unsigned short row[32];
    // entries per lane in use here, and further chunks of 4 entries: info >> 4 & 0xff of them,
    // from chunk info >> 12
    int info, pad[3];
};
static_assert(sizeof(SweepSlice) % 16 == 0, "one bulk copy");

// One sweep, phase by phase (dependency levels or colors), 1 << shift lanes per row. Phase p has
// the `width` slices from width * p (some possibly without rows), staged as one copy; phases
// wider than that go on in slices [extra[p], extra[p + 1]), which their warps read from memory.
// `empty` is a slice without rows.
struct SweepView {
    int nph, shift, warps, width, depth, empty;
    int count;                       // most entries per lane; rows of one lane and one chunk: plain
    bool plain;
    const SweepSlice* slices; const int* extra;
    const int* mc; const double* mv;     // further chunks: 32 x 4 columns / values each
};

struct SmallArgs {
    int n, nslices;
    const int4* meta; const int* ci; const double* val;     // full rows, one lane each
    const double* wd; const double* b;
    double scale;                                           // 2 - omega
    double *x, *r, *d, *z, *q;
    SweepView fwd, bwd;
    double tol2;
    int use_zr_rule, max_iter, print_modulo;
    double print_tol;
    DeviceStatus* st;
};

// Doubles of the two vectors and the spare slot (an even count: copies land on 16 bytes).
__host__ __device__ constexpr int small_doubles(int n) { return 2 * n + 2; }

// v != 0 without the FP64 comparison (its warp instruction takes the SM 19 cycles too)
__device__ __forceinline__ bool nonzero(double v) { return (__double_as_longlong(v) << 1) != 0; }

__device__ __forceinline__ unsigned smem_addr(const void* p) { return (unsigned)__cvta_generic_to_shared(p); }
__device__ __forceinline__ void bar_init(unsigned long long* bar) {
    asm volatile("mbarrier.init.shared.b64 [%0], 1;" ::"r"(smem_addr(bar)) : "memory");
}
// `bytes` into shared memory (one lane): the barrier completes when they have landed.
__device__ __forceinline__ void load_slices(void* dst, const void* src, unsigned bytes, unsigned long long* bar) {
    asm volatile("mbarrier.arrive.expect_tx.shared.b64 _, [%0], %1;" ::"r"(smem_addr(bar)), "r"(bytes) : "memory");
    asm volatile("cp.async.bulk.shared::cta.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(smem_addr(dst)),
                 "l"(src), "r"(bytes), "r"(smem_addr(bar))
                 : "memory");
}
// Waits for a copy; gives up after kWaitNanos (status FEEC_TIMEOUT).
__device__ __forceinline__ bool wait_slices(unsigned long long* bar, unsigned parity, DeviceStatus* st) {
    unsigned long long t0 = 0;
    for (unsigned n = 1;; n++) {
        unsigned ok;
        asm volatile("{ .reg .pred p; mbarrier.try_wait.parity.shared.b64 p, [%1], %2; selp.u32 %0, 1, 0, p; }"
                     : "=r"(ok)
                     : "r"(smem_addr(bar)), "r"(parity)
                     : "memory");
        if (ok) return true;
        if ((n & 15u) == 0) {      // a try itself waits for a while
            const unsigned long long t = globaltimer_ns();
            if (t0 == 0) t0 = t;
            if (t - t0 > kWaitNanos) break;
        }
    }
    atomicExch(&st->abort, 1);
    atomicCAS(&st->status, FEEC_OK, FEEC_TIMEOUT);
    return false;
}

struct SweepEntries {
    int row, info;
    ushort4 c;
    double v[kSweepEntries];
};
__device__ __forceinline__ void read_slice(SweepEntries& e, const SweepSlice& s, int lane) {
    const double2 a = *reinterpret_cast<const double2*>(&s.v[lane][0]), b = *reinterpret_cast<const double2*>(&s.v[lane][2]);
    e.v[0] = a.x; e.v[1] = a.y; e.v[2] = b.x; e.v[3] = b.y;
    e.c = *reinterpret_cast<const ushort4*>(&s.c[lane][0]);
    e.row = s.row[lane];
    e.info = s.info;
}

// x[row] -= sum v x[c] for the slice in `e` (padding entries: column 0, value 0); `between` runs
// while the gathers travel. The row's factor is in v and, before the sweep, in x, so behind the
// gathers stand the products alone. COUNT entries per lane; PLAIN: no more, one lane per row.
template <int COUNT, bool PLAIN, typename F>
__device__ __forceinline__ void sweep_slice(const SweepEntries& e, const SweepView& s, double* x, int lane, F&& between) {
    const bool own = PLAIN || (lane & ((1 << s.shift) - 1)) == 0;
    const unsigned short c[4] = {e.c.x, e.c.y, e.c.z, e.c.w};
    double g[COUNT];
    #pragma unroll
    for (int k = 0; k < COUNT; k++) g[k] = x[c[k]];
    double acc = own ? x[e.row] : 0.0;
    between();
    #pragma unroll
    for (int k = 0; k < COUNT; k++) acc = fma(-e.v[k], g[k], acc);
    if constexpr (!PLAIN) {
        for (int t = 0; t < (e.info >> 4 & 0xff); t++) {
            #pragma unroll
            for (int k = 0; k < kSweepEntries; k++) {
                const int o = (kSweepEntries * ((e.info >> 12) + t) + k) * 32 + lane;
                acc = fma(-__ldg(&s.mv[o]), x[__ldg(&s.mc[o])], acc);
            }
        }
        acc = row_sum<double>(acc, s.shift);
    }
    if (own) x[e.row] = acc;
}

__device__ __forceinline__ void sweep_barrier(int warps) {
    asm volatile("bar.sync 1, %0;" ::"r"(warps * 32) : "memory");
}

// A whole sweep by the first s.warps warps of the block and the last warp, which stages the slices,
// s.depth phases ahead: it issues a phase's copy when the slot's last readers have passed a
// barrier, and comes to the barrier that ends phase p only when phase p + 2 has landed, so the
// others never look at a copy's barrier and read the next phase's slice while this phase's gathers
// travel. (Staging by the sweeping warps themselves put 500 cycles of issue and waiting into
// each phase; entries requested into registers phases ahead did not shorten the phases: a warp
// has six scoreboards for its loads and waits for the youngest load on one.) `phase` holds
// the parity of each slot's barrier. False when a copy never landed.
// FAR: more warps than slices in a slot; warp `width` and those after it read their first slice of a
// phase from memory, a phase ahead. A kernel of its own: in one kernel with the others it slows
// their phases by 3 - 13 %.
template <int COUNT, bool PLAIN, bool FAR = false>
__device__ __forceinline__ bool sweep_as(const SweepView& s, double* x, SweepSlice* ring, unsigned long long* bars,
                                      unsigned& phase, DeviceStatus* st) {
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const bool stager = warp == kSmallWarps - 1;      // of every sweep: it keeps the slots' parities
    if ((warp >= s.warps && !stager) || s.nph == 0) return true;
    if (stager) {
        bool ok = true;
        const unsigned bytes = (unsigned)(s.width * sizeof(SweepSlice));
        auto issue = [&](int p, int slot) {
            if (lane == 0 && p < s.nph) load_slices(ring + slot * s.width, s.slices + (long long)p * s.width, bytes, bars + slot);
        };
        auto landed = [&](int p, int slot) {
            if (p >= s.nph) return;
            ok = ok && wait_slices(bars + slot, phase >> slot & 1u, st);
            phase ^= 1u << slot;
        };
        for (int k = 0; k < s.depth; k++) issue(k, k);
        landed(0, 0);
        landed(1, 1);
        sweep_barrier(s.warps + 1);
        int slot = 0, two = 2;      // slots of phases p and p + 2
        for (int p = 0; p < s.nph; p++) {
            landed(p + 2, two);
            sweep_barrier(s.warps + 1);
            issue(p + s.depth, slot);
            slot = slot + 1 == s.depth ? 0 : slot + 1;
            two = two + 1 == s.depth ? 0 : two + 1;
        }
        return ok;
    }
    sweep_barrier(s.warps + 1);
    const bool staged = !FAR || warp < s.width;
    auto beyond = [&](int p) {
        if (p >= s.nph) return s.empty;
        const int at = __ldg(&s.extra[p]) + warp - s.width;
        return at < __ldg(&s.extra[p + 1]) ? at : s.empty;
    };
    SweepEntries even, odd;
    const SweepSlice* here = ring + warp;
    int far = 0;                             // not staged: the warp's slice of the next phase
    if (staged) read_slice(even, *here, lane);
    else { read_slice(even, s.slices[beyond(0)], lane); far = beyond(1); }
    int slot = 0;
    auto step = [&](int p, const SweepEntries& e, SweepEntries& next) {
        slot = slot + 1 == s.depth ? 0 : slot + 1;
        const SweepSlice* ahead = ring + slot * s.width + warp;
        sweep_slice<COUNT, PLAIN>(e, s, x, lane, [&] {
            if (p + 1 >= s.nph) return;
            if (staged) read_slice(next, *ahead, lane);
            else { read_slice(next, s.slices[far], lane); far = beyond(p + 2); }
        });
        if (!FAR && s.width > s.warps)
            for (int k = s.warps; warp + k < s.width; k += s.warps) {
                SweepEntries f;
                read_slice(f, here[k], lane);
                sweep_slice<COUNT, PLAIN>(f, s, x, lane, [] {});
            }
        if (s.extra)
            for (int sl = __ldg(&s.extra[p]) + warp + (FAR ? s.warps - s.width : 0); sl < __ldg(&s.extra[p + 1]); sl += s.warps) {
                SweepEntries f;
                read_slice(f, s.slices[sl], lane);
                sweep_slice<COUNT, PLAIN>(f, s, x, lane, [] {});
            }
        sweep_barrier(s.warps + 1);      // phase p is complete
        here = ahead;
    };
    for (int p = 0; p < s.nph; p += 2) {
        step(p, even, odd);
        if (p + 1 < s.nph) step(p + 1, odd, even);
    }
    return true;
}

template <bool FAR>
__device__ __forceinline__ bool sweep(const SweepView& s, double* x, SweepSlice* ring, unsigned long long* bars,
                                      unsigned& phase, DeviceStatus* st) {
    if constexpr (FAR) {
        if (s.warps > s.width) return sweep_as<kSweepEntries, false, true>(s, x, ring, bars, phase, st);
        return sweep_as<kSweepEntries, false>(s, x, ring, bars, phase, st);
    }
    if (!s.plain) return sweep_as<kSweepEntries, false>(s, x, ring, bars, phase, st);
    if (s.count <= 2) return sweep_as<2, true>(s, x, ring, bars, phase, st);
    if (s.count == 3) return sweep_as<3, true>(s, x, ring, bars, phase, st);
    return sweep_as<4, true>(s, x, ring, bars, phase, st);
}

// Block sum, returned to warp 0. All values meet in shared memory first: summing 512 threads
// takes 12 + 20 + 3 warp additions instead of the 85 of a tree per warp (19 cycles each).
__device__ __forceinline__ double small_sum(double v, double* s_val) {
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    s_val[threadIdx.x] = v;
    __syncthreads();
    if (warp < 4) {
        double a = s_val[threadIdx.x];
        #pragma unroll
        for (int k = 1; k < kSmallThreads / 128; k++) a += s_val[threadIdx.x + 128 * k];
        #pragma unroll
        for (int off = 16; off > 0; off >>= 1) a += __shfl_xor_sync(0xffffffffu, a, off);
        if (lane == 0) s_val[kSmallThreads + warp] = a;
    }
    __syncthreads();
    if (warp != 0) return 0.0;
    return (s_val[kSmallThreads] + s_val[kSmallThreads + 1]) + (s_val[kSmallThreads + 2] + s_val[kSmallThreads + 3]);
}

// acc - sum over entries [k0, k0 + len) of the lane of val * X[col] with X in shared memory; the
// next chunk is requested with the products of the current one.
__device__ __forceinline__ double small_minus(const SmallArgs& a, long long off, int len, int lane, const double* X, double acc) {
    constexpr int CH = 4;
    const int* cp = a.ci + off + lane;
    const double* vp = a.val + off + lane;
    int c[CH];
    double v[CH];
    #pragma unroll
    for (int u = 0; u < CH; u++) {
        c[u] = u < len ? __ldg(cp + 32 * u) : -1;
        v[u] = u < len ? __ldg(vp + 32 * u) : 0.0;
    }
    for (int k = 0; k < len; k += CH) {
        int cn[CH];
        double vn[CH];
        #pragma unroll
        for (int u = 0; u < CH; u++) {
            const bool ok = k + CH + u < len;
            cn[u] = ok ? __ldg(cp + 32 * (k + CH + u)) : -1;
            vn[u] = ok ? __ldg(vp + 32 * (k + CH + u)) : 0.0;
        }
        #pragma unroll
        for (int u = 0; u < CH; u++)
            if (k + u < len) acc = fma(-v[u], c[u] >= 0 ? X[c[u]] : 0.0, acc);
        #pragma unroll
        for (int u = 0; u < CH; u++) { c[u] = cn[u]; v[u] = vn[u]; }
    }
    return acc;
}

template <bool FAR>
__global__ void __launch_bounds__(kSmallThreads, 1) small_pcg(SmallArgs a) {
    extern __shared__ __align__(16) double smem[];
    const int n = a.n;
    double* sd_ = smem;              // d
    // the sweeps' vector, in place: (omega / D) r, then m as the forward sweep passes (a row's own
    // value is read by the row alone, before its m is written), (2 - omega) m, then z as the
    // backward sweep passes; 0 throughout in rows with D == 0 (factor 0), which the sweeps skip.
    // Its slot n belongs to the lanes without a row.
    double* su = smem + n;
    SweepSlice* ring = reinterpret_cast<SweepSlice*>(smem + small_doubles(n));
    __shared__ double s_val[kSmallThreads + 4];
    __shared__ unsigned long long s_bar[kMaxSweepDepth];
    __shared__ double s_scal;
    __shared__ int s_ctl;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    unsigned phase = 0;
    bool ok = true;

    for (int i = threadIdx.x; i < small_doubles(n); i += kSmallThreads) smem[i] = 0.0;   // work vectors start at 0
    if (threadIdx.x < kMaxSweepDepth) bar_init(&s_bar[threadIdx.x]);
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    __syncthreads();

    // every row, one lane each: body(slice, row, has a row)
    auto rows = [&](auto&& body) {
        int4 next = warp < a.nslices ? __ldg(&a.meta[warp]) : make_int4(0, 0, 0, 0);
        for (int s = warp; s < a.nslices; s += kSmallWarps) {
            const FlowSlice f = flow_slice(next);
            if (s + kSmallWarps < a.nslices) next = __ldg(&a.meta[s + kSmallWarps]);
            body(f, f.row0 + lane, lane < f.nrow);
        }
    };
    // m = (D/w + L)^-1 r, z = (D/w + U)^-1 S m (:528-575, :647-699 / :1118-1170, :1241-1307), in su;
    // returns z.r (warp 0)
    auto precondition = [&]() {
        ok = sweep<FAR>(a.fwd, su, ring, s_bar, phase, a.st) && ok;
        __syncthreads();
        if (a.scale != 1.0) {
            for (int i = threadIdx.x; i < n; i += kSmallThreads) su[i] *= a.scale;
            __syncthreads();
        }
        ok = sweep<FAR>(a.bwd, su, ring, s_bar, phase, a.st) && ok;
        __syncthreads();
        double zr = 0.0;
        for (int i = threadIdx.x; i < n; i += kSmallThreads)
            if (nonzero(__ldg(&a.wd[i]))) zr = fma(su[i], a.r[i], zr);
        return small_sum(zr, s_val);
    };

    // ---- restart (sparsesolver.cpp:506-588 / :1072-1175): r = b - A x for rows with D != 0 ----
    rows([&](const FlowSlice& f, int i, bool act) {
        double acc = act ? __ldg(&a.b[i]) : 0.0;
        acc = small_minus(a, f.off, part_len<kFlowAll>(f), lane, a.x, acc);
        const double w = act ? __ldg(&a.wd[i]) : 0.0;
        if (nonzero(w)) { a.r[i] = acc; su[i] = acc * w; }
    });
    __syncthreads();
    double z_r = precondition();
    for (int i = threadIdx.x; i < n; i += kSmallThreads) sd_[i] = su[i];
    __syncthreads();

    // scalar control by thread 0 (z_r is its copy); the others read s_scal and s_ctl
    int K = 0, status = FEEC_MAXITER;
    while (K < a.max_iter) {
        if (threadIdx.x == 0) {
            if (a.print_modulo > 0 && K % a.print_modulo == 0)
                printf("(%d/%d)   INTERIM: Residual norm is %.9le < %.9le\n", K, n, sqrt(z_r), a.print_tol);
            s_ctl = a.use_zr_rule && abs_below(z_r, a.tol2) ? 1 : 0;                          // :601-604 / :1187-1190
        }
        double dq = 0.0;                                                                      // :614-628 / :1197-1212
        rows([&](const FlowSlice& f, int i, bool act) {
            const double q = -small_minus(a, f.off, part_len<kFlowAll>(f), lane, sd_, 0.0);
            if (act) {
                const double qi = nonzero(__ldg(&a.wd[i])) ? q : 0.0;
                a.q[i] = qi;
                dq = fma(sd_[i], qi, dq);
            }
        });
        const double d_Ad = small_sum(dq, s_val);    // its barriers also order q before it is read
        if (threadIdx.x == 0 && s_ctl == 0) {
            if (!isfinite(z_r) || below_zero(z_r) || !isfinite(d_Ad) || below_zero(d_Ad)) s_ctl = 2;
            else if (energy_small(d_Ad)) s_ctl = 3;
            s_scal = z_r / d_Ad;
        }
        if (__syncthreads_or(!ok)) return;       // a staged copy never landed (FEEC_TIMEOUT)
        if (s_ctl) { status = s_ctl == 1 ? FEEC_OK : s_ctl == 2 ? FEEC_BREAKDOWN : FEEC_SMALL_ENERGY; break; }
        const double alpha = s_scal;
        // :640-667 / :1230-1240, the update of x and r (rows with D != 0)
        for (int i0 = threadIdx.x; i0 < n; i0 += 4 * kSmallThreads) {
            double w[4], x[4], r[4], q[4];
            #pragma unroll
            for (int k = 0; k < 4; k++) {       // four rows' values requested together
                const int i = i0 + k * kSmallThreads;
                const bool in = i < n;
                w[k] = in ? __ldg(&a.wd[i]) : 0.0;
                x[k] = in ? a.x[i] : 0.0;
                r[k] = in ? a.r[i] : 0.0;
                q[k] = in ? a.q[i] : 0.0;
            }
            #pragma unroll
            for (int k = 0; k < 4; k++) {
                const int i = i0 + k * kSmallThreads;
                if (nonzero(w[k])) {
                    a.x[i] = fma(alpha, sd_[i], x[k]);
                    const double rn = fma(-alpha, q[k], r[k]);
                    a.r[i] = rn;
                    su[i] = rn * w[k];
                }
            }
        }
        __syncthreads();
        const double z_r_new = precondition();
        if (threadIdx.x == 0) {                                                               // :701-706 / :1309-1318
            s_scal = z_r_new / z_r;
            z_r = z_r_new;
        }
        __syncthreads();
        const double beta = s_scal;
        for (int i = threadIdx.x; i < n; i += kSmallThreads)
            sd_[i] = fma(beta, sd_[i], su[i]);   // 0 where D == 0
        __syncthreads();
        K++;
    }
    for (int i = threadIdx.x; i < n; i += kSmallThreads) { a.d[i] = sd_[i]; a.z[i] = su[i]; }
    finish(a.st, status, K, z_r, 0.0);
}

// A warp waits for a copy that nobody starts (feec_selftest_wait).
__global__ void missing_copy_kernel(DeviceStatus* st) {
    __shared__ unsigned long long bar;
    if (threadIdx.x == 0) bar_init(&bar);
    __syncwarp();
    wait_slices(&bar, 0, st);
}

// Static shared memory of the kernel, left out of the vectors' share.
constexpr int kSmallStatic = 8 * (kSmallThreads + 4) + 8 * kMaxSweepDepth + 256;

int optin_bytes() {
    int dev = 0, optin = 0;
    if (cudaGetDevice(&dev) != cudaSuccess) return 0;
    if (cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev) != cudaSuccess) return 0;
    return optin;
}

// One sweep's slices from the host copy of the layout.
struct SweepHost {
    std::vector<int> extra, mc;
    std::vector<double> mv;
    std::vector<SweepSlice> slices;
    int shift = 0, warps = 1, width = 1, depth = 3, empty = 0, count = 0;
    bool plain = true;
};

// `room`: slices of the shared memory's ring. False when a row is too long for the form.
bool build_sweep(SweepHost& h, int nph, const int* pptr, const int* list, const int* from, const int* to,
                 const int* ci, const double* val, const double* wd, int room, int n) {
    long long entries = 0;
    const int rows = pptr[nph];
    for (int k = 0; k < rows; k++) { const int i = list ? list[k] : k; entries += to[i] - from[i]; }
    // lanes per row: the average part in one chunk per lane, but one where a phase fills the
    // block's warps anyway (colors: bound by the SM's FP64 units)
    const bool wide = rows >= 32 * kSmallWarps / 2 * nph;
    while (!wide && h.shift < 5 && entries > (long long)rows * (kSweepEntries << h.shift)) h.shift++;
    const int width = 1 << h.shift, per = 32 >> h.shift;
    int widest = 1;
    long long real = 0;
    for (int p = 0; p < nph; p++) {
        const int c = (pptr[p + 1] - pptr[p] + per - 1) / per;
        widest = std::max(widest, c);
        real += std::max(c, 1);
    }
    // A warp for each slice of the widest phase, and that phase in a slot, or as much of it as three
    // slots leave room for; warps without a slice in the slot only where they are more than half
    // (us per iteration with and without them: 3D P1, 13,000 rows 261 / 340, 13,500 rows 277 / 550; 3D P2,
    // 13,500 rows 658 / 1418; but 3D P1, 11,000 rows 239 / 221; 2D P1, 13,300 rows 276 / 247, 13,569 rows
    // 294 / 286). Where few phases are that wide (a slot each would be mostly
    // empty: the slices of 3,000 levels of one row beside one of 1,500 rows took 196 MB, and their
    // copies 0.99 us a phase), as many warps as keep the rounds of the wide ones to an eighth of
    // the phases.
    h.warps = std::min(widest, kSmallWarps - 1);
    h.width = std::max(1, std::min(widest, room / 3));
    if (2 * h.width >= h.warps) h.warps = std::min(h.width, h.warps);
    if ((long long)nph * h.width > kMaxPadding * real) {
        for (h.warps = 1; h.warps < std::min(widest, kSmallWarps - 1); h.warps++) {
            long long more = 0;
            for (int p = 0; p < nph; p++) more += std::max(0, (pptr[p + 1] - pptr[p] + per * h.warps - 1) / (per * h.warps) - 1);
            if (8 * more <= nph) break;
        }
        h.width = std::max(1, std::min(h.width, std::min(h.warps, (int)(kMaxPadding * real / nph))));
    }
    h.depth = std::max(3, std::min(kMaxSweepDepth, room / h.width));
    std::vector<SweepSlice> more;
    bool any = false;
    h.extra.assign(1, nph * h.width);
    for (int p = 0; p < nph; p++) {
        int at = 0;
        for (int k0 = pptr[p]; at < h.width || k0 < pptr[p + 1]; k0 += per, at++) {
            SweepSlice s;
            std::memset(&s, 0, sizeof(s));
            for (int l = 0; l < 32; l++) s.row[l] = (unsigned short)n;
            const int k1 = std::min(pptr[p + 1], k0 + per);
            int longest = 0;
            for (int k = k0; k < k1; k++) { const int i = list ? list[k] : k; longest = std::max(longest, (to[i] - from[i] + width - 1) / width); }
            const int chunks = std::max(0, (longest + kSweepEntries - 1) / kSweepEntries - 1);
            const int first = (int)(h.mc.size() / (32 * kSweepEntries));
            if (chunks > 0xff || first >= 1 << 19) return false;
            s.info = std::min(longest, kSweepEntries) | chunks << 4 | first << 12;
            h.count = std::max(h.count, std::min(longest, kSweepEntries));
            if (chunks > 0) h.plain = false;
            h.mc.resize(h.mc.size() + (size_t)32 * kSweepEntries * chunks, 0);
            h.mv.resize(h.mc.size(), 0.0);
            for (int k = k0; k < k1; k++) {
                const int i = list ? list[k] : k, base = (k - k0) * width;
                for (int t = 0; t < width; t++) s.row[base + t] = (unsigned short)i;
                for (int j = 0; j < to[i] - from[i]; j++) {
                    const int e = j / width, lane = base + j % width, chunk = e / kSweepEntries;
                    if (chunk == 0) {
                        s.c[lane][e] = (unsigned short)ci[from[i] + j];
                        s.v[lane][e] = val[from[i] + j] * wd[i];
                    } else {
                        const size_t o = ((size_t)kSweepEntries * (first + chunk - 1) + e % kSweepEntries) * 32 + lane;
                        h.mc[o] = ci[from[i] + j];
                        h.mv[o] = val[from[i] + j] * wd[i];
                    }
                }
            }
            if (at < h.width) h.slices.push_back(s);
            else { more.push_back(s); any = true; }
        }
        h.extra.push_back(nph * h.width + (int)more.size());
    }
    h.slices.insert(h.slices.end(), more.begin(), more.end());
    if (!any) h.extra.clear();
    SweepSlice none;
    std::memset(&none, 0, sizeof(none));
    for (int l = 0; l < 32; l++) none.row[l] = (unsigned short)n;
    h.empty = (int)h.slices.size();
    h.slices.push_back(none);
    if (h.shift > 0) h.plain = false;
    return true;
}

int upload_sweep(DevArena& m, cudaStream_t st, const SweepHost& h, int nph, SweepView& v) {
    int *extra = nullptr, *mc;
    double* mv;
    SweepSlice* slices;
    FEEC_TRY(m.alloc(slices, h.slices.size())); FEEC_TRY(m.alloc(mc, h.mc.size())); FEEC_TRY(m.alloc(mv, h.mv.size()));
    FEEC_TRY(cudaMemcpyAsync(slices, h.slices.data(), sizeof(SweepSlice) * h.slices.size(), cudaMemcpyHostToDevice, st));
    FEEC_TRY(cudaMemcpyAsync(mc, h.mc.data(), 4 * h.mc.size(), cudaMemcpyHostToDevice, st));
    FEEC_TRY(cudaMemcpyAsync(mv, h.mv.data(), 8 * h.mv.size(), cudaMemcpyHostToDevice, st));
    if (!h.extra.empty()) {
        FEEC_TRY(m.alloc(extra, h.extra.size()));
        FEEC_TRY(cudaMemcpyAsync(extra, h.extra.data(), 4 * h.extra.size(), cudaMemcpyHostToDevice, st));
    }
    FEEC_TRY(cudaStreamSynchronize(st));   // the host arrays leave scope
    v.nph = nph; v.shift = h.shift; v.warps = h.warps; v.width = h.width; v.depth = h.depth; v.empty = h.empty; v.count = h.count; v.plain = h.plain;
    v.slices = slices; v.extra = extra; v.mc = mc; v.mv = mv;
    return FEEC_OK;
}

// Slices of the ring beside the two vectors.
int ring_room(int n) {
    return (int)(((long long)optin_bytes() - kSmallStatic - 8ll * small_doubles(n)) / (long long)sizeof(SweepSlice));
}

}  // namespace

// Slices and sweep schedules, kept with the layout.
struct SmallData {
    DevArena mem;
    SmallArgs args{};
};

void small_release(feec_system* s) {
    if (!s->small) return;
    s->small->mem.release();
    delete s->small;
    s->small = nullptr;
}

size_t small_bytes(const feec_system* s) { return s->small ? s->small->mem.bytes : 0; }

bool small_pcg_fits(const feec_system* s) {
    if (s->n >= 0xffff || ring_room(s->n) < 8) return false;
    return s->prepared == FEEC_METHOD_SSOR || (s->prepared == FEEC_METHOD_RAINBOW && s->n <= kSmallColorRows);
}

namespace {

int small_build(feec_system* s) {
    if (s->small) return FEEC_OK;
    HomeStreamScope home(s);
    cudaStream_t st = s->stream;
    const int n = s->n;
    s->small = new SmallData();
    s->small->mem.stream = st;
    DevArena& M = s->small->mem;
    SmallArgs& a = s->small->args;
    std::vector<int> rp((size_t)n + 1), ls((size_t)n), us((size_t)n);
    std::vector<int> fptr((size_t)s->nf + 1), bptr((size_t)s->nbw + 1), brows((size_t)n), ci((size_t)s->nnz);
    std::vector<double> val((size_t)s->nnz), wd((size_t)n);
    FEEC_TRY(cudaMemcpyAsync(rp.data(), s->rp, 4 * rp.size(), cudaMemcpyDeviceToHost, st));
    FEEC_TRY(cudaMemcpyAsync(ls.data(), s->lsplit, 4 * ls.size(), cudaMemcpyDeviceToHost, st));
    FEEC_TRY(cudaMemcpyAsync(us.data(), s->usplit, 4 * us.size(), cudaMemcpyDeviceToHost, st));
    FEEC_TRY(cudaMemcpyAsync(fptr.data(), s->fptr, 4 * fptr.size(), cudaMemcpyDeviceToHost, st));
    FEEC_TRY(cudaMemcpyAsync(bptr.data(), s->bptr, 4 * bptr.size(), cudaMemcpyDeviceToHost, st));
    FEEC_TRY(cudaMemcpyAsync(brows.data(), s->brows, 4 * brows.size(), cudaMemcpyDeviceToHost, st));
    FEEC_TRY(cudaMemcpyAsync(ci.data(), s->ci, 4 * ci.size(), cudaMemcpyDeviceToHost, st));
    FEEC_TRY(cudaMemcpyAsync(val.data(), s->val, 8 * val.size(), cudaMemcpyDeviceToHost, st));
    FEEC_TRY(cudaMemcpyAsync(wd.data(), s->wd, 8 * wd.size(), cudaMemcpyDeviceToHost, st));
    FEEC_TRY(cudaStreamSynchronize(st));
    // full rows, one lane each: one SM's FP64 units are the bound
    std::vector<int4> meta;
    long long units = 0;
    for (int r0 = 0; r0 < n; r0 += 32) {
        const int nr = std::min(32, n - r0);
        int l = 0, e = 0, u = 0;
        for (int i = r0; i < r0 + nr; i++) {
            l = std::max(l, ls[i] - rp[i]);
            e = std::max(e, us[i] - ls[i]);
            u = std::max(u, rp[i + 1] - us[i]);
        }
        if (l > 0xffff || u > 0xffff || e > 0x7fff) return FEEC_BADARG;
        meta.push_back(make_int4(r0, nr | e << 16, l | (int)((unsigned)u << 16), (int)units));
        units += l + e + u;
    }
    int4* dmeta; int* dci; double* dval;
    FEEC_TRY(M.alloc(dmeta, meta.size())); FEEC_TRY(M.alloc(dci, (size_t)units * 32)); FEEC_TRY(M.alloc(dval, (size_t)units * 32));
    FEEC_TRY(cudaMemcpyAsync(dmeta, meta.data(), sizeof(int4) * meta.size(), cudaMemcpyHostToDevice, st));
    FEEC_TRY(flow_fill((int)meta.size(), dmeta, s->rp, s->lsplit, s->usplit, s->ci, s->val, dci, dval, nullptr, st));
    a.n = n; a.nslices = (int)meta.size(); a.meta = dmeta; a.ci = dci; a.val = dval;
    SweepHost f, b;
    const int room = ring_room(n);
    if (!build_sweep(f, s->nf, fptr.data(), nullptr, rp.data(), ls.data(), ci.data(), val.data(), wd.data(), room, n) ||
        !build_sweep(b, s->nbw, bptr.data(), brows.data(), us.data(), rp.data() + 1, ci.data(), val.data(), wd.data(), room, n))
        return FEEC_BADARG;
    const int e = upload_sweep(M, st, f, s->nf, a.fwd);
    return e != FEEC_OK ? e : upload_sweep(M, st, b, s->nbw, a.bwd);
}

}  // namespace

int small_pcg_prepare(feec_system* s) {
    const int e = small_build(s);
    if (e != FEEC_OK) {
        cudaGetLastError();
        small_release(s);
    }
    return e;
}

cudaError_t launch_missing_copy(DeviceStatus* st, cudaStream_t s) {
    note_launch();
    missing_copy_kernel<<<1, 32, 0, s>>>(st);
    return cudaGetLastError();
}

int launch_small_pcg(feec_system* s, const PcgArgs<double>& p, LaunchShape& shape) {
    SmallArgs a = s->small->args;
    a.wd = p.wd; a.scale = 2.0 - p.omega; a.b = p.b; a.x = p.x; a.r = p.r; a.d = p.d; a.z = p.z; a.q = p.q;
    a.tol2 = p.tol2; a.use_zr_rule = p.use_zr_rule; a.max_iter = p.max_iter; a.print_modulo = p.print_modulo;
    a.print_tol = p.print_tol; a.st = p.st;
    const int ring = std::max(a.fwd.width * a.fwd.depth, a.bwd.width * a.bwd.depth);
    const size_t bytes = 8 * (size_t)small_doubles(s->n) + (size_t)ring * sizeof(SweepSlice);
    shape.blocks = 1;
    shape.threads = kSmallThreads;
    shape.lanes = 1 << a.fwd.shift;
    note_launch();
    const auto kernel = a.fwd.warps > a.fwd.width || a.bwd.warps > a.bwd.width ? small_pcg<true> : small_pcg<false>;
    // the most that any system uses, not this one's: the attribute belongs to the kernel, and other
    // threads launch it for other systems
    FEEC_TRY(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, optin_bytes() - kSmallStatic));
    kernel<<<1, kSmallThreads, bytes, s->stream>>>(a);
    return cuda_status(cudaGetLastError());
}

}  // namespace feec
