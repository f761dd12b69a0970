// Building blocks of the dataflow solvers (kernels_flow.cu): published values that carry
// their own readiness, gathers that wait for them, and the grid-wide sums.
//
// A value that other warps gather is published with one relaxed store into a buffer whose
// slots hold a sentinel (all bits set) until then; a gather re-reads the slots that still
// hold it. The value is its own flag, so a dependence costs the store's and the load's way
// through L2 (0.6 us measured) instead of a grid barrier with its release and acquire
// fences around the same two trips (a phase of the barrier form measured 2.6 us with its
// entries loaded ahead). Every buffer slot is reset by its owner at a time when a grid-wide
// sum (a release / acquire barrier) separates the reset from the last gather before it and
// from the next publication's gathers after it.
//
// Progress: the grid is launched cooperatively, so every warp is resident; each warp walks
// its slices in one global topological order (phases ascending or descending), so the
// first unfinished slice never waits on another unfinished one. Every wait is bounded
// (time and polls) and leaves through the status word.
#pragma once

#include "feec_device.cuh"
#include "feec_internal.h"

namespace feec {

// Measured on 3D P1 refined 7 times, 3D P2 refined 5 times and 2D P2 refined 7 times: 16 warps
// per SM and chunks of 8 (188 / 68 / 20.9 us per FP64 iteration) against 8 warps and chunks of 16
// (305 / 79 / 21.2), 16 warps and chunks of 12 (199 / 73 / 21.9) or of 16 (213 / 79 / 24.9; spills).
constexpr int kFlowThreads = 512;
constexpr int kFlowWarps = kFlowThreads / 32;
constexpr int kFlowChunk = 8;       // entries per lane gathered together (a multiple of 4)

__device__ __forceinline__ double ld_flow(const double* p) {
    double v;
    asm volatile("ld.relaxed.gpu.global.f64 %0, [%1];" : "=d"(v) : "l"(p));
    return v;
}
__device__ __forceinline__ float ld_flow(const float* p) {
    float v;
    asm volatile("ld.relaxed.gpu.global.f32 %0, [%1];" : "=f"(v) : "l"(p));
    return v;
}
__device__ __forceinline__ bool is_sentinel(double v) { return __double_as_longlong(v) == -1ll; }
__device__ __forceinline__ bool is_sentinel(float v) { return __float_as_int(v) == -1; }
// Publishes v (a NaN with the sentinel's bits is stored as the default NaN).
__device__ __forceinline__ void st_flow(double* p, double v) {
    if (is_sentinel(v)) v = __longlong_as_double(0x7ff8000000000000ll);
    asm volatile("st.relaxed.gpu.global.f64 [%0], %1;" ::"l"(p), "d"(v) : "memory");
}
__device__ __forceinline__ void st_flow(float* p, float v) {
    if (is_sentinel(v)) v = __int_as_float(0x7fc00000);
    asm volatile("st.relaxed.gpu.global.f32 [%0], %1;" ::"l"(p), "f"(v) : "memory");
}
__device__ __forceinline__ void reset_flow(double* p) {
    asm volatile("st.relaxed.gpu.global.b64 [%0], %1;" ::"l"(p), "l"(-1ll) : "memory");
}
__device__ __forceinline__ void reset_flow(float* p) {
    asm volatile("st.relaxed.gpu.global.b32 [%0], %1;" ::"l"(p), "r"(-1) : "memory");
}

// One warp's slice: 32 >> shift rows, 1 << shift lanes each, its entries column-major
// ([L | E | U] blocks of `len` entries per lane) from (long long)off * 32.
struct FlowSlice {
    int row0, nrow, shift, len_l, len_e, len_u;
    long long off;
};
// Parts of a slice's entries that a sweep reads.
enum { kFlowL = 0, kFlowU = 1, kFlowAll = 2 };
template <int PART>
__device__ __forceinline__ long long part_off(const FlowSlice& s) {
    return PART == kFlowU ? s.off + 32ll * (s.len_l + s.len_e) : s.off;
}
template <int PART>
__device__ __forceinline__ int part_len(const FlowSlice& s) {
    return PART == kFlowU ? s.len_u : PART == kFlowL ? s.len_l : s.len_l + s.len_e + s.len_u;
}
__device__ __forceinline__ FlowSlice flow_slice(const int4 m) {
    FlowSlice f;
    f.row0 = m.x;
    f.nrow = m.y & 0xff;
    f.shift = (m.y >> 8) & 0xff;
    f.len_e = (m.y >> 16) & 0xffff;
    f.len_l = m.z & 0xffff;
    f.len_u = (m.z >> 16) & 0xffff;
    f.off = (long long)(unsigned)m.w * 32;
    return f;
}

// The lane's row of a slice: lane 0 of the row's group owns the row.
struct FlowRow {
    int i;
    bool own;
};
__device__ __forceinline__ FlowRow flow_row(const FlowSlice& s, int lane) {
    const int k = lane >> s.shift;
    return FlowRow{s.row0 + k, k < s.nrow && (lane & ((1 << s.shift) - 1)) == 0};
}

// A wait's bound: polls are counted, and every 4096 of them the abort flag and the clock are
// looked at. Returns false once the wait has to be given up (status and abort are set).
static __device__ __noinline__ bool flow_wait_goes_on(DeviceStatus* st, unsigned long long& t0, int site) {
    if (ld_volatile_i32(&st->abort)) return false;
    const unsigned long long t = globaltimer_ns();
    if (t0 == 0) t0 = t;
    if (t - t0 <= kWaitNanos) return true;
    atomicExch(&st->abort, 1);
    atomicCAS(&st->status, FEEC_OK, FEEC_TIMEOUT);
    atomicExch(&st->timeout_site, site);
    return false;
}

// The slices of one warp. Slice j of `mine` is slice gw + j * nw of the grid, so that
// consecutive slices of a phase are on different SMs.
struct FlowWarp {
    const int4* meta;
    int gw, nw, mine, lane;
    __device__ __forceinline__ void init(const int4* m, int nslices) {
        meta = m;
        lane = threadIdx.x & 31;
        nw = gridDim.x * (blockDim.x >> 5);
        gw = (threadIdx.x >> 5) * gridDim.x + blockIdx.x;
        mine = gw < nslices ? (nslices - 1 - gw) / nw + 1 : 0;
    }
    // descriptor of slice j (an empty slice past the ends)
    __device__ __forceinline__ int4 raw(int j) const {
        return j >= 0 && j < mine ? __ldg(&meta[gw + j * nw]) : make_int4(0, 0, 0, 0);
    }
};

// A lane's next columns (-1: none).
struct FlowCols {
    int c[kFlowChunk];
    __device__ __forceinline__ void load(const int* __restrict__ ci, long long off, int len, int lane) {
        #pragma unroll
        for (int u = 0; u < kFlowChunk; u++) c[u] = u < len ? __ldg(ci + off + 32 * u + lane) : -1;
    }
};

// acc - sum over entries [0, len) of the lane of val * X[col], X published while the kernel
// runs, in two halves: begin() requests the first chunk's values and gathers and the columns
// after it, so that the caller's own-row work runs while they travel; finish() waits. `cols`
// holds the part's first columns on entry and, after finish(), those at (next_off, next_len).
// A lane's entries are in the order in which their columns are published, and are added in
// groups of four as the groups arrive: behind the last arrival stand at most four dependent
// FP64 operations (64 cycles each). Unused slots are jumped over, not masked: a masked FP64
// instruction takes as long.
template <typename T>
struct FlowGather {
    T v[kFlowChunk], g[kFlowChunk];
    FlowCols ahead;

    __device__ __forceinline__ void request(const int* __restrict__ ci, const T* __restrict__ val, long long off, int k0,
                                            int len, const FlowCols& cols, long long next_off, int next_len, int lane,
                                            const T* X) {
        #pragma unroll
        for (int u = 0; u < kFlowChunk; u++) {
            g[u] = T(0);
            if (cols.c[u] >= 0) g[u] = ld_flow(X + cols.c[u]);
        }
        const T* vp = val + off + 32ll * k0 + lane;
        #pragma unroll
        for (int u = 0; u < kFlowChunk; u++) v[u] = k0 + u < len ? __ldg(vp + 32 * u) : T(0);
        const bool last = k0 + kFlowChunk >= len;
        ahead.load(ci, last ? next_off : off + 32ll * (k0 + kFlowChunk), last ? next_len : len - k0 - kFlowChunk, lane);
    }
    __device__ __forceinline__ void begin(const int* __restrict__ ci, const T* __restrict__ val, long long off, int len,
                                          const FlowCols& cols, long long next_off, int next_len, int lane, const T* X) {
        request(ci, val, off, 0, len, cols, next_off, next_len, lane, X);
    }
    // Waits for the chunk in flight (m entries of it, at most kFlowChunk) and subtracts it.
    __device__ __forceinline__ T wait(const FlowCols& cols, int m, const T* X, T acc, DeviceStatus* st, int site,
                                      bool& live) {
        unsigned spins = 0;
        unsigned long long t0 = 0;
        #pragma unroll
        for (int b = 0; b < kFlowChunk; b += 4) {
            if (b < m) {
                while (live) {
                    int missing = is_sentinel(g[b]) || is_sentinel(g[b + 1]) || is_sentinel(g[b + 2]) ||
                                  is_sentinel(g[b + 3]);
                    asm volatile("" : "+r"(missing));     // one vote for all lanes, whatever their columns
                    if (!__any_sync(0xffffffffu, missing)) break;
                    if ((++spins & 4095u) == 0) {
                        if (!flow_wait_goes_on(st, t0, site)) live = false;
                        live = __all_sync(0xffffffffu, live);
                    }
                    #pragma unroll
                    for (int u = b; u < kFlowChunk; u++)
                        if (is_sentinel(g[u])) g[u] = ld_flow(X + cols.c[u]);
                }
                switch (m - b) {
                    default: acc = fma(-v[b], g[b], acc); acc = fma(-v[b + 1], g[b + 1], acc);
                             acc = fma(-v[b + 2], g[b + 2], acc); acc = fma(-v[b + 3], g[b + 3], acc); break;
                    case 3: acc = fma(-v[b], g[b], acc); acc = fma(-v[b + 1], g[b + 1], acc);
                            acc = fma(-v[b + 2], g[b + 2], acc); break;
                    case 2: acc = fma(-v[b], g[b], acc); acc = fma(-v[b + 1], g[b + 1], acc); break;
                    case 1: acc = fma(-v[b], g[b], acc); break;
                }
            }
        }
        return acc;
    }
    __device__ __forceinline__ T finish(const int* __restrict__ ci, const T* __restrict__ val, long long off, int len,
                                        FlowCols& cols, long long next_off, int next_len, int lane, const T* X, T acc,
                                        DeviceStatus* st, int site, bool& live) {
        for (int k0 = 0;;) {
            acc = wait(cols, len - k0, X, acc, st, site, live);
            cols = ahead;
            k0 += kFlowChunk;
            if (k0 >= len) return acc;
            request(ci, val, off, k0, len, cols, next_off, next_len, lane, X);
        }
    }
};

// Walks the warp's slices (descending if BACK): body(slice, the first columns of its PART, offset
// and length of the next slice's PART). Descriptors are requested two slices ahead.
template <int PART, bool BACK, typename F>
__device__ __forceinline__ void flow_sweep(const FlowWarp& w, const int* __restrict__ ci, F&& body) {
    constexpr int step = BACK ? -1 : 1;
    int j = BACK ? w.mine - 1 : 0;
    FlowSlice s = flow_slice(w.raw(j));
    int4 r = w.raw(j + step);
    FlowCols cols;
    cols.load(ci, part_off<PART>(s), part_len<PART>(s), w.lane);
    for (int k = 0; k < w.mine; k++) {
        const FlowSlice next = flow_slice(r);
        r = w.raw(j + 2 * step);
        body(s, cols, part_off<PART>(next), part_len<PART>(next));
        s = next;
        j += step;
    }
}

// acc - sum over entries [0, len) of the lane, X unchanged while it is read (the restart).
template <typename T>
__device__ __forceinline__ T direct_minus(const int* __restrict__ ci, const T* __restrict__ val, long long off, int len,
                                          int lane, const T* X, T acc) {
    for (int k = 0; k < len; k++) {
        const int c = __ldg(&ci[off + 32ll * k + lane]);
        if (c >= 0) acc = fma(-__ldg(&val[off + 32ll * k + lane]), X[c], acc);
    }
    return acc;
}

// Sum over the 1 << shift lanes of a row (every lane of the row receives it).
template <typename T>
__device__ __forceinline__ T row_sum(T s, int shift) {
    for (int off = 1 << shift >> 1; off > 0; off >>= 1) s += __shfl_xor_sync(0xffffffffu, s, off);
    return s;
}

// |a| < bound and a < 0 on the bits (bound > 0): the control thread's FP64 comparisons would
// take 64 cycles each. Both are false for NaN, as the comparisons are.
__device__ __forceinline__ bool abs_below(double a, double bound) {
    return (__double_as_longlong(a) & 0x7fffffffffffffffll) < __double_as_longlong(bound);
}
__device__ __forceinline__ bool below_zero(double a) {
    const long long b = __double_as_longlong(a);
    return b < 0 && (b << 1) != 0 && (unsigned long long)(b << 1) <= 0xffe0000000000000ull;
}
// sqrt|a| < the reference's machine epsilon 2^-52 (sparsesolver.cpp:153-157)
__device__ __forceinline__ bool energy_small(double a) { return abs_below(a, 4.9303806576313238e-32); }

// a * b added to a running sum: FP64 by one fused operation; FP32 with the product's
// rounding error kept (fma(a, b, -ab) is exact) in the compensated pair.
__device__ __forceinline__ double acc_product(double acc, double a, double b) { return fma(a, b, acc); }
__device__ __forceinline__ CompF acc_product(CompF acc, float a, float b) {
    const float p = a * b;
    acc = comp_add(acc, p);
    acc.c += fmaf(a, b, -p);
    return acc;
}

struct FlowShared {
    double warp_sum[32][4];   // a block has at most 32 warps
    double total[4][4];
    int ok;
};

// The block's and the grid's part of flow_reduce: every warp has put its NV sums into
// sh.warp_sum[warp].
template <int NV>
__device__ __forceinline__ bool flow_reduce_warps(double* part, DeviceStatus* st, unsigned long long& epoch, int site,
                                                  bool live, FlowShared& sh, double (&tot)[NV]) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, warps = blockDim.x >> 5;
    const int dead = __syncthreads_or(live ? 0 : 1);   // also orders the block's writes before the release
    if (dead) return false;
    const int nb = gridDim.x;
    if (warp == 0) {
        const int i = lane & 3;
        double a = i < NV && (lane >> 2) < warps ? sh.warp_sum[lane >> 2][i] : 0.0;
        for (int w = (lane >> 2) + 8; w < warps; w += 8)
            if (i < NV) a += sh.warp_sum[w][i];
        for (int off = 4; off < 4 * warps && off < 32; off <<= 1) a += __shfl_xor_sync(0xffffffffu, a, off);
        if (lane < NV) {
            if (nb == 1) sh.total[0][lane] = a;
            else part[4 * blockIdx.x + lane] = a;
        }
        __syncwarp();
        if (lane == 0) {
            sh.ok = 1;
            if (nb > 1) {
                epoch += 1;
                arrive_release(&st->barrier);
                sh.ok = wait_counter(st, epoch * (unsigned long long)nb, site, kWaitNanos) ? 1 : 0;
            }
        }
    }
    __syncthreads();
    if (!sh.ok) return false;
    if (nb == 1) {
        #pragma unroll
        for (int i = 0; i < NV; i++) tot[i] = sh.total[0][i];
        __syncthreads();
        return true;
    }
    const int readers = warps < 4 ? warps : 4;
    if (warp < readers) {
        const int i = lane & 3;
        double a = 0.0;
        // five blocks' partials requested together (all of them on 152 blocks), then added
        for (int b0 = warp * 8 + (lane >> 2); b0 < nb; b0 += 40 * readers) {
            double p[5];
            #pragma unroll
            for (int k = 0; k < 5; k++) {
                const int b = b0 + 8 * readers * k;
                p[k] = i < NV && b < nb ? __ldcg(&part[4 * b + i]) : 0.0;
            }
            #pragma unroll
            for (int k = 0; k < 5; k++)
                if (b0 - (lane >> 2) + 8 * readers * k < nb) a += p[k];
        }
        #pragma unroll
        for (int off = 4; off < 32; off <<= 1) a += __shfl_xor_sync(0xffffffffu, a, off);
        if (lane < NV) sh.total[warp][lane] = a;
    }
    __syncthreads();
    if (warp == 0) {
        const int i = lane & 3;
        double a = i < NV ? sh.total[0][i] : 0.0;
        for (int w = 1; w < readers; w++) a += i < NV ? sh.total[w][i] : 0.0;
        #pragma unroll
        for (int j = 0; j < NV; j++) tot[j] = __shfl_sync(0xffffffffu, a, j);
    }
    return true;
}

// A warp's part of flow_reduce: its NV sums into sh.warp_sum. With four sums the tree halves the
// number of values each step (6 additions instead of 20: an FP64 addition costs a warp 64 cycles).
template <typename T, int NV>
__device__ __forceinline__ void flow_warp_sums(const typename AccT<T>::type (&v)[NV], FlowShared& sh) {
    static_assert(NV == 1 || NV == 2 || NV == 4, "sums per reduction");
    using A = AccT<T>;
    using Acc = typename A::type;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    Acc k = v[0];
    int idx = 0, rest = 16;
    if constexpr (NV == 4) {
        const bool hi = lane & 16;
        Acc k0 = A::merge(hi ? v[2] : v[0], A::shfl_xor(hi ? v[0] : v[2], 16));
        Acc k1 = A::merge(hi ? v[3] : v[1], A::shfl_xor(hi ? v[1] : v[3], 16));
        const bool mid = lane & 8;
        k = A::merge(mid ? k1 : k0, A::shfl_xor(mid ? k0 : k1, 8));
        idx = (hi ? 2 : 0) + (mid ? 1 : 0);
        rest = 4;
    } else if constexpr (NV == 2) {
        const bool hi = lane & 16;
        k = A::merge(hi ? v[1] : v[0], A::shfl_xor(hi ? v[0] : v[1], 16));
        idx = hi ? 1 : 0;
        rest = 8;
    }
    for (int off = rest; off > 0; off >>= 1) k = A::merge(k, A::shfl_xor(k, off));
    if ((lane & (2 * rest - 1)) == 0) sh.warp_sum[warp][idx] = A::value(k);
}

// Grid-wide sums of NV (at most 4) accumulators per thread, which is also the iteration's
// barrier: everything written before it in any block is visible after it in every block.
// The totals are returned to warp 0 of every block (identical bits in every block: fixed
// shuffle trees and a fixed order over blocks). `part` must not be one that some block may
// still be reading (callers alternate two). Returns false in every thread when a wait gave up
// here or, `live` false, before.
template <typename T, int NV>
__device__ __forceinline__ bool flow_reduce(typename AccT<T>::type (&v)[NV], double* part, DeviceStatus* st,
                                            unsigned long long& epoch, int site, bool live, FlowShared& sh,
                                            double (&tot)[NV]) {
    flow_warp_sums<T, NV>(v, sh);
    return flow_reduce_warps<NV>(part, st, epoch, site, live, sh, tot);
}

}  // namespace feec
