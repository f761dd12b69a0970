// Cuts the rows of a layout into the slices of the dataflow solvers (FlowSlice, flow_device.cuh), on
// the device: a solve of a few iterations takes a millisecond or two, so the cut must not cost
// more than that. Set-up beside the first solve, walking the rows on the host once for each choice of
// lanes per row -> here: multicolor 3D P1 refined 7 times (2,146,689 rows) 50 -> 0.9 ms, 6 times 6.7 ->
// 0.3, 3D P2 refined 5 times (274,625 rows) 7.4 -> 0.5; natural order 13.3 -> 0.4, 2.6 -> 0.3, 3.3 -> 0.4;
// 2D P1 refined 6 times (4,225 rows) 0.15 -> 0.20. Bound by the walk's chain of loads and votes, and for
// the large ones by the fill of the slices.
//
// Rows are cut window by window, a warp per window and choice, greedily from the window's first row:
// a slice takes the following rows as long as they need no more lanes than its first and fit 32
// lanes. Windows are multiples of 32 rows from the start of a color (or of the matrix), so that rows
// of one length fill their slices.
//
// Lanes per row of each slice. A warp's FP64 instruction holds its scheduler 64 cycles and the SM's
// FP64 units 19 (measured), and a chunk of kFlowChunk entries takes a trip to L2 of about 500. With p
// entries per lane a phase therefore lasts at least as long as its slowest slice, 64 (p + log2
// lanes + 1) + 500 per chunk, and at least 19 cycles per instruction of its slices over the SMs: few
// entries per lane shorten the chain, many lanes per row issue the row's other ~12 operations for
// fewer rows at once. Each color takes the bound on p with the smallest sum over the two sweeps of
// the larger of the two. (3D P2: one lane for the first seven colors, four to eight for the
// 65-entry rows after them. FP32 was fastest on the same slices: with at most 8 entries per lane
// everywhere 67 us per iteration on 3D P2 refined 5 times against 55.) The natural-order solvers have
// one phase, whose lanes are also added by shuffles behind the products (92 cycles a step).
#include <algorithm>
#include <climits>
#include <vector>

#include "flow_device.cuh"
#include "feec_system.h"

namespace feec {
namespace {

// Windows of 1,024 and 2,048 rows: 0.6 ms for the natural order of 3D P2 refined 5 times (0.4 here).
constexpr int kWindow = 256;
constexpr int kRowOps = 12, kNaturalRowOps = 7;   // FP64 operations of a row besides its entries
constexpr int kMaxChoices = 8;
constexpr unsigned kAll = 0xffffffffu;

struct CutChoices {
    int count, most[kMaxChoices];      // entries per lane and part, at most (with up to 32 lanes)
};

struct CutRows {
    const int *rp, *lsplit, *usplit;   // colors: [L | E | U] rows
    const int* len;                    // natural order: entries per row
};

struct CutStats {
    int chain[2], slices, longest, bad, pad;
    long long ops[2], units;
};

struct CutTotal {
    long long units;
    int slices, longest, bad, pad;
};

__device__ __forceinline__ int per_lane(int entries, int shift) { return (entries + (1 << shift) - 1) >> shift; }

// body(first row, rows, shift, entries per lane of L, E and U) for the slices of rows [lo, hi), by a warp.
template <bool NATURAL, typename F>
__device__ __forceinline__ void cut_window(const CutRows& rows, int lo, int hi, int most, F&& body) {
    const int lane = threadIdx.x & 31;
    for (int i = lo; i < hi;) {
        const int k = i + lane;
        int l = 0, e = 0, u = 0;
        if (k < hi) {
            if constexpr (NATURAL) {
                u = __ldg(&rows.len[k]);
            } else {
                const int a = __ldg(&rows.rp[k]), b = __ldg(&rows.lsplit[k]), c = __ldg(&rows.usplit[k]), d = __ldg(&rows.rp[k + 1]);
                l = b - a; e = c - b; u = d - c;
            }
        }
        const int longest = max(l, u);
        int need = 0;
        while (need < 5 && per_lane(longest, need) > most) need++;
        const int shift = __shfl_sync(kAll, need, 0);
        const unsigned fits = __ballot_sync(kAll, k < hi && lane < (32 >> shift) && need <= shift);
        const int nrow = fits == kAll ? 32 : __ffs(~fits) - 1;
        const bool in = lane < nrow;
        const int pl = NATURAL ? 0 : __reduce_max_sync(kAll, in ? per_lane(l, shift) : 0);
        const int pe = NATURAL ? 0 : __reduce_max_sync(kAll, in ? per_lane(e, shift) : 0);
        const int pu = __reduce_max_sync(kAll, in ? per_lane(u, shift) : 0);
        body(i, nrow, shift, pl, pe, pu);
        i += nrow;
    }
}

template <bool NATURAL>
__global__ void __launch_bounds__(128) cut_measure_kernel(int nwindows, const int4* __restrict__ windows, CutChoices choices,
                                                          CutRows rows, CutStats* __restrict__ stats) {
    const int gw = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    if (gw >= nwindows * choices.count) return;
    const int4 w = __ldg(&windows[gw / choices.count]);
    CutStats s{};
    cut_window<NATURAL>(rows, w.y, w.z, choices.most[gw % choices.count], [&](int, int, int shift, int l, int e, int u) {
        const int part[2] = {NATURAL ? u : l, u};
        #pragma unroll
        for (int k = 0; k < (NATURAL ? 1 : 2); k++) {
            const int chunks = (part[k] + kFlowChunk - 1) / kFlowChunk;
            s.chain[k] = max(s.chain[k], 64 * (part[k] + 1) + (NATURAL ? 92 : 64) * shift + 500 * chunks);
            s.ops[k] += part[k] + shift + (NATURAL ? kNaturalRowOps : kRowOps);
        }
        s.slices++;
        s.units += l + e + u;
        s.longest = max(s.longest, u);
        s.bad |= l > 0xffff || u > 0xffff || e > 0xff;
    });
    if ((threadIdx.x & 31) == 0) stats[gw] = s;
}

// One block per color: the choice with the smallest modelled time, among those of at most max_slices
// slices and max_longest entries per lane where there are any.
__global__ void __launch_bounds__(256) cut_choose_kernel(const int* __restrict__ first, CutChoices choices, int sms,
                                                         int max_slices, int max_longest, const CutStats* __restrict__ stats,
                                                         int* __restrict__ best) {
    __shared__ CutStats part[8];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    double cost = -1.0;
    bool within = false;
    int pick = 0;
    for (int o = 0; o < choices.count; o++) {
        CutStats s{};
        for (int w = first[blockIdx.x] + threadIdx.x; w < first[blockIdx.x + 1]; w += blockDim.x) {
            const CutStats& t = stats[(long long)w * choices.count + o];
            for (int k = 0; k < 2; k++) { s.chain[k] = max(s.chain[k], t.chain[k]); s.ops[k] += t.ops[k]; }
            s.slices += t.slices;
            s.longest = max(s.longest, t.longest);
        }
        for (int off = 16; off > 0; off >>= 1) {
            for (int k = 0; k < 2; k++) s.ops[k] += __shfl_xor_sync(kAll, s.ops[k], off);
            s.slices += __shfl_xor_sync(kAll, s.slices, off);
        }
        for (int k = 0; k < 2; k++) s.chain[k] = __reduce_max_sync(kAll, s.chain[k]);
        s.longest = __reduce_max_sync(kAll, s.longest);
        if (lane == 0) part[warp] = s;
        __syncthreads();
        if (threadIdx.x == 0) {
            for (int v = 1; v < 8; v++) {
                for (int k = 0; k < 2; k++) { s.chain[k] = max(s.chain[k], part[v].chain[k]); s.ops[k] += part[v].ops[k]; }
                s.slices += part[v].slices;
                s.longest = max(s.longest, part[v].longest);
            }
            double c = 0.0;
            for (int k = 0; k < 2; k++) c += fmax((double)s.chain[k], 19.0 * (double)s.ops[k] / sms);
            const bool in = s.slices <= max_slices && s.longest <= max_longest;
            if (cost < 0.0 || (in && !within) || (in == within && c < cost)) { cost = c; within = in; pick = o; }
        }
        __syncthreads();
    }
    if (threadIdx.x == 0) best[blockIdx.x] = pick;
}

// First slice and unit of every window (one block), and the totals.
__global__ void __launch_bounds__(1024) cut_scan_kernel(int nwindows, const int4* __restrict__ windows, CutChoices choices,
                                                        const CutStats* __restrict__ stats, const int* __restrict__ best,
                                                        int* __restrict__ slice0, long long* __restrict__ unit0, CutTotal* total) {
    __shared__ long long su[1024];
    __shared__ int ss[1024], sl[32], sb[32];
    const int t = threadIdx.x, each = (nwindows + 1023) / 1024;
    const int lo = min(t * each, nwindows), hi = min(lo + each, nwindows);
    auto at = [&](int w) -> const CutStats& { return stats[(long long)w * choices.count + best[windows[w].x]]; };
    long long units = 0;
    int slices = 0, longest = 0, bad = 0;
    for (int w = lo; w < hi; w++) {
        const CutStats& s = at(w);
        units += s.units; slices += s.slices; longest = max(longest, s.longest); bad |= s.bad;
    }
    su[t] = units; ss[t] = slices;
    longest = __reduce_max_sync(kAll, longest);
    bad = __reduce_or_sync(kAll, (unsigned)bad);
    if ((t & 31) == 0) { sl[t >> 5] = longest; sb[t >> 5] = bad; }
    __syncthreads();
    for (int off = 1; off < 1024; off <<= 1) {
        const long long u = t >= off ? su[t - off] : 0;
        const int s = t >= off ? ss[t - off] : 0;
        __syncthreads();
        su[t] += u; ss[t] += s;
        __syncthreads();
    }
    long long u = su[t] - units;
    int k = ss[t] - slices;
    for (int w = lo; w < hi; w++) {
        slice0[w] = k; unit0[w] = u;
        const CutStats& s = at(w);
        k += s.slices; u += s.units;
    }
    if (t == 0) {
        CutTotal r{su[1023], ss[1023], 0, 0, 0};
        for (int v = 0; v < 32; v++) { r.longest = max(r.longest, sl[v]); r.bad |= sb[v]; }
        *total = r;
    }
}

template <bool NATURAL>
__global__ void __launch_bounds__(128) cut_emit_kernel(int nwindows, const int4* __restrict__ windows, CutChoices choices,
                                                       const int* __restrict__ best, CutRows rows, const int* __restrict__ slice0,
                                                       const long long* __restrict__ unit0, int4* __restrict__ meta) {
    const int gw = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    if (gw >= nwindows) return;
    const int4 w = __ldg(&windows[gw]);
    int k = slice0[gw];
    long long at = unit0[gw];
    cut_window<NATURAL>(rows, w.y, w.z, choices.most[best[w.x]], [&](int row0, int nrow, int shift, int l, int e, int u) {
        if ((threadIdx.x & 31) == 0)
            meta[k] = make_int4(row0, nrow | shift << 8 | e << 16, l | (int)((unsigned)u << 16), (int)(unsigned)at);
        k++;
        at += l + e + u;
    });
}

// Rows of each window of kSortWindow sorted by length, longest first, equal lengths in their order (one
// block per window, a bitonic network over (length, row)): perm, iperm and the lengths in that order.
__global__ void __launch_bounds__(kSortWindow / 2) sort_rows_kernel(int n, const int* __restrict__ rp, int* __restrict__ perm,
                                                                    int* __restrict__ iperm, int* __restrict__ len) {
    __shared__ unsigned long long key[kSortWindow];
    const int base = blockIdx.x * kSortWindow, t = threadIdx.x;
    for (int k = t; k < kSortWindow; k += kSortWindow / 2) {
        const int i = base + k;
        const int L = i < n ? rp[i + 1] - rp[i] : -1;
        key[k] = (unsigned long long)(0x7fffffffu - (unsigned)L) << 32 | (unsigned)k;    // -1: behind every row
    }
    __syncthreads();
    for (int size = 2; size <= kSortWindow; size <<= 1)
        for (int step = size >> 1; step > 0; step >>= 1) {
            const int a = 2 * t - (t & (step - 1)), b = a + step;
            const unsigned long long ka = key[a], kb = key[b];
            if ((ka > kb) == ((a & size) == 0)) { key[a] = kb; key[b] = ka; }
            __syncthreads();
        }
    for (int k = t; k < kSortWindow && base + k < n; k += kSortWindow / 2) {
        const int i = base + (int)(unsigned)key[k];
        perm[base + k] = i;
        iperm[i] = base + k;
        len[base + k] = (int)(0x7fffffffu - (unsigned)(key[k] >> 32));
    }
}

// Windows and their colors from the host, the four steps, and D's slices, units and longest part.
template <bool NATURAL>
int cut(FlowData& D, cudaStream_t st, int sms, const std::vector<int>& ranges, const CutChoices& choices,
        int max_slices, int max_longest, const CutRows& rows) {
    std::vector<int4> windows;
    std::vector<int> first(1, 0);
    const int colors = (int)ranges.size() - 1;
    for (int c = 0; c < colors; c++) {
        for (int lo = ranges[c]; lo < ranges[c + 1]; lo += kWindow) windows.push_back(make_int4(c, lo, std::min(lo + kWindow, ranges[c + 1]), 0));
        first.push_back((int)windows.size());
    }
    const int nw = (int)windows.size();
    DevArena tmp;
    tmp.stream = st;
    struct Release { DevArena& m; ~Release() { m.release(); } } rel{tmp};
    int4* dw; int *dfirst, *best, *slice0; long long* unit0; CutStats* stats; CutTotal* dtot;
    FEEC_TRY(tmp.alloc(dw, windows.size())); FEEC_TRY(tmp.alloc(dfirst, first.size())); FEEC_TRY(tmp.alloc(best, (size_t)colors));
    FEEC_TRY(tmp.alloc(slice0, windows.size())); FEEC_TRY(tmp.alloc(unit0, windows.size()));
    FEEC_TRY(tmp.alloc(stats, windows.size() * choices.count)); FEEC_TRY(tmp.alloc(dtot, 1));
    FEEC_TRY(cudaMemcpyAsync(dw, windows.data(), sizeof(int4) * windows.size(), cudaMemcpyHostToDevice, st));
    FEEC_TRY(cudaMemcpyAsync(dfirst, first.data(), sizeof(int) * first.size(), cudaMemcpyHostToDevice, st));
    for (int k = 0; k < 4; k++) note_launch();
    cut_measure_kernel<NATURAL><<<(nw * choices.count + 3) / 4, 128, 0, st>>>(nw, dw, choices, rows, stats);
    cut_choose_kernel<<<colors, 256, 0, st>>>(dfirst, choices, sms, max_slices, max_longest, stats, best);
    cut_scan_kernel<<<1, 1024, 0, st>>>(nw, dw, choices, stats, best, slice0, unit0, dtot);
    FEEC_TRY(cudaGetLastError());
    CutTotal total{};
    FEEC_TRY(cudaMemcpyAsync(&total, dtot, sizeof(total), cudaMemcpyDeviceToHost, st));
    FEEC_TRY(cudaStreamSynchronize(st));
    // a slice's first unit is 32 bits, its parts 16 and its E part 8
    if (total.bad || total.slices <= 0 || total.units > 0x7fffffffll) return FEEC_BADARG;
    D.nslices = total.slices;
    D.units = total.units;
    D.longest = total.longest;
    FEEC_TRY(D.mem.alloc(D.meta, (size_t)D.nslices));
    cut_emit_kernel<NATURAL><<<(nw + 3) / 4, 128, 0, st>>>(nw, dw, choices, best, rows, slice0, unit0, D.meta);
    FEEC_TRY(cudaGetLastError());
    return FEEC_OK;
}

}  // namespace

int cut_colors(FlowData& D, cudaStream_t st, int sms, const std::vector<int>& ranges, const int* rp, const int* lsplit,
               const int* usplit) {
    const CutChoices choices{8, {1, 2, 4, 8, 12, 16, 24, 32}};
    return cut<false>(D, st, sms, ranges, choices, INT_MAX, INT_MAX, CutRows{rp, lsplit, usplit, nullptr});
}

int cut_natural(FlowData& D, cudaStream_t st, int sms, int n, const int* rp) {
    FEEC_TRY(D.mem.alloc(D.perm, (size_t)n)); FEEC_TRY(D.mem.alloc(D.iperm, (size_t)n));
    DevArena tmp;
    tmp.stream = st;
    struct Release { DevArena& m; ~Release() { m.release(); } } rel{tmp};
    int* len;
    FEEC_TRY(tmp.alloc(len, (size_t)n));
    note_launch();
    sort_rows_kernel<<<(n + kSortWindow - 1) / kSortWindow, kSortWindow / 2, 0, st>>>(n, rp, D.perm, D.iperm, len);
    FEEC_TRY(cudaGetLastError());
    // many rows: few lanes each, without weighing the alternatives
    const bool many = n > 32 * 64 * sms;
    const CutChoices choices = many ? CutChoices{1, {32}} : CutChoices{6, {1, 2, 4, 8, 16, 32}};
    // the register form where a choice fits it (flow_natural_form)
    return cut<true>(D, st, sms, {0, n}, choices, sms * kFlowWarps, kFlowChunk, CutRows{nullptr, nullptr, nullptr, len});
}

}  // namespace feec
