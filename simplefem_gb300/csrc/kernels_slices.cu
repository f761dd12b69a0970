// Cuts the rows of a layout into the slices of the dataflow solvers (FlowSlice, flow_device.cuh), on
// the device: a solve of a few iterations takes a millisecond or two, so the cut must not cost
// more than that. First solves less later ones, with the rows walked on the host once for each choice of
// lanes per row -> here: colors of 3D P1 refined 7 times (2,146,689 rows) 50 -> 1.0 ms, 6 times 6.7 -> 0.3,
// 3D P2 refined 5 times (274,625 rows) 7.4 -> 0.5; natural order 13.3 -> 0.7, 2.6 -> 0.3, 3.3 -> 0.3; 2D P1
// refined 6 times (4,225 rows) 0.15 -> 0.20. Bound by the chains of a window's walk (80 to 90 us on 3D P2
// refined 5 times) and, for colors, by the fill of the slices (190 us).
//
// The rows of a color (or of a matrix) are cut greedily from the first: a slice takes the following
// rows as long as they need no more lanes than its first and fit 32 lanes. So that windows of rows
// can be cut at the same time, each is cut from all the rows where the slice before it may end,
// one per lane: its first to its 32nd. The windows' ends are then chained (cut_choose_kernel), which
// gives the one cut that starts at the color's first row.
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

// Rows per window: short ones walk faster, many take longer to chain (one warp chains a matrix's).
constexpr int window_rows(bool natural) { return natural ? 512 : 256; }
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

// Of the slices that start in a window.
struct CutStats {
    int chain[2], ops[2], slices, longest, units, bad;
};

struct CutTotal {
    long long units;
    int slices, longest, bad, pad;
};

__device__ __forceinline__ int per_lane(int entries, int shift) { return (entries + (1 << shift) - 1) >> shift; }

template <bool NATURAL>
__device__ __forceinline__ int3 row_parts(const CutRows& rows, int i) {
    if constexpr (NATURAL) return make_int3(0, 0, __ldg(&rows.len[i]));
    const int a = __ldg(&rows.rp[i]), b = __ldg(&rows.lsplit[i]), c = __ldg(&rows.usplit[i]), d = __ldg(&rows.rp[i + 1]);
    return make_int3(b - a, c - b, d - c);
}
__device__ __forceinline__ int shift_of(int longest, int most) {
    int s = 0;
    while (s < 5 && per_lane(longest, s) > most) s++;
    return s;
}

// A block per window (color, first row, end, end of the color) and a warp per choice: lane e cuts from
// the window's row e. ends: how many rows the last slice reaches into the next window.
template <bool NATURAL>
__global__ void __launch_bounds__(32 * kMaxChoices) cut_measure_kernel(const int4* __restrict__ windows, CutChoices choices,
                                                                       CutRows rows, CutStats* __restrict__ stats,
                                                                       unsigned char* __restrict__ ends) {
    constexpr int kSpan = window_rows(NATURAL) + 32;
    __shared__ int3 part[kSpan];
    __shared__ unsigned char need[kMaxChoices][kSpan];
    const int lane = threadIdx.x & 31, o = threadIdx.x >> 5;
    const int4 w = windows[blockIdx.x];
    const int len = w.z - w.y, span = min(len + 31, w.w - w.y);
    for (int k = threadIdx.x; k < span; k += blockDim.x) part[k] = row_parts<NATURAL>(rows, w.y + k);
    __syncthreads();
    for (int k = lane; k < span; k += 32) need[o][k] = (unsigned char)shift_of(max(part[k].x, part[k].z), choices.most[o]);
    __syncwarp();
    CutStats s{};
    int i = lane;
    while (i < len) {
        const int shift = need[o][i], cap = min(i + (32 >> shift), span);
        int l = 0, e = 0, u = 0, k = i;
        do {
            const int3 p = part[k++];
            l = max(l, p.x); e = max(e, p.y); u = max(u, p.z);
        } while (k < cap && need[o][k] <= shift);
        i = k;
        l = per_lane(l, shift); e = per_lane(e, shift); u = per_lane(u, shift);
        const int of[2] = {NATURAL ? u : l, u};
        #pragma unroll
        for (int d = 0; d < (NATURAL ? 1 : 2); d++) {
            const int chunks = (of[d] + kFlowChunk - 1) / kFlowChunk;
            s.chain[d] = max(s.chain[d], 64 * (of[d] + 1) + (NATURAL ? 92 : 64) * shift + 500 * chunks);
            s.ops[d] += of[d] + shift + (NATURAL ? kNaturalRowOps : kRowOps);
        }
        s.slices++;
        s.longest = max(s.longest, u);
        // a slice's parts are 16 bits, its E part 8
        if (l > 0xffff || u > 0xffff || e > 0xff) s.bad = 1;
        else s.units += l + e + u;
    }
    const long long at = ((long long)blockIdx.x * choices.count + o) * 32 + lane;
    stats[at] = s;
    ends[at] = (unsigned char)max(i - len, 0);
}

// A block per color, a warp per choice: chains the color's windows (starts[w]: rows of window w that
// belong to a slice before it) and takes the choice with the smallest modelled time, among those
// of at most max_slices slices and max_longest entries per lane where there are any.
__global__ void __launch_bounds__(32 * kMaxChoices) cut_choose_kernel(const int* __restrict__ first, CutChoices choices, int sms,
                                                                      int max_slices, int max_longest,
                                                                      const CutStats* __restrict__ stats,
                                                                      const unsigned char* __restrict__ ends,
                                                                      unsigned char* __restrict__ starts, int* __restrict__ best) {
    __shared__ double cost[kMaxChoices];
    __shared__ bool within[kMaxChoices];
    const int lane = threadIdx.x & 31, o = threadIdx.x >> 5, last = first[blockIdx.x + 1];
    int start = 0, chain[2] = {0, 0}, slices = 0, longest = 0;
    long long ops[2] = {0, 0};
    for (int w0 = first[blockIdx.x]; w0 < last; w0 += 32) {
        int mine = 0, end[32];
        #pragma unroll
        for (int k = 0; k < 32; k++)
            end[k] = w0 + k < last ? ends[((long long)(w0 + k) * choices.count + o) * 32 + lane] : 0;
        #pragma unroll
        for (int k = 0; k < 32; k++) {
            if (lane == k) mine = start;
            start = __shfl_sync(kAll, end[k], start);
        }
        const int w = w0 + lane;
        if (w < last) {
            const long long at = (long long)w * choices.count + o;
            starts[at] = (unsigned char)mine;
            const CutStats s = stats[at * 32 + mine];
            for (int d = 0; d < 2; d++) { chain[d] = max(chain[d], s.chain[d]); ops[d] += s.ops[d]; }
            slices += s.slices;
            longest = max(longest, s.longest);
        }
    }
    for (int off = 16; off > 0; off >>= 1)
        for (int d = 0; d < 2; d++) ops[d] += __shfl_xor_sync(kAll, ops[d], off);
    double c = 0.0;
    for (int d = 0; d < 2; d++) c += fmax((double)__reduce_max_sync(kAll, chain[d]), 19.0 * (double)ops[d] / sms);
    slices = __reduce_add_sync(kAll, slices);
    longest = __reduce_max_sync(kAll, longest);
    if (lane == 0) { cost[o] = c; within[o] = slices <= max_slices && longest <= max_longest; }
    __syncthreads();
    if (threadIdx.x == 0) {
        int pick = 0;
        for (int k = 1; k < choices.count; k++)
            if ((within[k] && !within[pick]) || (within[k] == within[pick] && cost[k] < cost[pick])) pick = k;
        best[blockIdx.x] = pick;
    }
}

// First slice and unit of every window (one block), and the totals.
__global__ void __launch_bounds__(1024) cut_scan_kernel(int nwindows, const int4* __restrict__ windows, CutChoices choices,
                                                        const CutStats* __restrict__ stats, const unsigned char* __restrict__ starts,
                                                        const int* __restrict__ best, int* __restrict__ slice0,
                                                        long long* __restrict__ unit0, CutTotal* total) {
    __shared__ long long su[1024];
    __shared__ int ss[1024], sl[32], sb[32];
    const int t = threadIdx.x, each = (nwindows + 1023) / 1024;
    const int lo = min(t * each, nwindows), hi = min(lo + each, nwindows);
    auto at = [&](int w) -> const CutStats& {
        const long long k = (long long)w * choices.count + best[windows[w].x];
        return stats[k * 32 + starts[k]];
    };
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

// A warp per window, which one lane walks: its slices' descriptors.
template <bool NATURAL>
__global__ void __launch_bounds__(64) cut_emit_kernel(int nwindows, const int4* __restrict__ windows, CutChoices choices,
                                                      const int* __restrict__ best, CutRows rows,
                                                      const unsigned char* __restrict__ starts, const int* __restrict__ slice0,
                                                      const long long* __restrict__ unit0, int4* __restrict__ meta) {
    constexpr int kSpan = window_rows(NATURAL) + 32;
    __shared__ int3 parts[2][kSpan];
    __shared__ unsigned char needs[2][kSpan];
    const int gw = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31;
    if (gw >= nwindows) return;
    int3* const part = parts[threadIdx.x >> 5];
    unsigned char* const need = needs[threadIdx.x >> 5];
    const int4 w = windows[gw];
    const int o = best[w.x], most = choices.most[o], len = w.z - w.y, span = min(len + 31, w.w - w.y);
    for (int k = lane; k < span; k += 32) {
        const int3 p = row_parts<NATURAL>(rows, w.y + k);
        part[k] = p;
        need[k] = (unsigned char)shift_of(max(p.x, p.z), most);
    }
    __syncwarp();
    if (lane != 0) return;
    int slice = slice0[gw];
    long long unit = unit0[gw];
    for (int i = starts[(long long)gw * choices.count + o]; i < len;) {
        const int first = i, shift = need[i], cap = min(i + (32 >> shift), span);
        int l = 0, e = 0, u = 0;
        do {
            const int3 p = part[i++];
            l = max(l, p.x); e = max(e, p.y); u = max(u, p.z);
        } while (i < cap && need[i] <= shift);
        l = per_lane(l, shift); e = per_lane(e, shift); u = per_lane(u, shift);
        meta[slice++] = make_int4(w.y + first, (i - first) | shift << 8 | e << 16, l | (int)((unsigned)u << 16), (int)(unsigned)unit);
        unit += l + e + u;
    }
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
    constexpr int kRows = window_rows(NATURAL);
    const int colors = (int)ranges.size() - 1;
    for (int c = 0; c < colors; c++) {
        for (int lo = ranges[c]; lo < ranges[c + 1]; lo += kRows)
            windows.push_back(make_int4(c, lo, std::min(lo + kRows, ranges[c + 1]), ranges[c + 1]));
        first.push_back((int)windows.size());
    }
    const int nw = (int)windows.size();
    DevArena tmp;
    tmp.stream = st;
    struct Release { DevArena& m; ~Release() { m.release(); } } rel{tmp};
    int4* dw; int *dfirst, *best, *slice0; long long* unit0; CutStats* stats; CutTotal* dtot;
    unsigned char *ends, *starts;
    const size_t cuts = windows.size() * choices.count;
    FEEC_TRY(tmp.alloc(dw, windows.size())); FEEC_TRY(tmp.alloc(dfirst, first.size())); FEEC_TRY(tmp.alloc(best, (size_t)colors));
    FEEC_TRY(tmp.alloc(slice0, windows.size())); FEEC_TRY(tmp.alloc(unit0, windows.size()));
    FEEC_TRY(tmp.alloc(stats, 32 * cuts)); FEEC_TRY(tmp.alloc(ends, 32 * cuts)); FEEC_TRY(tmp.alloc(starts, cuts));
    FEEC_TRY(tmp.alloc(dtot, 1));
    FEEC_TRY(cudaMemcpyAsync(dw, windows.data(), sizeof(int4) * windows.size(), cudaMemcpyHostToDevice, st));
    FEEC_TRY(cudaMemcpyAsync(dfirst, first.data(), sizeof(int) * first.size(), cudaMemcpyHostToDevice, st));
    for (int k = 0; k < 4; k++) note_launch();
    cut_measure_kernel<NATURAL><<<nw, 32 * choices.count, 0, st>>>(dw, choices, rows, stats, ends);
    cut_choose_kernel<<<colors, 32 * choices.count, 0, st>>>(dfirst, choices, sms, max_slices, max_longest, stats, ends, starts, best);
    cut_scan_kernel<<<1, 1024, 0, st>>>(nw, dw, choices, stats, starts, best, slice0, unit0, dtot);
    FEEC_TRY(cudaGetLastError());
    CutTotal total{};
    FEEC_TRY(cudaMemcpyAsync(&total, dtot, sizeof(total), cudaMemcpyDeviceToHost, st));
    FEEC_TRY(cudaStreamSynchronize(st));
    // a slice's first unit is 32 bits
    if (total.bad || total.slices <= 0 || total.units > 0x7fffffffll) return FEEC_BADARG;
    D.nslices = total.slices;
    D.units = total.units;
    D.longest = total.longest;
    FEEC_TRY(D.mem.alloc(D.meta, (size_t)D.nslices));
    cut_emit_kernel<NATURAL><<<(nw + 1) / 2, 64, 0, st>>>(nw, dw, choices, best, rows, starts, slice0, unit0, D.meta);
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
