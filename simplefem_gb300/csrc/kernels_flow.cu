// Dataflow forms of the multicolor SSOR solvers (one cooperative launch per solve):
//
//   flow_eisenstat — ConjugateGradientSolverCSR_Eisenstat_Rainbow (solver/sparsesolver.cpp:1338-1645),
//                    the FP64 product mode and the FP32 inner solves of the mixed mode
//   flow_pcg       — ConjugateGradientSolverCSR_Rainbow (:1002-1335)
//
// What bounds a sweep is not its memory traffic but its 2 * colors dependent phases. With a
// grid barrier between phases, as in the persistent kernels, a phase of the 3D P2 operator
// refined 5 times (N = 274,625, 17 colors) cost 6.4 us: the barrier (1.2 us: release fence,
// counter, acquire), its row bounds, columns, values and gathers one after the other, and
// FP64 instructions issued for rows of 4 and 16 lanes (GB300 holds a warp scheduler 64
// cycles for each, whatever its active lanes). Here a row's value is published the moment
// it is known and its readers wait for that value alone (flow_device.cuh), so phases
// overlap wherever the matrix lets them; the entries of a slice and the row's own values
// are requested before the wait; and rows take one lane each unless that leaves
// schedulers idle (kernels_slices.cu chooses lanes per slice). The only grid-wide barriers left
// are the sums: one per iteration (Eisenstat) and two (PCG).
//
// Row slices: every slice belongs to one warp, the same in both sweeps, so a row's own
// vectors (x, r, d and the rest) are only ever touched by the lane that owns the row and
// need no ordering across warps.
#include <algorithm>
#include <cmath>
#include <cstdio>
#include <vector>

#include "flow_device.cuh"
#include "feec_system.h"
#include "persistent_common.cuh"

namespace feec {
namespace {

template <typename T>
struct FlowArgs {
    int n, nslices;
    const int4* meta; const int* ci; const T* val;
    const T* wd; const T* sd;        // omega / D and D (2 - omega) / omega, never 0 here
    const T* b;
    T *x, *r, *d, *w, *q;            // own vectors (w: Eisenstat only; q: PCG only)
    T* pub[4];                       // published vectors, every slot the sentinel on entry
    double tol2, rr_stop;            // |z.r| < tol2 if use_zr_rule; z.r < rr_stop * (z.r at the start) if rr_stop > 0
    int use_zr_rule, max_iter, print_modulo;
    double print_tol;
    double* partials;                // 8 * gridDim.x doubles
    DeviceStatus* st;
    int keep_dir;                    // Eisenstat: see PcgArgs
    double zr_prev, scale;
};

enum { kGoOn = 0, kBreakdown = 1, kSmallEnergy = 2, kConverged = 3, kLastStep = 4 };

// ---------------------------------------------------------------------------
// Eisenstat's formulation. Per iteration: one backward sweep (technical m = (D/w + U)^-1 d,
// with the previous iteration's x, r and d updates formed as each row comes up), one forward
// sweep (auxiliary q = (D/w + L)^-1 (d - S m), w = q + m), and one grid-wide sum of z.r,
// d.w, z.w and w.Sw (z = S r). From those: alpha = z.r / d.w, and beta = (z.r)' / z.r with
// (z.r)' = z.r - 2 alpha z.w + alpha^2 w.Sw, the square expanded of r' = r - alpha w, so that
// no second sum is waited for; the next iteration sums (z.r)' itself for its alpha and the
// stopping rule, so nothing accumulates. Published: m in pub[0 / 1], q in pub[2 / 3], by the
// iteration's parity; an iteration's backward sweep resets the other parity's slots of its
// rows (read by nobody since the last sum).
// Measured, 3D P2 refined 5 times, per iteration: FP64 229 -> 66 us (the barrier-phase kernel
// -> this one), FP32 115 -> 55 us; 3D P1 refined 7 times, FP64: 329 -> 188 us. Without its
// waits (values wrong) the FP64 iteration takes 47 us and without anything but its FP64
// instructions 33, so what is left of the dependences is about 0.6 us for each of the 33 steps.
// ---------------------------------------------------------------------------
template <typename T>
__global__ void __launch_bounds__(kFlowThreads, 1) flow_eisenstat(FlowArgs<T> a) {
    using AT = AccT<T>;
    using Acc = typename AT::type;
    __shared__ FlowShared sh;
    __shared__ double s_scal[2];
    __shared__ int s_ctl;
    FlowWarp w;
    w.init(a.meta, a.nslices);
    const int lane = w.lane, mine = w.mine;
    unsigned long long epoch = 0;
    bool live = true;
    const bool keep = a.keep_dir != 0;
    DeviceStatus* st = a.st;

    // ---- restart (:1409-1478): r = (D/w + L)^-1 (b - A x), z = S r, d = z ----
    Acc sums[4] = {AT::zero(), AT::zero(), AT::zero(), AT::zero()};
    flow_sweep<kFlowL, false>(w, a.ci, [&](const FlowSlice& s, FlowCols& cols, long long noff, int nlen) {
        const FlowRow row = flow_row(s, lane);
        FlowGather<T> in;
        in.begin(a.ci, a.val, part_off<kFlowL>(s), part_len<kFlowL>(s), cols, noff, nlen, lane, a.pub[3]);
        T acc = row.own ? __ldg(&a.b[row.i]) : T(0);
        acc = direct_minus<T>(a.ci, a.val, s.off, part_len<kFlowAll>(s), lane, a.x, acc);
        acc = in.finish(a.ci, a.val, part_off<kFlowL>(s), part_len<kFlowL>(s), cols, noff, nlen, lane, a.pub[3], acc, st, 70, live);
        acc = row_sum<T>(acc, s.shift);
        if (row.own) {
            const T ri = acc * __ldg(&a.wd[row.i]);
            st_flow(a.pub[3] + row.i, ri);
            a.r[row.i] = ri;
            const T zi = ri * __ldg(&a.sd[row.i]);
            if (!keep) a.d[row.i] = zi;
            sums[0] = acc_product(sums[0], zi, ri);
        }
    });
    double tot[4];
    if (!flow_reduce<T, 4>(sums, a.partials + 4 * gridDim.x, st, epoch, 71, live, sh, tot)) return;
    double z_r = tot[0], z_r_prev = tot[0];   // thread 0 only
    const double z_r0 = tot[0];
    int K = 0;
    if (threadIdx.x == 0) {
        if (a.print_modulo > 0 && blockIdx.x == 0)
            printf("(%d/%d)   INTERIM: Residual norm is %.9le < %.9le\n", 0, a.n, sqrt(z_r), a.print_tol);
        s_ctl = (a.use_zr_rule && fabs(z_r) < a.tol2) ? kConverged : kGoOn;               // :1483-1490
        s_scal[1] = keep ? z_r / (a.zr_prev * a.scale) : 0.0;
    }
    __syncthreads();
    int status = FEEC_MAXITER;
    bool step = false;      // the last direction's step is still to be taken
    if (s_ctl == kConverged) status = FEEC_OK;
    else for (;;) {
        const bool first = K == 0;
        const T alpha = (T)s_scal[0], beta = (T)s_scal[1];
        T* const m_pub = a.pub[K & 1];
        T* const m_old = a.pub[(K & 1) ^ 1];
        T* const q_pub = a.pub[2 + (K & 1)];
        T* const q_old = a.pub[2 + ((K & 1) ^ 1)];
        #pragma unroll
        for (int i = 0; i < 4; i++) sums[i] = AT::zero();
        // backward sweep (:1506-1530) with the updates of the previous iteration (:1580-1618)
        flow_sweep<kFlowU, true>(w, a.ci, [&](const FlowSlice& s, FlowCols& cols, long long noff, int nlen) {
            const FlowRow row = flow_row(s, lane);
            FlowGather<T> in;
            in.begin(a.ci, a.val, part_off<kFlowU>(s), part_len<kFlowU>(s), cols, noff, nlen, lane, m_pub);
            T dv = T(0), wdv = T(0);
            if (row.own) {
                const int i = row.i;
                wdv = __ldg(&a.wd[i]);
                T ri = a.r[i];
                dv = a.d[i];
                const T sdv = __ldg(&a.sd[i]);
                if (!first) {
                    a.x[i] = fma(alpha, ld_flow(m_old + i), a.x[i]);
                    ri = fma(-alpha, a.w[i], ri);
                    a.r[i] = ri;
                }
                const T zi = ri * sdv;
                if (!first || keep) {
                    dv = fma(beta, dv, zi);
                    a.d[i] = dv;
                }
                sums[0] = acc_product(sums[0], zi, ri);
                reset_flow(m_old + i);
                reset_flow(q_old + i);
            }
            T acc = in.finish(a.ci, a.val, part_off<kFlowU>(s), part_len<kFlowU>(s), cols, noff, nlen, lane, m_pub, dv, st, 72, live);
            acc = row_sum<T>(acc, s.shift);
            if (row.own) st_flow(m_pub + row.i, acc * wdv);
        });
        // forward sweep (:1533-1571)
        flow_sweep<kFlowL, false>(w, a.ci, [&](const FlowSlice& s, FlowCols& cols, long long noff, int nlen) {
            const FlowRow row = flow_row(s, lane);
            FlowGather<T> in;
            in.begin(a.ci, a.val, part_off<kFlowL>(s), part_len<kFlowL>(s), cols, noff, nlen, lane, q_pub);
            T dv = T(0), mv = T(0), sdv = T(0), wdv = T(0), ri = T(0), acc = T(0);
            if (row.own) {
                const int i = row.i;
                dv = a.d[i];
                mv = ld_flow(m_pub + i);
                sdv = __ldg(&a.sd[i]);
                wdv = __ldg(&a.wd[i]);
                ri = a.r[i];
                acc = fma(-sdv, mv, dv);
            }
            acc = in.finish(a.ci, a.val, part_off<kFlowL>(s), part_len<kFlowL>(s), cols, noff, nlen, lane, q_pub, acc, st, 73, live);
            acc = row_sum<T>(acc, s.shift);
            if (row.own) {
                const T qv = acc * wdv;
                st_flow(q_pub + row.i, qv);
                const T wv = qv + mv;
                a.w[row.i] = wv;
                const T sw = wv * sdv;
                sums[1] = acc_product(sums[1], wv, dv);
                sums[2] = acc_product(sums[2], ri, sw);
                sums[3] = acc_product(sums[3], wv, sw);
            }
        });
        if (!flow_reduce<T, 4>(sums, a.partials + (K & 1) * 4 * gridDim.x, st, epoch, 74, live, sh, tot)) return;
        if (threadIdx.x == 0) {
            z_r_prev = K > 0 ? z_r : tot[0];
            z_r = tot[0];
            const double d_Ad = tot[1];
            int ctl = kGoOn;
            if (K > 0) {
                if (a.print_modulo > 0 && K % a.print_modulo == 0 && blockIdx.x == 0)
                    printf("(%d/%d)   INTERIM: Residual norm is %.9le < %.9le\n", K, a.n, sqrt(z_r), a.print_tol);
                if (a.use_zr_rule && abs_below(z_r, a.tol2)) ctl = kConverged;
                if (a.rr_stop > 0.0 && z_r < a.rr_stop * z_r0) ctl = kConverged;
            }
            const bool bad = !isfinite(z_r) || below_zero(z_r) || !isfinite(d_Ad) || below_zero(d_Ad);   // :918-933
            const bool tiny = !bad && energy_small(d_Ad);
            if (ctl == kConverged) {
                // an inner solve (no reference rule) takes the step it has already paid for
                if (!a.use_zr_rule && !bad && !tiny) ctl = kLastStep;
            } else if (bad) {
                ctl = kBreakdown;
            } else if (tiny) {
                ctl = kSmallEnergy;
            }
            const double al = z_r / d_Ad;
            s_scal[0] = al;
            s_scal[1] = fma(al, fma(al, tot[3], -2.0 * tot[2]), z_r) / z_r;
            s_ctl = ctl;
        }
        __syncthreads();
        const int ctl = s_ctl;
        if (ctl == kBreakdown) { status = FEEC_BREAKDOWN; break; }
        if (ctl == kSmallEnergy) { status = FEEC_SMALL_ENERGY; break; }
        if (ctl == kConverged) { status = FEEC_OK; break; }
        K++;
        if (ctl == kLastStep || K >= a.max_iter) {
            if (ctl == kLastStep) status = FEEC_OK;
            step = true;
            break;
        }
    }
    double zr_last[1] = {0.0};
    if (step) {
        Acc last[1] = {AT::zero()};
        const T alpha = (T)s_scal[0];
        T* const m_pub = a.pub[(K - 1) & 1];
        for (int j = 0; j < mine; j++) {
            const FlowSlice s = flow_slice(w.raw(j));
            const FlowRow row = flow_row(s, lane);
            if (row.own) {
                const T ri = fma(-alpha, a.w[row.i], a.r[row.i]);
                a.x[row.i] = fma(alpha, ld_flow(m_pub + row.i), a.x[row.i]);
                a.r[row.i] = ri;
                last[0] = acc_product(last[0], T(ri * __ldg(&a.sd[row.i])), ri);
            }
        }
        // the reported z.r is that of the final r, summed, not the expansion that beta is made of
        if (!flow_reduce<T, 1>(last, a.partials + (K & 1) * 4 * gridDim.x, st, epoch, 75, live, sh, zr_last)) return;
    }
    finish(st, status, K, step ? zr_last[0] : z_r, 0.0);
    if (blockIdx.x == 0 && threadIdx.x == 0) st->extra[0] = step ? z_r : z_r_prev;
}

// ---------------------------------------------------------------------------
// SSOR-PCG over full rows: q = A d, then the forward and backward sweeps. Published: d in
// pub[0] (gathered by the product), m in pub[1] (forward sweep), z in pub[2] (backward
// sweep). m and z are reset while d is published (their gathers ended before the z.r sum)
// and d in the forward sweep (its gathers ended before the d.q sum). Measured, 3D P2 refined 5
// times: 259 -> 97 us per iteration.
// ---------------------------------------------------------------------------
__global__ void __launch_bounds__(kFlowThreads, 1) flow_pcg(FlowArgs<double> a) {
    __shared__ FlowShared sh;
    __shared__ double s_scal[2];
    __shared__ int s_ctl;
    FlowWarp w;
    w.init(a.meta, a.nslices);
    const int lane = w.lane, mine = w.mine;
    unsigned long long epoch = 0;
    bool live = true;
    DeviceStatus* st = a.st;
    double* const d_pub = a.pub[0];
    double* const m_pub = a.pub[1];
    double* const z_pub = a.pub[2];

    // r = b - A x (restart, :1072-1116) or x += alpha d, r -= alpha q (:1230-1240), then the
    // forward sweep (:1118-1140 / :1241-1261)
    auto forward = [&](bool restart, double alpha) {
        flow_sweep<kFlowL, false>(w, a.ci, [&](const FlowSlice& s, FlowCols& cols, long long noff, int nlen) {
            const FlowRow row = flow_row(s, lane);
            FlowGather<double> in;
            in.begin(a.ci, a.val, part_off<kFlowL>(s), part_len<kFlowL>(s), cols, noff, nlen, lane, m_pub);
            const int i = row.i;
            double ri = 0.0, wdv = 0.0;
            if (row.own) wdv = __ldg(&a.wd[i]);
            if (restart) {
                ri = row.own ? __ldg(&a.b[i]) : 0.0;
                ri = direct_minus<double>(a.ci, a.val, s.off, part_len<kFlowAll>(s), lane, a.x, ri);
                ri = row_sum<double>(ri, s.shift);
                if (row.own) a.r[i] = ri;
                else ri = 0.0;
            } else if (row.own) {
                a.x[i] = fma(alpha, a.d[i], a.x[i]);
                ri = fma(-alpha, a.q[i], a.r[i]);
                a.r[i] = ri;
                reset_flow(d_pub + i);
            }
            double acc = in.finish(a.ci, a.val, part_off<kFlowL>(s), part_len<kFlowL>(s), cols, noff, nlen, lane, m_pub, ri, st, 80, live);
            acc = row_sum<double>(acc, s.shift);
            if (row.own) st_flow(m_pub + i, acc * wdv);
        });
    };
    // scaling and backward sweep (:1142-1170 / :1263-1307); returns the lane's part of z.r
    auto backward = [&]() {
        double zr = 0.0;
        flow_sweep<kFlowU, true>(w, a.ci, [&](const FlowSlice& s, FlowCols& cols, long long noff, int nlen) {
            const FlowRow row = flow_row(s, lane);
            FlowGather<double> in;
            in.begin(a.ci, a.val, part_off<kFlowU>(s), part_len<kFlowU>(s), cols, noff, nlen, lane, z_pub);
            const int i = row.i;
            double acc = 0.0, wdv = 0.0, ri = 0.0;
            if (row.own) {
                acc = ld_flow(m_pub + i) * __ldg(&a.sd[i]);
                wdv = __ldg(&a.wd[i]);
                ri = a.r[i];
            }
            acc = in.finish(a.ci, a.val, part_off<kFlowU>(s), part_len<kFlowU>(s), cols, noff, nlen, lane, z_pub, acc, st, 81, live);
            acc = row_sum<double>(acc, s.shift);
            if (row.own) {
                const double zi = acc * wdv;
                st_flow(z_pub + i, zi);
                zr = fma(zi, ri, zr);
            }
        });
        return zr;
    };

    forward(true, 0.0);
    double one[1] = {backward()}, tot[1];
    if (!flow_reduce<double, 1>(one, a.partials, st, epoch, 82, live, sh, tot)) return;
    double z_r = tot[0];
    int K = 0, status = FEEC_MAXITER;
    double beta = 0.0;
    for (;;) {
        if (threadIdx.x == 0) {
            if (a.print_modulo > 0 && K % a.print_modulo == 0 && blockIdx.x == 0)
                printf("(%d/%d)   INTERIM: Residual norm is %.9le < %.9le\n", K, a.n, sqrt(z_r), a.print_tol);
            s_ctl = (a.use_zr_rule && abs_below(z_r, a.tol2)) ? kConverged : kGoOn;       // :1187-1190
        }
        __syncthreads();
        if (s_ctl == kConverged) { status = FEEC_OK; break; }
        // d = z + beta d (:1309-1318), published; q = A d, d.q (:1197-1212)
        for (int j = 0; j < mine; j++) {
            const FlowSlice s = flow_slice(w.raw(j));
            const FlowRow row = flow_row(s, lane);
            if (row.own) {
                const int i = row.i;
                double dv = ld_flow(z_pub + i);
                if (K > 0) dv = fma(beta, a.d[i], dv);
                a.d[i] = dv;
                st_flow(d_pub + i, dv);
                reset_flow(z_pub + i);
                reset_flow(m_pub + i);
            }
        }
        double dq = 0.0;
        flow_sweep<kFlowAll, false>(w, a.ci, [&](const FlowSlice& s, FlowCols& cols, long long noff, int nlen) {
            const FlowRow row = flow_row(s, lane);
            FlowGather<double> in;
            in.begin(a.ci, a.val, part_off<kFlowAll>(s), part_len<kFlowAll>(s), cols, noff, nlen, lane, d_pub);
            double acc = in.finish(a.ci, a.val, part_off<kFlowAll>(s), part_len<kFlowAll>(s), cols, noff, nlen, lane, d_pub, 0.0, st, 83, live);
            acc = row_sum<double>(acc, s.shift);
            if (row.own) {
                a.q[row.i] = -acc;
                dq = fma(-acc, a.d[row.i], dq);
            }
        });
        one[0] = dq;
        if (!flow_reduce<double, 1>(one, a.partials + 4 * gridDim.x, st, epoch, 84, live, sh, tot)) return;
        if (threadIdx.x == 0) {
            const double d_Ad = tot[0];
            int ctl = kGoOn;
            if (!isfinite(z_r) || below_zero(z_r) || !isfinite(d_Ad) || below_zero(d_Ad)) ctl = kBreakdown;
            else if (energy_small(d_Ad)) ctl = kSmallEnergy;
            s_ctl = ctl;
            s_scal[0] = z_r / d_Ad;
        }
        __syncthreads();
        if (s_ctl == kBreakdown) { status = FEEC_BREAKDOWN; break; }
        if (s_ctl == kSmallEnergy) { status = FEEC_SMALL_ENERGY; break; }
        forward(false, s_scal[0]);
        one[0] = backward();
        if (!flow_reduce<double, 1>(one, a.partials, st, epoch, 85, live, sh, tot)) return;
        if (threadIdx.x == 0) {
            s_scal[1] = tot[0] / z_r;
            z_r = tot[0];
        }
        __syncthreads();
        beta = s_scal[1];
        K++;
        if (K >= a.max_iter) break;
    }
    finish(st, status, K, z_r, 0.0);
}

// Fills the slices: entry number p of a part of row row0 + r goes to lane r << shift | (p mod
// 2^shift), column p >> shift. L is ordered by ascending column and U by descending column:
// colors are contiguous in the permuted numbering, so that is the order in which the sweeps
// publish them. Padding: column -1, value 0. A part of more than kRankSegment entries is ordered
// within segments of that many, so that the set-up stays linear in a row's length: the order only
// decides which entry is waited for first. (Ranked against the whole part, a row of 200,000 entries
// took 36 s of set-up; 40 ms so.)
constexpr int kRankSegment = 256;
__global__ void flow_fill_kernel(int nslices, const int4* __restrict__ meta, const int* __restrict__ rp,
                                 const int* __restrict__ lsplit, const int* __restrict__ usplit,
                                 const int* __restrict__ ci_in, const double* __restrict__ val_in, int* __restrict__ ci,
                                 double* __restrict__ val64, float* __restrict__ val32) {
    const int sl = blockIdx.x * (blockDim.x / 32) + threadIdx.x / 32;
    const int lane = threadIdx.x & 31;
    if (sl >= nslices) return;
    const FlowSlice s = flow_slice(__ldg(&meta[sl]));
    const int width = 1 << s.shift, r = lane >> s.shift, t = lane & (width - 1);
    const bool act = r < s.nrow;
    const int i = s.row0 + r;
    const int lo = act ? rp[i] : 0, l = act ? lsplit[i] : 0, u = act ? usplit[i] : 0, hi = act ? rp[i + 1] : 0;
    const int from[3] = {lo, l, u}, to[3] = {l, u, hi}, len[3] = {s.len_l, s.len_e, s.len_u};
    long long o = s.off;
    for (int part = 0; part < 3; part++) {
        const int a = from[part], count = to[part] - a;
        for (int j = t; j < count; j += width) {
            const int c = ci_in[a + j];
            const int from_h = j & ~(kRankSegment - 1), to_h = min(count, from_h + kRankSegment);
            int rank = from_h;
            for (int h = from_h; h < to_h; h++) {
                const int ch = ci_in[a + h];
                rank += (part == 2 ? ch > c : ch < c) || (ch == c && h < j);
            }
            const long long dst = o + 32ll * (rank >> s.shift) + (r << s.shift) + (rank & (width - 1));
            const double v = val_in[a + j];
            if (ci) ci[dst] = c;
            if (val64) val64[dst] = v;
            if (val32) val32[dst] = (float)v;
        }
        for (int p = count + ((t - count) & (width - 1)); p < (len[part] << s.shift); p += width) {   // this lane's padding
            const long long dst = o + 32ll * (p >> s.shift) + lane;
            if (ci) ci[dst] = -1;
            if (val64) val64[dst] = 0.0;
            if (val32) val32[dst] = 0.0f;
        }
        o += 32ll * len[part];
    }
}

}  // namespace

cudaError_t flow_fill(int nslices, const int4* meta, const int* rp, const int* lsplit, const int* usplit, const int* ci_in,
                      const double* val_in, int* ci, double* val64, float* val32, cudaStream_t st) {
    if (nslices <= 0) return cudaSuccess;
    note_launch();
    flow_fill_kernel<<<(nslices + 7) / 8, 256, 0, st>>>(nslices, meta, rp, lsplit, usplit, ci_in, val_in, ci, val64, val32);
    return cudaGetLastError();
}

// Builds the slices of the multicolor layout (lazily, kept until the layout changes) and the
// values of the wanted precision.
int flow_build(feec_system* s, bool f32) {
    FlowData& D = s->flow;
    if (D.ready && (f32 ? (void*)D.val32 : (void*)D.val64)) return FEEC_OK;
    HomeStreamScope home(s);
    cudaStream_t st = s->stream;
    const int n = s->n;
    const bool first = !D.ready;
    if (first) {
        D.mem.release();
        D = FlowData{};
        D.mem.stream = st;
        int sms = 0;
        FEEC_TRY(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, s->dev));
        const int e = cut_colors(D, st, sms, s->color_ranges, s->rp, s->lsplit, s->usplit);
        if (e != FEEC_OK) return e;
        FEEC_TRY(D.mem.alloc(D.ci, (size_t)D.units * 32));
        FEEC_TRY(alloc_published(D, 4, n));
    }
    if (f32) FEEC_TRY(D.mem.alloc(D.val32, (size_t)D.units * 32));
    else FEEC_TRY(D.mem.alloc(D.val64, (size_t)D.units * 32));
    FEEC_TRY(flow_fill(D.nslices, D.meta, s->rp, s->lsplit, s->usplit, s->ci, s->val, first ? D.ci : nullptr,
                       f32 ? nullptr : D.val64, f32 ? D.val32 : nullptr, st));
    D.ready = true;
    return FEEC_OK;
}

namespace {

template <typename T>
int flow_launch(feec_system* s, const PcgArgs<T>& p, const void* fn, LaunchShape& shape) {
    const FlowData& D = s->flow;
    FlowArgs<T> a{};
    a.n = p.n; a.nslices = D.nslices; a.meta = D.meta; a.ci = D.ci;
    if constexpr (sizeof(T) == 8) a.val = D.val64;
    else a.val = D.val32;
    a.wd = p.wd; a.sd = p.sd; a.b = p.b; a.x = p.x; a.r = p.r; a.d = p.d; a.w = p.w; a.q = p.q;
    for (int k = 0; k < 4; k++) {
        a.pub[k] = reinterpret_cast<T*>(D.pub[k]);
        FEEC_TRY(cudaMemsetAsync(a.pub[k], 0xFF, sizeof(T) * (size_t)p.n, s->stream));
    }
    a.tol2 = p.tol2; a.rr_stop = p.rr_stop; a.use_zr_rule = p.use_zr_rule; a.max_iter = p.max_iter;
    a.print_modulo = p.print_modulo; a.print_tol = p.print_tol; a.partials = p.partials; a.st = p.st;
    a.keep_dir = p.keep_dir; a.zr_prev = p.zr_prev; a.scale = p.scale;
    int sms = 0;
    FEEC_TRY(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, s->dev));
    // One warp per scheduler and block before there are more blocks, as for plain CG: alone, a solve
    // takes the same time as over all SMs, and small solves on several streams share them (solves
    // per ms, 8 streams, blocks of 512 threads -> these: 2D P1, 1,089 rows FP64 1.74 -> 5.40, 8,500 rows
    // 0.35 -> 0.72, 6,000 rows by the two-sweep form 0.30 -> 1.29; 3D P1, 4,913 rows 0.53 -> 1.01).
    shape.blocks = std::max(1, std::min(sms, (D.nslices + 3) / 4));
    shape.threads = 32 * std::min((D.nslices + shape.blocks - 1) / shape.blocks, kFlowWarps);
    shape.lanes = 1;
    void* args[] = {&a};
    note_launch();
    FEEC_TRY(cudaLaunchCooperativeKernel(fn, dim3(shape.blocks), dim3(shape.threads), args, 0, s->stream));
    return FEEC_OK;
}

}  // namespace

int launch_flow_eisenstat(feec_system* s, const PcgArgs<double>& a, LaunchShape& shape) {
    return flow_launch<double>(s, a, (const void*)flow_eisenstat<double>, shape);
}
int launch_flow_eisenstat(feec_system* s, const PcgArgs<float>& a, LaunchShape& shape) {
    return flow_launch<float>(s, a, (const void*)flow_eisenstat<float>, shape);
}
int launch_flow_pcg(feec_system* s, const PcgArgs<double>& a, LaunchShape& shape) {
    return flow_launch<double>(s, a, (const void*)flow_pcg, shape);
}

}  // namespace feec
