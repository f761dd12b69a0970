// MINRES (MINRESCSR, solver/sparsesolver.cpp:2159-2425) and conjugate residuals
// (ConjugateResidualSolverCSR, :1687-1915, and its _textbook twin, :1918-2156) with one grid-wide
// sum per iteration, one cooperative launch per solve.
//
// The barrier-phase kernels (minres_persistent, cr_persistent) spend three and two grid barriers
// and as many block-wide FP64 reductions on an iteration. Here the vector that the product gathers
// is published row by row (flow_device.cuh), and the norm that the reference sums after the update
// is expanded from sums taken before it:
//   MINRES  t = A v1 - gamma v0, vn = t - delta v1:  vn.vn = t.t - 2 delta t.v1 + delta^2 v1.v1
//   CR      Adir' = Ares + beta Adir:  Adir'.Adir' = Ares.Ares + 2 beta Ares.Adir + beta^2 Adir.Adir
// all of them actual sums of the vectors at hand. Where the expansion cancels to less than kCancel
// of its terms, the norm is summed from the vector itself, with a reduction of its own: at 0.1 the
// iteration counts are the reference's to 2 on every fixture (at 1e-3 one of them, conjugate
// residuals on 343 rows of 3D P3, ends 5 of 175 steps early; with every norm summed 4 early), and
// the solves take the same time; summing every norm takes 1.4 times as long.
// Rows, slices and the two forms (vectors in registers or in memory) are those of plain CG
// (kernels_flow_cg.cu). What is left of an iteration is one publication's way through L2, the
// product and one reduction. Host calls against the barrier-phase kernels, to 1e-12: 3D P1 refined
// 5 times (35,937 rows) MINRES 6.85 -> 3.50 ms (358 iterations, 18.3 -> 8.6 us each), CR 4.50 ->
// 3.08; 3D P2 refined 4 times (35,937 rows, 27 entries each) 14.7 -> 6.6 and 11.5 -> 5.8; 2D P1
// refined 5 times (1,089 rows) 3.53 -> 1.53 and 2.43 -> 1.49.
#include <cmath>
#include <cstdio>

#include "flow_device.cuh"
#include "feec_system.h"
#include "flow_more.h"
#include "persistent_common.cuh"

namespace feec {
namespace {

constexpr double kCancel = 0.1;

// One row per lane group with its entries in registers (every lane of the group carries the row),
// or all of a warp's slices with the vectors in memory.
template <bool REG>
struct Rows {
    FlowWarp w;
    FlowSlice s;
    FlowCols cols;
    double v[kFlowChunk];
    int i;
    bool in, own;            // the lane carries a row; it is the row's first lane

    __device__ __forceinline__ void init(const FlowMoreArgs& a) {
        w.init(a.meta, a.nslices);
        if constexpr (REG) {
            s = flow_slice(w.raw(0));
            const FlowRow r = flow_row(s, w.lane);
            i = r.i; own = r.own;
            in = (w.lane >> s.shift) < s.nrow;
            cols.load(a.ci, s.off, s.len_u, w.lane);
            #pragma unroll
            for (int u = 0; u < kFlowChunk; u++) v[u] = u < s.len_u ? __ldg(a.val + s.off + 32 * u + w.lane) : 0.0;
        }
    }
    // body(i) for the rows the lane owns
    template <typename F>
    __device__ __forceinline__ void each(F&& body) {
        for (int j = 0; j < w.mine; j++) {
            const FlowSlice q = flow_slice(w.raw(j));
            const FlowRow r = flow_row(q, w.lane);
            if (r.own) body(r.i);
        }
    }
    // body(i, own, b - A x) for every slice, x unchanged while it is read
    template <typename F>
    __device__ __forceinline__ void residual(const FlowMoreArgs& a, F&& body) {
        for (int j = 0; j < w.mine; j++) {
            const FlowSlice q = flow_slice(w.raw(j));
            const FlowRow r = flow_row(q, w.lane);
            double acc = r.own ? __ldg(&a.b[r.i]) : 0.0;
            acc = row_sum<double>(direct_minus<double>(a.ci, a.val, q.off, q.len_u, w.lane, a.x, acc), q.shift);
            body(r.i, r.own, acc);
        }
    }
    // REG: (A X)[i] of the published X, in every lane of the row
    __device__ __forceinline__ double product(const double* X, DeviceStatus* st, int site, bool& live) {
        if (w.mine == 0) return 0.0;
        FlowGather<double> in_flight;
        #pragma unroll
        for (int u = 0; u < kFlowChunk; u++) {
            in_flight.g[u] = 0.0;
            if (cols.c[u] >= 0) in_flight.g[u] = ld_flow(X + cols.c[u]);
            in_flight.v[u] = v[u];
        }
        return -row_sum<double>(in_flight.wait(cols, s.len_u, X, 0.0, st, site, live), s.shift);
    }
    // otherwise: body(i, own, (A X)[i]) for every slice; pre(i) is called for owned rows while the
    // gathers travel
    template <typename Pre, typename F>
    __device__ __forceinline__ void products(const FlowMoreArgs& a, const double* X, int site, bool& live, Pre&& pre, F&& body) {
        flow_sweep<kFlowU, false>(w, a.ci, [&](const FlowSlice& q, FlowCols& c, long long noff, int nlen) {
            const FlowRow r = flow_row(q, w.lane);
            FlowGather<double> in_flight;
            in_flight.begin(a.ci, a.val, q.off, q.len_u, c, noff, nlen, w.lane, X);
            if (r.own) pre(r.i);
            const double acc = in_flight.finish(a.ci, a.val, q.off, q.len_u, c, noff, nlen, w.lane, X, 0.0, a.st, site, live);
            body(r.i, r.own, -row_sum<double>(acc, q.shift));
        });
    }
};

// Four sums of products p[k] q[k] of one row per lane group: spread over four of the row's lanes
// where it has them (a warp's FP64 operation takes its scheduler 64 cycles whatever its active
// lanes: 4 operations instead of 10).
__device__ __forceinline__ bool reduce_row4(const Rows<true>& rows, const double (&p)[4], const double (&q)[4], double* part,
                                            DeviceStatus* st, unsigned long long& epoch, int site, bool live, FlowShared& sh,
                                            double (&tot)[4]) {
    const int lane = rows.w.lane, shift = rows.s.shift;
    if (shift >= 2) {
        // lanes beyond a row's fourth hold 0, so the tree over strides from 4 adds each row once
        const int t = lane & ((1 << shift) - 1);
        double k = rows.in && t < 4 ? (t == 0 ? p[0] : t == 1 ? p[1] : t == 2 ? p[2] : p[3]) *
                                          (t == 0 ? q[0] : t == 1 ? q[1] : t == 2 ? q[2] : q[3]) : 0.0;
        for (int off = 4; off < 32; off <<= 1) k += __shfl_xor_sync(0xffffffffu, k, off);
        if (lane < 4) sh.warp_sum[threadIdx.x >> 5][lane] = k;
    } else {
        double sums[4] = {0.0, 0.0, 0.0, 0.0};
        if (rows.own)
            #pragma unroll
            for (int k = 0; k < 4; k++) sums[k] = p[k] * q[k];
        flow_warp_sums<double, 4>(sums, sh);
    }
    return flow_reduce_warps<4>(part, st, epoch, site, live, sh, tot);
}

struct MoreControl {
    double a, b, c, d, e, f;
    int status;      // -1: go on
    int exact;       // the expanded norm cancelled: sum it
};

// ---------------------------------------------------------------------------
// MINRES
// ---------------------------------------------------------------------------

// Scalar state, in warp 0 of every block (identical bits in every block).
struct MinresState {
    double gamma, eta, s0, s1, c0, c1;
};

// Rotations of one step (:2338-2362) from delta and vn.vn. The two square roots and the four
// divisions run in different lanes at once. Out: a = alpha_2, b = alpha_3, c = 1 / alpha_1,
// d = cn eta, e = 1 / gamma_n, f = gamma_n.
__device__ __forceinline__ void minres_rotate(MinresState& m, double delta, double gn2, int K, int n, double tol,
                                              int print_modulo, MoreControl& c) {
    const int lane = threadIdx.x & 31;
    const double alpha_0 = m.c1 * delta - m.c0 * m.s1 * m.gamma;
    const double alpha_2 = m.s1 * delta + m.c0 * m.c1 * m.gamma;
    const double alpha_3 = m.s0 * m.gamma;
    const double root = sqrt(lane == 0 ? gn2 : fma(alpha_0, alpha_0, gn2));
    const double gamma_n = __shfl_sync(0xffffffffu, root, 0), alpha_1 = __shfl_sync(0xffffffffu, root, 1);
    const double div = (lane == 0 ? alpha_0 : lane == 1 ? gamma_n : 1.0) / (lane == 3 ? gamma_n : alpha_1);
    const double cn = __shfl_sync(0xffffffffu, div, 0), sn = __shfl_sync(0xffffffffu, div, 1);
    const double inv_a = __shfl_sync(0xffffffffu, div, 2), inv_g = __shfl_sync(0xffffffffu, div, 3);
    if (lane == 0) {
        c.a = alpha_2; c.b = alpha_3; c.c = inv_a; c.d = cn * m.eta; c.e = inv_g; c.f = gamma_n;
        c.exact = 0;
    }
    m.eta = -sn * m.eta;
    m.c0 = m.c1; m.s0 = m.s1; m.c1 = cn; m.s1 = sn;
    m.gamma = gamma_n;
    if (lane == 0) {
        if (blockIdx.x == 0 && print_modulo > 0 && K % print_modulo == 0)
            printf("(%d/%d)   INTERIM: Residual norm is %.9le < %.9le\n", K, n, m.eta, tol);
        c.status = abs_below(m.eta, tol) ? FEEC_OK : -1;                                    // :2290-2293
    }
}

template <bool REG>
__global__ void __launch_bounds__(kFlowThreads, 1) flow_minres(FlowMoreArgs a) {
    __shared__ FlowShared sh;
    __shared__ MoreControl ctl;
    __shared__ double s_delta;
    Rows<REG> rows;
    rows.init(a);
    unsigned long long epoch = 0;
    bool live = true;
    DeviceStatus* st = a.st;
    int turn = 0, K = 0, status = FEEC_MAXITER;
    auto part = [&]() { return a.partials + (turn++ & 1) * 4 * gridDim.x; };
    double *v0 = a.w[0], *v1 = a.w[1], *w0 = a.w[2], *w1 = a.w[3], *t = a.w[4];
    double x_ = 0.0, v0_ = 0.0, v1_ = 0.0, w0_ = 0.0, w1_ = 0.0, t_ = 0.0;      // REG

    // restart (:2233-2283): v0 = w0 = w1 = 0, v1 = (b - A x) / gamma
    {
        double acc[1] = {0.0}, sum[1];
        rows.residual(a, [&](int i, bool own, double r) {
            if constexpr (REG) v1_ = r;
            if (own) {
                if constexpr (REG) { }
                else { v0[i] = 0.0; w0[i] = 0.0; w1[i] = 0.0; v1[i] = r; }
                acc[0] = fma(r, r, acc[0]);
            }
        });
        if constexpr (REG)
            if (rows.in) x_ = a.x[rows.i];
        if (!flow_reduce<double, 1>(acc, part(), st, epoch, 96, live, sh, sum)) return;
        if (threadIdx.x < 32) {
            const double gamma = sqrt(sum[0]);
            if (threadIdx.x == 0) { ctl.e = 1.0 / gamma; ctl.f = gamma; ctl.status = abs_below(gamma, a.tol) ? FEEC_OK : -1; }
        }
        __syncthreads();
    }
    MinresState m{ctl.f, ctl.f, 0.0, 0.0, 1.0, 1.0};
    double gamma = ctl.f;
    {
        const double inv = ctl.e;
        if constexpr (REG) v1_ *= inv;
        else rows.each([&](int i) { v1[i] *= inv; });
    }
    status = ctl.status;
    while (status < 0) {
        double* const pub = a.pub[K & 1];
        double* const old = a.pub[(K & 1) ^ 1];
        double tot[4];
        // t = A v1 - gamma v0; sums [delta = p.v1, t.t, t.v1, v1.v1] (:2297-2313)
        if constexpr (REG) {
            if (rows.own) { st_flow(pub + rows.i, v1_); reset_flow(old + rows.i); }
            const double p = rows.product(pub, st, 97, live);
            t_ = fma(-gamma, v0_, p);
            const double f[4] = {p, t_, t_, v1_}, g[4] = {v1_, t_, v1_, v1_};
            if (!reduce_row4(rows, f, g, part(), st, epoch, 98, live, sh, tot)) return;
        } else {
            rows.each([&](int i) { st_flow(pub + i, v1[i]); reset_flow(old + i); });
            double sums[4] = {0.0, 0.0, 0.0, 0.0};
            double mine = 0.0, last = 0.0;
            rows.products(a, pub, 97, live, [&](int i) { mine = v1[i]; last = v0[i]; }, [&](int i, bool own, double p) {
                if (own) {
                    const double ti = fma(-gamma, last, p);
                    t[i] = ti;
                    sums[0] = fma(p, mine, sums[0]);
                    sums[1] = fma(ti, ti, sums[1]);
                    sums[2] = fma(ti, mine, sums[2]);
                    sums[3] = fma(mine, mine, sums[3]);
                }
            });
            if (!flow_reduce<double, 4>(sums, part(), st, epoch, 98, live, sh, tot)) return;
        }
        if (threadIdx.x < 32) {
            const double delta = tot[0];
            const double gn2 = fma(delta, fma(delta, tot[3], -2.0 * tot[2]), tot[1]);
            const bool cancelled = !(gn2 >= kCancel * tot[1]);
            if (threadIdx.x == 0) { s_delta = delta; ctl.exact = cancelled; }
            __syncwarp();
            if (!cancelled) minres_rotate(m, delta, gn2, K, a.n, a.tol, a.print_modulo, ctl);
        }
        __syncthreads();
        const double delta = s_delta;
        if (ctl.exact) {
            double acc[1] = {0.0}, sum[1];
            if constexpr (REG) {
                const double u = fma(-delta, v1_, t_);
                if (rows.own) acc[0] = u * u;
            } else {
                rows.each([&](int i) {
                    const double u = fma(-delta, v1[i], t[i]);
                    acc[0] = fma(u, u, acc[0]);
                });
            }
            if (!flow_reduce<double, 1>(acc, part(), st, epoch, 99, live, sh, sum)) return;
            if (threadIdx.x < 32) minres_rotate(m, delta, sum[0], K, a.n, a.tol, a.print_modulo, ctl);
            __syncthreads();
        }
        const double alpha_2 = ctl.a, alpha_3 = ctl.b, inv_a = ctl.c, ce = ctl.d, inv_g = ctl.e;
        gamma = ctl.f;
        status = ctl.status;
        // :2332-2378: wn = (v1 - alpha_2 w1 - alpha_3 w0) / alpha_1, x += cn eta wn, the next v1
        if constexpr (REG) {
            const double wn = fma(-alpha_3, w0_, fma(-alpha_2, w1_, v1_)) * inv_a;
            const double vn = fma(-delta, v1_, t_) * inv_g;
            x_ = fma(ce, wn, x_);
            w0_ = w1_; w1_ = wn;
            v0_ = v1_; v1_ = vn;
        } else {
            rows.each([&](int i) {
                const double vi = v1[i];
                const double wn = fma(-alpha_3, w0[i], fma(-alpha_2, w1[i], vi)) * inv_a;
                a.x[i] = fma(ce, wn, a.x[i]);
                w0[i] = wn;
                v0[i] = fma(-delta, vi, t[i]) * inv_g;
            });
            double* s = v0; v0 = v1; v1 = s;      // the new vectors replaced the oldest ones
            s = w0; w0 = w1; w1 = s;
        }
        K++;
        if (K >= a.max_iter) { status = FEEC_MAXITER; break; }
    }
    // :2397-2403: res = b - A x
    if constexpr (REG)
        if (rows.own) a.x[rows.i] = x_;
    if (!grid_barrier(st, epoch, 100)) return;
    rows.residual(a, [&](int i, bool own, double r) {
        if (own) a.res[i] = r;
    });
    finish(st, status, K, m.eta, gamma);
}

// ---------------------------------------------------------------------------
// Conjugate residuals
// ---------------------------------------------------------------------------

// Stopping rules and the step (:1804-1840) from Ad_r and Ad_Ad; a = alpha.
__device__ __forceinline__ void cr_step(double ad_r, double ad_ad, int K, int n, double tol, int print_modulo, MoreControl& c) {
    if ((threadIdx.x & 31) != 0) return;
    if (print_modulo > 0 && K % print_modulo == 0 && blockIdx.x == 0)
        printf("(%d/%d)   INTERIM: Residual norm is %.9le < %.9le\n", K, n, sqrt(ad_r), tol);
    int status = -1;
    if (!isfinite(ad_r) || below_zero(ad_r)) status = FEEC_BREAKDOWN;
    else if (abs_below(ad_r, tol * tol)) status = FEEC_OK;
    else if (!isfinite(ad_ad) || below_zero(ad_ad)) status = FEEC_BREAKDOWN;
    else if (energy_small(ad_ad)) status = FEEC_SMALL_ENERGY;
    c.status = status;
    c.a = ad_r / ad_ad;
}

template <bool REG>
__global__ void __launch_bounds__(kFlowThreads, 1) flow_cr(FlowMoreArgs a) {
    __shared__ FlowShared sh;
    __shared__ MoreControl ctl;
    Rows<REG> rows;
    rows.init(a);
    unsigned long long epoch = 0;
    bool live = true;
    DeviceStatus* st = a.st;
    int turn = 0, K = 0, status = FEEC_MAXITER;
    auto part = [&]() { return a.partials + (turn++ & 1) * 4 * gridDim.x; };
    double *dir = a.w[0], *adir = a.w[1], *ares = a.w[2];
    double x_ = 0.0, r_ = 0.0, dir_ = 0.0, adir_ = 0.0, ares_ = 0.0;            // REG
    double ad_r = 0.0, ad_ad = 0.0;                                             // warp 0

    // restart (:1749-1790): res = b - A x, dir = res, Adir = A dir, Ares = Adir
    rows.residual(a, [&](int i, bool own, double r) {
        if constexpr (REG) { r_ = r; dir_ = r; }
        if (own) {
            if constexpr (!REG) { a.res[i] = r; dir[i] = r; }
            st_flow(a.pub[0] + i, r);
        }
    });
    {
        double acc[2] = {0.0, 0.0}, sum[2];
        if constexpr (REG) {
            if (rows.in) x_ = a.x[rows.i];
            adir_ = rows.product(a.pub[0], st, 101, live);
            ares_ = adir_;
            if (rows.own) { acc[0] = adir_ * r_; acc[1] = adir_ * adir_; }
        } else {
            double r = 0.0;
            rows.products(a, a.pub[0], 101, live, [&](int i) { r = a.res[i]; }, [&](int i, bool own, double s) {
                if (own) {
                    adir[i] = s;
                    ares[i] = s;
                    acc[0] = fma(s, r, acc[0]);
                    acc[1] = fma(s, s, acc[1]);
                }
            });
        }
        if (!flow_reduce<double, 2>(acc, part(), st, epoch, 102, live, sh, sum)) return;
        if (threadIdx.x < 32) {
            ad_r = sum[0]; ad_ad = sum[1];
            cr_step(ad_r, ad_ad, 0, a.n, a.tol, a.print_modulo, ctl);
        }
        __syncthreads();
    }
    while (true) {
        status = ctl.status;
        if (status >= 0) break;
        const double alpha = ctl.a;
        double* const pub = a.pub[(K & 1) ^ 1];
        double* const old = a.pub[K & 1];
        double tot[4];
        // :1846-1863: vil = A Adir; x, res, Ares; sums [Ares.res, Ares.Ares, Ares.Adir, Adir.Adir]
        if constexpr (REG) {
            if (rows.own) { st_flow(pub + rows.i, adir_); reset_flow(old + rows.i); }
            const double vil = rows.product(pub, st, 103, live);
            x_ = fma(alpha, dir_, x_);
            r_ = fma(-alpha, adir_, r_);
            ares_ = fma(-alpha, vil, ares_);
            const double f[4] = {ares_, ares_, ares_, adir_}, g[4] = {r_, ares_, adir_, adir_};
            if (!reduce_row4(rows, f, g, part(), st, epoch, 104, live, sh, tot)) return;
        } else {
            rows.each([&](int i) { st_flow(pub + i, adir[i]); reset_flow(old + i); });
            double sums[4] = {0.0, 0.0, 0.0, 0.0};
            double ad = 0.0, ar = 0.0, r = 0.0;
            rows.products(a, pub, 103, live, [&](int i) {
                ad = adir[i]; ar = ares[i];
                a.x[i] = fma(alpha, dir[i], a.x[i]);
                r = fma(-alpha, ad, a.res[i]);
                a.res[i] = r;
            }, [&](int i, bool own, double vil) {
                if (own) {
                    ar = fma(-alpha, vil, ar);
                    ares[i] = ar;
                    sums[0] = fma(ar, r, sums[0]);
                    sums[1] = fma(ar, ar, sums[1]);
                    sums[2] = fma(ar, ad, sums[2]);
                    sums[3] = fma(ad, ad, sums[3]);
                }
            });
            if (!flow_reduce<double, 4>(sums, part(), st, epoch, 104, live, sh, tot)) return;
        }
        K++;
        if (threadIdx.x < 32) {
            const double beta = tot[0] / ad_r;                                              // :1865
            ad_r = tot[0];
            ad_ad = fma(beta, fma(beta, tot[3], 2.0 * tot[2]), tot[1]);
            const bool cancelled = !(ad_ad >= kCancel * fma(beta * beta, tot[3], tot[1]));
            if (threadIdx.x == 0) { ctl.b = beta; ctl.exact = cancelled; }
            if (!cancelled && K < a.max_iter) cr_step(ad_r, ad_ad, K, a.n, a.tol, a.print_modulo, ctl);
        }
        __syncthreads();
        const double beta = ctl.b;
        // :1867-1880: dir, Adir
        if constexpr (REG) {
            dir_ = fma(beta, dir_, r_);
            adir_ = fma(beta, adir_, ares_);
        } else {
            rows.each([&](int i) {
                dir[i] = fma(beta, dir[i], a.res[i]);
                adir[i] = fma(beta, adir[i], ares[i]);
            });
        }
        if (ctl.exact) {
            double acc[1] = {0.0}, sum[1];
            if constexpr (REG) {
                if (rows.own) acc[0] = adir_ * adir_;
            } else {
                rows.each([&](int i) { const double v = adir[i]; acc[0] = fma(v, v, acc[0]); });
            }
            if (!flow_reduce<double, 1>(acc, part(), st, epoch, 105, live, sh, sum)) return;
            if (threadIdx.x < 32) {
                ad_ad = sum[0];
                if (K < a.max_iter) cr_step(ad_r, ad_ad, K, a.n, a.tol, a.print_modulo, ctl);
            }
            __syncthreads();
        }
        if (K >= a.max_iter) { status = FEEC_MAXITER; break; }
    }
    if constexpr (REG)
        if (rows.own) { a.x[rows.i] = x_; a.res[rows.i] = r_; }
    finish(st, status, K, ad_r, ad_ad);
}

}  // namespace

cudaError_t launch_flow_more(bool minres, const FlowForm& form, const FlowMoreArgs& a, cudaStream_t st) {
    const void* fn = minres ? (form.registers ? (const void*)flow_minres<true> : (const void*)flow_minres<false>)
                            : (form.registers ? (const void*)flow_cr<true> : (const void*)flow_cr<false>);
    FlowMoreArgs copy = a;
    void* args[] = {&copy};
    note_launch();
    return cudaLaunchCooperativeKernel(fn, dim3(form.blocks), dim3(form.threads), args, 0, st);
}

}  // namespace feec
