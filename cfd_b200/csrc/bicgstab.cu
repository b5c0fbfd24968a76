// Jacobi-preconditioned BiCGStab on an engine's level-0 operator (the momentum solver of the
// reference's accelerator layer, krylov_kernels.inc:97-169, selected by Method::BiCgStab).
//
// The iteration follows the reference's recurrences and stopping rules step by step (rho from
// r0.r, the pp / ph / v / s / sh / t updates, omega = (t.s) / (t.t) or 0, the early exit on
// |s| and the exits on rho == 0, omega == 0 and r0.v == 0; iterations capped at the maximum).
// Every update rounds each product and sum separately in the reference's operand order. Dot
// products are the tile reductions of the CG kernels (reproducible; they differ from
// the reference's sequential sums only in summation order).
//
// The scalars live on the device (BcgState): each dot product is part of the kernel that makes
// its operands, and that kernel's last CTA takes the scalar step, so an iteration is five
// kernels captured in one graph, launched without waiting for any of its scalars. Before, four
// dot kernels a iteration were read back and added on the host: a scalar step on the graded
// 80^3 box spent 2.50 ms, of which the solve's kernels ran 0.99 ms.
#include <algorithm>
#include <type_traits>

#include "engine.hpp"

namespace cfdb {

struct BcgState {
    double tol;
    double res;
    double rho, alpha, omega, beta;
    int it, max_it;
    int iters_out;
    int active;
    int converged;
    int half; // |s| met the tolerance: this iteration ends with x += alpha ph
};

namespace {

__device__ __forceinline__ bool bcg_active(const BcgState* st) {
    return *reinterpret_cast<volatile const int*>(&st->active) != 0;
}

__device__ __forceinline__ void bcg_stop(BcgState& s, int iterations, int converged, int* n_active) {
    s.iters_out = iterations;
    s.converged = converged;
    s.active = 0;
    *n_active = 0;
}

// r = b - A x, r0 = r, pp = v = 0; |r|
template <int V>
static __global__ void __launch_bounds__(kBlock, (kMinBlocks<double, V, false>)) k_bcg_init(
    Sell<double> a, Tiles tiles, BcgState* st, const double* __restrict__ b, const double* __restrict__ x,
    double* __restrict__ r, double* __restrict__ r0, double* __restrict__ pp, double* __restrict__ v, Reduce red,
    int* n_active) {
    pdl_launch();
    const TileCtx c = tile_of(tiles);
    reduce_begin(c.tile, c.s, red);
    Visit<V, double> vis;
    vis.begin(a, c.r0, c.r1);
    pdl_wait();
    double rr = 0.0, unused = 0.0;
    vis.run(a, c.r0, c.r1, [x](int j) { return x[j]; }, [&](int row) { return b[row]; },
            [&](int row, double ax, double bi) {
                const double ri = __dsub_rn(bi, ax);
                r[row] = ri;
                r0[row] = ri;
                pp[row] = 0.0;
                v[row] = 0.0;
                rr = __dadd_rn(rr, __dmul_rn(ri, ri));
            });
    if (reduce_system(rr, unused, c.tile, red) && threadIdx.x == 0) {
        BcgState& s = *st;
        s.res = sqrt(rr);
        if (s.res <= s.tol) {
            bcg_stop(s, 0, 1, n_active);
        } else if (s.max_it < 1) {
            bcg_stop(s, s.max_it, 0, n_active);
        } else {
            // rho = alpha = omega = 1 before the first iteration; r0 . r = |r|^2
            s.rho = rr;
            s.beta = rr;
            s.omega = 1.0;
        }
    }
}

// pp = r + beta (pp - omega v); ph = pp * dinv
static __global__ void __launch_bounds__(kBlock) k_bcg_p(Tiles tiles, const BcgState* st, const double* __restrict__ r,
                                                         const double* __restrict__ v,
                                                         const double* __restrict__ dinv, double* __restrict__ pp,
                                                         double* __restrict__ ph) {
    pdl_launch();
    const TileCtx c = tile_of(tiles);
    pdl_wait();
    if (!bcg_active(st)) return;
    const double beta = st->beta, omega = st->omega;
    for (int r0 = c.r0 + threadIdx.x; r0 < c.r1; r0 += 2 * kBlock) {
        double ri[2], pi[2], vi[2], di[2];
#pragma unroll
        for (int u = 0; u < 2; ++u) {
            const int row = r0 + u * kBlock;
            const bool ok = row < c.r1;
            ri[u] = ok ? r[row] : 0.0;
            pi[u] = ok ? pp[row] : 0.0;
            vi[u] = ok ? v[row] : 0.0;
            di[u] = ok ? dinv[row] : 0.0;
        }
#pragma unroll
        for (int u = 0; u < 2; ++u) {
            const int row = r0 + u * kBlock;
            if (row >= c.r1) continue;
            const double p = __dadd_rn(ri[u], __dmul_rn(beta, __dsub_rn(pi[u], __dmul_rn(omega, vi[u]))));
            pp[row] = p;
            ph[row] = __dmul_rn(p, di[u]);
        }
    }
}

// kSecond = false: v = A ph and r0 . v -> alpha = rho / (r0 . v); kSecond: t = A sh, t . t and t . s
// -> omega (w is r0 or s)
template <int V, bool kSecond>
static __global__ void __launch_bounds__(kBlock, (kMinBlocks<double, V, false>)) k_bcg_spmv(
    Sell<double> a, Tiles tiles, BcgState* st, const double* __restrict__ in, const double* __restrict__ w,
    double* __restrict__ out, Reduce red, int* n_active) {
    pdl_launch();
    const TileCtx c = tile_of(tiles);
    reduce_begin(c.tile, c.s, red);
    Visit<V, double> vis;
    vis.begin(a, c.r0, c.r1);
    pdl_wait();
    if (!bcg_active(st)) return;
    if (kSecond && st->half != 0) return;
    double d0 = 0.0, d1 = 0.0;
    vis.run(a, c.r0, c.r1, [in](int j) { return in[j]; }, [&](int row) { return w[row]; },
            [&](int row, double q, double wi) {
                out[row] = q;
                if (kSecond) {
                    d0 = __dadd_rn(d0, __dmul_rn(q, q));
                    d1 = __dadd_rn(d1, __dmul_rn(q, wi));
                } else {
                    d0 = __dadd_rn(d0, __dmul_rn(wi, q));
                }
            });
    if (reduce_system(d0, d1, c.tile, red) && threadIdx.x == 0) {
        BcgState& s = *st;
        if (kSecond) {
            s.omega = d0 > 0.0 ? d1 / d0 : 0.0;
        } else if (d0 == 0.0) {
            bcg_stop(s, s.it, 0, n_active);
        } else {
            s.alpha = s.rho / d0;
        }
    }
}

// s = r - alpha v; sh = s * dinv; |s| (at the tolerance: the iteration ends with x += alpha ph)
static __global__ void __launch_bounds__(kBlock) k_bcg_s(Tiles tiles, BcgState* st, const double* __restrict__ r,
                                                         const double* __restrict__ v,
                                                         const double* __restrict__ dinv, double* __restrict__ s,
                                                         double* __restrict__ sh, Reduce red) {
    pdl_launch();
    const TileCtx c = tile_of(tiles);
    reduce_begin(c.tile, c.s, red);
    pdl_wait();
    if (!bcg_active(st)) return;
    const double alpha = st->alpha;
    double ss = 0.0, unused = 0.0;
    for (int r0 = c.r0 + threadIdx.x; r0 < c.r1; r0 += 2 * kBlock) {
        double ri[2], vi[2], di[2];
#pragma unroll
        for (int u = 0; u < 2; ++u) {
            const int row = r0 + u * kBlock;
            const bool ok = row < c.r1;
            ri[u] = ok ? r[row] : 0.0;
            vi[u] = ok ? v[row] : 0.0;
            di[u] = ok ? dinv[row] : 0.0;
        }
#pragma unroll
        for (int u = 0; u < 2; ++u) {
            const int row = r0 + u * kBlock;
            if (row >= c.r1) continue;
            const double si = __dsub_rn(ri[u], __dmul_rn(alpha, vi[u]));
            s[row] = si;
            sh[row] = __dmul_rn(si, di[u]);
            ss = __dadd_rn(ss, __dmul_rn(si, si));
        }
    }
    if (reduce_system(ss, unused, c.tile, red) && threadIdx.x == 0) {
        BcgState& q = *st;
        const double norm = sqrt(ss);
        q.half = norm <= q.tol ? 1 : 0;
        if (q.half) q.res = norm;
    }
}

// x += alpha ph + omega sh; r = s - omega t; |r| and r0 . r -> the next iteration's rho and beta
// (half: x += alpha ph only, converged)
static __global__ void __launch_bounds__(kBlock) k_bcg_xr(Tiles tiles, BcgState* st, const double* __restrict__ ph,
                                                          const double* __restrict__ sh,
                                                          const double* __restrict__ s,
                                                          const double* __restrict__ t,
                                                          const double* __restrict__ rs, double* __restrict__ x,
                                                          double* __restrict__ r, Reduce red, int* n_active) {
    pdl_launch();
    const TileCtx c = tile_of(tiles);
    reduce_begin(c.tile, c.s, red);
    pdl_wait();
    if (!bcg_active(st)) return;
    const double alpha = st->alpha, omega = st->omega;
    const bool half = st->half != 0;
    double rr = 0.0, rho = 0.0;
    for (int r0 = c.r0 + threadIdx.x; r0 < c.r1; r0 += 2 * kBlock) {
        double xi[2], pi[2], hi[2], si[2], ti[2], ri[2];
#pragma unroll
        for (int u = 0; u < 2; ++u) {
            const int row = r0 + u * kBlock;
            const bool ok = row < c.r1;
            xi[u] = ok ? x[row] : 0.0;
            pi[u] = ok ? ph[row] : 0.0;
            hi[u] = ok && !half ? sh[row] : 0.0;
            si[u] = ok && !half ? s[row] : 0.0;
            ti[u] = ok && !half ? t[row] : 0.0;
            ri[u] = ok && !half ? rs[row] : 0.0;
        }
#pragma unroll
        for (int u = 0; u < 2; ++u) {
            const int row = r0 + u * kBlock;
            if (row >= c.r1) continue;
            if (half) {
                x[row] = __dadd_rn(xi[u], __dmul_rn(alpha, pi[u]));
            } else {
                x[row] = __dadd_rn(xi[u], __dadd_rn(__dmul_rn(alpha, pi[u]), __dmul_rn(omega, hi[u])));
                const double rn = __dsub_rn(si[u], __dmul_rn(omega, ti[u]));
                r[row] = rn;
                rr = __dadd_rn(rr, __dmul_rn(rn, rn));
                rho = __dadd_rn(rho, __dmul_rn(ri[u], rn));
            }
        }
    }
    if (reduce_system(rr, rho, c.tile, red) && threadIdx.x == 0) {
        BcgState& q = *st;
        if (half) {
            bcg_stop(q, q.it, 1, n_active);
            return;
        }
        q.res = sqrt(rr);
        if (q.res <= q.tol) {
            bcg_stop(q, q.it, 1, n_active);
            return;
        }
        q.it += 1;
        if (q.it > q.max_it) {
            bcg_stop(q, q.max_it, 0, n_active);
        } else if (rho == 0.0 || omega == 0.0) {
            bcg_stop(q, q.it, 0, n_active);
        } else {
            q.beta = (rho / q.rho) * (alpha / omega);
            q.rho = rho;
        }
    }
}

} // namespace

// The initial residual, or the five kernels of one iteration.
void Engine::enqueue_bicgstab(bool init) {
    const DevLevel& d = lv_[0];
    const size_t n = static_cast<size_t>(d.n_rows);
    double* r0 = bcg_;
    double* v = r0 + n;
    double* s = v + n;
    double* t = s + n;
    double* ph = t + n;
    double* sh = ph + n;
    const bool pdl = tuning_.pdl != 0;
    auto run = [&](auto V) {
        constexpr int kV = decltype(V)::value;
        if (init) {
            launch_k(pdl, k_bcg_init<kV>, d.n_tiles, kBlock, 0, stream_, d.a.s64, d.tiles, bcg_st_, b_, x_, r_, r0, p_, v, red_,
                       n_active_);
            return;
        }
        launch_k(pdl, k_bcg_p, d.n_tiles, kBlock, 0, stream_, d.tiles, bcg_st_, r_, v, dinv0_, p_, ph);
        launch_k(pdl, k_bcg_spmv<kV, false>, d.n_tiles, kBlock, 0, stream_, d.a.s64, d.tiles, bcg_st_, ph, r0, v, red_, n_active_);
        launch_k(pdl, k_bcg_s, d.n_tiles, kBlock, 0, stream_, d.tiles, bcg_st_, r_, v, dinv0_, s, sh, red_);
        launch_k(pdl, k_bcg_spmv<kV, true>, d.n_tiles, kBlock, 0, stream_, d.a.s64, d.tiles, bcg_st_, sh, s, t, red_, n_active_);
        launch_k(pdl, k_bcg_xr, d.n_tiles, kBlock, 0, stream_, d.tiles, bcg_st_, ph, sh, s, t, r0, x_, r_, red_, n_active_);
    };
    with_krylov_visit(krylov_visit(), run);
}

SolveResult Engine::solve_bicgstab(const SolveRequest& rq, bool want_true) {
    CFDB_CUDA(cudaSetDevice(device_));
    if (n_sys_ != 1) fail(1, "solve_bicgstab: single-system plans only");
    const DevLevel& d = lv_[0];
    if (bcg_ == nullptr) {
        bcg_ = arena_.alloc<double>(6 * static_cast<size_t>(d.n_rows));
        bcg_st_ = arena_.alloc<BcgState>(1);
    }
    capture(kBcgGraphs, kInit, [&] { enqueue_bicgstab(true); });
    capture(kBcgGraphs, kIterate, [&] {
        enqueue_bicgstab(false);
        enqueue_publish();
    });
    struct Upload {
        BcgState s;
        SysState cg;
        int words[2];
    };
    Upload* h = static_cast<Upload*>(host_state(sizeof(Upload)));
    h->s = BcgState{};
    h->s.tol = rq.tol;
    h->s.max_it = rq.max_it;
    h->s.it = 1;
    h->s.active = 1;
    h->words[0] = 1; // active systems
    h->words[1] = 0; // error flag
    CFDB_CUDA(cudaMemcpyAsync(bcg_st_, &h->s, sizeof(BcgState), cudaMemcpyHostToDevice, stream_));
    CFDB_CUDA(cudaMemcpyAsync(n_active_, h->words, 2 * sizeof(int), cudaMemcpyHostToDevice, stream_));
    launch_graph(kBcgGraphs, kInit);
    iterate(kBcgGraphs, std::max(rq.max_it, 0) + 1LL);
    h->cg.true_res = -1.0;
    if (want_true) {
        // |b - A x| of the returned solution, as the CG paths report it
        with_krylov_visit(krylov_visit(), [&](auto V) {
            launch_k(tuning_.pdl != 0, k_true_residual<decltype(V)::value>, d.n_tiles, kBlock, 0, stream_, d.a.s64, d.tiles,
                     st_, b_, x_, red_);
        });
        ++launches_;
        CFDB_CUDA(cudaGetLastError());
        CFDB_CUDA(cudaMemcpyAsync(&h->cg, st_, sizeof(SysState), cudaMemcpyDeviceToHost, stream_));
    }
    CFDB_CUDA(cudaMemcpyAsync(&h->s, bcg_st_, sizeof(BcgState), cudaMemcpyDeviceToHost, stream_));
    CFDB_CUDA(cudaStreamSynchronize(stream_));
    SolveResult out;
    out.iterations = h->s.active ? rq.max_it : h->s.iters_out;
    out.residual = h->s.res;
    out.converged = h->s.converged != 0;
    out.true_residual = h->cg.true_res;
    return out;
}

} // namespace cfdb
