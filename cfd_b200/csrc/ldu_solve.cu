// Residual norms of an engine's level-0 system, for the persistent LDU solve
// (LduMatrix::solve_persistent, ldu_matrix.cpp:287-366, and LduMatrix::residual_norms,
// ldu_matrix.cpp:69-103).
//
// Row i of A x is summed over the engine's SELL slots, which hold the LDU matrix's CSR pattern in
// column order with its values already scattered: coalesced columns and values, where a pass over
// the CSR pattern with each value fetched through the LDU value map took 44 us per call on the
// 1.3M-cell tet box (and two host round trips). The mean of x stays on the device between the
// two kernels. Sums are the tile reductions of the CG kernels: reproducible, and different from the
// reference's face-loop sums only in summation order.
#include "ldu_solve.hpp"

#include "engine.hpp"

namespace cfdb {

struct NormState {
    double x_ref;
    double res, norm, r2;
};

namespace {

// x_ref = sum of x over the n user rows / n
__global__ void __launch_bounds__(kBlock) k_ldu_mean(Tiles tiles, int n, const double* __restrict__ x, Reduce red,
                                                     NormState* out) {
    pdl_launch();
    const TileCtx c = tile_of(tiles);
    reduce_begin(c.tile, c.s, red);
    pdl_wait();
    double s = 0.0, unused = 0.0;
    for (int r0 = c.r0 + threadIdx.x; r0 < c.r1; r0 += 4 * kBlock) {
        double v[4];
#pragma unroll
        for (int u = 0; u < 4; ++u) v[u] = r0 + u * kBlock < min(c.r1, n) ? x[r0 + u * kBlock] : 0.0;
#pragma unroll
        for (int u = 0; u < 4; ++u) s += v[u];
    }
    if (reduce_system(s, unused, c.tile, red) && threadIdx.x == 0) out->x_ref = s / static_cast<double>(n);
}

// sum |b - Ax|, sum |Ax - rs x_ref| + |b - rs x_ref| (rs = row sum), sum (b - Ax)^2 over the n user
// rows. B: entries of a row taken in one batch.
template <int B>
__global__ void __launch_bounds__(kBlock) k_ldu_norms(Sell<double> m, Tiles tiles, int n, const double* __restrict__ b,
                                                      const double* __restrict__ x, Reduce red, Reduce red2,
                                                      NormState* out) {
    pdl_launch();
    const TileCtx c = tile_of(tiles);
    reduce_begin(c.tile, c.s, red);
    pdl_wait();
    const double x_ref = *reinterpret_cast<volatile const double*>(&out->x_ref);
    double res = 0.0, norm = 0.0, r2 = 0.0, unused = 0.0;
    for (int row = c.r0 + threadIdx.x; row < min(c.r1, n); row += kBlock) {
        SellRow r = sell_row_at(m, row);
        const double bi = b[row];
        double ax = 0.0, rs = 0.0;
        for (; r.k < r.e; r.k += 32 * B) {
            double v[B], xv[B];
            int cc[B];
            sell_load<B>(m, r.k, r.e, 0, v, cc);
#pragma unroll
            for (int u = 0; u < B; ++u) xv[u] = cc[u] >= 0 ? x[cc[u]] : 0.0;
#pragma unroll
            for (int u = 0; u < B; ++u)
                if (cc[u] >= 0) {
                    ax = __dadd_rn(ax, __dmul_rn(v[u], xv[u]));
                    rs = __dadd_rn(rs, v[u]);
                }
        }
        const double ax_ref = __dmul_rn(rs, x_ref);
        const double ri = __dsub_rn(bi, ax);
        res += fabs(ri);
        norm += fabs(ax - ax_ref) + fabs(bi - ax_ref);
        r2 += __dmul_rn(ri, ri);
    }
    if (reduce_system(res, norm, c.tile, red) && threadIdx.x == 0) {
        out->res = res;
        out->norm = norm;
    }
    if (reduce_system(r2, unused, c.tile, red2) && threadIdx.x == 0) out->r2 = r2;
}

} // namespace

LduNorms Engine::residual_norms() {
    CFDB_CUDA(cudaSetDevice(device_));
    if (n_sys_ != 1) fail(1, "residual_norms: single-system plans only");
    const DevLevel& d = lv_[0];
    if (norms_ == nullptr) {
        norms_ = arena_.alloc<NormState>(1);
        // a second set of partials and tickets: the norms are three sums
        const size_t groups = static_cast<size_t>(ceil_div(d.n_tiles, kGroupTiles)) + 1;
        red2_ = red_;
        red2_.partials = arena_.alloc<double>(2 * static_cast<size_t>(std::max(d.n_tiles, 1)));
        red2_.gpartials = arena_.alloc<double>(2 * groups);
        int* cnt = arena_.alloc<int>(2 * groups);
        CFDB_CUDA(cudaMemsetAsync(cnt, 0, sizeof(int) * 2 * groups, stream_));
        red2_.counters = cnt;
        red2_.gcounters = cnt + groups;
    }
    const bool pdl = tuning_.pdl != 0;
    const int n = n_of_[0];
    launch_k(pdl, k_ldu_mean, d.n_tiles, kBlock, 0, stream_, d.tiles, n, x_, red_, norms_);
    if (row_width(d.a) <= 5.25)
        launch_k(pdl, k_ldu_norms<5>, d.n_tiles, kBlock, 0, stream_, d.a.s64, d.tiles, n, b_, x_, red_, red2_, norms_);
    else
        launch_k(pdl, k_ldu_norms<7>, d.n_tiles, kBlock, 0, stream_, d.a.s64, d.tiles, n, b_, x_, red_, red2_, norms_);
    launches_ += 2;
    NormState* h = static_cast<NormState*>(host_state(sizeof(NormState)));
    CFDB_CUDA(cudaMemcpyAsync(h, norms_, sizeof(NormState), cudaMemcpyDeviceToHost, stream_));
    CFDB_CUDA(cudaStreamSynchronize(stream_));
    return LduNorms{h->res, h->norm, h->r2};
}

} // namespace cfdb
