// Pressure gradient and velocity correction of FlowSolver::pressure_correction on the device
// (the Gauss branch of FlowSolver::pressure_gradient, flow_solver.cpp:339-372, and the velocity
// correction, flow_solver.cpp:843-846).
//
// The reference accumulates face by face: each internal face adds S_f p_f to its owner and
// subtracts it from its neighbour, then each boundary face adds S_f p_b to its owner. Here
// one thread per cell walks its internal faces in ascending face order and then its boundary
// faces in ascending order, so every cell receives the same contributions in the same order;
// every product and sum is rounded separately (no FMA). Vectors are xyz-interleaved.
//
// The cell kernels are bound by the chain of dependent gathers of a cell's faces (slot -> face and
// cell across -> values), so a cell's slots are taken in batches of kFaceBatch whose loads are in
// flight together, and each slot holds the cell across its face beside the face, which saves the
// owner and neighbour gathers.
#include "../../include/cfdb.h"

#include <algorithm>
#include <cmath>
#include <string>
#include <vector>

#include "common.hpp"
#include "fv_step.hpp"

static_assert(CFDB_ERR_NO_DEVICE == 4, "require_cuda_device (common.hpp) reports status 4");

namespace cfdb {
void set_thread_error(const std::string& msg);
} // namespace cfdb

using namespace cfdb;

struct cfdb_fv {
    int device = 0;
    int n = 0, nf = 0, ni = 0;
    cudaStream_t st = nullptr;
    DeviceArena mem;
    int* owner = nullptr;     // n_faces
    int* neighbour = nullptr; // internal faces
    double* w = nullptr;      // internal faces
    double* sf = nullptr;     // 3 n_faces
    double* cf = nullptr;     // 3 n_faces
    double* cc = nullptr;     // 3 n_cells
    double* vol = nullptr;    // n_cells
    int* kind = nullptr;      // boundary faces: cfdb_boundary_kind
    double* pout = nullptr;   // boundary faces: outlet pressure
    int* iptr = nullptr;      // cell -> internal faces (ascending)
    int2* islot = nullptr;    // face, and the cell across: c' >= 0 when this cell owns the face, else -1 - c'
    int* bptr = nullptr;      // cell -> boundary faces (ascending)
    int* bface = nullptr;
    double* delta = nullptr;  // n_faces: delta coefficients (fv_geometry.cpp:43-50)
    double* corr = nullptr;   // 3 internal faces: non-orthogonal corrections S - d delta
    ~cfdb_fv() {
        if (st != nullptr) {
            cudaStreamSynchronize(st);
            cudaStreamDestroy(st);
        }
    }
};

namespace {

constexpr int kFaceBatch = 4; // a tet's internal faces; a hex takes two batches

// Calls f(slot values) for the slots [k0, k1) in order, kFaceBatch at a time: load(j, slot) fills
// entry j of the caller's registers for every slot of a batch first, then use(j, slot) runs in order.
template <class L, class U>
__device__ __forceinline__ void for_faces(const int2* __restrict__ islot, int k0, int k1, L load, U use) {
    for (int k = k0; k < k1; k += kFaceBatch) {
        int2 s[kFaceBatch];
#pragma unroll
        for (int j = 0; j < kFaceBatch; ++j) s[j] = k + j < k1 ? __ldg(&islot[k + j]) : make_int2(-1, 0);
#pragma unroll
        for (int j = 0; j < kFaceBatch; ++j)
            if (s[j].x >= 0) load(j, s[j]);
#pragma unroll
        for (int j = 0; j < kFaceBatch; ++j)
            if (s[j].x >= 0) use(j, s[j]);
    }
}

__device__ __forceinline__ bool owned(const int2& slot) { return slot.y >= 0; }
__device__ __forceinline__ int across(const int2& slot) { return slot.y >= 0 ? slot.y : -1 - slot.y; }

// Pressure gradient of one cell in two passes (flow_solver.cpp:348-370): the sum over its internal
// faces of +-S_f (w p_P + (1 - w) p_N), then of S_f p_b over its boundary faces, over the volume.
// Pass 2 extrapolates p_b of every boundary face but pressure outlets tangentially with the
// first-pass gradient of the cell: p_b = p_P + g_P . (d - (d . n) n), d = face centre - cell centre,
// n = S / |S|. The second pass reads the first one's result of its own cell alone, so both run in
// one thread, and cells without boundary faces need one. As three kernels with the sums in memory
// between them the gradient took 106 us on the 1.3M-cell tet box. With u also the velocity
// correction u = HbyA - rAU grad (flow_solver.cpp:843-846).
__global__ void __launch_bounds__(256) k_gradient(int n, int ni, const int* __restrict__ iptr, const int2* __restrict__ islot,
                           const double* __restrict__ w, const int* __restrict__ bptr,
                           const int* __restrict__ bface, const int* __restrict__ kind,
                           const double* __restrict__ pout, const double* __restrict__ sf,
                           const double* __restrict__ cf, const double* __restrict__ cc,
                           const double* __restrict__ vol, const double* __restrict__ p,
                           double* __restrict__ grad, const double* __restrict__ hbya,
                           const double* __restrict__ rau, double* __restrict__ u) {
    const int c = blockIdx.x * blockDim.x + threadIdx.x;
    if (c >= n) return;
    const int k0 = iptr[c], k1 = iptr[c + 1], b0 = bptr[c], b1 = bptr[c + 1];
    const double pc = p[c], v = vol[c];
    double g[3] = {0.0, 0.0, 0.0};
    double wf[kFaceBatch], pa[kFaceBatch], s0[kFaceBatch], s1[kFaceBatch], s2[kFaceBatch];
    for_faces(islot, k0, k1,
              [&](int j, const int2& s) {
                  wf[j] = w[s.x];
                  pa[j] = p[across(s)];
                  s0[j] = sf[3 * s.x];
                  s1[j] = sf[3 * s.x + 1];
                  s2[j] = sf[3 * s.x + 2];
              },
              [&](int j, const int2& s) {
                  const bool mine = owned(s);
                  const double po = mine ? pc : pa[j], pn = mine ? pa[j] : pc;
                  const double pf = __dadd_rn(__dmul_rn(wf[j], po), __dmul_rn(__dsub_rn(1.0, wf[j]), pn));
                  const double f0 = __dmul_rn(s0[j], pf), f1 = __dmul_rn(s1[j], pf), f2 = __dmul_rn(s2[j], pf);
                  g[0] = mine ? __dadd_rn(g[0], f0) : __dsub_rn(g[0], f0);
                  g[1] = mine ? __dadd_rn(g[1], f1) : __dsub_rn(g[1], f1);
                  g[2] = mine ? __dadd_rn(g[2], f2) : __dsub_rn(g[2], f2);
              });
    double out[3];
    for (int pass = b0 < b1 ? 1 : 2; pass <= 2; ++pass) {
        double a0 = g[0], a1 = g[1], a2 = g[2];
        for (int k = b0; k < b1; ++k) {
            const int f = bface[k];
            const int b = f - ni;
            const bool outlet = kind[b] == CFDB_BC_PRESSURE_OUTLET;
            double pb = outlet ? pout[b] : pc;
            const double t0 = sf[3 * f], t1 = sf[3 * f + 1], t2 = sf[3 * f + 2];
            if (pass == 2 && !outlet) {
                const double area = __dsqrt_rn(__dadd_rn(__dadd_rn(__dmul_rn(t0, t0), __dmul_rn(t1, t1)), __dmul_rn(t2, t2)));
                const double n0 = __ddiv_rn(t0, area), n1 = __ddiv_rn(t1, area), n2 = __ddiv_rn(t2, area);
                const double d0 = __dsub_rn(cf[3 * f], cc[3 * c]);
                const double d1 = __dsub_rn(cf[3 * f + 1], cc[3 * c + 1]);
                const double d2 = __dsub_rn(cf[3 * f + 2], cc[3 * c + 2]);
                const double dn = __dadd_rn(__dadd_rn(__dmul_rn(d0, n0), __dmul_rn(d1, n1)), __dmul_rn(d2, n2));
                const double e0 = __dsub_rn(d0, __dmul_rn(dn, n0));
                const double e1 = __dsub_rn(d1, __dmul_rn(dn, n1));
                const double e2 = __dsub_rn(d2, __dmul_rn(dn, n2));
                const double e = __dadd_rn(__dadd_rn(__dmul_rn(out[0], e0), __dmul_rn(out[1], e1)), __dmul_rn(out[2], e2));
                pb = __dadd_rn(pb, e);
            }
            a0 = __dadd_rn(a0, __dmul_rn(t0, pb));
            a1 = __dadd_rn(a1, __dmul_rn(t1, pb));
            a2 = __dadd_rn(a2, __dmul_rn(t2, pb));
        }
        out[0] = __ddiv_rn(a0, v);
        out[1] = __ddiv_rn(a1, v);
        out[2] = __ddiv_rn(a2, v);
    }
#pragma unroll
    for (int i = 0; i < 3; ++i) grad[3 * c + i] = out[i];
    if (u != nullptr) {
        const double r = rau[c];
#pragma unroll
        for (int i = 0; i < 3; ++i) u[3 * c + i] = __dsub_rn(hbya[3 * c + i], __dmul_rn(r, out[i]));
    }
}

// u = HbyA - rAU grad p
__global__ void k_correct_velocity(int n, const double* __restrict__ hbya, const double* __restrict__ rau,
                                   const double* __restrict__ grad, double* __restrict__ u) {
    const int c = blockIdx.x * blockDim.x + threadIdx.x;
    if (c >= n) return;
    const double r = rau[c];
    for (int i = 0; i < 3; ++i) u[3 * c + i] = __dsub_rn(hbya[3 * c + i], __dmul_rn(r, grad[3 * c + i]));
}

// HbyA = (source - offdiag(U) U) / diag and rAU = V / mean(diag) (flow_solver.cpp:688-707),
// per component; the off-diagonal product gathers the cell's faces in ascending order
// (ldu_matrix.cpp:39-49: upper * x[N] for owned faces, lower * x[P] otherwise). One walk over the
// faces serves the three components (three walks took 81 us on the 1.3M-cell tet box).
__global__ void __launch_bounds__(256) k_hbya_rau(int n, const int* __restrict__ iptr, const int2* __restrict__ islot,
                           const double* __restrict__ upper, const double* __restrict__ lower,
                           const double* __restrict__ diag, const double* __restrict__ source,
                           const double* __restrict__ u, const double* __restrict__ vol,
                           double* __restrict__ hbya, double* __restrict__ rau) {
    const int c = blockIdx.x * blockDim.x + threadIdx.x;
    if (c >= n) return;
    const int k0 = iptr[c], k1 = iptr[c + 1];
    double d[3], src[3], off[3] = {0.0, 0.0, 0.0};
#pragma unroll
    for (int i = 0; i < 3; ++i) {
        d[i] = diag[3 * c + i];
        src[i] = source[3 * c + i];
    }
    double a[kFaceBatch], x[kFaceBatch][3];
    for_faces(islot, k0, k1,
              [&](int j, const int2& s) {
                  a[j] = owned(s) ? upper[s.x] : lower[s.x];
                  const int o = across(s);
#pragma unroll
                  for (int i = 0; i < 3; ++i) x[j][i] = u[3 * o + i];
              },
              [&](int j, const int2&) {
#pragma unroll
                  for (int i = 0; i < 3; ++i) off[i] = __dadd_rn(off[i], __dmul_rn(a[j], x[j][i]));
              });
#pragma unroll
    for (int i = 0; i < 3; ++i) hbya[3 * c + i] = __ddiv_rn(__dsub_rn(src[i], off[i]), d[i]);
    const double mean = __ddiv_rn(__dadd_rn(__dadd_rn(d[0], d[1]), d[2]), 3.0);
    rau[c] = __ddiv_rn(vol[c], mean);
}

__device__ __forceinline__ double dot3(const double* a, const double* b) {
    return __dadd_rn(__dadd_rn(__dmul_rn(a[0], b[0]), __dmul_rn(a[1], b[1])), __dmul_rn(a[2], b[2]));
}

// predicted face flux and face rAU (flow_solver.cpp:709-733), with the relaxation-independent
// correction when u_prev / phi_prev are given (flow_solver.cpp:735-752)
__global__ void k_face_flux(int nf, int ni, const int* __restrict__ owner, const int* __restrict__ neighbour,
                            const double* __restrict__ w, const double* __restrict__ sf,
                            const int* __restrict__ kind, const double* __restrict__ hbya,
                            const double* __restrict__ rau, const double* __restrict__ ufix,
                            const double* __restrict__ u_prev, const double* __restrict__ phi_prev, double beta,
                            double* __restrict__ phi, double* __restrict__ rau_f) {
    const int f = blockIdx.x * blockDim.x + threadIdx.x;
    if (f >= nf) return;
    const int o = owner[f];
    const double* s = sf + 3 * f;
    double ph, rf;
    if (f < ni) {
        const int nb = neighbour[f];
        const double wf = w[f], wn = __dsub_rn(1.0, wf);
        double v[3];
        for (int i = 0; i < 3; ++i) v[i] = __dadd_rn(__dmul_rn(wf, hbya[3 * o + i]), __dmul_rn(wn, hbya[3 * nb + i]));
        ph = dot3(v, s);
        rf = __dadd_rn(__dmul_rn(wf, rau[o]), __dmul_rn(wn, rau[nb]));
        if (u_prev != nullptr) {
            double uf[3];
            for (int i = 0; i < 3; ++i) uf[i] = __dadd_rn(__dmul_rn(wf, u_prev[3 * o + i]), __dmul_rn(wn, u_prev[3 * nb + i]));
            ph = __dadd_rn(ph, __dmul_rn(beta, __dsub_rn(phi_prev[f], dot3(uf, s))));
        }
    } else {
        const int b = f - ni;
        rf = rau[o];
        const int k = kind[b];
        if (k == CFDB_BC_VELOCITY_INLET || k == CFDB_BC_WALL) {
            ph = dot3(ufix + 3 * b, s);
        } else if (k == CFDB_BC_PRESSURE_OUTLET) {
            ph = dot3(hbya + 3 * o, s);
            if (u_prev != nullptr) ph = __dadd_rn(ph, __dmul_rn(beta, __dsub_rn(phi_prev[f], dot3(u_prev + 3 * o, s))));
        } else {
            ph = 0.0;
        }
    }
    phi[f] = ph;
    rau_f[f] = rf;
}

// boundary terms of the pressure equation (flow_solver.cpp:784-796): source -= phi_HbyA for
// every boundary face, and for outlets diag += rAU_f delta, source += rAU_f delta p_out; then
// set_reference(ref_cell, ref_value) (ldu_matrix.cpp:105-109) unless ref_cell < 0
__global__ void k_pressure_boundary(int n, int ni, const int* __restrict__ bptr, const int* __restrict__ bface,
                                    const int* __restrict__ kind, const double* __restrict__ pout,
                                    const double* __restrict__ phi, const double* __restrict__ rau_f,
                                    const double* __restrict__ delta, int ref_cell, double ref_value,
                                    double* __restrict__ diag, double* __restrict__ source) {
    const int c = blockIdx.x * blockDim.x + threadIdx.x;
    if (c >= n) return;
    double d = diag[c], s = source[c];
    for (int k = bptr[c]; k < bptr[c + 1]; ++k) {
        const int f = bface[k];
        const int b = f - ni;
        s = __dsub_rn(s, phi[f]);
        if (kind[b] == CFDB_BC_PRESSURE_OUTLET) {
            const double coeff = __dmul_rn(rau_f[f], delta[f]);
            d = __dadd_rn(d, coeff);
            s = __dadd_rn(s, __dmul_rn(coeff, pout[b]));
        }
    }
    if (c == ref_cell) {
        s = __dadd_rn(s, __dmul_rn(d, ref_value));
        d = __dadd_rn(d, d);
    }
    diag[c] = d;
    source[c] = s;
}

// non-orthogonal correction fluxes rAU_f k . (w gp_P + (1 - w) gp_N) (flow_solver.cpp:808-815)
__global__ void k_non_orth_faces(int ni, const int* __restrict__ owner, const int* __restrict__ neighbour,
                                 const double* __restrict__ w, const double* __restrict__ corr,
                                 const double* __restrict__ rau_f, const double* __restrict__ grad,
                                 double* __restrict__ non_orth) {
    const int f = blockIdx.x * blockDim.x + threadIdx.x;
    if (f >= ni) return;
    const int o = owner[f], nb = neighbour[f];
    const double wf = w[f], wn = __dsub_rn(1.0, wf);
    double v[3];
    for (int i = 0; i < 3; ++i) v[i] = __dadd_rn(__dmul_rn(wf, grad[3 * o + i]), __dmul_rn(wn, grad[3 * nb + i]));
    non_orth[f] = __dmul_rn(rau_f[f], dot3(corr + 3 * f, v));
}

// source = base + (owned faces) non_orth - (neighbour faces) non_orth, faces in ascending order
__global__ void __launch_bounds__(256) k_non_orth_source(int n, const int* __restrict__ iptr, const int2* __restrict__ islot,
                                  const double* __restrict__ non_orth, const double* __restrict__ base,
                                  double* __restrict__ source) {
    const int c = blockIdx.x * blockDim.x + threadIdx.x;
    if (c >= n) return;
    double t = base[c];
    double e[kFaceBatch];
    for_faces(islot, iptr[c], iptr[c + 1], [&](int j, const int2& s) { e[j] = non_orth[s.x]; },
              [&](int j, const int2& s) { t = owned(s) ? __dadd_rn(t, e[j]) : __dsub_rn(t, e[j]); });
    source[c] = t;
}

// conservative face flux on every face (flow_solver.cpp:818-833)
__global__ void k_fv_correct_flux(int nf, int ni, const int* __restrict__ owner, const int* __restrict__ neighbour,
                                  const int* __restrict__ kind, const double* __restrict__ pout,
                                  const double* __restrict__ phi_hbya, const double* __restrict__ rau_f,
                                  const double* __restrict__ delta, const double* __restrict__ non_orth,
                                  const double* __restrict__ p, double* __restrict__ phi) {
    const int f = blockIdx.x * blockDim.x + threadIdx.x;
    if (f >= nf) return;
    const int o = owner[f];
    const double coeff = __dmul_rn(rau_f[f], delta[f]);
    if (f < ni) {
        const double v = __dsub_rn(phi_hbya[f], __dmul_rn(coeff, __dsub_rn(p[neighbour[f]], p[o])));
        phi[f] = __dsub_rn(v, non_orth != nullptr ? non_orth[f] : 0.0);
    } else {
        const int b = f - ni;
        double v = phi_hbya[f];
        if (kind[b] == CFDB_BC_PRESSURE_OUTLET) v = __dsub_rn(v, __dmul_rn(coeff, __dsub_rn(pout[b], p[o])));
        phi[f] = v;
    }
}

// p = p_prev + alpha (p_new - p_prev) (flow_solver.cpp:837-840)
__global__ void k_fv_relax(int n, const double* __restrict__ p_prev, const double* __restrict__ p_new,
                           double alpha, double* __restrict__ p) {
    const int c = blockIdx.x * blockDim.x + threadIdx.x;
    if (c >= n) return;
    p[c] = __dadd_rn(p_prev[c], __dmul_rn(alpha, __dsub_rn(p_new[c], p_prev[c])));
}

int grid_cells(int n) { return std::max(1, (n + 255) / 256); }

template <class F> int guarded_fv(F&& f) {
    try {
        f();
        return CFDB_OK;
    } catch (const Error& e) {
        set_thread_error(e.what());
        return e.code;
    } catch (const std::exception& e) {
        set_thread_error(e.what());
        return CFDB_ERR_INTERNAL;
    }
}

} // namespace

// The launches behind the entry points: arguments checked, work enqueued on the geometry's stream.
namespace cfdb {

int fv_device(const cfdb_fv* fv) { return fv->device; }

cudaStream_t fv_stream(const cfdb_fv* fv) { return fv->st; }

void fv_gradient(cfdb_fv* fv, const double* p, double* grad, const double* hbya, const double* rau, double* u) {
    if (fv == nullptr || p == nullptr || grad == nullptr) fail(CFDB_ERR_BAD_ARG, "null argument");
    CFDB_CUDA(cudaSetDevice(fv->device));
    k_gradient<<<grid_cells(fv->n), 256, 0, fv->st>>>(fv->n, fv->ni, fv->iptr, fv->islot, fv->w, fv->bptr, fv->bface, fv->kind,
                                                fv->pout, fv->sf, fv->cf, fv->cc, fv->vol, p, grad, hbya, rau, u);
    CFDB_CUDA(cudaGetLastError());
}

void fv_hbya_rau(cfdb_fv* fv, const double* mom_diag, const double* mom_upper, const double* mom_lower,
                 const double* mom_source, const double* u, double* hbya, double* rau) {
    if (fv == nullptr || !mom_diag || !mom_source || !u || !hbya || !rau || (fv->ni > 0 && (!mom_upper || !mom_lower)))
        fail(CFDB_ERR_BAD_ARG, "null argument");
    CFDB_CUDA(cudaSetDevice(fv->device));
    k_hbya_rau<<<grid_cells(fv->n), 256, 0, fv->st>>>(fv->n, fv->iptr, fv->islot, mom_upper, mom_lower, mom_diag, mom_source, u,
                                                fv->vol, hbya, rau);
    CFDB_CUDA(cudaGetLastError());
}

void fv_face_flux(cfdb_fv* fv, const double* hbya, const double* rau, const double* fixed_velocity, const double* u_prev,
                  const double* phi_prev, double beta, double* phi_hbya, double* rau_f) {
    if (fv == nullptr || !hbya || !rau || !phi_hbya || !rau_f || (fv->nf > fv->ni && !fixed_velocity) ||
        ((u_prev == nullptr) != (phi_prev == nullptr)))
        fail(CFDB_ERR_BAD_ARG, "null argument (u_prev and phi_prev go together)");
    CFDB_CUDA(cudaSetDevice(fv->device));
    k_face_flux<<<grid_cells(fv->nf), 256, 0, fv->st>>>(fv->nf, fv->ni, fv->owner, fv->neighbour, fv->w, fv->sf, fv->kind, hbya,
                                                  rau, fixed_velocity, u_prev, phi_prev, beta, phi_hbya, rau_f);
    CFDB_CUDA(cudaGetLastError());
}

void fv_pressure_boundary(cfdb_fv* fv, const double* phi_hbya, const double* rau_f, int ref_cell, double ref_value,
                          double* diag, double* source) {
    if (fv == nullptr || !phi_hbya || !rau_f || !diag || !source) fail(CFDB_ERR_BAD_ARG, "null argument");
    if (ref_cell >= fv->n) fail(CFDB_ERR_BAD_ARG, "reference cell out of range");
    CFDB_CUDA(cudaSetDevice(fv->device));
    k_pressure_boundary<<<grid_cells(fv->n), 256, 0, fv->st>>>(fv->n, fv->ni, fv->bptr, fv->bface, fv->kind, fv->pout, phi_hbya,
                                                         rau_f, fv->delta, ref_cell, ref_value, diag, source);
    CFDB_CUDA(cudaGetLastError());
}

void fv_non_orth(cfdb_fv* fv, const double* grad, const double* rau_f, const double* base_source, double* non_orth,
                 double* source) {
    if (fv == nullptr || !grad || !rau_f || !base_source || !non_orth || !source) fail(CFDB_ERR_BAD_ARG, "null argument");
    CFDB_CUDA(cudaSetDevice(fv->device));
    if (fv->ni > 0)
        k_non_orth_faces<<<grid_cells(fv->ni), 256, 0, fv->st>>>(fv->ni, fv->owner, fv->neighbour, fv->w, fv->corr, rau_f, grad,
                                                             non_orth);
    k_non_orth_source<<<grid_cells(fv->n), 256, 0, fv->st>>>(fv->n, fv->iptr, fv->islot, non_orth, base_source, source);
    CFDB_CUDA(cudaGetLastError());
}

void fv_correct_flux(cfdb_fv* fv, const double* phi_hbya, const double* rau_f, const double* non_orth,
                     const double* p_new, double* phi) {
    if (fv == nullptr || !phi_hbya || !rau_f || !p_new || !phi) fail(CFDB_ERR_BAD_ARG, "null argument");
    CFDB_CUDA(cudaSetDevice(fv->device));
    k_fv_correct_flux<<<grid_cells(fv->nf), 256, 0, fv->st>>>(fv->nf, fv->ni, fv->owner, fv->neighbour, fv->kind, fv->pout,
                                                        phi_hbya, rau_f, fv->delta, non_orth, p_new, phi);
    CFDB_CUDA(cudaGetLastError());
}

void fv_relax(cfdb_fv* fv, const double* p_prev, const double* p_new, double alpha, double* p) {
    if (fv == nullptr || !p_prev || !p_new || !p) fail(CFDB_ERR_BAD_ARG, "null argument");
    CFDB_CUDA(cudaSetDevice(fv->device));
    k_fv_relax<<<grid_cells(fv->n), 256, 0, fv->st>>>(fv->n, p_prev, p_new, alpha, p);
    CFDB_CUDA(cudaGetLastError());
}

} // namespace cfdb

extern "C" {

int cfdb_fv_create(int n_cells, int n_faces, int n_internal_faces, const int* owner, const int* neighbour,
                   const double* face_areas, const double* face_centres, const double* cell_centres,
                   const double* cell_volumes, const double* weights, const int* boundary_kind,
                   const double* boundary_pressure, cfdb_fv** out) {
    return guarded_fv([&] {
        if (out == nullptr || n_cells <= 0 || n_internal_faces < 0 || n_faces < n_internal_faces)
            fail(CFDB_ERR_BAD_ARG, "cfdb_fv_create: bad sizes");
        const int nb = n_faces - n_internal_faces;
        if (!owner || (n_internal_faces > 0 && (!neighbour || !weights)) || !face_areas || !face_centres ||
            !cell_centres || !cell_volumes || (nb > 0 && (!boundary_kind || !boundary_pressure)))
            fail(CFDB_ERR_BAD_ARG, "cfdb_fv_create: null array");
        for (int f = 0; f < n_faces; ++f) {
            if (owner[f] < 0 || owner[f] >= n_cells || (f < n_internal_faces && (neighbour[f] < 0 || neighbour[f] >= n_cells)))
                fail(CFDB_ERR_BAD_ARG, "cfdb_fv_create: face " + std::to_string(f) + " addresses a cell out of range");
        }
        for (int b = 0; b < nb; ++b)
            if (boundary_kind[b] < CFDB_BC_VELOCITY_INLET || boundary_kind[b] > CFDB_BC_EMPTY)
                fail(CFDB_ERR_BAD_ARG, "cfdb_fv_create: unknown boundary kind");
        require_cuda_device();
        auto* fv = new cfdb_fv;
        try {
            CFDB_CUDA(cudaGetDevice(&fv->device));
            CFDB_CUDA(cudaStreamCreateWithFlags(&fv->st, cudaStreamNonBlocking));
            fv->n = n_cells;
            fv->nf = n_faces;
            fv->ni = n_internal_faces;
            // cell -> face lists in ascending face order
            std::vector<int> iptr(n_cells + 1, 0), bptr(n_cells + 1, 0);
            for (int f = 0; f < n_internal_faces; ++f) {
                ++iptr[owner[f] + 1];
                ++iptr[neighbour[f] + 1];
            }
            for (int f = n_internal_faces; f < n_faces; ++f) ++bptr[owner[f] + 1];
            for (int c = 0; c < n_cells; ++c) {
                iptr[c + 1] += iptr[c];
                bptr[c + 1] += bptr[c];
            }
            std::vector<int2> islot(iptr[n_cells]);
            std::vector<int> bface(bptr[n_cells]);
            std::vector<int> fi(iptr.begin(), iptr.end() - 1), fb(bptr.begin(), bptr.end() - 1);
            for (int f = 0; f < n_internal_faces; ++f) {
                islot[fi[owner[f]]++] = make_int2(f, neighbour[f]);
                islot[fi[neighbour[f]]++] = make_int2(f, -1 - owner[f]);
            }
            for (int f = n_internal_faces; f < n_faces; ++f) bface[fb[owner[f]]++] = f;
            auto up = [&](const auto* src, size_t cnt) {
                using T = std::remove_const_t<std::remove_pointer_t<decltype(src)>>;
                std::vector<T> h(src, src + cnt);
                return fv->mem.upload(h, fv->st);
            };
            fv->owner = up(owner, n_faces);
            fv->neighbour = up(neighbour, n_internal_faces);
            fv->w = up(weights, n_internal_faces);
            fv->sf = up(face_areas, 3 * static_cast<size_t>(n_faces));
            fv->cf = up(face_centres, 3 * static_cast<size_t>(n_faces));
            fv->cc = up(cell_centres, 3 * static_cast<size_t>(n_cells));
            fv->vol = up(cell_volumes, n_cells);
            fv->kind = up(boundary_kind, nb);
            fv->pout = up(boundary_pressure, nb);
            fv->iptr = fv->mem.upload(iptr, fv->st);
            fv->islot = fv->mem.upload(islot, fv->st);
            fv->bptr = fv->mem.upload(bptr, fv->st);
            fv->bface = fv->mem.upload(bface, fv->st);
            // delta coefficients of every face and non-orthogonal corrections of the internal ones
            // (fv_geometry.cpp:34-50): delta = |S|^2 / max(S.d, 0.05 |S||d|), k = S - d delta,
            // d = centre of the neighbour (or of the boundary face) minus centre of the owner
            std::vector<double> delta(n_faces), corr(3 * static_cast<size_t>(n_internal_faces));
            auto dot = [](const double* a, const double* b) { return (a[0] * b[0] + a[1] * b[1]) + a[2] * b[2]; };
            for (int f = 0; f < n_faces; ++f) {
                const double* s = face_areas + 3 * static_cast<size_t>(f);
                const double* cp = cell_centres + 3 * static_cast<size_t>(owner[f]);
                const double* to = f < n_internal_faces ? cell_centres + 3 * static_cast<size_t>(neighbour[f])
                                                        : face_centres + 3 * static_cast<size_t>(f);
                const double d[3] = {to[0] - cp[0], to[1] - cp[1], to[2] - cp[2]};
                const double area = std::sqrt(dot(s, s));
                const double s_dot_d = std::max(dot(s, d), 0.05 * area * std::sqrt(dot(d, d)));
                if (!(area > 0.0) || !(s_dot_d > 0.0)) fail(CFDB_ERR_BAD_ARG, "cfdb_fv_create: degenerate face " + std::to_string(f));
                delta[f] = area * area / s_dot_d;
                if (f < n_internal_faces)
                    for (int i = 0; i < 3; ++i) corr[3 * static_cast<size_t>(f) + i] = s[i] - d[i] * delta[f];
            }
            fv->delta = fv->mem.upload(delta, fv->st);
            fv->corr = fv->mem.upload(corr, fv->st);
            CFDB_CUDA(cudaStreamSynchronize(fv->st));
        } catch (...) {
            delete fv;
            throw;
        }
        *out = fv;
    });
}

int cfdb_fv_destroy(cfdb_fv* fv) {
    if (fv != nullptr) {
        cudaSetDevice(fv->device);
        delete fv;
    }
    return CFDB_OK;
}

int cfdb_fv_pressure_gradient_device(cfdb_fv* fv, const double* p, double* grad) {
    return guarded_fv([&] {
        fv_gradient(fv, p, grad, nullptr, nullptr, nullptr);
        CFDB_CUDA(cudaStreamSynchronize(fv->st));
    });
}

int cfdb_fv_sizes(const cfdb_fv* fv, int* n_cells, int* n_faces, int* n_internal_faces) {
    if (fv == nullptr) return CFDB_ERR_BAD_ARG;
    if (n_cells) *n_cells = fv->n;
    if (n_faces) *n_faces = fv->nf;
    if (n_internal_faces) *n_internal_faces = fv->ni;
    return CFDB_OK;
}

int cfdb_fv_delta_device(const cfdb_fv* fv, const double** delta) {
    if (fv == nullptr || delta == nullptr) return CFDB_ERR_BAD_ARG;
    *delta = fv->delta;
    return CFDB_OK;
}

int cfdb_fv_hbya_rau_device(cfdb_fv* fv, const double* mom_diag, const double* mom_upper, const double* mom_lower,
                            const double* mom_source, const double* u, double* hbya, double* rau) {
    return guarded_fv([&] {
        fv_hbya_rau(fv, mom_diag, mom_upper, mom_lower, mom_source, u, hbya, rau);
        CFDB_CUDA(cudaStreamSynchronize(fv->st));
    });
}

int cfdb_fv_face_flux_device(cfdb_fv* fv, const double* hbya, const double* rau, const double* fixed_velocity,
                             const double* u_prev, const double* phi_prev, double beta, double* phi_hbya,
                             double* rau_f) {
    return guarded_fv([&] {
        fv_face_flux(fv, hbya, rau, fixed_velocity, u_prev, phi_prev, beta, phi_hbya, rau_f);
        CFDB_CUDA(cudaStreamSynchronize(fv->st));
    });
}

int cfdb_fv_pressure_boundary_device(cfdb_fv* fv, const double* phi_hbya, const double* rau_f, int ref_cell,
                                     double ref_value, double* diag, double* source) {
    return guarded_fv([&] {
        fv_pressure_boundary(fv, phi_hbya, rau_f, ref_cell, ref_value, diag, source);
        CFDB_CUDA(cudaStreamSynchronize(fv->st));
    });
}

int cfdb_fv_non_orth_device(cfdb_fv* fv, const double* grad, const double* rau_f, const double* base_source,
                            double* non_orth, double* source) {
    return guarded_fv([&] {
        fv_non_orth(fv, grad, rau_f, base_source, non_orth, source);
        CFDB_CUDA(cudaStreamSynchronize(fv->st));
    });
}

int cfdb_fv_correct_flux_device(cfdb_fv* fv, const double* phi_hbya, const double* rau_f, const double* non_orth,
                                const double* p_new, double* phi) {
    return guarded_fv([&] {
        fv_correct_flux(fv, phi_hbya, rau_f, non_orth, p_new, phi);
        CFDB_CUDA(cudaStreamSynchronize(fv->st));
    });
}

int cfdb_fv_relax_device(cfdb_fv* fv, const double* p_prev, const double* p_new, double alpha, double* p) {
    return guarded_fv([&] {
        fv_relax(fv, p_prev, p_new, alpha, p);
        CFDB_CUDA(cudaStreamSynchronize(fv->st));
    });
}

int cfdb_fv_correct_velocity_device(cfdb_fv* fv, const double* hbya, const double* rau, const double* grad,
                                    double* u) {
    return guarded_fv([&] {
        if (fv == nullptr || hbya == nullptr || rau == nullptr || grad == nullptr || u == nullptr)
            fail(CFDB_ERR_BAD_ARG, "null argument");
        CFDB_CUDA(cudaSetDevice(fv->device));
        k_correct_velocity<<<grid_cells(fv->n), 256, 0, fv->st>>>(fv->n, hbya, rau, grad, u);
        CFDB_CUDA(cudaGetLastError());
        CFDB_CUDA(cudaStreamSynchronize(fv->st));
    });
}

} // extern "C"
