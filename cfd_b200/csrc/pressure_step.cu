// FlowSolver::pressure_correction (flow_solver.cpp:673-847) as one C-ABI call, composed in C++
// from the library's device entry points in the reference's order, every array in device
// memory: HbyA and rAU from the momentum system (flow_solver.cpp:688-708), the predicted face
// flux and face rAU with the relaxation-independent term (:710-755), the pressure equation
// with its boundary terms and reference cell (:757-796), the non-orthogonal correctors around
// the persistent LDU solve with its AmgCache (:798-822), the conservative flux, pressure
// relaxation and velocity correction (:824-846). Each step is the device kernel that is
// bit-identical to the reference's face or cell loop; the solve is cfdb_system_solve_ldu's.
//
// The loops run on the geometry's stream and the assembly and the solves on the system's; events
// order the two, and the host waits only where a solve reads its scalars back (waiting after every
// launch cost about 20 stream drains a step). The matrix is scattered into the solver once per step:
// the correctors change the source alone.
#include "../../include/cfdb.h"

#include <string>

#include "common.hpp"
#include "fv_step.hpp"
#include "system_step.hpp"

namespace cfdb {
void set_thread_error(const std::string& msg); // capi.cu
}

namespace {

void ok(int rc, const char* what) {
    if (rc != CFDB_OK) {
        char msg[512];
        cfdb_last_error(msg, sizeof msg);
        cfdb::fail(rc, std::string(what) + ": " + msg);
    }
}

// Orders two streams without the host: after(a, b) makes b's later work wait for a's earlier work.
struct Order {
    cudaEvent_t e = nullptr;
    Order() { CFDB_CUDA(cudaEventCreateWithFlags(&e, cudaEventDisableTiming)); }
    ~Order() {
        if (e != nullptr) cudaEventDestroy(e);
    }
    Order(const Order&) = delete;
    Order& operator=(const Order&) = delete;
    void after(cudaStream_t a, cudaStream_t b) const {
        CFDB_CUDA(cudaEventRecord(e, a));
        CFDB_CUDA(cudaStreamWaitEvent(b, e, 0));
    }
};

} // namespace

extern "C" int cfdb_pressure_correction_device(cfdb_system* sys, cfdb_fv* fv, const double* mom_diag,
                                               const double* mom_upper, const double* mom_lower,
                                               const double* mom_source, double* u, double* p,
                                               const double* fixed_velocity, const double* u_prev,
                                               const double* phi_prev, const cfdb_pressure_settings* s,
                                               const cfdb_pressure_workspace* w, cfdb_ldu_result* results,
                                               double* initial_residual) {
    try {
        if (sys == nullptr || fv == nullptr || s == nullptr || w == nullptr || u == nullptr || p == nullptr)
            cfdb::fail(CFDB_ERR_BAD_ARG, "cfdb_pressure_correction_device: null argument");
        int n = 0, nf = 0, ni = 0;
        ok(cfdb_fv_sizes(fv, &n, &nf, &ni), "fv sizes");
        int sys_n = 0, sys_nf = 0;
        ok(cfdb_system_sizes(sys, &sys_n, &sys_nf), "system sizes");
        if (sys_n != n || sys_nf != ni)
            cfdb::fail(CFDB_ERR_BAD_ARG, "cfdb_pressure_correction_device: the system and the geometry differ in size");
        if (s->n_non_orth_correctors < 0) cfdb::fail(CFDB_ERR_BAD_ARG, "negative non-orthogonal correctors");
        if (!w->hbya || !w->rau || !w->phi_hbya || !w->rau_f || !w->diag || !w->source || !w->base_source ||
            !w->p_prev || !w->p_new || !w->non_orth || !w->grad || !w->phi || (ni > 0 && (!w->upper || !w->lower)))
            cfdb::fail(CFDB_ERR_BAD_ARG, "cfdb_pressure_correction_device: workspace array missing");
        const size_t bn = sizeof(double) * static_cast<size_t>(n);
        void* sys_stream = nullptr;
        ok(cfdb_system_stream(sys, &sys_stream), "system stream");
        const cudaStream_t ss = static_cast<cudaStream_t>(sys_stream);
        const cudaStream_t fs = cfdb::fv_stream(fv);
        CFDB_CUDA(cudaSetDevice(cfdb::fv_device(fv))); // the event belongs to the streams' device
        Order order;
        auto copy = [&](double* dst, const double* src) { CFDB_CUDA(cudaMemcpyAsync(dst, src, bn, cudaMemcpyDeviceToDevice, fs)); };
        auto drain = [&]() {
            CFDB_CUDA(cudaStreamSynchronize(fs));
            CFDB_CUDA(cudaStreamSynchronize(ss));
        };
        try {
            // HbyA, rAU; predicted face flux and face rAU (relaxation-independent term when the
            // previous velocity and flux are given and alpha_u < 1)
            cfdb::fv_hbya_rau(fv, mom_diag, mom_upper, mom_lower, mom_source, u, w->hbya, w->rau);
            const bool majumdar = u_prev != nullptr && phi_prev != nullptr && s->alpha_u < 1.0;
            cfdb::fv_face_flux(fv, w->hbya, w->rau, fixed_velocity, majumdar ? u_prev : nullptr,
                               majumdar ? phi_prev : nullptr, majumdar ? 1.0 - s->alpha_u : 0.0, w->phi_hbya, w->rau_f);
            // pressure equation: internal faces (zero source0: base_source serves as it), then the
            // boundary faces and the reference cell
            CFDB_CUDA(cudaMemsetAsync(w->base_source, 0, bn, fs));
            const double* delta = nullptr;
            ok(cfdb_fv_delta_device(fv, &delta), "delta");
            order.after(fs, ss);
            ok(cfdb_system_assemble_pressure_device(sys, w->phi_hbya, w->rau_f, delta, nullptr, w->base_source, -1, 0.0,
                                                    w->upper, w->lower, w->diag, w->source),
               "pressure assembly");
            order.after(ss, fs);
            cfdb::fv_pressure_boundary(fv, w->phi_hbya, w->rau_f, s->ref_cell, s->ref_value, w->diag, w->source);
            copy(w->base_source, w->source);
            copy(w->p_prev, p);
            copy(w->p_new, p);
            // non-orthogonal correctors around the persistent solve
            const int n_solves = s->n_non_orth_correctors + 1;
            if (s->n_non_orth_correctors == 0 || ni == 0)
                CFDB_CUDA(cudaMemsetAsync(w->non_orth, 0, sizeof(double) * static_cast<size_t>(ni > 0 ? ni : 1), fs));
            for (int corr = 0; corr < n_solves; ++corr) {
                if (s->n_non_orth_correctors > 0) {
                    cfdb::fv_gradient(fv, w->p_new, w->grad, nullptr, nullptr, nullptr);
                    cfdb::fv_non_orth(fv, w->grad, w->rau_f, w->base_source, w->non_orth, w->source);
                }
                cfdb_ldu_result r{};
                order.after(fs, ss);
                cfdb::solve_ldu_step(sys, w->diag, w->upper, w->lower, w->source, w->p_new, s->p_solver, s->amg,
                                     /*same_matrix=*/corr > 0, r);
                if (corr == 0 && initial_residual != nullptr) *initial_residual = r.initial_residual;
                if (results != nullptr) results[corr] = r;
                order.after(ss, fs);
                if (w->solve_p != nullptr) copy(w->solve_p + static_cast<size_t>(corr) * n, w->p_new);
                if (w->solve_source != nullptr) copy(w->solve_source + static_cast<size_t>(corr) * n, w->source);
            }
            // conservative flux, relaxed pressure, velocity correction
            cfdb::fv_correct_flux(fv, w->phi_hbya, w->rau_f, w->non_orth, w->p_new, w->phi);
            if (s->relax_p) cfdb::fv_relax(fv, w->p_prev, w->p_new, s->alpha_p, p);
            else copy(p, w->p_new);
            cfdb::fv_gradient(fv, p, w->grad, w->hbya, w->rau, u);
        } catch (...) {
            // the caller's arrays are free to go once the call has returned
            cudaStreamSynchronize(fs);
            cudaStreamSynchronize(ss);
            throw;
        }
        drain();
        return CFDB_OK;
    } catch (const cfdb::Error& e) {
        cfdb::set_thread_error(e.what());
        return e.code;
    } catch (const std::exception& e) {
        cfdb::set_thread_error(e.what());
        return CFDB_ERR_INTERNAL;
    }
}
