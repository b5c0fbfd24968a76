// The launches behind the cfdb_fv_* entry points (fv.cu), for callers that compose a step from them
// without waiting between them: each checks its arguments and enqueues its kernels on the geometry's
// stream (fv_stream).
#pragma once

#include <cuda_runtime.h>

struct cfdb_fv;

namespace cfdb {

int fv_device(const cfdb_fv* fv);
cudaStream_t fv_stream(const cfdb_fv* fv);
// grad of p; with u also u = hbya - rau grad
void fv_gradient(cfdb_fv* fv, const double* p, double* grad, const double* hbya, const double* rau, double* u);
void fv_hbya_rau(cfdb_fv* fv, const double* mom_diag, const double* mom_upper, const double* mom_lower,
                 const double* mom_source, const double* u, double* hbya, double* rau);
void fv_face_flux(cfdb_fv* fv, const double* hbya, const double* rau, const double* fixed_velocity, const double* u_prev,
                  const double* phi_prev, double beta, double* phi_hbya, double* rau_f);
void fv_pressure_boundary(cfdb_fv* fv, const double* phi_hbya, const double* rau_f, int ref_cell, double ref_value,
                          double* diag, double* source);
void fv_non_orth(cfdb_fv* fv, const double* grad, const double* rau_f, const double* base_source, double* non_orth,
                 double* source);
void fv_correct_flux(cfdb_fv* fv, const double* phi_hbya, const double* rau_f, const double* non_orth,
                     const double* p_new, double* phi);
void fv_relax(cfdb_fv* fv, const double* p_prev, const double* p_new, double alpha, double* p);

} // namespace cfdb
