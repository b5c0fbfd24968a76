// Residual norms of an LDU system (LduMatrix::residual_norms, ldu_matrix.cpp:69-103), used by the
// persistent LDU solve of the C ABI (cfdb_system_solve_ldu; Engine::residual_norms).
#pragma once

#include "common.hpp"


namespace cfdb {

// res = sum |b - A x|, norm = sum (|A x - A x_ref| + |b - A x_ref|) with x_ref = mean(x) (the
// OpenFOAM normalisation; normalised residual = res / (norm + 1e-20)), r2 = sum (b - A x)^2.
struct LduNorms {
    double res = 0.0;
    double norm = 0.0;
    double r2 = 0.0;
};

} // namespace cfdb
