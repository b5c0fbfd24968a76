// The persistent LDU solve behind cfdb_system_solve_ldu (capi.cu), for callers that solve one matrix
// several times in a row.
#pragma once

#include "../../include/cfdb.h"

namespace cfdb {

// cfdb_system_solve_ldu on device arrays. same_matrix: diag, upper and lower are those of this
// system's last solve_ldu_step call and unchanged since, so the level-0 values are not scattered
// again. The arrays must be ready in the order of the system's stream; x is complete in that order
// when the call returns. Throws cfdb::Error.
void solve_ldu_step(cfdb_system* sys, const double* diag, const double* upper, const double* lower,
                    const double* source, double* x, const cfdb_ldu_settings& settings, const cfdb_amg_settings& amg,
                    bool same_matrix, cfdb_ldu_result& result);

} // namespace cfdb
