// Order of the records that a solve's iterations publish to the host (Progress in kernels.cuh). They
// are numbered modulo 2^32 over an engine's whole life: at 36 us an iteration a signed count would
// pass its end after 21 hours, and a record of the solve before would then be taken for the one that
// is waited for. At most two records are outstanding, so the difference decides. Kept free of CUDA
// headers so that a host-only test can check it.
#pragma once

namespace cfdb {

inline bool record_reached(unsigned have, unsigned want) { return static_cast<int>(have - want) >= 0; }

} // namespace cfdb
