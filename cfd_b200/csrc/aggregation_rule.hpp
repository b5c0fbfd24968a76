// Which levels of an AMG setup are aggregated on the device (dsetup.cu): before the start by their size,
// and while it runs by its progress. The result is the host's either way. Kept free of CUDA headers so
// that a host-only test can check it.
#pragma once

namespace cfdb {

// Levels aggregated on the device: those of at least 200K strong entries, but not the dense ones (the
// conflict lists grow with the square of the strong entries per row). The device's time is that of a chain of
// decisions and of some 20 launches, 0.3 to 0.6 ms on the smallest levels; the host's is a few nanoseconds a
// strong entry plus the strength graph's read-back. Measured, one level, device / host in us (strong
// entries, per row): 23K, 5.6: 358 / 116; 94K, 3.8: 345 / 252; 91K, 9.8: 661 / 384; 156K, 9.8: 742 / 624; 190K,
// 5.8: 574 / 235 (box) and 576 / 269 (graded); 237K, 8.6: 782 / 978; 326K, 9.6: 1109 / 1289; 350K, 11.0:
// 1313 / 1261; 374K, 5.8: 725 / 742 (box) and 710 / 954 (graded); 632K, 3.9: 520 / 841; 1.9M, 8.7:
// 1811 / 3178; 2.9M, 3.9: 1113 / 3620.
inline bool device_aggregation(int n, long long ns) { return ns >= 200000 && ns <= 20LL * n; }

// Whether the aggregation of n rows with ns strong entries, `decided` of the rows after `sweeps` sweeps
// (a multiple of 4), is better left to the host: a sweep takes 50 to 95 us, the host's pass 1 to 4 ns a strong
// entry, so that 16 + ns / 100K sweeps are about the host's time. A level gives up when its projected
// sweeps pass 1.5 times that, or 4 times that after the first 4, when a front has only set out. Sweeps
// used, projected after 4 and after 8, and that time in sweeps: box 100^3 24, 47, 21, 75; its second level 24,
// 31, 21, 29; box 160^3 48, 138, 60, 260; its second level 40, 105, 51, 68; tet 95^3x6 28, 28, 27, 220; its second
// level 36, 95, 51, 102. Given up: a band of 200K rows (3100 sweeps, 3100 projected after 4, 19), box 5 x 5
// x 20000 (424, 430, 25), tet 3 x 3 x 4000 x 6 (252, 260, 21; its second level 256, 262, 19), box 1000 x 500 x 1
// (52, 250, 35), box 15 x 15 x 2000 (48, 46 after 8, 24). Aggregation of the first three without the rule, with
// it and on the host alone: 156 / 1.2 / 0.7 ms, 32 / 3.6 / 2.5, 25 / 3.7 / 3.0.
inline bool slow_sweeps(long long sweeps, int n, int ns, int decided) {
    const long long fair = 16 + ns / 100000;
    const long long allowed = sweeps < 8 ? 4 * fair : fair + fair / 2;
    return sweeps * n > allowed * decided;
}

} // namespace cfdb
