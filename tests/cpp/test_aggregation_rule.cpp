// Host-only check of the rules by which a level of an AMG setup is aggregated on the device or on the
// host (cfd_b200/csrc/aggregation_rule.hpp), on the progress that levels showed on a B200.
#include "aggregation_rule.hpp"

#include <cstdio>

namespace {

struct Level {
    const char* name;
    int n, ns;
    bool stays;       // settles on the device
    double done[6];   // share of the rows decided after 4, 8, 12, ... sweeps (0: not reached)
};

const Level kLevels[] = {
    {"box 40^3", 64000, 374400, true, {0.557}},
    {"box 64^3", 262144, 1548288, true, {0.262, 0.754, 0.999}},
    {"box 64^3, level 1", 31868, 344128, true, {0.320, 0.736, 0.9999}},
    {"box 100^3", 1000000, 5940000, true, {0.085, 0.382, 0.705, 0.938, 0.999}},
    {"box 100^3, level 1", 121207, 1301600, true, {0.128, 0.387, 0.642, 0.891, 0.9999}},
    {"box 160^3", 4096000, 24422400, true, {0.029, 0.134, 0.227, 0.320, 0.422}},
    {"box 160^3, level 1", 495902, 5298662, true, {0.038, 0.158, 0.310, 0.457, 0.593}},
    {"box 160^3, level 2", 27725, 242252, true, {0.523}},
    {"tet 40^3x6, level 1", 65045, 644286, true, {0.298, 0.760, 0.995}},
    {"tet 60^3x6", 1296000, 5140386, true, {0.546, 0.964}},
    {"tet 60^3x6, level 1", 217904, 2171522, true, {0.132, 0.386, 0.679, 0.916, 0.9999}},
    {"tet 95^3x6", 5144250, 20467076, true, {0.145, 0.292, 0.459, 0.635, 0.822}},
    {"tet 95^3x6, level 1", 861530, 8610926, true, {0.042, 0.156, 0.312, 0.492, 0.678}},
    {"box 400x40x40, level 2", 71862, 721136, true, {0.137, 0.434, 0.771, 0.980}},
    {"box 5x5x20000", 500000, 999950, false, {0.009}},
    {"box 20000x5x5", 500000, 999950, false, {0.013, 0.026, 0.038, 0.051}},
    {"box 500000x1x1", 500000, 999998, false, {0.0005}},
    {"box 1000x500x1", 500000, 1996984, false, {0.016, 0.061, 0.134, 0.234, 0.350}},
    {"box 15x15x2000", 450000, 899550, false, {0.087, 0.175, 0.263, 0.352, 0.441}},
    {"tet 3x3x4000x6", 216000, 563642, false, {0.015, 0.030, 0.046}},
    {"tet 3x3x4000x6, level 1", 59140, 335362, false, {0.015, 0.030, 0.047}},
    {"band of 3 entries", 200000, 399998, false, {0.0013}},
    {"band of 21 entries", 200000, 2828998, false, {0.0009}},
};

} // namespace

int main() {
    int fails = 0;
    for (const Level& l : kLevels) {
        bool left = false;
        for (int b = 0; b < 6 && l.done[b] > 0.0 && !left; ++b)
            left = cfdb::slow_sweeps(4LL * (b + 1), l.n, l.ns, static_cast<int>(l.done[b] * l.n));
        if (left == l.stays || !cfdb::device_aggregation(l.n, l.ns)) {
            std::printf("FAIL %s\n", l.name);
            ++fails;
        }
        // never more than about 1.5 times the host's time, whatever the progress
        if (!cfdb::slow_sweeps(2 * (16 + l.ns / 100000) + 4, l.n, l.ns, l.n - 1)) {
            std::printf("FAIL limit %s\n", l.name);
            ++fails;
        }
    }
    // small, dense and the largest possible levels
    if (cfdb::device_aggregation(32768, 190464) || cfdb::device_aggregation(20000, 400001)) {
        std::printf("FAIL size\n");
        ++fails;
    }
    if (!cfdb::device_aggregation(2147483647, 2147483647) || cfdb::slow_sweeps(4, 2147483647, 2147483647, 2147483647)) {
        std::printf("FAIL largest\n");
        ++fails;
    }
    if (fails == 0) std::printf("ok\n");
    return fails == 0 ? 0 : 1;
}
