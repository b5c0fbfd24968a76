// Host-only check of the order of a solve's progress records (cfd_b200/csrc/progress_rule.hpp),
// where their number passes the ends of the signed and the unsigned range.
#include "progress_rule.hpp"

#include <cstdio>
#include <initializer_list>

int main() {
    using cfdb::record_reached;
    int fails = 0;
    for (const unsigned at : {1u, 1000u, 0x7ffffffeu, 0x7fffffffu, 0x80000000u, 0xfffffffeu, 0xffffffffu, 0u}) {
        for (unsigned behind = 0; behind <= 2; ++behind) {
            // the record `at` is waited for while the newest one is `behind` before it, then after it
            if (record_reached(at - behind, at) != (behind == 0) || !record_reached(at + behind, at)) {
                std::printf("FAIL at %u, %u\n", at, behind);
                ++fails;
            }
        }
    }
    if (fails == 0) std::printf("ok\n");
    return fails == 0 ? 0 : 1;
}
