// Check of ldp::share_out (how a persistent FP32 launch shares few items out
// over its warps) over shapes and item counts: one launch whose lanes are all
// idle claims every item by its warps' shares alone, and no warp has a share
// that the others' hold already.
// Prints "ok" or the first violation and exits non-zero.
#include <algorithm>
#include <cstdio>
#include <initializer_list>

#include "ldp_share.h"

int main() {
    for (unsigned sms : {1u, 2u, 7u, 148u})
        for (unsigned wps = 1; wps <= 48; ++wps) {
            const unsigned warps = sms * wps, lanes = warps * 32, step = lanes > 4096 ? 13 : 1;
            for (unsigned n = 1; n <= lanes + 2; n += n + 64 > lanes ? 1 : step) {
                const ldp::Share s = ldp::share_out(n, sms, wps);
                const bool fits = s.warps >= 1 && s.warps <= warps && s.lanes >= 1 && s.lanes <= 32;
                const unsigned long long first = (unsigned long long)s.warps * s.lanes;
                const bool claimed = first >= std::min(n, lanes);
                const bool few = (s.warps == warps && s.lanes == 32) || (s.warps - 1) * (unsigned long long)s.lanes < n;
                if (!fits || !claimed || !few) {
                    std::printf("%u SMs, %u warps each, %u items: %u warps of %u lanes\n", sms, wps, n, s.warps, s.lanes);
                    return 1;
                }
            }
            if (ldp::share_out(0, sms, wps).lanes != 32) {
                std::printf("no items\n");
                return 1;
            }
        }
    std::printf("ok\n");
    return 0;
}
