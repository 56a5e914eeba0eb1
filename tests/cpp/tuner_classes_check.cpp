// Checks that merged FP64 sets whose grid is fixed (one chunk per block) share
// no autotuner class with larger ones: run by tests/test_tuner_classes.py.
#include <cstdio>

#include "../../ns3d_gb300/csrc/tuner.h"

int main() {
    for (int sms : {132, 152, 160})
        for (int share = 1; share <= 16; ++share) {
            const long limit = sms / share;  // plan_krylov: one chunk per block up to here
            for (long n = 1; n <= limit; ++n)
                for (long m = limit + 1; m < 4 * limit; ++m)
                    if (ns3d::tuner_key(0, ns3d::fixed_grid_units(n, limit), share) == ns3d::tuner_key(0, m, share)) {
                        std::printf("FAILED %d SMs, %d lanes: %ld and %ld chunks\n", sms, share, n, m);
                        return 1;
                    }
        }
    std::printf("OK\n");
    return 0;
}
