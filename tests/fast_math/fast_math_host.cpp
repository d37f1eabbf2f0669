// Host build of the step loops' reciprocal and square root (rt_fast_math.h) from a
// given seed, for the CPU check against IEEE division and root.  Test-only.
#include "rt_fast_math.h"

extern "C" void host_refine(const double* v, const double* rcp_seed, const double* rsqrt_seed, long n, double* rcp,
                            double* root) {
    for (long i = 0; i < n; ++i) {
        rcp[i] = relsim::refine_rcp(v[i], rcp_seed[i]);
        root[i] = relsim::refine_sqrt(v[i], rsqrt_seed[i]);
    }
}
