// Host build of the blackbody colour's table (rt_planck.h), for the CPU check of the
// look-up against the sum it replaces.  Test-only.
#include <vector>

#include "rt_planck.h"

extern "C" void host_planck(const double* lambda_um, const double* weight, const double* t, long n, double* sum,
                            double* looked_up) {
    const double(*w)[3] = reinterpret_cast<const double(*)[3]>(weight);
    std::vector<double> table(relsim::kPlanckTableDoubles);
    relsim::planck_table_fill(lambda_um, w, table.data());
    for (long i = 0; i < n; ++i) {
        relsim::planck_sum(lambda_um, w, t[i], sum + 3 * i);
        relsim::planck_lookup(table.data(), t[i], looked_up + 3 * i);
    }
}
