// Host check of the resident solves' launch shapes (resident_plan.h): reads
// lines "rows width bytes_per_value sms smem_max" from stdin and prints the
// plan for each, and whether GMRES runs resident.
#include <cstdio>

#include "resident_plan.h"

int main()
{
    long long rows = 0;
    int width = 0, real = 0, sms = 0;
    unsigned long long smem = 0;
    while (std::scanf("%lld %d %d %d %llu", &rows, &width, &real, &sms, &smem) == 5) {
        const mhfem::ResidentPlan P = mhfem::plan_resident(rows, width, (size_t)real, sms, (size_t)smem);
        std::printf("%d %d %d %d %d %d %d %d %d %llu %d %d\n", P.ok, P.two, P.cluster, P.mats, P.recomp, P.x_in_smem,
                    P.ctas, P.threads, P.rc, (unsigned long long)P.smem, P.two ? mhfem::kPassThreads : mhfem::kMaxThreads,
                    mhfem::gmres_resident_fits(rows, width));
    }
    return 0;
}
