// The FP64 BiCGStab resident on the SMs (resident.cuh).
#include "resident.cuh"

namespace mhfem {

bool krylov_resident_fits(int64_t rows, int width, bool fp32)
{
    int dev = 0;
    ResidentPlan P;
    return device_plan(rows, width, fp32 ? sizeof(float) : sizeof(double), &dev, &P) == cudaSuccess && P.ok;
}

cudaError_t krylov_resident_fp64(const EllMatrix& A, const double* b, double tol, int max_iter, const int32_t* stop,
                                 double* x, KrylovWork& W, KrylovScalars* host, int iters, cudaStream_t s)
{
    return iterate_resident<double>(A, A.vals, b, tol, max_iter, stop, x, W.r, W.rh, W.p, W.v, W.s, W.t, W.sc, host,
                                    W, iters, s);
}

}  // namespace mhfem
