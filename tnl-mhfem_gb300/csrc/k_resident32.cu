// The mixed form's FP32 inner BiCGStab resident on the SMs (resident.cuh).
#include "resident.cuh"

namespace mhfem {

cudaError_t krylov_resident_fp32(const EllMatrix& A, KrylovWork& W, KrylovScalars* host, int iters, cudaStream_t s)
{
    return iterate_resident<float>(A, A.vals32, nullptr, 0, 0, nullptr, W.x32, W.r32, W.rh32, W.p32, W.v32, W.s32,
                                   W.t32, W.sc32, host, W, iters, s);
}

}  // namespace mhfem
