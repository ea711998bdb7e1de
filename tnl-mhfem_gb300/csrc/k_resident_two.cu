// The resident BiCGStab with two reductions per iteration (resident_two.cuh).
#include "resident_two.cuh"

namespace mhfem {

namespace {

template <typename R>
cudaError_t launch_two_t(int width, bool cluster, int ctas, int threads, size_t smem, const ResidentArgs<R>& a, int dev,
                         cudaStream_t s)
{
    cudaError_t e = cudaErrorInvalidValue;
    MHFEM_WIDTH_DISPATCH(width, e = (cluster ? launch_group<true>(k_bicgstab_two<R, WW, true>, ctas, threads, smem, a, dev, s)
                                             : launch_group<false>(k_bicgstab_two<R, WW, false>, ctas, threads, smem, a, dev, s)));
    return e;
}

}  // namespace

cudaError_t launch_two(int width, bool cluster, int ctas, int threads, size_t smem, const ResidentArgs<double>& a,
                       int dev, cudaStream_t s)
{
    return launch_two_t<double>(width, cluster, ctas, threads, smem, a, dev, s);
}

cudaError_t launch_two(int width, bool cluster, int ctas, int threads, size_t smem, const ResidentArgs<float>& a, int dev,
                       cudaStream_t s)
{
    return launch_two_t<float>(width, cluster, ctas, threads, smem, a, dev, s);
}

}  // namespace mhfem
