// The FP64 BiCGStab resident on the SMs (resident.cuh), and the check of the
// waits between its CTAs.
#include <vector>

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

// ---- check of the bounded waits ----------------------------------------------------

namespace {

constexpr int kCheckThreads = 256;

// Every CTA but `skip` (none if negative) goes through a reduction and a barrier
// of the group, as the solves do, and reports 1 (passed both) or 0 (gave up);
// CTA `skip` never arrives and reports -1, so the others' waits run out after
// max_polls.
__global__ void __launch_bounds__(kCheckThreads) k_wait_check(unsigned int* counters, double* partials, int skip,
                                                              unsigned int max_polls, int* result)
{
    __shared__ double col[kSums * kCheckThreads], tot[kSums];
    __shared__ int bad;
    if ((int)blockIdx.x == skip) {
        if (threadIdx.x == 0) result[blockIdx.x] = -1;
        return;
    }
    if (threadIdx.x == 0) bad = 0;
    Group<false, CheckPolls> G{col,  tot, nullptr, &bad, partials, counters + kBarrierFirst,
                               reinterpret_cast<int*>(counters + kBarrierError), nullptr, -1, {max_polls}};
    G.begin();
    __syncthreads();
    const double one[1] = {threadIdx.x == 0 ? 1.0 : 0.0};
    bool ok = G.reduce(one, 0);
    ok = ok && tot[0] == (double)gridDim.x && G.barrier();  // the same in every thread
    if (ok) G.end();
    if (threadIdx.x == 0) result[blockIdx.x] = ok ? 1 : 0;
}

}  // namespace

cudaError_t grid_barrier_check(int ctas, int skip, unsigned int max_polls, int* passed, int* gave_up, int* flag)
{
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    int nb = 0;
    e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&nb, k_wait_check, kCheckThreads, 0);
    if (e != cudaSuccess) return e;
    if (ctas < 1 || ctas > nb * sm_count(dev)) return cudaErrorInvalidValue;
    // the counters, the CTAs' results, the partial sums
    const size_t words = kCounterWords + (size_t)ctas, sums = (words + 1) / 2;
    double* buf = nullptr;
    e = cudaMalloc(&buf, sizeof(double) * (sums + (size_t)kSums * ctas));
    if (e != cudaSuccess) return e;
    std::vector<unsigned int> res(words, 0);
    e = cudaMemset(buf, 0, sizeof(double) * sums);
    if (e == cudaSuccess) {
        unsigned int* counters = reinterpret_cast<unsigned int*>(buf);
        double* partials = buf + sums;
        int* result = reinterpret_cast<int*>(counters + kCounterWords);
        void* args[] = {(void*)&counters, (void*)&partials, (void*)&skip, (void*)&max_polls, (void*)&result};
        e = cudaLaunchCooperativeKernel((const void*)k_wait_check, dim3(ctas), dim3(kCheckThreads), args, 0, 0);
        if (e == cudaSuccess) e = cudaMemcpy(res.data(), buf, sizeof(unsigned int) * words, cudaMemcpyDeviceToHost);
    }
    cudaFree(buf);
    if (e != cudaSuccess) return e;
    *passed = 0;
    *gave_up = 0;
    for (int b = 0; b < ctas; ++b) {
        const int r = (int)res[kCounterWords + b];
        *passed += r == 1;
        *gave_up += r == 0;
    }
    *flag = (int)res[kBarrierError];
    return cudaSuccess;
}

}  // namespace mhfem
