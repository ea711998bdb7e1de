#pragma once
// BiCGStab with the system resident on the SMs (sm_103a): the FP64 solve
// (k_resident.cu) and the mixed form's FP32 inner solve (k_resident32.cu).
//
// One launch runs a chunk of iterations.  Every CTA owns a contiguous block
// of rows and keeps their Krylov vectors in shared memory for the whole
// launch (for the smaller systems the rows' ELL words too), so that only
// what the SpMVs gather goes through memory, and an iteration is three (or
// four) phases separated by group-wide reductions instead of five kernels
// (the smallest systems take resident_two.cuh's form of two):
//   A. v = A p, (rh, v) -> alpha;
//   B. s = r - alpha v, t = A s, (t, s), (t, t), (rh, s), (rh, t) -> omega and
//      beta;
//   C. x += alpha p + omega s, r = s - omega t, p = r + beta (p - omega v),
//      (r, r), (rh, r) -> the convergence and restart tests.
// beta needs rho' = (rh, r) before r exists; it is taken from the sums of
// phase B, (rh, s) - omega (rh, t), so that p is updated in the pass that
// forms r.  The next alpha uses the rho' summed over r itself in phase C, so
// the recurrence's rounding does not accumulate.
//
// What bounds it.  GB300 issues FP64 at 1.68 lanes per clock per SM (saturated
// by four warps) with 64 cycles of latency, so a small system's iteration is a
// chain of dependent FP64 additions, divisions and synchronisations: a warp
// reduction takes 0.2 us, a division 0.27 us, a grid barrier 1.5 us.  Hence:
//  - a reduction's sums go to different warps (one per FP64 unit of the SM),
//    with one arrival and one polling thread per CTA and no thread fence beyond
//    the counter's own release and acquire;
//  - the scalars take one quotient of six dependent operations per reduction
//    (fp_recip.h), square roots only near the decisions they belong to;
//  - the systems of a few thousand rows run in one thread-block cluster
//    (resident_two.cuh): its barrier takes 0.5 us and the gathers read the
//    neighbours' shared memory.
// Every wait on a grid counter is bounded: a CTA that polls kBarrierPolls
// times records the failure in *bar_err and in pinned memory and returns, and
// the others then fail their next waits.  The first CTA may have passed the
// last wait and have written a result all the same, so the host looks at the
// pinned word after every launch, whatever the result says.
#include <algorithm>
#include <mutex>
#include <set>
#include <utility>

#include "fp_convert.h"
#include "krylov_common.cuh"
#include "resident_plan.h"

namespace mhfem {

template <typename T>
struct ResidentArgs {
    const int32_t* cols;
    const T* vals;
    int W;
    int64_t rows;
    int rc;             // rows per CTA
    T *x, *r, *rh, *p, *v, *s, *t;
    const T* b;             // right-hand side: the launch begins the solve (r = b - A x); null: it goes on
    double tol;             // with b: the solve's limits
    int max_iter;
    const int32_t* stop;    // with b: non-zero word: end at once with KS_ASSEMBLY (may be null)
    KrylovScalars* sc;
    KrylovScalars* host;    // pinned copy of sc for the host (may be null)
    double* partials;   // [4 reductions][kSums][CTA]
    unsigned int* bar;  // arrival count, and its value at the last launch's end
    int* bar_err;
    int* host_wait;     // pinned: set by a CTA whose wait gave up (may be null)
    int give_up;        // the CTA whose waits give up (a check of the report; -1: none)
    int max_its;
    int check_mask;     // streamed forms: iterations between the sums over r, less one (1, 2, 4, ... less one)
};

namespace {

__device__ __forceinline__ uint32_t smem_u32(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }

// Address of the same shared variable in CTA `rank` of the cluster.
__device__ __forceinline__ uint32_t map_rank(uint32_t addr, uint32_t rank)
{
    uint32_t a;
    asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(a) : "r"(addr), "r"(rank));
    return a;
}
template <typename T>
__device__ __forceinline__ T ld_cluster(uint32_t addr)
{
    T v;
    if constexpr (sizeof(T) == 8) asm volatile("ld.shared::cluster.f64 %0, [%1];" : "=d"(v) : "r"(addr) : "memory");
    else asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(v) : "r"(addr) : "memory");
    return v;
}
__device__ __forceinline__ void st_cluster(uint32_t addr, double v)
{
    asm volatile("st.shared::cluster.f64 [%0], %1;" ::"r"(addr), "d"(v) : "memory");
}
__device__ __forceinline__ void cluster_arrive() { asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory"); }
__device__ __forceinline__ void cluster_wait() { asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory"); }
__device__ __forceinline__ void cluster_barrier()
{
    cluster_arrive();
    cluster_wait();
}

__device__ __forceinline__ double warp_sum(double v)
{
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

// A thread's sums enter the reductions as FP64 (converted off the FP64 pipe).
__device__ __forceinline__ double widen(double v) { return v; }
__device__ __forceinline__ double widen(float v) { return f32_to_f64(v); }

// Sum of col[lane], col[lane + 32], ... over n values in four chains.
__device__ __forceinline__ double lane_sum(const double* col, int lane, int n)
{
    double a[4] = {0, 0, 0, 0};
    for (int j = lane; j < n; j += 128) {
#pragma unroll
        for (int k = 0; k < 4; ++k)
            if (j + 32 * k < n) a[k] = (j == lane) ? col[j + 32 * k] : a[k] + col[j + 32 * k];
    }
    return (a[0] + a[1]) + (a[2] + a[3]);
}

// Polls after which a wait gives up: kBarrierPolls in the solves (known when
// they are compiled), a parameter of the check of the waits.
struct SolvePolls {
    __device__ __forceinline__ operator unsigned int() const { return kBarrierPolls; }
};
struct CheckPolls {
    unsigned int polls;
    __device__ __forceinline__ operator unsigned int() const { return polls; }
};

// The CTAs of the launch as one group: reductions over all of them and a
// barrier.  CL: one cluster; else the whole (cooperatively launched) grid.
template <bool CL, typename Polls = SolvePolls>
struct Group {
    double* col;     // [kSums][threads]
    double* tot;     // [kSums]
    double* slots;   // cluster: [kinds of reduction][kSums][kMaxCluster]
    int* bad;        // shared: a wait gave up
    double* partials;
    unsigned int* bar;
    int* err;
    int* host_wait;
    int give_up;
    Polls polls;
    // Arrivals that the counter has seen (in the first warp).  The count runs
    // on from launch to launch: the word behind it holds its value at the last
    // launch's end.
    unsigned int target = 0;

    __device__ __forceinline__ void begin()
    {
        if (!CL && threadIdx.x < 32) target = __ldcg(bar + 1);
    }
    // Call once every CTA has passed the launch's last wait.
    __device__ __forceinline__ void end()
    {
        if (!CL && blockIdx.x == 0 && threadIdx.x == 0) bar[1] = target;
    }

    // One thread of the CTA: arrives and waits for the others.  (A poll limit
    // per CTA for give_up, in a register over the kernel, made the streamed forms'
    // iteration 3 to 4% longer.)
    __device__ __forceinline__ void wait()
    {
        if (arrive_and_wait(bar, err, target, polls) && (int)blockIdx.x != give_up) return;
        atomicExch(err, 1);
        *bad = 1;
        if (host_wait) *(volatile int*)host_wait = 1;
    }

    // Barrier of the first NV warps.
    template <int NV>
    __device__ __forceinline__ void sum_warps_sync()
    {
        if constexpr (NV == 1) __syncwarp();
        else asm volatile("bar.sync 1, %0;" ::"n"(NV * 32) : "memory");
    }

    // tot[q] = the sum of every thread's acc[q]; also a barrier that makes
    // the global (or cluster-shared) writes before it visible after it.
    // Reductions of different `kind` alternate, so a kind's buffer is free
    // again when it is written next.  The warps that have no sum to take run
    // side() while the others wait.
    template <int NV, typename T_>
    __device__ __forceinline__ bool reduce(const T_ (&acc)[NV], int kind)
    {
        return reduce<NV>(acc, kind, [](int) {});
    }
    template <int NV, typename T_, typename Side>
    __device__ __forceinline__ bool reduce(const T_ (&acc)[NV], int kind, Side&& side)
    {
        const int T = blockDim.x, lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nc = gridDim.x;
#pragma unroll
        for (int q = 0; q < NV; ++q) col[q * T + threadIdx.x] = widen(acc[q]);
        __syncthreads();
        if constexpr (CL) {
            double* mine = slots + (kind * kSums + warp) * kMaxCluster;
            if (warp < NV) {
                const double v = warp_sum(lane_sum(col + warp * T, lane, T));
                if (lane < nc) st_cluster(map_rank(smem_u32(mine + blockIdx.x), lane), v);
            }
            cluster_arrive();
            if (warp >= NV) side(warp - NV);
            cluster_wait();
            if (warp < NV) {
                double v = lane < nc ? mine[lane] : 0.0;
#pragma unroll
                for (int o = kMaxCluster / 2; o > 0; o >>= 1)
                    if (o < nc) v += __shfl_xor_sync(0xffffffffu, v, o);
                if (lane == 0) tot[warp] = v;
            }
            __syncthreads();
            return true;
        }
        else {
            if (warp < NV) {
                double* mine = partials + (int64_t)(kind * kSums + warp) * nc;
                const double v = warp_sum(lane_sum(col + warp * T, lane, T));
                if (lane == 0) __stcg(mine + blockIdx.x, v);
                // one arrival and one polling thread per CTA for all the sums:
                // more of either slow the counter's line down
                sum_warps_sync<NV>();
                if (warp == 0) {
                    target += nc;
                    if (lane == 0) wait();
                }
                sum_warps_sync<NV>();
                const bool ok = *(volatile int*)bad == 0;
                double a[5] = {0, 0, 0, 0, 0};  // at most one CTA per SM: 152 partials in one pass
                if (ok)
                    for (int b = lane; b < nc; b += 160) {
                        double w[5];
#pragma unroll
                        for (int k = 0; k < 5; ++k) w[k] = b + 32 * k < nc ? __ldcg(mine + b + 32 * k) : 0.0;
#pragma unroll
                        for (int k = 0; k < 5; ++k) a[k] = b == lane ? w[k] : a[k] + w[k];
                    }
                const double s = warp_sum(((a[0] + a[1]) + (a[2] + a[3])) + a[4]);
                if (lane == 0) tot[warp] = s;
            }
            else
                side(warp - NV);
            __syncthreads();
            return *bad == 0;
        }
    }

    __device__ __forceinline__ bool barrier() { return barrier([](int) {}); }
    // The warps behind the first run side() while it waits.
    template <typename Side>
    __device__ __forceinline__ bool barrier(Side&& side)
    {
        if constexpr (CL) {
            cluster_barrier();
            return true;
        }
        else {
            __syncthreads();
            if (threadIdx.x < 32) {
                target += gridDim.x;
                if (threadIdx.x == 0) wait();
            }
            else
                side((int)(threadIdx.x >> 5) - 1);
            __syncthreads();
            return *bad == 0;
        }
    }
};

// Limits that decide a common iteration's end without a square root or a
// quotient: (tol ||b||)^2 and (kRestartEps ||rh||)^2, each with a margin far
// above the rounding of the comparison it stands for.
struct EndLimits {
    double conv2, restart2;
};
__device__ __forceinline__ EndLimits end_limits(const KrylovScalars& S)
{
    const double thr = S.tol * S.bnorm, e = kRestartEps * S.rhnorm;
    return {thr * thr * (1.0 + 1e-12), e * e * (1.0 + 1e-9)};
}

// The decisions at the end of an iteration, as scalars_beta's (k_krylov.cu):
// non-finite, converged, iteration cap, breakdown, restart.  S->res holds the
// residual when the solve or the chunk ends.
__device__ __forceinline__ void end_of_iteration(KrylovScalars* S, EndLimits* lim, double rr, double rho,
                                                 bool last_of_chunk)
{
    const double rho2 = rho * rho, bound2 = lim->restart2 * rr;
    S->it += 1;
    S->rr = rr;
    if (!last_of_chunk && S->it < S->max_iter && finite_bits(rr) && finite_bits(rho2) &&
        greater_bits(lim->conv2, kTiny) && greater_bits(rr, lim->conv2) && greater_bits(bound2, kTiny) &&
        greater_bits(rho2, bound2) && !zero_bits(S->omega) && !zero_bits(S->rho)) {
        S->rho = rho;
        S->restart = 0;
        return;
    }
    S->res = sqrt(rr) / S->bnorm;
    S->restart = 0;
    if (!finite(S->res)) { S->status = KS_NOTFINITE; S->done = 1; }
    else if (S->res < S->tol) { S->status = KS_CONVERGED; S->done = 1; }
    else if (S->it >= S->max_iter) { S->status = KS_MAXITER; S->done = 1; }
    else if (S->omega == 0 || S->rho == 0) { S->status = KS_BREAKDOWN; S->done = 1; }
    else if (fabs(rho) <= kRestartEps * sqrt(rr) * S->rhnorm) {
        // shadow residual (numerically) orthogonal to r: restart with rh = p = r
        S->restart = 1;
        S->rho = rr;
        S->rhnorm = sqrt(rr);
        *lim = end_limits(*S);
    }
    else
        S->rho = rho;
}

// The end of an iteration of the streamed forms that did not sum over r, with
// rho' from phase B's sums.  False, and nothing changed, if by end_of_iteration's
// conditions with the last known ||r|| it may end the solve or restart it: then
// the sums are formed after all and end_of_iteration decides on the residual
// itself (r may have vanished, and with it rho').
__device__ __forceinline__ bool end_unchecked(KrylovScalars* S, const EndLimits* lim, double rho)
{
    const double rho2 = rho * rho, bound2 = lim->restart2 * S->rr;
    if (!finite_bits(rho2) || !greater_bits(bound2, kTiny) || !greater_bits(rho2, bound2) || zero_bits(S->omega) ||
        zero_bits(S->rho))
        return false;
    S->it += 1;
    S->restart = 0;
    S->rho = rho;
    return true;
}

// What a launch begins with: the scalars of a new solve (or those the last
// launch left), nothing else to do if the solve is over.  False when it is.
template <typename R>
__device__ __forceinline__ bool begin_resident(const ResidentArgs<R>& g, KrylovScalars* S, EndLimits* limits, int* bad)
{
    if (threadIdx.x == 0) {
        if (g.b) {
            *S = KrylovScalars{};
            S->tol = g.tol;
            S->max_iter = g.max_iter;
            if (g.stop && *g.stop) {
                S->status = KS_ASSEMBLY;
                S->done = 1;
            }
        }
        else {
            *S = *g.sc;
            *limits = end_limits(*S);
        }
        *bad = 0;
    }
    __syncthreads();
    if (!S->done) return true;  // the same in every CTA
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        *g.sc = *S;
        if (g.host) *g.host = *S;
    }
    return false;
}

// ||r||, ||b|| of a new solve.
__device__ __forceinline__ void first_residual(KrylovScalars* S, EndLimits* limits, double rr, double bb)
{
    const double rn = sqrt(rr), bn = sqrt(bb);
    S->bnorm = bn == 0 ? 1.0 : bn;
    S->rho = S->rr = rr;
    S->rhnorm = rn;
    S->res = rn / S->bnorm;
    if (!finite(S->res)) { S->status = KS_NOTFINITE; S->done = 1; }
    else if (S->res < S->tol) { S->status = KS_CONVERGED; S->done = 1; }
    *limits = end_limits(*S);
}

// Two quotients in threads 0 and 32, side by side: omega = ts / tt (and rho' = (rh, s) -
// omega (rh, t) when rho_next is not null), then beta from tt / ts.
__device__ __forceinline__ void scalars_omega_beta(KrylovScalars* S, const double* tot, double inv_rv, double* rho_next)
{
    const double ts = tot[0], tt = tot[1];
    const double num = threadIdx.x == 0 ? ts : tt, den = threadIdx.x == 0 ? tt : ts;
    const double r = recip_newton(den);
    if (threadIdx.x == 0) {
        const double q = quotient(num, den, r);
        S->ts = ts;
        S->tt = tt;
        S->omega = q;
        if (rho_next) *rho_next = fma(-q, tot[3], tot[2]);
        S->half = 0;
        if (!finite_bits(ts) || !finite_bits(tt)) {
            S->status = KS_NOTFINITE;
            S->done = 1;
            S->res = sqrt(S->rr) / S->bnorm;
        }
        // no omega: the solve ends with the half step (scalars_half_step)
        else if (zero_bits(tt)) S->half = 1;
    }
    else
        // beta = (rho' / rho) (alpha / omega) with alpha = rho / (rh, v).  (rh, s) is
        // zero but for rounding, by the choice of alpha: its factor 1 / omega needs
        // no correction.
        S->beta = quotient(fma(tot[2], quotient_product(num, den, r), -tot[3]), S->rv, inv_rv);
}

// A s = 0, with ss = (s, s): with a nonsingular matrix s = 0, and x + alpha p
// solves the system; with a singular one s need not be zero, and the iteration
// breaks down.  (In every other case a half step that would meet the tolerance
// ends its iteration with a smaller ||r||, so ||s|| is formed only here.)
__device__ __forceinline__ void scalars_half_step(KrylovScalars* S, double ss)
{
    S->snorm = sqrt(ss) / S->bnorm;
    S->done = 1;
    if (S->snorm < S->tol) {
        S->res = S->snorm;
        S->it += 1;
        S->status = KS_CONVERGED;
    }
    else {
        S->res = sqrt(S->rr) / S->bnorm;
        S->status = KS_BREAKDOWN;
    }
}

// WW: compile-time ELL width (0: run-time).  MATS: the CTA's ELL words are
// copied to shared memory once.  RECOMP: phase B forms s at each gathered neighbour from its
// r and v (W more FP64 operations per row) instead of publishing s behind a
// barrier of its own.  XS: x in shared memory.
template <typename R, int WW, bool MATS, bool RECOMP, bool XS>
__global__ void __launch_bounds__(kMaxThreads, 1) k_bicgstab_resident(const ResidentArgs<R> g)
{
    extern __shared__ double smem[];
    __shared__ KrylovScalars S;
    __shared__ double tot[kSums];
    __shared__ double s_inv_rv, s_rho_next;
    __shared__ int s_sum;
    __shared__ int bad;
    const int T = blockDim.x, rc = g.rc, W = WW > 0 ? WW : g.W;
    const int64_t base = (int64_t)blockIdx.x * rc, rows = g.rows;
    const int n = (int)max((int64_t)0, min((int64_t)rc, rows - base));
    __shared__ EndLimits limits;
    const bool first = g.b != nullptr;
    if (!begin_resident(g, &S, &limits, &bad)) return;

    double* col = smem;
    R* sr = reinterpret_cast<R*>(col + kSums * T);
    R* srh = sr + rc;
    R* sp = srh + rc;
    R* sv = sp + rc;
    R* st = sv + rc;
    R* ss = RECOMP ? st + rc : sr;  // without RECOMP s takes r's place, and the next r that of t
    R* sa = st + (RECOMP ? 2 : 1) * rc;
    R* const xp = XS ? sa : g.x + base;
    if (XS) sa += rc;
    uint32_t* scol = reinterpret_cast<uint32_t*>(sa + (int64_t)(MATS ? W : 0) * rc);

    for (int m = threadIdx.x; m < n; m += T) {
        if (!first) {
            sr[m] = __ldcg(g.r + base + m);
            srh[m] = __ldcg(g.rh + base + m);
            sp[m] = __ldcg(g.p + base + m);
        }
        if (XS) xp[m] = g.x[base + m];
    }
    if constexpr (MATS)
        for (int k = 0; k < W; ++k)
            for (int m = threadIdx.x; m < n; m += T) {
                const int64_t o = (int64_t)k * rows + base + m;
                const uint32_t c = (uint32_t)__ldg(g.cols + o);
                sa[k * rc + m] = __ldg(g.vals + o);
                scol[k * rc + m] = c;
            }
    Group<false> G{col, tot, nullptr, &bad, g.partials, g.bar, g.bar_err, g.host_wait, g.give_up, {}};
    G.begin();
    __syncthreads();

    // y = self + sum_k a_k gather(c_k) over the CTA's rows; body(m, y).  The
    // streamed form loads the next row's ELL words before the current gathers.
    auto spmv = [&](auto&& self, auto&& gather, auto&& body) {
        if constexpr (MATS) {
            for (int m = threadIdx.x; m < n; m += T) {
                R y = self(m);
                if constexpr (WW > 0) {
                    R xg[WW];
#pragma unroll
                    for (int k = 0; k < WW; ++k) xg[k] = gather(scol[k * rc + m]);
#pragma unroll
                    for (int k = 0; k < WW; ++k) y = fma(sa[k * rc + m], xg[k], y);
                }
                else {
                    for (int k = 0; k < W; ++k) y = fma(sa[k * rc + m], gather(scol[k * rc + m]), y);
                }
                body(m, y);
            }
        }
        else if constexpr (WW > 0 && WW <= 6) {
            int32_t c[WW];
            R a[WW];
            auto load = [&](int m, int32_t(&cc)[WW], R(&aa)[WW]) {
#pragma unroll
                for (int k = 0; k < WW; ++k) {
                    cc[k] = __ldg(g.cols + (int64_t)k * rows + base + m);
                    aa[k] = __ldg(g.vals + (int64_t)k * rows + base + m);
                }
            };
            int m = threadIdx.x;
            if (m < n) load(m, c, a);
            for (; m < n; m += T) {
                int32_t cn[WW];
                R an[WW];
                if (m + T < n) load(m + T, cn, an);
                R xg[WW];
#pragma unroll
                for (int k = 0; k < WW; ++k) xg[k] = gather((uint32_t)c[k]);
                R y = self(m);
#pragma unroll
                for (int k = 0; k < WW; ++k) y = fma(a[k], xg[k], y);
                body(m, y);
#pragma unroll
                for (int k = 0; k < WW; ++k) {
                    c[k] = cn[k];
                    a[k] = an[k];
                }
            }
        }
        else {
            for (int m = threadIdx.x; m < n; m += T) {
                R y = self(m);
                if constexpr (WW > 0) {
                    int32_t c[WW];
                    R a[WW], xg[WW];
#pragma unroll
                    for (int k = 0; k < WW; ++k) {
                        c[k] = __ldg(g.cols + (int64_t)k * rows + base + m);
                        a[k] = __ldg(g.vals + (int64_t)k * rows + base + m);
                    }
#pragma unroll
                    for (int k = 0; k < WW; ++k) xg[k] = gather((uint32_t)c[k]);
#pragma unroll
                    for (int k = 0; k < WW; ++k) y = fma(a[k], xg[k], y);
                }
                else {
                    for (int k = 0; k < W; ++k) {
                        const int64_t o = (int64_t)k * rows + base + m;
                        y = fma(__ldg(g.vals + o), gather((uint32_t)__ldg(g.cols + o)), y);
                    }
                }
                body(m, y);
            }
        }
    };

    if (first) {
        // rh = p = r = b - A x (x gathered from memory), ||r||, ||b||
        R acc[2] = {0, 0};
        for (int m = threadIdx.x; m < n; m += T) {
            R y = g.x[base + m];
            for (int k = 0; k < W; ++k) {
                const int64_t o = (int64_t)k * rows + base + m;
                y = fma(MATS ? sa[k * rc + m] : __ldg(g.vals + o), g.x[__ldg(g.cols + o)], y);
            }
            const R bm = g.b[base + m], rv = bm - y;
            sr[m] = rv;
            srh[m] = rv;
            sp[m] = rv;
            __stcg(g.p + base + m, rv);
            if (RECOMP) __stcg(g.r + base + m, rv);
            acc[0] = fma(rv, rv, acc[0]);
            acc[1] = fma(bm, bm, acc[1]);
        }
        if (!G.reduce(acc, 2)) return;
        if (threadIdx.x == 0) first_residual(&S, &limits, tot[0], tot[1]);
        __syncthreads();
    }

    for (int k = 0; k < g.max_its && !S.done; ++k) {
        // A. v = A p, (rh, v) -> alpha
        {
            R acc[1] = {0};
            spmv([&](int m) { return sp[m]; },
                 [&](uint32_t c) { return g.p[c]; },
                 [&](int m, R y) {
                     sv[m] = y;
                     if (RECOMP) __stcg(g.v + base + m, y);
                     acc[0] = fma(srh[m], y, acc[0]);
                 });
            if (!G.reduce(acc, 0)) return;
            if (threadIdx.x == 0) {
                const double rv = tot[0], inv = recip_newton(rv);
                S.rv = rv;
                S.alpha = quotient(S.rho, rv, inv);
                s_inv_rv = inv;
                if (!finite_bits(rv) || zero_bits(rv)) {
                    S.status = finite_bits(rv) ? KS_BREAKDOWN : KS_NOTFINITE;
                    S.done = 1;
                    S.res = sqrt(S.rr) / S.bnorm;
                }
            }
            __syncthreads();
            if (S.done) break;
        }
        const R alpha = (R)S.alpha;
        // x += f y over the CTA's rows, in the warps that wait for a barrier
        // or a reduction (`used` of them do not): two FP64 operations per row
        // and iteration leave the critical path.  Streamed forms only: with
        // few rows the waiting reduction needs the FP64 pipe more (49,408 rows
        // 12.4 us per iteration without, 12.7 with it).  With x in memory only
        // at width 4, where registers are left to load four rows together: the
        // wait does not cover a load per pass (1,515,000 rows in FP32, width 6:
        // 42.8 us without, 53.8 with it).
        constexpr bool side_x = !MATS && (XS || WW == 4);
        auto add_to_x = [&](R f, const R* y, int w, int used) {
            const int step = T - 32 * used;
            constexpr int U = WW == 4 ? 4 : 1;
            for (int m0 = w * 32 + (threadIdx.x & 31); m0 < n; m0 += U * step) {
                R xv[U];
#pragma unroll
                for (int u = 0; u < U; ++u)
                    if (m0 + u * step < n) xv[u] = xp[m0 + u * step];
#pragma unroll
                for (int u = 0; u < U; ++u)
                    if (m0 + u * step < n) xp[m0 + u * step] = fma(f, y[m0 + u * step], xv[u]);
            }
        };
        // B. s, t = A s, the four sums -> omega, beta
        {
            R acc[4] = {0, 0, 0, 0};
            auto dots = [&](int m, R sv_, R y) {
                const R h = srh[m];
                acc[0] = fma(y, sv_, acc[0]);
                acc[1] = fma(y, y, acc[1]);
                acc[2] = fma(h, sv_, acc[2]);
                acc[3] = fma(h, y, acc[3]);
            };
            if constexpr (RECOMP) {
                spmv([&](int m) { return ss[m] = fma(-alpha, sv[m], sr[m]); },
                     [&](uint32_t c) { return fma(-alpha, g.v[c], g.r[c]); },
                     [&](int m, R y) {
                         st[m] = y;
                         dots(m, ss[m], y);
                     });
            }
            else {
                for (int m = threadIdx.x; m < n; m += T) {
                    const R sv_ = fma(-alpha, sv[m], sr[m]);
                    ss[m] = sv_;
                    __stcg(g.s + base + m, sv_);
                }
                if (!G.barrier([&](int w) { if (side_x) add_to_x(alpha, sp, w, 1); })) return;
                spmv([&](int m) { return ss[m]; }, [&](uint32_t c) { return g.s[c]; },
                     [&](int m, R y) {
                         st[m] = y;
                         dots(m, ss[m], y);
                     });
            }
            if (!G.reduce(acc, 1)) return;
            if (threadIdx.x == 0 || threadIdx.x == 32) scalars_omega_beta(&S, tot, s_inv_rv, &s_rho_next);
            __syncthreads();
            if (S.done) break;
        }
        if (S.half) {
            R acc[1] = {0};
            for (int m = threadIdx.x; m < n; m += T) {
                if (!side_x) xp[m] = fma(alpha, sp[m], xp[m]);
                acc[0] = fma(ss[m], ss[m], acc[0]);
            }
            if (!G.reduce(acc, 2)) return;
            if (threadIdx.x == 0) scalars_half_step(&S, tot[0]);
            __syncthreads();
            break;
        }
        // C. r, p (and x, while the sums go round), (r, r), (rh, r) -> convergence, restart
        {
            const R omega = (R)S.omega, beta = (R)S.beta;
            const bool check = MATS || ((S.it + 1) & g.check_mask) == 0 || k + 1 == g.max_its ||
                               S.it + 1 >= S.max_iter;
            R acc[2] = {0, 0};
            R* const rnew = RECOMP ? sr : st;
            for (int m = threadIdx.x; m < n; m += T) {
                const R sv_ = ss[m], pv = sp[m];
                if (!side_x) xp[m] = fma(omega, sv_, fma(alpha, pv, xp[m]));
                const R rv = fma(-omega, st[m], sv_);
                const R pn = fma(beta, fma(-omega, sv[m], pv), rv);
                rnew[m] = rv;
                sp[m] = pn;
                __stcg(g.p + base + m, pn);
                if (RECOMP) __stcg(g.r + base + m, rv);
                if (check) {
                    acc[0] = fma(rv, rv, acc[0]);
                    acc[1] = fma(srh[m], rv, acc[1]);
                }
            }
            if (check) {
                if (!G.reduce(acc, 2, [&](int w) { if (side_x) add_to_x(omega, ss, w, 2); })) return;
                if (threadIdx.x == 0) end_of_iteration(&S, &limits, tot[0], tot[1], k + 1 == g.max_its);
            }
            else {
                if (!G.barrier([&](int w) { if (side_x) add_to_x(omega, ss, w, 1); })) return;
                if (threadIdx.x == 0) s_sum = !end_unchecked(&S, &limits, s_rho_next);
                __syncthreads();
                if (s_sum) {
                    for (int m = threadIdx.x; m < n; m += T) {
                        const R rv = rnew[m];
                        acc[0] = fma(rv, rv, acc[0]);
                        acc[1] = fma(srh[m], rv, acc[1]);
                    }
                    if (!G.reduce(acc, 2)) return;
                    if (threadIdx.x == 0) end_of_iteration(&S, &limits, tot[0], tot[1], k + 1 == g.max_its);
                }
            }
            if constexpr (!RECOMP) {  // r is where t was; the next s takes its place, the next t that of this s
                st = ss;
                sr = ss = rnew;
            }
            __syncthreads();
            if (S.done) break;
            if (S.restart) {  // rh = p = r; rho = (r, r)
                acc[0] = 0;
                for (int m = threadIdx.x; m < n; m += T) {
                    const R rv = sr[m];
                    srh[m] = rv;
                    sp[m] = rv;
                    __stcg(g.p + base + m, rv);
                    acc[0] = fma(rv, rv, acc[0]);
                }
                const R sum[1] = {acc[0]};
                if (!G.reduce(sum, 3)) return;
                if (threadIdx.x == 0) {
                    S.rho = S.rr = tot[0];
                    S.rhnorm = sqrt(tot[0]);
                    limits = end_limits(S);
                }
                __syncthreads();
            }
        }
    }
    for (int m = threadIdx.x; m < n; m += T) {
        if (XS) g.x[base + m] = xp[m];
        g.r[base + m] = sr[m];
        g.rh[base + m] = srh[m];
        g.p[base + m] = sp[m];
    }
    G.end();
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        *g.sc = S;
        if (g.host) *g.host = S;
    }
}

// ---- launches --------------------------------------------------------------------

// Launches a resident kernel: as one cluster (CL) or cooperatively, so that
// every CTA is resident.  cudaErrorCooperativeLaunchTooLarge when the device
// (or a partition of it) has no room; nothing ran then.
template <bool CL, typename Args>
cudaError_t launch_group(void (*kernel)(Args), int ctas, int threads, size_t smem, const Args& a, int dev,
                         cudaStream_t s)
{
    {
        static std::mutex mu;
        static std::set<std::pair<int, const void*>> done;  // (device, kernel) whose attributes are set
        std::lock_guard<std::mutex> lock(mu);
        if (!done.count({dev, (const void*)kernel})) {
            int most = 0;
            cudaError_t e = cudaDeviceGetAttribute(&most, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev);
            cudaFuncAttributes fa{};
            if (e == cudaSuccess) e = cudaFuncGetAttributes(&fa, kernel);
            if (e == cudaSuccess)
                e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         most - (int)fa.sharedSizeBytes);
            if (CL && e == cudaSuccess)
                e = cudaFuncSetAttribute(kernel, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
            if (e != cudaSuccess) return e;
            done.insert({dev, (const void*)kernel});
        }
    }
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3(ctas);
    cfg.blockDim = dim3(threads);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = s;
    cudaLaunchAttribute at[1];
    if (CL) {
        at[0].id = cudaLaunchAttributeClusterDimension;
        at[0].val.clusterDim.x = ctas;
        at[0].val.clusterDim.y = 1;
        at[0].val.clusterDim.z = 1;
    }
    else {
        at[0].id = cudaLaunchAttributeCooperative;
        at[0].val.cooperative = 1;
    }
    cfg.attrs = at;
    cfg.numAttrs = 1;
    const cudaError_t e = cudaLaunchKernelEx(&cfg, kernel, a);
    return e == cudaErrorInvalidClusterSize ? cudaErrorCooperativeLaunchTooLarge : e;
}

template <typename R, int WW, bool MATS, bool RECOMP, bool XS>
cudaError_t launch_resident(const ResidentPlan& P, const ResidentArgs<R>& a, int dev, cudaStream_t s)
{
    return launch_group<false>(k_bicgstab_resident<R, WW, MATS, RECOMP, XS>, P.ctas, P.threads, P.smem, a, dev, s);
}

template <typename R, int WW>
cudaError_t launch_form(const ResidentPlan& P, const ResidentArgs<R>& a, int dev, cudaStream_t s)
{
    if (P.mats && P.recomp) return launch_resident<R, WW, true, true, true>(P, a, dev, s);
    if constexpr (sizeof(R) == 8)
        if (P.mats) return launch_resident<R, WW, true, false, true>(P, a, dev, s);
    if (P.x_in_smem) return launch_resident<R, WW, false, false, true>(P, a, dev, s);
    return launch_resident<R, WW, false, false, false>(P, a, dev, s);
}

}  // namespace
// resident_two.cuh, compiled apart (k_resident_two.cu)
cudaError_t launch_two(int width, bool cluster, int ctas, int threads, size_t smem, const ResidentArgs<double>& a,
                       int dev, cudaStream_t s);
cudaError_t launch_two(int width, bool cluster, int ctas, int threads, size_t smem, const ResidentArgs<float>& a,
                       int dev, cudaStream_t s);
namespace {

cudaError_t device_plan(int64_t rows, int width, size_t real, int* dev, ResidentPlan* P)
{
    cudaError_t e = cudaGetDevice(dev);
    if (e != cudaSuccess) return e;
    int most = 0;
    e = cudaDeviceGetAttribute(&most, cudaDevAttrMaxSharedMemoryPerBlockOptin, *dev);
    if (e != cudaSuccess) return e;
    *P = plan_resident(rows, width, real, sm_count(*dev), (size_t)most);
    return cudaSuccess;
}

// b: begins the solve of A x = b (tol, max_iter, stop); null: goes on with it.
template <typename R>
cudaError_t iterate_resident(const EllMatrix& A, const R* vals, const R* b, double tol, int max_iter,
                             const int32_t* stop, R* x, R* r, R* rh, R* p, R* v, R* sv, R* t, KrylovScalars* sc,
                             KrylovScalars* host, KrylovWork& W, int iters, cudaStream_t s)
{
    int dev = 0;
    ResidentPlan P;
    cudaError_t e = device_plan(A.rows, A.width, sizeof(R), &dev, &P);
    if (e != cudaSuccess) return e;
    if (!P.ok || (int64_t)4 * kSums * P.ctas > (int64_t)W.grid * kPartStride) return cudaErrorCooperativeLaunchTooLarge;
    const ResidentArgs<R> a{A.cols, vals, A.width, A.rows, P.rc, x, r, rh, p, v, sv, t, b, tol,
                            max_iter, stop, sc, host, W.partials, W.counters + kBarrierFirst,
                            reinterpret_cast<int*>(W.counters + kBarrierError), W.host_wait, W.give_up, iters,
                            P.check_every - 1};
    if (P.two) return launch_two(A.width, P.cluster, P.ctas, P.threads, P.smem, a, dev, s);
    MHFEM_WIDTH_DISPATCH(A.width, e = (launch_form<R, WW>(P, a, dev, s)));
    return e;
}

}  // namespace

}  // namespace mhfem
