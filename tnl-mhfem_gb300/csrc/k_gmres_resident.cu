// Restarted GMRES resident on the SMs (sm_103a, FP64), for the systems of
// gmres_resident_fits: one launch runs up to `max_its` Arnoldi
// iterations, restarts included.  CTAs, rows, clusters, reductions and bounded
// waits are those of the resident BiCGStab (resident.cuh); the algorithm, the
// unnormalized basis (v_i = inv_i u_i) and the solve state are k_gmres.cu's.
//
//  A. z = A u_j -> u_{j+1} and the dot products (z, u_i), i <= j -> h_ij, c_i
//     (with the reorthogonalization, A2: u_{j+1} -= sum c_i u_i and the dot
//     products again);
//  B. u_{j+1} -= sum c_i u_i, ||u_{j+1}||^2, the rotations of the new column;
//  at the end of a cycle x += sum_i y_i inv_i u_i, then r = b - A x -> u_0 and
//  the next cycle's length by the adaptive rule (gmres_restart.h).
//
// What bounds it: like the resident BiCGStab the chain of FP64 latencies, and
// here the sums of up to 32 dot products over the threads and the CTAs (13.2 us
// per iteration on 30,200 rows; 32 us with two fenced grid barriers, a shuffle
// tree per dot product and one thread for the state).  Hence:
//  - a warp adds eight dot products over its lanes in nine additions: each
//    step halves the values a lane still holds instead of adding all of them
//    at every step;
//  - the sums over the CTAs are split over all warps, as many CTAs to a warp
//    load as the number of products leaves lanes;
//  - the state's vectors (Hessenberg column, multipliers, back substitution)
//    go one entry to a lane, and the earlier rotations of a column run in a
//    warp that would wait for the norm's reduction;
//  - the rows' basis vectors stay in shared memory while they fit (read twice
//    per iteration), as do the ELL words.
// Every CTA holds its own copy of the state and applies the same operations to
// the same values, so the copies stay identical and the result deterministic.
#include "gmres_restart.h"
#include "resident.cuh"

namespace mhfem {

namespace {

constexpr int kDots = 32;         // dot products of an iteration at most (kGmresMaxM)
constexpr int kDotChunk = 8;
constexpr int kGmresThreads = 256;
static_assert(kGmresMaxM <= kDots, "one lane per dot product");

struct GmresArgs {
    const int32_t* cols;
    const double* vals;
    int W;
    int64_t rows;
    int rc;
    int reorth;
    int vectors;        // basis vectors held (restart length + 1)
    const double* b;
    double *x, *U;
    GmresState* st;
    GmresCtl* host;     // pinned copy of st->ctl
    double* pdots;      // [2][CTA][kDots]
    double* partials;
    unsigned int* bar;
    int* bar_err;
    int* host_wait;     // as ResidentArgs'
    int give_up;
    int max_its;
};

// Sums of eight values over the warp's lanes: value 4 (lane bit 4) + 2 (bit 3)
// + (bit 2) ends in the lane (and in the four lanes that differ in the low
// two bits).
__device__ __forceinline__ double warp_sum8(double (&a)[kDotChunk], int lane)
{
#pragma unroll
    for (int half = 4; half > 0; half /= 2) {
        const bool hi = (lane & (4 * half)) != 0;
#pragma unroll
        for (int k = 0; k < half; ++k) {
            const double send = hi ? a[k] : a[k + half], keep = hi ? a[k + half] : a[k];
            a[k] = keep + __shfl_xor_sync(0xffffffffu, send, 4 * half);
        }
    }
    double v = a[0];
    v += __shfl_xor_sync(0xffffffffu, v, 2);
    v += __shfl_xor_sync(0xffffffffu, v, 1);
    return v;
}

// WW: compile-time ELL width (0: run-time).  CL: one cluster, everything in
// shared memory.  MEM: basis vectors and ELL words read from memory.
template <int WW, bool CL, bool MEM>
__global__ void __launch_bounds__(kGmresThreads, 1) k_gmres_resident(const GmresArgs g)
{
    static_assert(!(CL && MEM), "the cluster form keeps everything in shared memory");
    constexpr int kWarps = kGmresThreads / 32;
    extern __shared__ double smem[];
    __shared__ GmresState S;
    __shared__ double tot[kSums];
    __shared__ double slots[CL ? 3 * kSums * kMaxCluster : 1];
    __shared__ double dslots[CL ? 2 * kMaxCluster * kDots : 1];
    __shared__ double sh[kWarps][kDots];  // per-warp sums of the dot products, then of their CTA sums
    __shared__ double d[kDots];
    __shared__ double inv_bnorm;
    __shared__ int bad;
    const int T = blockDim.x, rc = g.rc, W = WW > 0 ? WW : g.W, nw = T / 32;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int64_t base = (int64_t)blockIdx.x * rc, rows = g.rows;
    const int n = (int)max((int64_t)0, min((int64_t)rc, rows - base));
    {
        const unsigned long long* src = reinterpret_cast<const unsigned long long*>(g.st);
        unsigned long long* dst = reinterpret_cast<unsigned long long*>(&S);
        for (int k = threadIdx.x; k < (int)(sizeof(GmresState) / 8); k += T) dst[k] = __ldcg(src + k);
        if (threadIdx.x == 0) bad = 0;
    }
    __syncthreads();
    if (S.ctl.done) {  // the same in every CTA
        if (blockIdx.x == 0 && threadIdx.x == 0) *g.host = S.ctl;
        return;
    }
    if (threadIdx.x == 0) inv_bnorm = recip_newton(S.ctl.bnorm);

    double* col = smem;
    double* su = col + kSums * T;  // [vectors][rc]
    double* sa = su + (MEM ? 0 : (int64_t)g.vectors * rc);
    uint32_t* scol = reinterpret_cast<uint32_t*>(sa + (MEM ? 0 : (int64_t)W * rc));
    if constexpr (!MEM) {
        for (int i = 0; i <= S.j; ++i)
            for (int m = threadIdx.x; m < n; m += T) su[i * rc + m] = __ldcg(g.U + (int64_t)i * rows + base + m);
        for (int k = 0; k < W; ++k)
            for (int m = threadIdx.x; m < n; m += T) {
                const int64_t o = (int64_t)k * rows + base + m;
                const uint32_t c = (uint32_t)__ldg(g.cols + o);
                sa[k * rc + m] = __ldg(g.vals + o);
                // cluster: the column's address in its owner's copy of u_0
                scol[k * rc + m] = CL ? map_rank(smem_u32(su + c % rc), c / rc) : c;
            }
    }
    Group<CL> G{col, tot, slots, &bad, g.partials, g.bar, g.bar_err, g.host_wait, g.give_up, {}};
    G.begin();
    if constexpr (CL) cluster_barrier();
    else __syncthreads();

    // the CTA's rows of u_i
    auto u = [&](int i) -> double* { return MEM ? g.U + (int64_t)i * rows + base : su + i * rc; };

    // tot over CTAs of the dot products' block sums sh[warp][0 .. nv) -> d
    auto sum_dots = [&](int nv, int kind) -> bool {
        __syncthreads();
        double v = 0;
        if (lane < nv && (CL || warp == 0))
            for (int w = 0; w < nw; ++w) v += sh[w][lane];
        const double* src;
        int nc = gridDim.x;
        if constexpr (CL) {
            double* mine = dslots + kind * kMaxCluster * kDots;
            if (lane < nv)
                for (int r = warp; r < nc; r += nw)
                    st_cluster(map_rank(smem_u32(mine + blockIdx.x * kDots + lane), r), v);
            cluster_barrier();
            src = mine;
        }
        else {
            double* mine = g.pdots + (int64_t)kind * nc * kDots;
            if (warp == 0) {
                if (lane < nv) __stcg(mine + blockIdx.x * kDots + lane, v);
                __syncwarp();
                G.target += nc;
                if (lane == 0) G.wait();
            }
            __syncthreads();
            if (bad) return false;
            src = mine;
        }
        // `per` CTAs to a warp load, `width` lanes to a CTA
        const int width = nv <= 8 ? 8 : nv <= 16 ? 16 : 32, per = 32 / width, i = lane & (width - 1);
        double a[4] = {0, 0, 0, 0};
        const int step = nw * per;
        for (int c = warp * per + lane / width; c < nc; c += 4 * step) {
            double w[4];
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                const int cc = c + k * step;
                w[k] = cc < nc && i < nv ? (CL ? src[cc * kDots + i] : __ldcg(src + cc * kDots + i)) : 0.0;
            }
#pragma unroll
            for (int k = 0; k < 4; ++k)
                if (c + k * step < nc) a[k] += w[k];
        }
        double s = (a[0] + a[1]) + (a[2] + a[3]);
        if (width <= 16) s += __shfl_xor_sync(0xffffffffu, s, 16);
        if (width <= 8) s += __shfl_xor_sync(0xffffffffu, s, 8);
        __syncthreads();  // sh has been read
        if (lane < nv) sh[warp][lane] = s;
        __syncthreads();
        if (warp == 0) {
            double t = 0;
            if (lane < nv)
                for (int w = 0; w < nw; ++w) t += sh[w][lane];
            d[lane] = t;
        }
        return true;
    };
    // block sums of (u_{j+1}, u_i), i <= j, into sh; u_{j+1} = A u_j first when spmv
    auto dots = [&](int j, bool spmv) {
        double* un = u(j + 1);
        const double* uj = u(j);
        for (int c0 = 0; c0 <= j; c0 += kDotChunk) {
            const int nk = min(kDotChunk, j + 1 - c0);
            double acc[kDotChunk];
#pragma unroll
            for (int k = 0; k < kDotChunk; ++k) acc[k] = 0;
            for (int m = threadIdx.x; m < n; m += T) {
                double z;
                if (spmv && c0 == 0) {
                    const uint32_t off = CL ? (uint32_t)(j * rc * sizeof(double)) : 0u;
                    const double* gj = g.U + (int64_t)j * rows;
                    auto gather = [&](uint32_t c) { return CL ? ld_cluster<double>(c + off) : gj[c]; };
                    z = uj[m];
                    if constexpr (WW > 0) {
                        double a[WW], xg[WW];
                        uint32_t c[WW];
#pragma unroll
                        for (int k = 0; k < WW; ++k) {
                            const int64_t o = (int64_t)k * rows + base + m;
                            c[k] = MEM ? (uint32_t)__ldg(g.cols + o) : scol[k * rc + m];
                            a[k] = MEM ? __ldg(g.vals + o) : sa[k * rc + m];
                        }
#pragma unroll
                        for (int k = 0; k < WW; ++k) xg[k] = gather(c[k]);
#pragma unroll
                        for (int k = 0; k < WW; ++k) z = fma(a[k], xg[k], z);
                    }
                    else {
                        for (int k = 0; k < W; ++k) {
                            const int64_t o = (int64_t)k * rows + base + m;
                            const uint32_t c = MEM ? (uint32_t)__ldg(g.cols + o) : scol[k * rc + m];
                            z = fma(MEM ? __ldg(g.vals + o) : sa[k * rc + m], gather(c), z);
                        }
                    }
                    un[m] = z;
                }
                else
                    z = un[m];
                if (nk == kDotChunk) {
#pragma unroll
                    for (int k = 0; k < kDotChunk; ++k) acc[k] = fma(z, u(c0 + k)[m], acc[k]);
                }
                else {
#pragma unroll
                    for (int k = 0; k < kDotChunk; ++k)
                        if (k < nk) acc[k] = fma(z, u(c0 + k)[m], acc[k]);
                }
            }
            const double v = warp_sum8(acc, lane);
            if ((lane & 3) == 0) sh[warp][c0 + (lane >> 2 & 1) + (lane >> 3 & 1) * 2 + (lane >> 4) * 4] = v;
        }
    };
    // h_ij and c_i from the dot products, one lane each
    auto column = [&](int j, bool second) {
        if (warp == 0 && lane <= j) {
            const double invj = S.inv[j], invi = S.inv[lane], e = invi * d[lane], h = invj * e;
            S.H[lane][j] = second ? S.H[lane][j] + h : h;
            S.c[lane] = invi * e;
        }
        __syncthreads();
    };
    // u_{j+1} -= sum_{i <= j} c_i u_i; its value for row m
    auto orth = [&](int j, int m) {
        double t = u(j + 1)[m];
#pragma unroll 4
        for (int i = 0; i <= j; ++i) t = fma(-S.c[i], u(i)[m], t);
        return t;
    };

    for (int it = 0; it < g.max_its; ++it) {
        const int j = S.j;
        dots(j, true);
        if (!sum_dots(j + 1, 0)) return;
        __syncwarp();
        column(j, false);
        if (g.reorth) {
            double* un = u(j + 1);
            for (int m = threadIdx.x; m < n; m += T) un[m] = orth(j, m);
            dots(j, false);
            if (!sum_dots(j + 1, 1)) return;
            __syncwarp();
            column(j, true);
        }
        // B
        {
            double* un = u(j + 1);
            double acc[1] = {0};
            for (int m = threadIdx.x; m < n; m += T) {
                const double t = orth(j, m);
                un[m] = t;
                if (!CL && !MEM) __stcg(g.U + (int64_t)(j + 1) * rows + base + m, t);
                acc[0] = fma(t, t, acc[0]);
            }
            // the earlier rotations of column j, in one of the warps that wait
            auto rotate = [&](int w) {
                if (w != 0) return;
                const double cs = lane < j ? S.cs[lane] : 0.0, sn = lane < j ? S.sn[lane] : 0.0;
                const double next = lane < j ? S.H[lane + 1][j] : 0.0, cn = cs * next;
                double t = S.H[0][j], before = t;
                for (int k = 0; k < j; ++k) {
                    if (lane == k) before = t;
                    t = fma(-__shfl_sync(0xffffffffu, sn, k), t, __shfl_sync(0xffffffffu, cn, k));
                }
                if (lane < j) S.H[lane][j] = fma(cs, before, sn * next);
                if (lane == 0) S.H[j][j] = t;
            };
            if (!G.reduce(acc, 0, rotate)) return;
            if (warp == 0) {
                // sqrt and reciprocal of ||u||^2 (lane 0) and of the rotated diagonal's square (lane 1)
                const double a = S.H[j][j], invj = S.inv[j], sum = tot[0];
                const double den2 = fma(a, a, (invj * invj) * sum);
                const double r = sqrt(lane == 0 ? sum : den2), ri = r > 0 ? recip_newton(r) : 0.0;
                const double nrm = __shfl_sync(0xffffffffu, r, 0), nrmi = __shfl_sync(0xffffffffu, ri, 0);
                const double den = __shfl_sync(0xffffffffu, r, 1), deni = __shfl_sync(0xffffffffu, ri, 1);
                const double hn = invj * nrm;  // h_{j+1,j}
                // the rotation's cosine and sine and 1 / ||u|| in one pass, a quotient to a lane
                const double top = lane == 0 ? a : lane == 1 ? hn : 1.0, bot = lane < 2 ? den : nrm;
                const double val = bot > 0 ? quotient(top, bot, lane < 2 ? deni : nrmi) : lane == 0 ? 1.0 : 0.0;
                const double cs = __shfl_sync(0xffffffffu, val, 0), sn = __shfl_sync(0xffffffffu, val, 1);
                const double inv = __shfl_sync(0xffffffffu, val, 2);
                // the estimate that ends the cycle; the residual that is reported is formed at the restart
                const double gj = S.g[j], gn = -sn * gj, res = quotient_product(fabs(gn), S.ctl.bnorm, inv_bnorm);
                __syncwarp();
                if (lane == 0) {
                    S.cs[j] = cs;
                    S.sn[j] = sn;
                    S.H[j][j] = den;
                    S.g[j + 1] = gn;
                    S.g[j] = cs * gj;
                    S.inv[j + 1] = inv;
                    GmresCtl& C = S.ctl;
                    C.res = res;
                    C.it += 1;
                    S.j = j + 1;
                    if (!finite_bits(res) || !finite_bits(den)) { C.status = KS_NOTFINITE; C.done = 1; }
                    else if (res < S.tol || j + 1 >= S.m || zero_bits(nrm) || C.it >= S.max_iter) C.cycle_end = 1;
                }
            }
            __syncthreads();
        }
        if (S.ctl.done) break;
        if (!S.ctl.cycle_end) continue;
        // the end of the cycle: y from R y = g column by column, x += sum_i y_i inv_i u_i
        if (warp == 0) {
            const int k = S.j;
            double gi = lane < k ? S.g[lane] : 0.0, y = 0;
            const double ri = lane < k ? recip_newton(S.H[lane][lane]) : 0.0;
            for (int i = k - 1; i >= 0; --i) {
                const double yi = __shfl_sync(0xffffffffu, lane < k ? quotient(gi, S.H[lane][lane], ri) : 0.0, i);
                if (lane == i) y = yi;
                if (lane < i) gi = fma(-S.H[lane][i], yi, gi);
            }
            S.c[lane] = lane < k ? y * S.inv[lane] : 0.0;
        }
        __syncthreads();
        {
            const int k = S.j;
            for (int m = threadIdx.x; m < n; m += T) {
                double t = g.x[base + m];
#pragma unroll 4
                for (int i = 0; i < k; ++i) t = fma(S.c[i], u(i)[m], t);
                __stcg(g.x + base + m, t);
            }
        }
        if (!G.barrier()) return;
        // the restart: r = b - A x -> u_0, the true residual, the next length
        {
            double acc[1] = {0};
            double* u0 = u(0);
            for (int m = threadIdx.x; m < n; m += T) {
                double y = __ldcg(g.x + base + m);
                for (int k = 0; k < W; ++k) {
                    const int64_t o = (int64_t)k * rows + base + m;
                    y = fma(MEM ? __ldg(g.vals + o) : sa[k * rc + m], __ldcg(g.x + __ldg(g.cols + o)), y);
                }
                const double r = g.b[base + m] - y;
                u0[m] = r;
                if (!CL && !MEM) __stcg(g.U + base + m, r);
                acc[0] = fma(r, r, acc[0]);
            }
            if (!G.reduce(acc, 1)) return;
            if (threadIdx.x == 0) {
                GmresCtl& C = S.ctl;
                const double beta = sqrt(tot[0]);
                C.res = beta / C.bnorm;
                S.g[0] = beta;
                S.inv[0] = beta > 0 ? 1.0 / beta : 0.0;
                S.j = 0;
                C.cycle_end = 0;
                if (!finite(C.res)) { C.status = KS_NOTFINITE; C.done = 1; }
                else if (C.res < S.tol) { C.status = KS_CONVERGED; C.done = 1; }
                else if (C.it >= S.max_iter) { C.status = KS_MAXITER; C.done = 1; }
                else {
                    const RestartRule R{S.m_min, S.m_max, S.step_min, S.step_max};
                    S.m = next_restart_with(S.m, S.res_prev > 0 ? C.res / S.res_prev : 0.0, R, S.max_cr, S.min_cr);
                }
                S.res_prev = C.res;
            }
            __syncthreads();
            if (S.ctl.done) break;
        }
    }
    if constexpr (CL) {
        // the basis goes back to memory for the next launch (the grid forms wrote it as they went)
        if (!S.ctl.done)
            for (int i = 0; i <= S.j; ++i)
                for (int m = threadIdx.x; m < n; m += T) g.U[(int64_t)i * rows + base + m] = su[i * rc + m];
    }
    G.end();
    if (blockIdx.x == 0) {
        if (threadIdx.x == 0) *g.host = S.ctl;
        const unsigned long long* src = reinterpret_cast<const unsigned long long*>(&S);
        unsigned long long* dst = reinterpret_cast<unsigned long long*>(g.st);
        for (int k = threadIdx.x; k < (int)(sizeof(GmresState) / 8); k += T) dst[k] = src[k];
    }
    if constexpr (CL) cluster_barrier();  // no CTA leaves while another may still read its shared memory
}

struct GmresPlan {
    bool cluster = false, mem = false;
    int ctas = 0, threads = 0, rc = 0;
    size_t smem = 0;
};

GmresPlan plan_gmres(int64_t rows, int width, int vectors, int sms, size_t smem_max)
{
    GmresPlan P;
    auto fill = [&](int64_t ctas) {
        P.ctas = (int)std::max<int64_t>(1, ctas);
        P.rc = (int)((rows + P.ctas - 1) / P.ctas);
        P.threads = std::min(kGmresThreads, group_threads(P.rc, kGmresThreads));
        P.smem = sizeof(double) * (size_t)kSums * P.threads +
                 (P.mem ? 0 : (sizeof(double) * (vectors + width) + sizeof(int32_t) * width) * (size_t)P.rc);
        return P.smem <= smem_max;
    };
    if (rows <= kClusterRows) {
        int c = 1;
        while (c < kMaxCluster && (int64_t)c * 128 < rows) c *= 2;
        P.cluster = true;
        if (fill(c)) return P;
        P.cluster = false;
    }
    const int64_t ctas = std::min<int64_t>((rows + 127) / 128, sms);
    if (!fill(ctas)) {
        P.mem = true;
        fill(ctas);
    }
    if (P.rc > 0) P.ctas = (int)((rows + P.rc - 1) / P.rc);
    return P;
}

template <int WW, bool CL, bool MEM>
cudaError_t launch_gmres(const GmresPlan& P, const GmresArgs& a, int dev, cudaStream_t s)
{
    return launch_group<CL>(k_gmres_resident<WW, CL, MEM>, P.ctas, P.threads, P.smem, a, dev, s);
}

template <int WW>
cudaError_t launch_gmres_form(const GmresPlan& P, const GmresArgs& a, int dev, cudaStream_t s)
{
    if (P.cluster) return launch_gmres<WW, true, false>(P, a, dev, s);
    if (P.mem) return launch_gmres<WW, false, true>(P, a, dev, s);
    return launch_gmres<WW, false, false>(P, a, dev, s);
}

}  // namespace

cudaError_t gmres_resident(const EllMatrix& A, const double* b, double* x, GmresWork& G, KrylovWork& W, bool reorth,
                           int iters, cudaStream_t s)
{
    int dev = 0, most = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e == cudaSuccess) e = cudaDeviceGetAttribute(&most, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev);
    if (e != cudaSuccess) return e;
    constexpr size_t kStatic = 24 << 10;  // the static shared variables (the solve state, the dot products' slots)
    const GmresPlan P = plan_gmres(A.rows, A.width, G.m + 1, sm_count(dev), (size_t)most - kStatic);
    if ((int64_t)3 * kSums * P.ctas > (int64_t)W.grid * kPartStride ||
        (int64_t)2 * P.ctas * kDots > (int64_t)krylov_grid() * kGmStride)
        return cudaErrorCooperativeLaunchTooLarge;
    const GmresArgs a{A.cols, A.vals, A.width, A.rows, P.rc, reorth ? 1 : 0, G.m + 1, b, x, G.U, G.st, G.host, G.partials,
                      W.partials, W.counters + kBarrierFirst, reinterpret_cast<int*>(W.counters + kBarrierError),
                      W.host_wait, W.give_up, iters};
    MHFEM_WIDTH_DISPATCH(A.width, e = launch_gmres_form<WW>(P, a, dev, s));
    return e;
}

}  // namespace mhfem
