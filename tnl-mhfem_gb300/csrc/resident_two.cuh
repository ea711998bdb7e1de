#pragma once
// The resident BiCGStab with two reductions per iteration (sm_103a, FP64 and
// FP32), for the systems whose iteration is mostly synchronisation: up to
// kTwoEntries off-diagonal entries.
//
// resident.cuh's iteration ends in a barrier because the next SpMV gathers p,
// which the neighbours have to form first.  Here every CTA keeps, for each
// entry of its rows, a copy of the neighbour's p, v and r (or s) in shared
// memory and updates it by the neighbour's own operations, so the copies stay
// bitwise equal to the originals; only v and t are gathered, each behind the
// reduction that its phase ends with anyway:
//   A. x += alpha p + omega s, r = s - omega t, p = r + beta (p - omega v), the
//      same r and p at the neighbours (t gathered); v = A p, (rh, v), (r, r),
//      (rh, r) -> the tests on the finished iteration, alpha;
//   B. s = r - alpha v, the same at the neighbours (v gathered); t = A s, (t, s),
//      (t, t), (rh, s), (rh, t) -> omega, beta.
// Against three reductions an entry costs three more FP64 operations: worth it
// while a reduction (2.5 us over 152 CTAs, 1 us in a cluster) is dearer.
#include "resident.cuh"

namespace mhfem {

namespace {

template <typename R, int WW, bool CL>
__global__ void __launch_bounds__(kPassThreads, 1) k_bicgstab_two(const ResidentArgs<R> g)
{
    extern __shared__ double smem[];
    __shared__ KrylovScalars S;
    __shared__ EndLimits limits;
    __shared__ double tot[kSums];
    __shared__ double s_inv_rv;
    __shared__ int s_rv_status;  // KS_RUNNING, or why (rh, v) ends the solve
    __shared__ double slots[CL ? 4 * kSums * kMaxCluster : 1];
    __shared__ int bad;
    const int T = blockDim.x, rc = g.rc, W = WW > 0 ? WW : g.W;
    const int64_t base = (int64_t)blockIdx.x * rc, rows = g.rows;
    const int n = (int)max((int64_t)0, min((int64_t)rc, rows - base));
    const bool first = g.b != nullptr;
    if (!begin_resident(g, &S, &limits, &bad)) return;

    double* col = smem;
    R* sr = reinterpret_cast<R*>(col + kSums * T);
    R* srh = sr + rc;
    R* sp = srh + rc;
    R* sv = sp + rc;
    R* ss = sv + rc;
    R* st = ss + rc;
    R* sx = st + rc;
    // per entry [k][row]: the matrix value, the neighbour's r or s, p, v, and
    // its column (cluster: the address in its owner's copy of sr)
    R* ea = sx + rc;
    R* er = ea + W * rc;
    R* ep = er + W * rc;
    R* ev = ep + W * rc;
    uint32_t* ec = reinterpret_cast<uint32_t*>(ev + W * rc);

    for (int m = threadIdx.x; m < n; m += T) {
        if (!first) {
            sr[m] = __ldcg(g.r + base + m);
            srh[m] = __ldcg(g.rh + base + m);
            sp[m] = __ldcg(g.p + base + m);
        }
        sx[m] = g.x[base + m];
    }
    for (int k = 0; k < W; ++k)
        for (int m = threadIdx.x; m < n; m += T) {
            const int64_t o = (int64_t)k * rows + base + m;
            const uint32_t c = (uint32_t)__ldg(g.cols + o);
            ea[k * rc + m] = __ldg(g.vals + o);
            ec[k * rc + m] = CL ? map_rank(smem_u32(sr + c % rc), c / rc) : c;
        }
    Group<CL> G{col, tot, slots, &bad, g.partials, g.bar, g.bar_err, g.host_wait, g.give_up, {}};
    G.begin();
    if constexpr (CL) cluster_barrier();
    else __syncthreads();
    const uint32_t off_p = (uint32_t)((char*)sp - (char*)sr), off_v = (uint32_t)((char*)sv - (char*)sr),
                   off_t = (uint32_t)((char*)st - (char*)sr);
    auto gather = [&](const R* mem, uint32_t off, uint32_t c) { return CL ? ld_cluster<R>(c + off) : mem[c]; };
    // y += sum_k a_k fn(e), e the position of row m's entry k; its gathered
    // values are loaded first, by pre(c)
    auto entries = [&](int m, R y, auto&& pre, auto&& fn) {
        if constexpr (WW > 0) {
            R xg[WW];
#pragma unroll
            for (int k = 0; k < WW; ++k) xg[k] = pre(ec[k * rc + m]);
#pragma unroll
            for (int k = 0; k < WW; ++k) y = fma(ea[k * rc + m], fn(k * rc + m, xg[k]), y);
        }
        else {
            for (int k = 0; k < W; ++k) y = fma(ea[k * rc + m], fn(k * rc + m, pre(ec[k * rc + m])), y);
        }
        return y;
    };

    if (first) {
        // rh = p = r = b - A x (x gathered from memory), ||r||, ||b||
        R acc[2] = {0, 0};
        for (int m = threadIdx.x; m < n; m += T) {
            R y = sx[m];
            for (int k = 0; k < W; ++k) y = fma(ea[k * rc + m], g.x[__ldg(g.cols + (int64_t)k * rows + base + m)], y);
            const R bm = g.b[base + m], rv = bm - y;
            sr[m] = rv;
            srh[m] = rv;
            sp[m] = rv;
            if (!CL) {
                __stcg(g.r + base + m, rv);
                __stcg(g.p + base + m, rv);
            }
            acc[0] = fma(rv, rv, acc[0]);
            acc[1] = fma(bm, bm, acc[1]);
        }
        if (!G.reduce(acc, 2)) return;
        if (threadIdx.x == 0) first_residual(&S, &limits, tot[0], tot[1]);
        __syncthreads();
    }

    // x += alpha p + omega s, r = s - omega t, p = r + beta (p - omega v) of row m
    auto advance = [&](int m, R alpha, R omega, R beta) {
        const R s = ss[m], p = sp[m];
        sx[m] = fma(omega, s, fma(alpha, p, sx[m]));
        const R r = fma(-omega, st[m], s);
        sr[m] = r;
        return sp[m] = fma(beta, fma(-omega, sv[m], p), r);
    };
    bool load = true;  // the neighbours' r and p are to be gathered (the first iteration of a launch, a restart)
    for (int k = 0; k < g.max_its && !S.done;) {
        // A. (x, r, p of the last iteration,) v = A p -> its tests, alpha
        {
            R acc[3] = {0, 0, 0};
            const R alpha = (R)S.alpha, omega = (R)S.omega, beta = (R)S.beta;
            for (int m = threadIdx.x; m < n; m += T) {
                R y;
                if (load) {
                    const R p = sp[m];
                    y = entries(m, p, [&](uint32_t c) { return gather(g.p, off_p, c); },
                                [&](int e, R pj) {
                                    er[e] = gather(g.r, 0, ec[e]);
                                    return ep[e] = pj;
                                });
                }
                else
                    y = entries(m, advance(m, alpha, omega, beta), [&](uint32_t c) { return gather(g.t, off_t, c); },
                                [&](int e, R tj) {
                                    const R rj = fma(-omega, tj, er[e]);
                                    er[e] = rj;
                                    return ep[e] = fma(beta, fma(-omega, ev[e], ep[e]), rj);
                                });
                sv[m] = y;
                if (!CL) __stcg(g.v + base + m, y);
                const R h = srh[m], r = sr[m];
                acc[0] = fma(h, y, acc[0]);
                acc[1] = fma(r, r, acc[1]);
                acc[2] = fma(h, r, acc[2]);
            }
            if (!G.reduce(acc, 0)) return;
            // the tests on the finished iteration and alpha side by side: a
            // thread's FP64 operations take 64 cycles each
            const double rho = load ? S.rho : tot[2];
            if (threadIdx.x == 0) {
                if (!load) end_of_iteration(&S, &limits, tot[1], rho, false);
            }
            else if (threadIdx.x == 32) {
                const double rv = tot[0], inv = recip_newton(rv);
                S.rv = rv;
                S.alpha = quotient(rho, rv, inv);
                s_inv_rv = inv;
                s_rv_status = !finite_bits(rv) ? KS_NOTFINITE : zero_bits(rv) ? KS_BREAKDOWN : KS_RUNNING;
            }
            __syncthreads();
            if (s_rv_status != KS_RUNNING) {
                __syncthreads();
                if (threadIdx.x == 0 && !S.done && !S.restart) {
                    S.status = s_rv_status;
                    S.done = 1;
                    S.res = sqrt(S.rr) / S.bnorm;
                }
                __syncthreads();
            }
            if (S.done) break;
            if (S.restart) {  // rh = p = r, and phase A again
                for (int m = threadIdx.x; m < n; m += T) {
                    const R r = sr[m];
                    srh[m] = r;
                    sp[m] = r;
                    if (!CL) {
                        __stcg(g.r + base + m, r);
                        __stcg(g.p + base + m, r);
                    }
                }
                if (!G.barrier()) return;
                if (threadIdx.x == 0) S.restart = 0;
                __syncthreads();
                load = true;
                continue;
            }
            load = false;
        }
        const R alpha = (R)S.alpha;
        // B. s, t = A s, the four sums -> omega, beta
        {
            R acc[4] = {0, 0, 0, 0};
            for (int m = threadIdx.x; m < n; m += T) {
                const R s = ss[m] = fma(-alpha, sv[m], sr[m]);
                const R y = entries(m, s, [&](uint32_t c) { return gather(g.v, off_v, c); },
                                    [&](int e, R vj) {
                                        ev[e] = vj;
                                        return er[e] = fma(-alpha, vj, er[e]);
                                    });
                st[m] = y;
                if (!CL) __stcg(g.t + base + m, y);
                const R h = srh[m];
                acc[0] = fma(y, s, acc[0]);
                acc[1] = fma(y, y, acc[1]);
                acc[2] = fma(h, s, acc[2]);
                acc[3] = fma(h, y, acc[3]);
            }
            if (!G.reduce(acc, 1)) return;
            if (threadIdx.x == 0 || threadIdx.x == 32) scalars_omega_beta(&S, tot, s_inv_rv, nullptr);
            __syncthreads();
            if (S.done) break;
        }
        if (S.half) {
            R acc[1] = {0};
            for (int m = threadIdx.x; m < n; m += T) {
                sx[m] = fma(alpha, sp[m], sx[m]);
                acc[0] = fma(ss[m], ss[m], acc[0]);
            }
            if (!G.reduce(acc, 2)) return;
            if (threadIdx.x == 0) scalars_half_step(&S, tot[0]);
            __syncthreads();
            break;
        }
        if (++k == g.max_its) {  // the launch ends: finish the iteration without the next v
            R acc[2] = {0, 0};
            const R omega = (R)S.omega, beta = (R)S.beta;
            for (int m = threadIdx.x; m < n; m += T) {
                advance(m, alpha, omega, beta);
                const R r = sr[m];
                acc[0] = fma(r, r, acc[0]);
                acc[1] = fma(srh[m], r, acc[1]);
            }
            if (!G.reduce(acc, 2)) return;
            if (threadIdx.x == 0) {
                end_of_iteration(&S, &limits, tot[0], tot[1], true);
            }
            __syncthreads();
            if (!S.done && S.restart) {
                for (int m = threadIdx.x; m < n; m += T) srh[m] = sp[m] = sr[m];
                __syncthreads();
                if (threadIdx.x == 0) S.restart = 0;
            }
        }
    }
    __syncthreads();
    for (int m = threadIdx.x; m < n; m += T) {
        g.x[base + m] = sx[m];
        g.r[base + m] = sr[m];
        g.rh[base + m] = srh[m];
        g.p[base + m] = sp[m];
    }
    G.end();
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        *g.sc = S;
        if (g.host) *g.host = S;
    }
    if constexpr (CL) cluster_barrier();  // no CTA leaves while another may still read its shared memory
}

}  // namespace

}  // namespace mhfem
