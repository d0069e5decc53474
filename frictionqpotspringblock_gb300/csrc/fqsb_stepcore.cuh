/*
 * Parts shared by the step kernels (fqsb_step.cu) and the resident run kernel (fqsb_run.cu): position
 * update, force sum without interactions, the search of a chunk window, and the bookkeeping and stop
 * tests of a finished step.
 */
#ifndef FQSB_STEPCORE_CUH
#define FQSB_STEPCORE_CUH

#include "fqsb_internal.h"

namespace fqsb {

template <unsigned SOFT = 0u>
__device__ __forceinline__ double u_next(const DevSys& s, const double* u0, const double* v0, const double* a0,
                                         int64_t q)
{
    return S_ADD(3, S_ADD(2, u0[q], S_MULC(0, s.f_dt, s.dt, v0[q])), S_MULC(1, s.f_hdt2, s.hdt2, a0[q]));
}

/* f + the Laplace2d force of a particle with neighbours above, below, left and right, in the step's operations (sites
 * 7, 8): 4 u is exact, so its subtraction is one fma (as f + k (...), for a power of two k). */
template <unsigned SOFT>
__device__ __forceinline__ double grid_force(const DevSys& s, double f, double uU, double uD, double uL, double u,
                                             double uR)
{
    const double lap = FQ_FMA(u, -4.0, S_ADD(7, S_ADD(8, FQ_ADD(uU, uD), uL), uR));
    return scale_add(lap, s.s_k, f);
}

/*
 * The force sum of a particle without interactions and damping, f_frame + f_potential, and f_frame itself.
 * d: centre - u of a Cuspy well (the others take w).  k_frame is most often a power of two or general:
 * for a power of two f_frame is exact and one fma forms the sum (site 6, add_scaled; where f_frame is also needed and
 * latency counts, SOFT = 0, the sum is formed from it).
 */
template <int POT, unsigned SOFT = 0u>
__device__ __forceinline__ double frame_pot(const DevSys& s, const double4_32a& w, double d, double up, double uf,
                                            double& ff)
{
    const double fp = POT == POT_CUSPY ? scale<SOFT != 0u>(d, s.s_mu) : pot_force<POT>(s, w, up);
    double x = S_SUB(4, uf, up);
    if (SOFT == 0u) {
        ff = scale(x, s.s_kf);
        return FQ_ADD(ff, fp);
    }
    if (s.s_kf.mode == SCALE_GENERAL) {
        x = fq_smulc(x, s.s_kf.f);
        ff = x;
    }
    else {
        ff = scale(x, s.s_kf); /* read for the residual and frame-force sums only */
    }
    return add_scaled(x, s.s_kf, fp);
}

__device__ __forceinline__ long long absll(long long x)
{
    return x < 0 ? -x : x;
}

__device__ __forceinline__ uint64_t globaltimer()
{
    uint64_t t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}

__device__ __forceinline__ void set_loop(const DevSys& s, unsigned v)
{
    if (s.in_graph) {
        cudaGraphSetConditional((cudaGraphConditionalHandle)s.h_while, v);
    }
}

__device__ __forceinline__ void set_branch(const DevSys& s, unsigned v)
{
    if (s.in_graph) {
        cudaGraphSetConditional((cudaGraphConditionalHandle)s.h_if, v);
    }
}

/* The residual of a step (residual, detail.h:1512-1520) from its sums of f^2 and f_frame^2, if the run asks for it */
__device__ __forceinline__ double residual_of(int flags, double sf, double sff)
{
    if (!(flags & RF_RESID)) {
        return 0.0;
    }
    const double r_fres = FQ_SQRT(sf), r_fext = FQ_SQRT(sff);
    return r_fext != 0.0 ? FQ_DIV(r_fres, r_fext) : r_fres;
}

/*
 * Bookkeeping and stop tests of one finished step on a run-control block c (global memory for the
 * graph path, shared memory for the one-cluster path) and its StopList window `ring`: step and
 * increment counters, frame position, plastic activity, NaN / yield-search errors, the StopList
 * residual test (GooseFEM::Iterate::StopList, detail.h:1780-1783), event, truncation and step limits.
 * sf: the sum of f_frame (RF_FFSUM); r: the residual; now: the time, for the start of a launch.
 */
template <typename CTL>
__device__ __forceinline__ void finalize_ctl(CTL* c, double* ring, double uf, double sf, double r, uint64_t now)
{
    int flags = c->flags;
    c->ticket = 0;
    c->ticket_redo = 0;
    c->n_pending_cta = 0;
    c->n_regen = 0;
    if (flags & RF_FFSUM) {
        c->rec_ffsum[c->step] = sf;
    }
    if (flags & RF_SCHEDULE) {
        c->u_frame = uf;
    }
    c->step += 1;
    if (!(flags & RF_NOINC)) {
        c->inc += 1;
    }
    c->cur ^= 1;
    if (flags & RF_FLOW) {
        c->u_frame = uf;
    }
    if (c->launch_steps == 0) {
        c->launch_t0 = now;
    }
    c->launch_steps += 1;
    if (c->nan_flag) {
        c->error = DERR_NAN;
    }
    else if (c->walk_flag) {
        c->error = DERR_WALK;
    }
    else {
        if (flags & (RF_ACT | RF_TRUNCATE)) {
            long long sv = c->s_sum;
            if (sv != c->s_n) {
                if (c->init) {
                    c->init = 0;
                    c->qs_first = c->inc;
                }
                c->qs_last = c->inc;
            }
            c->s_n = sv;
        }
        if ((flags & RF_EVENT) && c->a_count != 0) {
            c->done = RUN_EVENT;
        }
        if (!c->done && (flags & RF_RESID)) {
            c->last_residual = r;
            int64_t n = c->niter_tol;
            if (n > 0) {
                int64_t pos = c->sl_pos;
                double old = ring[pos];
                if (old >= c->tol) {
                    c->sl_ge_tol -= 1;
                }
                if (old >= c->tol2) {
                    c->sl_ge_tol2 -= 1;
                }
                if (n >= 2) {
                    double second = ring[pos + 1 < n ? pos + 1 : 0];
                    if (second > old) {
                        c->sl_asc -= 1;
                    }
                    double newest = ring[pos > 0 ? pos - 1 : n - 1];
                    if (r > newest) {
                        c->sl_asc += 1;
                    }
                }
                ring[pos] = r;
                c->sl_pos = pos + 1 < n ? pos + 1 : 0;
                if (r >= c->tol) {
                    c->sl_ge_tol += 1;
                }
                if (r >= c->tol2) {
                    c->sl_ge_tol2 += 1;
                }
            }
            if ((c->sl_asc == 0 && c->sl_ge_tol == 0) || c->sl_ge_tol2 == 0) {
                c->done = RUN_CONVERGED;
            }
        }
        if (!c->done && (flags & RF_TRUNCATE)) {
            if ((c->A_truncate > 0 && c->a_count >= c->A_truncate) ||
                (c->S_truncate > 0 && c->s_sum >= c->S_truncate)) {
                c->done = RUN_TRUNCATED;
            }
        }
        if (!c->done && c->step >= c->max_steps) {
            c->done = RUN_MAXITER;
        }
    }
}

/*
 * Stop tests of one finished step (thread 0 of the CTA that finishes the step last); sets the
 * run-loop condition.  sf / sff: sum of f^2 and of f_frame^2 over all particles.
 */
static __device__ __forceinline__ void finalize_step(const DevSys& s, double uf, double sf, double sff)
{
    Ctl* c = s.ctl;
    finalize_ctl(c, s.ring, uf, sf, residual_of(c->flags, sf, sff), globaltimer());
    bool more = !c->done && !c->error && (globaltimer() - c->launch_t0) < c->budget_ns;
    __threadfence();
    set_loop(s, more ? 1u : 0u);
}

/* Commits well li of particle p, between yield positions yl and yr, in the window that starts at `start`. */
__device__ __forceinline__ void commit_well(const DevSys& s, int64_t p, int64_t start, int64_t li, double yl, double yr,
                                            double4_32a& w)
{
    s.cidx[p] = (int32_t)li;
    s.gidx[p] = start + li;
    w = make_wc(s, yl, yr);
    store_well(s, p, w);
}

/*
 * Searches particle p's current chunk window for the well of u (y[i] <= u < y[i+1], the prrng
 * align rule) and commits it when it lies inside the window's margins [min_margin, W - buffer).
 * Returns false when the window must move (then nothing is changed).  On entry w holds the yield
 * positions of the particle's present well (chunk index cidx), which u has left, or NaNs where they
 * are not known.
 *
 * Nearly always u is in the next well on one side: its far yield position is the only load that waits for
 * another one.  (The general search reads the window's ends, the index, and the positions one after the
 * other; a warp waits for whichever lane leaves its well.)
 */
__device__ __forceinline__ bool window_search(const DevSys& s, int64_t p, double u, double4_32a& w)
{
    const int64_t W = s.W;
    const double* y = s.data + p * W;
    int64_t li = s.cidx[p];
    const int64_t start = s.start[p];
    if (w.y <= u) {
        if (li + 2 < W && li + 1 >= s.min_margin && li + 1 < W - s.buffer) {
            const double yr = y[li + 2];
            if (u < yr) {
                commit_well(s, p, start, li + 1, w.y, yr, w);
                return true;
            }
        }
    }
    else if (u < w.x) {
        if (li - 1 >= s.min_margin && li - 1 < W - s.buffer) {
            const double yl = y[li - 1];
            if (yl <= u) {
                commit_well(s, p, start, li - 1, yl, w.x, w);
                return true;
            }
        }
    }
    if (!(y[0] <= u && u < y[W - 1])) {
        return false;
    }
    if (y[li] <= u) {
        while (li + 1 < W && y[li + 1] <= u) {
            ++li;
        }
    }
    else {
        while (li > 0 && y[li] > u) {
            --li;
        }
    }
    if (li < s.min_margin || li >= W - s.buffer) {
        return false;
    }
    commit_well(s, p, start, li, y[li], y[li + 1], w);
    return true;
}

__device__ __forceinline__ bool non_finite(double x)
{
    return (__double_as_longlong(x) & 0x7fffffffffffffffLL) >= 0x7ff0000000000000LL;
}

/* Pairwise sums of x and of y over the 32 lanes (fixed order; both sums share instructions as in
 * cta_tree2): lane 0 gets both. */
__device__ __forceinline__ double2 warp_tree2(double x, double y)
{
    const unsigned full = 0xffffffffu;
    const int lane = threadIdx.x & 31;
    double v;
    {
        const double xa = __shfl_sync(full, x, (2 * lane) & 31), xb = __shfl_sync(full, x, (2 * lane + 1) & 31);
        const double ya = __shfl_sync(full, y, (2 * lane) & 31), yb = __shfl_sync(full, y, (2 * lane + 1) & 31);
        v = add_nospec(lane < 16 ? xa : ya, lane < 16 ? xb : yb);
    }
#pragma unroll
    for (int h = 16; h >= 2; h >>= 1) {
        const double a = __shfl_sync(full, v, (2 * lane) & 31), b = __shfl_sync(full, v, (2 * lane + 1) & 31);
        if (lane < h) {
            v = add_nospec(a, b);
        }
    }
    return make_double2(v, __shfl_sync(full, v, 1));
}

/* Pairwise sum of n = 1, 2, 4 or 8 consecutive values */
__device__ __forceinline__ double sum_consecutive(const double* x, int n)
{
    double r = x[0];
    if (n >= 2) {
        r = add_nospec(r, x[1]);
    }
    if (n >= 4) {
        r = add_nospec(r, add_nospec(x[2], x[3]));
    }
    if (n >= 8) {
        r = add_nospec(r, add_nospec(add_nospec(x[4], x[5]), add_nospec(x[6], x[7])));
    }
    return r;
}

} // namespace fqsb

#endif
