/*
 * Runs of small Line1d / Particles systems in one thread-block cluster (sm_103a, FP64).
 */
#include "fqsb_stepcore.cuh"

#include <cooperative_groups.h>

namespace fqsb {

/*
 * A whole run of a small Line1d / Particles system in one launch of one thread-block cluster (up to
 * 16 CTAs on 16 SMs).  For small N a step on all SMs takes the latency of its grid barrier (4.6 us at
 * N = 1024); here the state stays in registers for the whole run, one particle per thread, the new
 * positions at tile edges cross CTA boundaries through distributed shared memory, and the only wait
 * of a step is one cluster barrier, whose latency is overlapped with what needs no neighbour.
 * What bounds a step: the serial chain of three velocity evaluations (65 cycles per binary64 operation)
 * and the barrier.  N = 1024, Cuspy, us per step, flow and minimise: 1.5 and 2.2; before the neighbours' positions
 * were pushed, the barrier split and the stop tests taken off the chain, 2.0 and 3.1.
 *
 * Every CTA has its particle threads and one control warp (the last warp; that of CTA 0 works).  Time step t:
 *   position update, the tile's outermost positions written to the neighbours' CTAs -> cluster barrier A_t,
 *   beside it frame and potential forces, the first damping force and the well test -> interactions,
 *   velocities, the warp's residual subtree written to CTA 0's slot t % 2 -> positions of step t + 1 -> A_{t+1}
 * Meanwhile, after A_{t+1}, CTA 0's control warp sums step t's subtrees, applies its counters and runs the
 * same stop tests as the graph path (finalize_ctl), and writes its decision to every CTA, which reads it
 * after A_{t+2}.  The decision thus comes two barriers late: when it says stop after step t, the threads
 * have already taken step t + 1, and they restore the state from before that step (positions,
 * velocities, accelerations, and the well and chunk window as they were) -- the step's counters were
 * never applied.  Neither the stop tests nor reads of another CTA's memory are then on the critical path.
 * Arithmetic, the residual tree (aligned power-of-two tiles) and the stop tests are those of
 * k_step_line, and chunk windows move as k_regen moves them, so the results equal the graph path's
 * bit for bit.  Runs that record a trajectory (adjoint) use the graph path.
 */

/* Named barrier 1 over the particle threads of the CTA (the control warp is not in it). */
__device__ __forceinline__ void particle_bar(int n)
{
    asm volatile("bar.sync 1, %0;" ::"r"(n) : "memory");
}

/* particle_bar that also returns whether any particle thread passed a non-zero flag */
__device__ __forceinline__ int particle_bar_or(int n, int flag)
{
    int r;
    asm volatile("{\n\t.reg .pred p, q;\n\tsetp.ne.s32 p, %1, 0;\n\tbar.red.or.pred q, 1, %2, p;\n\t"
                 "selp.s32 %0, 1, 0, q;\n\t}"
                 : "=r"(r)
                 : "r"(flag), "r"(n)
                 : "memory");
    return r;
}

template <int POT, int INTER, bool TH>
__global__ void __launch_bounds__(SMALL_THREADS_MAX + 32, 1) k_run_small(const __grid_constant__ DevSys s)
{
    namespace cg = cooperative_groups;
    cg::cluster_group cluster = cg::this_cluster();
    /* per step parity: the tile's new positions; those of the ring neighbours outside it, written there by the
     * neighbours' CTAs; the decision that the next but one step reads, written by CTA 0 */
    __shared__ double sh_un[2][SMALL_THREADS_MAX];
    __shared__ double sh_edge[2][2];
    __shared__ int sh_stop[2];
    /* CTA 0 keeps the run-control block and the StopList window, and per step parity the warps' residual
     * subtrees and the counters of all CTAs, written there by them */
    __shared__ Ctl sc;
    __shared__ double sring[SMALL_RING_MAX];
    __shared__ double2 spart[2][SMALL_MAX_CTAS * SMALL_THREADS_MAX / 32];
    __shared__ unsigned long long sl_ds[2], sl_da[2];
    __shared__ int sl_nan[2], sl_walk[2];
    /* window moves of this step shared by the CTA's particle threads (fwd_move_*) */
    constexpr int SMALL_MOVES = 64;
    __shared__ FwdMove sh_moves[SMALL_MOVES];
    __shared__ int sh_nmove;

    if (TH && (s.ctl->done || s.ctl->error)) {
        /* launched beside others that ended the run (no CTA writes the control block before all have read it) */
        if (blockIdx.x == 0 && threadIdx.x == 0) {
            s.ctl->th_commit = 0;
        }
        return;
    }
    const unsigned rank = cluster.block_rank();
    const unsigned G = cluster.num_blocks();
    const int tid = threadIdx.x;
    const int pt = (int)blockDim.x - 32; /* particle threads; the last warp is the control warp */
    const bool ctrl = tid >= pt;
    const int64_t N = s.N;
    const int64_t tile = (int64_t)pt;
    const int64_t base = (int64_t)rank * tile;
    const int64_t p = base + (int64_t)tid; /* this thread's particle */
    const Ctl* gc = s.ctl;
    const int flags = gc->flags;
    const bool act = (flags & (RF_ACT | RF_TRUNCATE | RF_EVENT)) != 0;
    const bool resid = (flags & RF_RESID) != 0;
    const double vdt = gc->vdt;
    double uf = gc->u_frame;
    int cur = gc->cur;
    const int64_t nring = (resid && gc->niter_tol > 0) ? gc->niter_tol : 0;
    if (tid < 2) {
        sh_stop[tid] = 0;
        sl_ds[tid] = 0ull;
        sl_da[tid] = 0ull;
        sl_nan[tid] = 0;
        sl_walk[tid] = 0;
    }
    if (tid == 0) {
        sh_nmove = 0;
    }
    if (rank == 0) {
        if (tid == 0) {
            sc = *gc;
        }
        for (int64_t i = tid; i < nring; i += blockDim.x) {
            sring[i] = s.ring[i];
        }
    }

    /* ring neighbours of the tile's first and last particle: the CTAs that hold them, and their slots for this
     * tile's outermost positions */
    const int64_t plast = (base + tile < N ? base + tile : N) - 1;
    const int64_t pl = base == 0 ? N - 1 : base - 1;
    const int64_t pr = plast + 1 == N ? 0 : plast + 1;
    double* to_left = cluster.map_shared_rank(&sh_edge[0][0], (unsigned)(pl / tile)) + 1;
    double* to_right = cluster.map_shared_rank(&sh_edge[0][0], (unsigned)(pr / tile));
    Ctl* sc0 = cluster.map_shared_rank(&sc, 0);
    const int warps = pt >> 5; /* of particle threads */
    double2* part0 = cluster.map_shared_rank(&spart[0][0], 0) + rank * warps + (tid >> 5);
    unsigned long long* sl_ds0 = cluster.map_shared_rank(&sl_ds[0], 0);
    unsigned long long* sl_da0 = cluster.map_shared_rank(&sl_da[0], 0);
    int* sl_nan0 = cluster.map_shared_rank(&sl_nan[0], 0);
    int* sl_walk0 = cluster.map_shared_rank(&sl_walk[0], 0);

    double u, v, a;
    double4_32a w;
    /* the state before the latest step, kept for the rollback of a step taken after the stop; window starts */
    double pu, pv, pa;
    int64_t start, pstart;
    if (!ctrl && p < N) {
        u = s.u[cur][p];
        v = s.v[cur][p];
        a = s.a[cur][p];
        w = load_well(s, p);
        start = s.start[p];
    }
    else {
        u = v = a = 0.0;
        w = make_double4_32a(0.0, 0.0, 0.0, 0.0);
        start = 0;
    }
    pu = u;
    pv = v;
    pa = a;
    pstart = start;
    /* thermal forces: the values in use, and what step t + 1 draws, loaded a step ahead (planned draws) */
    double fth = 0.0, fnew = 0.0;
    uint32_t draw = 0u, draw_next = 0u;
    const uint32_t* th_mask = TH ? s.th_mask + (p < N ? p >> 5 : 0) : nullptr;
    if (TH && !ctrl) {
        draw = p < N ? th_mask[0] : 0u;
        draw_next = p < N ? th_mask[s.th_words] : 0u;
        fth = p < N ? s.f_th[p] : 0.0;
        fnew = p < N && (draw >> (p & 31) & 1u) ? s.th_val[p] : 0.0;
    }
    /* pcg32 stride of pt steps, x -> mv_a x + mv_c, for the shared draws of window moves */
    const uint64_t mv_c = pcg_advance(0ULL, (uint64_t)pt);
    const uint64_t mv_a = pcg_advance(1ULL, (uint64_t)pt) - mv_c;
    int64_t steps_taken = 0;
    uint64_t now = 0;
    double uf_prev = uf;
    double uf_t = (flags & RF_FLOW) ? FQ_ADD(uf, vdt) : uf;
    /* every CTA's shared memory is set up before another one writes to it */
    cluster.sync();
    for (int64_t t = 0;; ++t) {
        const int q = (int)(t & 1);
        double un = 0.0, sfp = 0.0, ff = 0.0, fd = 0.0;
        bool out = false;
        if (!ctrl) {
            un = FQ_ADD(FQ_ADD(u, FQ_MUL(s.dt, v)), FQ_MUL(s.hdt2, a));
            sh_un[q][tid] = un;
            if (inter_ring(INTER)) {
                if (p == base) {
                    to_left[2 * q] = un;
                }
                if (p == plast) {
                    to_right[2 * q] = un;
                }
            }
        }
        /* A_t: every tile's new positions; the decision after step t - 2 (slot t % 2) */
        cluster.barrier_arrive();
        /* beside the barrier: what does not need the neighbours */
        if (!ctrl) {
            sfp = frame_pot<POT>(s, w, POT == POT_CUSPY ? FQ_SUB(w.z, un) : 0.0, un, uf_t, ff);
            fd = FQ_MUL(s.me, FQ_ADD(v, FQ_MUL(s.dt, a)));
            out = p < N && !in_well(w.x, w.y, un);
        }
        cluster.barrier_wait();
        if (t >= 2 && ((volatile int*)sh_stop)[q]) {
            /* stopped after step t - 2: restore the state before step t - 1 */
            steps_taken = t - 1;
            u = pu;
            v = pv;
            a = pa;
            if (!ctrl && p < N) {
                bool placed = false;
                if (start != pstart) {
                    /* the window moved in the step taken after the stop: put it back */
                    double acc;
                    seq_fill(s, p, pstart, s.W, s.data + p * s.W, &acc);
                    s.start[p] = pstart;
                    s.acc_end[p] = acc;
                    placed = true;
                }
                /* the well of the restored position (index, cached well) in the restored window */
                double4_32a ww = load_well(s, p);
                if (placed) {
                    /* not a well of the restored window: the search starts from its index alone */
                    ww.x = ww.y = __longlong_as_double(0x7ff8000000000000LL);
                }
                if ((placed || !in_well(ww.x, ww.y, u)) && !non_finite(u) && !window_search(s, p, u, ww)) {
                    dev_align(s, p, u);
                }
            }
            break;
        }
        const double uf_last = uf_prev; /* u_frame of step t - 1, for its stop tests */
        uf_prev = uf_t;
        const double uf_now = uf_t;
        if (flags & RF_FLOW) {
            uf_t = FQ_ADD(uf_t, vdt);
        }
        if (ctrl) {
            if (rank == 0 && t >= 1) {
                /* the decision after step t - 1.  This warp's work of a step has to fit into a step: the residual's
                 * two square roots beside each other, the time now and then */
                const int lane = tid - pt, r = (int)((t - 1) & 1);
                double res = 0.0;
                if (resid) {
                    /* the canonical tree over the warps' subtrees, zero padded to 16 CTAs */
                    const int per = warps <= 2 ? 1 : warps / 2, n = (int)G * warps;
                    double x[4], y[4];
#pragma unroll
                    for (int i = 0; i < 4; ++i) {
                        const int k = per * lane + i;
                        const bool in = i < per && k < n;
                        x[i] = in ? spart[r][k].x : 0.0;
                        y[i] = in ? spart[r][k].y : 0.0;
                    }
                    const double2 tot = warp_tree2(sum_consecutive(x, per), sum_consecutive(y, per));
                    const double ty = __shfl_sync(0xffffffffu, tot.y, 0);
                    const double root = FQ_SQRT(lane == 1 ? ty : tot.x);
                    const double r_fres = __shfl_sync(0xffffffffu, root, 0), r_fext = __shfl_sync(0xffffffffu, root, 1);
                    res = r_fext != 0.0 ? FQ_DIV(r_fres, r_fext) : r_fres;
                }
                if ((t & 63) == 1) {
                    now = globaltimer();
                }
                int stop = 0;
                if (lane == 0) {
                    if (sl_ds[r]) {
                        sc.s_sum = (long long)((unsigned long long)sc.s_sum + sl_ds[r]);
                        sl_ds[r] = 0ull;
                    }
                    if (sl_da[r]) {
                        sc.a_count = (long long)((unsigned long long)sc.a_count + sl_da[r]);
                        sl_da[r] = 0ull;
                    }
                    if (sl_nan[r]) {
                        sc.nan_flag = 1;
                    }
                    if (sl_walk[r]) {
                        sc.walk_flag = 1;
                    }
                    finalize_ctl(&sc, sring, uf_last, 0.0, res, now);
                    stop = (sc.done || sc.error || now - sc.launch_t0 >= sc.budget_ns || (TH && t >= s.th_K)) ? 1 : 0;
                }
                stop = __shfl_sync(0xffffffffu, stop, 0);
                if ((unsigned)lane < G) {
                    *(volatile int*)(cluster.map_shared_rank(&sh_stop[0], (unsigned)lane) + r) = stop;
                }
            }
            continue;
        }
        /* the particle threads take step t */
        uf = uf_now;
        pu = u;
        pv = v;
        pa = a;
        pstart = start;
        /* plastic activity of a particle whose well index went from gold to gnew */
        auto count_move = [&](int64_t p, int64_t gold, int64_t gnew) {
            if (act && gnew != gold) {
                int64_t ref = s.i_n[p];
                long long ds = absll(gnew - ref) - absll(gold - ref);
                long long da = (long long)(gnew != ref) - (long long)(gold != ref);
                atomicAdd(sl_ds0 + q, (unsigned long long)ds);
                atomicAdd(sl_da0 + q, (unsigned long long)da);
            }
        };
        /* wells: a search inside the chunk window, or a window move */
        int64_t gold = 0;
        bool mv = false;
        if (out) {
            if (is_nan_bits(un)) {
                atomicOr(sl_nan0 + q, 1);
            }
            if (!non_finite(un)) {
                gold = s.gidx[p];
                if (window_search(s, p, un, w)) {
                    count_move(p, gold, s.gidx[p]);
                    sfp = frame_pot<POT>(s, w, FQ_SUB(w.z, un), un, uf, ff);
                }
                else {
                    mv = true;
                }
            }
        }
        if (particle_bar_or(pt, mv ? 1 : 0)) {
            /* moves planned here are drawn by all particle threads of the CTA, then summed by their
             * owners; the others (more than SMALL_MOVES, or not a forward move) go through dev_align */
            int slot = -1;
            if (mv) {
                int k = atomicAdd(&sh_nmove, 1);
                if (k < SMALL_MOVES) {
                    FwdMove m;
                    const bool ready = next_window_ready(s, p);
                    if (fwd_move_plan(s, p, un, m)) {
                        m.next = ready ? 1 : 0;
                        sh_moves[k] = m;
                        slot = k;
                    }
                    else {
                        sh_moves[k].p = -1;
                    }
                }
            }
            if (tid == 0) {
                /* the moved windows' next-window buffers are out of date after this run */
                atomicOr(&sc0->nx_stale, 1);
            }
            particle_bar(pt);
            const int nm = sh_nmove < SMALL_MOVES ? sh_nmove : SMALL_MOVES;
            for (int k = 0; k < nm; ++k) {
                if (sh_moves[k].p >= 0) {
                    if (sh_moves[k].next) {
                        fwd_move_copy(s, sh_moves[k], tid, pt);
                    }
                    else {
                        fwd_move_draws(s, sh_moves[k], tid, pt, mv_a, mv_c);
                    }
                }
            }
            particle_bar(pt);
            if (tid == 0) {
                sh_nmove = 0; /* (the next step's moves come after its cluster barrier) */
            }
            if (mv) {
                if (slot >= 0) {
                    if (sh_moves[slot].next) {
                        fwd_move_finish(s, sh_moves[slot]);
                    }
                    else {
                        fwd_move_sum(s, sh_moves[slot]);
                    }
                }
                else {
                    dev_align(s, p, un); /* moves the chunk window; a failed search sets walk_flag */
                    if (((volatile Ctl*)s.ctl)->walk_flag) {
                        atomicOr(sl_walk0 + q, 1);
                    }
                }
                w = load_well(s, p);
                start = s.start[p];
                sfp = frame_pot<POT>(s, w, FQ_SUB(w.z, un), un, uf, ff);
                count_move(p, gold, s.gidx[p]);
            }
        }
        double f = 0.0;
        if (p < N) {
            double sum;
            if (inter_ring(INTER)) {
                const double uL = tid > 0 ? sh_un[q][tid - 1] : sh_edge[q][0];
                const double uR = p < plast ? sh_un[q][tid + 1] : sh_edge[q][1];
                sum = add_ring_force<INTER, 0u>(s, sfp, uL, un, uR);
            }
            else {
                sum = add_zero(sfp);
            }
            if (TH) {
                /* step t's draw, then the load for step t + 1 (row th_K of the plan is empty) */
                if (draw >> (p & 31) & 1u) {
                    fth = fnew;
                }
                if (draw_next >> (p & 31) & 1u) {
                    fnew = s.th_val[(t + 1) * N + p];
                }
            }
            /* verlet_velocity, its first damping force formed above */
            f = with_thermal<TH>(FQ_ADD(sum, fd), fth);
            double an = scale(f, s.s_im);
            double vn = FQ_ADD(v, FQ_MUL(s.hdt, FQ_ADD(a, an)));
            f = with_thermal<TH>(FQ_ADD(sum, FQ_MUL(s.me, vn)), fth);
            an = scale(f, s.s_im);
            vn = FQ_ADD(v, FQ_MUL(s.hdt, FQ_ADD(a, an)));
            f = with_thermal<TH>(FQ_ADD(sum, FQ_MUL(s.me, vn)), fth);
            an = scale(f, s.s_im);
            u = un;
            v = vn;
            a = an;
        }
        if (resid) {
            const double f2 = p < N ? mul_nospec(f, f) : 0.0, ff2 = p < N ? mul_nospec(ff, ff) : 0.0;
            const double2 part = warp_tree2(f2, ff2);
            if ((tid & 31) == 0) {
                part0[q * (SMALL_MAX_CTAS * SMALL_THREADS_MAX / 32)] = part;
            }
        }
        if (TH) {
            draw = draw_next;
            draw_next = p < N ? th_mask[(t + 2 < s.th_K ? t + 2 : s.th_K) * s.th_words] : 0u;
        }
    }
    cur = sc0->cur;
    if (!ctrl && p < N) {
        s.u[cur][p] = u;
        s.v[cur][p] = v;
        s.a[cur][p] = a;
    }
    if (rank == 0) {
        for (int64_t i = tid; i < nring; i += blockDim.x) {
            s.ring[i] = sring[i];
        }
        if (tid == 0) {
            if (TH) {
                sc.th_commit = steps_taken;
            }
            *s.ctl = sc;
        }
    }
    /* no CTA may exit while others still read its shared memory */
    cluster.sync();
}

/*
 * One particle per thread, up to 256 of them per CTA: N <= 4096 in a cluster of 16, Smooth systems N <= 2048.
 * Beyond, the resident run kernel on all SMs takes a step in less time (flow, us per step, cluster and run kernel:
 * Cuspy N = 4096 2.4 and 4.7, 8192 (two particles per thread) 5.6 and 4.8, 16384 (four) 11.4 and 4.8; Smooth
 * N = 2048 6.8 and 9.0, 4096 11.2 and 9.4).
 */
SmallGeom small_geometry(int64_t N, int pot, int max_ctas)
{
    SmallGeom g;
    int64_t per = (N + max_ctas - 1) / max_ctas;
    int64_t tile = 32;
    while (tile < per) {
        tile <<= 1;
    }
    g.threads = (int)tile;
    g.ctas = (int)((N + tile - 1) / tile);
    g.ok = N >= 1 && tile <= SMALL_THREADS_MAX && max_ctas <= SMALL_MAX_CTAS && (pot != POT_SMOOTH || N <= 2048);
    return g;
}

template <int POT, int INTER, bool TH = false>
static const void* small_kernel_t()
{
    return (const void*)k_run_small<POT, INTER, TH>;
}

static const void* small_kernel(const DevSys& s)
{
    if (s.f_th) {
        /* RandomNormalForcing systems: Cuspy with Laplace1d, Quartic1d or no interactions */
        switch (s.inter) {
            case INTER_LAPLACE1D: return small_kernel_t<POT_CUSPY, INTER_LAPLACE1D, true>();
            case INTER_QUARTIC1D: return small_kernel_t<POT_CUSPY, INTER_QUARTIC1D, true>();
            default: return small_kernel_t<POT_CUSPY, INTER_NONE, true>();
        }
    }
    /* the Quartic interactions exist with the Cuspy potential only (Line1d.h:428, :562) */
    if (s.inter == INTER_QUARTIC1D) {
        return small_kernel_t<POT_CUSPY, INTER_QUARTIC1D>();
    }
    if (s.inter == INTER_QUARTICGRAD1D) {
        return small_kernel_t<POT_CUSPY, INTER_QUARTICGRAD1D>();
    }
    if (s.inter == INTER_LAPLACE1D) {
        return s.pot == POT_CUSPY ? small_kernel_t<POT_CUSPY, INTER_LAPLACE1D>()
               : s.pot == POT_SEMISMOOTH ? small_kernel_t<POT_SEMISMOOTH, INTER_LAPLACE1D>()
                                         : small_kernel_t<POT_SMOOTH, INTER_LAPLACE1D>();
    }
    return s.pot == POT_CUSPY ? small_kernel_t<POT_CUSPY, INTER_NONE>()
           : s.pot == POT_SEMISMOOTH ? small_kernel_t<POT_SEMISMOOTH, INTER_NONE>()
                                     : small_kernel_t<POT_SMOOTH, INTER_NONE>();
}

static void small_launch_config(const SmallGeom& g, cudaStream_t st, cudaLaunchConfig_t& cfg, cudaLaunchAttribute* attr)
{
    cfg = {};
    cfg.gridDim = dim3((unsigned)g.ctas);
    cfg.blockDim = dim3((unsigned)g.threads + 32u); /* particle threads and the control warp */
    cfg.dynamicSmemBytes = 0;
    cfg.stream = st;
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = (unsigned)g.ctas;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
}

bool small_cluster_fits(const DevSys& s, const SmallGeom& g)
{
    const void* f = small_kernel(s);
    if (cudaFuncSetAttribute(f, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) != cudaSuccess) {
        cudaGetLastError();
        return false;
    }
    cudaLaunchConfig_t cfg;
    cudaLaunchAttribute attr[1];
    small_launch_config(g, nullptr, cfg, attr);
    int n = 0;
    if (cudaOccupancyMaxActiveClusters(&n, f, &cfg) != cudaSuccess) {
        cudaGetLastError();
        return false;
    }
    return n >= 1;
}

cudaError_t launch_small_run(const DevSys& s, const SmallGeom& g, cudaStream_t st)
{
    const void* f = small_kernel(s);
    if (g.ctas > 8) {
        /* clusters above the portable size of 8 must be allowed per kernel */
        cudaError_t e = cudaFuncSetAttribute(f, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
        if (e != cudaSuccess) {
            return e;
        }
    }
    cudaLaunchConfig_t cfg;
    cudaLaunchAttribute attr[1];
    small_launch_config(g, st, cfg, attr);
    DevSys arg = s;
    arg.in_graph = 0; /* not inside the run graph: no conditional handles to set */
    void* args[] = {(void*)&arg};
    return cudaLaunchKernelExC(&cfg, f, args);
}

} // namespace fqsb
