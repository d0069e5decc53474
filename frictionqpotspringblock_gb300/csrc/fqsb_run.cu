/*
 * Resident run kernel of Line1d, Particles and Laplace2d systems (sm_103a, FP64): many time steps
 * (System::timeStep, include/FrictionQPotSpringBlock/detail.h:1539-1570) in one cooperative launch.
 *
 * Why.  With one kernel per time step inside the run graph's WHILE loop every step pays the loop's
 * iteration, the launch, each CTA's read of the run state and its ticket: 13 us at N = 1024, 18 us at
 * N = 2^22.  Here the CTAs (one per SM) stay, and a grid barrier (2 us with the start of the next step)
 * separates the steps.  Measured per step, one kernel per step and this kernel: N = 65536 17.3 and 6.6 us,
 * 2^20 50 and 37 us, 2^22 177 and 136 us (minimise 221 and 161 us).  It is then bound by the fp64 and the
 * ALU pipe together (61% and 64% of their practical rates) and by how well the warps' phases interleave.
 *
 * Work split.  The ring is cut into strips of 32 to 256 consecutive particles; each warp takes whole
 * strips and needs no barrier with the others inside a step (in the one-kernel-per-step form the warps
 * spend a third of their time at the CTA's barrier between position update and forces, and around the
 * ticket).  A warp first updates its strip's positions and those of the two neighbours outside, into
 * shared memory, and tests the wells; the particles of the strip that may have left theirs are then
 * looked at together, a lane each; and it walks over the strip again, one particle per lane, for forces
 * and velocities.  One particle per lane and rolled loops keep the code within the instruction cache.
 * Strips are as long as they can be (the two outside positions cost an extra pass) while every warp
 * still gets one (run_geometry).
 *
 * Stop tests.  The last CTA of the grid holds no strips: it sums step t - 1's residual and runs its stop
 * tests (finalize_ctl) while the others take step t.  When step t - 1 turns out to be the last, step t
 * is dropped: its output went to the other half of the double-buffered state, its counters to its own
 * slot, and the wells it changed are looked up again (restore_wells).
 *
 * Residual.  The sums follow the fixed pairwise tree over the flat index: in a strip, over the strips of
 * a node, over the nodes (control CTA), all aligned powers of two.
 *
 * Chunk windows.  A step in which a particle leaves its window ends the launch unfinished; the graph's
 * IF branch moves the windows, repeats the marked strips and finishes the step (fqsb_step.cu), and the
 * loop launches this kernel again.
 *
 * The kernel's waits are on CTAs that a cooperative launch keeps resident, and end after Ctl::wait_ns (5 s).  The host
 * then sets RunSync and the marks of pending strips back (run(), fqsb_capi.cu).
 */
#include "fqsb_stepcore.cuh"

namespace fqsb {

/* Warps per CTA: 28 (72 registers a thread); Smooth's double-double sine needs 128 registers. */
template <int POT>
struct RunWarps {
    static constexpr int value = POT == POT_SMOOTH ? 16 : 28;
};

constexpr int RUN_RING = 1024; /* StopList windows up to this length are kept in shared memory */

/* Why a launch ends after step t: the run stopped after step t - 1 (step t is dropped); particles of step
 * t left their windows; t was the last step asked for; the barrier ran out. */
enum : int { END_NOT = 0, END_STOPPED = 1, END_PENDING = 2, END_LAST = 3, END_BARRIER = 4 };

__device__ __forceinline__ unsigned long long load_acquire(const unsigned long long* p)
{
    unsigned long long v;
    asm volatile("ld.acquire.gpu.u64 %0, [%1];" : "=l"(v) : "l"(p) : "memory");
    return v;
}

/* Waits until a counter of s.sync has reached `want`; false when the wait ran out. */
__device__ __forceinline__ bool wait_for(const DevSys& s, const unsigned long long* counter, unsigned long long want)
{
    RunSync* y = s.sync;
    uint64_t t0 = 0;
    for (unsigned k = 1; load_acquire(counter) < want; ++k) {
        if ((k & 255u) == 0u) {
            if (((volatile RunSync*)y)->failed) {
                return false;
            }
            const uint64_t now = globaltimer();
            t0 = t0 == 0 ? now : t0;
            if (now - t0 > s.ctl->wait_ns) {
                atomicOr(&y->failed, 1);
                return false;
            }
        }
    }
    return true;
}

/* Grid barrier up to `want` arrivals, for thread 0 of a CTA (the others wait at a CTA barrier on both sides);
 * false when it ran out. */
__device__ __forceinline__ bool grid_barrier(const DevSys& s, unsigned long long want)
{
    __threadfence();
    atomicAdd(&s.sync->arrived, 1ull);
    return wait_for(s, &s.sync->arrived, want);
}

/* The barrier after step t; returns how the launch goes on. */
__device__ __forceinline__ int barrier_after(const DevSys& s, unsigned long long base, int64_t t, bool last)
{
    if (!grid_barrier(s, base + (unsigned long long)(t + 1) * gridDim.x)) {
        return END_BARRIER;
    }
    const volatile RunSync* vy = s.sync;
    if (vy->stop[t & 1]) {
        return END_STOPPED;
    }
    if (vy->pending[t & 1]) {
        return END_PENDING;
    }
    return last ? END_LAST : END_NOT;
}

/*
 * Particle p at its new position un, which may have left its well: searches its window, counts the change
 * in the slot of step t (act) and commits the new well; d becomes centre - un (Cuspy).  Returns whether
 * the window must move.
 */
template <int POT>
static __device__ __noinline__ bool leave_well(const DevSys& s, int64_t p, double un, bool act, int64_t t, double& d,
                                               int64_t* moved)
{
    const double2 wy = __ldcg(s.wy + p);
    const int64_t gold = s.gidx[p];
    if (is_nan_bits(un)) {
        s.sync->nan[t & 1] = 1;
    }
    if (in_well(wy.x, wy.y, un) || non_finite(un)) {
        return false;
    }
    double4_32a w = make_double4_32a(wy.x, wy.y, 0.0, 0.0);
    if (!window_search(s, p, un, w)) {
        return true;
    }
    *moved = t + 1;
    if (POT == POT_CUSPY) {
        d = FQ_SUB(w.z, un);
    }
    const int64_t gnew = s.gidx[p];
    if (act && gnew != gold) {
        const int64_t ref = s.i_n[p];
        const long long ds = absll(gnew - ref) - absll(gold - ref);
        const long long da = (long long)(gnew != ref) - (long long)(gold != ref);
        atomicAdd((unsigned long long*)&s.sync->ds[t & 1], (unsigned long long)ds);
        atomicAdd((unsigned long long*)&s.sync->da[t & 1], (unsigned long long)da);
    }
    return false;
}

/* The well of particle p at position u looked up again in its window, after a dropped step (the window has
 * not moved since u was reached, and contains it). */
static __device__ __noinline__ void restore_well(const DevSys& s, int64_t p, double u)
{
    const double2 wy = __ldcg(s.wy + p);
    if (in_well(wy.x, wy.y, u) || non_finite(u)) {
        return;
    }
    const double* y = s.data + p * s.W;
    int64_t li = s.cidx[p];
    while (li + 1 < s.W - 1 && y[li + 1] <= u) {
        ++li;
    }
    while (li > 0 && y[li] > u) {
        --li;
    }
    s.cidx[p] = (int32_t)li;
    s.gidx[p] = s.start[p] + li;
    store_well(s, p, make_wc(s, y[li], y[li + 1]));
}

/* What the steps of one launch share within a warp */
struct Strip {
    double *un, *v, *d; /* shared memory: positions (un[0], un[1 + S] outside), velocities, Cuspy centre - un */
    uint8_t* list;      /* particles of the strip that may have left their wells */
    int groups;         /* S / 32 */
};

/*
 * One time step of the strip of particles p0 .. p0 + n - 1 (n <= S) by one warp; returns the strip's sums
 * of f^2 and f_frame^2 (or of f_frame) in lane 0.
 *
 * A grid (Laplace2d) is taken in the order of its flat index, so a strip has most of its particles' left and
 * right neighbours; those above and below are in other strips.  Their positions are read, not recomputed: every step
 * leaves its particles' next positions in s.ahead (for the first step of a launch a pass of its own does).
 * That is 8 B more written per particle and step, but no position is updated twice (a tile of 16 x 32 updates 96 of
 * its neighbours' besides its own 512), and no launches: flow, us per step, by tiles in the run graph and here:
 * 301 x 257 21.1 and 6.7, 1024 x 1024 51.6 and 40.0, 2048 x 2048 173 and 163, 4096 x 3000 480 and 446.
 */
template <int POT, int INTER, int MODE, bool TH>
__device__ __forceinline__ double2 strip_step(const DevSys& s, const Strip& st, int64_t p0, int n, int cur, double uf,
                                              int flags, int64_t step, int64_t t, int64_t th_used, bool& pending,
                                              int64_t* moved)
{
    /* one more addition on the integer pipes where they do not also square the residual: at N = 2^22 142 us per
     * step instead of 144 us, but 173 us instead of 169 us with the squares */
    constexpr unsigned SOFT = MODE == KMODE_PLAIN ? STEP_SOFT | (1u << 11) : STEP_SOFT;
    const int lane = threadIdx.x & 31;
    const bool general = MODE == KMODE_GENERAL;
    const bool act = general && (flags & (RF_ACT | RF_TRUNCATE | RF_EVENT)) != 0;
    const bool resid = MODE == KMODE_RESID || (general && (flags & RF_RESID) != 0);
    const bool ffsum = general && (flags & RF_FFSUM) != 0;
    const int64_t N = s.N;
    const double *u0 = s.u[cur], *v0 = s.v[cur], *a0 = s.a[cur];
    double *u1 = s.u[cur ^ 1], *v1 = s.v[cur ^ 1], *a1 = s.a[cur ^ 1];
    const int G = st.groups;

    /* positions: pass i < G the strip's particles, pass G its two neighbours outside (lanes 0 and 1); the
     * loads of a pass are issued a pass ahead */
    constexpr bool GRID = inter_grid(INTER);
    const int passes = inter_ring(INTER) || GRID ? G + 1 : G;
    /* grid: positions of this step by the step before, and where this step leaves those of the next */
    const double* ahead = GRID ? s.ahead + (t & 1 ? 0 : N) : nullptr;
    double* ahead_next = GRID ? s.ahead + (t & 1 ? N : 0) : nullptr;
    auto index = [&](int i) -> int64_t {
        if (i < G) {
            return p0 + i * 32 + lane;
        }
        return lane == 0 ? (p0 == 0 ? N - 1 : p0 - 1) : (p0 + n == N ? 0 : p0 + n);
    };
    double ul, vl, al;
    double2 wl = __ldcg((POT == POT_CUSPY ? s.wk : s.wy) + p0 + lane);
    {
        const int64_t p = index(0);
        if (GRID) {
            ul = lane < n ? __ldcg(ahead + p) : 0.0;
            vl = __ldcg(v0 + p);
            al = 0.0;
        }
        else {
            ul = __ldcg(u0 + p);
            vl = __ldcg(v0 + p);
            al = __ldcg(a0 + p);
        }
    }
    int leaving = 0;
#pragma unroll 1
    for (int i = 0; i < passes; ++i) {
        const double u = ul, v = vl, a = al;
        const double2 w = wl;
        const int64_t p = index(i);
        if (i + 1 < passes) {
            const int64_t pn = index(i + 1);
            if (GRID) {
                ul = (i + 1 < G ? (i + 1) * 32 + lane < n : lane < 2) ? __ldcg(ahead + pn) : 0.0;
            }
            else {
                ul = __ldcg(u0 + pn);
                al = __ldcg(a0 + pn);
            }
            vl = __ldcg(v0 + pn);
            if (i + 1 < G) {
                wl = __ldcg((POT == POT_CUSPY ? s.wk : s.wy) + pn);
            }
        }
        const double un =
            GRID ? u : S_ADD(3, S_ADD(2, u, S_MULC(0, s.f_dt, s.dt, v)), S_MULC(1, s.f_hdt2, s.hdt2, a));
        if (i < G) {
            const int k = i * 32 + lane;
            st.v[k] = v;
            if (k < n) {
                st.un[1 + k] = un;
                u1[p] = un;
            }
            /* Cuspy: the force's centre - un also tells that the particle stays in its well */
            bool out;
            if (POT == POT_CUSPY) {
                const double d = S_SUB(5, w.x, un);
                st.d[k] = d;
                out = !surely_in_well(w, d);
            }
            else {
                out = !in_well(w.x, w.y, un);
            }
            const unsigned m = __ballot_sync(0xffffffffu, out && k < n);
            if (out && k < n) {
                st.list[leaving + __popc(m & ((1u << lane) - 1u))] = (uint8_t)k;
            }
            leaving += __popc(m);
        }
        else if (lane < 2) {
            st.un[lane == 0 ? 0 : 1 + n] = un;
        }
    }
    __syncwarp();

    /* the particles that may have left their wells, a lane each: one wait for all of the strip */
    bool pend = false;
    for (int j = lane; j < leaving; j += 32) {
        const int k = st.list[j];
        if (leave_well<POT>(s, p0 + k, st.un[1 + k], act, t, st.d[k], moved)) {
            pend = true;
            s.regen_list[atomicAdd(&s.ctl->n_regen, 1)] = (int32_t)(p0 + k);
        }
    }
    __syncwarp();

    /* wells, forces and velocities */
    al = __ldcg(a0 + p0 + lane);
    /* grid: column of the lane's particle, the positions above and below it (loaded a pass ahead) */
    int64_t col = 0, col_step = 0;
    double upper = 0.0, lower = 0.0;
    auto above = [&](int64_t p) { return __ldcg(ahead + (p >= s.cols ? p - s.cols : p + (N - s.cols))); };
    auto below = [&](int64_t p) { return __ldcg(ahead + (p < N - s.cols ? p + s.cols : p - (N - s.cols))); };
    if (GRID) {
        col = (p0 + lane) % s.cols;
        col_step = 32 % s.cols;
        if (lane < n) {
            upper = above(p0 + lane);
            lower = below(p0 + lane);
        }
    }
#pragma unroll 1
    for (int i = 0; i < G; ++i) {
        const int k = i * 32 + lane;
        const int64_t p = p0 + k;
        const double a = al;
        const double uU = upper, uD = lower;
        if (i + 1 < G) {
            al = __ldcg(a0 + p + 32);
            if (GRID && k + 32 < n) {
                upper = above(p + 32);
                lower = below(p + 32);
            }
        }
        const double up = st.un[1 + k], d = POT == POT_CUSPY ? st.d[k] : 0.0;
        double4_32a w = make_double4_32a(0.0, 0.0, 0.0, 0.0);
        if (POT != POT_CUSPY) {
            const double2 wy = __ldcg(s.wy + p), wk = __ldcg(s.wk + p);
            w = make_double4_32a(wy.x, wy.y, wk.x, wk.y);
        }
        double ff;
        double sfi = frame_pot<POT, SOFT>(s, w, d, up, uf, ff);
        if (inter_ring(INTER)) {
            sfi = add_ring_force<INTER, SOFT>(s, sfi, st.un[k], up, st.un[2 + k]);
        }
        else if (GRID) {
            double uL = st.un[k], uR = st.un[2 + k];
            if (k < n && col == 0) {
                uL = __ldcg(ahead + p + s.cols - 1);
            }
            if (k < n && col == s.cols - 1) {
                uR = __ldcg(ahead + p - (s.cols - 1));
            }
            col += col_step;
            col -= col >= s.cols ? s.cols : 0;
            sfi = grid_force<SOFT>(s, sfi, uU, uD, uL, up, uR);
        }
        else {
            sfi = add_zero(sfi);
        }
        double vn, an, f;
        double fth = 0.0;
        if (TH && k < n) {
            /* the planned draw of step t, or the force of the step before */
            const uint32_t draw = __ldcg(s.th_mask + (th_used + t) * s.th_words + (p >> 5));
            fth = draw >> (p & 31) & 1u ? __ldcg(s.th_val + (th_used + t) * N + p)
                                        : __ldcg((t == 0 ? s.f_th : s.th_w[(t - 1) & 1]) + p);
            s.th_w[t & 1][p] = fth;
        }
        verlet_velocity<SOFT, TH>(s, sfi, st.v[k], a, vn, an, f, fth);
        if (k < n) {
            v1[p] = vn;
            a1[p] = an;
            if (GRID) {
                ahead_next[p] = S_ADD(3, S_ADD(2, up, S_MULC(0, s.f_dt, s.dt, vn)), S_MULC(1, s.f_hdt2, s.hdt2, an));
            }
        }
        if (resid) {
            st.v[k] = k < n ? fq_smul(f, f) : 0.0;
            st.d[k] = k < n ? fq_smul(ff, ff) : 0.0;
        }
        else if (ffsum) {
            st.v[k] = k < n ? ff : 0.0;
            st.d[k] = 0.0;
        }
        if (general && (flags & RF_RECORD) && k < n) {
            const size_t o = (size_t)step * (size_t)N + (size_t)p;
            s.ctl->rec_u[o] = up;
            s.ctl->rec_v[o] = vn;
            s.ctl->rec_a[o] = an;
            s.ctl->rec_w[o] = load_well(s, p);
        }
    }
    pending = __any_sync(0xffffffffu, pend);
    double2 sum = make_double2(0.0, 0.0);
    if (resid || ffsum) {
        __syncwarp();
        sum = warp_tree2(sum_consecutive(st.v + G * lane, G), sum_consecutive(st.d + G * lane, G));
    }
    __syncwarp();
    return sum;
}

/* Steps that a launch takes at most: those the run has left, and with thermal forcing those left of the plan */
__device__ __forceinline__ int64_t steps_of_launch(const DevSys& s)
{
    const int64_t left = s.ctl->max_steps - s.ctl->step;
    return s.f_th && s.th_K - s.ctl->th_used < left ? s.th_K - s.ctl->th_used : left;
}

/* The CTA without strips: sums and stop tests of each step, one step behind the others */
static __device__ __noinline__ void run_control(const DevSys& s, const RunGeom& g)
{
    __shared__ Ctl sc;
    __shared__ double ring[RUN_RING];
    __shared__ double red[64];
    __shared__ int how_sh;
    constexpr int T = 512; /* threads of the sum over the nodes */
    const int tid = threadIdx.x;
    RunSync* y = s.sync;
    const int flags = s.ctl->flags;
    const bool tree = (flags & (RF_RESID | RF_FFSUM)) != 0;
    unsigned long long base = y->base;
    const int64_t left = steps_of_launch(s), step0 = s.ctl->step;
    const double vdt = s.ctl->vdt;
    const int64_t nring = (flags & RF_RESID) ? s.ctl->niter_tol : 0;
    const bool shared_ring = nring <= RUN_RING;
    double uf = s.ctl->u_frame;
    __syncthreads();
    if (tid == 0) {
        sc = *s.ctl;
        sc.n_regen = 0;
        sc.n_pending_cta = 0;
    }
    for (int64_t i = tid; shared_ring && i < nring; i += blockDim.x) {
        ring[i] = s.ring[i];
    }
    if (inter_grid(s.inter)) {
        base += gridDim.x; /* the barrier after the first positions (when it runs out, so does the first step's) */
        if (tid == 0) {
            grid_barrier(s, base);
        }
    }
    __syncthreads();

    /* step k finished everywhere: its counters, its residual, its stop tests */
    auto finish = [&](int64_t k, double ufk) {
        const int q = (int)(k & 1);
        double2 tot = make_double2(0.0, 0.0);
        if (tree) {
            const double2* node = s.nodes + (size_t)q * RUN_NODES_MAX;
            const int64_t per = next_pow2(g.nnodes) > T ? next_pow2(g.nnodes) / T : 1;
            double2 x = make_double2(0.0, 0.0);
            if (tid < T) {
                x = serial_tree2([&](int64_t i) { return i < g.nnodes ? __ldcg(node + i) : make_double2(0.0, 0.0); },
                                 (int64_t)tid * per, per);
                x = warp_tree2(x.x, x.y);
            }
            if (tid < T && (tid & 31) == 0) {
                red[tid >> 5] = x.x;
                red[32 + (tid >> 5)] = x.y;
            }
            __syncthreads();
            if (tid < 32) {
                tot = warp_tree2(tid < T / 32 ? red[tid] : 0.0, tid < T / 32 ? red[32 + tid] : 0.0);
            }
        }
        if (tid == 0) {
            volatile RunSync* vy = y;
            sc.s_sum = (long long)((unsigned long long)sc.s_sum + (unsigned long long)vy->ds[q]);
            sc.a_count = (long long)((unsigned long long)sc.a_count + (unsigned long long)vy->da[q]);
            vy->ds[q] = 0;
            vy->da[q] = 0;
            if (vy->nan[q]) {
                sc.nan_flag = 1;
            }
            finalize_ctl(&sc, shared_ring ? ring : s.ring, ufk, tot.x, residual_of(flags, tot.x, tot.y), globaltimer());
        }
    };

    int64_t t = 0;
    for (;; ++t) {
        double uf_t = uf;
        if (flags & RF_FLOW) {
            uf_t = FQ_ADD(uf, vdt);
        }
        if (flags & RF_SCHEDULE) {
            uf_t = sc.sched[step0 + t];
        }
        if (t > 0) {
            finish(t - 1, uf);
        }
        if (tid == 0) {
            const bool stop =
                t > 0 && (sc.done || sc.error || (globaltimer() - sc.launch_t0) >= sc.budget_ns);
            ((volatile RunSync*)y)->stop[t & 1] = stop ? 1 : 0;
            how_sh = barrier_after(s, base, t, t + 1 == left);
        }
        __syncthreads();
        uf = uf_t;
        if (how_sh != END_NOT) {
            break;
        }
    }
    const int how = how_sh;
    __syncthreads();
    if (how == END_LAST) {
        finish(t, uf);
    }
    __syncthreads();
    for (int64_t i = tid; shared_ring && i < nring; i += blockDim.x) {
        s.ring[i] = ring[i];
    }
    if (tid == 0) {
        volatile RunSync* vy = y;
        const int q = (int)(t & 1);
        /* the flags below are cleared for the next launch: every CTA has to have read them after its last barrier */
        if (how == END_BARRIER || vy->failed || !wait_for(s, &y->left, gridDim.x - 1u)) {
            sc.error = DERR_BARRIER;
        }
        vy->left = 0;
        if (how == END_PENDING) {
            /* step t is finished by the repeat of its pending strips; what its other strips counted stays */
            sc.s_sum = (long long)((unsigned long long)sc.s_sum + (unsigned long long)vy->ds[q]);
            sc.a_count = (long long)((unsigned long long)sc.a_count + (unsigned long long)vy->da[q]);
            if (vy->nan[q]) {
                sc.nan_flag = 1;
            }
            sc.n_regen = ((volatile Ctl*)s.ctl)->n_regen;
            sc.n_pending_cta = vy->pending[q];
        }
        for (int k = 0; k < 2; ++k) {
            vy->stop[k] = 0;
            vy->pending[k] = 0;
            vy->nan[k] = 0;
            vy->ds[k] = 0;
            vy->da[k] = 0;
        }
        vy->base = base + (unsigned long long)(t + 1) * gridDim.x;
        sc.th_commit = how == END_BARRIER || how == END_STOPPED ? t : t + 1;
        sc.th_from = sc.th_used;
        sc.th_used += sc.th_commit;
        if (sc.th_used >= s.th_K) {
            sc.th_used = 0;
        }
        *s.ctl = sc;
        const bool more = !sc.done && !sc.error && (sc.launch_steps == 0 || globaltimer() - sc.launch_t0 < sc.budget_ns);
        __threadfence();
        set_branch(s, how == END_PENDING ? 1u : 0u);
        set_loop(s, how == END_PENDING || more ? 1u : 0u);
    }
}

template <int POT, int INTER, int MODE, bool TH>
__global__ void __launch_bounds__(32 * RunWarps<POT>::value, 1)
    k_run_line(const __grid_constant__ DevSys s, const __grid_constant__ RunGeom g)
{
    extern __shared__ double dyn[];
    __shared__ int how_sh, next_sh[2]; /* next strip to take, per step parity */
    __shared__ int64_t moved_sh; /* 1 + the last step in which a particle of this CTA changed its well */
    if (s.ctl->done || s.ctl->error) {
        if (blockIdx.x == 0 && threadIdx.x == 0) {
            s.ctl->th_commit = 0;
            set_branch(s, 0u);
            set_loop(s, 0u);
        }
        return;
    }
    if (blockIdx.x == gridDim.x - 1) {
        run_control(s, g);
        return;
    }
    const int wid = threadIdx.x >> 5, lane = threadIdx.x & 31, NW = blockDim.x >> 5;
    const int S = g.S;
    Strip st;
    st.un = dyn + (size_t)wid * (3 * S + 2);
    st.v = st.un + S + 2;
    st.d = st.v + S;
    st.list = reinterpret_cast<uint8_t*>(dyn + (size_t)NW * (3 * S + 2)) + (size_t)wid * S;
    st.groups = S / 32;
    RunSync* y = s.sync;
    unsigned long long base = y->base;
    const int flags = s.ctl->flags;
    const int cur0 = s.ctl->cur;
    const int64_t step0 = s.ctl->step, left = steps_of_launch(s), th_used = TH ? s.ctl->th_used : 0;
    const double vdt = s.ctl->vdt;
    const double* sched = s.ctl->sched;
    const bool tree = MODE == KMODE_RESID || (MODE == KMODE_GENERAL && (flags & (RF_RESID | RF_FFSUM)) != 0);
    double uf = s.ctl->u_frame;
    const int64_t W = gridDim.x - 1;
    const int64_t n0 = g.nnodes * blockIdx.x / W, n1 = g.nnodes * (blockIdx.x + 1) / W;
    /* strips of this CTA: those of its nodes; without sums an even share */
    int64_t s0 = n0 * g.node_strips, s1 = n1 * g.node_strips < g.nstrips ? n1 * g.node_strips : g.nstrips;
    if (MODE == KMODE_PLAIN) {
        s0 = g.nstrips * blockIdx.x / W;
        s1 = g.nstrips * (blockIdx.x + 1) / W;
    }
    if (threadIdx.x == 0) {
        moved_sh = 0;
        next_sh[0] = next_sh[1] = NW;
    }
    if (inter_grid(INTER)) {
        /* the positions of the first step */
        base += gridDim.x;
        const int64_t end = s1 * S < s.N ? s1 * S : s.N;
        for (int64_t p = s0 * S + threadIdx.x; p < end; p += blockDim.x) {
            s.ahead[s.N + p] = u_next<STEP_SOFT>(s, s.u[cur0], s.v[cur0], s.a[cur0], p);
        }
        __syncthreads();
        if (threadIdx.x == 0) {
            grid_barrier(s, base);
        }
    }
    __syncthreads();
    int64_t t = 0;
    for (;; ++t) {
        const int q = (int)(t & 1);
        if (flags & RF_FLOW) {
            uf = FQ_ADD(uf, vdt);
        }
        if (MODE == KMODE_GENERAL && (flags & RF_SCHEDULE)) {
            uf = sched[step0 + t];
        }
        /* the first strips by warp, then whichever warp is ready takes the next */
        for (int64_t k = s0 + wid; k < s1;) {
            const int64_t p0 = k * S;
            bool pending;
            const double2 sum = strip_step<POT, INTER, MODE, TH>(s, st, p0, (int)(s.N - p0 < S ? s.N - p0 : S), cur0 ^ q, uf,
                                                             flags, step0 + t, t, th_used, pending, &moved_sh);
            if (lane == 0) {
                if (tree) {
                    s.partials[k] = sum;
                }
                if (pending) {
                    s.cta_pending[k] = 1;
                    atomicAdd(&y->pending[q], 1);
                }
            }
            int j = 0;
            if (lane == 0) {
                j = atomicAdd(&next_sh[q], 1);
            }
            k = s0 + __shfl_sync(0xffffffffu, j, 0);
        }
        __syncthreads();
        if (tree) {
            /* the strips' sums of each node, pairwise */
            const int64_t per = g.node_strips > 32 ? g.node_strips / 32 : 1;
            for (int64_t m = n0 + wid; m < n1; m += NW) {
                const int64_t k0 = m * g.node_strips;
                const int64_t k1 = k0 + g.node_strips < g.nstrips ? k0 + g.node_strips : g.nstrips;
                const double2 x = serial_tree2(
                    [&](int64_t i) { return i < k1 ? __ldcg(s.partials + i) : make_double2(0.0, 0.0); },
                    k0 + lane * per, per);
                const double2 sum = warp_tree2(x.x, x.y);
                if (lane == 0) {
                    s.nodes[(size_t)q * RUN_NODES_MAX + m] = sum;
                }
            }
            __syncthreads();
        }
        if (threadIdx.x == 0) {
            next_sh[q] = NW;
            how_sh = barrier_after(s, base, t, t + 1 == left);
        }
        __syncthreads();
        if (how_sh != END_NOT) {
            break;
        }
    }
    if (threadIdx.x == 0) {
        __threadfence();
        atomicAdd(&y->left, 1ull);
    }
    if (how_sh == END_STOPPED) {
        /* drop step t: its wells back to those of its input state, its marks cleared */
        const double* u0 = s.u[cur0 ^ (int)(t & 1)];
        for (int64_t k = s0 + wid; k < s1; k += NW) {
            if (lane == 0) {
                s.cta_pending[k] = 0;
            }
            for (int i = lane; moved_sh == t + 1 && i < S && k * S + i < s.N; i += 32) {
                restore_well(s, k * S + i, __ldcg(u0 + k * S + i));
            }
        }
    }
}

/* ------------------------------------------------------------- host side */

template <int POT, int INTER>
static const void* run_kernel_t(int mode)
{
    return mode == KMODE_PLAIN   ? (const void*)k_run_line<POT, INTER, KMODE_PLAIN, false>
           : mode == KMODE_RESID ? (const void*)k_run_line<POT, INTER, KMODE_RESID, false>
                                 : (const void*)k_run_line<POT, INTER, KMODE_GENERAL, false>;
}

const void* run_kernel(const DevSys& s, int mode)
{
    if (s.f_th) {
        /* RandomNormalForcing systems: Cuspy with Laplace1d, Quartic1d or no interactions */
        switch (s.inter) {
            case INTER_LAPLACE1D: return (const void*)k_run_line<POT_CUSPY, INTER_LAPLACE1D, KMODE_GENERAL, true>;
            case INTER_QUARTIC1D: return (const void*)k_run_line<POT_CUSPY, INTER_QUARTIC1D, KMODE_GENERAL, true>;
            default: return (const void*)k_run_line<POT_CUSPY, INTER_NONE, KMODE_GENERAL, true>;
        }
    }
    switch (s.inter) {
        case INTER_LAPLACE2D:
            return s.pot == POT_CUSPY        ? run_kernel_t<POT_CUSPY, INTER_LAPLACE2D>(mode)
                   : s.pot == POT_SEMISMOOTH ? run_kernel_t<POT_SEMISMOOTH, INTER_LAPLACE2D>(mode)
                                             : run_kernel_t<POT_SMOOTH, INTER_LAPLACE2D>(mode);
        case INTER_QUARTIC1D: return run_kernel_t<POT_CUSPY, INTER_QUARTIC1D>(mode);
        case INTER_QUARTICGRAD1D: return run_kernel_t<POT_CUSPY, INTER_QUARTICGRAD1D>(mode);
        case INTER_LAPLACE1D:
            return s.pot == POT_CUSPY        ? run_kernel_t<POT_CUSPY, INTER_LAPLACE1D>(mode)
                   : s.pot == POT_SEMISMOOTH ? run_kernel_t<POT_SEMISMOOTH, INTER_LAPLACE1D>(mode)
                                             : run_kernel_t<POT_SMOOTH, INTER_LAPLACE1D>(mode);
        default:
            return s.pot == POT_CUSPY        ? run_kernel_t<POT_CUSPY, INTER_NONE>(mode)
                   : s.pot == POT_SEMISMOOTH ? run_kernel_t<POT_SEMISMOOTH, INTER_NONE>(mode)
                                             : run_kernel_t<POT_SMOOTH, INTER_NONE>(mode);
    }
}

static size_t run_smem(int S, int64_t warps)
{
    return (sizeof(double) * (3 * (size_t)S + 2) + (size_t)S) * (size_t)warps;
}

constexpr int RUN_STRIP_MAX = 256;

RunGeom run_geometry(const DevSys& s)
{
    RunGeom g = {};
    if (!(inter_ring(s.inter) || s.inter == INTER_NONE || s.inter == INTER_LAPLACE2D)) {
        return g;
    }
    int dev = 0, sms = 0, coop = 0;
    if (cudaGetDevice(&dev) != cudaSuccess ||
        cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess ||
        cudaDeviceGetAttribute(&coop, cudaDevAttrCooperativeLaunch, dev) != cudaSuccess || !coop || sms < 2) {
        cudaGetLastError();
        return g;
    }
    g.threads = 32 * (s.pot == POT_SMOOTH ? RunWarps<POT_SMOOTH>::value : RunWarps<POT_CUSPY>::value);
    /* strips as long as they can be while a CTA's strips still occupy as many warps as possible: 32 to 256 */
    const int64_t workers = sms - 1, warps = g.threads / 32;
    g.S = 32;
    while (g.S < RUN_STRIP_MAX && (s.N + g.S - 1) / g.S > workers * warps) {
        g.S *= 2;
    }
    g.nstrips = (s.N + g.S - 1) / g.S;
    /* nodes: a power of two of strips, at most RUN_NODES_MAX of them; CTAs take whole nodes */
    g.node_strips = 1;
    while ((g.nstrips + g.node_strips - 1) / g.node_strips > RUN_NODES_MAX) {
        g.node_strips *= 2;
    }
    g.nnodes = (g.nstrips + g.node_strips - 1) / g.node_strips;
    g.ctas = (int)(g.nnodes < workers ? g.nnodes : workers) + 1;
    g.smem = run_smem(g.S, warps);
    g.smem_max = run_smem(RUN_STRIP_MAX, warps);
    return g;
}

} // namespace fqsb
