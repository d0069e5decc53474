/*
 * Fused velocity-Verlet step kernels (sm_103a, FP64) and the device-side run loop.
 *
 * One launch of k_step_line / k_step_grid = one System::timeStep
 * (include/FrictionQPotSpringBlock/detail.h:1539-1570) over all particles, fused with everything
 * timeStep calls: the u update (:1549), updated_u -> potential force with the well search
 * (Cuspy::force :139-170 / SemiSmooth :236-277 / Smooth :379-409), the interaction
 * (Laplace1d::force :474-487 / Laplace2d::force :545-583), the frame force (:1353-1356), the three
 * velocity updates with damping and force sums (:1552-1565, :1321-1395) and the NaN check
 * (:1567-1569); when the run asks for it also the residual terms of minimise /
 * timeStepsUntilEvent (residual :1512-1520, StopList test :1780-1783) and the plastic-activity
 * bookkeeping (:1768-1778, :1855-1866).
 *
 * Run loop.  A run (timeSteps, flowSteps, minimise, minimise_truncate, timeStepsUntilEvent) is one
 * CUDA graph: a conditional WHILE node whose body is many steps of the resident run kernel
 * (fqsb_run.cu), or one step of the kernels here: QuarticGradient2d, LongRange1d, single steps of grids
 * and of thermal systems, thermal systems of more than 2^21 particles, and GPUs on which the run kernel's grid
 * does not fit.  The last CTA to finish a step
 * evaluates the stop tests and sets the loop condition (cudaGraphSetConditional), so the host
 * launches the graph once and synchronises once.  A launch also yields after a device-time budget
 * (%globaltimer), so the host regains control every ~0.2 s of a long run.
 *
 * Chunk windows.  The step kernels only search a particle's current chunk window (a few loads).
 * When the new well lies outside the window's margins the window must move and be regenerated from
 * the particle's pcg32 stream (heavy code: distribution transforms).  That code is kept out of the
 * step kernels (it would raise them to 128 registers and cost ~12% throughput); instead the CTA (or the
 * run kernel's strip) is marked pending, a conditional IF branch of the same graph iteration regenerates the marked
 * particles' windows (k_regen) and repeats the marked CTAs or strips (redo pass).  The step is a pure function
 * of the old state, so the redo reproduces exactly the reference's step.
 *
 * State is double buffered (u, v, a)[cur] -> (u, v, a)[cur ^ 1].  Arithmetic uses explicit
 * __dadd_rn / __dmul_rn in the reference's order (no fma contraction), so results equal the CPU
 * oracle bit for bit.  Only exact rewrites save fp64 issue slots (the fp64 pipe, 1.68 operations per
 * clock per SM on GB300, is the binding unit):
 *   - the partial sum f_frame + f_potential + f_interactions is formed once per step (it is the
 *     same in every computeForce of the step);
 *   - multiplications by parameters equal to 1 are skipped; a product by a power of two is exact, so where
 *     it only feeds an addition (2 u, 4 u, and f_frame, f_interactions with k_frame or k a power of two)
 *     one fma does both;
 *   - the NaN test and, where it is needed at all, the well test yl <= u < yr run on order-preserving
 *     integer keys; a Cuspy particle is first tested against its well's centre and half width, which
 *     reads 16 bytes of the well instead of 32 and takes 2 instructions.
 * Measured at N = 2^22 (Line1d Cuspy, kernel alone): 193 us per step with the sums formed separately, the
 * well test on keys always and the previous integer-pipe operations, 159 us as it is; the 2048 x 2048
 * grid 229 and 195 us.
 */
#include "fqsb_stepcore.cuh"

namespace fqsb {

/*
 * Resident CTAs of 256 threads per SM the step kernels are compiled for (register cap 48 at 5).  The
 * integer-pipe operations are long dependent chains; occupancy hides them (4.9 G particle-steps/s
 * slower at the 93-112 registers the compiler picks unbounded).  The Smooth potential's
 * double-double sine needs more registers than the cap allows without spilling.
 */
template <int POT>
struct StepOcc {
    static constexpr int value = POT == POT_SMOOTH ? 2 : 5;
};

/* Whole-CTA canonical tree over partials[0..G) (zero padded to a power of two). */
static __device__ __noinline__ double2 tree_partials(const double2* partials, int64_t G, double* sh)
{
    int64_t P = next_pow2(G);
    int T = blockDim.x;
    double x = 0.0, y = 0.0;
    if (P <= T) {
        if (threadIdx.x < G) {
            double2 q = __ldcg(partials + threadIdx.x);
            x = q.x;
            y = q.y;
        }
    }
    else {
        int64_t per = P / T;
        int64_t lo = (int64_t)threadIdx.x * per;
        const double2 t = serial_tree2(
            [&](int64_t i) { return i < G ? __ldcg(partials + i) : make_double2(0.0, 0.0); }, lo, per);
        x = t.x;
        y = t.y;
    }
    return cta_tree2(x, y, sh);
}

struct StepShared {
    int exit_flag;
    int cur;
    int flags;
    int last;
    int nan;
    int pending;
    double uf;
    unsigned long long ds;
    unsigned long long da;
    double red[64];
};

/* Reads the run state; returns false when the run is already over (then CTA 0 ends the loop). */
__device__ __forceinline__ bool step_prologue(const DevSys& s, StepShared& sh, bool graph_loop)
{
    int tid = threadIdx.x + threadIdx.y * blockDim.x;
    if (tid == 0) {
        volatile Ctl* c = s.ctl;
        sh.exit_flag = (c->done != 0) || (c->error != 0);
        sh.cur = c->cur;
        sh.flags = c->flags;
        double uf = c->u_frame;
        if (sh.flags & RF_FLOW) {
            uf = FQ_ADD(uf, c->vdt);
        }
        if (sh.flags & RF_SCHEDULE) {
            uf = c->sched[c->step];
        }
        sh.uf = uf;
        sh.nan = 0;
        sh.pending = 0;
        sh.ds = 0ull;
        sh.da = 0ull;
        sh.last = 0;
        if (sh.exit_flag && graph_loop && blockIdx.x == 0 && blockIdx.y == 0) {
            set_loop(s, 0u);
        }
    }
    __syncthreads();
    return sh.exit_flag == 0;
}

/*
 * Well check of particle p at its new position un, from the constants wk of its cached well (loaded by the
 * caller).  Cuspy: d = centre - un, which the force needs anyway, also tells that the particle stays in
 * its well without reading the yield positions; only where it cannot tell is the exact test made (and
 * un looked at for a NaN, which d carries).  The other potentials read the yield positions always.
 * Returns the (possibly new) well, its yield positions unset where the Cuspy test sufficed.  `regen` is set
 * when the chunk window must move; the pass-1 caller then marks its CTA pending.
 */
template <int POT, unsigned SOFT = 0u>
__device__ __forceinline__ double4_32a well_of(const DevSys& s, int64_t p, double un, bool act, StepShared& sh,
                                               double2 wk, double& d, bool& regen)
{
    regen = false;
    double4_32a w = make_double4_32a(0.0, 0.0, wk.x, wk.y);
    d = 0.0;
    if (POT == POT_CUSPY) {
        d = S_SUB(5, wk.x, un);
        if (surely_in_well(wk, d)) {
            return w;
        }
    }
    const double2 wy = s.wy[p];
    w.x = wy.x;
    w.y = wy.y;
    if (is_nan_bits(un)) {
        sh.nan = 1;
    }
    if (!in_well(w.x, w.y, un) && !non_finite(un)) {
        int64_t gold = s.gidx[p];
        if (window_search(s, p, un, w)) {
            int64_t gnew = s.gidx[p];
            if (act && gnew != gold) {
                int64_t ref = s.i_n[p];
                long long ds = absll(gnew - ref) - absll(gold - ref);
                long long da = (long long)(gnew != ref) - (long long)(gold != ref);
                atomicAdd(&sh.ds, (unsigned long long)ds);
                atomicAdd(&sh.da, (unsigned long long)da);
            }
            if (POT == POT_CUSPY) {
                d = fq_s_hw_add(w.z, -un); /* a call: not predicated into the path of the others */
            }
        }
        else {
            regen = true;
        }
    }
    return w;
}

/* Role of the CTA epilogue in the step's kernels. */
enum : int {
    EPI_LINE = 0,      /* 1d pass 1: last CTA finalises, or opens the regeneration branch */
    EPI_GRID_STEP = 1, /* 2d pass 1: last CTA opens (or closes) the regeneration branch */
    EPI_REDO = 2,      /* 1d redo of the pending CTAs: the last of them finalises */
    EPI_REDUCE = 3     /* 2d reduction: last CTA finalises */
};

/*
 * End of a CTA's part of a step: commits activity / NaN flags and the CTA's residual subtree; the CTA
 * that finishes last (ticket) finalises the step or steers the regeneration branch, per `mode`.
 */
__device__ __forceinline__ void step_epilogue(const DevSys& s, StepShared& sh, int mode, double rf, double rff)
{
    const bool resid = (sh.flags & (RF_RESID | RF_FFSUM)) != 0;
    const bool tree = resid && mode != EPI_GRID_STEP;
    double sf = 0.0, sff = 0.0;
    if (tree) {
        double2 t = cta_tree2(rf, rff, sh.red);
        sf = t.x;
        sff = t.y;
    }
    __syncthreads();
    int tid = threadIdx.x + threadIdx.y * blockDim.x;
    int64_t bid = blockIdx.x + (int64_t)blockIdx.y * gridDim.x;
    Ctl* c = s.ctl;
    if (tid == 0) {
        if (tree) {
            s.partials[bid] = make_double2(sf, sff);
        }
        if (sh.ds) {
            atomicAdd((unsigned long long*)&c->s_sum, sh.ds);
        }
        if (sh.da) {
            atomicAdd((unsigned long long*)&c->a_count, sh.da);
        }
        if (sh.nan && !sh.pending) {
            atomicOr(&c->nan_flag, 1);
        }
        if (sh.pending) {
            s.cta_pending[bid] = 1;
            atomicAdd(&c->n_pending_cta, 1);
        }
        __threadfence();
        if (mode == EPI_REDO) {
            unsigned t = atomicAdd(&c->ticket_redo, 1u);
            sh.last = (t == (unsigned)c->n_pending_cta - 1u) ? 1 : 0;
        }
        else {
            unsigned t = atomicAdd(&c->ticket, 1u);
            sh.last = (t == gridDim.x * gridDim.y - 1) ? 1 : 0;
        }
    }
    __syncthreads();
    if (!sh.last) {
        return;
    }
    __threadfence();
    if (mode == EPI_LINE || mode == EPI_GRID_STEP) {
        bool pend = c->n_pending_cta > 0;
        if (pend || mode == EPI_GRID_STEP) {
            if (tid == 0) {
                c->ticket = 0;
                set_branch(s, pend ? 1u : 0u);
            }
            return;
        }
        if (tid == 0) {
            set_branch(s, 0u);
        }
    }
    double2 tot = make_double2(0.0, 0.0);
    if (resid) {
        tot = tree_partials(s.partials, (int64_t)gridDim.x * gridDim.y, sh.red);
    }
    if (tid == 0) {
        finalize_step(s, sh.uf, tot.x, tot.y);
    }
}

/*
 * Line1d (INTER_LAPLACE1D) or Particles (INTER_NONE) step.  Thread t of CTA b owns the PPT consecutive
 * particles b*T*PPT + t*PPT + [0, PPT): a CTA covers an aligned power-of-two range of the flat index,
 * so the residual sums follow the fixed pairwise tree over the flat index.  Updated positions are
 * exchanged through shared memory (one barrier); the two particles just outside the CTA are recomputed
 * from the old state.  State arrays are padded to a multiple of 1024 entries.  redo = 1: only CTAs
 * marked pending run (after k_regen moved their particles' windows).
 */
template <int POT, int INTER, int PPT, unsigned SOFT = STEP_SOFT, bool TH = false>
__global__ void __launch_bounds__(256, StepOcc<POT>::value) k_step_line(const __grid_constant__ DevSys s, int redo)
{
    __shared__ StepShared sh;
    __shared__ double sh_un[256 * PPT];
    __shared__ double sh_halo[2]; /* ring neighbours left of the tile's first particle, right of its last */
    if (!step_prologue(s, sh, true)) {
        return;
    }
    if (redo) {
        if (!s.cta_pending[blockIdx.x]) {
            return;
        }
        __syncthreads();
        if (threadIdx.x == 0) {
            s.cta_pending[blockIdx.x] = 0;
        }
    }
    const int cur = sh.cur;
    const bool act = (sh.flags & (RF_ACT | RF_TRUNCATE | RF_EVENT)) != 0;
    const bool resid = (sh.flags & RF_RESID) != 0;
    const bool ffsum = (sh.flags & RF_FFSUM) != 0;
    const bool record = (sh.flags & RF_RECORD) != 0;
    const int64_t rec_step = record ? ((volatile Ctl*)s.ctl)->step : 0;
    const double uf = sh.uf;
    const int64_t N = s.N;
    const int T = blockDim.x;
    const int64_t base = (int64_t)blockIdx.x * T * PPT;
    const int64_t p0 = base + (int64_t)threadIdx.x * PPT;
    const double* u0 = s.u[cur];
    const double* v0 = s.v[cur];
    const double* a0 = s.a[cur];
    double* u1 = s.u[cur ^ 1];
    double* v1 = s.v[cur ^ 1];
    double* a1 = s.a[cur ^ 1];

    double un[PPT], vr[PPT], ar[PPT];
    /* the cached wells are loaded together with the state, so that their latency overlaps the
     * position update and the neighbour exchange instead of following them */
    double2 wpre[PPT];
#pragma unroll
    for (int j = 0; j < PPT; ++j) {
        wpre[j] = s.wk[p0 + j];
    }
    if (PPT == 2) {
        double2 uu = *reinterpret_cast<const double2*>(u0 + p0);
        double2 vv = *reinterpret_cast<const double2*>(v0 + p0);
        double2 aa = *reinterpret_cast<const double2*>(a0 + p0);
        vr[0] = vv.x;
        vr[PPT - 1] = vv.y;
        ar[0] = aa.x;
        ar[PPT - 1] = aa.y;
        un[0] = S_ADD(3, S_ADD(2, uu.x, S_MULC(0, s.f_dt, s.dt, vr[0])), S_MULC(1, s.f_hdt2, s.hdt2, ar[0]));
        un[PPT - 1] = S_ADD(3, S_ADD(2, uu.y, S_MULC(0, s.f_dt, s.dt, vr[PPT - 1])),
                            S_MULC(1, s.f_hdt2, s.hdt2, ar[PPT - 1]));
    }
    else {
#pragma unroll
        for (int j = 0; j < PPT; ++j) {
            vr[j] = v0[p0 + j];
            ar[j] = a0[p0 + j];
            un[j] = S_ADD(3, S_ADD(2, u0[p0 + j], S_MULC(0, s.f_dt, s.dt, vr[j])), S_MULC(1, s.f_hdt2, s.hdt2, ar[j]));
        }
    }
    if (inter_ring(INTER)) {
#pragma unroll
        for (int j = 0; j < PPT; ++j) {
            sh_un[threadIdx.x * PPT + j] = un[j];
        }
        if (threadIdx.x < 2) {
            /* the two neighbours outside the tile, recomputed from the old state by two lanes of one
             * warp (one pass through the position update instead of one in each of two warps) */
            const int64_t last = (base + (int64_t)T * PPT < N ? base + (int64_t)T * PPT : N) - 1;
            const int64_t q = threadIdx.x == 0 ? (base == 0 ? N - 1 : base - 1) : (last + 1 == N ? 0 : last + 1);
            sh_halo[threadIdx.x] = u_next(s, u0, v0, a0, q);
        }
        __syncthreads();
    }
    double rf = 0.0, rff = 0.0;
    bool pending = false;
    double vo[PPT], ao[PPT];
#pragma unroll
    for (int j = 0; j < PPT; ++j) {
        int64_t p = p0 + j;
        vo[j] = 0.0;
        ao[j] = 0.0;
        if (p >= N) {
            continue;
        }
        double up = un[j];
        bool regen;
        double d;
        double4_32a w = well_of<POT, SOFT>(s, p, up, act, sh, wpre[j], d, regen);
        pending |= regen;
        double ff;
        double sfi = frame_pot<POT, SOFT>(s, w, d, up, uf, ff);
        if (inter_ring(INTER)) {
            int li = threadIdx.x * PPT + j;
            double uL = li > 0 ? sh_un[li - 1] : sh_halo[0];
            double uR = (li + 1 < T * PPT && p + 1 < N) ? sh_un[li + 1] : sh_halo[1];
            sfi = add_ring_force<INTER, SOFT>(s, sfi, uL, up, uR);
        }
        else if (inter_grid(INTER)) {
            /* Laplace2d, the repeat of the run kernel's pending strips: neighbours recomputed from the old state */
            const int64_t C = s.cols, col = p % C;
            const double uU = u_next(s, u0, v0, a0, p >= C ? p - C : p + (N - C));
            const double uD = u_next(s, u0, v0, a0, p < N - C ? p + C : p - (N - C));
            const double uL = u_next(s, u0, v0, a0, col == 0 ? p + (C - 1) : p - 1);
            const double uR = u_next(s, u0, v0, a0, col == C - 1 ? p - (C - 1) : p + 1);
            sfi = grid_force<SOFT>(s, sfi, uU, uD, uL, up, uR);
        }
        else {
            sfi = add_zero(sfi);
        }
        double f;
        verlet_velocity<SOFT, TH>(s, sfi, vr[j], ar[j], vo[j], ao[j], f, TH ? s.f_th[p] : 0.0);
        if (resid) {
            /* squares on the integer pipes (bit-identical), sums on the fp64 pipe */
            double f2 = fq_smul(f, f), ff2 = fq_smul(ff, ff);
            if (j == 0) {
                rf = f2;
                rff = ff2;
            }
            else {
                rf = add_nospec(rf, f2);
                rff = add_nospec(rff, ff2);
            }
        }
        else if (ffsum) {
            rf = j == 0 ? ff : add_nospec(rf, ff);
        }
        if (record) {
            size_t o = (size_t)rec_step * (size_t)N + (size_t)p;
            s.ctl->rec_u[o] = up;
            s.ctl->rec_v[o] = vo[j];
            s.ctl->rec_a[o] = ao[j];
            s.ctl->rec_w[o] = load_well(s, p);
        }
    }
    if (p0 < N) {
        if (PPT == 2) {
            *reinterpret_cast<double2*>(u1 + p0) = make_double2(un[0], un[PPT - 1]);
            *reinterpret_cast<double2*>(v1 + p0) = make_double2(vo[0], vo[PPT - 1]);
            *reinterpret_cast<double2*>(a1 + p0) = make_double2(ao[0], ao[PPT - 1]);
        }
        else {
#pragma unroll
            for (int j = 0; j < PPT; ++j) {
                u1[p0 + j] = un[j];
                v1[p0 + j] = vo[j];
                a1[p0 + j] = ao[j];
            }
        }
    }
    if (pending && !redo) {
        sh.pending = 1;
        for (int j = 0; j < PPT; ++j) {
            /* record the particles of this thread that need a new window */
            int64_t p = p0 + j;
            if (p < N) {
                double2 w = s.wy[p];
                if (!in_well(w.x, w.y, un[j]) && !non_finite(un[j])) {
                    int k = atomicAdd(&s.ctl->n_regen, 1);
                    s.regen_list[k] = (int32_t)p;
                }
            }
        }
    }
    if (pending && redo) {
        /* the window could not be moved (yield search bound): reported by the finalisation */
        atomicOr(&s.ctl->walk_flag, 1);
    }
    step_epilogue(s, sh, redo ? EPI_REDO : EPI_LINE, rf, rff);
}

/*
 * Line2d step: CTA tile of 8 rows x 32 columns, one particle per thread, the neighbourhood read from
 * a haloed shared tile (the halo of 84 positions recomputed by three whole warps).  The residual terms are
 * written per particle (sq2) and summed in the flat-index pairwise order by k_reduce_grid, which
 * also finalises the step.
 */
template <int POT, int INTER = INTER_LAPLACE2D, unsigned SOFT = STEP_SOFT>
__global__ void __launch_bounds__(256, StepOcc<POT>::value) k_step_grid(const __grid_constant__ DevSys s, int redo)
{
    __shared__ StepShared sh;
    /* the tile's new positions at [1 + row][1 + column], with the halo around its nr x nc valid
     * particles: rows 0 and 1 + nr, columns 0 and 1 + nc, and the four corners */
    __shared__ double sh_un[10][34];
    if (!step_prologue(s, sh, true)) {
        return;
    }
    const int64_t bid = blockIdx.x + (int64_t)blockIdx.y * gridDim.x;
    if (redo) {
        if (!s.cta_pending[bid]) {
            return;
        }
        __syncthreads();
        if (threadIdx.x == 0 && threadIdx.y == 0) {
            s.cta_pending[bid] = 0;
        }
    }
    const int cur = sh.cur;
    const bool act = (sh.flags & (RF_ACT | RF_TRUNCATE | RF_EVENT)) != 0;
    const bool resid = (sh.flags & RF_RESID) != 0;
    const double uf = sh.uf;
    const int64_t R = s.rows, C = s.cols;
    const int tx = threadIdx.x, ty = threadIdx.y;
    const int64_t row0 = (int64_t)blockIdx.y * 8, col0 = (int64_t)blockIdx.x * 32;
    const int nr = (int)(R - row0 < 8 ? R - row0 : 8);
    const int nc = (int)(C - col0 < 32 ? C - col0 : 32);
    const int64_t i = row0 + ty;
    const int64_t jc = col0 + tx;
    const bool valid = i < R && jc < C;
    const double* u0 = s.u[cur];
    const double* v0 = s.v[cur];
    const double* a0 = s.a[cur];
    const int64_t p = i * C + jc;
    double up = 0.0, vr = 0.0, ar = 0.0;
    double2 wk = make_double2(0.0, 0.0);
    if (valid) {
        wk = s.wk[p];
        vr = v0[p];
        ar = a0[p];
        up = S_ADD(3, S_ADD(2, u0[p], S_MULC(0, s.f_dt, s.dt, vr)), S_MULC(1, s.f_hdt2, s.hdt2, ar));
        sh_un[1 + ty][1 + tx] = up;
    }
    {
        /* the halo, recomputed from the old state (periodic) by whole warps: warp 0 the row above,
         * warp 1 the row below, warp 2 the side columns (lanes 0-7 left, 8-15 right) and the corners
         * (lanes 16-19) */
        const int64_t rt = (row0 + R - 1) % R, rb = (row0 + nr) % R;
        const int64_t cl = (col0 + C - 1) % C, cr = (col0 + nc) % C;
        if (ty == 0 && tx < nc) {
            sh_un[0][1 + tx] = u_next(s, u0, v0, a0, rt * C + jc);
        }
        else if (ty == 1 && tx < nc) {
            sh_un[1 + nr][1 + tx] = u_next(s, u0, v0, a0, rb * C + jc);
        }
        else if (ty == 2 && tx < 20) {
            int r, c;
            int64_t q;
            if (tx < 16) {
                const int k = tx & 7;
                r = 1 + k;
                c = tx < 8 ? 0 : 1 + nc;
                q = (row0 + k) * C + (tx < 8 ? cl : cr);
            }
            else {
                const int k = tx - 16;
                r = k < 2 ? 0 : 1 + nr;
                c = (k & 1) ? 1 + nc : 0;
                q = (k < 2 ? rt : rb) * C + ((k & 1) ? cr : cl);
            }
            if (tx >= 16 || (tx & 7) < nr) {
                sh_un[r][c] = u_next(s, u0, v0, a0, q);
            }
        }
    }
    __syncthreads();
    if (valid) {
        bool regen;
        double d;
        double4_32a w = well_of<POT, SOFT>(s, p, up, act, sh, wk, d, regen);
        if (regen) {
            if (!redo) {
                sh.pending = 1;
                int k = atomicAdd(&s.ctl->n_regen, 1);
                s.regen_list[k] = (int32_t)p;
            }
            else {
                atomicOr(&s.ctl->walk_flag, 1);
            }
        }
        double ff;
        double sfp = frame_pot<POT, SOFT>(s, w, d, up, uf, ff);
        double fi;
        if (INTER == INTER_LAPLACE2D) {
            const double uU = sh_un[ty][1 + tx];
            const double uD = sh_un[ty + 2][1 + tx];
            const double uL = sh_un[1 + ty][tx];
            const double uR = sh_un[1 + ty][tx + 2];
            fi = scale(FQ_SUB(FQ_ADD(FQ_ADD(FQ_ADD(uU, uD), uL), uR), scale_pow2(up, 2, 4.0)), s.s_k);
        }
        else {
            /* 3 x 3 neighbourhood from the haloed tile */
            auto nb = [&](int di, int dj) -> double { return sh_un[1 + ty + di][1 + tx + dj]; };
            fi = qg2d_force(s, up, nb(1, 0), nb(-1, 0), nb(0, 1), nb(0, -1), nb(1, 1), nb(1, -1), nb(-1, 1), nb(-1, -1));
        }
        double sfi = S_ADD(9, sfp, fi);
        double vv, aa, f;
        verlet_velocity<SOFT>(s, sfi, vr, ar, vv, aa, f);
        s.u[cur ^ 1][p] = up;
        s.v[cur ^ 1][p] = vv;
        s.a[cur ^ 1][p] = aa;
        if (resid) {
            s.sq2[p] = make_double2(fq_smul(f, f), fq_smul(ff, ff));
        }
    }
    if (redo) {
        /* the reduction kernel after the branch finalises; only the counters are committed here */
        __syncthreads();
        if (threadIdx.x == 0 && threadIdx.y == 0) {
            if (sh.ds) {
                atomicAdd((unsigned long long*)&s.ctl->s_sum, sh.ds);
            }
            if (sh.da) {
                atomicAdd((unsigned long long*)&s.ctl->a_count, sh.da);
            }
            if (sh.nan) {
                atomicOr(&s.ctl->nan_flag, 1);
            }
        }
        return;
    }
    step_epilogue(s, sh, EPI_GRID_STEP, 0.0, 0.0);
}

/*
 * Line2d Laplace2d step with two rows per thread: CTA tile of 16 rows x 32 columns (blockDim 32 x 8,
 * thread (x, y) owns rows 2y and 2y + 1 of column x).  All four neighbours come from shared memory:
 * the tile's new positions and a recomputed halo of 96 positions per 512 particles, computed by three
 * whole warps (the 8 x 32 tiles of k_step_grid recompute their side columns in one lane per warp and
 * row).  Per particle the same operations in the same order as k_step_grid, so the same results.
 * Takes single steps and the kernel-by-kernel form of the run loop; longer runs take the run kernel.
 */
template <int POT, unsigned SOFT = STEP_SOFT>
__global__ void __launch_bounds__(256, StepOcc<POT>::value) k_step_grid2(const __grid_constant__ DevSys s, int redo)
{
    __shared__ StepShared sh;
    /* the tile's new positions at [1 + row][1 + column], with the four halo lines around them: row 0
     * and row 1 + nr (the rows above and below the tile's nr valid rows), column 0 and column 1 + nc */
    __shared__ double sh_un[18][34];
    if (!step_prologue(s, sh, true)) {
        return;
    }
    const int64_t bid = blockIdx.x + (int64_t)blockIdx.y * gridDim.x;
    if (redo) {
        if (!s.cta_pending[bid]) {
            return;
        }
        __syncthreads();
        if (threadIdx.x == 0 && threadIdx.y == 0) {
            s.cta_pending[bid] = 0;
        }
    }
    const int cur = sh.cur;
    const bool act = (sh.flags & (RF_ACT | RF_TRUNCATE | RF_EVENT)) != 0;
    const bool resid = (sh.flags & RF_RESID) != 0;
    const double uf = sh.uf;
    const int64_t R = s.rows, C = s.cols;
    const int tx = threadIdx.x, ty = threadIdx.y;
    const int64_t row0 = (int64_t)blockIdx.y * 16, col0 = (int64_t)blockIdx.x * 32;
    const int nr = (int)(R - row0 < 16 ? R - row0 : 16);
    const int nc = (int)(C - col0 < 32 ? C - col0 : 32);
    const int64_t jc = col0 + tx;
    const int64_t i0 = row0 + 2 * ty;
    const double* u0 = s.u[cur];
    const double* v0 = s.v[cur];
    const double* a0 = s.a[cur];
    double up[2], vr[2], ar[2];
    double2 wk[2];
#pragma unroll
    for (int q = 0; q < 2; ++q) {
        const int64_t i = i0 + q;
        up[q] = vr[q] = ar[q] = 0.0;
        wk[q] = make_double2(0.0, 0.0);
        if (i < R && jc < C) {
            const int64_t p = i * C + jc;
            wk[q] = s.wk[p];
            vr[q] = v0[p];
            ar[q] = a0[p];
            up[q] = S_ADD(3, S_ADD(2, u0[p], S_MULC(0, s.f_dt, s.dt, vr[q])), S_MULC(1, s.f_hdt2, s.hdt2, ar[q]));
            sh_un[1 + 2 * ty + q][1 + tx] = up[q];
        }
    }
    /* the halo, recomputed from the old state (periodic): warp 0 the row above, warp 1 the row below,
     * warp 2 the columns left (lanes 0-15) and right (lanes 16-31); whole warps, no divergent lanes */
    if (ty == 0 && tx < nc) {
        sh_un[0][1 + tx] = u_next(s, u0, v0, a0, ((row0 + R - 1) % R) * C + jc);
    }
    else if (ty == 1 && tx < nc) {
        sh_un[1 + nr][1 + tx] = u_next(s, u0, v0, a0, ((row0 + nr) % R) * C + jc);
    }
    else if (ty == 2 && (tx & 15) < nr) {
        const int r = tx & 15;
        const int64_t c = tx < 16 ? (col0 + C - 1) % C : (col0 + nc) % C;
        sh_un[1 + r][tx < 16 ? 0 : 1 + nc] = u_next(s, u0, v0, a0, (row0 + r) * C + c);
    }
    __syncthreads();
#pragma unroll
    for (int q = 0; q < 2; ++q) {
        const int64_t i = i0 + q;
        if (!(i < R && jc < C)) {
            continue;
        }
        const int64_t p = i * C + jc;
        const int r = 2 * ty + q;
        bool regen;
        double d;
        double4_32a w = well_of<POT, SOFT>(s, p, up[q], act, sh, wk[q], d, regen);
        if (regen) {
            if (!redo) {
                sh.pending = 1;
                int k = atomicAdd(&s.ctl->n_regen, 1);
                s.regen_list[k] = (int32_t)p;
            }
            else {
                atomicOr(&s.ctl->walk_flag, 1);
            }
        }
        double ff;
        double sfp = frame_pot<POT, SOFT>(s, w, d, up[q], uf, ff);
        const double uU = sh_un[r][1 + tx];
        const double uD = sh_un[r + 2][1 + tx];
        const double uL = sh_un[1 + r][tx];
        const double uR = sh_un[1 + r][tx + 2];
        const double sfi = grid_force<SOFT>(s, sfp, uU, uD, uL, up[q], uR);
        double vv, aa, f;
        verlet_velocity<SOFT>(s, sfi, vr[q], ar[q], vv, aa, f);
        s.u[cur ^ 1][p] = up[q];
        s.v[cur ^ 1][p] = vv;
        s.a[cur ^ 1][p] = aa;
        if (resid) {
            s.sq2[p] = make_double2(fq_smul(f, f), fq_smul(ff, ff));
        }
    }
    if (redo) {
        /* the reduction kernel after the branch finalises; only the counters are committed here */
        __syncthreads();
        if (threadIdx.x == 0 && threadIdx.y == 0) {
            if (sh.ds) {
                atomicAdd((unsigned long long*)&s.ctl->s_sum, sh.ds);
            }
            if (sh.da) {
                atomicAdd((unsigned long long*)&s.ctl->a_count, sh.da);
            }
            if (sh.nan) {
                atomicOr(&s.ctl->nan_flag, 1);
            }
        }
        return;
    }
    step_epilogue(s, sh, EPI_GRID_STEP, 0.0, 0.0);
}

/* Rows of a CTA tile of the 2d step kernel: 16 for Laplace2d (k_step_grid2), 8 otherwise. */
static int64_t grid_tile_rows(const DevSys& s)
{
    return s.inter == INTER_LAPLACE2D ? 16 : 8;
}

/* Pairwise reduction of the 2d step's sq2 in flat-index order (1024 per CTA) + step finalisation. */
__global__ void __launch_bounds__(256) k_reduce_grid(DevSys s)
{
    __shared__ StepShared sh;
    if (!step_prologue(s, sh, true)) {
        return;
    }
    const bool resid = (sh.flags & RF_RESID) != 0;
    double rf = 0.0, rff = 0.0;
    if (resid) {
        int64_t lo = (int64_t)blockIdx.x * 1024 + threadIdx.x * 4;
        double x[4], y[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            if (lo + j < s.N) {
                double2 q = s.sq2[lo + j];
                x[j] = q.x;
                y[j] = q.y;
            }
            else {
                x[j] = 0.0;
                y[j] = 0.0;
            }
        }
        rf = FQ_ADD(FQ_ADD(x[0], x[1]), FQ_ADD(x[2], x[3]));
        rff = FQ_ADD(FQ_ADD(y[0], y[1]), FQ_ADD(y[2], y[3]));
    }
    step_epilogue(s, sh, EPI_REDUCE, rf, rff);
}

/* Regeneration branch: move the chunk windows of the particles recorded by pass 1. */
__global__ void __launch_bounds__(128) k_regen(DevSys s)
{
    Ctl* c = s.ctl;
    if (c->done || c->error) {
        return;
    }
    const int cur = c->cur;
    const bool act = (c->flags & (RF_ACT | RF_TRUNCATE | RF_EVENT)) != 0;
    const int n = c->n_regen;
    auto count_move = [&](int64_t p, int64_t gold) {
        int64_t gnew = s.gidx[p];
        if (act && gnew != gold) {
            int64_t ref = s.i_n[p];
            long long ds = absll(gnew - ref) - absll(gold - ref);
            long long da = (long long)(gnew != ref) - (long long)(gold != ref);
            atomicAdd((unsigned long long*)&c->s_sum, (unsigned long long)ds);
            atomicAdd((unsigned long long*)&c->a_count, (unsigned long long)da);
        }
    };
    if (n >= (int)(gridDim.x * blockDim.x) / 4) {
        /* many moves: one thread per particle keeps every thread busy */
        for (int k = blockIdx.x * blockDim.x + threadIdx.x; k < n; k += gridDim.x * blockDim.x) {
            int64_t p = s.regen_list[k];
            int64_t gold = s.gidx[p];
            dev_align(s, p, u_next(s, s.u[cur], s.v[cur], s.a[cur], p));
            count_move(p, gold);
        }
        return;
    }
    /* few moves: one CTA per particle, its threads sharing the draws (fwd_move_*); the same values */
    __shared__ FwdMove m_sh;
    __shared__ int ok_sh;
    __shared__ long long gold_sh;
    const uint64_t mv_c = pcg_advance(0ULL, (uint64_t)blockDim.x);
    const uint64_t mv_a = pcg_advance(1ULL, (uint64_t)blockDim.x) - mv_c;
    for (int k = blockIdx.x; k < n; k += gridDim.x) {
        const int64_t p = s.regen_list[k];
        if (threadIdx.x == 0) {
            double un = u_next(s, s.u[cur], s.v[cur], s.a[cur], p);
            gold_sh = s.gidx[p];
            FwdMove m;
            ok_sh = fwd_move_plan(s, p, un, m) ? 1 : 0;
            if (ok_sh) {
                m_sh = m;
            }
            else {
                dev_align(s, p, un);
            }
        }
        __syncthreads();
        if (ok_sh) {
            fwd_move_draws(s, m_sh, (int)threadIdx.x, (int)blockDim.x, mv_a, mv_c);
        }
        __syncthreads();
        if (threadIdx.x == 0) {
            if (ok_sh) {
                fwd_move_sum(s, m_sh);
            }
            count_move(p, gold_sh);
        }
        __syncthreads();
    }
}

/*
 * Next-window buffers of a small system, refreshed before a run of the one-cluster kernel: each CTA
 * takes particles blockIdx.x, blockIdx.x + gridDim.x, ...; a particle whose buffer does not follow
 * its current window (next_window_ready) gets the W draws after the window end from all the CTA's
 * threads, then their running sum from one thread.  A particle whose buffer is current costs one
 * comparison, so the kernel is cheap when few windows moved.
 */
__global__ void __launch_bounds__(128) k_next_window(DevSys s)
{
    __shared__ int need_sh, kind_sh;
    __shared__ uint64_t st_sh;
    __shared__ long long end_sh;
    const uint64_t mv_c = pcg_advance(0ULL, (uint64_t)blockDim.x);
    const uint64_t mv_a = pcg_advance(1ULL, (uint64_t)blockDim.x) - mv_c;
    for (int64_t p = blockIdx.x; p < s.N; p += gridDim.x) {
        if (threadIdx.x == 0) {
            const int64_t end = s.start[p] + s.W - 1;
            int kind;
            int64_t ko;
            uint64_t sto;
            need_sh = s.nx_end[p] != end && next_window_applies(s, p, end, kind, ko, sto);
            if (need_sh) {
                kind_sh = kind;
                end_sh = end;
                st_sh = pcg_advance(sto, (uint64_t)(end + 1 - ko));
            }
        }
        __syncthreads();
        if (need_sh) {
            seq_draws(s, s.nx + p * s.W, s.W, st_sh, (int)threadIdx.x, (int)blockDim.x, mv_a, mv_c);
            __syncthreads();
            if (threadIdx.x == 0) {
                next_window_sum(s, p, end_sh, kind_sh);
                s.nx_end[p] = end_sh;
            }
        }
        __syncthreads();
    }
}

cudaError_t launch_next_window(const DevSys& s, cudaStream_t st)
{
    if (s.nx == nullptr) {
        return cudaSuccess;
    }
    const int64_t grid = s.N < 4 * 152 ? s.N : 4 * 152;
    k_next_window<<<(unsigned)grid, 128, 0, st>>>(s);
    return cudaGetLastError();
}

/* ------------------------------------------------------------- long-range interactions */

/*
 * Line1d System_Cuspy_LongRange (Line1d.h:617-675): every particle interacts with all others,
 * f_int(p) = sum over i != p, in index order, of (u'(i) - u'(p)) k / d^(alpha+1), d the ring distance
 * (LongRange1d::force, detail.h:844-866).  All new positions are needed before any interaction, so
 * the step is two launches: k_lr_position writes u' for all particles; k_lr_step (same pass-1 / redo
 * roles and epilogue as k_step_line) reads the new positions through shared-memory tiles, keeps each
 * particle's sum in the reference's sequential order, and does wells, forces, velocity updates and
 * the residual.
 */
__global__ void __launch_bounds__(256) k_lr_position(DevSys s)
{
    __shared__ StepShared sh;
    if (!step_prologue(s, sh, true)) {
        return;
    }
    const int cur = sh.cur;
    const int64_t p = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (p < s.N) {
        s.u[cur ^ 1][p] = u_next(s, s.u[cur], s.v[cur], s.a[cur], p);
    }
}

template <int POT, int PPT>
__global__ void __launch_bounds__(256) k_lr_step(const __grid_constant__ DevSys s, int redo)
{
    constexpr int LR_TILE = 1024;
    __shared__ StepShared sh;
    __shared__ double tile[LR_TILE];
    if (!step_prologue(s, sh, true)) {
        return;
    }
    if (redo) {
        if (!s.cta_pending[blockIdx.x]) {
            return;
        }
        __syncthreads();
        if (threadIdx.x == 0) {
            s.cta_pending[blockIdx.x] = 0;
        }
    }
    const int cur = sh.cur;
    const bool act = (sh.flags & (RF_ACT | RF_TRUNCATE | RF_EVENT)) != 0;
    const bool resid = (sh.flags & RF_RESID) != 0;
    const double uf = sh.uf;
    const int64_t N = s.N;
    const int64_t p0 = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) * PPT;
    const double* un = s.u[cur ^ 1];
    double up[PPT], fi[PPT];
#pragma unroll
    for (int j = 0; j < PPT; ++j) {
        up[j] = p0 + j < N ? un[p0 + j] : 0.0;
        fi[j] = 0.0;
    }
    for (int64_t t0 = 0; t0 < N; t0 += LR_TILE) {
        const int cnt = (int)(N - t0 < LR_TILE ? N - t0 : LR_TILE);
        __syncthreads();
        for (int k = threadIdx.x; k < cnt; k += blockDim.x) {
            tile[k] = un[t0 + k];
        }
        __syncthreads();
#pragma unroll
        for (int j = 0; j < PPT; ++j) {
            const int64_t p = p0 + j;
            if (p >= N) {
                continue;
            }
            double acc = fi[j];
            for (int k = 0; k < cnt; ++k) {
                const int64_t i = t0 + k;
                if (i == p) {
                    continue;
                }
                int64_t d = i > p ? i - p : p - i;
                if (d > s.lr_m) {
                    d = N - d;
                }
                acc = FQ_ADD(acc, FQ_MUL(FQ_SUB(tile[k], up[j]), __ldg(s.lr_pref + d)));
            }
            fi[j] = acc;
        }
    }
    double rf = 0.0, rff = 0.0;
    bool pending = false;
#pragma unroll
    for (int j = 0; j < PPT; ++j) {
        const int64_t p = p0 + j;
        if (p >= N) {
            continue;
        }
        bool regen;
        double d;
        double4_32a w = well_of<POT>(s, p, up[j], act, sh, s.wk[p], d, regen);
        pending |= regen;
        double ff;
        double sfp = frame_pot<POT>(s, w, d, up[j], uf, ff);
        double sfi = FQ_ADD(sfp, fi[j]);
        double vo, ao, f;
        verlet_velocity(s, sfi, s.v[cur][p], s.a[cur][p], vo, ao, f);
        s.v[cur ^ 1][p] = vo;
        s.a[cur ^ 1][p] = ao;
        if (resid) {
            double f2 = fq_smul(f, f), ff2 = fq_smul(ff, ff);
            if (j == 0) {
                rf = f2;
                rff = ff2;
            }
            else {
                rf = add_nospec(rf, f2);
                rff = add_nospec(rff, ff2);
            }
        }
    }
    if (pending && !redo) {
        sh.pending = 1;
        for (int j = 0; j < PPT; ++j) {
            const int64_t p = p0 + j;
            if (p < N) {
                double2 w = s.wy[p];
                if (!in_well(w.x, w.y, up[j]) && !non_finite(up[j])) {
                    int k = atomicAdd(&s.ctl->n_regen, 1);
                    s.regen_list[k] = (int32_t)p;
                }
            }
        }
    }
    if (pending && redo) {
        atomicOr(&s.ctl->walk_flag, 1);
    }
    step_epilogue(s, sh, redo ? EPI_REDO : EPI_LINE, rf, rff);
}

/* ------------------------------------------------------------- no-passing minimiser */

/*
 * minimise of System_Cuspy_Laplace_Nopassing (detail.h:1694-1753, class Line1d.h:173-238): one Jacobi
 * sweep per loop iteration, in the same run graph form as the dynamics (WHILE node, stop test on the
 * device).  k_nopass_update: from the previous sweep's positions (buffer cur, the reference's v_n
 * snapshot) each particle takes
 *     u = ((k (u[p-1] + u[p+1]) + k_frame u_frame) + mu umin) / ((2 k + k_frame) + mu),
 * umin the centre of its current well; the chunk is aligned at u (moving the window when needed) and,
 * while the local chunk index changes, u is recomputed with the new well.  Writes u (buffer cur ^ 1),
 * f_frame and f_potential.  k_nopass_force: f_interactions of the new positions,
 * f = (f_potential + f_interactions) + f_frame, the residual subtrees; the last CTA runs the StopList
 * test (finalize_step with RF_NOINC: no time passes).
 */
__global__ void __launch_bounds__(256) k_nopass_update(DevSys s, NopassArgs A)
{
    __shared__ StepShared sh;
    if (!step_prologue(s, sh, true)) {
        return;
    }
    const int cur = sh.cur;
    const double uf = sh.uf;
    const int64_t N = s.N;
    const double* u0 = s.u[cur];
    const int64_t p0 = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) * A.ppt;
    for (int j = 0; j < A.ppt; ++j) {
        const int64_t p = p0 + j;
        if (p >= N) {
            break;
        }
        const double uneigh = p == 0       ? FQ_ADD(u0[N - 1], u0[1])
                              : p == N - 1 ? FQ_ADD(u0[N - 2], u0[0])
                                           : FQ_ADD(u0[p - 1], u0[p + 1]);
        const double* y = s.data + p * s.W;
        int64_t i = s.cidx[p];
        double umin = 0.0, u = 0.0;
        for (int it = 0;; ++it) {
            if (it >= NOPASS_MAX_REALIGN) {
                atomicOr(&s.ctl->walk_flag, 1); /* reported as an error by the finalisation */
                break;
            }
            umin = FQ_MUL(0.5, FQ_ADD(y[i], y[i + 1]));
            u = FQ_DIV(FQ_ADD(FQ_ADD(FQ_MUL(s.k, uneigh), FQ_MUL(s.k_frame, uf)), FQ_MUL(s.mu, umin)), A.den);
            dev_align(s, p, u);
            const int64_t jj = s.cidx[p];
            if (jj == i) {
                break;
            }
            i = jj;
        }
        s.u[cur ^ 1][p] = u;
        s.v[cur ^ 1][p] = s.v[cur][p];
        s.a[cur ^ 1][p] = s.a[cur][p];
        A.f_frame[p] = FQ_MUL(s.k_frame, FQ_SUB(uf, u));
        A.f_pot[p] = FQ_MUL(s.mu, FQ_SUB(umin, u));
    }
}

__global__ void __launch_bounds__(256) k_nopass_force(DevSys s, NopassArgs A)
{
    __shared__ StepShared sh;
    if (!step_prologue(s, sh, true)) {
        return;
    }
    const int cur = sh.cur;
    const int64_t N = s.N;
    const double* u1 = s.u[cur ^ 1];
    const int64_t p0 = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) * A.ppt;
    double rf = 0.0, rff = 0.0;
    for (int j = 0; j < A.ppt; ++j) {
        const int64_t p = p0 + j;
        if (p >= N) {
            break;
        }
        const double u = u1[p];
        const double uL = u1[p == 0 ? N - 1 : p - 1], uR = u1[p == N - 1 ? 0 : p + 1];
        const double fi = scale(FQ_ADD(FQ_SUB(uL, scale_pow2(u, 1, 2.0)), uR), s.s_k);
        const double ff = A.f_frame[p];
        const double f = FQ_ADD(FQ_ADD(A.f_pot[p], fi), ff);
        A.f_int[p] = fi;
        A.f[p] = f;
        const double f2 = FQ_MUL(f, f), ff2 = FQ_MUL(ff, ff);
        if (j == 0) {
            rf = f2;
            rff = ff2;
        }
        else {
            rf = FQ_ADD(rf, f2);
            rff = FQ_ADD(rff, ff2);
        }
    }
    step_epilogue(s, sh, EPI_LINE, rf, rff);
}

cudaError_t launch_nopass_iteration(const DevSys& s, const LineGeom& g, const NopassArgs& A, cudaStream_t st)
{
    k_nopass_update<<<(unsigned)g.grid, (unsigned)g.threads, 0, st>>>(s, A);
    k_nopass_force<<<(unsigned)g.grid, (unsigned)g.threads, 0, st>>>(s, A);
    return cudaGetLastError();
}

/* ------------------------------------------------------------- geometry */

LineGeom line_geometry(int64_t N)
{
    LineGeom g;
    /* enough CTAs to fill 152 SMs when N allows, power-of-two tiles for the canonical reduction */
    int64_t tile = 512;
    while (tile > 32 && (N + tile - 1) / tile < 2 * 152) {
        tile >>= 1;
    }
    g.ppt = tile >= 512 ? 2 : 1;
    g.threads = (int)(tile / g.ppt);
    g.grid = (N + tile - 1) / tile;
    return g;
}

LineGeom strip_geometry(int64_t N, int S)
{
    LineGeom g;
    g.ppt = 1;
    g.threads = S;
    g.grid = (N + S - 1) / S;
    return g;
}

int64_t grid_reduce_ctas(int64_t N)
{
    return (N + 1023) / 1024;
}

int64_t step_ctas(const DevSys& s, const LineGeom& g)
{
    if (inter_grid(s.inter)) {
        return ((s.cols + 31) / 32) * ((s.rows + grid_tile_rows(s) - 1) / grid_tile_rows(s));
    }
    return g.grid;
}

/* ------------------------------------------------------------- run graph */

template <int POT, int INTER, bool TH = false>
static void* line_kernel_t(int ppt)
{
    return ppt == 2 ? (void*)k_step_line<POT, INTER, 2, STEP_SOFT, TH> : (void*)k_step_line<POT, INTER, 1, STEP_SOFT, TH>;
}

static void* step_kernel(const DevSys& s, const LineGeom& g)
{
    if (s.f_th) {
        /* RandomNormalForcing systems: Cuspy with Laplace1d, Quartic1d or no interactions */
        switch (s.inter) {
            case INTER_LAPLACE1D: return line_kernel_t<POT_CUSPY, INTER_LAPLACE1D, true>(g.ppt);
            case INTER_QUARTIC1D: return line_kernel_t<POT_CUSPY, INTER_QUARTIC1D, true>(g.ppt);
            default: return line_kernel_t<POT_CUSPY, INTER_NONE, true>(g.ppt);
        }
    }
    if (s.inter == INTER_LONGRANGE1D) {
        return g.ppt == 2 ? (void*)k_lr_step<POT_CUSPY, 2> : (void*)k_lr_step<POT_CUSPY, 1>;
    }
    if (s.inter == INTER_QUARTICGRAD2D) {
        return (void*)k_step_grid<POT_CUSPY, INTER_QUARTICGRAD2D>;
    }
    if (s.inter == INTER_QUARTIC1D) {
        return line_kernel_t<POT_CUSPY, INTER_QUARTIC1D>(g.ppt);
    }
    if (s.inter == INTER_QUARTICGRAD1D) {
        return line_kernel_t<POT_CUSPY, INTER_QUARTICGRAD1D>(g.ppt);
    }
    if (s.inter == INTER_LAPLACE2D) {
        switch (s.pot) {
            case POT_CUSPY: return (void*)k_step_grid2<POT_CUSPY>;
            case POT_SEMISMOOTH: return (void*)k_step_grid2<POT_SEMISMOOTH>;
            default: return (void*)k_step_grid2<POT_SMOOTH>;
        }
    }
    if (s.inter == INTER_LAPLACE1D) {
        switch (s.pot) {
            case POT_CUSPY: return line_kernel_t<POT_CUSPY, INTER_LAPLACE1D>(g.ppt);
            case POT_SEMISMOOTH: return line_kernel_t<POT_SEMISMOOTH, INTER_LAPLACE1D>(g.ppt);
            default: return line_kernel_t<POT_SMOOTH, INTER_LAPLACE1D>(g.ppt);
        }
    }
    switch (s.pot) {
        case POT_CUSPY: return line_kernel_t<POT_CUSPY, INTER_NONE>(g.ppt);
        case POT_SEMISMOOTH: return line_kernel_t<POT_SEMISMOOTH, INTER_NONE>(g.ppt);
        default: return line_kernel_t<POT_SMOOTH, INTER_NONE>(g.ppt);
    }
}

/* The kernel that repeats the run kernel's pending strips */
static void* redo_kernel(const DevSys& s, const LineGeom& g)
{
    if (s.inter == INTER_LAPLACE2D) {
        switch (s.pot) {
            case POT_CUSPY: return (void*)k_step_line<POT_CUSPY, INTER_LAPLACE2D, 1>;
            case POT_SEMISMOOTH: return (void*)k_step_line<POT_SEMISMOOTH, INTER_LAPLACE2D, 1>;
            default: return (void*)k_step_line<POT_SMOOTH, INTER_LAPLACE2D, 1>;
        }
    }
    return step_kernel(s, g);
}

static cudaError_t add_kernel(cudaGraphNode_t* node, cudaGraph_t graph, const cudaGraphNode_t* deps, size_t ndeps,
                              void* func, dim3 grid, dim3 block, void** args)
{
    cudaKernelNodeParams kp = {};
    kp.func = func;
    kp.gridDim = grid;
    kp.blockDim = block;
    kp.sharedMemBytes = 0;
    kp.kernelParams = args;
    kp.extra = nullptr;
    return cudaGraphAddKernelNode(node, graph, deps, ndeps, &kp);
}

static cudaError_t add_conditional(cudaGraphNode_t* node, cudaGraph_t graph, const cudaGraphNode_t* deps, size_t ndeps,
                                   cudaGraphConditionalHandle h, cudaGraphConditionalNodeType type, cudaGraph_t* body)
{
    cudaGraphNodeParams np = {};
    np.type = cudaGraphNodeTypeConditional;
    np.conditional.handle = h;
    np.conditional.type = type;
    np.conditional.size = 1;
    cudaError_t e = cudaGraphAddNode(node, graph, deps, nullptr, ndeps, &np);
    if (e == cudaSuccess) {
        *body = np.conditional.phGraph_out[0];
    }
    return e;
}

/*
 * Host-driven form of one loop iteration (no conditional nodes, e.g. for profilers that cannot
 * profile kernels inside conditional graphs): pass 1, the regeneration kernel and the redo are always
 * launched; the latter two do nothing when no CTA is pending.
 */
cudaError_t launch_iteration(const DevSys& s, const LineGeom& g0, cudaStream_t st)
{
    bool is2d = inter_grid(s.inter);
    dim3 grid, block;
    if (is2d) {
        grid = dim3((unsigned)((s.cols + 31) / 32), (unsigned)((s.rows + grid_tile_rows(s) - 1) / grid_tile_rows(s)));
        block = dim3(32, 8);
    }
    else {
        grid = dim3((unsigned)g0.grid);
        block = dim3((unsigned)g0.threads);
    }
    void* fstep = step_kernel(s, g0);
    int pass1 = 0, pass2 = 1;
    void* args1[] = {(void*)&s, (void*)&pass1};
    void* args2[] = {(void*)&s, (void*)&pass2};
    void* argsr[] = {(void*)&s};
    cudaError_t e = cudaSuccess;
    if (s.f_th) {
        e = launch_thermal_step(s, st);
    }
    if (e == cudaSuccess && s.inter == INTER_LONGRANGE1D) {
        e = cudaLaunchKernel((void*)k_lr_position, dim3((unsigned)((s.N + 255) / 256)), dim3(256), argsr, 0, st);
    }
    if (e == cudaSuccess) {
        e = cudaLaunchKernel(fstep, grid, block, args1, 0, st);
    }
    if (e == cudaSuccess) {
        e = cudaLaunchKernel((void*)k_regen, dim3(4 * 152), dim3(128), argsr, 0, st);
    }
    if (e == cudaSuccess) {
        e = cudaLaunchKernel(fstep, grid, block, args2, 0, st);
    }
    if (e == cudaSuccess && is2d) {
        e = cudaLaunchKernel((void*)k_reduce_grid, dim3((unsigned)grid_reduce_ctas(s.N)), dim3(256), argsr, 0, st);
    }
    return e;
}

#define GR(expr)                                                                                       \
    do {                                                                                               \
        cudaError_t e_ = (expr);                                                                       \
        if (e_ != cudaSuccess) {                                                                       \
            cudaGraphDestroy(g);                                                                       \
            return e_;                                                                                 \
        }                                                                                              \
    } while (0)

/*
 * The run graph: WHILE(h_while) { step pass 1, or the resident run kernel's many steps (rg) ; IF(h_if) { regenerate
 * windows ; redo pending CTAs or strips } ; [grid by tiles: reduce + finalise] }.  `s` is updated with the two
 * conditional handles (kernel arguments).
 */
cudaError_t build_run_graph(DevSys& s, const LineGeom& g0, const RunGeom& rg, cudaGraphExec_t* exec, int mode)
{
    cudaGraph_t g;
    cudaError_t e = cudaGraphCreate(&g, 0);
    if (e != cudaSuccess) {
        return e;
    }
    cudaGraphConditionalHandle hw, hi;
    GR(cudaGraphConditionalHandleCreate(&hw, g, 1, cudaGraphCondAssignDefault));
    cudaGraphNode_t wnode;
    cudaGraph_t body;
    GR(add_conditional(&wnode, g, nullptr, 0, hw, cudaGraphCondTypeWhile, &body));
    GR(cudaGraphConditionalHandleCreate(&hi, body, 0, cudaGraphCondAssignDefault));
    s.h_while = hw;
    s.h_if = hi;
    s.in_graph = 1;

    const bool is2d = inter_grid(s.inter) && !rg.ctas; /* tiles of the grid, else strips of the flat index */
    dim3 grid, block;
    if (is2d) {
        grid = dim3((unsigned)((s.cols + 31) / 32), (unsigned)((s.rows + grid_tile_rows(s) - 1) / grid_tile_rows(s)));
        block = dim3(32, 8);
    }
    else {
        grid = dim3((unsigned)g0.grid);
        block = dim3((unsigned)g0.threads);
    }
    void* fstep = rg.ctas ? redo_kernel(s, g0) : step_kernel(s, g0);
    int pass1 = 0, pass2 = 1;
    void* args1[] = {(void*)&s, (void*)&pass1};
    void* args2[] = {(void*)&s, (void*)&pass2};
    void* argsr[] = {(void*)&s};
    cudaGraphNode_t nstep, nif;
    if (s.f_th && !rg.ctas) {
        /* updated_inc of the step: thermal draws before the step's forces */
        cudaGraphNode_t ndraw;
        GR(add_thermal_step(&ndraw, body, s));
        GR(add_kernel(&nstep, body, &ndraw, 1, fstep, grid, block, args1));
    }
    else if (s.inter == INTER_LONGRANGE1D) {
        /* all new positions before the all-pairs interaction */
        cudaGraphNode_t npos;
        GR(add_kernel(&npos, body, nullptr, 0, (void*)k_lr_position, dim3((unsigned)((s.N + 255) / 256)), dim3(256),
                      argsr));
        GR(add_kernel(&nstep, body, &npos, 1, fstep, grid, block, args1));
    }
    else if (rg.ctas) {
        /* many steps per launch; its CTAs wait on one another, so all of them must be resident */
        void* argsl[] = {(void*)&s, (void*)&rg};
        cudaKernelNodeParams kp = {};
        kp.func = const_cast<void*>(run_kernel(s, mode));
        kp.gridDim = dim3((unsigned)rg.ctas);
        kp.blockDim = dim3((unsigned)rg.threads);
        kp.sharedMemBytes = (unsigned)rg.smem;
        /* the limit is the kernel's, not this graph's: the same for every handle (another thread may be building one) */
        GR(cudaFuncSetAttribute(kp.func, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)rg.smem_max));
        kp.kernelParams = argsl;
        cudaGraphNode_t nplan;
        if (s.f_th) {
            /* the thermal draws of the launch's steps ahead of it */
            GR(add_thermal_plan(&nplan, body, s, s.th_K));
        }
        GR(cudaGraphAddKernelNode(&nstep, body, s.f_th ? &nplan : nullptr, s.f_th ? 1 : 0, &kp));
        cudaKernelNodeAttrValue coop = {};
        coop.cooperative = 1;
        GR(cudaGraphKernelNodeSetAttribute(nstep, cudaLaunchAttributeCooperative, &coop));
        if (s.f_th) {
            GR(add_thermal_commit(&nstep, body, &nstep, s));
        }
    }
    else {
        GR(add_kernel(&nstep, body, nullptr, 0, fstep, grid, block, args1));
    }
    cudaGraph_t ifbody;
    GR(add_conditional(&nif, body, &nstep, 1, hi, cudaGraphCondTypeIf, &ifbody));
    cudaGraphNode_t nregen, nredo;
    GR(add_kernel(&nregen, ifbody, nullptr, 0, (void*)k_regen, dim3(4 * 152), dim3(128), argsr));
    GR(add_kernel(&nredo, ifbody, &nregen, 1, fstep, grid, block, args2));
    if (is2d) {
        cudaGraphNode_t nred;
        GR(add_kernel(&nred, body, &nif, 1, (void*)k_reduce_grid, dim3((unsigned)grid_reduce_ctas(s.N)), dim3(256),
                      argsr));
    }
    e = cudaGraphInstantiate(exec, g, 0);
    cudaGraphDestroy(g);
    return e;
}

/*
 * The no-passing minimiser's graph: WHILE(h_while) { k_nopass_update ; k_nopass_force }.  Launched in the shape of
 * line_geometry, not in the run kernel's strips: each CTA takes a ticket and the last one sums all of their partials,
 * so CTAs of one warp are dear (N = 131072, us a sweep: strips of 32 58.2, CTAs of 256 threads 36.2).
 */
cudaError_t build_nopass_graph(const DevSys& s0, const LineGeom& g0, const NopassArgs& A, cudaGraphExec_t* exec)
{
    DevSys s = s0;
    cudaGraph_t g;
    cudaError_t e = cudaGraphCreate(&g, 0);
    if (e != cudaSuccess) {
        return e;
    }
    cudaGraphConditionalHandle hw;
    GR(cudaGraphConditionalHandleCreate(&hw, g, 1, cudaGraphCondAssignDefault));
    cudaGraphNode_t wnode;
    cudaGraph_t body;
    GR(add_conditional(&wnode, g, nullptr, 0, hw, cudaGraphCondTypeWhile, &body));
    s.h_while = hw;
    s.h_if = 0;
    s.in_graph = 1;
    NopassArgs a = A;
    void* args[] = {(void*)&s, (void*)&a};
    cudaGraphNode_t nup, nforce;
    GR(add_kernel(&nup, body, nullptr, 0, (void*)k_nopass_update, dim3((unsigned)g0.grid), dim3((unsigned)g0.threads),
                  args));
    GR(add_kernel(&nforce, body, &nup, 1, (void*)k_nopass_force, dim3((unsigned)g0.grid), dim3((unsigned)g0.threads),
                  args));
    e = cudaGraphInstantiate(exec, g, 0);
    cudaGraphDestroy(g);
    return e;
}

} // namespace fqsb
