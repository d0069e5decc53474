/*
 * RandomNormalForcing::force (detail.h:930-942), run by updated_inc at the start of every time step
 * (timeStep :1540-1544) and by refresh / set_inc: in particle order, every particle with inc >= next[p]
 * takes the next draw of one pcg32 stream, f_thermal[p] = mean + (stddev sqrt 2) erfinv(2 r - 1)
 * (r = u32 2^-32), and next[p] += dinc[p].
 *
 * Which particles draw when does not depend on the dynamics, so the draws of many steps are made ahead of
 * them (a plan): k_th_mask marks who draws in each step, k_th_count numbers the draws (step by step, in
 * particle order), k_th_list lists them, and k_th_eval computes one per thread from the stream's state
 * jumped ahead, so that the erfinv work (600 fp64 operations, one after the other) is dense and not in the
 * path of a step.  The run kernels then only read the drawn forces.  k_th_commit makes the steps that a
 * launch has taken the system's state (f_thermal, next, the stream).  A plan serves the launches of a run until it
 * is used up: steps in which chunk windows move end a launch early (N = 65536, one in most steps: 266 us a step with
 * a plan for every launch, 118 us).  Per time step of 1000 particles, each redrawn every 100 steps: 46.4 us with the draws
 * of each step made before it (four launches in the run graph's loop), 3.1 us planned for 256 steps and
 * taken by the one-cluster kernel.
 */
#include "fqsb_stepcore.cuh"

namespace fqsb {

/* The increment of the plan's first step, and in K its steps (no more than the run has left); false when the
 * run is over or takes no time steps, or the plan that it has is not used up.  Every thread reads the control block, so by plain loads that the first-level
 * cache serves (volatile ones all go to one line of the second: 2^22 particles, k_th_mask 18 us and 202 us,
 * k_th_commit 23 us and 103 us). */
__device__ __forceinline__ bool th_first_inc(const DevSys& s, int from, int64_t inc_arg, int64_t& inc, int& K)
{
    if (from == TH_AT_INC) {
        inc = inc_arg;
        return true;
    }
    const Ctl* c = s.ctl;
    if (c->done || c->error || (c->flags & RF_NOINC) || c->th_used != 0) {
        return false;
    }
    inc = c->inc + 1;
    const int64_t left = c->max_steps - c->step;
    K = left < K ? (int)left : K;
    return true;
}

__global__ void __launch_bounds__(256) k_th_mask(const __grid_constant__ DevSys s, int K, int from, int64_t inc_arg)
{
    int64_t inc;
    if (!th_first_inc(s, from, inc_arg, inc, K)) {
        return;
    }
    const int64_t p = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    int64_t next = 0, dinc = 0;
    if (p < s.N) {
        next = s.th_next[p];
        dinc = s.th_dinc[p];
    }
    for (int k = 0; k < K; ++k) {
        const bool draw = p < s.N && inc + k >= next;
        next += draw ? dinc : 0;
        const unsigned word = __ballot_sync(0xffffffffu, draw);
        if ((threadIdx.x & 31) == 0 && p < s.N) {
            s.th_mask[(int64_t)k * s.th_words + (p >> 5)] = word;
        }
    }
}

/* Exclusive prefix of x over the CTA's threads (whole warps); *total gets the CTA's sum.  sh: a word per warp. */
__device__ __forceinline__ int64_t cta_exclusive_scan(int64_t x, int64_t* sh, int64_t* total)
{
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, warps = blockDim.x >> 5;
    int64_t incl = x;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        int64_t y = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o) {
            incl += y;
        }
    }
    if (lane == 31) {
        sh[warp] = incl;
    }
    __syncthreads();
    int64_t before = 0, all = 0;
    for (int w = 0; w < warps; ++w) {
        int64_t t = sh[w];
        before += w < warp ? t : 0;
        all += t;
    }
    __syncthreads();
    *total = all;
    return before + incl - x;
}

/*
 * The CTA (b, k) counts the draws of 8192 particles (256 words of the mask) in planned step k; the last one turns
 * the counts into the draws before each of them.  (One CTA per step, whatever the size, left the GPU idle in plans
 * of few steps over many particles: a step of 2^22 particles took 300 us longer.)
 */
__global__ void __launch_bounds__(256) k_th_count(const __grid_constant__ DevSys s, int K, int from, int64_t inc_arg)
{
    __shared__ int64_t sh8[8];
    __shared__ int sh_last;
    int64_t inc;
    if (!th_first_inc(s, from, inc_arg, inc, K)) {
        return;
    }
    const int64_t B = gridDim.x, w = (int64_t)blockIdx.x * 256 + threadIdx.x;
    int64_t n = 0, total;
    if ((int)blockIdx.y < K && w < s.th_words) {
        n = __popc(s.th_mask[(int64_t)blockIdx.y * s.th_words + w]);
    }
    cta_exclusive_scan(n, sh8, &total);
    if (threadIdx.x == 0) {
        s.th_cnt[blockIdx.y * B + blockIdx.x] = total;
        __threadfence();
        sh_last = atomicAdd(&s.th->ticket, 1u) == gridDim.x * gridDim.y - 1u ? 1 : 0;
    }
    __syncthreads();
    if (!sh_last) {
        return;
    }
    __threadfence();
    /* consecutive counts to each thread */
    const int64_t M = (int64_t)K * B, per = (M + 255) / 256, i0 = threadIdx.x * per, i1 = i0 + per < M ? i0 + per : M;
    int64_t x = 0;
    for (int64_t i = i0; i < i1; ++i) {
        x += __ldcg(s.th_cnt + i);
    }
    int64_t before = cta_exclusive_scan(x, sh8, &total);
    for (int64_t i = i0; i < i1; ++i) {
        s.th_cum[i] = before;
        before += __ldcg(s.th_cnt + i);
        s.th_cnt[i] = 0;
    }
    if (threadIdx.x == 0) {
        s.th_cum[M] = total;
        s.th->total = total;
        s.th->ticket = 0u;
        s.th->base = s.th->state;
    }
}

/*
 * One step, whose draws k_th_eval makes the system's state: marked, counted by blocks and numbered in one kernel (the
 * last CTA to finish; the stream moves on).
 */
__global__ void __launch_bounds__(1024) k_th_one(const __grid_constant__ DevSys s, int from, int64_t inc_arg)
{
    __shared__ int64_t sh[32];
    __shared__ int sh_last;
    int64_t inc;
    int K = 1;
    if (!th_first_inc(s, from, inc_arg, inc, K)) {
        return;
    }
    const int64_t T = blockDim.x, B = th_blocks(s.th_words), p = (int64_t)blockIdx.x * T + threadIdx.x;
    const bool draw = p < s.N && inc >= s.th_next[p];
    const unsigned word = __ballot_sync(0xffffffffu, draw);
    if ((threadIdx.x & 31) == 0 && p < s.N) {
        s.th_mask[p >> 5] = word;
    }
    const int n = __syncthreads_count(draw);
    if (threadIdx.x == 0) {
        if (n) {
            atomicAdd((unsigned long long*)s.th_cnt + (p >> 13), (unsigned long long)n);
            __threadfence();
        }
        sh_last = atomicAdd(&s.th->ticket, 1u) == gridDim.x - 1u ? 1 : 0;
    }
    __syncthreads();
    if (!sh_last) {
        return;
    }
    __threadfence();
    const int64_t per = (B + T - 1) / T, i0 = threadIdx.x * per, i1 = i0 + per < B ? i0 + per : B;
    int64_t x = 0, total;
    for (int64_t i = i0; i < i1; ++i) {
        x += __ldcg(s.th_cnt + i);
    }
    int64_t before = cta_exclusive_scan(x, sh, &total);
    for (int64_t i = i0; i < i1; ++i) {
        s.th_cum[i] = before;
        before += __ldcg(s.th_cnt + i);
        s.th_cnt[i] = 0;
    }
    if (threadIdx.x == 0) {
        Thermal* th = s.th;
        th->total = total;
        th->ticket = 0u;
        th->base = th->state;
        th->state = pcg_advance_inc(th->state, (uint64_t)total, th->inc);
    }
}

/* The CTA (b, k) lists the draws of its 8192 particles in planned step k in particle order. */
__global__ void __launch_bounds__(256) k_th_list(const __grid_constant__ DevSys s, int K, int from, int64_t inc_arg)
{
    __shared__ int64_t sh8[8];
    int64_t inc;
    if (!th_first_inc(s, from, inc_arg, inc, K)) {
        return;
    }
    if ((int)blockIdx.y >= K) {
        return;
    }
    const int64_t w = (int64_t)blockIdx.x * 256 + threadIdx.x;
    uint32_t word = w < s.th_words ? s.th_mask[(int64_t)blockIdx.y * s.th_words + w] : 0u;
    int64_t total;
    int64_t k = cta_exclusive_scan(__popc(word), sh8, &total);
    k += s.th_cum[(int64_t)blockIdx.y * gridDim.x + blockIdx.x];
    for (; word; word &= word - 1u) {
        s.th_list[k++] = (int64_t)blockIdx.y * s.N + 32 * w + (__ffs((int)word) - 1);
    }
}

/* One thread per draw: entry k of the list takes output k of the stream.  now: the draws are the system's state. */
__global__ void __launch_bounds__(128) k_th_eval(const __grid_constant__ DevSys s, int from, int64_t inc_arg, int now)
{
    int64_t inc;
    int K = 0;
    if (!th_first_inc(s, from, inc_arg, inc, K)) {
        return;
    }
    const int64_t total = s.th->total;
    const uint64_t base = s.th->base, sinc = s.th->inc;
    for (int64_t k = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; k < total; k += (int64_t)gridDim.x * blockDim.x) {
        const uint32_t u32 = pcg_output(pcg_advance_inc(base, (uint64_t)k, sinc));
        const double r = FQ_MUL((double)u32, 0x1p-32);
        const double z = fq_erfinv(FQ_SUB(FQ_MUL(2.0, r), 1.0));
        const double f = FQ_ADD(s.th_mean, FQ_MUL(s.th_sc, z));
        const int64_t e = s.th_list[k]; /* now: of step 0, the particle */
        if (now) {
            s.f_th[e] = f;
            s.th_next[e] += s.th_dinc[e];
        }
        else {
            s.th_val[e] = f;
        }
    }
}

__global__ void __launch_bounds__(256) k_th_commit(const __grid_constant__ DevSys s)
{
    const int64_t from = s.ctl->th_from, steps = s.ctl->th_commit;
    const int64_t p = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (p < s.N) {
        int64_t draws = 0, last = -1;
        for (int64_t k = from; k < from + steps; ++k) {
            if (s.th_mask[k * s.th_words + (p >> 5)] >> (p & 31) & 1u) {
                ++draws;
                last = k;
            }
        }
        if (draws) {
            s.f_th[p] = s.th_val[last * s.N + p];
            s.th_next[p] += draws * s.th_dinc[p];
        }
    }
    if (p == 0 && steps > 0) {
        Thermal* th = s.th;
        const int64_t B = th_blocks(s.th_words);
        th->state = pcg_advance_inc(th->state, (uint64_t)(s.th_cum[(from + steps) * B] - s.th_cum[from * B]), th->inc);
    }
}

/* CTAs of k_th_eval (72 registers, 128 threads): 4 per SM, 78 k draws per pass, grid-stride beyond */
constexpr unsigned TH_EVAL_CTAS = 4 * 152;

struct ThLaunch {
    void* f;
    dim3 grid, block;
    void** args;
};

template <class F>
static cudaError_t for_plan(const DevSys& s, int64_t K, int from, int64_t inc, int now, F launch)
{
    int k = (int)K;
    void* args[] = {(void*)&s, (void*)&k, (void*)&from, (void*)&inc};
    void* args_one[] = {(void*)&s, (void*)&from, (void*)&inc};
    void* args_eval[] = {(void*)&s, (void*)&from, (void*)&inc, (void*)&now};
    /* one step: few CTAs where their tickets would count */
    const unsigned T = now && s.N > (1 << 18) ? 1024u : 256u;
    const dim3 parts((unsigned)((s.N + T - 1) / T)), blocks((unsigned)th_blocks(s.th_words), (unsigned)K);
    const ThLaunch list = {(void*)k_th_list, blocks, dim3(256), args};
    const ThLaunch eval = {(void*)k_th_eval, dim3(TH_EVAL_CTAS), dim3(128), args_eval};
    const ThLaunch step[] = {{(void*)k_th_one, parts, dim3(T), args_one}, list, eval};
    const ThLaunch plan[] = {{(void*)k_th_mask, parts, dim3(T), args}, {(void*)k_th_count, blocks, dim3(256), args}, list, eval};
    const ThLaunch *l = now ? step : plan, *end = now ? step + 3 : plan + 4;
    for (; l != end; ++l) {
        const cudaError_t e = launch(*l);
        if (e != cudaSuccess) {
            return e;
        }
    }
    return cudaSuccess;
}

static cudaError_t launch_plan(const DevSys& s, int64_t K, int from, int64_t inc, int now, cudaStream_t st)
{
    return for_plan(s, K, from, inc, now,
                    [&](const ThLaunch& l) { return cudaLaunchKernel(l.f, l.grid, l.block, l.args, 0, st); });
}

cudaError_t launch_thermal_plan(const DevSys& s, int64_t K, cudaStream_t st)
{
    return launch_plan(s, K, TH_FROM_RUN, 0, 0, st);
}

cudaError_t launch_thermal_step(const DevSys& s, cudaStream_t st)
{
    return launch_plan(s, 1, TH_FROM_RUN, 0, 1, st);
}

cudaError_t launch_thermal_draw(const DevSys& s, int64_t inc, cudaStream_t st)
{
    return launch_plan(s, 1, TH_AT_INC, inc, 1, st);
}

cudaError_t launch_thermal_commit(const DevSys& s, cudaStream_t st)
{
    k_th_commit<<<(unsigned)((s.N + 255) / 256), 256, 0, st>>>(s);
    return cudaGetLastError();
}

static cudaError_t add_node(cudaGraphNode_t* node, cudaGraph_t body, const cudaGraphNode_t* dep, const ThLaunch& l)
{
    cudaKernelNodeParams kp = {};
    kp.func = l.f;
    kp.gridDim = l.grid;
    kp.blockDim = l.block;
    kp.kernelParams = l.args;
    cudaGraphNode_t n;
    const cudaError_t e = cudaGraphAddKernelNode(&n, body, dep, dep ? 1 : 0, &kp);
    *node = n;
    return e;
}

static cudaError_t add_plan(cudaGraphNode_t* node, cudaGraph_t body, const DevSys& s, int64_t K, int now)
{
    bool first = true;
    return for_plan(s, K, TH_FROM_RUN, 0, now, [&](const ThLaunch& l) {
        const cudaError_t e = add_node(node, body, first ? nullptr : node, l);
        first = false;
        return e;
    });
}

cudaError_t add_thermal_plan(cudaGraphNode_t* node, cudaGraph_t body, const DevSys& s, int64_t K)
{
    return add_plan(node, body, s, K, 0);
}

cudaError_t add_thermal_step(cudaGraphNode_t* node, cudaGraph_t body, const DevSys& s)
{
    return add_plan(node, body, s, 1, 1);
}

cudaError_t add_thermal_commit(cudaGraphNode_t* node, cudaGraph_t body, const cudaGraphNode_t* dep, const DevSys& s)
{
    void* args[] = {(void*)&s};
    return add_node(node, body, dep, {(void*)k_th_commit, dim3((unsigned)((s.N + 255) / 256)), dim3(256), args});
}

} // namespace fqsb
