/*
 * Internal host-side interface between the C-ABI layer (fqsb_capi.cu) and the
 * kernel translation units.  Not installed; the public ABI is include/fqsb.h.
 */
#ifndef FQSB_INTERNAL_H
#define FQSB_INTERNAL_H

#include <nvtx3/nvToolsExt.h>
#include <cuda_runtime.h>

#include <string>

#include "fqsb_device.cuh"

namespace fqsb {

/* Launch geometry of the 1d step kernel: threads per CTA and particles per thread. */
struct LineGeom {
    int threads;
    int ppt;
    int64_t grid;
};

LineGeom line_geometry(int64_t N);
/* The step kernel's launch shape beside the resident run kernel: one CTA per strip. */
LineGeom strip_geometry(int64_t N, int S);

/* Message returned by fqsb_last_error(NULL) (errors of calls that have no handle). */
void set_global_error(const std::string& msg);

/* Per-particle canonical reduction of the step's residual terms (used by the 2d path). */
int64_t grid_reduce_ctas(int64_t N);

/* Number of CTAs of the step kernel (size of DevSys::cta_pending and DevSys::partials). */
int64_t step_ctas(const DevSys& s, const LineGeom& g);

/* The run graph: a device-side WHILE loop over fused steps, with the chunk-regeneration branch.
 * Writes the conditional handles into s (they are kernel arguments of the graph's nodes). */
/* Run-kernel instantiations: the general one, and two specialised ones -- runs without activity, residual,
 * frame-force sums or recording (timeSteps / flowSteps), and runs with the residual only (minimise) -- with
 * the other code compiled out.  KMODE_ONE: runs of one step on a grid, by tiles (k_step_grid2): the run kernel's pass
 * for the first positions is not worth one step (N = 4194304, a call of timeStep: 192 us by tiles, 334 us with the first
 * step's positions recomputed where they are read).  And of thermal systems, whose plan and commit are not (N = 1000, a
 * call of timeStep: 72 us in the one-cluster kernel, 66 us so). */
enum : int { KMODE_GENERAL = 0, KMODE_PLAIN = 1, KMODE_RESID = 2, KMODE_ONE = 3 };
struct RunGeom;
cudaError_t build_run_graph(DevSys& s, const LineGeom& g, const RunGeom& rg, cudaGraphExec_t* exec,
                            int mode = KMODE_GENERAL);

/* Resident run kernel of Line1d / Particles / Laplace2d systems (fqsb_run.cu): many steps in one cooperative launch. */
static const int64_t RUN_NODES_MAX = 1216; /* 8 per SM: the control CTA sums them in one pass */
struct RunGeom {
    int S;               /* particles per strip: 32 .. 256, a power of two */
    int threads, ctas;   /* launch shape (the last CTA is the control CTA); ctas = 0: not available */
    int64_t nstrips, node_strips, nnodes;
    size_t smem, smem_max; /* shared memory of a CTA; that of the longest strips */
};
RunGeom run_geometry(const DevSys& s);
const void* run_kernel(const DevSys& s, int mode);

/* Small Line1d / Particles systems: a whole run in one launch of one thread-block cluster. */
static const int SMALL_MAX_CTAS = 16;   /* cluster size limit (above 8 needs the non-portable opt-in) */
static const int SMALL_RING_MAX = 1024; /* StopList windows up to this length stay in shared memory */
/* small systems keep a next-window buffer (N x nchunk doubles) up to this many values */
static const int64_t NX_MAX_VALUES = (int64_t)1 << 25;
static const int SMALL_THREADS_MAX = 256; /* particle threads per CTA (each CTA adds one control warp) */
struct SmallGeom {
    int threads; /* per CTA, power of two in [32, 256] */
    int ctas;    /* CTAs of the cluster */
    bool ok;     /* N fits and gains from it */
};
SmallGeom small_geometry(int64_t N, int pot, int max_ctas);
cudaError_t launch_small_run(const DevSys& s, const SmallGeom& g, cudaStream_t st);
/* refreshes the next-window buffers of a small system (no-op when it has none) */
cudaError_t launch_next_window(const DevSys& s, cudaStream_t st);
/* Whether a cluster of g.ctas CTAs of this kernel can be co-scheduled (sizes above 8 are opt-in). */
bool small_cluster_fits(const DevSys& s, const SmallGeom& g);

/* Arguments of the no-passing minimiser's kernels (the force arrays are the handle's stored forces). */
struct NopassArgs {
    double *f_pot, *f_int, *f_frame, *f;
    double den; /* (2 k + k_frame) + mu */
    int ppt;    /* particles per thread (the step's launch shape, for the canonical residual tree) */
};
static const int NOPASS_MAX_REALIGN = 1 << 20; /* bound on one particle's well updates in one sweep */
cudaError_t build_nopass_graph(const DevSys& s, const LineGeom& g, const NopassArgs& A, cudaGraphExec_t* exec);
cudaError_t launch_nopass_iteration(const DevSys& s, const LineGeom& g, const NopassArgs& A, cudaStream_t st);

/*
 * RandomNormalForcing (fqsb_thermal.cu).  A plan holds the draws of the next K steps of a run; it changes nothing of
 * the system's state.  Committing the steps of it that a launch has taken (Ctl::th_commit) updates f_thermal, the next
 * increments and the stream.  The draws of one step, or at an increment, do that at once.
 */
enum : int { TH_AT_INC = 0, TH_FROM_RUN = 1 };
static const int64_t TH_STEPS_MAX = 256;
static const int64_t TH_RUN_STEPS = 8; /* fewer planned steps are not worth a launch of the run kernel */
/* blocks of 256 words of the mask: the plan counts and lists the draws of each in each step */
__host__ __device__ inline int64_t th_blocks(int64_t words)
{
    return (words + 255) / 256;
}
cudaError_t launch_thermal_plan(const DevSys& s, int64_t K, cudaStream_t st);
cudaError_t launch_thermal_commit(const DevSys& s, cudaStream_t st);
cudaError_t launch_thermal_step(const DevSys& s, cudaStream_t st);
cudaError_t launch_thermal_draw(const DevSys& s, int64_t inc, cudaStream_t st);
/* the same as nodes of a graph: plan and step first in `body` (the last node in *node), the commit after *dep */
cudaError_t add_thermal_plan(cudaGraphNode_t* node, cudaGraph_t body, const DevSys& s, int64_t K);
cudaError_t add_thermal_step(cudaGraphNode_t* node, cudaGraph_t body, const DevSys& s);
cudaError_t add_thermal_commit(cudaGraphNode_t* node, cudaGraph_t body, const cudaGraphNode_t* dep, const DevSys& s);

/* One loop iteration launched kernel by kernel by the host (s.in_graph must be 0). */
cudaError_t launch_iteration(const DevSys& s, const LineGeom& g, cudaStream_t st);

/* NVTX range over one C-ABI call: each stepping / construction call shows as a named range on a
 * profiler timeline (header-only NVTX 3; a no-op unless a tool is attached). */
struct ApiRange {
    explicit ApiRange(const char* name)
    {
        nvtxRangePushA(name);
    }
    ~ApiRange()
    {
        nvtxRangePop();
    }
    ApiRange(const ApiRange&) = delete;
    ApiRange& operator=(const ApiRange&) = delete;
};
#define FQSB_API_RANGE() fqsb::ApiRange fqsb_api_range_(__func__)

/* Arguments of one backward step of the adjoint (fqsb_adjoint.cu). */
struct AdjArgs {
    const double *u_in, *v_in, *a_in; /* input state of the step */
    const double* up;                 /* output positions of the step */
    const double4_32a* w;             /* wells used by the step */
    double uf;                        /* u_frame of the step */
    double wff;                       /* dL / d f_frame[p] of the step (loss window) */
    const double *lu_out, *lv_out, *la_out;
    double *lu_in, *lv_in, *la_in;
    double4_32a* partials; /* per CTA */
    double* step_out;      /* 4 doubles: sum k_frame dL/df_frame, dL/deta, dL/dmu, dL/dk of the step */
    unsigned* ticket;
};

cudaError_t launch_adjoint_step(const DevSys& s, const AdjArgs& A, cudaStream_t st);
int64_t adjoint_ctas(int64_t N);

} // namespace fqsb

#endif
