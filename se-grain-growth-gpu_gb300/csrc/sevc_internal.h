/*
 * Internal launch interface between the engine (sevc_engine.cu) and the
 * kernel translation units.  Every launcher enqueues on `s` and returns
 * without synchronising.
 */
#ifndef SEVC_INTERNAL_H
#define SEVC_INTERNAL_H

#include "sevc.h"
#include "sevc_device.cuh"
#include <curand_kernel.h>

/* Scratch shared by launches of one handle.  Arrays marked "per instance"
 * hold one block for each instance of a batched handle. */
struct DevScratch {
    /* index lists (capacity max(nb, ng), any order) and their lengths, zero
     * between steps: flip candidates; qualifying boundaries of the 2x3 loop;
     * failed threads of a polling iteration, then 3-sided candidates */
    int *list_a, *list_b, *list_c;
    int *n_a, *n_b, *n_c, *n_fail;
    int *extra;                      /* dynamic insertions of the 2x3 pass, EXTRA_CAP per instance */
    /* polling predicate, see poll_fail (zero between iterations): one flag
     * per grid thread, failed threads per grid block, failed blocks, all per
     * instance */
    int *threadfail, *pblock, *pcnt;
    int *piters;                     /* polling iterations this step, per instance */
    int *nrun;                       /* violations counted by check_data */
    int *segcnt;                     /* 2x3 count of each pass (20), per instance */
    double *block_area;              /* nucleated-area partial per block, per instance */
    int *counters;                   /* CTR_COUNT device counters per instance, see CTR_* */
    curandState *rng, *rng_saved;    /* 8192 cuRAND states + pre-attempt copy, per instance */
    int *nucl_buf;                   /* 96 ints per instance: per-block pick, alive count, pick's rank */
    int *nucl_on;                    /* per instance: attempt a nucleation this step */
    void *reserved;                  /* pieces of the block no kernel uses: they keep its layout (checkpoint files) */
    int *flags;                      /* 4 ints: the step's output decision, see launch_two_three_first */
    int *summary;                    /* the step's summary packed for one readback */
    int *three, *n_three;            /* the enabled 3-sided grains, listed by the grain pass (any order) */
    unsigned long long *digest;      /* SEVC_DIGEST_FIELDS sums of sevc_state_digest */
    /* events applied in parallel (removals, flips): reservation keys of
     * every vertex and boundary, the deferred events (also the grains a 2x3
     * pass left with three sides) */
    unsigned long long *vown, *bown;
    int *ehits, *n_ehits;
};
/* The reference's launch grid (n_blocks x n_threads), whose partition the
 * polling predicate shows: thread t of a block enters the block's result
 * through the shared-memory tree of topological.h:526-537, which halves its
 * width (rounding down) each round, so for a width that is not a power of
 * two some threads never do (counts). */
struct PollGrid {
    int blocks, tpb;
    int counting;      /* threads of a block that enter its result */
    __host__ __device__ int threads() const { return blocks * tpb; }
    __host__ __device__ static bool counts(int t, int w)
    {
        while (w > 1) {
            int h = w / 2;
            if (t >= 2 * h) return false;
            if (t >= h) t -= h;
            w = h;
        }
        return true;
    }
};
constexpr int EXTRA_CAP = 1024;
constexpr int TWO_THREE_PASSES = 20;  /* src/main.cu:227 */
constexpr int RNG_GRID = 8192;        /* the reference's 32 x 256 nucleation grid */

enum {
    CTR_NGRAINS = 0,     /* current_n_grains */
    CTR_CONVERGED = 1,   /* polling predicate result */
    CTR_FLIPS = 2,
    CTR_REMOVALS = 3,
    CTR_TWO_THREE = 4,
    CTR_NUCLEATIONS = 5,
    CTR_CANDIDATE = 6,   /* vrt_id_candidate (persists across attempts) */
    CTR_NUCL_ATTEMPT = 7,
    CTR_COUNT = 16
};
#define CTR_NUCL_AREA_SLOT 8 /* double stored at counters + 8 (two ints) */

/* launch shapes the autotuner may change (results do not depend on them);
 * the defaults are what it picked on the 1M-grain mesh */
struct LaunchShape {
    int tpb_vertex = 128;    /* threads per block of the vertex pass (meshes that vertex_lanes accepts: always 128) */
    int tpb_boundary = 128;  /* of the per-boundary passes (geometry, t_ext) */
    int wide_sides = 12;     /* 9..11: grains of this many sides or more get a warp each; 12: of 32 or more */
    int grain_occ = 6;       /* grain pass: 4 or 5: 64 grains a block; 6 or 8: 8, 16 or 32 by the mesh's size */
};

struct StepParams {
    double dt, eps, scaling, MC_k;
    int n_blocks, n_threads; /* reference launch grid, drives observable partitions */
    int ninst;               /* instances in the handle */
    double mu;               /* mobility (velocity factor); 1 in the reference */
    LaunchShape shape;
};

/* The handle's launch shapes (tpb_vertex, tpb_boundary, wide_sides,
 * grain_occ), for tests of every shape the autotuner may pick; SEVC_ERR_ARG
 * for others. */
extern "C" sevc_status sevc_set_launch_shape(sevc_handle *h, const int *shape);

/* geometry (sevc_geometry.cu) */
void launch_boundary_geometry(const DevMesh &m, double eps, double scaling, const LaunchShape &sh, cudaStream_t s);
/* grain pass: areas, moved areas, and the list of 3-sided grains */
void launch_grain_pass(const DevMesh &m, const DevScratch &x, const LaunchShape &sh, cudaStream_t s);
/* unit_gamma: every boundary energy is exactly 1 (GB_eps = 0, GB_scaling = 1) */
void launch_vertex_fd(const DevMesh &m, double mu, bool unit_gamma, const LaunchShape &sh, cudaStream_t s);
bool vertex_lanes(const DevMesh &m);   /* whether it takes six lanes per vertex */
void launch_grain_dadt(const DevMesh &m, const DevScratch &x, cudaStream_t s);
/* also lists the candidates and starts the polling's first comparison */
void launch_text_label(const DevMesh &m, const DevScratch &x, const StepParams &p, cudaStream_t s);
void launch_counts(const DevMesh &m, const DevScratch &x, const StepParams &p, cudaStream_t s);
/* the host's part of the output decision, flags[1..3], into x.flags; and n
 * ints into pinned host memory, both in stream order */
cudaError_t launch_set_flags(const DevScratch &x, int full, int min_grains, int grains, cudaStream_t s);
cudaError_t launch_read_out(const int *from, int *host, int n, cudaStream_t s);
/* counters | events | error bits | polling iterations | 2x3 counts | output decision, into out */
void launch_pack_summary(const DevMesh &m, const DevScratch &x, int *out, cudaStream_t s);

/* topology (sevc_topology.cu) */
PollGrid poll_grid(const StepParams &p);
/* The first 2x3 count (x.list_b, from the 3-sided grains of this step's
 * grain pass), the decision x.flags[0] ([1] the host's part of it, [2]
 * min_grains, [3] current grain count), and the next step stamp of the
 * events' save-on-write (m.stamp). */
void launch_two_three_first(const DevMesh &m, const DevScratch &x, cudaStream_t s);
/* The sparse phases (k_tail): all of them, the position update, the counts
 * and the summary in one launch for meshes that tail_whole accepts; else the
 * removals and the flips, each with the edits of its list fix-up, and the
 * position update with the rest of the flips' fix-up.  dense: the events of
 * both are applied over the whole GPU (two launches more each). */
bool tail_whole(const DevMesh &m);
void launch_tail_whole(const DevMesh &m, const DevScratch &x, const StepParams &p, int cap, int *summary, cudaStream_t s);
void launch_tail_removals(const DevMesh &m, const DevScratch &x, const StepParams &p, int cap, bool dense, cudaStream_t s);
void launch_tail_flips(const DevMesh &m, const DevScratch &x, const StepParams &p, bool dense, cudaStream_t s);
void launch_update_positions(const DevMesh &m, double dt, cudaStream_t s);
void launch_fill_instance_ids(const DevMesh &m, cudaStream_t s);

/* The mesh in the layout of sevc_mesh_host, written by the device through
 * pointers it can store to.  part: EXPORT_GRAINS, EXPORT_REST or both. */
enum { EXPORT_GRAINS = 1, EXPORT_REST = 2 };
cudaError_t launch_export(const DevMesh &m, const sevc_mesh_host &o, int part, cudaStream_t s);

/* check_data on the device (sevc_check.cu): violations counted into *out */
void launch_check(const DevMesh &m, int *out, cudaStream_t s);
/* per-field digests of the state (sevc_state_digest) into out[SEVC_DIGEST_FIELDS] */
void launch_digest(const DevMesh &m, unsigned long long *out, cudaStream_t s);

/* nucleation (sevc_nucleation.cu) */
void launch_rng_init(curandState *st, int n, cudaStream_t s);
void launch_nucleation(const DevMesh &m, const DevScratch &x, const StepParams &p, cudaStream_t s);
int rng_record(int nstreams, int ndraws, double *host_out);

/* adjoint (sevc_adjoint.cu) */
struct AdjointBuffers {
    double2 *lam;    /* adjoint of the positions (current step boundary) */
    double2 *lx, *lv;/* adjoint of the post-event positions / of the velocities */
    double *gse;     /* dL/dSE per grain (accumulated) */
    double *gmu;     /* dL/dmu per vertex (accumulated) */
    double *ggam;    /* dL/dGB_scaling per vertex (accumulated) */
    double *dlda;    /* dL/dA per grain of the statistic */
    double *scalars; /* reduced dL/dmu, dL/dGB_scaling */
};
/* one step's record on the tape (pieces of one allocation, each padded to
 * 256 bytes) */
struct TapeRecord {
    double2 *pos, *vel1;
    int4 *vb, *vg;
    int2 *bv;
    int *glist, *gvlen;
    uint8_t *ven, *ven1, *ben, *gen, *gtype;
    signed char *sgn;   /* signs of the grains' areas, by launch_adjoint_signs */
};
void launch_tape_record(const DevMesh &m, const TapeRecord &r, const EventLog &log, bool start, cudaStream_t s);
void launch_tape_after(const DevMesh &m, const TapeRecord &r, cudaStream_t s);
/* the signs of `steps` records, `bytes` apart */
void launch_adjoint_signs(const DevMesh &m, const TapeRecord &first, size_t bytes, int steps, cudaStream_t s);
/* soft histogram of a_g = |A_g| sc over nbins bins of [0, amax), divided by
 * nnorm; part: stat_doubles(nbins) doubles of scratch */
size_t stat_doubles(int nbins);
cudaError_t launch_histogram(const DevMesh &m, int nbins, double amax, double sc, double nnorm, double *part,
                             double *hist, cudaStream_t s);
/* lam = d(sum_k dldh_k h_k)/dx at the current state; zero_sum: see
 * k_hist_grad_area */
void launch_hist_seed(const DevMesh &m, int nbins, double amax, double sc, double nnorm, const double *dldh,
                      double zero_sum, double *dlda, double2 *lam, cudaStream_t s);
/* one step backward: `rec` views the mesh as recorded at the step's start,
 * log / ven1 / vel1 its events and the enabled flags and velocities after
 * it; nucleation: the log may hold nucleations */
void launch_adjoint_step(const DevMesh &rec, const AdjointBuffers &a, double dt, double mu, double eps, double s_gb,
                         const EventRec *log, const int *nlog, const uint8_t *ven1, const double2 *vel1,
                         const signed char *sgn, bool nucleation, cudaStream_t s);
/* *out = the sum of a[0..n); part: stat_doubles(1) doubles of scratch */
void launch_sum_ordered(const DevMesh &m, const double *a, int n, double *part, double *out, cudaStream_t s);
/* out[0..6] = count, sum |A|, sum A^2, sum vlen, 3-sided count, min |A|, max
 * |A| over grains [lo, hi); part: stat_doubles(1) doubles of scratch */
void launch_grain_stats(const DevMesh &m, int lo, int hi, double *part, double *out, cudaStream_t s);

#define SEVC_CUDA_OK(expr) ((expr) == cudaSuccess)

/* kernels launched by this process (reported per step) */
extern long long sevc_kernel_launches;
/* counts the next launches that must go without the programmatic-
 * serialisation attribute (a kernel with two predecessors) */
extern thread_local int sevc_pdl_skip;
#define COUNT_LAUNCHES(k) (sevc_kernel_launches += (k))

/* Launch and return the launch's own status.  (cudaGetLastError after a
 * launch also returns what any earlier failed call of this thread, of this
 * library or not, left behind.) */
template <typename... P, typename... A>
inline cudaError_t launch_status(void (*k)(P...), dim3 grid, dim3 block, size_t smem, cudaStream_t s, A &&...args)
{
    COUNT_LAUNCHES(1);
    return [&](P... p) {
        void *at[] = { &p... };
        return cudaLaunchKernel(reinterpret_cast<const void *>(k), grid, block, at, smem, s);
    }(static_cast<A &&>(args)...);
}

/* Launch with programmatic dependent launch allowed: the grid may be
 * scheduled while the previous kernel of the stream drains, which hides
 * most of the launch gap between the short kernels of the step's sparse
 * half.  Every kernel launched this way calls griddep_wait() before its
 * first global memory access; that returns once the previous kernel has
 * completed and its writes are visible, so only the scheduling overlaps. */
template <typename... P, typename... A>
inline void launch_dep(void (*k)(P...), dim3 grid, dim3 block, cudaStream_t s, A &&...args)
{
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[0].val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid;
    cfg.blockDim = block;
    cfg.dynamicSmemBytes = 0;
    cfg.stream = s;
    cfg.attrs = at;
    bool plain = sevc_pdl_skip > 0;
    if (sevc_pdl_skip > 0) sevc_pdl_skip--;
    cfg.numAttrs = plain ? 0 : 1;
    COUNT_LAUNCHES(1);
    cudaLaunchKernelEx(&cfg, k, static_cast<A &&>(args)...);
}

#endif
