/*
 * Device code of the step's end that runs either inside the one-cluster
 * kernel of the sparse phases (small meshes) or as kernels of its own over
 * the whole GPU beside it (large ones): position update, counts, summary;
 * and the polling predicate's marks, which the t_ext labels start.
 */
#ifndef SEVC_TAIL_CUH
#define SEVC_TAIL_CUH

#include "sevc_internal.h"

/* Boundary b changed its candidate state in this polling iteration
 * (flips_per_block, src/topological.h:486-511): grid thread (b mod grid), b
 * counted within its instance, fails.  A block of the reference's grid
 * passes while one of its threads that enter its result has not failed;
 * x.pblock counts the failed ones, x.pcnt the blocks of an instance where
 * all have.  b is listed for poll_reset. */
__device__ __forceinline__ void poll_fail(const DevMesh &m, const DevScratch &x, const PollGrid &pg, int b)
{
    int inst = m.binst[b], t = (b - m.boff[inst]) % pg.threads();
    if (atomicExch(x.threadfail + (size_t)inst * pg.threads() + t, 1)) return;
    x.list_c[atomicAdd(x.n_fail, 1)] = b;
    if (!PollGrid::counts(t % pg.tpb, pg.tpb)) return;
    if (atomicAdd(x.pblock + (size_t)inst * pg.blocks + t / pg.tpb, 1) == pg.counting - 1) atomicAdd(x.pcnt + inst, 1);
}

/* update_vertices_positions, src/calculus.h:391-404 */
__device__ __forceinline__ void update_vertex(const DevMesh &m, int v, double dt)
{
    if (!m.ven[v]) return;
    double2 p = m.pos[v], w = m.vel[v];
    p.x += w.x * dt;
    p.y += w.y * dt;
    p.x = dmod(p.x, m.D);
    p.y = dmod(p.y, m.D);
    m.pos[v] = p;
}

/* current_n_grains (src/calculus.h:264-313): an integer count per
 * instance, added into counters[inst * CTR_COUNT + CTR_NGRAINS] (zeroed
 * before), one atomic per warp whose grains share an instance */
__device__ __forceinline__ void count_grains(const DevMesh &m, int *counters, int tid, int n)
{
    for (int g0 = tid & ~31; g0 < m.ng; g0 += n) {
        int g = g0 + (tid & 31);
        bool on = g < m.ng && m.gen[g];
        int inst = g < m.ng ? m.ginst[g] : -1, lead = __shfl_sync(0xffffffffu, inst, 0);
        unsigned all = __ballot_sync(0xffffffffu, on), other = __ballot_sync(0xffffffffu, on && inst != lead);
        if (other) {
            if (on) atomicAdd(counters + (size_t)inst * CTR_COUNT + CTR_NGRAINS, 1);
        } else if ((tid & 31) == 0 && all) {
            atomicAdd(counters + (size_t)inst * CTR_COUNT + CTR_NGRAINS, __popc(all));
        }
    }
}

/* nucl_area_per_block (src/calculus.h:322-348) on the reference's grid, so
 * that the floating-point sum order is the same: per-thread strided partial
 * sums over the instance's grain indices, then the shared-memory tree.
 * CUDA block `rank` of `nranks` (at least tpb threads each) takes the
 * reference's blocks rank, rank + nranks, ...; those of an instance that
 * never held a nucleated grain are left out (their sums are 0). */
__device__ __forceinline__ void nucl_area_blocks(const DevMesh &m, double *block_out, int nblocks, int tpb, int rank,
                                                 int nranks)
{
    __shared__ double t[256];
    for (int u = rank; u < nblocks * m.ninst; u += nranks) {
        const int inst = u / nblocks, go = m.goff[inst], nn = m.nnlist[inst];
        if (nn == 0) continue;
        const int tid = (u - inst * nblocks) * tpb + threadIdx.x, stride = nblocks * tpb;
        const int *nl = m.nlist + go;
        if ((int)threadIdx.x < tpb) {
            double a = 0.0;
            /* the thread's stride set in ascending order, restricted to the
             * slots that can be NUCLEATED (the instance's nlist part is
             * ascending) */
            for (int i = 0; i < nn; i++) {
                int g = nl[i];
                if ((g - go) % stride == tid && m.gen[g] && m.gtype[g] == GT_NUCLEATED) a += m.garea[g];
            }
            t[threadIdx.x] = a;
        }
        __syncthreads();
        for (int i = tpb / 2; i != 0; i /= 2) {
            if ((int)threadIdx.x < i) t[threadIdx.x] += t[threadIdx.x + i];
            __syncthreads();
        }
        if (threadIdx.x == 0) block_out[u] = t[0];
        __syncthreads();
    }
}
/* host loop of nucleated_fraction_area, src/calculus.h:373-377, one thread
 * per instance */
__device__ __forceinline__ void nucl_area_final(const DevMesh &m, const double *block_out, int nblocks, int *counters,
                                                int tid, int n)
{
    for (int i = tid; i < m.ninst; i += n) {
        double s = 0.0;
        if (m.nnlist[i] > 0)
            for (int b = 0; b < nblocks; b++) s += __ldcg(block_out + (size_t)i * nblocks + b);
        *reinterpret_cast<double *>(counters + (size_t)i * CTR_COUNT + CTR_NUCL_AREA_SLOT) = 100 * s / (m.D * m.D);
    }
}

/* The step's summary in one buffer, for one readback: counters, events,
 * error bits, polling iterations, 2x3 pass counts (all per instance) and
 * the output decision.  Each per-step record it packs (event counts, error
 * bits, polling iterations and convergence, 2x3 pass counts) is zeroed once
 * read, and so are the exactness marks of the grains' dA/dt and the lengths
 * of the step's lists, so the next step starts from zeros without resets of
 * its own (the reset each step would otherwise begin with: src/main.cu's
 * per-step clears of these values). */
__device__ __forceinline__ void pack_summary(const DevMesh &m, const DevScratch &x, int *out, int tid, int n)
{
    const size_t I = m.ninst, nc = I * CTR_COUNT, ne = I * EVT_COUNT, ns = I * TWO_THREE_PASSES;
    const size_t total = nc + ne + 4 + I + ns + 1;
    for (size_t i = tid; i < total; i += n) {
        size_t k = i;
        int v;
        if (k < nc) v = x.counters[k];
        else if ((k -= nc) < ne) { v = m.evt[k]; m.evt[k] = 0; }
        else if ((k -= ne) < 4) { v = m.err[k]; m.err[k] = 0; }
        else if ((k -= 4) < I) { v = x.piters[k]; x.piters[k] = 0; m.pdone[k] = 0; }
        else if ((k -= I) < ns) { v = x.segcnt[k]; x.segcnt[k] = 0; }
        else { v = x.flags[0]; *x.n_a = *x.n_b = *x.n_c = *x.n_ehits = *x.n_three = *m.nfix = *m.nmod = 0; }
        out[i] = v;
    }
    const size_t nw = (size_t)m.ng / 16;                   /* gexact as 16-byte words (256-byte aligned array) */
    for (size_t i = tid; i < nw; i += n) reinterpret_cast<uint4 *>(m.gexact)[i] = make_uint4(0, 0, 0, 0);
    for (size_t i = 16 * nw + tid; i < (size_t)m.ng; i += n) m.gexact[i] = 0;
}

#endif
