/*
 * Topological transitions of one time step (src/topological.h of the
 * reference): the polling system, conflict resolution, removal of adjacent
 * 3-sided pairs, 3-sided grain removal, T1 flips and the deferred grain-list
 * edits.
 *
 * All of it works on short lists (the candidates the t_ext labels append,
 * the 3-sided grains the grain pass lists, the grains an event queues), and
 * it is a chain of about twenty dependent phases.  One thread-block cluster
 * runs the chain: a phase boundary is the cluster's hardware barrier
 * instead of a kernel launch, and the polling and 2x3 loops are loops (see
 * k_tail).  Edits whose order is observable have the result of the
 * reference's ascending index order; the list edits (ADD -> REMOVE ->
 * REPLACE) touch only the grain being edited and run one warp per grain,
 * which gives the reference's serial result.
 */
#include "sevc_tail.cuh"

namespace {

constexpr int TPB = 256;
constexpr int WL_BLOCKS = 152;
/* the cluster of the sparse phases */
constexpr int TAIL_BLOCKS = 16, TAIL_TPB = 512, TAIL_WARPS = TAIL_TPB / 32;

/* ------------------------------------------------------------------ */
/* grain-list primitives, src/geometry.h:614-734                       */
/* ------------------------------------------------------------------ */
__device__ int glist_find(const DevMesh &m, int g, int v)          /* grain_contains_vertex :703 */
{
    /* rows are 400 bytes in a 256-byte aligned array: four entries a load */
    const int4 *L = reinterpret_cast<const int4 *>(m.glist + (size_t)SEVC_MAXV * g);
    int n = m.gvlen[g];
    for (int i = 0; i < n; i += 4) {
        int4 q = L[i / 4];
        if (q.x == v) return i;
        if (i + 1 < n && q.y == v) return i + 1;
        if (i + 2 < n && q.z == v) return i + 2;
        if (i + 3 < n && q.w == v) return i + 3;
    }
    return -1;
}
__device__ int glist_consecutive(const DevMesh &m, int g, int A, int B) /* :724 */
{
    const int *L = m.glist + (size_t)SEVC_MAXV * g;
    int n = m.gvlen[g];
    for (int i = 0; i < n; i++) {
        if (L[i] == A && L[(i + 1) % n] == B) return 1;
        if (L[i] == B && L[(i + 1) % n] == A) return 2;
    }
    return -1;
}
/* Set flags[i] (a 0/1 byte) to 1; true for the one caller that changed
 * it.  Events that run concurrently may queue the same grain. */
__device__ __forceinline__ bool claim_byte(uint8_t *flags, int i)
{
    uintptr_t a = (uintptr_t)(flags + i);
    unsigned bit = 1u << (8 * (unsigned)(a & 3));
    return !(atomicOr((unsigned *)(a & ~(uintptr_t)3), bit) & bit);
}
/* queue a grain for the fix-up pass (grain.fix = true) */
__device__ void mark_fix(const DevMesh &m, int g)
{
    if (!claim_byte(m.gfix, g)) return;
    int i = atomicAdd(m.nfix, 1);
    if (i < m.fixcap) m.fixlist[i] = g; else raise_err(m, ERRB_WORKLIST);
}
/* write a deferred edit into vertex v's mod slot (mod_t, src/geometry.h:26);
 * prev < -1 keeps the slot's previous vrt_prev_id, as the reference does
 * when it only assigns fix/vrt/grn */
__device__ void set_mod(const DevMesh &m, int v, int slot, int fix, int grn, int vrt, int prev)
{
    int4 *md = m.vmod + 4 * (size_t)v + slot;
    int4 x = *md;
    x.x = grn; x.y = vrt; if (prev >= -1) x.z = prev; x.w = fix;
    *md = x;
    if (!m.vmodmark[v]) {
        m.vmodmark[v] = 1;
        int i = atomicAdd(m.nmod, 1);
        if (i < m.modcap) m.modlist[i] = v; else raise_err(m, ERRB_WORKLIST);
    }
}

/* ------------------------------------------------------------------ */
/* the team                                                            */
/* ------------------------------------------------------------------ */
/* Every thread of the grid.  In k_tail the grid is exactly one cluster and a
 * phase ends at sync(): what any thread wrote before it, any thread reads
 * after it (release / acquire at cluster scope). */
struct Team {
    int tid, n;            /* thread of the team, threads */
    int warp, nwarps, lane;/* consecutive warps lie in different blocks: a few events spread over all SMs */
    __device__ Team()
    {
        lane = threadIdx.x & 31;
        warp = (threadIdx.x >> 5) * gridDim.x + blockIdx.x;
        tid = 32 * warp + lane;
        n = gridDim.x * blockDim.x;
        nwarps = n >> 5;
    }
    __device__ __forceinline__ void sync() const
    {
        asm volatile("barrier.cluster.arrive.release;\n\tbarrier.cluster.wait.acquire;" ::: "memory");
    }
};

/* ids[0..n) (distinct) in ascending order into out, by rank; the caller
 * syncs.  Short lists: the reference's serial order of rare events. */
__device__ void rank_sort(const Team &T, const int *ids, int n, int *out)
{
    for (int i = T.tid; i < n; i += T.n) {
        int v = ids[i], r = 0;
        for (int j = 0; j < n; j++) r += ids[j] < v;
        out[r] = v;
    }
}

/* ------------------------------------------------------------------ */
/* polling system, src/topological.h:362-578                           */
/* ------------------------------------------------------------------ */
/* What the phases up to the removals read of a listed boundary's
 * surroundings.  Polling and conflicts change flags, never the mesh, so each
 * thread loads this for its first item when the kernel starts, the three kinds
 * in different warps so that their chains of dependent loads (some 1,000
 * cycles each) run side by side, and a phase is left with the loads of the
 * flags it tests: 49,000 -> 25,000 cycles for polling and conflicts at 150
 * candidates.  Items beyond the team's size load theirs as they come. */
/* a flag of boundary b, 0 for an empty slot (phases read the slots' flags
 * before they know whether they need them) */
__device__ __forceinline__ uint8_t flag_at(const uint8_t *flags, int nb, int b)
{
    return (unsigned)b < (unsigned)nb ? flags[b] : 0;
}
struct PollItem { int b, inst, en, buf; bool vi, ve; int4 si, se; };   /* a candidate, its ends' slots */
struct ConfItem { int c, b; int4 si, se; };                    /* a candidate, a boundary beside it, its ends' slots */
struct LabelItem { int b, g; };                                /* a candidate, a 3-sided grain on it (-1: none) */
__device__ __forceinline__ PollItem poll_item(const DevMesh &m, const int *list, int i, int n)
{
    PollItem p;
    p.b = i < n ? list[i] : -1;
    p.inst = p.en = p.buf = 0;
    p.vi = p.ve = false;
    p.si = p.se = make_int4(-1, -1, -1, -1);
    if (p.b >= 0) {
        const int2 e = m.bv[p.b];
        p.inst = m.binst[p.b];
        p.en = m.ben[p.b];
        p.buf = m.bcandbuf[p.b];
        p.si = m.vb[e.x]; p.se = m.vb[e.y];
        p.vi = m.ven[e.x]; p.ve = m.ven[e.y];
    }
    return p;
}
__device__ __forceinline__ ConfItem conf_item(const DevMesh &m, const int *list, int t, int n)
{
    ConfItem f;
    f.c = f.b = -1;
    f.si = f.se = make_int4(-1, -1, -1, -1);
    if (t < 6 * n) {
        const int i = t / 6, r = t - 6 * i, c = list[i];
        const int2 e = m.bv[c];
        const int b = slot3(m.vb[r < 3 ? e.x : e.y], r < 3 ? r : r - 3);
        if (b != c && (unsigned)b < (unsigned)m.nb) {
            const int2 w = m.bv[b];
            f.c = c;
            f.b = b;
            if ((unsigned)w.x < (unsigned)m.nv) f.si = m.vb[w.x];
            if ((unsigned)w.y < (unsigned)m.nv) f.se = m.vb[w.y];
        }
    }
    return f;
}
__device__ __forceinline__ LabelItem label_item(const DevMesh &m, const int *list, int t, int n)
{
    LabelItem l;
    l.b = l.g = -1;
    if (t < 3 * n) {
        const int i = t / 3, j = t - 3 * i, b = list[i];
        const int2 e = m.bv[b];
        const int4 ga = m.vg[e.x], gb = m.vg[e.y];
        const int g = slot3(ga, j);
        const bool first = !(j > 0 && g == ga.x) && !(j > 1 && g == ga.y);
        if ((unsigned)g < (unsigned)m.ng && first && (g == gb.x || g == gb.y || g == gb.z)) {
            const int len = m.gvlen[g];
            if (m.ben[b] && m.gen[g] && len == 3) { l.b = b; l.g = g; }
        }
    }
    return l;
}

/* vertices_vote (:362) for one vertex (its slots sb; on: enabled): its
 * boundary with the smallest extinction time among the candidates (the last
 * such slot) */
__device__ __forceinline__ int vertex_vote(const DevMesh &m, int4 sb, bool on)
{
    if (!on) return -1;
    double t[3];
    uint8_t c[3];
#pragma unroll
    for (int j = 0; j < 3; j++) {
        const int b = slot3(sb, j);
        c[j] = flag_at(m.bcand, m.nb, b);
        t[j] = (unsigned)b < (unsigned)m.nb ? m.btext[b] : 0.0;
    }
    double mt = 99999999;
    int am = sb.x;
#pragma unroll
    for (int j = 0; j < 3; j++)
        if (t[j] <= mt && c[j]) { mt = t[j]; am = slot3(sb, j); }
    return am;
}

/* One polling loop (:549-578) over the candidate list.  An iteration:
 *   votes    vertices_vote and count_boundaries_votes (:406): whether both
 *            ends of a candidate vote for it
 *   unlabel  (:441) a two-vote candidate clears its neighbours.  It is never
 *            adjacent to another two-vote candidate (their shared vertex
 *            votes once), so the parallel writes change no decision.
 *   compare  write_candidate_results (:466-477) and flips_per_block
 *            (:486-511): a mismatch marks its thread of the reference's grid
 *            (poll_fail).  Only listed boundaries can mismatch here: the
 *            t_ext labels compared and wrote every other one, whose flag no
 *            iteration changes.
 *   result   compare_candidates (:526-537): an instance with no block whose
 *            threads all failed has converged and takes no further
 *            iteration this step
 * Leaves the marks to the caller (poll_reset). */
__device__ void poll_reset(const DevMesh &m, const DevScratch &x, const Team &T, const PollGrid &pg, int nfail)
{
    for (int i = T.tid; i < nfail; i += T.n) {
        int b = x.list_c[i], inst = m.binst[b], t = (b - m.boff[inst]) % pg.threads();
        x.threadfail[(size_t)inst * pg.threads() + t] = 0;
        x.pblock[(size_t)inst * pg.blocks + t / pg.tpb] = 0;
    }
    for (int i = T.tid; i < m.ninst; i += T.n) x.pcnt[i] = 0;
    if (T.tid == 0) *x.n_fail = 0;
}
__device__ int poll_loop(const DevMesh &m, const DevScratch &x, const Team &T, const PollGrid &pg, int cap, PollItem &first)
{
    const int *list = x.list_a;
    const int n = *x.n_a;
    auto item = [&](int i) { return i == T.tid ? first : poll_item(m, list, i, n); };
    for (int it = 1;; it++) {
        if (n > 0) {
            bool two = false, done = false;          /* the first item's */
            for (int i = T.tid; i < n; i += T.n) {
                const PollItem p = item(i);
                const uint8_t over = m.pdone[p.inst], c = m.bcand[p.b];
                const int vi = vertex_vote(m, p.si, p.vi), ve = vertex_vote(m, p.se, p.ve);
                if (i == T.tid) done = over;
                if (!(p.en && c) || over) continue;
                const bool v = vi == p.b && ve == p.b;
                m.bvotes[p.b] = v ? 2 : 0;
                if (i == T.tid) two = v;
            }
            T.sync();
            for (int i = T.tid; i < n; i += T.n) {
                const PollItem p = item(i);
                if (i == T.tid ? !two : !(p.en && m.bcand[p.b] && m.bvotes[p.b] == 2) || m.pdone[p.inst]) continue;
#pragma unroll
                for (int j = 0; j < 3; j++) {
                    int u = slot3(p.si, j), w = slot3(p.se, j);
                    if (u != p.b) m.bcand[u] = 0;
                    if (w != p.b) m.bcand[w] = 0;
                }
            }
            T.sync();
            for (int i = T.tid; i < n; i += T.n) {
                PollItem p = item(i);
                if (i == T.tid ? done : m.pdone[p.inst] != 0) continue;
                const uint8_t c = m.bcand[p.b];
                if (p.en && c != p.buf) poll_fail(m, x, pg, p.b);
                m.bcandbuf[p.b] = p.en ? c : 0;
                if (i == T.tid) first.buf = p.en ? c : 0;
            }
            T.sync();
        }
        /* every block forms the result for itself; block 0 records it (the
         * others see an instance it marks as done either way) */
        bool run = false;
        for (int i = threadIdx.x; i < m.ninst; i += blockDim.x) {
            const uint8_t over = m.pdone[i];
            const bool again = x.pcnt[i] != 0;
            if (over) continue;
            run |= again;
            if (blockIdx.x == 0) {
                x.piters[i]++;
                if (!again) m.pdone[i] = 1;
            }
        }
        const int nfail = *x.n_fail;
        run = __syncthreads_or(run);
        if (run && it >= cap) {
            if (T.tid == 0) atomicOr(m.err, ERRB_NONCONVERGED);
            run = false;
        }
        if (!run) return nfail;
        T.sync();
        poll_reset(m, x, T, pg, nfail);
        T.sync();
    }
}

/* ------------------------------------------------------------------ */
/* conflicts, src/topological.h:83-155                                 */
/* ------------------------------------------------------------------ */
/* check_conflictive_boundaries for every non-candidate boundary adjacent
 * to a candidate (the only ones it can mark); one thread per candidate and
 * slot of its ends, so the six neighbours' load chains run side by side
 * (every visit of a boundary writes the same winner) */
__device__ void conflict_check(const DevMesh &m, const Team &T, const int *list, int n, const ConfItem &first)
{
    const int t0 = T.n - 1 - T.tid;
    for (int t = t0; t < 6 * n; t += T.n) {
        const ConfItem f = t == t0 ? first : conf_item(m, list, t, n);
        if (f.b < 0) continue;
        const uint8_t en = m.ben[f.b], cb = m.bcand[f.b], ec = m.ben[f.c], cc = m.bcand[f.c];
        uint8_t ci[3], ce[3];
#pragma unroll
        for (int j = 0; j < 3; j++) {
            ci[j] = flag_at(m.bcand, m.nb, slot3(f.si, j));
            ce[j] = flag_at(m.bcand, m.nb, slot3(f.se, j));
        }
        if (!(ec && cc) || !(en && !cb)) continue;
        int bi = -1, be = -1;
#pragma unroll
        for (int j = 2; j >= 0; j--) {                     /* the first of each end */
            const int x = slot3(f.si, j), y = slot3(f.se, j);
            if (x != f.b && ci[j]) bi = x;
            if (y != f.b && ce[j]) be = y;
        }
        if (bi >= 0 && be >= 0) {
            double ti = m.btext[bi], te = m.btext[be];
            int w;
            if (ti == te) w = bi < be ? bi : be;
            else w = ti < te ? bi : be;
            /* b is reached from each candidate next to it and every visit
             * writes the same w; the first writer (bconf was -1) counts the
             * mark */
            if (atomicExch(&m.bconf[f.b], w) == -1) atomicAdd(&m.evt[EVT_COUNT * m.binst[f.b] + EVT_CONFLICTS], 1);
        }
    }
}
__device__ void conflict_unlabel(const DevMesh &m, const Team &T, const int *list, int n, const PollItem &first)
{
    for (int i = T.tid; i < n; i += T.n) {
        const PollItem p = i == T.tid ? first : poll_item(m, list, i, n);
        const uint8_t c = m.bcand[p.b];
        bool drop = false;
#pragma unroll
        for (int j = 0; j < 3; j++) {
            const int u = slot3(p.si, j), w = slot3(p.se, j);
            const int fu = (unsigned)u < (unsigned)m.nb ? m.bconf[u] : -1, fw = (unsigned)w < (unsigned)m.nb ? m.bconf[w] : -1;
            drop |= (u != p.b && fu != -1 && fu != p.b) || (w != p.b && fw != -1 && fw != p.b);
        }
        if (p.en && c && drop) m.bcand[p.b] = 0;
    }
}

/* ------------------------------------------------------------------ */
/* removal of two adjacent 3-sided grains, src/topological.h:840-985   */
/* ------------------------------------------------------------------ */
/* remove_two_grains (:840-955); returns the rewired boundary CE or -1 */
__device__ __noinline__ int remove_two_grains_dev(const DevMesh &m, int bnd, const int *gnic)
{
    int2 eb = m.bv[bnd];
    int A = eb.x, B = eb.y;
    int4 sa = m.vb[A], sbv = m.vb[B];
    int AC = -1, BD = -1;
    for (int i = 0; i < 3; i++) if (slot3(sa, i) == bnd) { AC = slot3(sa, (i + 1) % 3); break; }
    for (int j = 0; j < 3; j++) if (slot3(sbv, j) == bnd) { BD = slot3(sbv, (j + 1) % 3); break; }
    if (AC < 0 || BD < 0) { raise_err(m, ERRB_TOPOLOGY); return -1; }
    int C = other_end(m.bv[AC], A);
    int D = other_end(m.bv[BD], B);
    int4 sc = m.vb[C], sd = m.vb[D];
    int CE = -1, DF = -1;
    for (int k = 0; k < 3; k++) if (slot3(sc, k) == AC) { CE = slot3(sc, (k + 2) % 3); break; }
    for (int l = 0; l < 3; l++) if (slot3(sd, l) == BD) { DF = slot3(sd, (l + 2) % 3); break; }
    if (CE < 0 || DF < 0) { raise_err(m, ERRB_TOPOLOGY); return -1; }
    int F = other_end(m.bv[DF], D);
    int2 ce = m.bv[CE];
    if (ce.x == C) ce.x = F; else ce.y = F;
    save_ends(m, CE);
    m.bv[CE] = ce;
    int4 sf = m.vb[F];
    for (int p = 0; p < 3; p++) if (slot3(sf, p) == DF) { set_slot3(sf, p, CE); break; }
    m.vb[F] = sf;
    if (gnic[0] < 0 || gnic[1] < 0) { raise_err(m, ERRB_TOPOLOGY); return -1; }
    int G3, G4;
    if (glist_find(m, gnic[0], A) >= 0) { G3 = gnic[0]; G4 = gnic[1]; } else { G3 = gnic[1]; G4 = gnic[0]; }
    set_mod(m, A, 0, FIX_REMOVE, G3, A, -2); mark_fix(m, G3);
    set_mod(m, A, 1, FIX_REMOVE, G3, C, -2);
    set_mod(m, A, 2, FIX_REMOVE, G3, D, -2);
    set_mod(m, B, 0, FIX_REMOVE, G4, B, -2); mark_fix(m, G4);
    set_mod(m, B, 1, FIX_REMOVE, G4, C, -2);
    set_mod(m, B, 2, FIX_REMOVE, G4, D, -2);
    sa = m.vb[A]; sbv = m.vb[B];
    for (int i = 0; i < 3; i++) {
        m.ben[slot3(sa, i)] = 0;
        m.ben[slot3(sbv, i)] = 0;
    }
    m.ben[DF] = 0;
    m.ben[bnd] = 0;
    m.ven[A] = 0; m.ven[D] = 0; m.ven[C] = 0; m.ven[B] = 0;
    return CE;
}

__device__ bool two_three_qualifies(const DevMesh &m, int b, int *gic)
{
    if (!m.ben[b]) return false;
    int2 e = m.bv[b];
    if (gintersect(m.vg[e.x], m.vg[e.y], gic) < 2) return false;
    return m.gvlen[gic[0]] == 3 && m.gvlen[gic[1]] == 3;
}

/* Qualifying boundaries among those at the vertices of the 3-sided grains
 * a[0..na) and then b[0..): a qualifying boundary lies on two of them, so
 * testing these gives every one; each is appended once, by the smaller of its
 * two grains at its first end.  t: one (grain, vertex, slot). */
__device__ __forceinline__ void find_two_three(const DevMesh &m, const int *a, int na, const int *b, int t, int *out,
                                               int *n_out)
{
    int i = t / 9, r = t - 9 * i, k = r / 3, j = r - 3 * k, g = i < na ? a[i] : b[i - na];
    if (!m.gen[g] || m.gvlen[g] != 3) return;
    int v = m.glist[(size_t)SEVC_MAXV * g + k], e = slot3(m.vb[v], j), gic[2];
    if (m.bv[e].x != v || !two_three_qualifies(m, e, gic)) return;
    if (g == (gic[0] < gic[1] ? gic[0] : gic[1])) out[atomicAdd(n_out, 1)] = e;
}
/* The boundaries that qualify after a pass of the 2x3 loop, given that every
 * listed one was visited by it.  Whether a boundary qualifies depends on its
 * flag, its ends, the grains at these and their side counts; a pass takes
 * flags away, re-wires the boundaries ce[0..nce) and leaves the grains
 * three[0..n3) with three sides, and nothing else can make one qualify.  So
 * these are tested, each appended once: by the smaller of its grains in
 * three[], as a re-wired one if neither is (and by the first of equal
 * entries).  The search over every 3-sided grain (some 3% of all) that
 * finds the same took 81,000 cycles a pass at 73,000 grains. */
__device__ bool unsorted_contains(const int *a, int n, int x)
{
    for (int i = 0; i < n; i++)
        if (a[i] == x) return true;
    return false;
}
__device__ void find_two_three_again(const DevMesh &m, const Team &T, const int *three, int n3, const int *ce, int nce,
                                     int *out, int *n_out)
{
    for (int t = T.tid; t < 9 * n3 + nce; t += T.n) {
        int e, g = -1, gic[2];
        if (t < 9 * n3) {
            const int i = t / 9, r = t - 9 * i, k = r / 3;
            g = three[i];
            if (!m.gen[g] || m.gvlen[g] != 3) continue;
            const int v = m.glist[(size_t)SEVC_MAXV * g + k];
            e = slot3(m.vb[v], r - 3 * k);
            if (m.bv[e].x != v) continue;
        } else {
            e = ce[t - 9 * n3];
            if (e < 0 || unsorted_contains(ce, t - 9 * n3, e)) continue;
        }
        if (!two_three_qualifies(m, e, gic)) continue;
        const int lo = gic[0] < gic[1] ? gic[0] : gic[1], hi = gic[0] < gic[1] ? gic[1] : gic[0];
        const int by = unsorted_contains(three, n3, lo) ? lo : unsorted_contains(three, n3, hi) ? hi : -1;
        if (by != g || !m.gen[lo] || glist_find(m, lo, m.bv[e].x) < 0) continue;
        out[atomicAdd(n_out, 1)] = e;
    }
}
/* The step's first 2x3 count (topological.h:228), from the 3-sided grains
 * the grain pass listed.  The last block then decides whether the step
 * computes every output-only value (extinction times of all boundaries,
 * dA/dt of all grains): when it can export or is asked to (flags[1], set by
 * the host), or when it could end at the stop threshold (a final export):
 * every removal takes a 3-sided grain, and a pass of the 2x3 loop can make
 * at most two per pair; the bound is generous, as the threshold is crossed
 * once per run.  Else only what the step can observe is computed.  flags[0]
 * = the decision, taken on the device so that no host round trip separates
 * the step's first half from its second. */
__global__ void k_two_three_first(DevMesh m, DevScratch x)
{
    const int n3 = *x.n_three;
    for (int t = blockIdx.x * blockDim.x + threadIdx.x; t < 9 * n3; t += gridDim.x * blockDim.x)
        find_two_three(m, x.three, n3, nullptr, t, x.list_b, x.n_b);
    const bool last = last_block(m.lastblk + 2);
    if (last && threadIdx.x == 0) {
        __threadfence();
        int mg = x.flags[2], curr = x.flags[3];
        long long reach = (long long)curr - n3 - 40LL * __ldcg(x.n_b) - 64;
        x.flags[0] = x.flags[1] || (mg > 0 && reach <= mg);
        *m.stamp += 1;   /* a new step: every value saved by the last step's events is stale */
    }
}

__device__ bool sorted_contains(const int *a, int lo, int hi, int x)
{
    int end = hi;
    while (lo < hi) {
        int mid = (lo + hi) >> 1;
        if (a[mid] < x) lo = mid + 1; else hi = mid;
    }
    return lo < end && a[lo] == x;
}

/* remove_two_grains_configurations (:965-985) is one thread scanning every
 * boundary in index order.  Only listed boundaries (those qualifying at the
 * count) and boundaries re-wired during the scan (CE) can qualify, so the
 * scan visits exactly those, in index order, re-testing each on visit.
 * One thread per instance, each over its own part of the ascending list;
 * the grains it removes are appended to gone, two a pair, and the pair's
 * re-wired boundary is kept at its place in ce (while there is room). */
__device__ void remove_two_three(const DevMesh &m, const int *list, int n, int *extra, int *segcnt, int *gone,
                                 int *n_gone, int *ce, int ce_cap, int inst)
{
    int i = lower_bound_i(list, n, m.boff[inst]);
    int N = lower_bound_i(list, n, m.boff[inst + 1]);
    segcnt[inst] = N - i;
    extra += (size_t)inst * EXTRA_CAP;
    int *evt = m.evt + EVT_COUNT * inst;
    int ne = 0;
    while (i < N || ne > 0) {
        int b;
        if (ne > 0 && (i >= N || extra[0] < list[i])) {
            b = extra[0];
            for (int k = 1; k < ne; k++) extra[k - 1] = extra[k];
            ne--;
        } else {
            b = list[i++];
        }
        int gic[2];
        if (!two_three_qualifies(m, b, gic)) continue;
        int2 e = m.bv[b];
        int gnic[2];
        gsymdiff(m.vg[e.x], m.vg[e.y], gnic);
        int CE = remove_two_grains_dev(m, b, gnic);
        m.gen[gic[0]] = 0;
        m.gen[gic[1]] = 0;
        int o = atomicAdd(n_gone, 2);
        gone[o] = gic[0];
        gone[o + 1] = gic[1];
        if (o / 2 < ce_cap) ce[o / 2] = CE;
        evt[EVT_TWO_THREE]++;
        if (CE > b && !sorted_contains(list, i, N, CE)) {
            int g2[2];
            if (two_three_qualifies(m, CE, g2)) {
                bool dup = false;
                for (int k = 0; k < ne; k++) dup |= extra[k] == CE;
                if (!dup) {
                    if (ne >= EXTRA_CAP) { raise_err(m, ERRB_WORKLIST); continue; }
                    int k = ne++;
                    while (k > 0 && extra[k - 1] > CE) { extra[k] = extra[k - 1]; k--; }
                    extra[k] = CE;
                }
            }
        }
    }
}

/* ------------------------------------------------------------------ */
/* 3-sided grain removal, src/topological.h:614-822, :994-1004         */
/* ------------------------------------------------------------------ */
/* label_3sided_grains (:994-1004) for the 3-sided grain g: -1, or, if g is
 * to be removed, its lowest enabled boundary with 0 <= t_ext <= dt (there is
 * one: a flip candidate is such a boundary, and so are all three in the
 * reference's other case).  L, bs: its vertices and their boundaries. */
__device__ int label3_first(const DevMesh &m, int g, double dt, int (&L)[3], int (&bs)[9])
{
    /* The reference breaks out of a vertex's boundary loop once a flip
     * candidate inside the grain is found; that sets the result to 1 for
     * good, so testing every boundary gives the same answer and lets all
     * nine records load at once. */
    const int *row = m.glist + (size_t)SEVC_MAXV * g;
    L[0] = row[0]; L[1] = row[1]; L[2] = row[2];
    int4 s[3] = { m.vb[L[0]], m.vb[L[1]], m.vb[L[2]] };
    int2 e[9];
#pragma unroll
    for (int j = 0; j < 9; j++) bs[j] = slot3(s[j / 3], j % 3);
#pragma unroll
    for (int j = 0; j < 9; j++) e[j] = m.bv[bs[j]];
    bool cand = false;
    int ans = 0, low = INT_MAX;
#pragma unroll
    for (int j = 0; j < 9; j++) {
        bool ii = e[j].x == L[0] || e[j].x == L[1] || e[j].x == L[2];
        bool ee = e[j].y == L[0] || e[j].y == L[1] || e[j].y == L[2];
        if (ii && ee) {
            int b = bs[j];
            uint8_t en = m.ben[b], ca = m.bcand[b];
            double t = m.btext[b];
            cand |= ca && en;
            if (t >= 0 && t <= dt && en) {
                ans++;
                low = b < low ? b : low;
            }
        }
    }
    return cand || ans / 2 == 3 ? low : -1;
}

/* remove_grain (:687-822) */
__device__ __noinline__ void remove_grain_dev(const DevMesh &m, int grn)
{
    const int *L = m.glist + (size_t)SEVC_MAXV * grn;
    int A = L[0], B = L[1], C = L[2];
    double D = m.D;
    double2 pa = m.pos[A], pb = m.pos[B], pc = m.pos[C];
    log_event(m, EV_REMOVE, A, B, C, pa, pb, pc);
    double nAB = arclen(pa, pb, D), nBC = arclen(pb, pc, D), nCA = arclen(pc, pa, D);
    double denom = nAB + nBC + nCA;
    double x0 = 0, y0 = 0;                                      /* adjust_origin_for_points, 3 points */
    double x1 = x0 + wrapd(pb.x, pa.x, D), y1 = y0 + wrapd(pb.y, pa.y, D);
    double x2 = x1 + wrapd(pc.x, pb.x, D), y2 = y1 + wrapd(pc.y, pb.y, D);
    pa.x += (nBC * x0 + nCA * x1 + nAB * x2) / denom;
    pa.y += (nBC * y0 + nCA * y1 + nAB * y2) / denom;
    pa.x = dmod(pa.x, D);
    pa.y = dmod(pa.y, D);
    save_vertex(m, A);
    m.pos[A] = pa;
    int gbc[2], gab[2], gac[2];
    gintersect(m.vg[B], m.vg[C], gbc);
    int G3 = gbc[0] == grn ? gbc[1] : gbc[0];
    gintersect(m.vg[A], m.vg[B], gab);
    int G2 = gab[0] == grn ? gab[1] : gab[0];
    gintersect(m.vg[A], m.vg[C], gac);
    int G1 = gac[0] == grn ? gac[1] : gac[0];
    if (G1 < 0 || G2 < 0 || G3 < 0) { raise_err(m, ERRB_TOPOLOGY); return; }
    m.vel[A] = make_double2(0.0, 0.0);
    int4 sc = m.vb[C], sb = m.vb[B];
    for (int i = 0; i < 3; i++) {
        int x = slot3(sc, i);
        int2 e = m.bv[x];
        if ((e.x == B && e.y == C) || (e.y == B && e.x == C)) { m.ben[x] = 0; break; }
    }
    int BE = -1, CF = -1;
    for (int i = 0; i < 3; i++) {
        int x = slot3(sb, i);
        int2 e = m.bv[x];
        if (!(e.x == A || e.y == A) && !(e.x == C || e.y == C)) { BE = x; break; }
    }
    for (int i = 0; i < 3; i++) {
        int x = slot3(sc, i);
        int2 e = m.bv[x];
        if (!(e.x == A || e.y == A) && !(e.x == B || e.y == B)) { CF = x; break; }
    }
    if (BE < 0 || CF < 0) { raise_err(m, ERRB_TOPOLOGY); return; }
    int2 e;
    save_ends(m, BE);
    save_ends(m, CF);
    e = m.bv[BE]; if (e.x == B) e.x = A; else e.y = A; m.bv[BE] = e;
    e = m.bv[CF]; if (e.x == C) e.x = A; else e.y = A; m.bv[CF] = e;
    int4 sa = m.vb[A];
    for (int i = 0; i < 3; i++) {
        int x = slot3(sa, i);
        int2 f = m.bv[x];
        if (f.x == B || f.y == B) { m.ben[x] = 0; set_slot3(sa, i, BE); break; }
    }
    for (int i = 0; i < 3; i++) {
        int x = slot3(sa, i);
        int2 f = m.bv[x];
        if (f.x == C || f.y == C) { m.ben[x] = 0; set_slot3(sa, i, CF); break; }
    }
    m.vb[A] = sa;
    m.ven[B] = 0;
    m.ven[C] = 0;
    m.gen[grn] = 0;
    set_mod(m, B, 0, FIX_REMOVE, G2, B, -2); mark_fix(m, G2);
    set_mod(m, C, 0, FIX_REMOVE, G1, C, -2); mark_fix(m, G1);
    set_mod(m, B, 1, FIX_REMOVE, G3, B, -2); mark_fix(m, G3);
    set_mod(m, C, 1, FIX_REPLACE, G3, A, C);
    int4 ga = m.vg[A];
    for (int i = 0; i < 3; i++) if (slot3(ga, i) == grn) set_slot3(ga, i, G3);
    m.vg[A] = ga;
}

/* ------------------------------------------------------------------ */
/* Events in parallel with the serial order's result                    */
/* ------------------------------------------------------------------ */
/* The reference applies the 3-sided removals one at a time in ascending
 * grain order (remove_grains <<<1,1>>>, :994) and defines no order for the
 * flips; here both phases follow ascending index order.  An event reads and
 * writes only its footprint (its vertices and the boundaries in their
 * slots) plus grain-level records that commute: queueing a grain for the
 * fix-up (an atomic claim of its flag) and its mod slots (per vertex).  Two events with disjoint footprints therefore
 * commute, and the serial result is obtained by deterministic reservation:
 *   reserve  every event writes its key into each footprint record
 *            (atomicMin); the key orders events by grain or boundary index,
 *            the serial order (the lists themselves are in any order);
 *   apply    an event that holds every one of its records shares none
 *            with an earlier event: it runs at once, all such in parallel;
 *            any other is deferred;
 *   deferred the deferred events run one at a time in index order, after
 *            the parallel ones; each shares records only with earlier
 *            events, which have all run (in parallel or before it here),
 *            and commutes with every later parallel one.
 * Keys carry a per-phase epoch in their high half that grows every step,
 * so records never need clearing: an earlier step's key is larger and is
 * replaced by the first reservation of a later step. */
__device__ __forceinline__ unsigned long long resv_key(unsigned epoch, int id)
{
    return ((unsigned long long)(0xFFFFFFFFu - epoch) << 32) | (unsigned)id;
}
__device__ __forceinline__ bool valid_v(const DevMesh &m, int v) { return (unsigned)v < (unsigned)m.nv; }
__device__ __forceinline__ bool valid_b(const DevMesh &m, int b) { return (unsigned)b < (unsigned)m.nb; }
__device__ __forceinline__ bool valid_g(const DevMesh &m, int g) { return (unsigned)g < (unsigned)m.ng; }

/* bring a record into this SM's L1 (no register result, no wait) */
__device__ __forceinline__ void l1_touch(const void *p) { asm volatile("prefetch.global.L1 [%0];" ::"l"(p)); }
/* one thread reserves a vertex and the boundaries in its slots */
__device__ __forceinline__ void reserve_vertex(const DevMesh &m, const DevScratch &x, int v, int4 slots,
                                               unsigned long long key)
{
    atomicMin(x.vown + v, key);
#pragma unroll
    for (int k = 0; k < 3; k++) {
        int b = slot3(slots, k);
        if (valid_b(m, b)) atomicMin(x.bown + b, key);
    }
}
/* the records an event's single-thread code reads, brought into L1 by
 * the warp in two parallel rounds: the vertices' own records, then the
 * boundaries in their slots and the grains around them */
__device__ void prefetch_event(const DevMesh &m, const int *verts, int nverts, int lane)
{
    int j = lane / 3, k = lane - 3 * j;
    if (lane >= 3 * nverts) return;
    int v = verts[j];
    if (!valid_v(m, v)) return;
    if (k == 0) {
        l1_touch(m.pos + v); l1_touch(m.vel + v); l1_touch(m.vstamp + v); l1_touch(m.pos0 + v);
        l1_touch(m.vmod + 4 * (size_t)v); l1_touch(m.vmodmark + v);
    }
    int b = slot3(m.vb[v], k), h = slot3(m.vg[v], k);
    if (valid_b(m, b)) { l1_touch(m.bv + b); l1_touch(m.bstamp + b); l1_touch(m.bexact + b); l1_touch(m.ben + b); }
    if (valid_g(m, h)) { l1_touch(m.gfix + h); l1_touch(m.gexact + h); l1_touch(m.gvlen + h); }
}
/* whether every vertex of an event and every boundary in their slots hold
 * its key (lane 3j + k: vertex j, slot k); nothing but the event holding a
 * vertex writes its slots, so they are the reserved ones */
__device__ bool warp_holds(const DevMesh &m, const DevScratch &x, const int *verts, int nverts, unsigned long long key,
                           int lane)
{
    bool ok = true;
    if (lane < 3 * nverts) {
        int j = lane / 3, v = verts[j];
        ok = valid_v(m, v);
        if (ok) {
            int b = slot3(m.vb[v], lane - 3 * j);
            ok = x.vown[v] == key && valid_b(m, b) && x.bown[b] == key;
        }
    }
    return __all_sync(0xffffffffu, ok);
}

/* remove_grain_dev for the usual case: the same writes with the same
 * values, but every record it reads is loaded up front, in two rounds,
 * instead of behind the writes that precede it, and the work-list appends
 * take one atomic each (the fix-up edits each queued grain on its own, so
 * the order of the entries does not matter).  False, with nothing
 * written, when a boundary or grain the removal needs is not found or an
 * outer boundary also joins A: remove_grain_dev then does it step by step.
 * nAB, nBC, nCA: the triangle's sides. */
__device__ bool remove_planned(const DevMesh &m, int grn, double nAB, double nBC, double nCA)
{
    const int *row = m.glist + (size_t)SEVC_MAXV * grn;
    const int A = row[0], B = row[1], C = row[2];
    const double D = m.D;
    double2 pa = m.pos[A], pb = m.pos[B], pc = m.pos[C], va = m.vel[A];
    int4 sa = m.vb[A], sb = m.vb[B], sc = m.vb[C], ga = m.vg[A], gb = m.vg[B], gc = m.vg[C];
    int4 mB0 = m.vmod[4 * (size_t)B], mC0 = m.vmod[4 * (size_t)C], mB1 = m.vmod[4 * (size_t)B + 1];
    uint8_t mkB = m.vmodmark[B], mkC = m.vmodmark[C];
    unsigned st = *m.stamp, stA = m.vstamp[A];
    int2 ea[3], eb[3], ec[3];
#pragma unroll
    for (int i = 0; i < 3; i++) { ea[i] = m.bv[slot3(sa, i)]; eb[i] = m.bv[slot3(sb, i)]; ec[i] = m.bv[slot3(sc, i)]; }
    int BC = -1, BE = -1, CF = -1, AB = -1, CA = -1, iAB = 0, iCA = 0;
    int2 eBE = make_int2(0, 0), eCF = make_int2(0, 0);
#pragma unroll
    for (int i = 2; i >= 0; i--) {                  /* the first match of each search */
        if ((ec[i].x == B && ec[i].y == C) || (ec[i].y == B && ec[i].x == C)) BC = slot3(sc, i);
        if (!(eb[i].x == A || eb[i].y == A) && !(eb[i].x == C || eb[i].y == C)) { BE = slot3(sb, i); eBE = eb[i]; }
        if (!(ec[i].x == A || ec[i].y == A) && !(ec[i].x == B || ec[i].y == B)) { CF = slot3(sc, i); eCF = ec[i]; }
        if (ea[i].x == B || ea[i].y == B) { AB = slot3(sa, i); iAB = i; }
    }
#pragma unroll
    for (int i = 2; i >= 0; i--)
        if (!(AB >= 0 && i == iAB) && (ea[i].x == C || ea[i].y == C)) { CA = slot3(sa, i); iCA = i; }
    int gbc[2], gab[2], gac[2];
    gintersect(gb, gc, gbc);
    gintersect(ga, gb, gab);
    gintersect(ga, gc, gac);
    const int G3 = gbc[0] == grn ? gbc[1] : gbc[0], G2 = gab[0] == grn ? gab[1] : gab[0];
    const int G1 = gac[0] == grn ? gac[1] : gac[0];
    if (BC < 0 || BE < 0 || CF < 0 || AB < 0 || CA < 0 || G1 < 0 || G2 < 0 || G3 < 0 || BE == CF) return false;
    if (sa.x == BE || sa.y == BE || sa.z == BE || sa.x == CF || sa.y == CF || sa.z == CF) return false;
    unsigned sBE = m.bstamp[BE], sCF = m.bstamp[CF];
    log_event(m, EV_REMOVE, A, B, C, pa, pb, pc);
    /* mark_fix of the three grains: claims and appends */
    const int G[3] = { G2, G1, G3 };
    bool nf[3];
    int nfix = 0;
#pragma unroll
    for (int k = 0; k < 3; k++) {
        nf[k] = claim_byte(m.gfix, G[k]);
        nfix += nf[k];
    }
    const int nm = (mkB ? 0 : 1) + (mkC ? 0 : 1);
    int f0 = nfix ? atomicAdd(m.nfix, nfix) : 0, m0 = nm ? atomicAdd(m.nmod, nm) : 0;
    double denom = nAB + nBC + nCA;
    double x0 = 0, y0 = 0;                                      /* adjust_origin_for_points, 3 points */
    double x1 = x0 + wrapd(pb.x, pa.x, D), y1 = y0 + wrapd(pb.y, pa.y, D);
    double x2 = x1 + wrapd(pc.x, pb.x, D), y2 = y1 + wrapd(pc.y, pb.y, D);
    double2 q = pa;
    q.x += (nBC * x0 + nCA * x1 + nAB * x2) / denom;
    q.y += (nBC * y0 + nCA * y1 + nAB * y2) / denom;
    q.x = dmod(q.x, D);
    q.y = dmod(q.y, D);
    if (stA != st) { m.pos0[A] = pa; m.vel0[A] = va; m.vstamp[A] = st; }     /* save_vertex */
    m.pos[A] = q;
    m.vel[A] = make_double2(0.0, 0.0);
    m.ben[BC] = 0;
    m.ben[AB] = 0;
    m.ben[CA] = 0;
    if (sBE != st) { m.bv0[BE] = eBE; m.bstamp[BE] = st; }                   /* save_ends */
    if (sCF != st) { m.bv0[CF] = eCF; m.bstamp[CF] = st; }
    if (eBE.x == B) eBE.x = A; else eBE.y = A;
    if (eCF.x == C) eCF.x = A; else eCF.y = A;
    m.bv[BE] = eBE;
    m.bv[CF] = eCF;
    set_slot3(sa, iAB, BE);
    set_slot3(sa, iCA, CF);
    m.vb[A] = sa;
    m.ven[B] = 0;
    m.ven[C] = 0;
    m.gen[grn] = 0;
    /* set_mod(B, 0, REMOVE, G2, B), (C, 0, REMOVE, G1, C), (B, 1, REMOVE, G3,
     * B), (C, 1, REPLACE, G3, A, C) */
    mB0.x = G2; mB0.y = B; mB0.w = FIX_REMOVE;
    mC0.x = G1; mC0.y = C; mC0.w = FIX_REMOVE;
    mB1.x = G3; mB1.y = B; mB1.w = FIX_REMOVE;
    m.vmod[4 * (size_t)B] = mB0;
    m.vmod[4 * (size_t)C] = mC0;
    m.vmod[4 * (size_t)B + 1] = mB1;
    m.vmod[4 * (size_t)C + 1] = make_int4(G3, A, C, FIX_REPLACE);
    if (!mkB) {
        m.vmodmark[B] = 1;
        if (m0 < m.modcap) m.modlist[m0] = B; else raise_err(m, ERRB_WORKLIST);
        m0++;
    }
    if (!mkC) {
        m.vmodmark[C] = 1;
        if (m0 < m.modcap) m.modlist[m0] = C; else raise_err(m, ERRB_WORKLIST);
    }
#pragma unroll
    for (int k = 0; k < 3; k++)
        if (nf[k]) {
            if (f0 < m.fixcap) m.fixlist[f0] = G[k]; else raise_err(m, ERRB_WORKLIST);
            f0++;
        }
    for (int i = 0; i < 3; i++) if (slot3(ga, i) == grn) set_slot3(ga, i, G3);
    m.vg[A] = ga;
    return true;
}

/* clear_grains_state and label_3sided_grains (src/main.cu:252-255), then the
 * removals' reservations (remove_grains, :994): a removal disables only its
 * own grain, so the set is known up front.  A removable grain has an
 * enabled boundary with 0 <= t_ext <= dt, so it lies beside a boundary of
 * the candidate list: one thread per listed boundary and grain at its first
 * end; the grain is listed by its lowest such boundary.  first: this thread's
 * first item, null if the mesh has changed since it was loaded. */
__device__ __forceinline__ int label_start(const Team &T) { return T.tid < T.n / 2 ? T.tid + T.n / 2 : T.tid - T.n / 2; }
__device__ void label3_reserve(const DevMesh &m, const DevScratch &x, const Team &T, int na, double dt,
                               const LabelItem *first)
{
    const unsigned ep = 2u * *m.stamp;
    const int t0 = label_start(T);
    for (int t = t0; t < 3 * na; t += T.n) {
        const LabelItem l = t == t0 && first ? *first : label_item(m, x.list_a, t, na);
        if (l.g < 0) continue;
        int L[3], bs[9];
        if (label3_first(m, l.g, dt, L, bs) != l.b) continue;
        x.list_c[atomicAdd(x.n_c, 1)] = l.g;
        const unsigned long long key = resv_key(ep, l.g);
#pragma unroll
        for (int k = 0; k < 3; k++) reserve_vertex(m, x, L[k], make_int4(bs[3 * k], bs[3 * k + 1], bs[3 * k + 2], -1), key);
    }
}
/* One warp per removal: its lanes check that it holds its records and bring
 * them into L1, lane 0 applies it (or it defers, when an earlier removal
 * holds a record). */
__device__ void remove_warp(const DevMesh &m, int g, int inst, int lane)
{
    /* lane k < 3: the side from list vertex k to the next */
    const int *L = m.glist + (size_t)SEVC_MAXV * g;
    double side = 0;
    if (lane < 3) side = arclen(m.pos[L[lane]], m.pos[L[lane < 2 ? lane + 1 : 0]], m.D);
    const double s0 = __shfl_sync(0xffffffffu, side, 0), s1 = __shfl_sync(0xffffffffu, side, 1),
                 s2 = __shfl_sync(0xffffffffu, side, 2);
    if (lane == 0) {
        if (!remove_planned(m, g, s0, s1, s2)) remove_grain_dev(m, g);
        atomicAdd(&m.evt[EVT_COUNT * inst + EVT_REMOVALS], 1);
    }
    __syncwarp();
}
__device__ void remove_apply(const DevMesh &m, const DevScratch &x, const Team &T, const int *list, int n)
{
    const unsigned ep = 2u * *m.stamp;
    for (int i = T.warp; i < n; i += T.nwarps) {
        int g = list[i];
        const int *L = m.glist + (size_t)SEVC_MAXV * g;
        int verts[3] = { L[0], L[1], L[2] };
        prefetch_event(m, verts, 3, T.lane);
        bool own = warp_holds(m, x, verts, 3, resv_key(ep, g), T.lane);
        if (own) remove_warp(m, g, m.ginst[g], T.lane);
        else if (T.lane == 0) x.ehits[atomicAdd(x.n_ehits, 1)] = g;
    }
}
/* The deferred events x.ehits[0..nd) in ascending order, one warp per
 * instance over its own part (off: the instances' first indices). */
template <class Apply>
__device__ void run_deferred(const DevMesh &m, const DevScratch &x, const Team &T, int nd, const int *off, Apply apply)
{
    int *sorted = x.list_b;               /* the 2x3 list, done with */
    rank_sort(T, x.ehits, nd, sorted);
    T.sync();
    if (T.tid == 0) *x.n_ehits = 0;
    for (int inst = T.warp; inst < m.ninst; inst += T.nwarps) {
        int lo = 0, hi = nd;
        if (m.ninst > 1) {
            lo = lower_bound_i(sorted, nd, off[inst]);
            hi = lower_bound_i(sorted, nd, off[inst + 1]);
        }
        for (int i = lo; i < hi; i++) apply(sorted[i], inst);
    }
}

/* ------------------------------------------------------------------ */
/* T1 flip, src/topological.h:174-291                                  */
/* ------------------------------------------------------------------ */
__device__ __noinline__ void flip_dev(const DevMesh &m, int bnd, double eps)
{
    int2 eb = m.bv[bnd];
    int A = eb.x, B = eb.y;
    int gic[2], gnic[2];
    if (gintersect(m.vg[A], m.vg[B], gic) < 2) { raise_err(m, ERRB_TOPOLOGY); return; }
    gsymdiff(m.vg[A], m.vg[B], gnic);
    int4 sa = m.vb[A], sb = m.vb[B];
    int i = -1, j = -1, AC = -1, BE = -1;
    for (int k = 0; k < 3; k++) if (slot3(sa, k) == bnd) { i = (k + 1) % 3; AC = slot3(sa, i); break; }
    for (int k = 0; k < 3; k++) if (slot3(sb, k) == bnd) { j = (k + 1) % 3; BE = slot3(sb, j); break; }
    if (AC < 0 || BE < 0 || gnic[0] < 0 || gnic[1] < 0) { raise_err(m, ERRB_TOPOLOGY); return; }
    set_slot3(sa, i, BE);
    set_slot3(sb, j, AC);
    m.vb[A] = sa;
    m.vb[B] = sb;
    save_ends(m, AC);
    save_ends(m, BE);
    int2 e = m.bv[AC]; if (e.x == A) e.x = B; else e.y = B; m.bv[AC] = e;
    e = m.bv[BE]; if (e.x == B) e.x = A; else e.y = A; m.bv[BE] = e;
    int g1, g2, g3, g4;
    for (g2 = 0; g2 < 2; g2++) if (glist_consecutive(m, gic[g2], A, B) == 1) break;
    for (g4 = 0; g4 < 2; g4++) if (glist_consecutive(m, gic[g4], B, A) == 1) break;
    for (g3 = 0; g3 < 2; g3++) if (glist_find(m, gnic[g3], A) >= 0) break;
    for (g1 = 0; g1 < 2; g1++) if (glist_find(m, gnic[g1], B) >= 0) break;
    if (g2 < 2) { set_mod(m, A, 0, FIX_REMOVE, gic[g2], A, -2); mark_fix(m, gic[g2]); }
    if (g4 < 2) { set_mod(m, B, 0, FIX_REMOVE, gic[g4], B, -2); mark_fix(m, gic[g4]); }
    if (g3 < 2) { set_mod(m, A, 1, FIX_ADD, gnic[g3], B, A); mark_fix(m, gnic[g3]); }
    if (g1 < 2) { set_mod(m, B, 1, FIX_ADD, gnic[g1], A, B); mark_fix(m, gnic[g1]); }
    if (g1 == 2 || g2 == 2 || g3 == 2 || g4 == 2) { raise_err(m, ERRB_TOPOLOGY); return; }
    int4 ga = m.vg[A], gb = m.vg[B];
    for (int k = 0; k < 3; k++) {
        if (slot3(ga, k) == gic[g2]) set_slot3(ga, k, gnic[g1]);
        if (slot3(gb, k) == gic[g4]) set_slot3(gb, k, gnic[g3]);
    }
    m.vg[A] = ga;
    m.vg[B] = gb;
    double2 pa = m.pos[A], pb = m.pos[B];                 /* vector2_mean, src/geometry.h:311 */
    log_event(m, EV_FLIP, A, B, -1, pa, pb, pb);
    double2 c = pa;
    c.x += wrapd(pb.x, pa.x, m.D) / 2;
    c.y += wrapd(pb.y, pa.y, m.D) / 2;
    c.x = dmod(c.x, m.D);
    c.y = dmod(c.y, m.D);
    save_vertex(m, A);
    save_vertex(m, B);
    m.pos[A] = c;
    m.pos[B] = c;
    sa = m.vb[A]; { int t = sa.y; sa.y = sa.x; sa.x = t; } m.vb[A] = sa; /* vertex_invert_boundary_order */
    sb = m.vb[B]; { int t = sb.y; sb.y = sb.x; sb.x = t; } m.vb[B] = sb;
    /* boundary_compute_energy (no GB scaling here, as in the reference) */
    if (eps == 0.0) {
        m.benergy[bnd] = 1.0;
    } else {
        int g2c[2];
        if (gintersect(m.vg[A], m.vg[B], g2c) < 2) { raise_err(m, ERRB_TOPOLOGY); return; }
        m.benergy[bnd] = gb_energy(m.gori[g2c[0]] - m.gori[g2c[1]], eps);
    }
    m.vel[A] = make_double2(0, 0);
    m.vel[B] = make_double2(0, 0);
}

/* What flip_dev derives before it writes anything: the two ends, their
 * other boundaries AC and BE (the successors of bnd in their slot
 * orders, at slots i and j), the grains on both sides (gic) and at the
 * ends (gnic), the ends' slot and grain records, and which of those grains
 * get which list edit (g1..g4, as flip_dev names them). */
struct FlipPlan {
    int A, B, AC, BE, i, j, g1, g2, g3, g4;
    int gic[2], gnic[2];
    int4 sa, sb, ga, gb;
};

/* Every lane of the warp derives the flip's plan; eight lanes scan each of
 * the four grain lists (a flip edits no list, so the answers are the ones
 * flip_dev's own scans give: glist_consecutive(g, P, Q) is 1 when the first
 * place where P and Q are neighbours has P first).  Returns false on any
 * inconsistency; the flip then runs its own checks and reports it. */
__device__ bool flip_plan(const DevMesh &m, int bnd, int lane, FlipPlan &P)
{
    int2 eb = m.bv[bnd];
    int A = eb.x, B = eb.y;
    if (A < 0 || A >= m.nv || B < 0 || B >= m.nv || A == B) return false;
    P.A = A; P.B = B;
    P.ga = m.vg[A]; P.gb = m.vg[B]; P.sa = m.vb[A]; P.sb = m.vb[B];
    if (gintersect(P.ga, P.gb, P.gic) < 2) return false;
    gsymdiff(P.ga, P.gb, P.gnic);
    P.i = P.j = P.AC = P.BE = -1;
    for (int k = 0; k < 3; k++) if (slot3(P.sa, k) == bnd) { P.i = (k + 1) % 3; P.AC = slot3(P.sa, P.i); break; }
    for (int k = 0; k < 3; k++) if (slot3(P.sb, k) == bnd) { P.j = (k + 1) % 3; P.BE = slot3(P.sb, P.j); break; }
    if (P.AC < 0 || P.BE < 0 || P.gnic[0] < 0 || P.gnic[1] < 0) return false;
    const int q = lane >> 3, g = q < 2 ? P.gic[q] : P.gnic[q - 2];
    const int *L = m.glist + (size_t)SEVC_MAXV * g;
    const int n = m.gvlen[g];
    int ab = SEVC_MAXV, ba = SEVC_MAXV;             /* first i with (A, B), (B, A) at i, i + 1 */
    bool hasA = false, hasB = false;
    for (int i = lane & 7; i < n; i += 8) {
        int u = L[i], w = L[i + 1 < n ? i + 1 : 0];
        if (u == A && w == B && ab == SEVC_MAXV) ab = i;
        if (u == B && w == A && ba == SEVC_MAXV) ba = i;
        hasA |= u == A;
        hasB |= u == B;
    }
    for (int o = 4; o > 0; o >>= 1) {
        ab = min(ab, __shfl_xor_sync(0xffffffffu, ab, o));
        ba = min(ba, __shfl_xor_sync(0xffffffffu, ba, o));
    }
    const unsigned f = __ballot_sync(0xffffffffu, ab < SEVC_MAXV && ab <= ba);
    const unsigned r = __ballot_sync(0xffffffffu, ba < SEVC_MAXV && ba < ab);
    const unsigned hA = __ballot_sync(0xffffffffu, hasA), hB = __ballot_sync(0xffffffffu, hasB);
    P.g2 = (f & 0xffu) ? 0 : (f & 0xff00u) ? 1 : 2;
    P.g4 = (r & 0xffu) ? 0 : (r & 0xff00u) ? 1 : 2;
    P.g3 = (hA & 0xff0000u) ? 0 : (hA & 0xff000000u) ? 1 : 2;
    P.g1 = (hB & 0xff0000u) ? 0 : (hB & 0xff000000u) ? 1 : 2;
    return !(P.g1 == 2 || P.g2 == 2 || P.g3 == 2 || P.g4 == 2);
}

/* flip_dev from a plan, for the usual case AC != BE: the same writes with
 * the same values, but every record the flip reads is loaded up front in
 * one round trip instead of behind the writes that precede it, and the
 * work-list appends of the mod slots and of the fix-up grains take one
 * atomic each (the fix-up pass edits each queued grain on its own, so the
 * order of the entries does not matter). */
__device__ void flip_planned(const DevMesh &m, int bnd, double eps, const FlipPlan &P)
{
    const int A = P.A, B = P.B, AC = P.AC, BE = P.BE;
    const int G[4] = { P.gic[P.g2], P.gic[P.g4], P.gnic[P.g3], P.gnic[P.g1] };
    unsigned st = *m.stamp;
    unsigned sAC = m.bstamp[AC], sBE = m.bstamp[BE], stA = m.vstamp[A], stB = m.vstamp[B];
    int2 eAC = m.bv[AC], eBE = m.bv[BE];
    int4 mA0 = m.vmod[4 * (size_t)A], mB0 = m.vmod[4 * (size_t)B];
    uint8_t mkA = m.vmodmark[A], mkB = m.vmodmark[B];
    double2 pa = m.pos[A], pb = m.pos[B], va = m.vel[A], vb = m.vel[B];
    log_event(m, EV_FLIP, A, B, -1, pa, pb, pb);
    /* boundary slots, then vertex_invert_boundary_order */
    int4 sa = P.sa, sb = P.sb;
    set_slot3(sa, P.i, BE);
    set_slot3(sb, P.j, AC);
    { int t = sa.y; sa.y = sa.x; sa.x = t; }
    { int t = sb.y; sb.y = sb.x; sb.x = t; }
    m.vb[A] = sa;
    m.vb[B] = sb;
    if (sAC != st) { m.bv0[AC] = eAC; m.bstamp[AC] = st; }      /* save_ends */
    if (sBE != st) { m.bv0[BE] = eBE; m.bstamp[BE] = st; }
    if (eAC.x == A) eAC.x = B; else eAC.y = B;
    if (eBE.x == B) eBE.x = A; else eBE.y = A;
    m.bv[AC] = eAC;
    m.bv[BE] = eBE;
    /* set_mod(A, 0, REMOVE), (B, 0, REMOVE), (A, 1, ADD), (B, 1, ADD) */
    mA0.x = G[0]; mA0.y = A; mA0.w = FIX_REMOVE;
    mB0.x = G[1]; mB0.y = B; mB0.w = FIX_REMOVE;
    m.vmod[4 * (size_t)A] = mA0;
    m.vmod[4 * (size_t)B] = mB0;
    m.vmod[4 * (size_t)A + 1] = make_int4(G[2], B, A, FIX_ADD);
    m.vmod[4 * (size_t)B + 1] = make_int4(G[3], A, B, FIX_ADD);
    int nm = (mkA ? 0 : 1) + (mkB ? 0 : 1);
    if (nm) {
        int i0 = atomicAdd(m.nmod, nm);
        if (!mkA) {
            m.vmodmark[A] = 1;
            if (i0 < m.modcap) m.modlist[i0] = A; else raise_err(m, ERRB_WORKLIST);
            i0++;
        }
        if (!mkB) {
            m.vmodmark[B] = 1;
            if (i0 < m.modcap) m.modlist[i0] = B; else raise_err(m, ERRB_WORKLIST);
        }
    }
    /* mark_fix of the four grains; flips running at the same time may queue
     * the same grain, the claim decides */
    bool nf[4];
    int nfix = 0;
#pragma unroll
    for (int k = 0; k < 4; k++) {
        nf[k] = claim_byte(m.gfix, G[k]);
        nfix += nf[k];
    }
    if (nfix) {
        int i0 = atomicAdd(m.nfix, nfix);
#pragma unroll
        for (int k = 0; k < 4; k++)
            if (nf[k]) {
                if (i0 < m.fixcap) m.fixlist[i0] = G[k]; else raise_err(m, ERRB_WORKLIST);
                i0++;
            }
    }
    int4 ga = P.ga, gb = P.gb;
    for (int k = 0; k < 3; k++) {
        if (slot3(ga, k) == G[0]) set_slot3(ga, k, G[3]);
        if (slot3(gb, k) == G[1]) set_slot3(gb, k, G[2]);
    }
    m.vg[A] = ga;
    m.vg[B] = gb;
    double2 c = pa;                                         /* vector2_mean, src/geometry.h:311 */
    c.x += wrapd(pb.x, pa.x, m.D) / 2;
    c.y += wrapd(pb.y, pa.y, m.D) / 2;
    c.x = dmod(c.x, m.D);
    c.y = dmod(c.y, m.D);
    if (stA != st) { m.pos0[A] = pa; m.vel0[A] = va; m.vstamp[A] = st; }   /* save_vertex */
    if (stB != st) { m.pos0[B] = pb; m.vel0[B] = vb; m.vstamp[B] = st; }
    m.pos[A] = c;
    m.pos[B] = c;
    if (eps == 0.0) {
        m.benergy[bnd] = 1.0;
    } else {
        int g2c[2];
        if (gintersect(ga, gb, g2c) < 2) { raise_err(m, ERRB_TOPOLOGY); return; }
        m.benergy[bnd] = gb_energy(m.gori[g2c[0]] - m.gori[g2c[1]], eps);
    }
    m.vel[A] = make_double2(0, 0);
    m.vel[B] = make_double2(0, 0);
}

/* apply_flippings (:1016-1026): the reference flips every remaining
 * candidate in parallel, with unsynchronised writes when two share
 * records; here flips follow ascending boundary order, which is every
 * race-free outcome.  A flip changes no boundary's enabled or candidate
 * flag, so the flips are known up front.  Reservation, parallel
 * application and the deferred pass as for the removals (epoch 2 * stamp
 * + 1); the footprint is both ends with their slots. */
/* unlabel_boundaries_st2 (:588-606) for an enabled candidate, then its
 * reservation: it stays a candidate unless a grain on either side has 3
 * sides.  One thread per listed boundary. */
__device__ void flip_reserve(const DevMesh &m, const DevScratch &x, const Team &T, const int *list, int n)
{
    const unsigned ep = 2u * *m.stamp + 1u;
    for (int i = T.tid; i < n; i += T.n) {
        int b = list[i];
        if (!(m.ben[b] && m.bcand[b])) continue;
        int2 e = m.bv[b];
        int4 sa = m.vb[e.x], sb = m.vb[e.y];
        int gic[2];
        if (gintersect(m.vg[e.x], m.vg[e.y], gic) < 2) {       /* the step fails */
            raise_err(m, ERRB_TOPOLOGY);
            continue;
        }
        if (m.gvlen[gic[0]] == 3 || m.gvlen[gic[1]] == 3) {
            m.bcand[b] = 0;
            continue;
        }
        const unsigned long long key = resv_key(ep, b);
        reserve_vertex(m, x, e.x, sa, key);
        reserve_vertex(m, x, e.y, sb, key);
    }
}
/* a warp: its lanes derive the plan, lane 0 applies it */
__device__ void flip_warp(const DevMesh &m, int b, double eps, int lane)
{
    FlipPlan P;
    bool planned = flip_plan(m, b, lane, P) && P.AC != P.BE;
    __syncwarp();
    if (lane == 0) {
        if (planned) flip_planned(m, b, eps, P);
        else flip_dev(m, b, eps);
        atomicAdd(&m.evt[EVT_COUNT * m.binst[b] + EVT_FLIPS], 1);
    }
    __syncwarp();
}
__device__ void flip_apply(const DevMesh &m, const DevScratch &x, const Team &T, const int *list, int n, double eps)
{
    const unsigned ep = 2u * *m.stamp + 1u;
    for (int i = T.warp; i < n; i += T.nwarps) {
        int b = list[i];
        if (!(m.ben[b] && m.bcand[b])) continue;
        int2 e = m.bv[b];
        int verts[2] = { e.x, e.y };
        prefetch_event(m, verts, 2, T.lane);
        bool own = warp_holds(m, x, verts, 2, resv_key(ep, b), T.lane);
        if (own) flip_warp(m, b, eps, T.lane);
        else if (T.lane == 0) x.ehits[atomicAdd(x.n_ehits, 1)] = b;
    }
}

/* ------------------------------------------------------------------ */
/* fix_grain_lists, src/topological.h:1035-1227                        */
/* ------------------------------------------------------------------ */
/* perform_ADD_ops, perform_REMOVE_ops, perform_REPLACE_ops
 * (src/topological.h:1035-1148) for one queued grain.  The reference runs
 * each over all grains before the next; an edit only touches its own
 * grain's list and only reads the mods, which nothing writes meanwhile, so
 * running the three for one grain back to back gives the same lists.
 *
 * One warp per grain.  The lanes copy the list to shared memory and read
 * the four mod slots of every listed vertex at once, recording for each
 * entry whether one of them is an ADD, REMOVE or REPLACE for this grain;
 * lane 0 then runs the three passes exactly as written (same visiting
 * order, same first-match searches, same shifts and -1 fills) on the
 * shared copy, reading the mods again only for the entries that hold an
 * edit (and the flags of a vertex an edit brings into the list), and the
 * lanes write back every entry the passes touched.  The long chain of
 * dependent global reads of one thread per grain becomes one parallel
 * round and a few L1 hits. */
__device__ __forceinline__ unsigned mod_ops_for(const DevMesh &m, int v, int g)
{
    if ((unsigned)v >= (unsigned)m.nv) return 0;
    const int4 *md = m.vmod + 4 * (size_t)v;
    unsigned f = 0;
#pragma unroll
    for (int j = 0; j < 4; j++) {
        int4 x = md[j];
        if (x.x == g) f |= x.w == FIX_ADD ? 1u : x.w == FIX_REMOVE ? 2u : x.w == FIX_REPLACE ? 4u : 0u;
    }
    return f;
}
__device__ void fix_grain_serial(const DevMesh &m, int g, int *Ls, unsigned char *Fs, int *Ss, unsigned char *SFs,
                                 int &n, int &hi)
{
    for (int i = 0; i < n; i++) {                        /* ADD */
        if (!(Fs[i] & 1u)) continue;
        const int v = Ls[i];
        for (int j = 0; j < 4; j++) {
            int4 md = m.vmod[4 * (size_t)v + j];
            if (!(md.w == FIX_ADD && md.x == g)) continue;
            int pos = -1;                                /* glist_add_after(g, md.y, md.z) */
            for (int k = 0; k < n; k++)
                if (Ls[k] == md.z) { pos = k + 1; break; }
            if (pos < 0) { raise_err(m, ERRB_TOPOLOGY); continue; }
            if (n >= SEVC_MAXV) { raise_err(m, ERRB_CAPACITY); continue; }
            for (int k = n; k > pos; k--) { Ls[k] = Ls[k - 1]; Fs[k] = Fs[k - 1]; }
            Ls[pos] = md.y;
            Fs[pos] = (unsigned char)mod_ops_for(m, md.y, g);
            n++;
            hi = n > hi ? n : hi;
        }
    }
    const int n0 = n;                                    /* REMOVE over the list as it stood */
    for (int i = 0; i < n0; i++) { Ss[i] = Ls[i]; SFs[i] = Fs[i]; }
    for (int i = 0; i < n0; i++) {
        if (!(SFs[i] & 2u)) continue;
        const int v = Ss[i];
        for (int j = 0; j < 4; j++) {
            int4 md = m.vmod[4 * (size_t)v + j];
            if (!(md.w == FIX_REMOVE && md.x == g)) continue;
            for (int k = 0; k < n; k++)                  /* glist_remove(g, md.y) */
                if (Ls[k] == md.y) {
                    for (int q = k; q < n - 1; q++) { Ls[q] = Ls[q + 1]; Fs[q] = Fs[q + 1]; }
                    n--;
                    Ls[n] = -1;
                    Fs[n] = 0;
                    break;
                }
        }
    }
    for (int i = 0; i < n; i++) {                        /* REPLACE */
        if (!(Fs[i] & 4u)) continue;
        const int v = Ls[i];
        for (int j = 0; j < 4; j++) {
            int4 md = m.vmod[4 * (size_t)v + j];
            if (!(md.w == FIX_REPLACE && md.x == g)) continue;
            for (int k = 0; k < n; k++)                  /* glist_replace(g, md.z, md.y) */
                if (Ls[k] == md.z) {
                    Ls[k] = md.y;
                    Fs[k] = (unsigned char)mod_ops_for(m, md.y, g);
                    break;
                }
        }
    }
}
/* compute_area (RATE false: area_stream) or compute_dAdt (RATE true:
 * dadt_over, from the step's starting state) over the list L of n entries by
 * one warp, the same operations in the same order: each lane forms its
 * vertex's wrapped delta and its terms, and the additions whose order counts,
 * the running coordinates and the sum, go through the lanes in list order. */
template <bool RATE> __device__ __forceinline__ double warp_sum(const DevMesh &m, const int *L, int n, int lane, unsigned st)
{
    const unsigned all = 0xffffffffu;
    double acc = 0, X = 0, Y = 0, vx = 0, vy = 0;    /* the sum; the last vertex's coordinates and velocity */
    double2 pr = make_double2(0, 0), w0 = pr;        /* its position; the first vertex's velocity */
    for (int base = 0; base < n; base += 32) {
        const int k = base + lane, len = min(n - base, 32);
        double2 r = make_double2(0, 0), w = r;
        if (k < n) {
            const int v = L[k];
            r = m.pos[v];
            if (RATE) {
                w = m.vel[v];
                if (m.vstamp[v] == st) { r = m.pos0[v]; w = m.vel0[v]; }
            }
        }
        double2 q = make_double2(__shfl_up_sync(all, r.x, 1), __shfl_up_sync(all, r.y, 1));
        if (lane == 0) q = pr;
        double dx = 0, dy = 0, mx = 0, my = 0, px = X, py = Y;
        if (k > 0 && k < n) { dx = wrapd(r.x, q.x, m.D); dy = wrapd(r.y, q.y, m.D); }
#pragma unroll 1
        for (int j = 0; j < len; j++) {
            if (j == lane) { px = X; py = Y; }
            X += __shfl_sync(all, dx, j);
            Y += __shfl_sync(all, dy, j);
            if (j == lane) { mx = X; my = Y; }
        }
        double t, u = 0;
        if (RATE) {
            double2 z = make_double2(__shfl_up_sync(all, w.x, 1), __shfl_up_sync(all, w.y, 1));
            if (lane == 0) z = make_double2(vx, vy);
            t = z.x * my + px * w.y;
            u = z.y * mx + py * w.x;
            if (base == 0) w0 = make_double2(__shfl_sync(all, w.x, 0), __shfl_sync(all, w.y, 0));
            vx = __shfl_sync(all, w.x, len - 1);
            vy = __shfl_sync(all, w.y, len - 1);
        } else {
            t = px * my - py * mx;
        }
        pr = make_double2(__shfl_sync(all, r.x, len - 1), __shfl_sync(all, r.y, len - 1));
#pragma unroll 1
        for (int j = base ? 0 : (RATE ? 1 : 2); j < len; j++) {
            acc += __shfl_sync(all, t, j);
            if (RATE) acc -= __shfl_sync(all, u, j);
        }
    }
    if (RATE) {
        if (n > 0) {
            acc += (vx * 0.0 + X * w0.y);
            acc -= (vy * 0.0 + Y * w0.x);
        }
        return acc;
    }
    if (n > 0) acc = add_closing_term(acc, X, Y);
    return dscale_down<1>(acc);
}
template <int WARPS> struct EditShared {
    int Ls[WARPS][SEVC_MAXV], Ss[WARPS][SEVC_MAXV], Nw[WARPS][2];
    unsigned char Fs[WARPS][SEVC_MAXV], SFs[WARPS][SEVC_MAXV];
};
__device__ __noinline__ void settle_boundary(const DevMesh &m, int b) { finalize_boundary(m, b); }
/* fix_grain_lists (:1209-1227), the edits, with what belongs to a grain
 * before and after its own: one warp per queued grain and per removed one
 * (gone[0..ngone)), in this order
 *   settle   the output-only dA/dt (see DevMesh) over the list as it still
 *            is, from the step's starting state, which the events saved
 *   edit     the list (queued and enabled grains)
 *   area     compute_grain_areas after the removals (src/main.cu:266), if
 *            areas is set.  Only a grain whose list changed since the grain
 *            pass can have a new area (the vertex a 3-sided removal moves
 *            belongs only to grains that removal queues), and its list and
 *            vertices are final for the step here; a grain edited by several
 *            fix-ups (2x3 passes, then the removals) is computed again by
 *            each, the last one on the final positions; one that is removed
 *            after a 2x3 pass edited it gets its first area back.  The flips' fix-up
 *            comes after the counts and needs none (the next step's grain
 *            pass computes every area).
 * No warp reads another's grain, so nothing separates the three.  three,
 * n_three (may be null): grains the edit leaves with three sides are listed
 * there.
 *
 * Beside them, the extinction times of the boundaries at the removed grains'
 * vertices that are now disabled.  One costs some 400 FP64 operations
 * (atan2, cos, sin), so its threads are the k-th (k < 3) such boundary of each
 * removed grain, not its nine slots with mostly idle lanes; the third takes
 * any beyond. */
template <int WARPS>
__device__ void edit_grains(const DevMesh &m, const Team &T, EditShared<WARPS> &S, const int *gone, int ngone, bool areas,
                            int *three, int *n_three)
{
    const int lane = T.lane, wib = threadIdx.x >> 5;
    const int nf = min(*m.nfix, m.fixcap);
    const unsigned st = *m.stamp;
    for (int w = T.warp; w < nf + ngone; w += T.nwarps) {
        const int g = w < nf ? m.fixlist[w] : gone[w - nf];
        int *L = m.glist + (size_t)SEVC_MAXV * g;
        int n = m.gvlen[g];
        const bool due = !m.gexact[g], queued = w < nf && m.gen[g], edit = queued && m.gfix[g];
        if (edit) {
            for (int i = lane; i < n; i += 32) {
                int v = L[i];
                S.Ls[wib][i] = v;
                S.Fs[wib][i] = (unsigned char)mod_ops_for(m, v, g);
            }
        }
        if (due) {
            const double d = warp_sum<true>(m, L, n, lane, st);
            if (lane == 0) { m.gdadt[g] = d; m.gexact[g] = GEXACT_DADT; }
        }
        if (edit) {
            __syncwarp();
            if (lane == 0) {
                int nn = n, hi = n;
                fix_grain_serial(m, g, S.Ls[wib], S.Fs[wib], S.Ss[wib], S.SFs[wib], nn, hi);
                S.Nw[wib][0] = nn;
                S.Nw[wib][1] = hi;
                if (nn != n) m.gvlen[g] = nn;
                if (n_three && nn == 3 && n != 3) three[atomicAdd(n_three, 1)] = g;
            }
            __syncwarp();
            n = S.Nw[wib][0];
            const int hi = S.Nw[wib][1];
            for (int i = lane; i < hi; i += 32) L[i] = S.Ls[wib][i];
        }
        if (queued) {
            if (areas) {
                const double a = warp_sum<false>(m, edit ? S.Ls[wib] : L, n, lane, 0);
                if (lane == 0) {
                    if (n_three && !(m.gexact[g] & GEXACT_AREA)) {   /* a 2x3 pass: see DevMesh */
                        m.garea0[g] = m.garea[g];
                        m.gexact[g] |= GEXACT_AREA;
                    }
                    m.garea[g] = a;
                }
            }
            if (lane == 0) m.gfix[g] = 0;            /* clear_grains_fix_state (:1150-1163) */
        }
        if (w >= nf && lane == 0 && (m.gexact[g] & GEXACT_AREA)) m.garea[g] = m.garea0[g];
        __syncwarp();
    }
    /* the boundaries from the other end of the team, beside the grains */
    for (int t = T.n - 1 - T.tid; t < 3 * ngone; t += T.n) {
        const int i = t / 3, k = t - 3 * i;
        const int *L = m.glist + (size_t)SEVC_MAXV * gone[i];
        int b[9];
#pragma unroll
        for (int j = 0; j < 3; j++) {
            int4 s = m.vb[L[j]];
            b[3 * j] = s.x; b[3 * j + 1] = s.y; b[3 * j + 2] = s.z;
        }
        unsigned due = 0;
#pragma unroll
        for (int j = 0; j < 9; j++) {
            /* not by bexact, which the grain's other threads and those of the
             * grains around it set meanwhile: all must count alike */
            bool off = valid_b(m, b[j]) && !m.ben[b[j]];
#pragma unroll
            for (int q = 0; q < j; q++) off = off && b[q] != b[j];
            due |= off ? 1u << j : 0u;
        }
        for (int c = 0; c < k; c++) due &= due - 1;
        /* the first call is every thread's at once */
        for (; due; due &= due - 1) {
            const int j = __ffs(due) - 1;
            int x = b[0];
#pragma unroll
            for (int q = 1; q < 9; q++) x = q == j ? b[q] : x;
            settle_boundary(m, x);
            if (k < 2) break;
        }
    }
}
/* clear_grains_fix_state (:1150-1163), the rest: reset the mods of every
 * vertex listed by an enabled grain.  Only marked vertices can hold mods.
 * Thread tid of n: one marked vertex and grain around it; each that finds
 * the vertex listed writes the same. */
__device__ __forceinline__ void clear_mods(const DevMesh &m, int tid, int n)
{
    const int nm = min(*m.nmod, m.modcap);
    for (int t = tid; t < 3 * nm; t += n) {
        int w = t / 3, j = t - 3 * w, v = m.modlist[w];
        if (j == 0) m.vmodmark[v] = 0;
        int g = slot3(m.vg[v], j);
        if (g >= 0 && m.gen[g] && glist_find(m, g, v) >= 0)
            for (int k = 0; k < 4; k++) m.vmod[4 * (size_t)v + k] = make_int4(-1, -1, -1, FIX_NONE);
    }
}
typedef EditShared<TAIL_WARPS> FixShared;
/* the edits, then the clearing; both work lists empty afterwards.  Ends with
 * a sync. */
__device__ void fix_lists(const DevMesh &m, const Team &T, FixShared &S, const int *gone, int ngone, bool areas,
                          int *three, int *n_three)
{
    if (*m.nfix == 0 && *m.nmod == 0 && ngone == 0) return; /* the same in every block: written before the last sync */
    edit_grains(m, T, S, gone, ngone, areas, three, n_three);
    T.sync();
    clear_mods(m, T.tid, T.n);
    T.sync();
    if (T.tid == 0) *m.nfix = *m.nmod = 0;
    T.sync();
}

/* ------------------------------------------------------------------ */
/* the sparse phases                                                   */
/* ------------------------------------------------------------------ */
/* the 2x3 loop (src/main.cu:227-250) from its first count, n > 0 */
__device__ void two_three_loop(const DevMesh &m, const DevScratch &x, const Team &T, FixShared &S)
{
    int *sorted = x.list_c;
    int n = *x.n_b, known = 0;
    for (int pass = 0; n > 0 && pass < TWO_THREE_PASSES; pass++) {
        int *ce = sorted + n;
        const int ce_cap = m.nb - n;
        rank_sort(T, x.list_b, n, sorted);
        T.sync();
        if (T.tid == 0) *x.n_b = 0;
        T.sync();
        for (int i = T.tid; i < m.ninst; i += T.n)
            remove_two_three(m, sorted, n, x.extra, x.segcnt + (size_t)pass * m.ninst, x.list_b, x.n_b, ce, ce_cap,
                             i);
        T.sync();
        /* with the removed grains, listed by the removals */
        const int pairs = *x.n_b / 2;
        fix_lists(m, T, S, x.list_b, 2 * pairs, true, x.ehits, x.n_ehits);
        if (T.tid == 0) *x.n_b = 0;
        T.sync();
        const int n3 = *x.n_three, more = *x.n_ehits;
        if (pairs <= ce_cap) {
            find_two_three_again(m, T, x.ehits + known, more - known, ce, pairs, x.list_b, x.n_b);
        } else {
            for (int t = T.tid; t < 9 * (n3 + more); t += T.n)
                find_two_three(m, x.three, n3, x.ehits, t, x.list_b, x.n_b);
        }
        known = more;
        T.sync();
        n = *x.n_b;
    }
}

/* The part of a step after the t_ext labels (src/main.cu:219-325) as one
 * launch of one cluster.  PART selects what a launch covers:
 *   TAIL_REMOVE  polling (:219), conflicts (:222-225), the 2x3 loop
 *                (:227-250), 3-sided labels (:252-255), removals (:259)
 *   TAIL_FLIP    flips (:282-289)
 *   TAIL_END     the list fix-ups (:262-266, :294), position update (:314),
 *                counts (:317-325), step summary
 * On a large mesh TAIL_REMOVE and TAIL_FLIP are launches of their own and
 * the fix-ups run on the whole GPU behind each (k_edit).  TAIL_SPREAD: each
 * ends at its reservations, and k_apply and k_deferred behind it take the
 * events (see launch_tail_removals).
 *
 * What bounds it: nothing but the chain of its phases, each a handful of
 * dependent loads.  As ~25 kernels (programmatic dependent launch between
 * them) and two conditional graph nodes the chain took 100-150 us a step; a
 * cluster barrier costs well under a microsecond.  16 blocks of 512 are the
 * largest cluster; with a warp per event that is 256 events at once. */
constexpr int TAIL_WHOLE_NV = 64 * 1024;
enum { TAIL_REMOVE = 1, TAIL_FLIP = 2, TAIL_END = 4, TAIL_SPREAD = 8 };
template <int PART>
__global__ void __launch_bounds__(TAIL_TPB) k_tail(DevMesh m, DevScratch x, PollGrid pg, int cap, double dt, double eps,
                                                  int *summary)
{
    griddep_wait();
    __shared__ FixShared S;
    const Team T;
    const int na = *x.n_a;
    if (PART & TAIL_END)
        for (int i = T.tid; i < m.ninst; i += T.n) x.counters[(size_t)i * CTR_COUNT + CTR_NGRAINS] = 0;
    if (PART & TAIL_REMOVE) {
        PollItem pi = poll_item(m, x.list_a, T.tid, na);
        const ConfItem ci = conf_item(m, x.list_a, T.n - 1 - T.tid, na);
        const LabelItem li = label_item(m, x.list_a, label_start(T), na);
        const int nfail = poll_loop(m, x, T, pg, cap, pi);
        if (na > 0 || nfail > 0) {
            if (na > 0) conflict_check(m, T, x.list_a, na, ci);
            T.sync();
            if (na > 0) conflict_unlabel(m, T, x.list_a, na, pi);
            poll_reset(m, x, T, pg, nfail);
            T.sync();
        }
        const bool pairs = *x.n_b > 0;
        if (pairs) two_three_loop(m, x, T, S);
        if (na > 0) {
            label3_reserve(m, x, T, na, dt, pairs ? nullptr : &li);
            if (T.tid == 0) *x.n_ehits = 0;          /* the grains a 2x3 pass left with three sides */
            T.sync();
        }
        const int nc = na > 0 && !(PART & TAIL_SPREAD) ? *x.n_c : 0;
        if (nc > 0) {
            remove_apply(m, x, T, x.list_c, nc);
            T.sync();
            const int nd = *x.n_ehits;
            if (nd > 0) {
                run_deferred(m, x, T, nd, m.goff, [&](int g, int inst) { remove_warp(m, g, inst, T.lane); });
                T.sync();
            }
            if (PART & TAIL_END) fix_lists(m, T, S, x.list_c, nc, true, nullptr, nullptr);
        }
    }
    if ((PART & TAIL_FLIP) && !(PART & TAIL_END)) {
        /* the rest of the removals' fix-up, after k_edit */
        const bool queued = *m.nfix > 0 || *m.nmod > 0;
        if (queued) {
            clear_mods(m, T.tid, T.n);
            T.sync();
            if (T.tid == 0) *m.nfix = *m.nmod = 0;
            T.sync();
        }
    }
    if ((PART & TAIL_FLIP) && na > 0) {
        flip_reserve(m, x, T, x.list_a, na);
        if (PART & TAIL_SPREAD) return;
        T.sync();
        flip_apply(m, x, T, x.list_a, na, eps);
        T.sync();
        const int nd = *x.n_ehits;
        if (nd > 0) {
            run_deferred(m, x, T, nd, m.boff, [&](int b, int) { flip_warp(m, b, eps, T.lane); });
            T.sync();
        }
    }
    if (PART & TAIL_END) {
        fix_lists(m, T, S, nullptr, 0, false, nullptr, nullptr);
        /* the counts were zeroed before the last sync unless no candidate
         * made one necessary */
        if (na == 0) T.sync();
        for (int v = T.tid; v < m.nv; v += T.n) update_vertex(m, v, dt);
        count_grains(m, x.counters, T.tid, T.n);
        nucl_area_blocks(m, x.block_area, pg.blocks, pg.tpb, blockIdx.x, gridDim.x);
        /* without nucleated grains (a plain handle) there is nothing to wait for */
        const bool nucleated = m.ninst > 1 || m.nnlist[0] > 0;
        if (nucleated) T.sync();
        nucl_area_final(m, x.block_area, pg.blocks, x.counters, T.tid, T.n);
        T.sync();
        pack_summary(m, x, summary, T.tid, T.n);
    }
}

/* The events behind their reservations, over the whole GPU: those that hold
 * their records, a warp each, then (one cluster) the deferred ones.  For steps
 * of many events (see DENSE_EVENTS): the cluster's 256 warps take 10,400
 * removals and 12,700 flips in rounds, 760 and 600 us with their fix-ups, and
 * such a step of 256 meshes (1.28M grains) went from 3.13 ms to 2.36. */
constexpr int APPLY_TPB = 256, APPLY_BLOCKS = 2 * WL_BLOCKS;
template <bool FLIPS>
__global__ void __launch_bounds__(APPLY_TPB) k_apply(DevMesh m, DevScratch x, double eps)
{
    griddep_wait();
    const Team T;
    if (FLIPS) flip_apply(m, x, T, x.list_a, *x.n_a, eps);
    else remove_apply(m, x, T, x.list_c, *x.n_c);
}
template <bool FLIPS>
__global__ void __launch_bounds__(TAIL_TPB) k_deferred(DevMesh m, DevScratch x, double eps)
{
    griddep_wait();
    const Team T;
    /* without candidates n_ehits still counts the 2x3 loop's list */
    const int nd = *x.n_a > 0 ? *x.n_ehits : 0;
    if (nd == 0) return;
    if (FLIPS) run_deferred(m, x, T, nd, m.boff, [&](int b, int) { flip_warp(m, b, eps, T.lane); });
    else run_deferred(m, x, T, nd, m.goff, [&](int g, int inst) { remove_warp(m, g, inst, T.lane); });
}

/* edit_grains over the whole GPU, after the removals (REMOVED) or the
 * flips; the clearing of the mods is left to the next kernel, TAIL_FLIP or
 * k_update.  With 70 removals and 50 flips a step (100K grains) some 300
 * grains are edited after each, with 200 and 350 (400K grains) some 1,000,
 * and the cluster's sixteen SMs took 60 and 93 thousand cycles over the
 * first, 60 and 110 over the second, bound by their FP64 pipes and by the
 * rounds of 256 warps; a launch costs some 3. */
constexpr int EDIT_TPB = 256;
template <bool REMOVED>
__global__ void __launch_bounds__(EDIT_TPB) k_edit(DevMesh m, DevScratch x)
{
    griddep_wait();
    __shared__ EditShared<EDIT_TPB / 32> S;
    const Team T;
    edit_grains(m, T, S, x.list_c, REMOVED ? *x.n_c : 0, REMOVED, nullptr, nullptr);
}
/* the position update and the rest of the flips' fix-up */
__global__ void __launch_bounds__(TPB) k_update(DevMesh m, double dt)
{
    griddep_wait();
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t < m.nv) update_vertex(m, t, dt);
    clear_mods(m, t, gridDim.x * blockDim.x);
}

/* instance of every boundary and grain from the offset tables */
__global__ void k_fill_instance_ids(DevMesh m)
{
    int stride = gridDim.x * blockDim.x;
    for (int b = blockIdx.x * blockDim.x + threadIdx.x; b < m.nb; b += stride)
        m.binst[b] = lower_bound_i(m.boff, m.ninst + 1, b + 1) - 1;
    for (int g = blockIdx.x * blockDim.x + threadIdx.x; g < m.ng; g += stride)
        m.ginst[g] = lower_bound_i(m.goff, m.ninst + 1, g + 1) - 1;
}

/* k as one cluster, after the previous kernel of the stream (or without
 * programmatic serialisation, see launch_dep) */
template <typename... P, typename... A>
void launch_cluster(void (*k)(P...), cudaStream_t s, A &&...args)
{
    cudaFuncSetAttribute(k, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
    cudaLaunchAttribute at[2];
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = TAIL_BLOCKS;
    at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
    at[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[1].val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = TAIL_BLOCKS;
    cfg.blockDim = TAIL_TPB;
    cfg.stream = s;
    cfg.attrs = at;
    bool plain = sevc_pdl_skip > 0;
    if (sevc_pdl_skip > 0) sevc_pdl_skip--;
    cfg.numAttrs = plain ? 1 : 2;
    COUNT_LAUNCHES(1);
    cudaLaunchKernelEx(&cfg, k, static_cast<A &&>(args)...);
}
template <int PART>
void launch_tail_part(const DevMesh &m, const DevScratch &x, const StepParams &p, int cap, int *summary, cudaStream_t s)
{
    launch_cluster(k_tail<PART>, s, m, x, poll_grid(p), cap, p.dt, p.eps, summary);
}

} // namespace

PollGrid poll_grid(const StepParams &p)
{
    PollGrid g;
    g.blocks = p.n_blocks;
    g.tpb = p.n_threads;
    g.counting = 0;
    for (int t = 0; t < g.tpb; t++) g.counting += PollGrid::counts(t, g.tpb);
    return g;
}

void launch_two_three_first(const DevMesh &m, const DevScratch &x, cudaStream_t s)
{
    /* nine threads per 3-sided grain, of which there are a few percent */
    int g = (m.ng + TPB - 1) / TPB;
    COUNT_LAUNCHES(1), k_two_three_first<<<g < 4 * WL_BLOCKS ? g : 4 * WL_BLOCKS, TPB, 0, s>>>(m, x);
}
bool tail_whole(const DevMesh &m) { return m.nv <= TAIL_WHOLE_NV; }
void launch_tail_whole(const DevMesh &m, const DevScratch &x, const StepParams &p, int cap, int *summary, cudaStream_t s)
{
    launch_tail_part<TAIL_REMOVE | TAIL_FLIP | TAIL_END>(m, x, p, cap, summary, s);
}
void launch_tail_removals(const DevMesh &m, const DevScratch &x, const StepParams &p, int cap, bool dense, cudaStream_t s)
{
    if (dense) {
        launch_tail_part<TAIL_REMOVE | TAIL_SPREAD>(m, x, p, cap, nullptr, s);
        launch_dep(k_apply<false>, APPLY_BLOCKS, APPLY_TPB, s, m, x, p.eps);
        launch_cluster(k_deferred<false>, s, m, x, p.eps);
    } else {
        launch_tail_part<TAIL_REMOVE>(m, x, p, cap, nullptr, s);
    }
    launch_dep(k_edit<true>, WL_BLOCKS, EDIT_TPB, s, m, x);
}
void launch_tail_flips(const DevMesh &m, const DevScratch &x, const StepParams &p, bool dense, cudaStream_t s)
{
    if (dense) {
        launch_tail_part<TAIL_FLIP | TAIL_SPREAD>(m, x, p, 0, nullptr, s);
        launch_dep(k_apply<true>, APPLY_BLOCKS, APPLY_TPB, s, m, x, p.eps);
        launch_cluster(k_deferred<true>, s, m, x, p.eps);
    } else {
        launch_tail_part<TAIL_FLIP>(m, x, p, 0, nullptr, s);
    }
    launch_dep(k_edit<false>, WL_BLOCKS, EDIT_TPB, s, m, x);
}
void launch_update_positions(const DevMesh &m, double dt, cudaStream_t s)
{
    launch_dep(k_update, (m.nv + TPB - 1) / TPB, TPB, s, m, dt);
}

void launch_fill_instance_ids(const DevMesh &m, cudaStream_t s)
{
    COUNT_LAUNCHES(1), k_fill_instance_ids<<<4 * WL_BLOCKS, TPB, 0, s>>>(m);
}
