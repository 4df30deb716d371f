/*
 * Geometry and kinetics kernels of one time step (src/calculus.h and
 * src/topological.h:303-353 of the reference): blocks of grains in the
 * grain pass, one thread or six lanes per vertex, one thread per boundary.
 *
 * The finite-difference velocity (src/calculus.h:19-73,143-154) is split
 * in two passes so that no thread re-reads another grain's polygon:
 *   grain pass   for every grain: its area, and for every list slot p the
 *                areas with that vertex moved by +eps in x and in y; the
 *                stored-energy terms SE*(|A'|-|A|) are scattered to the
 *                vertex's grain slot;
 *   vertex pass  for every vertex: the three perturbed arclengths, the
 *                boundary terms, the velocity, and the vertex energy.
 * Both passes repeat the reference's arithmetic in the same order, so the
 * results are the ones energy_diff computes.
 */
#include "sevc_tail.cuh"

#include <algorithm>
#include <cmath>
#include <cstring>

namespace {

constexpr int TPB = 256;
inline int nblk(int n) { return (n + TPB - 1) / TPB; }

/* src/calculus.h:83-114 */
__global__ void k_boundary_geometry(DevMesh m, double eps, double scaling)
{
    int b = blockIdx.x * blockDim.x + threadIdx.x;
    if (b >= m.nb || !m.ben[b]) return;
    int2 e = m.bv[b];
    double2 a = m.pos[e.x], c = m.pos[e.y];
    m.blen[b] = arclen(a, c, m.D);
    double gamma;
    if (!boundary_gamma(m, b, eps, scaling, gamma)) { raise_err(m, ERRB_TOPOLOGY); return; }
    m.benergy[b] = gamma;
}

/* Store the stored-energy finite-difference terms of list vertex v
 * (SE * (|A'| - |A|), src/calculus.h:60) in v's slot for grain g. */
__device__ __forceinline__ void put_contrib(const DevMesh &m, int g, int v, double se, double absA, double Ax,
                                           double Ay)
{
    int4 sg = m.vg[v];
    int j = sg.x == g ? 0 : (sg.y == g ? 1 : (sg.z == g ? 2 : -1));
    if (j >= 0) m.contrib[3 * v + j] = make_double2(se * (dabs(Ax) - absA), se * (dabs(Ay) - absA));
}

/* ------------------------------------------------------------------ */
/* grain pass                                                          */
/* ------------------------------------------------------------------ */
/* Every grain's area and the areas with each list vertex moved by +eps in
 * x and in y (compute_area of the polygon with vertex p moved, src/
 * geometry.h:757, :908), bit for bit.
 *
 * Certificate.  Let u be the ulp of a grain's smallest coordinate along an
 * axis, Rmin.  When every coordinate lies in [Rmin, 1.75 Rmin] (and below
 * Dlim, and no coordinate + eps leaves its binade), all coordinates are
 * multiples of u, no wrap occurs, and every wrapped delta, unwrapped
 * coordinate and moved coordinate the reference forms is a multiple of u
 * below 2^53 u: each of those additions and subtractions is exact.  So the
 * unwrapped coordinate of vertex k is R[k] - R[0] in one subtraction; the
 * moved vertex's is A[p] + d_p and, for p = 0, every later one A[k] - d_0,
 * where d_p = RN(R[p] + eps) - R[p] depends on R[p]'s exponent only (the
 * multiple of ulp(R[p]) nearest to eps; eps is never halfway); and the moved
 * chain is back on the unmoved values from p + 1 on.  Only the products,
 * the shoelace terms and their running sum round, and those are formed in
 * the reference's order.  On 1M grains (domain 1000) about 0.4% of the
 * grains fail the certificate (next to an axis, where ulps are finer, or
 * across the wrap); their chains are formed as written, the slots of a block's together
 * (moved_uncertified).
 *
 * What bounds it: the FP64 pipe (2 thread-operations per clock and SM, of
 * which independent chains reach 84%) together with the latency of the
 * phases below.  The certificate leaves 109 FP64 operations per grain (234
 * when the chains are recomputed): the integer pipe forms the exact
 * differences, and the product of the stored energy with an area difference
 * (mul_diff).  Forming the shoelace products on the integer pipe as well
 * gained nothing (389 us with all of them, 378 with half).
 *
 * Layout.  A block takes GPB consecutive grains, orders them by falling
 * side count in shared memory (no order over the whole mesh is needed), and
 * works on chunks of 32 of them in loops over shared memory:
 *   per slot            position and grain-slot loads;
 *   per grain, axis     certificate;
 *   per slot, axis      coordinates relative to vertex 0, and to vertex 0
 *                       moved;
 *   per slot, polygon   shoelace products and terms (the unmoved polygon
 *                       and the two with vertex 0 moved);
 *   per grain, polygon  running sum, area;
 *   per slot, axis      the area with its vertex moved: the slots in falling
 *                       number s = n - 2 - p of terms behind them (those of
 *                       one s are a prefix of the order), so that the lanes
 *                       of a warp run the same operations.
 * Afterwards a warp per grain takes the rest, vertex by vertex: grains of
 * `wide` or more sides or of fewer than 3, and those with a coordinate
 * outside the domain or + eps in the next binade.
 *
 * Measured (GB300): 1M grains 0.368 ms, FP64 pipe active 69% of the
 * cycles, 22 of 32 lanes per FP64 instruction (slots of different s or p in
 * one warp); 2,000 grains 15 us.  The form before it (a grain per thread,
 * polygon in registers, one unrolled body per side count, side-count order
 * of the whole mesh first, warp-per-grain kernel for 11 sides and more)
 * took 0.50 ms and 95 us: on a small mesh each unrolled body runs once and
 * its instruction fetch is the time. */
constexpr int GP_NMAX = 32;              /* side counts below this may take the ordered path (bits of AxisCert::up, lanes) */
constexpr int GP_E0 = 1023 - 20, GP_E1 = 1023 + 20;   /* biased exponents of certified coordinates */

/* significand of eps = 1e-8 = GP_EPS_M 2^(GP_EPS_E - 1075) */
#define GP_EPS_M 0x15798ee2308c3aLL
#define GP_EPS_E (1023 - 27)

/* 1/n as a pair (hi, lo) for the division below; 4 and 8 are exact */
#define INV_SPLIT(n) { InvSplit<n>::hi, InvSplit<n>::lo }
__constant__ double2 c_inv_split[11] = { { 0, 0 }, { 0, 0 }, { 0, 0 }, INV_SPLIT(3), { 0.25, 0.0 }, INV_SPLIT(5),
                                         INV_SPLIT(6), INV_SPLIT(7), { 0.125, 0.0 }, INV_SPLIT(9), INV_SPLIT(10) };

/* x / n for a side count n: a multiplication and an fma where the bound of
 * InvSplit holds, else the division */
__device__ __forceinline__ double div_sides(double x, int n)
{
    unsigned long long b = mag2(x);
    if (n >= 3 && n <= 10 && b >= (0x07B0000000000000ULL << 1) && b < (0x7830000000000000ULL << 1)) {
        double2 z = c_inv_split[n];
        return __fma_rn(x, z.x, __dmul_rn(x, z.y));
    }
    return ddiv_slow(x, (double)n);
}

static __device__ __noinline__ double mul_diff_slow(double se, double x, double y) { return se * (x - y); }
/* se * (x - y) for x, y >= 0 (src/calculus.h:60), each operation rounded, on
 * the integer pipe when x and y lie in one binade and differ by less than
 * 2^31 ulps: the difference is then k ulps exactly, and the product of k
 * and se's significand, a 96-bit integer, is rounded to nearest even. */
__device__ __forceinline__ double mul_diff(double se, double x, double y)
{
    const long long bx = dbits(x), by = dbits(y), k = bx - by, bs = dbits(se);
    const int E = (int)(by >> 52), es = (int)((bs >> 52) & 0x7ff);
    const unsigned a = (unsigned)((int)k < 0 ? -(int)k : (int)k);
    const int lz = __clz((int)a);
    int eb = 32 - lz + E + es - 1075;
    const unsigned hi_sign = ((unsigned)k ^ (unsigned)((unsigned long long)bs >> 32)) & 0x80000000u;
    /* one binade, k in 32 bits and not 0 or INT_MIN, se and the result well
     * inside the normal range */
    if ((int)(bx >> 52) != E || k != (long long)(int)k || a == 0 || a >> 31 || es == 0 || es == 0x7ff || E == 0 ||
        eb < 2 || eb > 2045)
        return mul_diff_slow(se, x, y);
    const unsigned ka = a << lz;
    const unsigned long long M = (((unsigned long long)bs & 0x000FFFFFFFFFFFFFULL) | (1ULL << 52)) << 11;
    const unsigned long long p0 = (unsigned long long)ka * (unsigned)M, p1 = (unsigned long long)ka * (unsigned)(M >> 32);
    unsigned long long h = p1 + (p0 >> 32);            /* bits 32 .. 95 of the product, its leading one at 95 or 94 */
    unsigned l = (unsigned)p0;
    if (!(h >> 63)) {
        h = (h << 1) | (l >> 31);
        l <<= 1;
        eb--;
    }
    unsigned long long q = h >> 11;
    const unsigned r = (unsigned)h & 0x7ffu;
    q += r > 0x400u || (r == 0x400u && (l != 0 || (q & 1)));
    const unsigned long long bits = ((unsigned long long)(eb - 1) << 52) + q;     /* a carry out of q raises the exponent */
    return __longlong_as_double((long long)(bits | ((unsigned long long)hi_sign << 32)));
}

/* area_stream over a polygon staged in shared memory (raw positions P[k]
 * of vertex k), same operations in the same order. */
__device__ __forceinline__ double area_shared(const double2 *P, int n, int ps, double2 pp, double D)
{
    double area = 0;
    if (n > 0) {
        double2 r0 = (ps == 0) ? pp : P[0];
        double ax = 0, ay = 0, rx = r0.x, ry = r0.y;
        for (int k = 1; k < n; k++) {
            double2 r = (k == ps) ? pp : P[k];
            double nx = ax + wrapd(r.x, rx, D);
            double ny = ay + wrapd(r.y, ry, D);
            if (k > 1) area += ax * ny - ay * nx;
            ax = nx; ay = ny; rx = r.x; ry = r.y;
        }
        area = add_closing_term(area, ax, ay);
    }
    return dscale_down<1>(area);
}

/* grain g by one warp, polygon staged in shared memory.  The 2n+1
 * areas (vertex p moved along x: task 2p, along y: task 2p+1, unmoved:
 * task 2n) are spread over the lanes, so a grain of up to 15 sides costs one
 * polygon walk per lane. */
__device__ __noinline__ void grain_by_warp(const DevMesh &m, int g, double2 *P, double *R, int lane)
{
    const double D = m.D;
    const int *L = m.glist + (size_t)SEVC_MAXV * g;
    int n = m.gvlen[g];
    for (int k = lane; k < n; k += 32) P[k] = m.pos[L[k]];
    __syncwarp();
    for (int t = lane; t <= 2 * n; t += 32) {
        int p = t >> 1;
        double2 pp = make_double2(0, 0);
        if (t < 2 * n) {
            double2 q = P[p];
            pp = (t & 1) ? make_double2(dmod(q.x, D), dmod(q.y + SEVC_GRAD_EPS_D, D))
                         : make_double2(dmod(q.x + SEVC_GRAD_EPS_D, D), dmod(q.y, D));
        } else {
            p = -1;
        }
        R[t] = area_shared(P, n, p, pp, D);
    }
    __syncwarp();
    double A = R[2 * n];
    double se = m.gse[g];
    if (lane == 0) {
        m.garea[g] = A;
        m.gq[g] = se * A / n;
    }
    double absA = dabs(A);
    for (int p = lane; p < n; p += 32) put_contrib(m, g, L[p], se, absA, R[2 * p], R[2 * p + 1]);
    __syncwarp();
}

/* one axis of a grain: the exponent of its smallest coordinate (index into
 * the tables) and the mask of the vertices one binade above it */
struct AxisCert { int e; unsigned up; };
enum { GP_REST = 0, GP_CERT = 1, GP_CHAIN = 2 };

constexpr int GP_CHUNK = 32;
template <int SLOTS> struct GrainChunk {
    double R[2][SLOTS];                        /* raw coordinates; then the terms k of the polygons with vertex 0 moved */
    double A[2][SLOTS];                        /* unwrapped coordinates */
    double M[2][SLOTS];                        /* the same with vertex 0 moved along the axis; then M[0]: sum of T up to k */
    double Q[2][SLOTS], T[SLOTS];              /* A[0][k] A[1][k+1], A[1][k] A[0][k+1], their difference */
    int dest[SLOTS];                           /* 3 v + grain slot */
    unsigned short moved[SLOTS], inner[SLOTS]; /* the slots in the order they are worked on */
    unsigned char owner[SLOTS];
    double se[GP_CHUNK], area[GP_CHUNK], sum0[2][GP_CHUNK];   /* sum0: twice the areas with vertex 0 moved */
    int sg[GP_CHUNK];
    unsigned short off[GP_CHUNK];              /* first slot */
    unsigned char n[GP_CHUNK];
    int ok[2][GP_CHUNK];                       /* GP_* of each axis */
    AxisCert c[2][GP_CHUNK];
    __device__ int state(int i) const          /* certified, walked as a chain, or left to the rest */
    {
        int x = ok[0][i], y = ok[1][i];
        return x && y ? (x > y ? x : y) : GP_REST;
    }
};
struct GrainRest { double2 P[SEVC_MAXV]; double R[2 * SEVC_MAXV + 1]; };   /* one per warp */
template <int NT, int SLOTS> struct GrainSmem {
    static constexpr size_t rest = sizeof(GrainRest) * (NT / 32), chunk = sizeof(GrainChunk<SLOTS>);
    static constexpr size_t bytes = chunk > rest ? chunk : rest;
};
/* d 2^(e - 1075) for |d| < 2^53: exact, on the integer pipe */
__device__ __forceinline__ double grid_value(long long d, int e)
{
    const unsigned long long u = (unsigned long long)(d < 0 ? -d : d);
    const int sh = __clzll((long long)u) - 11;
    const unsigned long long r = ((unsigned long long)(e - 1 - sh) << 52) + (u << sh);
    return d == 0 ? 0.0 : __longlong_as_double((long long)(r | ((unsigned long long)d & 0x8000000000000000ULL)));
}
/* a - b for positive binary64 patterns whose exponents are e or e + 1 and
 * whose difference is below 2^53 times 2^(e - 1075) */
__device__ __forceinline__ double sub_exact(long long a, long long b, int e)
{
    const long long M = 0x000FFFFFFFFFFFFFLL, H = 1LL << 52;
    const long long ma = ((a & M) | H) << ((int)(a >> 52) - e), mb = ((b & M) | H) << ((int)(b >> 52) - e);
    return grid_value(ma - mb, e);
}
/* a + n 2^(e - 1075) for a multiple a of 2^(e - 1075), |a| < 2^53 times it */
__device__ __forceinline__ double add_exact(double a, long long n, int e)
{
    const long long b = dbits(a);
    const int ea = (int)((b >> 52) & 0x7ff);
    long long m = ((b & 0x000FFFFFFFFFFFFFLL) | (1LL << 52)) >> (ea ? e - ea : 63);
    return grid_value((b < 0 ? -m : m) + n, e);
}

/* certificate of one axis over the raw coordinates r[0..n); that no
 * coordinate + eps leaves its binade is checked slot by slot.  A grain
 * with a coordinate outside [0, D) takes the rest's path. */
__device__ __forceinline__ int certify_axis(const double *r, int n, double D, long long dlim, AxisCert &c)
{
    long long lo = dbits(r[0]), hi = lo;
    for (int k = 1; k < n; k++) {
        long long b = dbits(r[k]);
        lo = b < lo ? b : lo;
        hi = b > hi ? b : hi;
    }
    int e = (int)(lo >> 52), e1 = (int)(hi >> 52);
    c.e = e - GP_E0;
    c.up = 0;
    if (lo < 0 || hi >= dbits(D)) return GP_REST;
    if (e < GP_E0 || e1 > GP_E1 || e1 > e + 1 || hi >= dlim) return GP_CHAIN;
    long long ml = (lo & 0x000FFFFFFFFFFFFFLL) | (1LL << 52), mh = ((hi & 0x000FFFFFFFFFFFFFLL) | (1LL << 52)) << (e1 - e);
    return mh - ml <= (ml >> 1) + (ml >> 2) ? GP_CERT : GP_CHAIN;
}

/* Twice the area with the vertex of slot q (not the grain's first) of an
 * uncertified grain moved along axis x, up to its sign (see the moved areas
 * of certified grains below): the chain is formed as the reference does from
 * the moved vertex on, and when it does not come back to the unmoved value at
 * the next vertex, bit for bit, it is walked to its end.  Some 10% of the
 * grains of a 2,000-grain mesh are uncertified (next to the axes and across
 * the wrap) and most of them have such a slot; a warp that walked all
 * 2 n + 1 polygons of each, and chains formed among the certified slots, where
 * a warp waits for one lane, made the pass of 64 meshes of that size (176,000
 * grains) 171 us; with their slots packed into whole warps it took 129 us. */
template <int SLOTS>
__device__ __forceinline__ double moved_uncertified(const DevMesh &m, const GrainChunk<SLOTS> &B, int q, int x)
{
    const int i = B.owner[q], o = B.off[i], p = q - o, nn = B.n[i];
    const double *F = B.A[x], *G = B.A[1 - x];
    auto raw = [&](int k) { return reinterpret_cast<const double *>(m.pos + B.dest[k] / 3)[x]; };
    const long long flip = x ? LLONG_MIN : 0;
    auto sgn = [&](double v) { return __longlong_as_double(dbits(v) ^ flip); };
    const double D = m.D, rm = raw(q - 1), mv = dmod(raw(q) + SEVC_GRAD_EPS_D, D), w = wrapd(mv, rm, D);
    double r = raw(p < nn - 1 ? q + 1 : q);
    const double f = p == 1 ? zero_plus(w) : F[q - 1] + w;
    double a = 0;
    if (p >= 2) {
        a = B.Q[x][q - 1] - G[q - 1] * f;                      /* term p - 1 */
        if (p > 2) a = sgn(B.M[0][q - 2]) + a;
    }
    if (p < nn - 1) {
        double g = f + wrapd(r, mv, D);                        /* the next vertex's coordinate */
        const bool joins = dbits(g) == dbits(F[q + 1]);
        const double t2 = f * G[q + 1] - G[q] * g;             /* term p */
        a = p == 1 ? t2 : a + t2;
        for (int k = q + 1; k < o + nn - 1; k++) {
            if (joins) {
                a = a + sgn(B.T[k]);
            } else {
                const double s = raw(k + 1), h = g + wrapd(s, r, D);
                a = a + (g * G[k + 1] - G[k] * h);
                g = h;
                r = s;
            }
        }
    }
    return a;
}

/* the listed slots (2 slot + axis); a call, so that its registers do not
 * spill the certified slots' */
template <int NT, int SLOTS>
__device__ __noinline__ void moved_uncertified_all(const DevMesh &m, const GrainChunk<SLOTS> &B, const unsigned short *odd,
                                                   int nodd)
{
    for (int t = threadIdx.x; t < nodd; t += NT) {
        const int x = odd[t] & 1, q = odd[t] >> 1, i = B.owner[q];
        const double a = moved_uncertified(m, B, q, x);
        reinterpret_cast<double *>(m.contrib + B.dest[q])[x] = mul_diff(B.se[i], dabs(dscale_down<1>(a)), dabs(B.area[i]));
    }
}

template <int GPB, int NT, int SLOTS>
__global__ void __launch_bounds__(NT, SLOTS == 208 ? 11 : 1) k_grain_pass(DevMesh m, int *three, int *n_three, int wide, long long dlim)
{
    __shared__ __align__(16) unsigned char smem[GrainSmem<NT, SLOTS>::bytes];
    GrainChunk<SLOTS> &B = *reinterpret_cast<GrainChunk<SLOTS> *>(smem);
    __shared__ int order[GPB];                 /* the block's grains by falling side count */
    __shared__ unsigned char sides[GPB];
    __shared__ int cnt[GP_NMAX], start[GP_NMAX];
    __shared__ int first[GP_NMAX];             /* first[j]: first entry of B.moved (and B.inner) with s + 2 = j */
    __shared__ int rest[GPB], nrest, listed, chunk, slots, nmoved, chains, nodd;
    __shared__ long long ntab[GP_E1 - GP_E0 + 1];
    constexpr int W = NT / 32;
    static_assert(GPB <= NT, "a thread per grain orders them");
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int g = blockIdx.x * GPB + tid;
    bool on = tid < GPB && g < m.ng;
    int n = 0, r = 0;
    if (on) {
        uint8_t en = m.gen[g];
        n = m.gvlen[g];
        on = en;
    }
    if (tid < GP_NMAX) cnt[tid] = 0;
    if (tid == 0) nrest = 0;
    for (int t = tid; t <= GP_E1 - GP_E0; t += NT) {
        /* RN(eps / ulp) for coordinates of this exponent */
        const int d = t + GP_E0 - GP_EPS_E;
        ntab[t] = (GP_EPS_M + (1LL << (d - 1))) >> d;
    }
    __syncthreads();
    /* the block's grains by falling side count */
    if (on) {
        if (n == 3) three[atomicAdd(n_three, 1)] = g;
        if (n < 3 || n >= wide || n >= GP_NMAX) {
            rest[atomicAdd(&nrest, 1)] = g;
            on = false;
        } else {
            r = atomicAdd(&cnt[n], 1);
        }
    }
    __syncthreads();
    if (warp == 0) {
        const int k = GP_NMAX - 1 - lane, c = cnt[k];
        int a = c;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            int y = __shfl_up_sync(0xffffffffu, a, o);
            if (lane >= o) a += y;
        }
        start[k] = a - c;                      /* grains of more than k sides */
        if (k == 0) listed = a;
    }
    __syncthreads();
    if (on) {
        order[start[n] + r] = g;
        sides[start[n] + r] = (unsigned char)n;
    }
    __syncthreads();
    /* chunks of up to 32 grains (and SLOTS list slots) of the order */
    for (int c0 = 0; c0 < listed;) {
    if (warp == 0) {
        const int i = c0 + lane, k = i < listed ? sides[i] : 0;
        int o = k;
#pragma unroll
        for (int d = 1; d < 32; d <<= 1) {
            int y = __shfl_up_sync(0xffffffffu, o, d);
            if (lane >= d) o += y;
        }
        const bool in = k > 0 && o <= SLOTS;
        const int c = __popc(__ballot_sync(0xffffffffu, in));
        o -= k;
        if (in) {
            const int gi = order[i];
            B.sg[lane] = gi;
            B.n[lane] = (unsigned char)k;
            B.off[lane] = (unsigned short)o;
            for (int j = 0; j < k; j++) B.owner[o + j] = (unsigned char)lane;
            if (lane == c - 1) { slots = o + k; chunk = c; }
        }
        /* class of s = q - 3: one slot of each grain of q or more sides */
        const int q = GP_NMAX - 1 - lane;
        int ge = (q > 0 ? start[q - 1] : listed) - c0;
        ge = ge < 0 ? 0 : (ge < c ? ge : c);
        int f = ge;
#pragma unroll
        for (int d = 1; d < 32; d <<= 1) {
            int y = __shfl_up_sync(0xffffffffu, f, d);
            if (lane >= d) f += y;
        }
        f -= ge;
        if (q >= 1) first[q - 1] = f;          /* j = s + 2 = q - 1; q = 2, 1: p = n - 1 and p = 0, every grain */
        else nmoved = f;
    } else if (warp == W - 1) {
        if (c0 + lane < listed) B.se[lane] = m.gse[order[c0 + lane]];
    }
    __syncthreads();
    const int total = chunk;                   /* read here: warp 0 sets the next chunk's behind the last barrier */
    /* per slot: position, where the vertex keeps this grain's terms, places
     * in the work orders */
#pragma unroll 2
    for (int q = tid; q < slots; q += NT) {
        const int i = B.owner[q], k = q - B.off[i], nn = B.n[i], gi = B.sg[i];
        const int v = m.glist[(size_t)SEVC_MAXV * gi + k];
        const double2 p = m.pos[v];
        const int4 sv = m.vg[v];
        B.moved[first[k == 0 ? 0 : nn - k] + i] = (unsigned short)q;
        if (k > 0 && k < nn - 1) B.inner[first[k + 1] + i] = (unsigned short)q;
        const int w = sv.x == gi ? 0 : (sv.y == gi ? 1 : (sv.z == gi ? 2 : -1));
        B.R[0][q] = p.x;
        B.R[1][q] = p.y;
        B.dest[q] = w >= 0 ? 3 * v + w : -1;
    }
    __syncthreads();
    /* per grain and axis: certificate */
    if (tid == 0) chains = nodd = 0;
    for (int t = tid; t < 2 * total; t += NT) {
        const int x = t >= total, i = x ? t - total : t;
        B.ok[x][i] = certify_axis(B.R[x] + B.off[i], B.n[i], m.D, dlim, B.c[x][i]);
    }
    __syncthreads();
    /* per slot and axis: coordinate relative to vertex 0, and to vertex 0
     * moved; of an uncertified grain the wrapped deltas that its chains add
     * up, each as the reference forms it */
    for (int t = tid; t < 2 * slots; t += NT) {
        const int x = t >= slots, q = x ? t - slots : t, i = B.owner[q], o = B.off[i], st = B.state(i);
        if (B.dest[q] < 0) B.ok[0][i] = GP_REST;
        if (st == GP_CERT) {
            const int e = B.c[x][i].e;
            const long long b = dbits(B.R[x][q]), b0 = dbits(B.R[x][o]);
            const int u = (int)(b >> 52) - GP_E0;
            if (((b + ntab[u]) ^ b) >> 52) B.ok[0][i] = GP_REST;
            if (u != e) atomicOr(&B.c[x][i].up, 1u << (q - o));
            B.A[x][q] = sub_exact(b, b0, e + GP_E0);
            B.M[x][q] = sub_exact(b, b0 + ntab[(int)(b0 >> 52) - GP_E0], e + GP_E0);
        } else if (st == GP_CHAIN) {
            chains = 1;
            const double rk = B.R[x][q];
            const double d = q == o ? 0.0 : wrapd(rk, B.R[x][q - 1], m.D);
            B.A[x][q] = d;
            B.M[x][q] = q == o + 1 ? zero_plus(wrapd(rk, dmod(B.R[x][o] + SEVC_GRAD_EPS_D, m.D), m.D)) : d;
        }
    }
    __syncthreads();
    if (chains) {                              /* the block has uncertified grains: their running sums */
        for (int t = tid; t < 4 * total; t += NT) {
            const int i = t >> 2, c = t & 3, o = B.off[i], nn = B.n[i];
            if (B.state(i) != GP_CHAIN) continue;
            double *Z = (c < 2 ? B.A[c] : B.M[c - 2]) + o, a = c < 2 ? zero_plus(Z[1]) : Z[1];
            Z[1] = a;
            for (int k = 2; k < nn; k++) Z[k] = a = a + Z[k];
        }
        __syncthreads();
    }
    /* per slot 0 < k < n - 1 (by falling k, those of one k a prefix of the
     * order) and polygon (unmoved, vertex 0 moved along x, along y): the
     * shoelace products and their difference.  Along y the difference has
     * the opposite sign: only magnitudes of moved areas are used. */
    const int ninner = first[1];
    for (int t = tid; t < 3 * ninner; t += NT) {
        const int c = t >= 2 * ninner ? 2 : (t >= ninner ? 1 : 0), q = B.inner[t - c * ninner];
        const double *F = c == 0 ? B.A[0] : B.M[c - 1], *G = c == 2 ? B.A[0] : B.A[1];
        const double q1 = F[q] * G[q + 1], q2 = G[q] * F[q + 1], d = q1 - q2;
        if (c == 0) {
            B.Q[0][q] = q1;
            B.Q[1][q] = q2;
            B.T[q] = d;
        } else {
            B.R[c - 1][q] = d;
        }
    }
    __syncthreads();
    /* per grain and polygon: the running sum; of the unmoved one, the area.
     * (Sums that only a magnitude is taken of leave out the reference's
     * 0.0 + first term and its closing +-0: those change the sign of a zero
     * at most.)  A grain's three sums lie side by side, so a warp's grains have
     * like numbers of sides: with a polygon per warp each waited for the
     * chunk's longest list (380 against 368 us at 1M grains). */
    for (int t = tid; t < 3 * total; t += NT) {
        const int i = t / 3, c = t - 3 * i, o = B.off[i], nn = B.n[i];
        if (B.state(i) == GP_REST) {
            if (c == 0) rest[atomicAdd(&nrest, 1)] = B.sg[i];
            continue;
        }
        const double *Z = c == 0 ? B.T : B.R[c - 1];
        double acc = zero_plus(Z[o + 1]);
        if (c == 0) B.M[0][o + 1] = acc;
        for (int k = 2; k < nn - 1; k++) {
            acc = acc + Z[o + k];
            if (c == 0) B.M[0][o + k] = acc;
        }
        if (c == 0) {
            acc = add_closing_term(acc, B.A[0][o + nn - 1], B.A[1][o + nn - 1]);
            const double A = dscale_down<1>(acc);
            B.area[i] = A;
            m.garea[B.sg[i]] = A;
        } else {
            B.sum0[c - 1][i] = acc;
        }
    }
    __syncthreads();
    /* per slot and axis: the area with its vertex moved along the axis.  With
     * F the moved axis and G the other one, the terms p - 1 and p are
     * F[p-1] G[p] - G[p-1] f and f G[p+1] - G[p] F[p+1] for x, minus those
     * for y; along y the whole sum is formed with the opposite sign. */
    const int per_axis = (nmoved + 31) & ~31;         /* no warp works on both axes */
    unsigned short *odd = reinterpret_cast<unsigned short *>(B.R[0]);   /* done with; 2 slot + axis */
    for (int t = tid; t < 2 * per_axis; t += NT) {
        const int x = t >= per_axis, w = x ? t - per_axis : t;
        if (w >= nmoved) continue;
        const int q = B.moved[w], i = B.owner[q], o = B.off[i], p = q - o, nn = B.n[i];
        const int st = B.state(i);
        if (st == GP_REST) continue;
        double a;         /* twice the moved area */
        if (p == 0) {
            a = B.sum0[x][i];
            if (x == 0) m.gq[B.sg[i]] = div_sides(B.se[i] * B.area[i], nn);
        } else if (st == GP_CHAIN) {
            odd[atomicAdd(&nodd, 1)] = (unsigned short)(2 * q + x);
            continue;
        } else {
            const double *F = B.A[x], *G = B.A[1 - x];
            const int e = B.c[x][i].e, up = (int)((B.c[x][i].up >> p) & 1u);
            const double f = add_exact(F[q], ntab[e + up] << up, e + GP_E0);
            const long long flip = x ? LLONG_MIN : 0;
            auto sgn = [&](double v) { return __longlong_as_double(dbits(v) ^ flip); };
            a = 0;
            if (p >= 2) {
                a = B.Q[x][q - 1] - G[q - 1] * f;                      /* term p - 1 */
                if (p > 2) a = sgn(B.M[0][q - 2]) + a;
            }
            if (p < nn - 1) {
                const double t2 = f * G[q + 1] - B.Q[1 - x][q];        /* term p */
                a = p == 1 ? t2 : a + t2;
                for (int k = q + 1; k < o + nn - 1; k++) a = a + sgn(B.T[k]);
            }
        }
        reinterpret_cast<double *>(m.contrib + B.dest[q])[x] = mul_diff(B.se[i], dabs(dscale_down<1>(a)), dabs(B.area[i]));
    }
    if (chains) {                              /* the uncertified grains' slots */
        __syncthreads();
        moved_uncertified_all<NT>(m, B, odd, nodd);
    }
    __syncthreads();
    c0 += total;
    }
    /* the rest, a warp per grain */
    GrainRest &Z = reinterpret_cast<GrainRest *>(smem)[warp];
    for (int q = warp; q < nrest; q += W) grain_by_warp(m, rest[q], Z.P, Z.R, lane);
}
constexpr int GRAIN_TINY = 6 * 1024, GRAIN_SMALL = 32 * 1024;   /* see launch_grain_pass */
constexpr int VERTEX_LANES_NV = 12 * 1024;                      /* see launch_vertex_fd */

/* vertex pass: src/calculus.h:19-73 (boundary part) and :143-154;
 * vertex_compute_energy src/geometry.h:472-479.
 *
 * UNIT_GAMMA: every boundary energy is exactly 1 this step (isotropic
 * boundaries, GB_scaling = 1: the geometry pass wrote 1 * 1 into every
 * enabled boundary), so the products gamma * x are x and are skipped.
 * Sums that the reference starts from 0.0 take their first term through
 * zero_plus, which keeps the first addition off the FP64 pipe. */
template <bool UNIT_GAMMA>
__global__ void k_vertex_fd(DevMesh m, double mu)
{
    int v = blockIdx.x * blockDim.x + threadIdx.x;
    if (v >= m.nv || !m.ven[v]) return;
    double2 p = m.pos[v];
    int4 sb = m.vb[v], sg = m.vg[v];
    double2 q[3];
    double gam[3], len[3];
    for (int j = 0; j < 3; j++) {
        int b = slot3(sb, j);
        q[j] = m.pos[other_end(m.bv[b], v)];
        gam[j] = m.benergy[b];
        len[j] = m.blen[b];
    }
    double2 cg[3];
    for (int j = 0; j < 3; j++) cg[j] = m.contrib[3 * v + j];
    DevMesh::FdTerms t;
    double vel[2];
#pragma unroll
    for (int c = 0; c < 2; c++) {
        double2 np = p;
        if (c == 0) np.x += SEVC_GRAD_EPS_D; else np.y += SEVC_GRAD_EPS_D;
        np.x = dmod(np.x, m.D);
        np.y = dmod(np.y, m.D);
        double bt = 0.0, gt = 0.0;
#pragma unroll
        for (int j = 0; j < 3; j++) {
            double Lj = arclen(np, q[j], m.D);
            double term = UNIT_GAMMA ? (Lj - len[j]) : (gam[j] * (Lj - len[j]));
            double gj = c == 0 ? cg[j].x : cg[j].y;
            if (j == 0) { bt = zero_plus(term); gt = zero_plus(gj); }
            else { bt += term; gt += gj; }
        }
        if (c == 0) { t.bx = bt; t.gx = gt; } else { t.by = bt; t.gy = gt; }
        vel[c] = div_grad_eps(-(bt + gt));
        if (mu != 1.0) vel[c] = mu * vel[c];   /* mobility; 1 * v is v exactly */
    }
    m.terms[v] = t;
    m.vel[v] = make_double2(vel[0], vel[1]);
    m.vspd[v] = speed_bound(vel[0], vel[1]);
    double e = 0.0;
#pragma unroll
    for (int j = 0; j < 3; j++) {
        int g = slot3(sg, j);
        double ej = dscale_down<1>(UNIT_GAMMA ? len[j] : (len[j] * gam[j]));
        e = j == 0 ? zero_plus(ej) : e + ej;
        e += g >= 0 ? m.gq[g] : 0.0;
    }
    m.venergy[v] = e;
}

/* The same for meshes that leave the GPU idle, by six lanes per vertex, five
 * vertices a warp: lane 3 c + j has the arclength of boundary j with the
 * vertex moved along c, and the sums pass through shuffles in the same order.
 * One thread's six arclengths are 20 KB of code that every warp of a small
 * mesh fetches for one pass through it, and a chain six times as long;
 * here every lane runs one.  Sums are formed by all six lanes, which costs
 * twice the FP64 instructions per vertex: see launch_vertex_fd. */
template <bool UNIT_GAMMA>
__global__ void __launch_bounds__(128) k_vertex_fd_lanes(DevMesh m, double mu)
{
    const unsigned all = 0xffffffffu;
    const int lane = threadIdx.x & 31, slot = lane / 6, r = lane - 6 * slot, c = r >= 3, j = r - 3 * c;
    const int v = 5 * ((blockIdx.x * blockDim.x + threadIdx.x) >> 5) + slot;
    const bool on = slot < 5 && v < m.nv && m.ven[v];
    double2 np = make_double2(0, 0), q = np;
    double gam = 0, len = 0, gj = 0, gq = 0;
    if (on) {
        np = m.pos[v];
        const int4 sb = m.vb[v], sg = m.vg[v];
        const int b = slot3(sb, j), g = slot3(sg, j);
        gj = reinterpret_cast<const double *>(m.contrib + 3 * v + j)[c];
        q = m.pos[other_end(m.bv[b], v)];
        gam = m.benergy[b];
        len = m.blen[b];
        gq = g >= 0 ? m.gq[g] : 0.0;
        const double moved = (c ? np.y : np.x) + SEVC_GRAD_EPS_D;
        if (c) np.y = moved; else np.x = moved;
        np.x = dmod(np.x, m.D);
        np.y = dmod(np.y, m.D);
    }
    const double Lj = arclen(np, q, m.D);
    const double term = UNIT_GAMMA ? (Lj - len) : (gam * (Lj - len));
    const double ej = dscale_down<1>(UNIT_GAMMA ? len : (len * gam));
    const int base = lane - j, first = lane - r;
    double bt = zero_plus(__shfl_sync(all, term, base)), gt = zero_plus(__shfl_sync(all, gj, base));
    double e = zero_plus(__shfl_sync(all, ej, first));
    e += __shfl_sync(all, gq, first);
#pragma unroll
    for (int k = 1; k < 3; k++) {
        bt += __shfl_sync(all, term, base + k);
        gt += __shfl_sync(all, gj, base + k);
        e += __shfl_sync(all, ej, first + k);
        e += __shfl_sync(all, gq, first + k);
    }
    double vel = div_grad_eps(-(bt + gt));
    if (mu != 1.0) vel = mu * vel;
    const double vy = __shfl_sync(all, vel, first + 3);
    if (!on || j) return;
    double *t = reinterpret_cast<double *>(m.terms + v);
    t[2 * c] = bt;
    t[2 * c + 1] = gt;
    reinterpret_cast<double *>(m.vel + v)[c] = vel;
    if (c) return;
    m.vspd[v] = speed_bound(vel, vy);
    m.venergy[v] = e;
}

/* compute_grain_dAdts, src/calculus.h:243 with compute_dAdt
 * src/geometry.h:779-787 streamed over the list */
__device__ void dadt_of(const DevMesh &m, int g);

/* every enabled grain, on a step that computes every output-only value
 * (flags[0]); on the others the events settle the grains they change */
__global__ void k_grain_dadt(DevMesh m, const int *flags)
{
    if (!flags[0]) return;
    int stride = gridDim.x * blockDim.x;
    for (int g = blockIdx.x * blockDim.x + threadIdx.x; g < m.ng; g += stride)
        if (m.gen[g]) dadt_of(m, g);
}

__device__ void dadt_of(const DevMesh &m, int g)
{
    m.gdadt[g] = dadt_from(m, g, m.pos, m.vel);
    m.gexact[g] = GEXACT_DADT;
}

/* compute_t_ext (src/topological.h:303-334) then label_boundaries
 * (:343-353), which runs on every slot including disabled ones */
/*
 * When flags[0] is 0 a boundary that provably is not a candidate skips
 * the transcendental evaluation and gets a t_ext outside [0, dt], so the
 * labels (this kernel's and label_3sided's) see what they would see; the
 * value itself is not observed: exports happen only on steps that compute
 * every value, and a boundary an event disables gets its exact value then
 * (finalize_boundary).  The proof that a boundary is not a candidate is the
 * binary32 certificate text_outside_dt.
 */
/* label_boundaries' result for boundary b.  A candidate joins the list the
 * polling and the flips work on.  For any other boundary the first polling
 * iteration's comparison (src/topological.h:466-511) happens here: its flag
 * is 0 and stays 0, so it mismatches if the buffer (buf, as the last step's
 * polling left it) holds 1, and the buffer becomes 0.  (A listed boundary is
 * enabled; a disabled one has its buffer cleared and never mismatches.) */
__device__ __forceinline__ void set_label(const DevMesh &m, const DevScratch &x, const PollGrid &pg, int b, uint8_t en,
                                          uint8_t buf, unsigned cand)
{
    m.bcand[b] = (uint8_t)cand;
    m.bconf[b] = -1;
    if (en && cand) {
        x.list_a[atomicAdd(x.n_a, 1)] = b;
    } else if (buf) {
        m.bcandbuf[b] = 0;
        if (en) poll_fail(m, x, pg, b);
    }
}
__device__ __forceinline__ void text_label_one(const DevMesh &m, const DevScratch &x, const PollGrid &pg, int b,
                                               uint8_t en, uint8_t buf, double2 pi, double2 pe, double2 vi, double2 ve,
                                               double dt, float Df, float hDf, float inv_dt, int full)
{
    long long tb;
    if (en) {
        if (!full && text_outside_dt(pi, pe, vi, ve, Df, hDf, inv_dt)) {
            /* not a candidate: its t_ext is outside [0, dt]; the value
             * itself is only observed if an event disables the boundary,
             * which then computes it (finalize_boundary) */
            m.btext[b] = SEVC_MAX_T_EXT_D;
            m.bexact[b] = 0;
            set_label(m, x, pg, b, en, buf, 0);
            return;
        }
        double text = text_exact_call(pi, pe, vi, ve, m.D);
        m.btext[b] = text;
        m.bexact[b] = 1;
        tb = dbits(text);
    } else {
        tb = dbits(m.btext[b]);
    }
    /* text >= 0 && text <= dt on the bit pattern (dt > 0): +-0, or a
     * non-negative pattern not above dt's; NaN fails as in the comparison.
     * Written in PTX so that it stays two integer comparisons (as C the
     * compiler may turn it back into FP64 ones). */
    unsigned cand;
    asm("{\n\t.reg .pred p, q, z;\n\t"
        "setp.ge.s64 p, %1, 0;\n\t"
        "setp.le.s64 q, %1, %2;\n\t"
        "setp.eq.s64 z, %1, 0x8000000000000000;\n\t"
        "and.pred p, p, q;\n\t"
        "or.pred p, p, z;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(cand) : "l"(tb), "l"(dbits(dt)));
    set_label(m, x, pg, b, en, buf, cand);
}
/* Two boundaries per thread (b and b + blockDim.x of the block's pair of
 * tiles), every load of both issued before either is labelled: the pass
 * waits on rounds of gathers, and twice the loads in flight per thread
 * hide more of that latency than the registers they cost.
 *
 * Speed bound.  A candidate has 0 <= t_ext = -|d| / (u.(ve - vi)) <= dt
 * (u = d/|d| through atan2/cos/sin, |u| <= 1 + 1e-15), so
 * |d| <= dt (|vi|_1 + |ve|_1) (1 + 1e-14).  The vertex pass leaves an upper
 * bound of each |v|_1 in binary32 (speed_bound); a boundary whose
 * arclength this step (blen, the same |d| up to 1e-15) cut down to binary32
 * exceeds dt_up (s_i + s_e), dt_up >= dt (1 + 1e-6), rounded up, is no
 * candidate, and is labelled as the certificate labels one (without
 * reading its ends' positions and velocities).  The others take the
 * certificate and, if undecided, the exact value. */
__global__ void k_text_label(DevMesh m, DevScratch x, PollGrid pg, double dt, float Df, float hDf, float inv_dt,
                             float dt_up)
{
    griddep_wait();
    int b0 = 2 * blockIdx.x * blockDim.x + threadIdx.x;
    int full = x.flags[0];
    uint8_t en[2], buf[2];
    int2 e[2];
#pragma unroll
    for (int k = 0; k < 2; k++) {
        int b = b0 + k * blockDim.x;
        bool in = b < m.nb;
        en[k] = in ? m.ben[b] : 0;
        buf[k] = in ? m.bcandbuf[b] : 0;
        e[k] = in ? m.bv[b] : make_int2(0, 0);   /* loaded beside the flag: one round trip less */
    }
    bool far[2] = { false, false };
    if (!full) {
        float bl[2] = { 0.f, 0.f }, si[2] = { 0.f, 0.f }, se[2] = { 0.f, 0.f };
#pragma unroll
        for (int k = 0; k < 2; k++)
            if (en[k]) { bl[k] = f32_cut(m.blen[b0 + k * blockDim.x]); si[k] = m.vspd[e[k].x]; se[k] = m.vspd[e[k].y]; }
#pragma unroll
        for (int k = 0; k < 2; k++) far[k] = en[k] && bl[k] > __fmul_ru(__fadd_ru(si[k], se[k]), dt_up);
    }
    double2 z = make_double2(0, 0), pi[2] = { z, z }, pe[2] = { z, z }, vi[2] = { z, z }, ve[2] = { z, z };
#pragma unroll
    for (int k = 0; k < 2; k++)
        if (en[k] && !far[k]) { pi[k] = m.pos[e[k].x]; pe[k] = m.pos[e[k].y]; vi[k] = m.vel[e[k].x]; ve[k] = m.vel[e[k].y]; }
#pragma unroll
    for (int k = 0; k < 2; k++) {
        int b = b0 + k * blockDim.x;
        if (b >= m.nb) continue;
        if (far[k]) {
            m.btext[b] = SEVC_MAX_T_EXT_D;       /* as text_label_one's certified skip */
            m.bexact[b] = 0;
            set_label(m, x, pg, b, en[k], buf[k], 0);
        } else {
            text_label_one(m, x, pg, b, en[k], buf[k], pi[k], pe[k], vi[k], ve[k], dt, Df, hDf, inv_dt, full);
        }
    }
}


__global__ void k_pack_summary(DevMesh m, DevScratch x, int *out)
{
    griddep_wait();
    pack_summary(m, x, out, blockIdx.x * blockDim.x + threadIdx.x, gridDim.x * blockDim.x);
}
/* The step's way in and out.  A copy of a few bytes between two steps goes to
 * another engine and back: with one for the host's flags and one for the
 * summary a step of 2,000 grains took 60 us of which 46 were its kernels,
 * with these 51 us. */
__global__ void k_set_flags(int *flags, int f1, int f2, int f3)
{
    flags[1] = f1; flags[2] = f2; flags[3] = f3;
}
__global__ void k_read_out(const int *from, int *to, int n)
{
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) to[i] = from[i];
}
__global__ void k_reset_ngrains(int *counters, int ninst)
{
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < ninst) counters[(size_t)i * CTR_COUNT + CTR_NGRAINS] = 0;
}
/* both counts; the last block finishes the nucleated area */
__global__ void __launch_bounds__(TPB) k_counts(DevMesh m, int *counters, double *block_area, int nblocks, int tpb)
{
    count_grains(m, counters, blockIdx.x * blockDim.x + threadIdx.x, gridDim.x * blockDim.x);
    nucl_area_blocks(m, block_area, nblocks, tpb, blockIdx.x, gridDim.x);
    const bool last = last_block(m.lastblk + 1);
    if (last) {
        __threadfence();
        nucl_area_final(m, block_area, nblocks, counters, threadIdx.x, blockDim.x);
    }
}

} // namespace

void launch_boundary_geometry(const DevMesh &m, double eps, double scaling, const LaunchShape &sh, cudaStream_t s)
{
    int t = sh.tpb_boundary;
    COUNT_LAUNCHES(1), k_boundary_geometry<<<(m.nb + t - 1) / t, t, 0, s>>>(m, eps, scaling);
}
void launch_grain_pass(const DevMesh &m, const DevScratch &x, const LaunchShape &sh, cudaStream_t s)
{
    /* coordinates from here on take the general path (adding eps could
     * reach D): a margin of 1e-7, or of a few ulps of a large D */
    double lim = m.D - std::max(1e-7, m.D * 0x1p-50);
    long long dlim;
    memcpy(&dlim, &lim, sizeof dlim);
    const int wide = sh.wide_sides >= 12 ? GP_NMAX : sh.wide_sides;
    auto go = [&](auto kernel, int gpb, int nt) {
        COUNT_LAUNCHES(1), kernel<<<(m.ng + gpb - 1) / gpb, nt, 0, s>>>(m, x.three, x.n_three, wide, dlim);
    };
    /* Large meshes want blocks on the SM: 32 grains, 208 slots (6.5 per
     * grain; 3% of the blocks need a second chunk) and 40 registers let
     * eleven in, 385 us at 1M grains against 397 with ten (blocks of 64 in two
     * chunks: 414, and 67 against 62 at 100K; they stay for the autotuner).
     * Below, an SM holds few blocks and the longest one is the time: 16
     * grains from GRAIN_SMALL down (31 us against 35 at 32,000 grains; above
     * it 41 against 39 at 50,000 and 68 against 56 at 100,000), 8 from
     * GRAIN_TINY down (16 us against 18 at 2,000, 17 against 18 at 6,000;
     * above it 23 against 19 at 10,000). */
    if (sh.grain_occ < 6) go(k_grain_pass<64, 128, 208>, 64, 128);
    else if (m.ng <= GRAIN_TINY) go(k_grain_pass<8, 128, 80>, 8, 128);
    else if (m.ng <= GRAIN_SMALL) go(k_grain_pass<16, 128, 144>, 16, 128);
    else go(k_grain_pass<32, 128, 208>, 32, 128);
}

bool vertex_lanes(const DevMesh &m) { return m.nv <= VERTEX_LANES_NV; }
void launch_vertex_fd(const DevMesh &m, double mu, bool unit_gamma, const LaunchShape &sh, cudaStream_t s)
{
    /* six lanes per vertex: 8 us against 12 at 2,000 grains, 10 against 12 at
     * 5,000, the same at 10,000, 18 against 14 at 20,000 */
    if (vertex_lanes(m)) {
        const int g = (m.nv + 19) / 20;               /* four warps of five vertices */
        if (unit_gamma) COUNT_LAUNCHES(1), k_vertex_fd_lanes<true><<<g, 128, 0, s>>>(m, mu);
        else COUNT_LAUNCHES(1), k_vertex_fd_lanes<false><<<g, 128, 0, s>>>(m, mu);
        return;
    }
    int t = sh.tpb_vertex;
    if (unit_gamma) COUNT_LAUNCHES(1), k_vertex_fd<true><<<(m.nv + t - 1) / t, t, 0, s>>>(m, mu);
    else COUNT_LAUNCHES(1), k_vertex_fd<false><<<(m.nv + t - 1) / t, t, 0, s>>>(m, mu);
}
void launch_grain_dadt(const DevMesh &m, const DevScratch &x, cudaStream_t s)
{
    int g = nblk(m.ng);
    COUNT_LAUNCHES(1), k_grain_dadt<<<g < 8 * 152 ? g : 8 * 152, TPB, 0, s>>>(m, x.flags);
}
void launch_text_label(const DevMesh &m, const DevScratch &x, const StepParams &p, cudaStream_t s)
{
    const double dt = p.dt;
    int t = p.shape.tpb_boundary;
    /* binary32 copies for the certificate (text_outside_dt): rounded to
     * nearest, within 2^-24 of the binary64 values */
    float Df = (float)m.D, hDf = (float)(m.D / 2.0), inv_dt = (float)(1.0 / dt);
    /* dt (1 + 1e-6) rounded up to binary32, for the speed bound */
    float dt_up = std::nextafter((float)(dt * (1.0 + 1e-6)), INFINITY);
    if ((double)dt_up < dt * (1.0 + 1e-6)) dt_up = std::nextafter(dt_up, INFINITY);
    if (m.nb > 0)
        launch_dep(k_text_label, (m.nb + 2 * t - 1) / (2 * t), t, s, m, x, poll_grid(p), dt, Df, hDf, inv_dt, dt_up);
}
void launch_pack_summary(const DevMesh &m, const DevScratch &x, int *out, cudaStream_t s)
{
    /* the exactness marks it zeroes, 16 at a time, outnumber the words it
     * packs: with blocks for the words alone (one, on a single mesh) it took
     * 17 us at 1M grains, with blocks for both 3 us */
    size_t words = (size_t)m.ninst * (CTR_COUNT + EVT_COUNT + 1 + TWO_THREE_PASSES) + 5, marks = (size_t)m.ng / 16 + 1;
    int g = (int)(((words > marks ? words : marks) + TPB - 1) / TPB);
    launch_dep(k_pack_summary, g < 152 ? g : 152, TPB, s, m, x, out);
}

cudaError_t launch_set_flags(const DevScratch &x, int full, int min_grains, int grains, cudaStream_t s)
{
    return launch_status(k_set_flags, 1, 1, 0, s, x.flags, full, min_grains, grains);
}
cudaError_t launch_read_out(const int *from, int *host, int n, cudaStream_t s)
{
    int g = nblk(n);
    return launch_status(k_read_out, g < 16 ? g : 16, TPB, 0, s, from, host, n);
}
void launch_counts(const DevMesh &m, const DevScratch &x, const StepParams &p, cudaStream_t s)
{
    COUNT_LAUNCHES(1), k_reset_ngrains<<<(p.ninst + 127) / 128, 128, 0, s>>>(x.counters, p.ninst);
    int g = nblk(m.ng);
    COUNT_LAUNCHES(1), k_counts<<<g < 152 ? g : 152, TPB, 0, s>>>(m, x.counters, x.block_area, p.n_blocks, p.n_threads);
}
