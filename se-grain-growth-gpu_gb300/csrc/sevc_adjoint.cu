/*
 * Adjoint of the time step over the positions, and the grain-area
 * histogram used as a differentiable statistic.  No counterpart in the
 * reference.
 *
 * Forward map of one step (fixed event sequence):
 *   v_i^c = mu * ( -[ sum_j gamma_j (L_j(x + eps e_i^c) - L_j(x))
 *                     + sum_g SE_g (|A_g(x + eps e_i^c)| - |A_g(x)|) ] / eps )
 *                                          (src/calculus.h:19-73, eps = 1e-8)
 *   events: a T1 flip sets both ends to their midpoint, a 3-sided removal
 *           moves the survivor to the length-weighted point of the three
 *           vertices (src/topological.h:174-291, :687-822); both zero the
 *           velocities of the vertices they move; disabled vertices stop
 *   x_{n+1} = x' + dt * v'                 (src/calculus.h:391-404)
 * with gamma_j = s * f_j (s = GB_scaling, f_j = 1 for GB_eps = 0).
 * A step with a nucleation first maps the positions by the inserted
 * triangle (src/nucleation2.cu:116-212 with the factor 0.99): with
 * A's boundaries ending at D, E, F, d_X = X - A (wrapped), u_X = d_X/|d_X|
 * and r = k * |d_X*| + 0.1 (X* the end of the shortest boundary, k = 0.8
 * times the replayed draw), the new A, B, C are A + 0.99 r u_D, u_E, u_F;
 * the rest of the step acts on that mesh.  The nucleated grain's stored
 * energy is 0, not a parameter.
 *
 * The adjoint below is the exact derivative of that map in real
 * arithmetic.  Two identities keep it cheap: the shoelace area is linear in
 * each coordinate of one vertex, so (|A(x + eps e)| - |A(x)|) / eps =
 * sign(A) dA/dx (away from a sign change), whose derivatives are constants
 * on the two list neighbours; and the arclength term's derivative is
 * (n' - n) / eps with n, n' the unit vectors of the unmoved and moved edge.
 * Every accumulation is a gather in a fixed order, so results do not depend
 * on scheduling.
 */
#include "sevc_internal.h"

namespace {

constexpr int TPB = 256;
constexpr int ADJ_BLOCK = 64;   /* of the backward pass's long threads: small meshes spread over the SMs */
inline int nblk(int n) { return (n + TPB - 1) / TPB; }

/* quadratic B-spline (partition of unity over unit-spaced bins) and its derivative */
__device__ __forceinline__ double bspline2(double s)
{
    double a = fabs(s);
    if (a <= 0.5) return 0.75 - s * s;
    if (a <= 1.5) { double t = 1.5 - a; return 0.5 * t * t; }
    return 0.0;
}
__device__ __forceinline__ double bspline2_d(double s)
{
    double a = fabs(s);
    if (a <= 0.5) return -2.0 * s;
    if (a <= 1.5) return s > 0 ? -(1.5 - a) : (1.5 - a);
    return 0.0;
}

/* signed area of grain g (src/geometry.h:757 order) */
__device__ __forceinline__ double grain_area(const DevMesh &m, int g)
{
    return area_stream(m.glist + (size_t)SEVC_MAXV * g, m.gvlen[g], m.pos, m.D);
}

/* list neighbours of vertex v in grain g (false: not listed); eight entries
 * of the list a load */
__device__ __forceinline__ bool list_neighbours(const DevMesh &m, int g, int v, int &prev, int &next)
{
    const int *L = m.glist + (size_t)SEVC_MAXV * g;
    const int n = m.gvlen[g];
    for (int base = 0; base < n; base += 8) {
        int e[8], at = -1;
        list_batch(L, n, base, e);
#pragma unroll
        for (int j = 7; j >= 0; j--) at = base + j < n && e[j] == v ? base + j : at;
        if (at >= 0) {
            prev = L[at == 0 ? n - 1 : at - 1];
            next = L[at == n - 1 ? 0 : at + 1];
            return true;
        }
    }
    return false;
}

/* ---------------- histogram of normalised grain areas ---------------- */
/* a_g = |A_g| sc with sc = N / (total domain area): N enabled grains tile
 * the domain, so 1/sc is their mean area;
 * h_k = (1/N) sum_g B2(a_g / w - k - 1/2), w = amax / nbins.
 *
 * Each grain touches the three bins around a_g / w.  T threads of a block
 * (the most whose private bins fit in shared memory) keep their own copy of
 * the bins, laid out bin by bin, so the additions of a warp run side by
 * side without atomics; a block's copies, then the blocks' partial bins (by
 * the last block to finish), are summed in a fixed order.  Bound by the
 * FP64 pipe: about 50 operations a grain for its area and 30 for the
 * splines.  500K grains 1.39 ms -> 0.1 ms (the form before it ran a
 * block-wide tree reduction for every bin). */
__device__ __forceinline__ double warp_sum(double s)
{
    for (int o = 16; o > 0; o >>= 1) s += __shfl_down_sync(0xffffffffu, s, o);
    return s;
}
__global__ void __launch_bounds__(TPB) k_hist(DevMesh m, int nbins, int T, double amax, double sc, double nnorm,
                                              double *blockbins, double *hist)
{
    extern __shared__ double bins[];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    for (int i = tid; i < nbins * T; i += TPB) bins[i] = 0.0;
    __syncthreads();
    const double w = amax / nbins;
    if (tid < T)
        for (int g = blockIdx.x * T + tid; g < m.ng; g += gridDim.x * T) {
            if (!m.gen[g]) continue;
            const double t = fabs(grain_area(m, g)) * sc / w;
            if (!(t < nbins + 2)) continue;
            const int c = (int)t;
            for (int k = c - 1; k <= c + 1; k++)
                if (k >= 0 && k < nbins) bins[k * T + tid] += bspline2(t - k - 0.5);
        }
    __syncthreads();
    for (int k = warp; k < nbins; k += TPB / 32) {
        double s = 0.0;
        for (int i = lane; i < T; i += 32) s += bins[k * T + i];
        s = warp_sum(s);
        if (lane == 0) blockbins[(size_t)blockIdx.x * nbins + k] = s;
    }
    const bool last = last_block(m.lastblk + 3);
    if (last) {
        __threadfence();
        for (int k = warp; k < nbins; k += TPB / 32) {
            double s = 0.0;
            for (int b = lane; b < (int)gridDim.x; b += 32) s += __ldcg(blockbins + (size_t)b * nbins + k);
            s = warp_sum(s);
            if (lane == 0) hist[k] = s / nnorm;
        }
    }
}

/* dL/dA_g of the histogram (signed area) given dL/dh: the three bins around
 * the grain's area have a derivative; zero_sum = 0.0 times the sum of dL/dh
 * (what the other bins contribute: nothing, or NaN if one is not finite) */
__global__ void k_hist_grad_area(DevMesh m, int nbins, double amax, double sc, double nnorm, const double *dldh,
                                 double zero_sum, double *dlda)
{
    int g = blockIdx.x * blockDim.x + threadIdx.x;
    if (g >= m.ng) return;
    if (!m.gen[g]) { dlda[g] = 0.0; return; }
    double A = grain_area(m, g);
    double w = amax / nbins, t = fabs(A) * sc / w;
    double d = zero_sum;
    if (t < nbins + 2) {
        const int c = (int)t;
        for (int k = c - 1; k <= c + 1; k++)
            if (k >= 0 && k < nbins) d += dldh[k] * bspline2_d(t - k - 0.5);
    }
    d *= sc / (w * nnorm);
    dlda[g] = A < 0 ? -d : d;
}

/* lambda_k = sum over k's grains of dL/dA_g dA_g/dx_k, with
 * dA/dx_k = (y_next - y_prev) / 2, dA/dy_k = (x_prev - x_next) / 2 */
__global__ void k_area_grad_to_vertices(DevMesh m, const double *dlda, double2 *lam)
{
    int v = blockIdx.x * blockDim.x + threadIdx.x;
    if (v >= m.nv) return;
    double2 out = make_double2(0, 0);
    if (m.ven[v]) {
        double2 p = m.pos[v];
        int4 sg = m.vg[v];
        for (int j = 0; j < 3; j++) {
            int g = slot3(sg, j);
            if (g < 0 || !m.gen[g]) continue;
            int pv, nx;
            if (!list_neighbours(m, g, v, pv, nx)) continue;
            double2 a = m.pos[pv], b = m.pos[nx];
            /* unwrapped neighbour coordinates relative to v */
            double xp = wrapd(a.x, p.x, m.D), yp = wrapd(a.y, p.y, m.D);
            double xn = wrapd(b.x, p.x, m.D), yn = wrapd(b.y, p.y, m.D);
            out.x += dlda[g] * 0.5 * (yn - yp);
            out.y += dlda[g] * 0.5 * (xp - xn);
        }
    }
    lam[v] = out;
}

/* ---------------- adjoint of one step ---------------- */
/* translation x_{n+1} = x' + dt v': lambda_x' = lambda (vertices alive
 * after the step), lambda_v = dt lambda (k_adj_events zeroes it for the
 * vertices an event moved); d/dmu of the step: dt * lambda . v' / mu */
__global__ void k_adj_translate(int nv, double dt, double mu, const double2 *lam, const uint8_t *ven1,
                                const double2 *vel1, double2 *lx, double2 *lv, double *gmu)
{
    griddep_wait();
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= nv) return;
    double2 l = ven1[i] ? lam[i] : make_double2(0, 0);
    lx[i] = l;
    lv[i] = make_double2(dt * l.x, dt * l.y);
    double2 w = vel1[i];
    gmu[i] += dt * (l.x * w.x + l.y * w.y) / mu;
}

/* one logged flip or 3-sided removal, backward */
__device__ void adj_event_one(double D, const EventRec &r, double2 *lx)
{
    if (r.type == EV_FLIP) {                          /* both ends -> midpoint */
        double2 a = lx[r.a], b = lx[r.b];
        double2 s = make_double2(0.5 * (a.x + b.x), 0.5 * (a.y + b.y));
        lx[r.a] = s;
        lx[r.b] = s;
        return;
    }
    if (r.type != EV_REMOVE) return;                  /* nucleations: k_adj_nucleation */
    /* A' = A + F(u, w), u = B - A, w = C - A,
     * F = (|w| u + |u| w) / (|u| + |w - u| + |w|) */
    double2 lp = lx[r.a];
    double ux = wrapd(r.pb.x, r.pa.x, D), uy = wrapd(r.pb.y, r.pa.y, D);
    double wx = ux + wrapd(r.pc.x, r.pb.x, D), wy = uy + wrapd(r.pc.y, r.pb.y, D);
    double nu = sqrt(ux * ux + uy * uy), nw = sqrt(wx * wx + wy * wy);
    double rx = wx - ux, ry = wy - uy, nr = sqrt(rx * rx + ry * ry);
    double S = nu + nr + nw;
    double Nx = nw * ux + nu * wx, Ny = nw * uy + nu * wy;
    double lN = lp.x * Nx + lp.y * Ny, lw = lp.x * wx + lp.y * wy, lu = lp.x * ux + lp.y * uy;
    double hux = ux / nu, huy = uy / nu, hwx = wx / nw, hwy = wy / nw, hrx = rx / nr, hry = ry / nr;
    if (nu == 0) { hux = 0; huy = 0; }                /* coincident vertices: zero subgradient */
    if (nw == 0) { hwx = 0; hwy = 0; }
    if (nr == 0) { hrx = 0; hry = 0; }
    if (!(S > 0)) return;                             /* degenerate triangle: the map is not moved */
    double S2 = S * S;
    /* J_u^T lambda' and J_w^T lambda' */
    double jux = (nw * lp.x + lw * hux) / S - lN * (hux - hrx) / S2;
    double juy = (nw * lp.y + lw * huy) / S - lN * (huy - hry) / S2;
    double jwx = (lu * hwx + nu * lp.x) / S - lN * (hrx + hwx) / S2;
    double jwy = (lu * hwy + nu * lp.y) / S - lN * (hry + hwy) / S2;
    lx[r.a] = make_double2(lp.x - jux - jwx, lp.y - juy - jwy);
    double2 b = lx[r.b], c = lx[r.c];
    lx[r.b] = make_double2(b.x + jux, b.y + juy);
    lx[r.c] = make_double2(c.x + jwx, c.y + jwy);
}

/* Walk the step's log from its end in chunks of ADJ_TPB records, one block
 * per instance: the threads test a chunk at once (record kind and the
 * instance of its first vertex) and thread 0 takes the hits in descending
 * log order.  Events of different instances touch disjoint vertices, so
 * the instances run side by side; within an instance the events keep the
 * reverse of the order they were applied in (the log order: the parallel
 * events, which share no vertex, then the deferred ones). */
constexpr int ADJ_TPB = 256;
template <class Want, class Take>
__device__ void walk_log_reverse(const EventRec *log, int n, Want want, Take take)
{
    __shared__ unsigned hit[ADJ_TPB / 32];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    for (int top = n; top > 0; top -= ADJ_TPB) {
        int e = top - 1 - (int)threadIdx.x;
        bool f = e >= 0 && want(e);
        unsigned w = __ballot_sync(0xffffffffu, f);
        if (lane == 0) hit[warp] = w;
        __syncthreads();
        if (threadIdx.x == 0)
            for (int k = 0; k < ADJ_TPB / 32; k++)
                for (unsigned h = hit[k]; h; h &= h - 1) take(top - 1 - (32 * k + __ffs(h) - 1));
        __syncthreads();
    }
}
__device__ __forceinline__ bool in_instance(const int *voff, int ninst, int inst, int v)
{
    return ninst <= 1 || (v >= voff[inst] && v < voff[inst + 1]);
}

/* the step's flips and 3-sided removals in reverse order, per instance; the
 * vertices they moved have no velocity (it was zeroed) */
__global__ void __launch_bounds__(ADJ_TPB) k_adj_events(double D, const EventRec *log, const int *nlog, double2 *lx,
                                                        double2 *lv, const int *voff, int ninst)
{
    griddep_wait();
    const int inst = blockIdx.x, n = *nlog;
    for (int i = threadIdx.x; i < n; i += ADJ_TPB) {
        const EventRec r = log[i];
        if ((r.type != EV_FLIP && r.type != EV_REMOVE) || !in_instance(voff, ninst, inst, r.a)) continue;
        lv[r.a] = lv[r.b] = make_double2(0, 0);
        if (r.type == EV_REMOVE) lv[r.c] = make_double2(0, 0);
    }
    walk_log_reverse(
        log, n,
        [&](int e) {
            EventRec r = log[e];
            return (r.type == EV_FLIP || r.type == EV_REMOVE) && in_instance(voff, ninst, inst, r.a);
        },
        [&](int e) { adj_event_one(D, log[e], lx); });
}

/* boundary weight f_j = gamma_j / s (k_boundary_geometry's definition) */
__device__ __forceinline__ double gb_weight(const DevMesh &m, int b, double eps)
{
    if (eps == 0.0) return 1.0;
    int2 e = m.bv[b];
    int gic[2];
    if (gintersect(m.vg[e.x], m.vg[e.y], gic) < 2) return 0.0;
    return gb_energy(m.gori[gic[0]] - m.gori[gic[1]], eps);
}

/* the nucleations of the step, last first: lambda of the positions
 * before it from lambda after it (one block per instance, as
 * k_adj_events).  For each new position Y = A + c u_X (c = 0.99 r):
 *   dY/dX = c (I - u u^T) / |d_X|,  dY/dA = I - dY/dX + u (dc/dA)^T,
 *   dc/dX* = 0.99 k u_X* = -dc/dA;
 * the new vertices B and C had no position before. */
__device__ void adj_nucleation_one(double D, const EventRec &r, const EventRec &x, double2 *lam)
{
    int Y[3] = { r.a, r.b, r.c }, X[3] = { x.a, x.b, x.c };
    double2 pa = r.pa, px[3] = { r.pb, r.pc, x.pa };
    double k = x.pb.x, c = 0.99 * x.pb.y;
    int is = (int)x.pc.x;
    double2 ly[3] = { lam[Y[0]], lam[Y[1]], lam[Y[2]] };
    double usx = wrapd(px[is].x, pa.x, D), usy = wrapd(px[is].y, pa.y, D);
    double ns = sqrt(usx * usx + usy * usy);
    usx = ns > 0 ? usx / ns : 0.0;
    usy = ns > 0 ? usy / ns : 0.0;
    double2 la = make_double2(0, 0);
    double2 lstar = make_double2(0, 0);
    for (int i = 0; i < 3; i++) {
        double dx = wrapd(px[i].x, pa.x, D), dy = wrapd(px[i].y, pa.y, D), n = sqrt(dx * dx + dy * dy);
        if (!(n > 0)) continue;
        double ux = dx / n, uy = dy / n, l_u = ux * ly[i].x + uy * ly[i].y;
        double gx = c / n * (ly[i].x - ux * l_u), gy = c / n * (ly[i].y - uy * l_u);
        double t = 0.99 * k * l_u;
        la.x += ly[i].x - gx - t * usx;
        la.y += ly[i].y - gy - t * usy;
        lam[X[i]].x += gx;
        lam[X[i]].y += gy;
        lstar.x += t * usx;
        lstar.y += t * usy;
    }
    lam[X[is]].x += lstar.x;
    lam[X[is]].y += lstar.y;
    lam[Y[0]] = la;
    lam[Y[1]] = make_double2(0, 0);
    lam[Y[2]] = make_double2(0, 0);
}
__global__ void __launch_bounds__(ADJ_TPB) k_adj_nucleation(double D, const EventRec *log, const int *nlog,
                                                            double2 *lam, const int *voff, int ninst)
{
    griddep_wait();
    const int inst = blockIdx.x, n = *nlog;
    walk_log_reverse(
        log, n,
        [&](int e) {
            if (e + 1 >= n) return false;
            EventRec r = log[e];
            return r.type == EV_NUCL && log[e + 1].type == EV_NUCL_AUX && in_instance(voff, ninst, inst, r.a);
        },
        [&](int e) { adj_nucleation_one(D, log[e], log[e + 1], lam); });
}

/* Sign of every grain's area at the start of each recorded step (area_stream's
 * sum), for a whole segment at once: blockIdx.y is the step, `bytes` the
 * distance of the records. */
__global__ void __launch_bounds__(TPB) k_adj_signs(TapeRecord r, size_t bytes, int ng, double D)
{
    griddep_wait();
    const int g = blockIdx.x * blockDim.x + threadIdx.x;
    if (g >= ng) return;
    const size_t o = blockIdx.y * bytes;
    auto at = [&](const void *p) { return static_cast<const char *>(p) + o; };
    int sign = 0;
    if (*reinterpret_cast<const uint8_t *>(at(r.gen + g))) {
        const double a = area_stream(reinterpret_cast<const int *>(at(r.glist + (size_t)SEVC_MAXV * g)),
                                     *reinterpret_cast<const int *>(at(r.gvlen + g)),
                                     reinterpret_cast<const double2 *>(at(r.pos)), D);
        sign = a > 0 ? 1 : (a < 0 ? -1 : 0);
    }
    r.sgn[o + g] = (signed char)sign;
}
/* per grain: dL/dSE_g += sum_p lambda_v(p) . (-mu sign(A) dA/dx_p) (not for a
 * nucleated grain, whose stored energy is 0, not a parameter).  Eight
 * vertices' positions and lambdas are loaded at once; the delta to a vertex's
 * predecessor is minus the predecessor's to it. */
__device__ __forceinline__ void adj_grain(const DevMesh &m, int g, double mu, const double2 *lv, const signed char *sgn,
                                          double *gse)
{
    if (g >= m.ng || !m.gen[g] || m.gtype[g] == GT_NUCLEATED) return;
    const int *L = m.glist + (size_t)SEVC_MAXV * g;
    const int n = m.gvlen[g];
    double acc = 0.0, px = 0, py = 0;                /* px, py: predecessor to vertex */
    double2 first = make_double2(0, 0);
    for (int base = 0; base < n; base += 8) {
        int v[8];
        double2 q[9], l[8];
        list_batch(L, n, base, v);
#pragma unroll
        for (int j = 0; j < 8; j++) { q[j] = m.pos[v[j]]; l[j] = lv[v[j]]; }
        q[8] = base + 8 < n ? m.pos[L[base + 8]] : make_double2(0, 0);
        if (base == 0) {
            first = q[0];
            const double2 last = m.pos[L[n - 1]];
            px = wrapd(first.x, last.x, m.D);
            py = wrapd(first.y, last.y, m.D);
        }
        const int end = n - base < 8 ? n - base : 8;
#pragma unroll 1
        for (int j = 0; j < end; j++) {
            const double2 c = q[j], b = base + j == n - 1 ? first : q[j + 1];
            const double xn = wrapd(b.x, c.x, m.D), yn = wrapd(b.y, c.y, m.D);
            acc += l[j].x * (0.5 * (yn + py)) + l[j].y * (0.5 * (-px - xn));
            px = xn; py = yn;
        }
    }
    gse[g] += -mu * (double)sgn[g] * acc;
}

/* For the edge vector d (length L) and its end moved by eps along axis c,
 * d' = d + eps e_c, L' = |d'|: *g = (d'/L' - d/L) / eps, the gradient with
 * respect to the moved end of (L' - L) / eps, and *s = (L' - L) / eps, both
 * in forms without cancellation:
 *   (L' - L) / eps = (2 d_c + eps) / (L + L')
 *   (d'/L' - d/L) / eps = e_c / L' - d (2 d_c + eps) / (L L' (L + L'))
 * (the same values as the difference quotients, which lose about eight
 * digits to cancellation).  L = 0, an edge whose ends coincide after a
 * flip, takes the zero subgradient for d/L. */
/*
 * The adjoint is checked against an FP64 reference and difference quotients
 * to a tolerance (it is not a bit-exact restatement), so its square roots
 * and reciprocals use a binary32 seed on the mantissa (the exponent split
 * off on the integer pipe) and one FP64 Newton step: ~2^-45 relative,
 * 3 and 2 FP64 instructions instead of ~8 each.  x > 0 and normal; other x
 * take the native operation.
 */
static __device__ __noinline__ double rsqrt_slow(double x) { return 1.0 / sqrt(x); }
static __device__ __noinline__ double rcp_slow(double x) { return 1.0 / x; }
__device__ __forceinline__ double rsqrt_newton(double x)
{
    long long b = dbits(x);
    int eb = (int)(b >> 52);
    if (eb < 2 || eb > 2045) return rsqrt_slow(x);
    int k = (eb - 1023) >> 1;                             /* x = m' 4^k, m' in [1, 4) */
    double mp = __longlong_as_double(b - (long long)(2 * k) * (1LL << 52));
    float y0 = rsqrt_seed(f32_cut(mp));
    double y = __longlong_as_double(dbits(f2d_bits(y0)) - (long long)k * (1LL << 52));
    double h = dscale_down<1>(x);
    double r = __fma_rn(-h * y, y, 0.5);                  /* 1/2 - x y^2 / 2 */
    return __fma_rn(y, r, y);
}
__device__ __forceinline__ double rcp_newton(double x)
{
    long long b = dbits(x);
    int eb = (int)(b >> 52);
    if (eb < 2 || eb > 2045) return rcp_slow(x);
    long long sh = (long long)(eb - 1023) * (1LL << 52);  /* x = m 2^e, m in [1, 2) */
    float y0 = rcp_seed(f32_cut(__longlong_as_double(b - sh)));
    double y = __longlong_as_double(dbits(f2d_bits(y0)) - sh);
    double e = __fma_rn(-x, y, 1.0);
    return __fma_rn(y, e, y);
}

/* The same quantities for the edge d (squared length L2, length L, 1/L,
 * 0 when L = 0) with the end moved by eps along axis c, written with one
 * reciprocal square root and one reciprocal:
 *   num = 2 d_c + eps, L'^2 = L2 + eps num, s = num / (L + L'),
 *   g = e_c / L' - d s / (L L'). */
__device__ __forceinline__ void edge_fd_grad(double dx, double dy, double L2, double L, double invL, double E, int c,
                                             double2 *g, double *s)
{
    double dc = c == 0 ? dx : dy, dother = c == 0 ? dy : dx;
    double num = __fma_rn(2.0, dc, E);
    double inv1 = rsqrt_newton(__fma_rn(E, num, L2));     /* 1 / L' */
    double L1 = __fma_rn(E, num, L2) * inv1;
    double sv = num * rcp_newton(L + L1);
    double t = sv * inv1 * invL;
    double gc = __fma_rn(-dc, t, inv1), go = -dother * t;
    *s = sv;
    *g = c == 0 ? make_double2(gc, go) : make_double2(go, gc);
}

/* per vertex k (gather): lambda_n[k] = lambda_x[k] + (J_v^T lambda_v)[k];
 * d/ds of k's own velocity into ggam[k].  Three lanes per vertex, ten
 * vertices a warp: lane j takes boundary j and grain j, so the three edges'
 * chains of dependent FP64 operations and the three list searches run side
 * by side; the first lane adds the parts in order. */
constexpr int ADJ_VPB = 10 * (ADJ_BLOCK / 32);     /* vertices per block */
__device__ __forceinline__ void adj_vertex(const DevMesh &m, double mu, double eps, double s_gb, const double2 *lx,
                                           const double2 *lv, const signed char *sgn, double2 *lam_out, double *ggam)
{
    const int lane = threadIdx.x & 31, q3 = lane / 3, j = lane - 3 * q3;
    const int k = blockIdx.x * ADJ_VPB + (threadIdx.x >> 5) * 10 + q3;
    const bool in = lane < 30 && k < m.nv, live = in && m.ven[k];
    const double E = SEVC_GRAD_EPS_D;
    double2 out = make_double2(0, 0);
    double dgam = 0.0;
    if (live) {
        const double2 p = m.pos[k], lk = lv[k];
        const int b = slot3(m.vb[k], j), g = slot3(m.vg[k], j);
        if (b >= 0) {
            int q = other_end(m.bv[b], k);
            double f = gb_weight(m, b, eps), gam = s_gb * f;
            double2 pq = m.pos[q], lq = lv[q];
            double dx = wrapd(p.x, pq.x, m.D), dy = wrapd(p.y, pq.y, m.D);
            double L2 = dx * dx + dy * dy;
            double invL = L2 > 0 ? rsqrt_newton(L2) : 0.0, L = L2 * invL;
            /* k moved along x / y (d -> d + eps e_c) and q moved (-d -> -d + eps e_c) */
            double2 gkx, gky, gqx, gqy;
            double skx, sky, sqx, sqy;
            edge_fd_grad(dx, dy, L2, L, invL, E, 0, &gkx, &skx);
            edge_fd_grad(dx, dy, L2, L, invL, E, 1, &gky, &sky);
            edge_fd_grad(-dx, -dy, L2, L, invL, E, 0, &gqx, &sqx);
            edge_fd_grad(-dx, -dy, L2, L, invL, E, 1, &gqy, &sqy);
            double cg = -mu * gam;
            out.x += cg * (lk.x * gkx.x + lk.y * gky.x);
            out.y += cg * (lk.x * gkx.y + lk.y * gky.y);
            dgam = -mu * f * (lk.x * skx + lk.y * sky);
            /* q's velocity: d/dx_k of -(gam/eps) (L(x_q + eps e_c) - L(x)) is
             * minus the gradient with respect to the moved end */
            double cq = mu * gam;
            out.x += cq * (lq.x * gqx.x + lq.y * gqy.x);
            out.y += cq * (lq.x * gqx.y + lq.y * gqy.y);
        }
        int pv, nx;
        if (g >= 0 && m.gen[g] && list_neighbours(m, g, k, pv, nx)) {
            double se = m.gtype[g] == GT_NUCLEATED ? 0.0 : m.gse[g];
            double c = 0.5 * mu * se * (double)sgn[g];
            double2 a = lv[pv], d = lv[nx];
            out.x += c * (a.y - d.y);
            out.y += c * (d.x - a.x);
        }
    }
    double2 sum = live && j == 0 ? lx[k] : make_double2(0, 0);
    double gsum = 0.0;
#pragma unroll
    for (int q = 0; q < 3; q++) {
        const int src = 3 * q3 + q < 32 ? 3 * q3 + q : 31;
        sum.x += __shfl_sync(0xffffffffu, out.x, src);
        sum.y += __shfl_sync(0xffffffffu, out.y, src);
        gsum += __shfl_sync(0xffffffffu, dgam, src);
    }
    if (j == 0 && in) {
        lam_out[k] = live ? sum : make_double2(0, 0);
        if (live) ggam[k] += gsum;
    }
}

/* both gathers of a step: the first vb blocks take the vertices, the others
 * the grains.  Neither fills the GPU at 10,000 grains; one after the other
 * they took 14 + 20 us, with the area signs in the first; this takes 22. */
__global__ void __launch_bounds__(ADJ_BLOCK) k_adj_gather(DevMesh m, double mu, double eps, double s_gb, const double2 *lx,
                                                          const double2 *lv, const signed char *sgn, double2 *lam_out,
                                                          double *ggam, double *gse, int vb)
{
    griddep_wait();
    if ((int)blockIdx.x < vb) adj_vertex(m, mu, eps, s_gb, lx, lv, sgn, lam_out, ggam);
    else adj_grain(m, (blockIdx.x - vb) * blockDim.x + threadIdx.x, mu, lv, sgn, gse);
}

/* ---- tape records (sevc_adjoint_histogram's replay) ---- */
/* What the adjoint of a step reads, in one launch instead of a copy per
 * array: the mesh the velocities are computed on, of the grain lists only the
 * used entries (24 of 400 bytes per grain on average).  blockIdx.y is the array:
 * one thread copying a piece of each waits for them in turn (10 us a step at
 * 10,000 grains, 7.5 so).  start: the record
 * is the step's first (the event log is emptied and switched on). */
__device__ __forceinline__ void copy_words(const void *src, void *dst, size_t bytes, size_t t, size_t n)
{
    /* 16-byte words; the arrays are padded to 256 bytes on both sides */
    const uint4 *a = static_cast<const uint4 *>(src);
    uint4 *b = static_cast<uint4 *>(dst);
    for (size_t i = t; i < (bytes + 15) / 16; i += n) b[i] = a[i];
}
__global__ void __launch_bounds__(TPB) k_tape_record(DevMesh m, TapeRecord r, EventLog log, int start)
{
    griddep_wait();
    const size_t t = blockIdx.x * (size_t)blockDim.x + threadIdx.x, n = (size_t)gridDim.x * blockDim.x;
    const size_t V = m.nv, B = m.nb, G = m.ng;
    switch (blockIdx.y) {
    case 0: copy_words(m.pos, r.pos, V * 16, t, n); break;
    case 1: copy_words(m.vb, r.vb, V * 16, t, n); break;
    case 2: copy_words(m.vg, r.vg, V * 16, t, n); break;
    case 3: copy_words(m.bv, r.bv, B * 8, t, n); break;
    case 4:
        copy_words(m.ven, r.ven, V, t, n);
        copy_words(m.ben, r.ben, B, t, n);
        break;
    case 5:
        copy_words(m.gvlen, r.gvlen, G * 4, t, n);
        copy_words(m.gen, r.gen, G, t, n);
        copy_words(m.gtype, r.gtype, G, t, n);
        break;
    default:
        for (size_t i = t; i < G * (SEVC_MAXV / 4); i += n) {
            const size_t g = i / (SEVC_MAXV / 4), j = i - g * (SEVC_MAXV / 4);
            if (4 * (int)j < m.gvlen[g]) reinterpret_cast<int4 *>(r.glist)[i] = reinterpret_cast<const int4 *>(m.glist)[i];
        }
    }
    if (start && t == 0 && blockIdx.y == 0) {
        *log.n = 0;
        *m.elog = log;
    }
}
/* enabled flags and velocities after the step; the log is switched off */
__global__ void __launch_bounds__(TPB) k_tape_after(DevMesh m, TapeRecord r)
{
    griddep_wait();
    const size_t t = blockIdx.x * (size_t)blockDim.x + threadIdx.x, n = (size_t)gridDim.x * blockDim.x;
    copy_words(m.vel, r.vel1, (size_t)m.nv * 16, t, n);
    copy_words(m.ven, r.ven1, m.nv, t, n);
    if (t == 0) *m.elog = EventLog{ nullptr, nullptr, 0 };
}

/* Grain statistics over grains [lo, hi): count, sum |A|, sum A^2, sum of
 * side counts, 3-sided count, min |A|, max |A|; per block into part, the
 * last block to finish sums the blocks (fixed order).  One block over all
 * grains took 12.7 ms at 500K grains; the FP64 work of the areas over the
 * whole GPU takes 0.06 ms. */
constexpr int NSTAT = 7;
__device__ __forceinline__ double stat_join(int k, double a, double b) { return k == 5 ? fmin(a, b) : (k == 6 ? fmax(a, b) : a + b); }
__global__ void __launch_bounds__(TPB) k_grain_stats(DevMesh m, int lo, int hi, double *part, double *out)
{
    __shared__ double red[NSTAT][TPB / 32];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    double v[NSTAT] = { 0, 0, 0, 0, 0, 1e300, 0 };
    for (int g = lo + blockIdx.x * TPB + threadIdx.x; g < hi; g += gridDim.x * TPB) {
        if (!m.gen[g]) continue;
        double a = fabs(grain_area(m, g));
        v[0] += 1;
        v[1] += a;
        v[2] += a * a;
        v[3] += m.gvlen[g];
        v[4] += m.gvlen[g] == 3;
        v[5] = fmin(v[5], a);
        v[6] = fmax(v[6], a);
    }
    for (int k = 0; k < NSTAT; k++) {
        for (int o = 16; o > 0; o >>= 1) v[k] = stat_join(k, v[k], __shfl_down_sync(0xffffffffu, v[k], o));
        if (lane == 0) red[k][warp] = v[k];
    }
    __syncthreads();
    if (threadIdx.x < NSTAT) {
        const int k = threadIdx.x;
        double s = red[k][0];
        for (int w = 1; w < TPB / 32; w++) s = stat_join(k, s, red[k][w]);
        part[blockIdx.x * NSTAT + k] = s;
    }
    const bool last = last_block(m.lastblk + 4);
    if (last && warp < NSTAT) {
        __threadfence();
        double s = warp == 5 ? 1e300 : 0.0;
        for (int b = lane; b < (int)gridDim.x; b += 32) s = stat_join(warp, s, __ldcg(part + b * NSTAT + warp));
        for (int o = 16; o > 0; o >>= 1) s = stat_join(warp, s, __shfl_down_sync(0xffffffffu, s, o));
        if (lane == 0) out[warp] = s;
    }
}

/* sum of a[0..n), in a fixed order: per block, then over the blocks by the
 * last one */
__global__ void __launch_bounds__(TPB) k_sum_ordered(const double *a, int n, double *part, int *ctr, double *out)
{
    __shared__ double red[TPB / 32];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    double s = 0.0;
    for (int i = blockIdx.x * TPB + threadIdx.x; i < n; i += gridDim.x * TPB) s += a[i];
    s = warp_sum(s);
    if (lane == 0) red[warp] = s;
    __syncthreads();
    if (threadIdx.x == 0) {
        double t = 0.0;
        for (int w = 0; w < TPB / 32; w++) t += red[w];
        part[blockIdx.x] = t;
    }
    const bool last = last_block(ctr);
    if (last && warp == 0) {
        __threadfence();
        double t = 0.0;
        for (int b = lane; b < (int)gridDim.x; b += 32) t += __ldcg(part + b);
        t = warp_sum(t);
        if (lane == 0) *out = t;
    }
}

} // namespace

/* blocks of the statistics kernels: two per SM cover the chip, more would
 * only add partial results */
static int stat_blocks(int n, int per) { int b = (n + per - 1) / per; return b < 1 ? 1 : (b < 2 * 152 ? b : 2 * 152); }
/* threads that keep private bins: as many as fit in 96 KB (two blocks per
 * SM), 16 at least (1024 bins: 128 KB); few grains take 64, which spreads
 * them over more blocks */
static int hist_threads(const DevMesh &m, int nbins)
{
    int T = TPB;
    while (T > 16 && (size_t)T * nbins * 8 > 96 * 1024) T /= 2;
    if (T > 64 && m.ng < 64 * 2 * 152) T = 64;
    return T;
}
size_t stat_doubles(int nbins) { return (size_t)2 * 152 * (nbins > NSTAT ? nbins : NSTAT); }
cudaError_t launch_histogram(const DevMesh &m, int nbins, double amax, double sc, double nnorm, double *part,
                             double *hist, cudaStream_t s)
{
    const int T = hist_threads(m, nbins);
    const size_t smem = (size_t)T * nbins * 8;
    /* the attribute belongs to the kernel, for every handle and thread: always
     * the largest any launch takes (1024 bins), never this one's size, under
     * which another thread's launch would be refused */
    cudaError_t e = cudaFuncSetAttribute(k_hist, cudaFuncAttributeMaxDynamicSharedMemorySize, 16 * 1024 * 8);
    if (e != cudaSuccess) return e;
    return launch_status(k_hist, stat_blocks(m.ng, T), TPB, smem, s, m, nbins, T, amax, sc, nnorm, part, hist);
}

void launch_hist_seed(const DevMesh &m, int nbins, double amax, double sc, double nnorm, const double *dldh,
                      double zero_sum, double *dlda, double2 *lam, cudaStream_t s)
{
    COUNT_LAUNCHES(1), k_hist_grad_area<<<nblk(m.ng), TPB, 0, s>>>(m, nbins, amax, sc, nnorm, dldh, zero_sum, dlda);
    COUNT_LAUNCHES(1), k_area_grad_to_vertices<<<nblk(m.nv), TPB, 0, s>>>(m, dlda, lam);
}

void launch_adjoint_step(const DevMesh &rec, const AdjointBuffers &a, double dt, double mu, double eps, double s_gb,
                         const EventRec *log, const int *nlog, const uint8_t *ven1, const double2 *vel1,
                         const signed char *sgn, bool nucleation, cudaStream_t s)
{
    launch_dep(k_adj_translate, nblk(rec.nv), TPB, s, rec.nv, dt, mu, a.lam, ven1, vel1, a.lx, a.lv, a.gmu);
    launch_dep(k_adj_events, rec.ninst, ADJ_TPB, s, rec.D, log, nlog, a.lx, a.lv, rec.voff, rec.ninst);
    const int vb = (rec.nv + ADJ_VPB - 1) / ADJ_VPB, gb = (rec.ng + ADJ_BLOCK - 1) / ADJ_BLOCK;
    launch_dep(k_adj_gather, vb + gb, ADJ_BLOCK, s, rec, mu, eps, s_gb, a.lx, a.lv, sgn, a.lam, a.ggam, a.gse, vb);
    if (nucleation) launch_dep(k_adj_nucleation, rec.ninst, ADJ_TPB, s, rec.D, log, nlog, a.lam, rec.voff, rec.ninst);
}

static int copy_blocks(const DevMesh &m) { int b = nblk(m.nv); return b < 4 * 152 ? b : 4 * 152; }
void launch_tape_record(const DevMesh &m, const TapeRecord &r, const EventLog &log, bool start, cudaStream_t s)
{
    const int b = copy_blocks(m);
    launch_dep(k_tape_record, dim3(b < 152 ? b : 152, 7), TPB, s, m, r, log, (int)start);
}
void launch_adjoint_signs(const DevMesh &m, const TapeRecord &first, size_t bytes, int steps, cudaStream_t s)
{
    for (int k = 0; k < steps; k += 65535) {
        TapeRecord r = first;
        auto shift = [&](auto *&p) { p = reinterpret_cast<std::remove_reference_t<decltype(p)>>((char *)p + k * bytes); };
        shift(r.pos); shift(r.glist); shift(r.gvlen); shift(r.gen); shift(r.sgn);
        launch_dep(k_adj_signs, dim3(nblk(m.ng), steps - k < 65535 ? steps - k : 65535), TPB, s, r, bytes, m.ng, m.D);
    }
}
void launch_tape_after(const DevMesh &m, const TapeRecord &r, cudaStream_t s)
{
    launch_dep(k_tape_after, copy_blocks(m), TPB, s, m, r);
}

void launch_grain_stats(const DevMesh &m, int lo, int hi, double *part, double *out, cudaStream_t s)
{
    COUNT_LAUNCHES(1), k_grain_stats<<<stat_blocks(hi - lo, TPB), TPB, 0, s>>>(m, lo, hi, part, out);
}

void launch_sum_ordered(const DevMesh &m, const double *a, int n, double *part, double *out, cudaStream_t s)
{
    COUNT_LAUNCHES(1), k_sum_ordered<<<stat_blocks(n, 4 * TPB), TPB, 0, s>>>(a, n, part, m.lastblk + 5, out);
}
