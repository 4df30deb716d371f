/*
 * Mesh invariants on the device: the checks of check_data
 * (src/utils.h:85-336, the tests that set is_valid = false), one thread
 * per boundary and vertex and a warp per grain, counted into one integer.  The host
 * restatement in sevc_host.c (sevc_host_check) counts the same violations
 * in the same way.  An index outside its array counts as one violation and
 * is not followed, so a damaged mesh is reported, never read out of bounds.
 */
#include "sevc_internal.h"
#include "sevc_host.h"

namespace {

constexpr int TPB = 256;

__device__ __forceinline__ bool inr(int x, int n) { return (unsigned)x < (unsigned)n; }

__device__ __forceinline__ void add_count(int *out, int bad)
{
    int s = bad;
    for (int o = 16; o > 0; o >>= 1) s += __shfl_down_sync(0xffffffffu, s, o);
    if ((threadIdx.x & 31) == 0 && s) atomicAdd(out, s);
}

__device__ __forceinline__ bool in_list(const DevMesh &m, int g, int v)
{
    const int *L = m.glist + (size_t)SEVC_MAXV * g;
    int n = min(max(m.gvlen[g], 0), SEVC_MAXV);
    for (int i = 0; i < n; i++)
        if (L[i] == v) return true;
    return false;
}

/* src/utils.h:85-158, per enabled boundary */
__device__ int check_boundary(const DevMesh &m, int b)
{
    int bad = 0;
    if (b < m.nb && m.ben[b]) {
        int2 e = m.bv[b];
        if (!inr(e.x, m.nv) || !inr(e.y, m.nv)) {
            bad = 1;
        } else {
            int4 sa = m.vb[e.x], sc = m.vb[e.y];
            bad += e.x == e.y;
            bad += !m.ven[e.x] || !m.ven[e.y];
            bad += sa.x != b && sa.y != b && sa.z != b;
            bad += sc.x != b && sc.y != b && sc.z != b;
            int s[6] = { sc.x, sc.y, sc.z, sa.x, sa.y, sa.z };
            bool ok_c = true, ok_a = true;
            for (int j = 0; j < 6; j++) {
                bool ok = inr(s[j], m.nb) && m.ben[s[j]];
                if (j < 3) ok_c &= ok; else ok_a &= ok;
            }
            bad += !ok_c;
            bad += !ok_a;
            int gic[2];
            int k = gintersect(m.vg[e.x], m.vg[e.y], gic);
            bad += k < 2 || gic[0] == gic[1];
        }
    }
    return bad;
}

/* src/utils.h:160-280, per enabled vertex */
__device__ int check_vertex(const DevMesh &m, int v)
{
    int bad = 0;
    if (v < m.nv && m.ven[v]) {
        int4 s4 = m.vb[v], g4 = m.vg[v];
        int s[3] = { s4.x, s4.y, s4.z }, g[3] = { g4.x, g4.y, g4.z }, nb[3] = { -1, -2, -3 };
        bad += s[0] == s[1] || s[1] == s[2] || s[2] == s[0];
        bad += g[0] == g[1] || g[1] == g[2] || g[2] == g[0];
        for (int j = 0; j < 3; j++) {
            bool gok = inr(g[j], m.ng);
            bad += !gok || !m.gen[g[j]];
            bad += !gok || !in_list(m, g[j], v);
            if (!inr(s[j], m.nb)) { bad += 1; continue; }
            int2 e = m.bv[s[j]];
            bad += !m.ben[s[j]];
            bad += e.x == e.y;
            nb[j] = e.x == v ? e.y : e.x;
            bad += e.x != v && e.y != v;
        }
        bad += nb[0] == nb[1] || nb[1] == nb[2] || nb[2] == nb[0];
    }
    return bad;
}

/* src/utils.h:282-336, per enabled grain, by a warp: its lanes read the
 * whole list (100 entries, all of them counted) side by side.  The lanes'
 * results add up to the grain's. */
__device__ int check_grain(const DevMesh &m, int g, int lane)
{
    if (g >= m.ng || !m.gen[g]) return 0;
    const int *L = m.glist + (size_t)SEVC_MAXV * g;
    const int n = m.gvlen[g];
    if (n < 0 || n > SEVC_MAXV) return lane == 0;
    int bad = 0, cnt = 0;
    bool out = false, stray = false;
    for (int j = lane; j < SEVC_MAXV; j += 32) {
        const int v = L[j];
        cnt += v != -1;
        if (j >= n) continue;
        if (!inr(v, m.nv)) { bad++; out = true; continue; }
        bad += !m.ven[v];
        int4 s = m.vg[v];
        stray |= s.x != g && s.y != g && s.z != g;
    }
    cnt = __reduce_add_sync(0xffffffffu, cnt);
    const bool any_out = __any_sync(0xffffffffu, out), any_stray = __any_sync(0xffffffffu, stray);
    if (lane == 0) bad += (!any_out && any_stray) + (cnt != n);
    return bad;
}

/* all three in one launch: blocks of boundaries, then of vertices, then of
 * grains (a warp each) */
__global__ void __launch_bounds__(TPB) k_check(DevMesh m, int bblocks, int vblocks, int *out)
{
    int k = blockIdx.x, bad;
    if (k < bblocks) bad = check_boundary(m, k * TPB + threadIdx.x);
    else if ((k -= bblocks) < vblocks) bad = check_vertex(m, k * TPB + threadIdx.x);
    else bad = check_grain(m, (k - vblocks) * (TPB / 32) + (threadIdx.x >> 5), threadIdx.x & 31);
    add_count(out, bad);
}

/* FP64 issue-rate probe: 8 independent fused multiply-add chains per
 * thread, so the pipe, not latency, limits the rate */
__global__ void k_fp64_rate(int iters, double a, double b, double *sink)
{
    double x[8];
    for (int k = 0; k < 8; k++) x[k] = threadIdx.x * 1e-3 + k;
    for (int i = 0; i < iters; i++)
#pragma unroll
        for (int k = 0; k < 8; k++) x[k] = fma(x[k], a, b);
    double s = 0;
    for (int k = 0; k < 8; k++) s += x[k];
    if (s == 12345.678) *sink = s;   /* keeps the chains live */
}


/* ---- the mesh for the host (sevc_get_state) ---- */
/* Every field in the host's layout, de-interleaved on the way: consecutive
 * threads store consecutive elements of one array, so that full lines go
 * over the link to host memory, which bounds the kernel (734 bytes per
 * grain at 170 GB/s measured: 4.3 ms at 1M grains). */
template <class T, class F> __device__ __forceinline__ void export_each(T *out, size_t n, F value)
{
    for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x)
        out[i] = value(i);
}
__global__ void __launch_bounds__(TPB) k_export(DevMesh m, sevc_mesh_host o, int part)
{
    const size_t V = m.nv, B = m.nb, G = m.ng;
    if (part & EXPORT_GRAINS) {
        const size_t n = G * SEVC_MAXV;
        if (((uintptr_t)o.glist & 15) == 0)
            export_each(reinterpret_cast<int4 *>(o.glist), n / 4, [&](size_t i) { return reinterpret_cast<const int4 *>(m.glist)[i]; });
        else
            export_each(o.glist, n, [&](size_t i) { return m.glist[i]; });
        export_each(o.gvlen, G, [&](size_t i) { return m.gvlen[i]; });
        export_each(o.garea, G, [&](size_t i) { return m.garea[i]; });
        export_each(o.gdadt, G, [&](size_t i) { return m.gdadt[i]; });
        export_each(o.gori, G, [&](size_t i) { return m.gori[i]; });
        export_each(o.gse, G, [&](size_t i) { return m.gse[i]; });
        export_each(o.gen, G, [&](size_t i) { return m.gen[i]; });
        export_each(o.gtype, G, [&](size_t i) { return m.gtype[i]; });
    }
    if (part & EXPORT_REST) {
        export_each(o.px, V, [&](size_t i) { return m.pos[i].x; });
        export_each(o.py, V, [&](size_t i) { return m.pos[i].y; });
        export_each(o.vx, V, [&](size_t i) { return m.vel[i].x; });
        export_each(o.vy, V, [&](size_t i) { return m.vel[i].y; });
        export_each(o.venergy, V, [&](size_t i) { return m.venergy[i]; });
        /* src/calculus.h:63-69: -term / grad_eps */
        export_each(o.vel_bnd_x, V, [&](size_t i) { return div_grad_eps(-m.terms[i].bx); });
        export_each(o.vel_grn_x, V, [&](size_t i) { return div_grad_eps(-m.terms[i].gx); });
        export_each(o.vel_bnd_y, V, [&](size_t i) { return div_grad_eps(-m.terms[i].by); });
        export_each(o.vel_grn_y, V, [&](size_t i) { return div_grad_eps(-m.terms[i].gy); });
        export_each(o.ven, V, [&](size_t i) { return m.ven[i]; });
        export_each(o.vb, 3 * V, [&](size_t i) { return reinterpret_cast<const int *>(m.vb)[4 * (i / 3) + i % 3]; });
        export_each(o.vg, 3 * V, [&](size_t i) { return reinterpret_cast<const int *>(m.vg)[4 * (i / 3) + i % 3]; });
        export_each(o.bini, B, [&](size_t i) { return m.bv[i].x; });
        export_each(o.bend, B, [&](size_t i) { return m.bv[i].y; });
        export_each(o.benergy, B, [&](size_t i) { return m.benergy[i]; });
        export_each(o.blen, B, [&](size_t i) { return m.blen[i]; });
        export_each(o.btext, B, [&](size_t i) { return m.btext[i]; });
        export_each(o.ben, B, [&](size_t i) { return m.ben[i]; });
        export_each(o.bcand, B, [&](size_t i) { return m.bcand[i]; });
    }
}

/* ---- state digests (sevc_state_digest) ---- */
__device__ __forceinline__ unsigned long long digest_mix(unsigned long long z)   /* splitmix64 finaliser */
{
    z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ULL;
    z = (z ^ (z >> 27)) * 0x94D049BB133111EBULL;
    return z ^ (z >> 31);
}
__device__ __forceinline__ unsigned long long ubits(int v) { return (unsigned long long)(unsigned)v; }
__device__ __forceinline__ unsigned long long ubits(double v) { return (unsigned long long)__double_as_longlong(v); }

/* elements of field f in the layout of sevc_get_state */
__device__ long long digest_len(const DevMesh &m, int f)
{
    if (f < 5) return m.nv;
    if (f < 7) return 3LL * m.nv;
    if (f < 13) return m.nb;
    if (f == 13) return (long long)SEVC_MAXV * m.ng;
    return m.ng;
}
__device__ unsigned long long digest_bits(const DevMesh &m, int f, long long i)
{
    switch (f) {
    case 0: return ubits(m.pos[i].x);
    case 1: return ubits(m.pos[i].y);
    case 2: return ubits(m.vel[i].x);
    case 3: return ubits(m.vel[i].y);
    case 4: return m.ven[i];
    case 5: return ubits(slot3(m.vb[i / 3], (int)(i % 3)));
    case 6: return ubits(slot3(m.vg[i / 3], (int)(i % 3)));
    case 7: return ubits(m.bv[i].x);
    case 8: return ubits(m.bv[i].y);
    case 9: return ubits(m.benergy[i]);
    case 10: return ubits(m.blen[i]);
    case 11: return m.ben[i];
    case 12: return m.bcand[i];
    case 13: return ubits(m.glist[i]);
    case 14: return ubits(m.gvlen[i]);
    case 15: return ubits(m.garea[i]);
    case 16: return ubits(m.gori[i]);
    case 17: return ubits(m.gse[i]);
    case 18: return m.gen[i];
    default: return m.gtype[i];
    }
}
/* blockIdx.y = field; the sum is order-independent, so the result does
 * not depend on the launch shape */
__global__ void k_digest(DevMesh m, unsigned long long *out)
{
    const int f = blockIdx.y;
    const long long n = digest_len(m, f);
    const unsigned long long salt = (unsigned long long)f << 56;
    unsigned long long acc = 0;
    for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x)
        acc += digest_mix(salt + (unsigned long long)i * 0x9E3779B97F4A7C15ULL + digest_bits(m, f, i));
    for (int o = 16; o > 0; o >>= 1) acc += __shfl_down_sync(0xffffffffu, acc, o);
    if ((threadIdx.x & 31) == 0) atomicAdd(out + f, acc);
}

} // namespace

/* FP64 multiply-add instructions (thread operations) per second on the
 * current device, measured with CUDA events */
extern "C" sevc_status sevc_measure_fp64_rate(double *ops_per_s)
{
    if (!ops_per_s) return SEVC_ERR_ARG;
    int dev = 0, nsm = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess)
        return SEVC_ERR_CUDA;
    double *sink = nullptr;
    cudaEvent_t e0, e1;
    if (cudaMalloc(&sink, sizeof(double)) != cudaSuccess) return SEVC_ERR_CUDA;
    cudaEventCreate(&e0);
    cudaEventCreate(&e1);
    int blocks = nsm * 8, threads = 256, iters = 4096;
    COUNT_LAUNCHES(1), k_fp64_rate<<<blocks, threads>>>(64, 1.0000001, 1e-9, sink);   /* warm-up */
    cudaEventRecord(e0);
    COUNT_LAUNCHES(1), k_fp64_rate<<<blocks, threads>>>(iters, 1.0000001, 1e-9, sink);
    cudaEventRecord(e1);
    float ms = 0;
    bool ok = cudaEventSynchronize(e1) == cudaSuccess && cudaEventElapsedTime(&ms, e0, e1) == cudaSuccess && ms > 0;
    cudaEventDestroy(e0);
    cudaEventDestroy(e1);
    cudaFree(sink);
    if (!ok) return SEVC_ERR_CUDA;
    *ops_per_s = (double)blocks * threads * iters * 8 / (ms * 1e-3);
    return SEVC_OK;
}

/* ---- self-test of the certified division / square root (vmag) ---- */
__device__ __forceinline__ unsigned long long mix64(unsigned long long z)   /* splitmix64 finaliser */
{
    z += 0x9E3779B97F4A7C15ULL;
    z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ULL;
    z = (z ^ (z >> 27)) * 0x94D049BB133111EBULL;
    return z ^ (z >> 31);
}
/* a double in [1, 2) from 52 random bits, times 2^k */
__device__ __forceinline__ double unit_pow2(unsigned long long u, int k)
{
    return __longlong_as_double((long long)((u & 0x000FFFFFFFFFFFFFULL) | ((unsigned long long)(1023 + k) << 52)));
}

/* counts: 0 divisions, 1 division mismatches, 2 divisions not certified,
 * 3 square roots, 4 square-root mismatches, 5 not certified, 6 vmag
 * evaluations, 7 vmag mismatches (a mismatch is a certified result whose
 * bits differ from the native operation's) */
__global__ void k_selftest_arith(long long n, unsigned long long seed, unsigned long long *counts)
{
    unsigned long long c[8] = {0, 0, 0, 0, 0, 0, 0, 0};
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x) {
        unsigned long long a = mix64(seed ^ (2 * i)), b = mix64(seed ^ (2 * i + 1)), kind = (a >> 60) & 7;
        /* division q / p with 0 <= q <= p */
        int kp = (int)((b >> 56) % 121) - 60;
        double p = unit_pow2(b, kp), q;
        if (kind < 4) {
            q = p * unit_pow2(a, -1 - (int)((a >> 52) & 7));          /* a general ratio */
        } else if (kind < 7) {
            /* q = RN(p m) for a rounding midpoint m = k 2^-53 + 2^-54 of (1/2, 1) */
            double kd = __longlong_as_double((long long)((a & 0x000FFFFFFFFFFFFFULL) | (1022ULL << 52)));
            q = __fma_rn(p, kd, p * 0x1p-54);
            if (kind == 6) q = __longlong_as_double(dbits(q) + (((a >> 59) & 1) ? 1 : -1));
            if (dbits(q) > dbits(p)) q = p;
        } else {
            int w = (int)((a >> 40) & 3);
            q = w == 0 ? p : (w == 1 ? 0.0 : p * 0x1p-1040);            /* r = 1, 0, subnormal q */
        }
        double r;
        c[0]++;
        if (div_fast(q, p, r)) { if (dbits(r) != dbits(q / p)) c[1]++; }
        else c[2]++;
        /* square root of t in [1, 2) */
        double t;
        if (kind < 4) {
            t = unit_pow2(a, 0);
        } else {
            /* t = RN(m^2) next to the square of a midpoint m = s + 2^-53 */
            double s = unit_pow2(a, 0);
            if (s > 1.4142135623730950) s = s - 0.4142135623730950;
            t = __fma_rn(s, s, s * 0x1p-52);
            if (kind == 6) t = __longlong_as_double(dbits(t) + (((a >> 59) & 1) ? 1 : -1));
            if ((dbits(t) >> 52) != 1023) t = 1.5;
        }
        c[3]++;
        if (sqrt_fast(t, r)) { if (dbits(r) != dbits(sqrt(t))) c[4]++; }
        else c[5]++;
        /* whole vector2_mag on coordinates of random sign and scale */
        double x = unit_pow2(mix64(a), (int)(b & 63) - 32), y = unit_pow2(mix64(b), (int)((a >> 8) & 63) - 32);
        if (kind == 7) y = ((a >> 44) & 1) ? x : 0.0;
        if ((a >> 48) & 1) x = -x;
        if ((b >> 48) & 1) y = -y;
        c[6]++;
        if (dbits(vmag(x, y)) != dbits(vmag_native(x, y))) c[7]++;
    }
    for (int k = 0; k < 8; k++) {
        unsigned long long v = c[k];
        for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
        if ((threadIdx.x & 31) == 0 && v) atomicAdd(counts + k, v);
    }
}

extern "C" sevc_status sevc_selftest_arith(long long n, unsigned long long seed, long long *counts)
{
    if (!counts || n < 0) return SEVC_ERR_ARG;
    unsigned long long *d = nullptr;
    if (cudaMalloc(&d, 8 * sizeof(unsigned long long)) != cudaSuccess) return SEVC_ERR_CUDA;
    bool ok = cudaMemset(d, 0, 8 * sizeof(unsigned long long)) == cudaSuccess;
    if (ok) {
        COUNT_LAUNCHES(1), k_selftest_arith<<<152 * 8, 256>>>(n, seed, d);
        unsigned long long h[8];
        ok = cudaGetLastError() == cudaSuccess && cudaMemcpy(h, d, sizeof h, cudaMemcpyDeviceToHost) == cudaSuccess;
        for (int k = 0; ok && k < 8; k++) counts[k] = (long long)h[k];
    }
    cudaFree(d);
    return ok ? SEVC_OK : SEVC_ERR_CUDA;
}

void launch_check(const DevMesh &m, int *out, cudaStream_t s)
{
    cudaMemsetAsync(out, 0, sizeof(int), s);
    const int bb = (m.nb + TPB - 1) / TPB, vb = (m.nv + TPB - 1) / TPB, gb = (m.ng + TPB / 32 - 1) / (TPB / 32);
    if (bb + vb + gb > 0) COUNT_LAUNCHES(1), k_check<<<bb + vb + gb, TPB, 0, s>>>(m, bb, vb, out);
}

cudaError_t launch_export(const DevMesh &m, const sevc_mesh_host &o, int part, cudaStream_t s)
{
    size_t n = (size_t)m.nv + m.nb;
    size_t g = (n + TPB - 1) / TPB;
    return launch_status(k_export, (unsigned)(g < 8 * 152 ? (g ? g : 1) : 8 * 152), TPB, 0, s, m, o, part);
}

void launch_digest(const DevMesh &m, unsigned long long *out, cudaStream_t s)
{
    long long n = (long long)SEVC_MAXV * m.ng;
    long long gx = (n + TPB - 1) / TPB;
    if (gx > 4 * 152) gx = 4 * 152;
    if (gx < 1) gx = 1;
    COUNT_LAUNCHES(1), k_digest<<<dim3((unsigned)gx, SEVC_DIGEST_FIELDS), TPB, 0, s>>>(m, out);
}
