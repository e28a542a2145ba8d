// The multigrid-preconditioned PCG direction solve of one scene as one cooperative launch.
//
// A solve is a chain of short dependent phases: the SpMV, the recurrences, and down and up the
// levels of the V-cycle (mg.cu describes the cycle).  As separate kernels replayed from a graph a
// phase cost 5 to 20 us whatever its size: a launch, a ramp, and too few CTAs, each bound by its own
// SM's FP64 pipe (one warp-wide FP64 instruction per ~19 clocks and SM on GB300).  Here one CTA per
// SM stays resident and the phases are separated by grid barriers.  What that changes:
//   * small scenes spread over all SMs: a level-0 slice of 32 rows is shared by up to 8 warps;
//   * contact rows (block CSR, some 20 blocks in a row, next to rows without any) are taken by
//     groups of 8 lanes over all warps of the CTA instead of one thread per row;
//   * the convergence test, the recurrences' scalars and the smoother weights are computed by every
//     CTA from the same per-CTA partial sums in the same order, so there is no single-CTA step;
//   * the post-smoothing of a level also prolongates its result into the next finer level.
// Per iteration: 3 L barriers for L levels.  Every sum runs in a fixed order for a given GPU and
// scene, so a solve is reproducible bit for bit.
// Per PCG iteration on a GB300, kernel chain against one launch: 1,458 vertices 40 us against 28, 1,736 with 608
// contact rows 65 / 50, 6,182 with 2,048 67 / 53, 10,376 with 5,133 70 / 55, 24,584 with 9,531 91 / 83 (system.cu has the
// line between them).  What is left of the small scenes' time is the
// barriers (1.1 us each) and, per phase, one or two dependent L2 accesses and a chain of FP64
// instructions at some 50 ns each.
#include <cooperative_groups.h>
#include <cuda_runtime.h>

#include "ctx.cuh"
#include "mg_node.cuh"
#include "pcg.cuh"

namespace cg = cooperative_groups;

namespace fipc {

constexpr int PP_THREADS = 512, PP_WARPS = PP_THREADS / 32;
constexpr int MG_POWER_ITERS = 8;          // power iterations per level and solve
constexpr unsigned FULL = 0xffffffffu;

struct PcgLoop {
    PCGArgs a;
    MgArgs m;
    const double* rhs;
    double rtol;
    int maxit, guess, contact;   // guess: x holds an initial guess; contact: the contact matrix has blocks
    int n_slices;
    double* part;                // [3][grid] dot products, then [2][levels][grid] power iteration norms
    double* omega;               // [levels] smoother weights
    double *pv0[MG_LEVELS_CAP], *pv1[MG_LEVELS_CAP];
};

struct PpShared {
    double row[3 * PP_THREADS];  // per-warp row sums
    double con[3 * PP_THREADS];  // contact sums
    double tot[8];
    double alpha, beta, gamma, inv_gamma, inv_alpha, tol2;   // scalars of the recurrences
    int done;
    int tiny;                    // gamma is subnormal (tolerance 0, a residual of some 1e-154) and its reciprocal may be infinite
    unsigned mask[PP_WARPS];     // rows of a slice with contact blocks
    int next;                    // next contact task of the pass
};

// Every phase has the form: loads that need nothing from the phases before (indices, and data that
// the same thread wrote), the barrier, the work.
__device__ __forceinline__ void barrier() { cg::this_grid().sync(); }

// ---------------------------------------------------------------- sums
// totals of n <= 8 per-CTA partials part[c * grid + cta] into sh.tot, the same order in every CTA;
// the loads of a lane are issued together (a dependent L2 access costs about half a microsecond).
// f maps a total (on one lane): scalar FP64 work is never repeated by a CTA's threads, since every
// warp's copy of it would take the SM's FP64 pipe for the same time.
template <class F>
__device__ __forceinline__ void grid_totals(const double* part, int n, PpShared& sh, F f) {
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    if (w < n) {
        double t = 0.0;
        for (int b0 = lane; b0 < (int)gridDim.x; b0 += 160) {
            double v[5];
#pragma unroll
            for (int q = 0; q < 5; ++q) v[q] = b0 + 32 * q < (int)gridDim.x ? __ldcg(part + w * gridDim.x + b0 + 32 * q) : 0.0;
            t += ((v[0] + v[1]) + (v[2] + v[3])) + v[4];
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) t += __shfl_down_sync(FULL, t, o);
        if (lane == 0) sh.tot[w] = f(t);
    }
    __syncthreads();
}

// the CTA's sums of NV values of its first n threads (n a multiple of 32) into part[c * grid + cta]
template <int NV>
__device__ __forceinline__ void cta_partials(const double (&v)[NV], int n, PpShared& sh, double* part) {
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    if ((int)threadIdx.x < n) {
#pragma unroll
        for (int c = 0; c < NV; ++c) sh.row[c * PP_THREADS + threadIdx.x] = v[c];
    }
    __syncthreads();
    if (w < NV) {
        double t = 0.0;
        for (int k = lane; k < n; k += 32) t += sh.row[w * PP_THREADS + k];
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) t += __shfl_down_sync(FULL, t, o);
        if (lane == 0) part[w * gridDim.x + blockIdx.x] = t;
    }
    __syncthreads();
}

// ---------------------------------------------------------------- level-0 rows
// Slice j of a CTA is gridDim.x j + (blockIdx.x + 61 j) mod gridDim.x: the shift keeps a CTA from
// meeting the same part of a regular mesh's cross-section in every slice (rows at the surface are
// shorter).  Slices are taken in passes of at most PP_WARPS; in a pass, warp q finishes the rows of
// its slice q, so a row belongs to the same thread in every phase.
struct Slices {
    int n, pass, G;   // slices of this CTA, slices per pass, warps per slice
};
__device__ __forceinline__ int slice_of(int cta, int j) { return gridDim.x * j + (cta + 61 * j) % gridDim.x; }
__device__ __forceinline__ Slices my_slices(const PcgLoop& P, int cta) {
    Slices s;
    const int full = P.n_slices / gridDim.x, rem = P.n_slices % gridDim.x;
    s.n = full + ((int)((cta + 61 * full) % gridDim.x) < rem ? 1 : 0);
    const int passes = (s.n + PP_WARPS - 1) / PP_WARPS;
    s.pass = passes ? (s.n + passes - 1) / passes : 1;
    s.G = min(PP_WARPS / s.pass, 8);
    return s;
}

template <class T>
struct Vec;
template <>
struct Vec<double> {
    static constexpr int NB = 1;   // blocks of a row in flight: FP64 issue binds, not latency
    const double* v;
    int st;
    // vectors change during the kernel: plain loads, never through the read-only path
    __device__ __forceinline__ void load(int j, double (&x)[3]) const {
        if (st == 4) {
            const double2 q = *reinterpret_cast<const double2*>(v + 4 * (size_t)j);
            x[0] = q.x;
            x[1] = q.y;
            x[2] = v[4 * (size_t)j + 2];
        } else {
            x[0] = v[3 * (size_t)j];
            x[1] = v[3 * (size_t)j + 1];
            x[2] = v[3 * (size_t)j + 2];
        }
    }
};
template <>
struct Vec<float> {
    static constexpr int NB = 2;
    const float* v;
    __device__ __forceinline__ void load(int j, float (&x)[3]) const {
        const float4 q = *reinterpret_cast<const float4*>(v + 4 * (size_t)j);
        x[0] = q.x;
        x[1] = q.y;
        x[2] = q.z;
    }
};

template <class T>
__device__ __forceinline__ void add_block(const T (&b)[9], const T (&x)[3], T (&s)[3]) {
    s[0] = fma(b[0], x[0], fma(b[1], x[1], fma(b[2], x[2], s[0])));
    s[1] = fma(b[3], x[0], fma(b[4], x[1], fma(b[5], x[2], s[1])));
    s[2] = fma(b[6], x[0], fma(b[7], x[1], fma(b[8], x[2], s[2])));
}

// a warp's share of a slice: its slots k, k + G, ...; the column ids of the next NB of them.  A slice's
// padding slots hold zero blocks and the row's own id; past the last vertex the id is clamped.
template <int NB>
struct RowCursor {
    int base, slots, k, col[NB];
    __device__ __forceinline__ void open(const PCGArgs& a, int s, int g, int G) {
        base = __ldg(a.soff + s);
        slots = __ldg(a.soff + s + 1) - base;
        k = g;
        cols(a, G);
    }
    __device__ __forceinline__ void cols(const PCGArgs& a, int G) {
#pragma unroll
        for (int q = 0; q < NB; ++q)
            if (k + q * G < slots) col[q] = min(__ldg(a.scol + (size_t)(base + k + q * G) * 32 + (threadIdx.x & 31)), a.nV - 1);
    }
};

// the contact blocks of a quarter of a slice's rows with contact: groups of 8 lanes take one row
// each, lane q of a group the row's blocks q, q + 8, ...; sums to cs[c][row of the pass]
template <class T>
__device__ __forceinline__ void contact_task(const PcgLoop& P, const T* __restrict__ cv, const Vec<T>& v, int s, int q, int part,
                                             PpShared& sh, T* cs) {
    const PCGArgs& a = P.a;
    const int lane = threadIdx.x & 31, sub = lane & 7, i = 32 * s + lane;
    int b = 0, e = 0;
    if (i < a.nV && !a.fixed[i]) {
        b = __ldg(a.crp + i);
        e = __ldg(a.crp + i + 1);
    }
    const unsigned mask = __ballot_sync(FULL, e > b);
    if (part == 0 && lane == 0) sh.mask[q] = mask;
    const int n = __popc(mask);
    for (int r0 = 4 * part; r0 < n; r0 += 16) {
        const int r = r0 + (lane >> 3);
        const int row = r < n ? nth_bit(mask, r) : 0;
        const int eb = __shfl_sync(FULL, b, row), ee = __shfl_sync(FULL, e, row);
        T y[3] = {T(0), T(0), T(0)};
        if (r < n) {
#pragma unroll 2
            for (int k = eb + sub; k < ee; k += 8) {
                T m[9], x[3];
                v.load(__ldg(a.cci + k), x);
#pragma unroll
                for (int c = 0; c < 9; ++c) m[c] = __ldg(cv + 9 * (size_t)k + c);
                add_block(m, x, y);
            }
        }
        __syncwarp();
#pragma unroll
        for (int o = 4; o > 0; o >>= 1)
#pragma unroll
            for (int c = 0; c < 3; ++c) y[c] += __shfl_xor_sync(FULL, y[c], o);
        if (sub == 0 && r < n) {
#pragma unroll
            for (int c = 0; c < 3; ++c) cs[c * PP_THREADS + 32 * q + row] = y[c];
        }
    }
}

// for every row i of the CTA: fin(i, st, y) with y = (A v)_i (zero at Dirichlet rows), A the elastic
// values ev (sliced ELL) plus the contact values cv (block CSR); st = own(i), what the row's thread
// loads while the CTA's other warps finish
template <bool SYNC, class T, class OWN, class FIN>
__device__ __forceinline__ void rows_apply(const PcgLoop& P, const T* __restrict__ ev, const T* __restrict__ cv, const Vec<T> v,
                                           PpShared& sh, OWN own, FIN fin) {
    constexpr int NB = Vec<T>::NB;
    const PCGArgs& a = P.a;
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    T* el = reinterpret_cast<T*>(sh.row);
    T* cs = reinterpret_cast<T*>(sh.con);
    const int me = (int)blockIdx.x;
    const Slices S = my_slices(P, me);
    if (threadIdx.x == 0) sh.next = 0;
    for (int j0 = 0; j0 < S.n || j0 == 0; j0 += S.pass) {
        const int nsl = min(S.pass, S.n - j0);
        RowCursor<NB> cur;
        const bool mine = w < nsl * S.G;
        if (mine) cur.open(a, slice_of(me, j0 + w / S.G), w % S.G, S.G);
        const int i = w < nsl ? 32 * slice_of(me, j0 + w) + lane : a.nV;
        if (j0 == 0 && SYNC) barrier();
        if (j0 == 0 && !SYNC) __syncthreads();
        if (mine) {
            T y[3] = {T(0), T(0), T(0)};
            while (cur.k + (NB - 1) * S.G < cur.slots) {
                T b[NB][9], x[NB][3];
#pragma unroll
                for (int q = 0; q < NB; ++q) {
                    const T* B = ev + (size_t)(cur.base + cur.k + q * S.G) * 288 + lane;
#pragma unroll
                    for (int c = 0; c < 9; ++c) b[q][c] = __ldg(B + 32 * c);
                    v.load(cur.col[q], x[q]);
                }
                cur.k += NB * S.G;
                cur.cols(a, S.G);
#pragma unroll
                for (int q = 0; q < NB; ++q) add_block(b[q], x[q], y);
            }
            if (NB > 1 && cur.k < cur.slots) {
                T b[9], x[3];
                const T* B = ev + (size_t)(cur.base + cur.k) * 288 + lane;
#pragma unroll
                for (int c = 0; c < 9; ++c) b[c] = __ldg(B + 32 * c);
                v.load(cur.col[0], x);
                add_block(b, x, y);
            }
#pragma unroll
            for (int c = 0; c < 3; ++c) el[c * PP_THREADS + threadIdx.x] = y[c];
        }
        decltype(own(0)) st{};
        if (i < a.nV) st = own(i);
        if (P.contact) {
            // tasks (slice, quarter of its contact rows), taken as warps come free
            for (;;) {
                int t = 0;
                if (lane == 0) t = atomicAdd(&sh.next, 1);
                t = __shfl_sync(FULL, t, 0);
                if (t >= 4 * nsl) break;
                contact_task<T>(P, cv, v, slice_of(me, j0 + (t >> 2)), t >> 2, t & 3, sh, cs);
            }
        }
        __syncthreads();
        if (threadIdx.x == 0) sh.next = 0;
        if (i < a.nV) {
            T y[3];
#pragma unroll
            for (int c = 0; c < 3; ++c) {
                const T* e = el + c * PP_THREADS + 32 * (w * S.G) + lane;
                y[c] = e[0];
                if (S.G == 8) y[c] = ((y[c] + e[32]) + (e[64] + e[96])) + ((e[128] + e[160]) + (e[192] + e[224]));
                else
                    for (int g = 1; g < S.G; ++g) y[c] += e[32 * g];
            }
            if (P.contact && (sh.mask[w] >> lane & 1)) {
#pragma unroll
                for (int c = 0; c < 3; ++c) y[c] += cs[c * PP_THREADS + 32 * w + lane];
            }
            if (a.fixed[i]) y[0] = y[1] = y[2] = T(0);
            fin(i, st, y);
        }
        __syncthreads();
    }
}

// fin(i, st) for every row of the CTA, by the same thread as in rows_apply; st = own(i) of the first
// pass is loaded before the work of `after` (the barrier and what follows it for the whole CTA)
template <class OWN, class AFTER, class FIN>
__device__ __forceinline__ void rows_each(const PcgLoop& P, OWN own, AFTER after, FIN fin) {
    const int me = (int)blockIdx.x;
    const Slices S = my_slices(P, me);
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    for (int j0 = 0; j0 < S.n || j0 == 0; j0 += S.pass) {
        const int i = w < min(S.pass, S.n - j0) ? 32 * slice_of(me, j0 + w) + lane : P.a.nV;
        decltype(own(0)) st{};
        if (i < P.a.nV) st = own(i);
        if (j0 == 0 && !after()) return;
        if (i < P.a.nV) fin(i, st);
    }
}
__device__ __forceinline__ Vec<double> vec4(const double* v) { return Vec<double>{v, 4}; }
struct None {};
struct D3 {
    double v[3];
};
__device__ __forceinline__ D3 ld_d3(const double* p, int i) {
    return D3{{p[3 * (size_t)i], p[3 * (size_t)i + 1], p[3 * (size_t)i + 2]}};
}

// a member i of a node and its offset; loaded before the barrier for a lane's first member
struct Member {
    int i;   // -1: none (past the end, or a Dirichlet vertex)
    double d0, d1, d2;
    __device__ __forceinline__ void open(const PcgLoop& P, const MgLev& L, int l, int k, int k1) {
        i = k < k1 ? __ldg(L.mem + k) : -1;
        if (i >= 0 && l == 1 && P.a.fixed[i]) i = -1;
        if (i < 0) return;
        d0 = __ldg(L.d + 3 * (size_t)i);
        d1 = __ldg(L.d + 3 * (size_t)i + 1);
        d2 = __ldg(L.d + 3 * (size_t)i + 2);
    }
};

// zf_i += P Y for member m of a node of level l (Y the node's six values).  Into level 0: stride 4,
// and the FP32 copy.
__device__ __forceinline__ void prolong_member(const PcgLoop& P, int l, const Member& m, const double (&Y)[6]) {
    if (m.i < 0) return;
    const double u0 = Y[0] + (Y[4] * m.d2 - Y[5] * m.d1), u1 = Y[1] + (Y[5] * m.d0 - Y[3] * m.d2), u2 = Y[2] + (Y[3] * m.d1 - Y[4] * m.d0);
    if (l == 1) {
        double* z = P.m.z0 + 4 * (size_t)m.i;
        const double2 q = *reinterpret_cast<const double2*>(z);
        const double z0 = q.x + u0, z1 = q.y + u1, z2 = z[2] + u2;
        *reinterpret_cast<double2*>(z) = make_double2(z0, z1);
        z[2] = z2;
        if (P.m.z0f) *reinterpret_cast<float4*>(P.m.z0f + 4 * (size_t)m.i) = make_float4((float)z0, (float)z1, (float)z2, 0.f);
    } else {
        double2* z = reinterpret_cast<double2*>(P.m.L[l - 1].z + 6 * (size_t)m.i);
        const double2 a = z[0], b = z[1], c = z[2];
        z[0] = make_double2(a.x + u0, a.y + u1);
        z[1] = make_double2(b.x + u2, b.y + Y[3]);
        z[2] = make_double2(c.x + Y[4], c.y + Y[5]);
    }
}

// ---------------------------------------------------------------- phases
// residual of the initial guess, block-Jacobi inverse, u = M^-1 r, |r|^2 and |b|^2; the start
// vectors of the power iterations and their norms
__device__ __forceinline__ void phase_start(const PcgLoop& P, PpShared& sh) {
    const PCGArgs& a = P.a;
    double acc[2] = {0.0, 0.0}, nrm = 0.0;
    auto fin = [&](int i, const double (&y)[3]) {
        const bool fx = a.fixed[i] != 0;
        double M[9], r[3];
        jacobi_block_inverse(a, i, fx, M);
        for (int k = 0; k < 9; ++k) a.minv[9 * (size_t)i + k] = M[k];
        for (int d = 0; d < 3; ++d) {
            const double b = fx ? 0.0 : P.rhs[3 * (size_t)i + d];
            r[d] = fx ? 0.0 : b - y[d];
            a.r[3 * (size_t)i + d] = r[d];
            a.p[3 * (size_t)i + d] = 0.0;
            a.s[3 * (size_t)i + d] = 0.0;
            acc[0] += r[d] * r[d];
            acc[1] += b * b;
            const unsigned long long h = ((unsigned long long)(3 * (long long)i + d) * 2654435761ull) % 1000ull;
            const double val = fx ? 0.0 : (double)h / 1000.0 - 0.5;
            P.pv0[0][4 * (size_t)i + d] = val;
            nrm += val * val;
        }
        P.pv0[0][4 * (size_t)i + 3] = 0.0;
        for (int d = 0; d < 3; ++d) a.u[4 * (size_t)i + d] = M[3 * d] * r[0] + M[3 * d + 1] * r[1] + M[3 * d + 2] * r[2];
        a.u[4 * (size_t)i + 3] = 0.0;
    };
    if (P.guess) {
        rows_apply<false, double>(P, a.sval, a.cva, Vec<double>{a.x, 3}, sh, [](int) { return None{}; },
                                  [&](int i, None, const double (&y)[3]) { fin(i, y); });
    } else {
        const double zero[3] = {0.0, 0.0, 0.0};
        rows_each(P, [](int) { return None{}; }, [] { return true; }, [&](int i, None) { fin(i, zero); });
    }
    cta_partials<2>(acc, PP_THREADS, sh, P.part);
    const double n0[1] = {nrm};
    double* np = P.part + 3 * gridDim.x;
    cta_partials<1>(n0, PP_THREADS, sh, np);
    for (int l = 1; l < P.m.levels - 1; ++l) {
        double s = 0.0;
        for (long long e = blockIdx.x * (long long)PP_THREADS + threadIdx.x; e < 6ll * P.m.L[l].n; e += (long long)gridDim.x * PP_THREADS) {
            const double val = (double)(((unsigned long long)e * 2654435761ull) % 1000ull) / 1000.0 - 0.5;
            P.pv0[l][e] = val;
            s += val * val;
        }
        const double v[1] = {s};
        cta_partials<1>(v, PP_THREADS, sh, np + l * gridDim.x);
    }
}

// after phase_start: the squared tolerance; true when the start already meets it
__device__ __forceinline__ bool phase_tolerance(const PcgLoop& P, PpShared& sh) {
    barrier();
    grid_totals(P.part, 2, sh, [](double t) { return t; });
    if (threadIdx.x == 0) {
        const double rr = sh.tot[0];
        sh.tol2 = P.rtol * P.rtol * sh.tot[1];
        sh.inv_gamma = sh.inv_alpha = 1.0;
        sh.tiny = 0;
        sh.done = rr == 0.0 || rr <= sh.tol2;
        if (blockIdx.x == 0 && sh.done) P.a.flag[0] = 1;
    }
    __syncthreads();
    return sh.done;
}

// power iteration k of every level at once: vout = D^-1 A (vin / |vin|)
__device__ __forceinline__ void phase_power(const PcgLoop& P, PpShared& sh, int k) {
    const PCGArgs& a = P.a;
    const int nl = P.m.levels - 1, lane = threadIdx.x & 31, w = threadIdx.x >> 5, p = lane % 6;
    const double* pin = P.part + (3 + (k & 1) * P.m.levels) * gridDim.x;
    double* pout = P.part + (3 + ((k + 1) & 1) * P.m.levels) * gridDim.x;
    barrier();
    grid_totals(pin, nl, sh, [](double t) { return 1.0 / sqrt(t); });
    const double sc = sh.tot[0];
    double s = 0.0;
    double* vout = (k & 1) ? P.pv0[0] : P.pv1[0];
    rows_apply<false, double>(P, a.sval, a.cva, vec4((k & 1) ? P.pv1[0] : P.pv0[0]), sh, [](int) { return None{}; },
                              [&](int i, None, double (&y)[3]) {
        const bool fx = a.fixed[i] != 0;
        for (int d = 0; d < 3; ++d) y[d] = fx ? 0.0 : y[d] * sc;
        const double* M = a.minv + 9 * (size_t)i;
        for (int d = 0; d < 3; ++d) {
            const double o = M[3 * d] * y[0] + M[3 * d + 1] * y[1] + M[3 * d + 2] * y[2];
            vout[4 * (size_t)i + d] = o;
            s += o * o;
        }
        vout[4 * (size_t)i + 3] = 0.0;
    });
    {
        const double v[1] = {s};
        cta_partials<1>(v, PP_THREADS, sh, pout);
    }
    for (int l = 1; l < nl; ++l) {
        const MgLev& L = P.m.L[l];
        const double sl = sh.tot[l];
        const double* vi = (k & 1) ? P.pv1[l] : P.pv0[l];
        double* vo = (k & 1) ? P.pv0[l] : P.pv1[l];
        s = 0.0;
        for (int I = blockIdx.x + gridDim.x * w; I < L.n; I += gridDim.x * PP_WARPS) {
            double y = 0.0;
            if (lane < 30) {
                NodeCursor<2> c;
                c.open(L, I, lane / 6, 5);
                y = node_row<true>(L, c, vi, p, 5);
            }
            __syncwarp();
            const double z = node_minv(L.minv + 36 * (size_t)I, node_gather(y, p) * sl, 1.0, 0, p);
            if (lane < 6) {
                vo[6 * (size_t)I + lane] = z;
                s += z * z;
            }
        }
        const double v[1] = {s};
        cta_partials<1>(v, PP_THREADS, sh, pout + l * gridDim.x);
    }
}

// smoother weights w_l = 4 / (3 * 1.05 * rho_l) from the last power iteration's norms, then z0 = w0 u
__device__ __forceinline__ void phase_weights(const PcgLoop& P, PpShared& sh) {
    const PCGArgs& a = P.a;
    const double* pn = P.part + (3 + (MG_POWER_ITERS & 1) * P.m.levels) * gridDim.x;
    barrier();
    grid_totals(pn, P.m.levels - 1, sh, [](double t) {
        const double rho = sqrt(t);
        return rho > 0.0 ? 4.0 / (3.0 * 1.05 * rho) : 1.0;
    });
    const double w0 = sh.tot[0];
    if (blockIdx.x == 0 && (int)threadIdx.x < P.m.levels - 1) P.omega[threadIdx.x] = sh.tot[threadIdx.x];
    rows_each(P, [](int) { return None{}; }, [] { return true; }, [&](int i, None) {
        double z[3];
        for (int d = 0; d < 3; ++d) {
            z[d] = w0 * a.u[4 * (size_t)i + d];
            P.m.z0[4 * (size_t)i + d] = z[d];
        }
        P.m.z0[4 * (size_t)i + 3] = 0.0;
        if (P.m.z0f) *reinterpret_cast<float4*>(P.m.z0f + 4 * (size_t)i) = make_float4((float)z[0], (float)z[1], (float)z[2], 0.f);
    });
}

// w = A u and the partial sums of (r, u), (w, u), (r, r)
__device__ __forceinline__ void phase_spmv(const PcgLoop& P, PpShared& sh) {
    const PCGArgs& a = P.a;
    struct Own {
        D3 u, r;
    };
    double acc[3] = {0.0, 0.0, 0.0};
    rows_apply<true, double>(P, a.sval, a.cva, vec4(a.u), sh,
                            [&](int i) {
                                const double* u = a.u + 4 * (size_t)i;
                                return Own{D3{{u[0], u[1], u[2]}}, ld_d3(a.r, i)};
                            },
                            [&](int i, const Own& o, const double (&y)[3]) {
#pragma unroll
                                for (int d = 0; d < 3; ++d) {
                                    a.w[3 * (size_t)i + d] = y[d];
                                    acc[0] = fma(o.r.v[d], o.u.v[d], acc[0]);
                                    acc[1] = fma(y[d], o.u.v[d], acc[1]);
                                    acc[2] = fma(o.r.v[d], o.r.v[d], acc[2]);
                                }
                            });
    cta_partials<3>(acc, 32 * my_slices(P, blockIdx.x).pass, sh, P.part);
}

// iteration k: convergence test, alpha and beta from the dot products (Chronopoulos-Gear), then
// p = u + beta p, s = w + beta s, x += alpha p, r -= alpha s, z0 = w0 M^-1 r.  True when converged.
__device__ __forceinline__ bool phase_update(const PcgLoop& P, PpShared& sh, int k) {
    const PCGArgs& a = P.a;
    struct Own {
        D3 u, p, w, s, x, r;
    };
    double alpha = 0.0, beta = 0.0, w0 = 0.0;
    rows_each(P,
              [&](int i) {
                  const double* u = a.u + 4 * (size_t)i;
                  return Own{D3{{u[0], u[1], u[2]}}, ld_d3(a.p, i), ld_d3(a.w, i), ld_d3(a.s, i), ld_d3(a.x, i), ld_d3(a.r, i)};
              },
              [&] {
                  barrier();
                  w0 = P.omega[0];
                  grid_totals(P.part, 3, sh, [](double t) { return t; });
                  if (threadIdx.x == 0) {
                      const double G = sh.tot[0];
                      sh.done = sh.tot[2] <= sh.tol2;
                      sh.beta = k == 0 ? 0.0 : G * sh.inv_gamma;
                      if (sh.tiny) {
                          sh.beta = G / sh.gamma;
                          sh.alpha = G / (sh.tot[1] - sh.beta * G / sh.alpha);
                          // subnormal sums hold few digits, or none: a step that they do not give is left out
                          if (!isfinite(sh.alpha) || !isfinite(sh.beta)) sh.alpha = sh.beta = 0.0;
                      } else {
                          sh.alpha = G / (sh.tot[1] - sh.beta * G * sh.inv_alpha);
                      }
                      if (blockIdx.x == 0) {
                          a.flag[3] = sh.done ? k : k + 1;
                          if (sh.done) {
                              a.flag[0] = 1;
                              a.flag[1] = k;
                          }
                      }
                  }
                  __syncthreads();
                  alpha = sh.alpha;
                  beta = sh.beta;
                  if (threadIdx.x == 0) {   // for the next iteration, off the critical path
                      sh.gamma = sh.tot[0];
                      sh.tiny = sh.gamma < 2.2250738585072014e-308;
                      sh.inv_gamma = 1.0 / sh.tot[0];
                      sh.inv_alpha = 1.0 / alpha;
                  }
                  return !sh.done;
              },
              [&](int i, const Own& o) {
                  double p[3], s[3], r[3], z[3], M[9];
#pragma unroll
                  for (int c = 0; c < 9; ++c) M[c] = a.minv[9 * (size_t)i + c];
#pragma unroll
                  for (int d = 0; d < 3; ++d) {
                      const size_t e = 3 * (size_t)i + d;
                      p[d] = o.u.v[d] + beta * o.p.v[d];
                      s[d] = o.w.v[d] + beta * o.s.v[d];
                      r[d] = o.r.v[d] - alpha * s[d];
                      a.p[e] = p[d];
                      a.s[e] = s[d];
                      a.x[e] = o.x.v[d] + alpha * p[d];
                      a.r[e] = r[d];
                  }
#pragma unroll
                  for (int d = 0; d < 3; ++d) z[d] = w0 * (M[3 * d] * r[0] + M[3 * d + 1] * r[1] + M[3 * d + 2] * r[2]);
                  *reinterpret_cast<double2*>(P.m.z0 + 4 * (size_t)i) = make_double2(z[0], z[1]);
                  P.m.z0[4 * (size_t)i + 2] = z[2];
                  if (P.m.z0f)
                      *reinterpret_cast<float4*>(P.m.z0f + 4 * (size_t)i) = make_float4((float)z[0], (float)z[1], (float)z[2], 0.f);
              });
    return sh.done;
}

// t0 = r - A z0 (Dirichlet vertices 0)
__device__ __forceinline__ void phase_res0(const PcgLoop& P, PpShared& sh) {
    const PCGArgs& a = P.a;
    auto own = [&](int i) { return ld_d3(a.r, i); };
    auto fin = [&](int i, const D3& r, double y0, double y1, double y2) {
        const bool fx = a.fixed[i] != 0;
        double* t = P.m.t0 + 3 * (size_t)i;
        t[0] = fx ? 0.0 : r.v[0] - y0;
        t[1] = fx ? 0.0 : r.v[1] - y1;
        t[2] = fx ? 0.0 : r.v[2] - y2;
    };
    if (P.m.z0f)
        rows_apply<true, float>(P, P.m.v32, P.m.c32, Vec<float>{P.m.z0f}, sh, own,
                               [&](int i, const D3& r, const float (&y)[3]) { fin(i, r, (double)y[0], (double)y[1], (double)y[2]); });
    else
        rows_apply<true, double>(P, a.sval, a.cva, vec4(P.m.z0), sh, own,
                                [&](int i, const D3& r, const double (&y)[3]) { fin(i, r, y[0], y[1], y[2]); });
}

// u = z0 + w0 D^-1 (r - A z0) (Dirichlet vertices 0)
__device__ __forceinline__ void phase_post0(const PcgLoop& P, PpShared& sh) {
    const PCGArgs& a = P.a;
    const double w = P.omega[0];
    auto own = [&](int i) { return ld_d3(a.r, i); };
    auto fin = [&](int i, const D3& r, double y0, double y1, double y2) {
        double* u = a.u + 4 * (size_t)i;
        if (a.fixed[i]) {
            u[0] = u[1] = u[2] = 0.0;
            return;
        }
        const double s0 = r.v[0] - y0, s1 = r.v[1] - y1, s2 = r.v[2] - y2;
        const double* M = a.minv + 9 * (size_t)i;
        const double2 z = *reinterpret_cast<const double2*>(P.m.z0 + 4 * (size_t)i);
        const double z2 = P.m.z0[4 * (size_t)i + 2];
        *reinterpret_cast<double2*>(u) = make_double2(z.x + w * (M[0] * s0 + M[1] * s1 + M[2] * s2), z.y + w * (M[3] * s0 + M[4] * s1 + M[5] * s2));
        u[2] = z2 + w * (M[6] * s0 + M[7] * s1 + M[8] * s2);
    };
    if (P.m.z0f)
        rows_apply<true, float>(P, P.m.v32, P.m.c32, Vec<float>{P.m.z0f}, sh, own,
                               [&](int i, const D3& r, const float (&y)[3]) { fin(i, r, (double)y[0], (double)y[1], (double)y[2]); });
    else
        rows_apply<true, double>(P, a.sval, a.cva, vec4(P.m.z0), sh, own,
                                [&](int i, const D3& r, const double (&y)[3]) { fin(i, r, y[0], y[1], y[2]); });
}

// restriction of the finer residual into level l (g), and below the coarsest z = w D^-1 g; a group
// of 8 lanes per node takes its members in turn
__device__ __forceinline__ void phase_restrict(const PcgLoop& P, PpShared& sh, int l) {
    const MgLev& L = P.m.L[l];
    const double* t = l == 1 ? P.m.t0 : P.m.L[l - 1].t;
    const bool coarsest = l == P.m.levels - 1;
    const int sub = threadIdx.x & 7, st = l == 1 ? 3 : 6, base = threadIdx.x & 24;
    const int per = gridDim.x * (PP_THREADS / 8), me = (int)blockIdx.x;
    double w = 0.0;
    for (int I0 = 0; I0 < L.n; I0 += per) {
        const int I = I0 + me + gridDim.x * (threadIdx.x >> 3);
        const bool any = I0 + me + (int)(gridDim.x * (threadIdx.x >> 5) * 4) < L.n;   // a node of the warp's four
        double g[8] = {0.0, 0.0, 0.0, 0.0, 0.0, 0.0, 0.0, 0.0};
        int k = 0, k1 = 0;
        if (I < L.n) {
            k = __ldg(L.mem_ptr + I) + sub;
            k1 = __ldg(L.mem_ptr + I + 1);
        }
        constexpr int NM = 4;   // members of a lane in flight: their ids are loaded before the barrier
        int id[NM];
        auto ids = [&] {
#pragma unroll
            for (int q = 0; q < NM; ++q) {
                id[q] = k + 8 * q < k1 ? __ldg(L.mem + k + 8 * q) : -1;
                if (l == 1 && id[q] >= 0 && P.a.fixed[id[q]]) id[q] = -1;
            }
        };
        ids();
        if (I0 == 0) {
            barrier();
            w = coarsest ? 0.0 : P.omega[l];
        }
        while (k < k1) {
            double f[NM][3], d[NM][3];
#pragma unroll
            for (int q = 0; q < NM; ++q) {
                const int i = id[q] < 0 ? 0 : id[q];   // a member left out reads member 0 and is not added
                const double* ti = t + (size_t)st * i;
#pragma unroll
                for (int c = 0; c < 3; ++c) {
                    f[q][c] = ti[c];
                    d[q][c] = __ldg(L.d + 3 * (size_t)i + c);
                }
                if (l > 1 && id[q] >= 0) {
                    g[3] += ti[3];
                    g[4] += ti[4];
                    g[5] += ti[5];
                }
            }
#pragma unroll
            for (int q = 0; q < NM; ++q) {
                if (id[q] < 0) continue;
                g[0] += f[q][0];
                g[1] += f[q][1];
                g[2] += f[q][2];
                g[3] = fma(d[q][1], f[q][2], fma(-d[q][2], f[q][1], g[3]));
                g[4] = fma(d[q][2], f[q][0], fma(-d[q][0], f[q][2], g[4]));
                g[5] = fma(d[q][0], f[q][1], fma(-d[q][1], f[q][0], g[5]));
            }
            k += 8 * NM;
            ids();
        }
        if (!any) continue;
        __syncwarp();
        const double gp = reduce8(g, sub);
        const bool live = I < L.n && sub < 6;
        if (live) L.g[6 * (size_t)I + sub] = gp;
        if (!coarsest) {
            const int q = sub < 6 ? sub : 0;
            const double z = node_minv(L.minv + 36 * (size_t)(I < L.n ? I : 0), gp, w, base, q);
            if (live) L.z[6 * (size_t)I + sub] = z;
        }
    }
}

// a level between: t = g - A z, or (POST) z2 = z + w D^-1 (g - A z) prolongated into level l - 1
template <bool POST>
__device__ __forceinline__ void phase_smooth(const PcgLoop& P, PpShared& sh, int l) {
    const MgLev& L = P.m.L[l];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, p = lane % 6;
    const double om = POST ? P.omega[l] : 0.0;
    const int me = (int)blockIdx.x;
    bool first = true;
    for (int I = me + gridDim.x * w; I < L.n || first; I += gridDim.x * PP_WARPS) {
        const bool in = I < L.n;
        NodeCursor<2> c;
        Member m;
        int k = 0, k1 = 0;
        if (in) {
            if (lane < 30) c.open(L, I, lane / 6, 5);
            if (POST) {
                k = __ldg(L.mem_ptr + I) + lane;
                k1 = __ldg(L.mem_ptr + I + 1);
                m.open(P, L, l, k, k1);
            }
        }
        if (first) barrier();
        first = false;
        if (!in) break;
        const double g = L.g[6 * (size_t)I + p], z0 = POST ? L.z[6 * (size_t)I + p] : 0.0;
        double y = 0.0;
        if (lane < 30) y = node_row<true>(L, c, L.z, p, 5);
        __syncwarp();
        const double r = g - node_gather(y, p);
        if (!POST) {
            if (lane < 6) L.t[6 * (size_t)I + lane] = r;
            continue;
        }
        const double z = z0 + node_minv(L.minv + 36 * (size_t)I, r, om, 0, p);
        double Y[6];
#pragma unroll
        for (int e = 0; e < 6; ++e) Y[e] = __shfl_sync(FULL, z, e);
        for (; k < k1; k += 32) {
            prolong_member(P, l, m, Y);
            m.open(P, L, l, k + 32, k1);
        }
        __syncwarp();
    }
}

// coarsest level: z = D^-1 g (dense), prolongated into the level above; one CTA per node, two warps
// per row of its six.  The inverse's entries of the first 960 columns (all of them: MG_COARSEST keeps
// the level that small) and the first members are loaded before the barrier.
__device__ __forceinline__ void phase_coarsest(const PcgLoop& P, PpShared& sh) {
    const int l = P.m.levels - 1, n = P.m.n_dense;
    const MgLev& L = P.m.L[l];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, p = w / 2, j0 = 32 * (w & 1) + lane;
    constexpr int ND = 15;
    static_assert(PP_WARPS >= 12, "two warps for each of six rows");
    bool first = true;
    for (int I = (int)blockIdx.x; I < L.n || first; I += gridDim.x) {
        double D[ND];
        Member m;
        int k = 0, k1 = 0;
        const double* Dr = P.m.dense + (size_t)(6 * I + p) * P.m.ld_dense;
        if (I < L.n) {
            if (p < 6) {
#pragma unroll
                for (int q = 0; q < ND; ++q) D[q] = j0 + 64 * q < n ? __ldg(Dr + j0 + 64 * q) : 0.0;
            }
            k = __ldg(L.mem_ptr + I) + threadIdx.x;
            k1 = __ldg(L.mem_ptr + I + 1);
            m.open(P, L, l, k, k1);
        }
        if (first) barrier();
        first = false;
        if (I >= L.n) break;
        if (p < 6) {
            double g[ND], t = 0.0, t1 = 0.0;
#pragma unroll
            for (int q = 0; q < ND; ++q) g[q] = j0 + 64 * q < n ? L.g[j0 + 64 * q] : 0.0;
#pragma unroll
            for (int q = 0; q < ND; q += 2) {
                if (64 * q < n) t = fma(D[q], g[q], t);
                if (q + 1 < ND && 64 * (q + 1) < n) t1 = fma(D[q + 1], g[q + 1], t1);
            }
            for (int j = j0 + 64 * ND; j < n; j += 64) t = fma(__ldg(Dr + j), L.g[j], t);
            t += t1;
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) t += __shfl_down_sync(FULL, t, o);
            if (lane == 0) sh.row[w] = t;
        }
        __syncthreads();
        double Y[6];
        if (k < k1) {
#pragma unroll
            for (int c = 0; c < 6; ++c) Y[c] = sh.row[2 * c] + sh.row[2 * c + 1];
        }
        for (; k < k1; k += PP_THREADS) {
            prolong_member(P, l, m, Y);
            m.open(P, L, l, k + PP_THREADS, k1);
        }
        __syncthreads();
    }
}

// ---------------------------------------------------------------- kernels
__global__ void __launch_bounds__(PP_THREADS, 1) k_pcg_run(PcgLoop P) {
    __shared__ PpShared sh;
    phase_start(P, sh);
    if (phase_tolerance(P, sh)) return;
    for (int k = 0; k < MG_POWER_ITERS; ++k) phase_power(P, sh, k);
    phase_weights(P, sh);
    const int nl = P.m.levels;
    for (int k = 0; k < P.maxit; ++k) {
        // V-cycle on r: from z0 = w0 D^-1 r to u
        phase_res0(P, sh);
        for (int l = 1; l < nl; ++l) {
            phase_restrict(P, sh, l);
            if (l < nl - 1) phase_smooth<false>(P, sh, l);
        }
        phase_coarsest(P, sh);
        for (int l = nl - 2; l >= 1; --l) phase_smooth<true>(P, sh, l);
        phase_post0(P, sh);
        phase_spmv(P, sh);
        if (phase_update(P, sh, k)) return;
    }
}

// ---------------------------------------------------------------- host side
int mg_loop_args(fipc_ctx* c, MgArgs* m, double** omega, double** pv0, double** pv1);

// the solve for a system whose multigrid levels mg_prepare has set up
int pcg_mg_run(fipc_ctx* c, const PCGArgs& a, double rtol, int maxit, int guess, int* iters, cudaStream_t s) {
    int dev = 0, nsm = 0, per = 0;
    FIPC_CUDA(cudaGetDevice(&dev));
    FIPC_CUDA(cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev));
    FIPC_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, k_pcg_run, PP_THREADS, 0));
    if (per < 1) return FIPC_ERR_CUDA;
    if (c->pcg_part.ensure(8ull * (3 + 2 * MG_LEVELS_CAP) * nsm + 64)) return FIPC_ERR_CUDA;
    PcgLoop P{};
    P.a = a;
    P.rhs = c->rhs;
    P.rtol = rtol;
    P.maxit = maxit;
    P.guess = guess;
    P.contact = c->c_nnzb > 0;
    P.n_slices = c->n_slices;
    P.part = c->pcg_part.as<double>();
    const int st = mg_loop_args(c, &P.m, &P.omega, P.pv0, P.pv1);
    if (st) return st;
    int h_flag[4] = {0, 0, 0, 0};
    void* args[] = {&P};
    FIPC_CUDA(cudaLaunchCooperativeKernel((const void*)k_pcg_run, dim3(nsm), dim3(PP_THREADS), args, 0, s));
    FIPC_LAUNCHED();
    FIPC_CUDA(cudaMemcpyAsync(h_flag, a.flag, sizeof(int) * 4, cudaMemcpyDeviceToHost, s));
    FIPC_CUDA(cudaStreamSynchronize(s));
    FIPC_CUDA(cudaGetLastError());
    if (iters) *iters = h_flag[0] ? h_flag[1] : maxit;
    return h_flag[0] ? FIPC_OK : FIPC_ERR_ITERATION;
}

}  // namespace fipc
