// Shared by the single-scene and batched PCG: the system operands and the per-row product
// w_i = sum_j A_ij v_j over the elastic sliced-ELL rows and the contact block-CSR rows.
#pragma once

#include "ctx.cuh"

namespace fipc {

struct PCGArgs {
    int nV;
    const int *soff, *scol, *rlen;   // elastic matrix, sliced-ELL
    const double* sval;
    const int *crp, *cci;            // contact matrix, block-CSR
    const double* cva;
    const unsigned char* fixed;
    const int* diag_spos;
    double *x, *r, *u, *w, *p, *s, *minv;   // u: stride 4 (padded); the others stride 3
    double* part;                    // [3][nblk]
    double* sc;                      // scalars, see SC_*
    int* flag;                       // [0] done, [1] iterations, [2] ticket
    // coarse space (cs_blocks = PCG blocks per aggregate; 0: block-Jacobi only)
    int cs_blocks;
    const double* cs_d;              // [V][3] vertex offset from its aggregate's centroid
    double* cs_part;                 // [nblk][6] per-block restriction (force, torque) of r
    double* cs_g;                    // [6 n_agg] restriction per aggregate
    double* cs_y;                    // [6 n_agg] coarse correction Ac^-1 g
    int* cs_ticket;                  // [n_agg] blocks of the aggregate done (reset by its last block)
    const double* cs_ainv;           // inverse coarse matrix, row stride cs_ld
    int cs_n, cs_ld;                 // 6 n_agg; padded row stride
    // multigrid preconditioner (mg non-null, host pointer): the update kernel writes the
    // pre-smoothed z0 = w0 D^-1 r (stride 4) instead of u, and the V-cycle produces u
    const struct MgArgs* mg;
    double* mg_z0;
    const double* mg_omega;          // [levels] smoother weights (device)
    float* mg_z0f;                   // FP32 copy of z0 (stride 4) for FP32 smoothing products, or null
};

// one level >= 1 of the multigrid hierarchy (6 DOFs per node), as the V-cycle kernels see it
struct MgLev {
    int n;                           // nodes
    const int *mem_ptr, *mem;        // members (finer-level ids) of each node
    const int* agg_of;               // node of each finer-level node
    const double* d;                 // [3 n_finer] offsets of the finer nodes from their node's centroid
    const int *s_rp, *s_ci;          // static pattern, 6x6 blocks
    const double* s_val;
    const int *c_rp, *c_ci;          // contact pattern (c_rp null: none)
    const double* c_val;
    const double* minv;              // [36 n] block-Jacobi inverses
    double *g, *z, *z2, *t;          // [6 n]: restricted residual, iterate, post-smoothed, residual
};
constexpr int MG_LEVELS_CAP = 8;
struct MgArgs {
    int levels;
    MgLev L[MG_LEVELS_CAP];          // L[1 .. levels - 1]
    double* z0;                      // [4 nV] level-0 iterate
    double* t0;                      // [3 nV] level-0 residual
    const double* omega;             // [levels]
    const double* dense;             // coarsest inverse, row stride ld_dense
    int n_dense, ld_dense;
    // FP32 smoothing products on level 0 (null: FP64): the elastic values in the sliced-ELL
    // layout and the contact values as FP32 copies, and z0 as FP32 (stride 4)
    const float *v32, *c32;
    float* z0f;
};
enum { SC_GAMMA = 0, SC_DELTA, SC_RR, SC_ALPHA, SC_BETA, SC_RR0, SC_TOL2, SC_COUNT };
constexpr int PCG_THREADS = 128;

// w_i = sum_j A_ij v_j over the elastic (sliced-ELL) and contact (block-CSR) rows of vertex i;
// v is stored with stride ST doubles per vertex (ST = 4: 32-byte aligned, two vector loads)
template <int ST>
__device__ __forceinline__ void load_v(const double* __restrict__ v, int j, double& a, double& b, double& c) {
    if (ST == 4) {
        const double2 ab = __ldg(reinterpret_cast<const double2*>(v + 4 * (size_t)j));
        a = ab.x;
        b = ab.y;
        c = __ldg(v + 4 * (size_t)j + 2);
    } else {
        a = __ldg(v + 3 * (size_t)j);
        b = __ldg(v + 3 * (size_t)j + 1);
        c = __ldg(v + 3 * (size_t)j + 2);
    }
}

// position of the r-th set bit of mask (r counts from 0)
__device__ __forceinline__ int nth_bit(unsigned mask, int r) {
    int pos = 0;
#pragma unroll
    for (int w = 16; w > 0; w >>= 1) {
        const int c = __popc((mask >> pos) & ((1u << w) - 1u));
        if (r >= c) {
            r -= c;
            pos += w;
        }
    }
    return pos;
}

// the contact part of y = A v for the rows of one warp (row(i) per lane, act: the lane has one), all
// lanes together: groups of 8 lanes take one row with contact each, lane q of a group its blocks q,
// q + 8, ..., and the group's sums go back to the row's lane.  (One lane per row waited for some 20
// dependent loads of its row while the lanes of rows without contact idled.)
template <class T, class LOAD>
__device__ __forceinline__ void contact_rows(const int* __restrict__ crp, const int* __restrict__ cci, const T* __restrict__ cva, int i,
                                             bool act, LOAD load, T& y0, T& y1, T& y2, int part = 0, int parts = 1) {
    const unsigned full = 0xffffffffu;
    const int lane = threadIdx.x & 31, sub = lane & 7;
    const int b = act ? __ldg(crp + i) : 0, e = act ? __ldg(crp + i + 1) : 0;
    const unsigned mask = __ballot_sync(full, e > b);
    const int n = __popc(mask), rank = __popc(mask & ((1u << lane) - 1u));
    for (int r0 = 4 * part; r0 < n; r0 += 4 * parts) {
        const int r = r0 + (lane >> 3), row = nth_bit(mask, r < n ? r : 0);
        const int eb = __shfl_sync(full, b, row), ee = __shfl_sync(full, e, row);
        T s[3] = {T(0), T(0), T(0)};
        if (r < n) {
#pragma unroll 2
            for (int k = eb + sub; k < ee; k += 8) {
                const T* B = cva + 9 * (size_t)k;
                T v0, v1, v2, m[9];
                load(__ldg(cci + k), v0, v1, v2);
#pragma unroll
                for (int q = 0; q < 9; ++q) m[q] = __ldg(B + q);
                s[0] = fma(m[0], v0, fma(m[1], v1, fma(m[2], v2, s[0])));
                s[1] = fma(m[3], v0, fma(m[4], v1, fma(m[5], v2, s[1])));
                s[2] = fma(m[6], v0, fma(m[7], v1, fma(m[8], v2, s[2])));
            }
        }
        __syncwarp();
        const bool mine = e > b && rank >= r0 && rank < r0 + 4;
        const int src = mine ? 8 * (rank - r0) : lane;
#pragma unroll
        for (int c = 0; c < 3; ++c) {
#pragma unroll
            for (int o = 4; o > 0; o >>= 1) s[c] += __shfl_xor_sync(full, s[c], o);
            s[c] = __shfl_sync(full, s[c], src);
        }
        if (mine) {
            y0 += s[0];
            y1 += s[1];
            y2 += s[2];
        }
    }
}

// Rows of a CTA of PCG_THREADS when PARTS warps share a slice of 32 rows, each taking every PARTS-th pair of
// blocks and group of contact rows; the sums of parts 1, .. reach part 0 in combine_parts.  For FP32 products of
// scenes that leave the SMs with few warps: a row's 14 blocks are then a chain of seven dependent loads
// with nothing to hide it.  (FP64 products are bound by the FP64 pipe and lose by the second part's adds.)
// Up to two dozen slices per SM: 61,700 rows (13 per SM) res0 22 -> 16 us, post0 28 -> 17; 182,000 (37 per
// SM) 23.5 -> 24.5 and 26.8 -> 27.1.
inline int row_parts(int nV) { return nV <= 24 * SMS * 32 ? 2 : 1; }
template <int PARTS>
struct RowPart {
    int i, part;
    __device__ __forceinline__ RowPart() {
        const int w = threadIdx.x >> 5;
        i = (blockIdx.x * (PCG_THREADS / 32 / PARTS) + w / PARTS) * 32 + (threadIdx.x & 31);
        part = w % PARTS;
    }
};
template <int PARTS, class T>
__device__ __forceinline__ void combine_parts(int part, T& y0, T& y1, T& y2) {
    if (PARTS == 1) return;
    __shared__ T sh[PCG_THREADS / 32][3][32];
    const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
    if (part) {
        sh[w][0][lane] = y0;
        sh[w][1][lane] = y1;
        sh[w][2][lane] = y2;
    }
    __syncthreads();
    if (part == 0)
#pragma unroll
        for (int q = 1; q < PARTS; ++q) {
            y0 += sh[w + q][0][lane];
            y1 += sh[w + q][1][lane];
            y2 += sh[w + q][2][lane];
        }
}

// act: the lane has a row; all lanes of a warp call.  WIDE: contact blocks by groups of lanes, else each
// row's by its own lane in order: the single-scene solve without the multigrid preconditioner, scenes of less than 1000
// vertices above all.  Their order of sums stays for its results, not for its time: ADMM iterations amplify another
// order's rounding (1e-12 of a direction) to 1e-8 of their variables.  us per iteration in order / by groups: 128 vertices
// 26.1 / 23.4, 686 27.5 / 24.7, 656 with 137 contact rows 31.3 / 27.8, 883 with 263 32.5 / 30.9.
template <int ST, bool WIDE = true>
__device__ __forceinline__ void row_apply(const PCGArgs& a, int i, bool act, const double* __restrict__ v, double& y0, double& y1,
                                          double& y2) {
    y0 = y1 = y2 = 0.0;
    const int sl = i >> 5, lane = i & 31;
    const int base = act ? a.soff[sl] : 0, len = act ? a.rlen[i] : 0;
    int k = 0;
    // two blocks per trip: their index, value and vector loads are independent
    for (; k + 1 < len; k += 2) {
        const size_t s0 = (size_t)(base + k), s1 = s0 + 1;
        const int j0 = __ldg(a.scol + s0 * 32 + lane), j1 = __ldg(a.scol + s1 * 32 + lane);
        const double* B = a.sval + s0 * 288 + lane;
        const double* C = a.sval + s1 * 288 + lane;
        double b[9], c[9];
#pragma unroll
        for (int q = 0; q < 9; ++q) {
            b[q] = __ldg(B + 32 * q);
            c[q] = __ldg(C + 32 * q);
        }
        double p0, p1, p2, q0, q1, q2;
        load_v<ST>(v, j0, p0, p1, p2);
        load_v<ST>(v, j1, q0, q1, q2);
        // pure FMA chains: three DFMA per block row
        y0 = fma(b[0], p0, fma(b[1], p1, fma(b[2], p2, y0)));
        y1 = fma(b[3], p0, fma(b[4], p1, fma(b[5], p2, y1)));
        y2 = fma(b[6], p0, fma(b[7], p1, fma(b[8], p2, y2)));
        y0 = fma(c[0], q0, fma(c[1], q1, fma(c[2], q2, y0)));
        y1 = fma(c[3], q0, fma(c[4], q1, fma(c[5], q2, y1)));
        y2 = fma(c[6], q0, fma(c[7], q1, fma(c[8], q2, y2)));
    }
    if (k < len) {
        const size_t s0 = (size_t)(base + k);
        const int j0 = __ldg(a.scol + s0 * 32 + lane);
        const double* B = a.sval + s0 * 288 + lane;
        double p0, p1, p2;
        load_v<ST>(v, j0, p0, p1, p2);
        y0 = fma(__ldg(B + 0), p0, fma(__ldg(B + 32), p1, fma(__ldg(B + 64), p2, y0)));
        y1 = fma(__ldg(B + 96), p0, fma(__ldg(B + 128), p1, fma(__ldg(B + 160), p2, y1)));
        y2 = fma(__ldg(B + 192), p0, fma(__ldg(B + 224), p1, fma(__ldg(B + 256), p2, y2)));
    }
    if (!WIDE) {
        if (act)
            for (int e = a.crp[i]; e < a.crp[i + 1]; ++e) {
                const int j = a.cci[e];
                const double* B = a.cva + 9 * (size_t)e;
                double v0, v1, v2;
                load_v<ST>(v, j, v0, v1, v2);
                y0 = fma(B[0], v0, fma(B[1], v1, fma(B[2], v2, y0)));
                y1 = fma(B[3], v0, fma(B[4], v1, fma(B[5], v2, y1)));
                y2 = fma(B[6], v0, fma(B[7], v1, fma(B[8], v2, y2)));
            }
        return;
    }
    __syncwarp();
    contact_rows<double>(a.crp, a.cci, a.cva, i, act, [&](int j, double& v0, double& v1, double& v2) { load_v<ST>(v, j, v0, v1, v2); },
                         y0, y1, y2);
}

// y = A v with FP32 copies of the values (v32: the sliced-ELL layout of sval; c32: the contact
// blocks) and an FP32 vector (stride 4), accumulated in FP32: the multigrid's smoothing products
template <int PARTS>
__device__ __forceinline__ void row_apply_f32(const PCGArgs& a, const float* __restrict__ v32, const float* __restrict__ c32, int i,
                                              bool act, const float4* __restrict__ v, float& y0, float& y1, float& y2, int part) {
    y0 = y1 = y2 = 0.f;
    const int sl = i >> 5, lane = i & 31;
    const int base = act ? a.soff[sl] : 0, len = act ? a.rlen[i] : 0;
    int k = 2 * part;
    for (; k + 1 < len; k += 2 * PARTS) {
        const size_t s0 = (size_t)(base + k), s1 = s0 + 1;
        const int j0 = __ldg(a.scol + s0 * 32 + lane), j1 = __ldg(a.scol + s1 * 32 + lane);
        const float* B = v32 + s0 * 288 + lane;
        const float* C = v32 + s1 * 288 + lane;
        float b[9], c[9];
#pragma unroll
        for (int q = 0; q < 9; ++q) {
            b[q] = __ldg(B + 32 * q);
            c[q] = __ldg(C + 32 * q);
        }
        const float4 p = __ldg(v + j0), q = __ldg(v + j1);
        y0 = fmaf(b[0], p.x, fmaf(b[1], p.y, fmaf(b[2], p.z, y0)));
        y1 = fmaf(b[3], p.x, fmaf(b[4], p.y, fmaf(b[5], p.z, y1)));
        y2 = fmaf(b[6], p.x, fmaf(b[7], p.y, fmaf(b[8], p.z, y2)));
        y0 = fmaf(c[0], q.x, fmaf(c[1], q.y, fmaf(c[2], q.z, y0)));
        y1 = fmaf(c[3], q.x, fmaf(c[4], q.y, fmaf(c[5], q.z, y1)));
        y2 = fmaf(c[6], q.x, fmaf(c[7], q.y, fmaf(c[8], q.z, y2)));
    }
    if (k < len) {
        const size_t s0 = (size_t)(base + k);
        const int j0 = __ldg(a.scol + s0 * 32 + lane);
        const float* B = v32 + s0 * 288 + lane;
        const float4 p = __ldg(v + j0);
        y0 = fmaf(__ldg(B + 0), p.x, fmaf(__ldg(B + 32), p.y, fmaf(__ldg(B + 64), p.z, y0)));
        y1 = fmaf(__ldg(B + 96), p.x, fmaf(__ldg(B + 128), p.y, fmaf(__ldg(B + 160), p.z, y1)));
        y2 = fmaf(__ldg(B + 192), p.x, fmaf(__ldg(B + 224), p.y, fmaf(__ldg(B + 256), p.z, y2)));
    }
    __syncwarp();
    contact_rows<float>(a.crp, a.cci, c32, i, act, [&](int j, float& v0, float& v1, float& v2) {
        const float4 p = __ldg(v + j);
        v0 = p.x;
        v1 = p.y;
        v2 = p.z;
    }, y0, y1, y2, part, PARTS);
}

// block sums of NV per-thread values into the shared array out[NV] (valid in every thread on
// return).  The values go through shared memory and warp c sums component c (four rows per lane,
// then a shuffle tree), so the block spends about 8 FP64 adds per component per lane of one warp
// instead of a full shuffle tree in every warp; the order is fixed.
template <int NV>
__device__ __forceinline__ void block_sums(const double (&v)[NV], double* out) {
    __shared__ double sv[NV][PCG_THREADS];
#pragma unroll
    for (int c = 0; c < NV; ++c) sv[c][threadIdx.x] = v[c];
    __syncthreads();
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    for (int c = wid; c < NV; c += PCG_THREADS / 32) {
        double x = sv[c][lane];
#pragma unroll
        for (int k = 1; k < PCG_THREADS / 32; ++k) x += sv[c][lane + 32 * k];
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) x += __shfl_down_sync(0xffffffffu, x, o);
        if (lane == 0) out[c] = x;
    }
    __syncthreads();
}

// restriction of one block's residuals onto the rigid-body modes of its aggregate: the block's
// sum over rows of (r_i, d_i x r_i) into cs_part[block] (fixed shuffle / shared order); the
// aggregate's last block to finish (atomic ticket) sums its blocks' partials in block order
// into cs_g, so the aggregate totals need no extra launch and are reproducible
__device__ __forceinline__ void block_restrict(const PCGArgs& a, bool valid, int i, const double (&r)[3], const double (&d)[3]) {
    __shared__ double tot[6];
    __shared__ bool last;
    double v[6] = {0, 0, 0, 0, 0, 0};
    if (valid) {
        v[0] = r[0];
        v[1] = r[1];
        v[2] = r[2];
        v[3] = d[1] * r[2] - d[2] * r[1];
        v[4] = d[2] * r[0] - d[0] * r[2];
        v[5] = d[0] * r[1] - d[1] * r[0];
    }
    block_sums<6>(v, tot);
    const int I = blockIdx.x / a.cs_blocks;
    if (threadIdx.x < 6) {
        a.cs_part[6 * (size_t)blockIdx.x + threadIdx.x] = tot[threadIdx.x];
        __threadfence();
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        const int nblocks = min((int)gridDim.x - I * a.cs_blocks, a.cs_blocks);
        last = atomicAdd(&a.cs_ticket[I], 1) == nblocks - 1;
    }
    __syncthreads();
    if (last && threadIdx.x < 6) {
        __threadfence();
        const int b0 = I * a.cs_blocks, b1 = min((int)gridDim.x, b0 + a.cs_blocks);
        double t = 0.0;
        for (int b = b0; b < b1; ++b) t += *(volatile double*)&a.cs_part[6 * (size_t)b + threadIdx.x];
        a.cs_g[6 * I + threadIdx.x] = t;
        if (threadIdx.x == 0) a.cs_ticket[I] = 0;
    }
}

// block-Jacobi preconditioner: the inverse of vertex i's 3x3 diagonal block (elastic + contact);
// identity at Dirichlet vertices
__device__ __forceinline__ void jacobi_block_inverse(const PCGArgs& a, int i, bool fx, double (&Mi)[9]) {
    if (fx) {
        for (int k = 0; k < 9; ++k) Mi[k] = (k % 4 == 0) ? 1.0 : 0.0;
    } else {
        double D[9];
        const double* E = a.sval + (size_t)(a.diag_spos[i] >> 5) * 288 + (a.diag_spos[i] & 31);
        for (int k = 0; k < 9; ++k) D[k] = E[32 * k];
        // the row's contact columns ascend
        int lo = a.crp[i], hi = a.crp[i + 1];
        const int end = hi;
        while (lo < hi) {
            const int m = (lo + hi) >> 1;
            if (a.cci[m] < i) lo = m + 1;
            else hi = m;
        }
        if (lo < end && a.cci[lo] == i)
            for (int q = 0; q < 9; ++q) D[q] += a.cva[9 * (size_t)lo + q];
        const double c00 = D[4] * D[8] - D[5] * D[7], c01 = D[5] * D[6] - D[3] * D[8], c02 = D[3] * D[7] - D[4] * D[6];
        const double id = 1.0 / (D[0] * c00 + D[1] * c01 + D[2] * c02);
        Mi[0] = c00 * id;
        Mi[1] = (D[2] * D[7] - D[1] * D[8]) * id;
        Mi[2] = (D[1] * D[5] - D[2] * D[4]) * id;
        Mi[3] = c01 * id;
        Mi[4] = (D[0] * D[8] - D[2] * D[6]) * id;
        Mi[5] = (D[2] * D[3] - D[0] * D[5]) * id;
        Mi[6] = c02 * id;
        Mi[7] = (D[1] * D[6] - D[0] * D[7]) * id;
        Mi[8] = (D[0] * D[4] - D[1] * D[3]) * id;
    }
}

}  // namespace fipc
