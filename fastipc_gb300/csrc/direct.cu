// Direct solve of the Newton system: the role of the reference's CHOLMOD factorisation
// (projects/FastIPC/NEWTON_IPC.py:764-776), for the iterations where PCG reaches its iteration
// limit, or for callers that want the reference's exact solve.
//
// A multifrontal Cholesky factorisation written for this GPU (no library factorisation):
//  * analysis on the host (mf_plan.h): nested-dissection ordering of the free vertices from the
//    elastic and contact block patterns, the assembly tree, one dense frontal matrix per tree
//    node, extend-add maps and the task tables of the numeric phase;
//  * the edited system's 3x3 blocks (Dirichlet rows and columns removed: their solution is 0,
//    as NEWTON_IPC.py:758-772 makes it) scattered into the fronts, elastic then contact;
//  * per tree height, children's update matrices pulled into their parents (each entry sums its
//    children in a fixed order), then every front of the height factored panel by panel: the
//    64 x 64 diagonal tile by one CTA, the rows below it 16 per CTA, and the trailing
//    update in 32 x 32 tiles (register blocks, operands staged in shared memory) across
//    all fronts of the height at once;
//  * forward and backward substitution through the tree by the same panels.
// Every sum runs in a fixed order, so the solve is deterministic.  FP64 throughout: the
// trailing update, which holds nearly all the flops, is bound by the FP64 pipe.
#include <cuda_runtime.h>

#include <algorithm>
#include <chrono>
#include <climits>
#include <vector>

#include "ctx.cuh"
#include "mf_plan.h"

namespace fipc {

int sell_to_bsr(fipc_ctx* c, double* out, cudaStream_t s);

namespace {

constexpr int MF_THREADS = 256;
constexpr int MF_LDS = MF_TILE + 1;   // padded shared-memory column stride of a tile

inline int nbd(long long n, int b) { return (int)((n + b - 1) / b); }

// device copy of the plan (pointers into one arena) and the numeric buffers
struct MfDev {
    double* F;                       // fronts
    double* W;                       // per-front solve vectors
    double* Y;                       // per-front pivot results of the forward sweep
    const int *nvf, *npiv, *piv0, *child0, *children, *cmap, *fidx, *order, *level_nodes, *task_front, *ext_front;
    const long long *foff, *woff, *cmap0, *fidx0, *task_chunk0, *task_tile0, *ext_col0;
    int* flag;                       // [0]: a non-positive or non-finite pivot
};

// ---------------------------------------------------------------- assembly into the fronts
// block k of a block matrix to its front position (column-major, leading dimension ld[k])
__global__ void k_mf_scatter(long long nb, const double* __restrict__ val, const long long* __restrict__ dst, const int* __restrict__ ld,
                             double* __restrict__ F, int add) {
    const long long k = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= nb) return;
    const long long d = dst[k];
    if (d < 0) return;
    const long long L = ld[k];
    for (int a = 0; a < 3; ++a)
        for (int b = 0; b < 3; ++b) {
            const double v = val[9 * k + 3 * a + b];
            double* p = F + d + a + b * L;
            *p = add ? *p + v : v;
        }
}

// extend-add, pull form: one CTA per (front, column j); each lower entry (i >= j) adds the
// matching entries of its children's update matrices, children in tree order
__global__ void __launch_bounds__(MF_THREADS) k_mf_extend(MfDev d, const int* __restrict__ fronts, const long long* __restrict__ col0,
                                                          int nf) {
    const long long q = blockIdx.x;
    const int e = mf_find(col0, nf + 1, q);
    const int f = fronts[e];
    const int j = (int)(q - col0[e]);
    const int N = 3 * d.nvf[f];
    double* F = d.F + d.foff[f];
    const int J = j / 3, jb = j % 3;
    for (int i = j + threadIdx.x; i < N; i += MF_THREADS) {
        const int I = i / 3, ib = i % 3;
        double v = 0.0;
        for (int t = d.child0[f]; t < d.child0[f + 1]; ++t) {
            const int c = d.children[t];
            const int* m = d.cmap + d.cmap0[c];
            const int ci = m[I], cj = m[J];
            if (ci < 0 || cj < 0) continue;
            const long long Nc = 3ll * d.nvf[c];
            v += d.F[d.foff[c] + (3 * ci + ib) + (3ll * cj + jb) * Nc];
        }
        F[i + (long long)j * N] += v;
    }
}

// ---------------------------------------------------------------- panel factorisation
struct PanelArgs {
    int k;                           // panel index: columns [k MF_TILE, k MF_TILE + kb)
    int n_fronts;
    long long t0;                    // offset into task_front
    const long long* chunk0;         // prefix of row chunks (n_fronts + 1)
    const long long* tile0;          // prefix of trailing tiles (n_fronts + 1)
};

__device__ __forceinline__ void panel_geometry(const MfDev& d, const PanelArgs& p, int e, int* f, int* N, int* c0, int* kb) {
    *f = d.task_front[p.t0 + e];
    *N = 3 * d.nvf[*f];
    *c0 = p.k * MF_TILE;
    *kb = min(MF_TILE, 3 * d.npiv[*f] - *c0);
}

// Cholesky of the diagonal tile, one CTA per front.  Bounded by the chain of its 64 pivots: the lower half
// stays in registers (four threads per row, thread q of them the columns q + 4 u), the unscaled column of a
// pivot goes through shared memory, and warp 0 carries all diagonals, so that the next pivot's
// reciprocal is formed while the others update: s_ij -= c_i c_j / p.  The columns are scaled to L
// at the end.  Rows are dealt to the warps so that the four schedulers (warp % 4) have the same FP64
// work.  Column by column in shared memory, with the square root, the division and the update behind one
// another, a tile took 94 us.
__global__ void __launch_bounds__(MF_THREADS) k_mf_potrf(MfDev d, PanelArgs p) {
    __shared__ double col[2][MF_TILE], pinv[2], piv[MF_TILE];
    int f, N, c0, kb;
    panel_geometry(d, p, blockIdx.x, &f, &N, &c0, &kb);
    double* F = d.F + d.foff[f] + c0 + (long long)c0 * N;
    const int t = threadIdx.x, w = t >> 5, lane = t & 31, rb = w < 4 ? w : 11 - w;
    const int i = 8 * rb + (lane >> 2), q = lane & 3;
    double e[16];
#pragma unroll
    for (int u = 0; u < 16; ++u) {
        const int j = q + 4 * u;
        e[u] = j <= i && i < kb ? F[i + (long long)j * N] : 0.0;
        if (j == 0) col[0][i] = e[u];
    }
    // the diagonals: rows lane and lane + 32
    double d0 = 0.0, d1 = 0.0;
    auto next_pivot = [&](int k, int b) {   // the calling lane holds diagonal k
        double v = k < 32 ? d0 : d1;
        if (!(v > 0.0) || !isfinite(v)) {
            atomicOr(d.flag, 1);
            v = 1.0;
        }
        piv[k] = v;
        pinv[b] = reciprocal(v);
    };
    if (w == 0) {
        if (lane < kb) d0 = F[lane + (long long)lane * N];
        if (lane + 32 < kb) d1 = F[lane + 32 + (long long)(lane + 32) * N];
        if (lane == 0) next_pivot(0, 0);
    }
    __syncthreads();
    for (int k = 0; k < kb; ++k) {
        const int b = k & 1;
        const double pin = pinv[b];
        if (w == 0 && k + 1 < kb) {
            const double x0 = col[b][lane], x1 = col[b][lane + 32];
            d0 = fma(-x0 * pin, x0, d0);
            d1 = fma(-x1 * pin, x1, d1);
            if (lane == ((k + 1) & 31)) next_pivot(k + 1, b ^ 1);
        }
        if (8 * rb + 7 > k) {
            const double r = col[b][i] * pin;
#pragma unroll
            for (int u = 0; u < 16; ++u) {
                if (4 * u + 3 <= k || 4 * u > 8 * rb + 7) continue;   // uniform over the warp
                const int j = q + 4 * u;
                if (j > k && j <= i) {
                    e[u] = fma(-r, col[b][j], e[u]);
                    if (j == k + 1) col[b ^ 1][i] = e[u];
                }
            }
        }
        __syncthreads();
    }
    // L_jj = sqrt(p_j), L_ij = c_ij / sqrt(p_j)
    if (t < kb) col[0][t] = 1.0 / sqrt(piv[t]);
    __syncthreads();
#pragma unroll
    for (int u = 0; u < 16; ++u) {
        const int j = q + 4 * u;
        if (j <= i && i < kb) F[i + (long long)j * N] = j == i ? sqrt(piv[j]) : e[u] * col[0][j];
    }
}

// the panel's diagonal tile into shared memory, scaled so that a substitution step is one FMA: column j
// divided by L_jj (forward: S[j][l] = L_lj / L_jj, l > j) or row i by L_ii (backward: S[i][j] = L_ij / L_ii,
// j < i), zero elsewhere; rinv = 1 / diagonal
template <bool FORWARD>
__device__ __forceinline__ void load_tile(const double* __restrict__ F, int N, int kb, double* __restrict__ S, double* __restrict__ rinv) {
    for (int j = threadIdx.x; j < MF_TILE; j += blockDim.x) rinv[j] = j < kb ? 1.0 / F[j + (long long)j * N] : 0.0;
    __syncthreads();
    for (int idx = threadIdx.x; idx < MF_TILE * MF_TILE; idx += blockDim.x) {
        const int l = idx % MF_TILE, j = idx / MF_TILE;   // row, column
        const double v = l > j && l < kb ? F[l + (long long)j * N] : 0.0;
        if (FORWARD) S[j * MF_LDS + l] = v * rinv[j];
        else S[l * MF_LDS + j] = v * rinv[l];
    }
    __syncthreads();
}

// rows below the diagonal tile: X L^T = B, 16 rows per CTA (a quarter of a 64-row chunk), 16 lanes per row
// with four columns each in registers.  A step is one shuffle and one to four FMAs, without a barrier;
// 64 rows per CTA and two barriers per column left most SMs idle on 100 us of one CTA's FP64 work.
constexpr int TRSM_ROWS = 16;
__global__ void __launch_bounds__(MF_THREADS) k_mf_trsm(MfDev d, PanelArgs p) {
    __shared__ double S[MF_TILE * MF_LDS], rinv[MF_TILE];
    const int chunk = blockIdx.x / (MF_TILE / TRSM_ROWS), part = blockIdx.x % (MF_TILE / TRSM_ROWS);
    const int e = mf_find(p.chunk0, p.n_fronts + 1, chunk);
    int f, N, c0, kb;
    panel_geometry(d, p, e, &f, &N, &c0, &kb);
    const int r0 = c0 + kb + (int)(chunk - p.chunk0[e]) * MF_TILE + part * TRSM_ROWS;
    if (r0 >= N) return;
    const int t = threadIdx.x & 15, r = r0 + (threadIdx.x >> 4);
    double* Fb = d.F + d.foff[f] + r + (long long)c0 * N;
    double b[4];
#pragma unroll
    for (int u = 0; u < 4; ++u) {
        const int j = t + 16 * u;
        b[u] = r < N && j < kb ? Fb[(long long)j * N] : 0.0;
    }
    load_tile<true>(d.F + d.foff[f] + c0 + (long long)c0 * N, N, kb, S, rinv);
#pragma unroll
    for (int u0 = 0; u0 < 4; ++u0)
        for (int jj = 0; jj < 16; ++jj) {
            const double bj = __shfl_sync(0xffffffffu, b[u0], jj, 16);
            const double* Sj = S + (16 * u0 + jj) * MF_LDS + t;
#pragma unroll
            for (int u = u0; u < 4; ++u) b[u] = fma(-bj, Sj[16 * u], b[u]);
        }
#pragma unroll
    for (int u = 0; u < 4; ++u) {
        const int j = t + 16 * u;
        if (r < N && j < kb) Fb[(long long)j * N] = b[u] * rinv[j];
    }
}

// trailing update of the lower tiles, C -= A_i A_j^T over the panel's kb columns, a quarter (32 x 32) of a
// 64 x 64 tile per CTA: bound by the FP64 pipe (19 us a quarter on one SM), and whole tiles left SMs idle
// in the panels with fewer tiles than SMs, and computed the upper quarter of diagonal tiles.
// Thread (tr, tc) owns rows tr + 16 a (a < 2) and columns tc + 8 b (b < 4).
constexpr int UPD_TILE = 32, UPD_THREADS = 128;
__global__ void __launch_bounds__(UPD_THREADS) k_mf_update(MfDev d, PanelArgs p) {
    __shared__ double As[MF_TILE * UPD_TILE], Bs[MF_TILE * UPD_TILE];   // [l][row]
    const int tile = blockIdx.x >> 2, qi = blockIdx.x >> 1 & 1, qj = blockIdx.x & 1;
    const int e = mf_find(p.tile0, p.n_fronts + 1, tile);
    int f, N, c0, kb;
    panel_geometry(d, p, e, &f, &N, &c0, &kb);
    int ti, tj;
    mf_tile(tile - p.tile0[e], &ti, &tj);
    if (ti == tj && qi < qj) return;
    const int s0 = c0 + kb;
    const int i0 = s0 + ti * MF_TILE + qi * UPD_TILE, j0 = s0 + tj * MF_TILE + qj * UPD_TILE;
    if (i0 >= N || j0 >= N) return;
    const int ni = min(UPD_TILE, N - i0), nj = min(UPD_TILE, N - j0);
    const double* F = d.F + d.foff[f];
    for (int idx = threadIdx.x; idx < UPD_TILE * kb; idx += UPD_THREADS) {
        const int r = idx % UPD_TILE, l = idx / UPD_TILE;
        As[idx] = r < ni ? F[(i0 + r) + (long long)(c0 + l) * N] : 0.0;
        Bs[idx] = r < nj ? F[(j0 + r) + (long long)(c0 + l) * N] : 0.0;
    }
    __syncthreads();
    const int tr = threadIdx.x & 15, tc = threadIdx.x >> 4;
    double acc[2][4] = {};
#pragma unroll 2
    for (int l = 0; l < kb; ++l) {
        double av[2], bv[4];
#pragma unroll
        for (int a = 0; a < 2; ++a) av[a] = As[l * UPD_TILE + tr + 16 * a];
#pragma unroll
        for (int b = 0; b < 4; ++b) bv[b] = Bs[l * UPD_TILE + tc + 8 * b];
#pragma unroll
        for (int a = 0; a < 2; ++a)
#pragma unroll
            for (int b = 0; b < 4; ++b) acc[a][b] = fma(av[a], bv[b], acc[a][b]);
    }
    double* C = d.F + d.foff[f];
#pragma unroll
    for (int b = 0; b < 4; ++b) {
        const int j = tc + 8 * b;
        if (j >= nj) continue;
#pragma unroll
        for (int a = 0; a < 2; ++a) {
            const int i = tr + 16 * a;
            if (i < ni) C[(i0 + i) + (long long)(j0 + j) * N] -= acc[a][b];
        }
    }
}

// ---------------------------------------------------------------- substitution
// By the panels of the factorisation: one CTA per front walking its columns one after the other, each a
// load from memory and a barrier, took 11.5 (forward) and 13.2 ms (backward) on a pile of 27 cubes (9,300
// vertices), nine heights and 61 panels.
//
// forward, per height: w = gathered right-hand side + children's updates (all rows)
__global__ void __launch_bounds__(MF_THREADS) k_mf_forward_gather(MfDev d, int h0, const double* __restrict__ rhs) {
    const int f = d.level_nodes[h0 + blockIdx.x];
    const int N = 3 * d.nvf[f];
    double* w = d.W + d.woff[f];
    for (int i = blockIdx.y * MF_THREADS + threadIdx.x; i < N; i += gridDim.y * MF_THREADS) {
        const int I = i / 3, ib = i % 3;
        double v = I < d.npiv[f] ? rhs[3ll * d.order[d.piv0[f] + I] + ib] : 0.0;
        for (int t = d.child0[f]; t < d.child0[f + 1]; ++t) {
            const int c = d.children[t];
            const int m = d.cmap[d.cmap0[c] + I];
            if (m >= 0) v += d.W[d.woff[c] + 3 * m + ib];
        }
        w[i] = v;
    }
}

// per panel: the tile's triangle (by warp 0, two rows per lane; x to shared memory), in every CTA of the
// front; the first n_fronts CTAs store it to Y, the others update 64 rows below, w -= L x, with
// their rows of L loaded before the chain
__global__ void __launch_bounds__(MF_THREADS) k_mf_forward(MfDev d, PanelArgs p) {
    __shared__ double S[MF_TILE * MF_LDS], rinv[MF_TILE], x[MF_TILE], sum[3][MF_TILE];
    const bool diag = (int)blockIdx.x < p.n_fronts;
    const int chunk = (int)blockIdx.x - p.n_fronts;
    const int e = diag ? (int)blockIdx.x : mf_find(p.chunk0, p.n_fronts + 1, chunk);
    int f, N, c0, kb;
    panel_geometry(d, p, e, &f, &N, &c0, &kb);
    const double* F = d.F + d.foff[f];
    double* w = d.W + d.woff[f];
    const int r0 = diag ? N : c0 + kb + (int)(chunk - p.chunk0[e]) * MF_TILE;
    const int r = r0 + (threadIdx.x & 63), part = threadIdx.x >> 6;   // 16 columns each
    double v[16];
#pragma unroll
    for (int c = 0; c < 16; ++c) v[c] = r < N && 16 * part + c < kb ? F[r + (long long)(c0 + 16 * part + c) * N] : 0.0;
    load_tile<true>(F + c0 + (long long)c0 * N, N, kb, S, rinv);
    if (threadIdx.x < 32) {
        const int l = threadIdx.x;
        double w0 = l < kb ? w[c0 + l] : 0.0, w1 = l + 32 < kb ? w[c0 + 32 + l] : 0.0;
#pragma unroll 4
        for (int j = 0; j < 32; ++j) {
            const double wj = __shfl_sync(0xffffffffu, w0, j);
            w0 = fma(-wj, S[j * MF_LDS + l], w0);
            w1 = fma(-wj, S[j * MF_LDS + l + 32], w1);
        }
#pragma unroll 4
        for (int j = 0; j < 32; ++j) w1 = fma(-__shfl_sync(0xffffffffu, w1, j), S[(j + 32) * MF_LDS + l + 32], w1);
        x[l] = w0 * rinv[l];
        x[l + 32] = w1 * rinv[l + 32];
    }
    __syncthreads();
    if (diag) {
        if (threadIdx.x < kb) d.Y[d.woff[f] + c0 + threadIdx.x] = x[threadIdx.x];
        return;
    }
    double a = 0.0;
#pragma unroll
    for (int c = 0; c < 16; ++c) a = fma(v[c], x[16 * part + c], a);
    if (part) sum[part - 1][threadIdx.x & 63] = a;
    __syncthreads();
    if (part == 0 && r < N) w[r] -= ((a + sum[0][threadIdx.x]) + sum[1][threadIdx.x]) + sum[2][threadIdx.x];
}

// backward, per height (parents first): y -= L^T x over the structure's rows, whose x the solution holds;
// 32 columns per CTA, four per warp
constexpr int BWD_COLS = 32, BWD_ROWS = 512;
__global__ void __launch_bounds__(MF_THREADS) k_mf_backward_gather(MfDev d, int h0, const double* __restrict__ sol) {
    __shared__ double x[BWD_ROWS];
    const int f = d.level_nodes[h0 + blockIdx.x];
    const int N = 3 * d.nvf[f], P = 3 * d.npiv[f];
    double* y = d.Y + d.woff[f];
    const double* F = d.F + d.foff[f];
    const int* fl = d.fidx + d.fidx0[f];
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    for (int j0 = blockIdx.y * BWD_COLS; j0 < P; j0 += gridDim.y * BWD_COLS) {
        const int j = j0 + 4 * wid;
        double a[4] = {0.0, 0.0, 0.0, 0.0};
        for (int i0 = P; i0 < N; i0 += BWD_ROWS) {
            const int n = min(BWD_ROWS, N - i0);
            __syncthreads();
            for (int i = threadIdx.x; i < n; i += MF_THREADS) x[i] = sol[3ll * d.order[fl[(i0 + i) / 3]] + (i0 + i) % 3];
            __syncthreads();
#pragma unroll 2
            for (int i = lane; i < n; i += 32) {
                const double xi = x[i];
#pragma unroll
                for (int c = 0; c < 4; ++c)
                    if (j + c < P) a[c] = fma(F[i0 + i + (long long)(j + c) * N], xi, a[c]);
            }
        }
#pragma unroll
        for (int c = 0; c < 4; ++c) {
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) a[c] += __shfl_down_sync(0xffffffffu, a[c], o);
            if (lane == 0 && j + c < P) y[j + c] -= a[c];
        }
    }
}

// per panel k, the last first: the tile's transposed triangle in every CTA of the front; CTA k of them
// stores it to the solution, CTA c < k updates the 64 columns of panel c, y -= L^T x
__global__ void __launch_bounds__(MF_THREADS) k_mf_backward(MfDev d, PanelArgs p, double* __restrict__ sol) {
    __shared__ double S[MF_TILE * MF_LDS], rinv[MF_TILE], x[MF_TILE];
    const int e = blockIdx.x / (p.k + 1), c = blockIdx.x % (p.k + 1);
    int f, N, c0, kb;
    panel_geometry(d, p, e, &f, &N, &c0, &kb);
    const double* F = d.F + d.foff[f];
    double* y = d.Y + d.woff[f];
    // rows t + 16 q of the panel, columns 64 c + g + 16 m
    const int t = threadIdx.x & 15, g = threadIdx.x >> 4;
    double v[4][4];
#pragma unroll
    for (int m = 0; m < 4; ++m)
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            const int row = t + 16 * q;
            v[m][q] = c < p.k && row < kb ? F[c0 + row + (long long)(MF_TILE * c + g + 16 * m) * N] : 0.0;
        }
    load_tile<false>(F + c0 + (long long)c0 * N, N, kb, S, rinv);
    if (threadIdx.x < 32) {
        const int l = threadIdx.x;
        double y0 = l < kb ? y[c0 + l] : 0.0, y1 = l + 32 < kb ? y[c0 + 32 + l] : 0.0;
#pragma unroll 4
        for (int j = 31; j >= 0; --j) {
            const double yj = __shfl_sync(0xffffffffu, y1, j);
            y0 = fma(-yj, S[(j + 32) * MF_LDS + l], y0);
            y1 = fma(-yj, S[(j + 32) * MF_LDS + l + 32], y1);
        }
#pragma unroll 4
        for (int j = 31; j >= 0; --j) y0 = fma(-__shfl_sync(0xffffffffu, y0, j), S[j * MF_LDS + l], y0);
        x[l] = y0 * rinv[l];
        x[l + 32] = y1 * rinv[l + 32];
    }
    __syncthreads();
    if (c == p.k) {
        const int j = threadIdx.x;
        if (j < kb) sol[3ll * d.order[d.piv0[f] + (c0 + j) / 3] + (c0 + j) % 3] = x[j];
        return;
    }
#pragma unroll
    for (int m = 0; m < 4; ++m) {
        double a = 0.0;
#pragma unroll
        for (int q = 0; q < 4; ++q) a = fma(v[m][q], x[t + 16 * q], a);
#pragma unroll
        for (int o = 8; o > 0; o >>= 1) a += __shfl_down_sync(0xffffffffu, a, o, 16);
        if (t == 0) y[MF_TILE * c + g + 16 * m] -= a;
    }
}

struct DevMem {
    void* p = nullptr;
    ~DevMem() {
        if (p) cudaFree(p);
    }
    bool alloc(size_t n) { return cudaMalloc(&p, n ? n : 16) == cudaSuccess; }
    template <class T>
    T* as() const { return (T*)p; }
};

// packs host vectors into one device arena (16-byte aligned pieces)
struct Arena {
    std::vector<char> host;
    std::vector<std::pair<size_t, const void**>> fix;
    template <class T>
    void add(const std::vector<T>& v, const T** out) {
        size_t off = (host.size() + 15) & ~size_t(15);
        host.resize(off + sizeof(T) * v.size());
        if (!v.empty()) memcpy(host.data() + off, v.data(), sizeof(T) * v.size());
        fix.push_back({off, (const void**)out});
    }
    bool upload(DevMem& m, cudaStream_t s) {
        if (!m.alloc(host.size())) return false;
        if (cudaMemcpyAsync(m.p, host.data(), host.size(), cudaMemcpyHostToDevice, s) != cudaSuccess) return false;
        for (auto& f : fix) *f.second = (const void*)((char*)m.p + f.first);
        return true;
    }
};

}  // namespace
}  // namespace fipc

using namespace fipc;

extern "C" {

int fipc_solve_system_direct(fipc_ctx* c, const unsigned char* fixed, double* sol, int* nnz_h, void* stream) {
    if (!c || !fixed || !sol) return FIPC_ERR_ARGUMENT;
    const int* crp_d = c->c_rowptr.as<int>();
    if (!crp_d) return FIPC_ERR_ARGUMENT;   // no system assembled
    cudaStream_t s = (cudaStream_t)stream;
    const int nV = c->nV;
    const int e_nnzb = c->nnzb, c_nnzb = c->c_nnzb;
    // patterns, Dirichlet mask and rest positions to the host for the analysis
    std::vector<int> rp(nV + 1), ci(e_nnzb), crp(nV + 1), cci(c_nnzb);
    std::vector<unsigned char> fx(nV);
    std::vector<double> x0(3ll * nV);
    FIPC_CUDA(cudaMemcpyAsync(rp.data(), c->row_ptr, 4ll * (nV + 1), cudaMemcpyDeviceToHost, s));
    if (e_nnzb) FIPC_CUDA(cudaMemcpyAsync(ci.data(), c->col_idx, 4ll * e_nnzb, cudaMemcpyDeviceToHost, s));
    FIPC_CUDA(cudaMemcpyAsync(crp.data(), crp_d, 4ll * (nV + 1), cudaMemcpyDeviceToHost, s));
    if (c_nnzb) FIPC_CUDA(cudaMemcpyAsync(cci.data(), c->c_col.p, 4ll * c_nnzb, cudaMemcpyDeviceToHost, s));
    FIPC_CUDA(cudaMemcpyAsync(fx.data(), fixed, nV, cudaMemcpyDeviceToHost, s));
    FIPC_CUDA(cudaMemcpyAsync(x0.data(), c->x0, 24ll * nV, cudaMemcpyDeviceToHost, s));
    FIPC_CUDA(cudaStreamSynchronize(s));
    MfPlan P;
    const auto t_an = std::chrono::steady_clock::now();
    if (mf_analyse(nV, rp.data(), ci.data(), c_nnzb ? crp.data() : nullptr, c_nnzb ? cci.data() : nullptr, fx.data(), x0.data(), P))
        return FIPC_ERR_ARGUMENT;
    c->mf_analyse_ms = std::chrono::duration<double, std::milli>(std::chrono::steady_clock::now() - t_an).count();
    c->mf_fronts = P.n_nodes;
    c->mf_front_doubles = P.f_total;
    c->mf_flops = P.flops;
    FIPC_CUDA(cudaMemsetAsync(sol, 0, 24ll * nV, s));
    if (nnz_h) {
        long long stored = 0;
        for (int f = 0; f < P.n_nodes; ++f) stored += 9ll * P.nvf[f] * (P.nvf[f] + 1) / 2 + 3ll * P.nvf[f];
        *nnz_h = (int)std::min<long long>(stored, INT_MAX);
    }
    if (P.n_nodes == 0) return FIPC_OK;
    // the fronts must fit
    size_t free_b = 0, total_b = 0;
    FIPC_CUDA(cudaMemGetInfo(&free_b, &total_b));
    const double need = 8.0 * ((double)P.f_total + 2.0 * (double)P.w_total) + 72.0 * e_nnzb;
    if (need > 0.85 * (double)free_b) return FIPC_ERR_CAPACITY;
    // extend-add tasks per height: fronts with children, prefix of their columns
    std::vector<int> ext_front;
    std::vector<long long> ext_col0;
    std::vector<long long> ext_at(P.height_max + 2, 0);   // per height: start in ext_front
    std::vector<long long> ext_pre_at(P.height_max + 2, 0);
    for (int h = 0; h <= P.height_max; ++h) {
        ext_at[h] = (long long)ext_front.size();
        ext_pre_at[h] = (long long)ext_col0.size();
        long long acc = 0;
        ext_col0.push_back(0);
        for (int q = P.lvl0[h]; q < P.lvl0[h + 1]; ++q) {
            const int f = P.level_nodes[q];
            if (P.child0[f + 1] == P.child0[f]) continue;
            ext_front.push_back(f);
            acc += 3ll * P.nvf[f];
            ext_col0.push_back(acc);
        }
    }
    ext_at[P.height_max + 1] = (long long)ext_front.size();
    MfDev d{};
    Arena ar;
    ar.add(P.nvf, &d.nvf);
    ar.add(P.npiv, &d.npiv);
    ar.add(P.piv0, &d.piv0);
    ar.add(P.child0, &d.child0);
    ar.add(P.children, &d.children);
    ar.add(P.cmap, &d.cmap);
    ar.add(P.fidx, &d.fidx);
    ar.add(P.order, &d.order);
    ar.add(P.level_nodes, &d.level_nodes);
    ar.add(P.task_front, &d.task_front);
    ar.add(ext_front, &d.ext_front);
    ar.add(P.foff, &d.foff);
    ar.add(P.woff, &d.woff);
    ar.add(P.cmap0, &d.cmap0);
    ar.add(P.fidx0, &d.fidx0);
    ar.add(P.task_chunk0, &d.task_chunk0);
    ar.add(P.task_tile0, &d.task_tile0);
    ar.add(ext_col0, &d.ext_col0);
    const long long *e_dst = nullptr, *c_dst = nullptr;
    const int *e_ld = nullptr, *c_ld = nullptr;
    ar.add(P.e_dst, &e_dst);
    ar.add(P.e_ld, &e_ld);
    ar.add(P.c_dst, &c_dst);
    ar.add(P.c_ld, &c_ld);
    DevMem plan, fronts, vecs, ev, flag;
    if (!ar.upload(plan, s)) return FIPC_ERR_CUDA;
    if (!fronts.alloc(8ull * P.f_total) || !vecs.alloc(16ull * P.w_total) || !ev.alloc(72ull * e_nnzb) || !flag.alloc(16))
        return FIPC_ERR_CUDA;
    d.F = fronts.as<double>();
    d.W = vecs.as<double>();
    d.Y = d.W + P.w_total;
    d.flag = flag.as<int>();
    FIPC_CUDA(cudaMemsetAsync(d.F, 0, 8ull * P.f_total, s));
    FIPC_CUDA(cudaMemsetAsync(d.flag, 0, 16, s));
    int st = sell_to_bsr(c, ev.as<double>(), s);
    if (st) return st;
    if (e_nnzb) {
        k_mf_scatter<<<nbd(e_nnzb, 256), 256, 0, s>>>(e_nnzb, ev.as<double>(), e_dst, e_ld, d.F, 0);
        FIPC_LAUNCHED();
    }
    if (c_nnzb) {
        k_mf_scatter<<<nbd(c_nnzb, 256), 256, 0, s>>>(c_nnzb, c->c_val.as<double>(), c_dst, c_ld, d.F, 1);
        FIPC_LAUNCHED();
    }
    auto panel = [&](size_t k) {
        const MfPlan::Panel& pl = P.panels[k];
        return PanelArgs{pl.k, pl.n_fronts, pl.t0, d.task_chunk0 + P.task_off[k], d.task_tile0 + P.task_off[k]};
    };
    size_t pn = 0;
    for (int h = 0; h <= P.height_max; ++h) {
        const int nf = (int)(ext_at[h + 1] - ext_at[h]);
        const long long cols = nf > 0 ? ext_col0[ext_pre_at[h] + nf] : 0;
        if (cols > 0) {
            k_mf_extend<<<(unsigned)cols, MF_THREADS, 0, s>>>(d, d.ext_front + ext_at[h], d.ext_col0 + ext_pre_at[h], nf);
            FIPC_LAUNCHED();
        }
        for (; pn < P.panels.size() && P.panels[pn].height == h; ++pn) {
            const MfPlan::Panel& pl = P.panels[pn];
            const PanelArgs pa = panel(pn);
            k_mf_potrf<<<pl.n_fronts, MF_THREADS, 0, s>>>(d, pa);
            FIPC_LAUNCHED();
            if (pl.n_chunks) {
                k_mf_trsm<<<(unsigned)(pl.n_chunks * (MF_TILE / TRSM_ROWS)), MF_THREADS, 0, s>>>(d, pa);
                FIPC_LAUNCHED();
            }
            if (pl.n_tiles) {
                k_mf_update<<<(unsigned)(4 * pl.n_tiles), UPD_THREADS, 0, s>>>(d, pa);
                FIPC_LAUNCHED();
            }
        }
    }
    // right-hand side with zeros at fixed vertices is implied: only free vertices are gathered
    std::vector<int> max_n(P.height_max + 1, 0), max_p(P.height_max + 1, 0);   // rows and pivots of a height's largest front
    for (int h = 0; h <= P.height_max; ++h)
        for (int q = P.lvl0[h]; q < P.lvl0[h + 1]; ++q) {
            max_n[h] = std::max(max_n[h], 3 * P.nvf[P.level_nodes[q]]);
            max_p[h] = std::max(max_p[h], 3 * P.npiv[P.level_nodes[q]]);
        }
    pn = 0;
    for (int h = 0; h <= P.height_max; ++h) {
        k_mf_forward_gather<<<dim3(P.lvl0[h + 1] - P.lvl0[h], std::max(1, std::min(16, nbd(max_n[h], MF_THREADS)))), MF_THREADS, 0, s>>>(
            d, P.lvl0[h], c->rhs);
        FIPC_LAUNCHED();
        for (; pn < P.panels.size() && P.panels[pn].height == h; ++pn) {
            k_mf_forward<<<(unsigned)(P.panels[pn].n_fronts + P.panels[pn].n_chunks), MF_THREADS, 0, s>>>(d, panel(pn));
            FIPC_LAUNCHED();
        }
    }
    for (int h = P.height_max; h >= 0; --h) {
        k_mf_backward_gather<<<dim3(P.lvl0[h + 1] - P.lvl0[h], std::max(1, std::min(64, nbd(max_p[h], BWD_COLS)))), MF_THREADS, 0, s>>>(
            d, P.lvl0[h], sol);
        FIPC_LAUNCHED();
        for (; pn > 0 && P.panels[pn - 1].height == h; --pn) {
            k_mf_backward<<<(unsigned)(P.panels[pn - 1].n_fronts * (P.panels[pn - 1].k + 1)), MF_THREADS, 0, s>>>(d, panel(pn - 1), sol);
            FIPC_LAUNCHED();
        }
    }
    FIPC_CUDA(cudaGetLastError());
    int bad = 0;
    FIPC_CUDA(cudaMemcpyAsync(&bad, d.flag, sizeof(int), cudaMemcpyDeviceToHost, s));
    FIPC_CUDA(cudaStreamSynchronize(s));
    return bad ? FIPC_ERR_NONFINITE : FIPC_OK;
}

int fipc_direct_stats(const fipc_ctx* c, int* fronts_h, long long* front_doubles_h, double* flops_h, double* analyse_ms_h) {
    if (!c) return FIPC_ERR_ARGUMENT;
    if (fronts_h) *fronts_h = c->mf_fronts;
    if (front_doubles_h) *front_doubles_h = c->mf_front_doubles;
    if (flops_h) *flops_h = c->mf_flops;
    if (analyse_ms_h) *analyse_ms_h = c->mf_analyse_ms;
    return FIPC_OK;
}

}  // extern "C"
