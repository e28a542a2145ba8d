// Device helpers of the multigrid levels with six DOFs per node, shared by the V-cycle's kernels
// (mg.cu) and the one-launch solve (pcg_mg.cu).  Iterates are read with plain loads, never through
// the read-only path: the one-launch solve changes them while it runs.
#pragma once

#include "pcg.cuh"

namespace fipc {

// A node's row product on a level of 6-DOF nodes (both patterns).  Two mappings onto a warp:
//   * one node per warp: lane = 6 kk + p (kk < 5; lanes 30, 31 idle) takes output p of the row's
//     blocks kk, kk + 5, ...; the five partial sums of an output are added in a fixed order;
//   * five nodes per warp (lane = 6 n + p takes output p of node n's whole row): a third fewer FP64
//     instructions per node (mg.cu has the rule).
// NB: blocks in flight.  Warps that hold five whole rows are few (8 per SM for 6,419 nodes), so each
// keeps four blocks in flight: a PCG iteration of the 960k-tet bar takes 218 us so, 226 us with two
// and 227 us with one node per warp.
template <int NB>
struct NodeCursor {
    int k, k1, kc, kc1, col[NB];   // static and contact ranges, the next blocks' columns
    __device__ __forceinline__ void open(const MgLev& L, int I, int kk, int step) {
        k = __ldg(L.s_rp + I) + kk;
        k1 = __ldg(L.s_rp + I + 1);
        kc = kc1 = 0;
        if (L.c_rp) {
            kc = __ldg(L.c_rp + I) + kk;
            kc1 = __ldg(L.c_rp + I + 1);
        }
        cols(L.s_ci, k, k1, step);
    }
    __device__ __forceinline__ void cols(const int* ci, int q, int q1, int step) {
#pragma unroll
        for (int c = 0; c < NB; ++c) col[c] = q + c * step < q1 ? __ldg(ci + q + c * step) : 0;
    }
};
__device__ __forceinline__ double node_dot(const double2 (&b)[3], const double2 (&v)[3], double y) {
    return fma(b[2].y, v[2].y, fma(b[2].x, v[2].x, fma(b[1].y, v[1].y, fma(b[1].x, v[1].x, fma(b[0].y, v[0].y, fma(b[0].x, v[0].x, y))))));
}
__device__ __forceinline__ void node_load(const double* val, const double* v, int p, size_t k, int col, double2 (&b)[3], double2 (&x)[3]) {
    const double2* B = reinterpret_cast<const double2*>(val + 36 * k + 6 * p);
    const double2* X = reinterpret_cast<const double2*>(v + 6 * (size_t)col);
#pragma unroll
    for (int q = 0; q < 3; ++q) {
        b[q] = __ldg(B + q);
        x[q] = X[q];
    }
}
// output p of the blocks [k, k1) of one pattern, `step` apart; the first blocks' columns are in cur.
// EVEN: full groups of NB first, the rest one by one (the one-launch solve: 7 us less per iteration);
// else every group with its blocks guarded (the chain's kernels: 15 us less on 5,039 nodes in contact)
template <int NB, bool EVEN>
__device__ __forceinline__ double node_blocks(NodeCursor<NB>& cur, const int* __restrict__ ci, const double* __restrict__ val, int k, int k1,
                                              const double* v, int p, int step) {
    double y[NB];
#pragma unroll
    for (int c = 0; c < NB; ++c) y[c] = 0.0;
    for (; EVEN ? k + (NB - 1) * step < k1 : k < k1; k += NB * step) {
        double2 b[NB][3], x[NB][3];
        bool in[NB];
#pragma unroll
        for (int c = 0; c < NB; ++c) {
            in[c] = EVEN || k + c * step < k1;
            if (in[c]) node_load(val, v, p, k + c * step, cur.col[c], b[c], x[c]);
        }
        cur.cols(ci, k + NB * step, k1, step);
#pragma unroll
        for (int c = 0; c < NB; ++c)
            if (in[c]) y[c] = node_dot(b[c], x[c], y[c]);
    }
    if (EVEN) {
#pragma unroll
        for (int c = 0; c < NB - 1; ++c)
            if (k + c * step < k1) {
                double2 b[3], x[3];
                node_load(val, v, p, k + c * step, cur.col[c], b, x);
                y[c] = node_dot(b, x, y[c]);
            }
    }
    double s = y[0];
#pragma unroll
    for (int c = 1; c < NB; ++c) s += y[c];
    return s;
}
template <bool EVEN, int NB>
__device__ __forceinline__ double node_row(const MgLev& L, NodeCursor<NB> c, const double* v, int p, int step) {
    double y = node_blocks<NB, EVEN>(c, L.s_ci, L.s_val, c.k, c.k1, v, p, step);
    if (c.kc < c.kc1) {
        c.cols(L.c_ci, c.kc, c.kc1, step);
        y += node_blocks<NB, EVEN>(c, L.c_ci, L.c_val, c.kc, c.kc1, v, p, step);
    }
    return y;
}
// sum of an output's five partial sums (one node per warp); every lane returns y for its p = lane % 6
__device__ __forceinline__ double node_gather(double y, int p) {
    const double y0 = __shfl_sync(0xffffffffu, y, p), y1 = __shfl_sync(0xffffffffu, y, p + 6), y2 = __shfl_sync(0xffffffffu, y, p + 12),
                 y3 = __shfl_sync(0xffffffffu, y, p + 18), y4 = __shfl_sync(0xffffffffu, y, p + 24);
    return ((y0 + y1) + (y2 + y3)) + y4;
}

// z_p = w sum_q M_pq s_q for the lane's p; s_q is held by lane base + q
__device__ __forceinline__ double node_minv(const double* __restrict__ M, double s, double w, int base, int p) {
    const double2* m = reinterpret_cast<const double2*>(M + 6 * p);
    double z0 = 0.0, z1 = 0.0;
#pragma unroll
    for (int q = 0; q < 3; ++q) {
        const double2 b = __ldg(m + q);
        z0 = fma(b.x, __shfl_sync(0xffffffffu, s, base + 2 * q), z0);
        z1 = fma(b.y, __shfl_sync(0xffffffffu, s, base + 2 * q + 1), z1);
    }
    return w * (z0 + z1);
}

// component `sub` of the sums over a group of 8 lanes of v[0..7]: seven adds instead of a tree for
// every component (each exchange halves the components a lane still carries)
__device__ __forceinline__ double reduce8(const double (&v)[8], int sub) {
    double a[4], b[2];
#pragma unroll
    for (int c = 0; c < 4; ++c) {
        const double keep = (sub & 4) ? v[c + 4] : v[c], send = (sub & 4) ? v[c] : v[c + 4];
        a[c] = keep + __shfl_xor_sync(0xffffffffu, send, 4);
    }
#pragma unroll
    for (int c = 0; c < 2; ++c) {
        const double keep = (sub & 2) ? a[c + 2] : a[c], send = (sub & 2) ? a[c] : a[c + 2];
        b[c] = keep + __shfl_xor_sync(0xffffffffu, send, 2);
    }
    const double keep = (sub & 1) ? b[1] : b[0], send = (sub & 1) ? b[0] : b[1];
    return keep + __shfl_xor_sync(0xffffffffu, send, 1);
}

}  // namespace fipc
