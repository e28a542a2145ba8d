// IPC barrier energy, gradient and PSD-projected Hessian per constraint row (host + device).
//
// Restates common/math/ipc.py:30-329 (PP/PE/PT/EE/EEM/PPM/PEM _energy, _g_and_H) with the
// distances of common/math/distance.py (PP_3D_E 955, PE_3D_E 684, PT_3D_E 976, EE_3D_E 192,
// EECN2_E 1345), the barrier of distance.py:22-44 and the mollifier of distance.py:1625-1673.
//
// Derivatives are hand-derived in translation-free reduced coordinates y = C x:
//   PT  (p,t0,t1,t2):    r = p-t0,  e1 = t1-t0, e2 = t2-t0,   d = (r.(e1 x e2))^2 / |e1 x e2|^2
//   EE* (a0,a1,b0,b1):   r = b0-a0, e1 = a1-a0, e2 = b1-b0,   d as above (EEM), |r|^2 (PPM),
//                        |r x e2|^2/|e2|^2 (PEM); the mollifier variable is |e1 x e2|^2
//   PE  (p,e0,e1):       q = e0-p,  e = e1-e0,                d = |q x e|^2 / |e|^2
//   PP  (a,b):           r = a-b,                             d = |r|^2
// Every energy is translation invariant, so the x-space Hessian H = C^T H_y C has the three
// rigid translations in its null space and H = Q M Q^T with Q the orthonormal (Helmert) basis
// of zero-sum vertex combinations and M = (CQ)^T H_y (CQ).  The PSD projection of the
// reference's n x n matrix (n = 12, 9, 6) therefore equals Q proj(M) Q^T with M of size
// 9, 6, 3: the projection of the mollified rows runs on the reduced matrix, that of the others on the
// one to five dimensions that its closed form below spans.
#pragma once

#include "common.cuh"
#include "eig.cuh"

namespace fipc {

// ---------------------------------------------------------------- barrier scalar function
FIPC_HD double barrier_E(double d, double dh2, double k) {
    return d < dh2 ? -k * (d - dh2) * (d - dh2) * log(d / dh2) : 0.0;
}
FIPC_HD double barrier_g(double d, double dh2, double k) {
    const double t2 = d - dh2;
    return d < dh2 ? k * (t2 * log(d / dh2) * -2.0 - (t2 * t2) / d) : 0.0;
}
FIPC_HD double barrier_H(double d, double dh2, double k) {
    const double t2 = d - dh2;
    return d < dh2 ? k * ((log(d / dh2) * -2.0 - t2 * 4.0 / d) + 1.0 / (d * d) * (t2 * t2)) : 0.0;
}

// ---------------------------------------------------------------- reduced-space helpers
// 9-dim y = (y0, y1, y2) blocks of 3; gradients g[9]; Hessians H[9*9] row-major.
FIPC_HD void put3(double* g, int blk, v3 a, double s) {
    g[3 * blk + 0] += s * a.x;
    g[3 * blk + 1] += s * a.y;
    g[3 * blk + 2] += s * a.z;
}
// H[blk_i][blk_j] += s * (a b^T)
FIPC_HD void put_outer(double* H, int bi, int bj, v3 a, v3 b, double s) {
    const double A[3] = {a.x, a.y, a.z}, B[3] = {b.x, b.y, b.z};
    for (int i = 0; i < 3; ++i)
        for (int j = 0; j < 3; ++j) H[(3 * bi + i) * 9 + 3 * bj + j] += s * A[i] * B[j];
}
FIPC_HD void put_ident(double* H, int bi, int bj, double s) {
    for (int i = 0; i < 3; ++i) H[(3 * bi + i) * 9 + 3 * bj + i] += s;
}
// H[bi][bj] += s [a]_x  (skew matrix with [a]_x b = a x b), and the transposed block
FIPC_HD void put_skew_pair(double* H, int bi, int bj, v3 a, double s) {
    const double S[9] = {0, -a.z, a.y, a.z, 0, -a.x, -a.y, a.x, 0};
    for (int i = 0; i < 3; ++i)
        for (int j = 0; j < 3; ++j) {
            H[(3 * bi + i) * 9 + 3 * bj + j] += s * S[i * 3 + j];
            H[(3 * bj + j) * 9 + 3 * bi + i] += s * S[i * 3 + j];
        }
}
FIPC_HD void sym_outer(double* H, const double* a, const double* b, double s, int n) {
    for (int i = 0; i < n; ++i)
        for (int j = 0; j < n; ++j) H[i * 9 + j] += s * (a[i] * b[j] + b[i] * a[j]);
}

// Value, gradient and Hessian of N = |u x w|^2 in blocks (bu, bw) of a 9-dim space.
FIPC_HD double cross_norm2(v3 u, v3 w, int bu, int bw, double* g, double* H) {
    const v3 c = cross(u, w);
    put3(g, bu, cross(w, c), 2.0);   // dN/du = 2 w x c
    put3(g, bw, cross(c, u), 2.0);   // dN/dw = 2 c x u
    const double uu = sq(u), ww = sq(w), uw = dot(u, w);
    put_ident(H, bu, bu, 2.0 * ww);
    put_outer(H, bu, bu, w, w, -2.0);
    put_ident(H, bw, bw, 2.0 * uu);
    put_outer(H, bw, bw, u, u, -2.0);
    // [u][w] block: 2 (u w^T - (u.w) I - [c]_x); [w][u] its transpose
    put_outer(H, bu, bw, u, w, 2.0);
    put_outer(H, bw, bu, w, u, 2.0);
    put_ident(H, bu, bw, -2.0 * uw);
    put_ident(H, bw, bu, -2.0 * uw);
    put_skew_pair(H, bu, bw, c, -2.0);
    return sq(c);
}

// squared point-plane style distance d = s^2 / D, s = r.(e1 x e2), D = |e1 x e2|^2 in blocks
// (0,1,2) = (r,e1,e2).  Also returns D with its gradient/Hessian (the mollifier variable).
FIPC_HD double triple_dist(v3 r, v3 e1, v3 e2, double* g, double* H, double* Dv, double* Dg, double* DH) {
    for (int i = 0; i < 9; ++i) Dg[i] = 0.0;
    for (int i = 0; i < 81; ++i) DH[i] = 0.0;
    const double D = cross_norm2(e1, e2, 1, 2, Dg, DH);
    const v3 n = cross(e1, e2);
    const double s = dot(r, n);
    double sg[9] = {0};
    put3(sg, 0, n, 1.0);
    put3(sg, 1, cross(e2, r), 1.0);
    put3(sg, 2, cross(r, e1), 1.0);
    const double iD = 1.0 / D, d = s * s * iD;
    for (int i = 0; i < 9; ++i) g[i] = 2.0 * s * iD * sg[i] - d * iD * Dg[i];
    for (int i = 0; i < 81; ++i) H[i] = -d * iD * DH[i];
    // s Hessian: [r][e1] = -[e2]_x, [r][e2] = [e1]_x, [e1][e2] = -[r]_x (plus transposes)
    const double k = 2.0 * s * iD;
    put_skew_pair(H, 0, 1, e2, -k);
    put_skew_pair(H, 0, 2, e1, k);
    put_skew_pair(H, 1, 2, r, -k);
    for (int i = 0; i < 9; ++i)
        for (int j = 0; j < 9; ++j)
            H[i * 9 + j] += 2.0 * iD * sg[i] * sg[j] + 2.0 * d * iD * iD * Dg[i] * Dg[j]
                            - 2.0 * s * iD * iD * (sg[i] * Dg[j] + Dg[i] * sg[j]);
    *Dv = D;
    return d;
}

// squared point-line distance d = |q x e|^2 / |e|^2 in blocks (bq, be)
FIPC_HD double line_dist(v3 q, v3 e, int bq, int be, double* g, double* H) {
    double Ng[9] = {0}, NH[81] = {0};
    const double N = cross_norm2(q, e, bq, be, Ng, NH);
    const double L = sq(e), iL = 1.0 / L, d = N * iL;
    double Lg[9] = {0};
    put3(Lg, be, e, 2.0);
    for (int i = 0; i < 9; ++i) g[i] = Ng[i] * iL - d * iL * Lg[i];
    for (int i = 0; i < 81; ++i) H[i] = NH[i] * iL;
    put_ident(H, be, be, -2.0 * d * iL);
    for (int i = 0; i < 9; ++i)
        for (int j = 0; j < 9; ++j)
            H[i * 9 + j] += -iL * iL * (Ng[i] * Lg[j] + Lg[i] * Ng[j]) + 2.0 * N * iL * iL * iL * Lg[i] * Lg[j];
    return d;
}

// ---------------------------------------------------------------- per-row evaluation
// Reduced-coordinate maps C[k][v] (rows: y blocks, columns: vertices of the row)
struct RowMap {
    int nv, ny;          // vertices, reduced blocks
    double C[3][4];
};
FIPC_HD RowMap row_map(int type) {
    RowMap m{};
    if (type == T_PP) {
        m.nv = 2; m.ny = 1;
        m.C[0][0] = 1; m.C[0][1] = -1;
    } else if (type == T_PE) {
        m.nv = 3; m.ny = 2;
        m.C[0][0] = -1; m.C[0][1] = 1;                 // q = e0 - p
        m.C[1][1] = -1; m.C[1][2] = 1;                 // e = e1 - e0
    } else if (type == T_PT) {
        m.nv = 4; m.ny = 3;
        m.C[0][0] = 1; m.C[0][1] = -1;                 // r = p - t0
        m.C[1][1] = -1; m.C[1][2] = 1;                 // e1 = t1 - t0
        m.C[2][1] = -1; m.C[2][3] = 1;                 // e2 = t2 - t0
    } else {
        m.nv = 4; m.ny = 3;
        m.C[0][0] = -1; m.C[0][2] = 1;                 // r = b0 - a0
        m.C[1][0] = -1; m.C[1][1] = 1;                 // e1 = a1 - a0
        m.C[2][2] = -1; m.C[2][3] = 1;                 // e2 = b1 - b0
    }
    return m;
}

// Orthonormal basis of zero-sum combinations of nv vertices (Helmert), Qb[v][a], a < nv-1: column a is
// (1, .., 1, -(a+1), 0, ..) / sqrt((a+1)(a+2)) with a+1 ones, whatever nv
struct Helmert {
    double q[4][3];
};
FIPC_HD Helmert helmert_basis() {
    constexpr double r2 = 0.70710678118654752440, r6 = 0.40824829046386301637, r12 = 0.28867513459481288225;
    return Helmert{{{r2, r6, r12}, {-r2, r6, r12}, {0.0, -2.0 * r6, r12}, {0.0, 0.0, -3.0 * r12}}};
}

// ---------------------------------------------------------------- unmollified rows in closed form
// The reduced Hessian of an unmollified row lives in a space of one to five dimensions that its
// geometry gives, so that the projection needs a 1x1, 3x3 or 5x5 eigenproblem instead of a 9x9 one
// (whose FP64 work on the device is 7 to 10 times this).
// With W_v the weights of the vertices in the vector whose length is the distance, W = |W| w,
// rho = sqrt(d) and K = 4 b'' d + 2 b':
//   PT, EE  signed distance s = r.n along the unit normal n of (e1, e2), r_t = alpha e1 + beta e2 the
//           tangential part of r, W = C_r - alpha C_e1 - beta C_e2.  A displacement changes s by
//           sigma = W.x_n to first order and by -omega.tau - s |omega|^2 / 2 to second, where
//           tau = W.x_t is tangential (2 components) and omega = E^-T q (q the normal components of
//           the changes of e1, e2; E = (e1 e2) in the tangent basis) is the normal's rotation.  So
//               M = K sigma^2 - 4 b' s omega.tau - 2 b' d |omega|^2
//           on tau along w (2 dimensions) and the zero-sum normal displacements (3).
//   PE      rho m = the part of q = e0 - p across the unit edge direction t, gamma = q.t / |e|,
//           W = C_q - gamma C_e, A = C_e:
//               M = K (W.x_m)^2 + 2 b' (W.x_b)^2 - 4 b' (rho/|e|) (A.x_m) (W.x_t) - 2 b' (rho/|e|)^2 (A.x_m)^2
//           with b = t x m.  b' < 0, so the x_b term projects to zero; the rest is on x_t along w (1
//           dimension) and the zero-sum x_m (2).
//   PP      M = K along the unit vector between the points, 2 b' < 0 (projected to zero) across it.
// The gradient is 2 b' rho W_v times the unit vector of the distance.

// A (N x N symmetric) <- the part of its spectral decomposition with positive eigenvalues (which is
// its PSD projection), by cyclic Jacobi rotations
template <int N>
FIPC_HD void positive_part(double (&A)[N][N]) {
    double V[N][N];
#pragma unroll
    for (int i = 0; i < N; ++i)
#pragma unroll
        for (int j = 0; j < N; ++j) V[i][j] = i == j ? 1.0 : 0.0;
#pragma unroll 1
    for (int sweep = 0; sweep < 16; ++sweep) {
        double off = 0.0, dia = 0.0;
#pragma unroll
        for (int i = 0; i < N; ++i) {
            dia += A[i][i] * A[i][i];
#pragma unroll
            for (int j = 0; j < i; ++j) off += A[j][i] * A[j][i];
        }
        if (!(off > 1e-32 * dia)) break;
#pragma unroll
        for (int p = 0; p < N - 1; ++p)
#pragma unroll
            for (int q = p + 1; q < N; ++q) {
                const double apq = A[p][q];
                if (apq == 0.0) continue;
                // t = sign(h) 2 apq / (|h| + sqrt(h^2 + 4 apq^2)): the smaller rotation
                const double h = A[q][q] - A[p][p], g = 2.0 * apq;
                const double t = (h >= 0.0 ? g : -g) / (fabs(h) + sqrt(h * h + g * g));
                const double c = 1.0 / sqrt(t * t + 1.0), s = t * c;
                A[p][p] -= t * apq;
                A[q][q] += t * apq;
                A[p][q] = 0.0;
#pragma unroll
                for (int k = 0; k < N; ++k) {
                    if (k != p && k != q) {
                        double& kp = k < p ? A[k][p] : A[p][k];
                        double& kq = k < q ? A[k][q] : A[q][k];
                        const double x = kp, y = kq;
                        kp = c * x - s * y;
                        kq = s * x + c * y;
                    }
                    const double x = V[k][p], y = V[k][q];
                    V[k][p] = c * x - s * y;
                    V[k][q] = s * x + c * y;
                }
            }
    }
    double lam[N];
#pragma unroll
    for (int k = 0; k < N; ++k) lam[k] = A[k][k] > 0.0 ? A[k][k] : 0.0;
#pragma unroll
    for (int i = 0; i < N; ++i)
#pragma unroll
        for (int j = i; j < N; ++j) {
            double s = 0.0;
#pragma unroll
            for (int k = 0; k < N; ++k) s += lam[k] * V[i][k] * V[j][k];
            A[i][j] = A[j][i] = s;
        }
}

// A (N x N symmetric, entries of order one, exactly NEG of its eigenvalues below zero) <- its PSD
// projection A - U C U^T, U an orthonormal basis of the negative invariant subspace, C = U^T A U.
// FP64 work is kept to the subspace: an FP32 Jacobi eigendecomposition gives U to a few digits and the
// preconditioner of the correction; the residual A U - U C, the update and the orthonormalisation are
// FP64, so that every pass multiplies the error by that of the FP32 vectors (1e-7 over the relative gap
// between the two groups of eigenvalues).  Only the gap across zero matters; clusters on one side
// do not.  Passes stop when the next one would move U by less than FP64 rounding.  Matrices graded
// beyond what FP32 separates do not converge in PASSES and take the FP64 Jacobi rotations.
template <int N, int NEG>
FIPC_HD void remove_negative(double (&A)[N][N]) {
    constexpr int PASSES = 8;
    float a[N][N], V[N][N];
#pragma unroll
    for (int i = 0; i < N; ++i)
#pragma unroll
        for (int j = 0; j < N; ++j) {
            a[i][j] = j >= i ? (float)A[i][j] : 0.f;
            V[i][j] = i == j ? 1.f : 0.f;
        }
#pragma unroll 1
    for (int sweep = 0; sweep < 8; ++sweep) {
        float off = 0.f, dia = 0.f;
#pragma unroll
        for (int i = 0; i < N; ++i) {
            dia += a[i][i] * a[i][i];
#pragma unroll
            for (int j = 0; j < i; ++j) off += a[j][i] * a[j][i];
        }
        if (!(off > 1e-15f * dia)) break;
#pragma unroll
        for (int p = 0; p < N - 1; ++p)
#pragma unroll
            for (int q = p + 1; q < N; ++q) {
                const float apq = a[p][q], h = a[q][q] - a[p][p], g = 2.f * apq;
                const float den = fabsf(h) + sqrtf(h * h + g * g);
                const float t = den > 0.f ? (h >= 0.f ? g : -g) / den : 0.f;
                const float c = 1.f / sqrtf(t * t + 1.f), s = t * c;
                a[p][p] -= t * apq;
                a[q][q] += t * apq;
                a[p][q] = 0.f;
#pragma unroll
                for (int k = 0; k < N; ++k) {
                    if (k != p && k != q) {
                        float& kp = k < p ? a[k][p] : a[p][k];
                        float& kq = k < q ? a[k][q] : a[q][k];
                        const float x = kp, y = kq;
                        kp = c * x - s * y;
                        kq = s * x + c * y;
                    }
                    const float x = V[k][p], y = V[k][q];
                    V[k][p] = c * x - s * y;
                    V[k][q] = s * x + c * y;
                }
            }
    }
    float lam[N];
#pragma unroll
    for (int k = 0; k < N; ++k) lam[k] = a[k][k];
    // the NEG smallest to the front
#pragma unroll
    for (int i = 0; i < NEG; ++i)
#pragma unroll
        for (int j = N - 1; j > i; --j) {
            const bool sw = lam[j] < lam[j - 1];
            const float l0 = lam[j - 1], l1 = lam[j];
            lam[j - 1] = sw ? l1 : l0;
            lam[j] = sw ? l0 : l1;
#pragma unroll
            for (int k = 0; k < N; ++k) {
                const float v0 = V[k][j - 1], v1 = V[k][j];
                V[k][j - 1] = sw ? v1 : v0;
                V[k][j] = sw ? v0 : v1;
            }
        }
    double U[NEG][N], C[NEG][NEG];
#pragma unroll
    for (int j = 0; j < NEG; ++j)
#pragma unroll
        for (int k = 0; k < N; ++k) U[j][k] = V[k][j];
    bool done = false;
    float before = 1.f;
#pragma unroll 1
    for (int pass = 0;; ++pass) {
        // orthonormalise; the norms are within the last update's square of one
#pragma unroll
        for (int j = 0; j < NEG; ++j) {
#pragma unroll
            for (int i = 0; i < j; ++i) {
                double o = 0.0;
#pragma unroll
                for (int k = 0; k < N; ++k) o += U[i][k] * U[j][k];
#pragma unroll
                for (int k = 0; k < N; ++k) U[j][k] -= o * U[i][k];
            }
            double n2 = 0.0;
#pragma unroll
            for (int k = 0; k < N; ++k) n2 += U[j][k] * U[j][k];
            n2 = 1.5 - 0.5 * n2;
#pragma unroll
            for (int k = 0; k < N; ++k) U[j][k] *= n2;
        }
        double MU[NEG][N];
#pragma unroll
        for (int j = 0; j < NEG; ++j)
#pragma unroll
            for (int i = 0; i < N; ++i) {
                double o = 0.0;
#pragma unroll
                for (int k = 0; k < N; ++k) o += A[i][k] * U[j][k];
                MU[j][i] = o;
            }
#pragma unroll
        for (int i = 0; i < NEG; ++i)
#pragma unroll
            for (int j = i; j < NEG; ++j) {
                double o = 0.0;
#pragma unroll
                for (int k = 0; k < N; ++k) o += U[i][k] * MU[j][k];
                C[i][j] = C[j][i] = o;
            }
        if (done || pass == PASSES) break;
        float move = 0.f;
#pragma unroll
        for (int j = 0; j < NEG; ++j) {
            float R[N], dU[N];
#pragma unroll
            for (int k = 0; k < N; ++k) {
                double o = MU[j][k];
#pragma unroll
                for (int i = 0; i < NEG; ++i) o -= C[i][j] * U[i][k];
                R[k] = (float)o;
                dU[k] = 0.f;
            }
#pragma unroll
            for (int q = NEG; q < N; ++q) {
                float o = 0.f;
#pragma unroll
                for (int k = 0; k < N; ++k) o += V[k][q] * R[k];
                o /= lam[q] - (float)C[j][j];
#pragma unroll
                for (int k = 0; k < N; ++k) dU[k] += o * V[k][q];
            }
#pragma unroll
            for (int k = 0; k < N; ++k) {
                move += fabsf(dU[k]);
                U[j][k] -= dU[k];
            }
        }
        // the next correction would be about move^2 / before
        done = move * move <= 1e-16f * before;   // false for NaN
        before = move;
    }
    if (!done) {
        positive_part<N>(A);
        return;
    }
#pragma unroll
    for (int i = 0; i < N; ++i) {
        double T[NEG];
#pragma unroll
        for (int p = 0; p < NEG; ++p) {
            T[p] = 0.0;
#pragma unroll
            for (int q = 0; q < NEG; ++q) T[p] += C[p][q] * U[q][i];
        }
#pragma unroll
        for (int j = i; j < N; ++j) {
            double o = A[i][j];
#pragma unroll
            for (int p = 0; p < NEG; ++p) o -= T[p] * U[p][j];
            A[i][j] = A[j][i] = o;
        }
    }
}

// component a of the Helmert basis (orthonormal, zero-sum) of a pattern over NV vertices
template <int NV>
FIPC_HD void helmert_components(const double (&w)[NV], double (&h)[NV - 1]) {
    const Helmert Q = helmert_basis();
    double sum = 0.0;
#pragma unroll
    for (int a = 0; a < NV - 1; ++a) {
        sum += w[a];
        h[a] = (sum - (a + 1) * w[a + 1]) * Q.q[0][a];
    }
}
// the pattern over the vertices of Helmert components h
template <int NV>
FIPC_HD void helmert_pattern(const double (&h)[NV - 1], double (&w)[NV]) {
    const Helmert Q = helmert_basis();
#pragma unroll
    for (int v = 0; v < NV; ++v) w[v] = 0.0;
#pragma unroll
    for (int a = 0; a < NV - 1; ++a) {
        const double s = h[a] * Q.q[0][a];
#pragma unroll
        for (int v = 0; v <= a; ++v) w[v] += s;
        w[a + 1] -= (a + 1) * s;
    }
}

// block (v, w) of the row's Hessian and its mirror image
FIPC_HD void store_pair(double* Hb, int v, int w, const double (&B)[3][3]) {
#pragma unroll
    for (int i = 0; i < 3; ++i)
#pragma unroll
        for (int j = 0; j < 3; ++j) {
            Hb[(v * 4 + w) * 9 + i * 3 + j] = B[i][j];
            if (v != w) Hb[(w * 4 + v) * 9 + j * 3 + i] = B[i][j];
        }
}

// PT (EE = false): vertices p, t0, t1, t2;  EE: a0, a1, b0, b1
template <bool EE>
FIPC_HD void barrier_row_plane(const v3* X, double dh2, double kappa, double* E, double* g, double* Hb) {
    const v3 r = EE ? X[2] - X[0] : X[0] - X[1], e1 = EE ? X[1] - X[0] : X[2] - X[1], e2 = EE ? X[3] - X[2] : X[3] - X[1];
    const v3 nn = cross(e1, e2);
    const double a = sqrt(sq(e1)), nl = sqrt(sq(nn));
    const v3 n = (1.0 / nl) * nn, t1 = (1.0 / a) * e1, t2 = cross(n, t1);
    const double s = dot(r, nn) / nl, d = s * s;           // from the unrounded normal
    const double bb = dot(e2, t1), dd = nl / a;            // E = [[a, bb], [0, dd]]
    const double beta = dot(r, t2) / dd, alpha = (dot(r, t1) - bb * beta) / a;
    const double b0 = barrier_E(d, dh2, kappa), b1 = barrier_g(d, dh2, kappa), b2 = barrier_H(d, dh2, kappa);
    *E = b0;
    double W[4], u[2][4];                                  // weights of the distance, of omega
    if (EE) {
        W[0] = -1.0 + alpha;
        W[1] = -alpha;
        W[2] = 1.0 + beta;
        W[3] = -beta;
    } else {
        W[0] = 1.0;
        W[1] = -1.0 + alpha + beta;
        W[2] = -alpha;
        W[3] = -beta;
    }
#pragma unroll
    for (int v = 0; v < 4; ++v) {
        g[3 * v] = 2.0 * b1 * s * W[v] * n.x;
        g[3 * v + 1] = 2.0 * b1 * s * W[v] * n.y;
        g[3 * v + 2] = 2.0 * b1 * s * W[v] * n.z;
        const double q1 = EE ? (v == 0 ? -1.0 : (v == 1 ? 1.0 : 0.0)) : (v == 1 ? -1.0 : (v == 2 ? 1.0 : 0.0));
        const double q2 = EE ? (v == 2 ? -1.0 : (v == 3 ? 1.0 : 0.0)) : (v == 1 ? -1.0 : (v == 3 ? 1.0 : 0.0));
        u[0][v] = q1 / a;
        u[1][v] = (q2 - (bb / a) * q1) / dd;
    }
    const double wl = sqrt(W[0] * W[0] + W[1] * W[1] + W[2] * W[2] + W[3] * W[3]);
    double w[4], wh[3], om[2][3];
#pragma unroll
    for (int v = 0; v < 4; ++v) w[v] = W[v] / wl;
    helmert_components<4>(w, wh);
    helmert_components<4>(u[0], om[0]);
    helmert_components<4>(u[1], om[1]);
    double K = (4.0 * b2 * d + 2.0 * b1) * wl * wl, c = -2.0 * b1 * s * wl, f = -2.0 * b1 * d;
    // M = K wh wh^T + f sum (om_i + (c/f) tau_i)(..)^T - (c^2/f) sum tau_i tau_i^T with K, f > 0 inside
    // the barrier: two negative eigenvalues.  Scaled to entries of order one for the FP32 part.
    const double size = fabs(K) + fabs(c) / dd + fabs(f) / (dd * dd);
    const double scale = size > 0.0 ? size : 1.0, inv = 1.0 / scale;
    K *= inv;
    c *= inv;
    f *= inv;
    double M[5][5];
    M[0][0] = M[0][1] = M[1][0] = M[1][1] = 0.0;
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        M[0][2 + k] = M[2 + k][0] = c * om[0][k];
        M[1][2 + k] = M[2 + k][1] = c * om[1][k];
#pragma unroll
        for (int l = 0; l < 3; ++l) M[2 + k][2 + l] = K * wh[k] * wh[l] + f * (om[0][k] * om[0][l] + om[1][k] * om[1][l]);
    }
    remove_negative<5, 2>(M);
#pragma unroll
    for (int i = 0; i < 5; ++i)
#pragma unroll
        for (int j = 0; j < 5; ++j) M[i][j] *= scale;
    // block (x, y) = w_x w_y T + w_x h_y n^T + w_y n h_x^T + N_xy n n^T
    const double nn3[3] = {n.x, n.y, n.z}, a3[3] = {t1.x, t1.y, t1.z}, b3[3] = {t2.x, t2.y, t2.z};
    double T[3][3], h[4][3], cols[3][4];
#pragma unroll
    for (int i = 0; i < 3; ++i) {
        const double pa = M[0][0] * a3[i] + M[0][1] * b3[i], pb = M[0][1] * a3[i] + M[1][1] * b3[i];
#pragma unroll
        for (int j = 0; j < 3; ++j) T[i][j] = pa * a3[j] + pb * b3[j];
    }
    {
        double hk[3] = {M[0][2], M[0][3], M[0][4]}, G0[4], G1[4];
        helmert_pattern<4>(hk, G0);
        hk[0] = M[1][2];
        hk[1] = M[1][3];
        hk[2] = M[1][4];
        helmert_pattern<4>(hk, G1);
#pragma unroll
        for (int v = 0; v < 4; ++v)
#pragma unroll
            for (int i = 0; i < 3; ++i) h[v][i] = G0[v] * a3[i] + G1[v] * b3[i];
#pragma unroll
        for (int k = 0; k < 3; ++k) {
            double hc[3] = {M[2 + k][2], M[2 + k][3], M[2 + k][4]};
            helmert_pattern<4>(hc, cols[k]);
        }
    }
#pragma unroll
    for (int x = 0; x < 4; ++x) {
        double hx[3] = {cols[0][x], cols[1][x], cols[2][x]}, N[4];
        helmert_pattern<4>(hx, N);
#pragma unroll
        for (int y = x; y < 4; ++y) {
            const double ww = w[x] * w[y];
            double p[3], q[3], B[3][3];
#pragma unroll
            for (int i = 0; i < 3; ++i) {
                p[i] = w[x] * h[y][i];
                q[i] = w[y] * h[x][i] + N[y] * nn3[i];
            }
#pragma unroll
            for (int i = 0; i < 3; ++i)
#pragma unroll
                for (int j = 0; j < 3; ++j) B[i][j] = ww * T[i][j] + p[i] * nn3[j] + nn3[i] * q[j];
            store_pair(Hb, x, y, B);
        }
    }
}

FIPC_HD void barrier_row_pe(const v3* X, double dh2, double kappa, double* E, double* g, double* Hb) {
    const v3 q = X[1] - X[0], e = X[2] - X[1];
    const double l = sqrt(sq(e));
    const v3 t = (1.0 / l) * e;
    // the part of q across the edge as (e x q) x e: no cancellation against the part along it
    const v3 eq = cross(e, q);
    const double l2 = sq(e), d = sq(eq) / l2, rho = sqrt(d), gamma = dot(q, t) / l;
    const v3 m = (1.0 / (rho * l2)) * cross(eq, e);
    const double b1 = barrier_g(d, dh2, kappa), b2 = barrier_H(d, dh2, kappa);
    *E = barrier_E(d, dh2, kappa);
    const double W[3] = {-1.0, 1.0 + gamma, -gamma}, A[3] = {0.0, -1.0, 1.0};
#pragma unroll
    for (int v = 0; v < 3; ++v) {
        g[3 * v] = 2.0 * b1 * rho * W[v] * m.x;
        g[3 * v + 1] = 2.0 * b1 * rho * W[v] * m.y;
        g[3 * v + 2] = 2.0 * b1 * rho * W[v] * m.z;
    }
    const double wl = sqrt(W[0] * W[0] + W[1] * W[1] + W[2] * W[2]);
    double w[3], wh[2], ah[2];
#pragma unroll
    for (int v = 0; v < 3; ++v) w[v] = W[v] / wl;
    helmert_components<3>(w, wh);
    helmert_components<3>(A, ah);
    // one negative eigenvalue, as above
    const double k = rho / l, K0 = (4.0 * b2 * d + 2.0 * b1) * wl * wl, c0 = -2.0 * b1 * k * wl, f0 = -2.0 * b1 * k * k;
    const double size = fabs(K0) + fabs(c0) + fabs(f0), scale = size > 0.0 ? size : 1.0, inv = 1.0 / scale;
    const double K = K0 * inv, c = c0 * inv, f = f0 * inv;
    double M[3][3];
    M[0][0] = 0.0;
#pragma unroll
    for (int i = 0; i < 2; ++i) {
        M[0][1 + i] = M[1 + i][0] = c * ah[i];
#pragma unroll
        for (int j = 0; j < 2; ++j) M[1 + i][1 + j] = K * wh[i] * wh[j] + f * ah[i] * ah[j];
    }
    remove_negative<3, 1>(M);
#pragma unroll
    for (int i = 0; i < 3; ++i)
#pragma unroll
        for (int j = 0; j < 3; ++j) M[i][j] *= scale;
    // block (x, y) = t (w_x w_y M_00 t + w_x G_y m)^T + m (w_y G_x t + N_xy m)^T
    const double t3[3] = {t.x, t.y, t.z}, m3[3] = {m.x, m.y, m.z};
    double G[3], cols[2][3];
    const double h0[2] = {M[0][1], M[0][2]}, h1[2] = {M[1][1], M[1][2]}, h2[2] = {M[2][1], M[2][2]};
    helmert_pattern<3>(h0, G);
    helmert_pattern<3>(h1, cols[0]);
    helmert_pattern<3>(h2, cols[1]);
#pragma unroll
    for (int x = 0; x < 3; ++x) {
        const double hx[2] = {cols[0][x], cols[1][x]};
        double N[3];
        helmert_pattern<3>(hx, N);
#pragma unroll
        for (int y = x; y < 3; ++y) {
            double p[3], q[3], B[3][3];
            const double ca = w[x] * w[y] * M[0][0], cb = w[x] * G[y], cc = w[y] * G[x];
#pragma unroll
            for (int i = 0; i < 3; ++i) {
                p[i] = ca * t3[i] + cb * m3[i];
                q[i] = cc * t3[i] + N[y] * m3[i];
            }
#pragma unroll
            for (int i = 0; i < 3; ++i)
#pragma unroll
                for (int j = 0; j < 3; ++j) B[i][j] = t3[i] * p[j] + m3[i] * q[j];
            store_pair(Hb, x, y, B);
        }
    }
}

FIPC_HD void barrier_row_pp(const v3* X, double dh2, double kappa, double* E, double* g, double* Hb) {
    const v3 r = X[0] - X[1];
    const double d = sq(r), b1 = barrier_g(d, dh2, kappa), b2 = barrier_H(d, dh2, kappa);
    *E = barrier_E(d, dh2, kappa);
    const double K = 4.0 * b2 * d + 2.0 * b1, k = K > 0.0 ? K / d : 0.0;
    const double rr[3] = {r.x, r.y, r.z};
#pragma unroll
    for (int i = 0; i < 3; ++i) {
        g[i] = 2.0 * b1 * rr[i];
        g[3 + i] = -g[i];
#pragma unroll
        for (int j = 0; j < 3; ++j) {
            const double h = k * rr[i] * rr[j];
            Hb[i * 3 + j] = Hb[5 * 9 + i * 3 + j] = h;
            Hb[9 + i * 3 + j] = Hb[4 * 9 + i * 3 + j] = -h;
        }
    }
}

// mollifier of the EE-type rows with its first two derivatives in D = |e1 x e2|^2: the threshold is of
// the rest shape (distance.py:1671-1673 and EEM_E/g/H)
struct Mollifier {
    double val, d1, d2;
};
FIPC_HD Mollifier mollifier(double D, const v3* X0) {
    Mollifier m{1.0, 0.0, 0.0};
    const double eps = 1.0e-3 * sq(X0[0] - X0[1]) * sq(X0[2] - X0[3]);
    if (D < eps) {
        const double q = D / eps;
        m.val = (-q + 2.0) * q;
        m.d1 = 2.0 * (1.0 / eps) * (-(1.0 / eps) * D + 1.0);
        m.d2 = -2.0 / (eps * eps);
    }
    return m;
}

// barrier energy of a row
FIPC_HD double barrier_energy(int type, const v3* X, const v3* X0, double dh2, double kappa) {
    const bool ee = type >= T_EE;
    const v3 r = type == T_PE ? X[1] - X[0] : (ee ? X[2] - X[0] : X[0] - X[1]);
    double f, D = 0.0;
    if (type == T_PP) {
        f = sq(r);
    } else if (type == T_PE) {
        const v3 e = X[2] - X[1];
        f = sq(cross(r, e)) * (1.0 / sq(e));
    } else {
        const v3 e1 = ee ? X[1] - X[0] : X[2] - X[1], e2 = ee ? X[3] - X[2] : X[3] - X[1];
        const v3 n = cross(e1, e2);
        D = sq(n);
        if (type == T_PPM) {
            f = sq(r);
        } else if (type == T_PEM) {
            f = sq(cross(r, e2)) * (1.0 / sq(e2));
        } else {
            const double s = dot(r, n);
            f = s * s * (1.0 / D);
        }
    }
    const double b = barrier_E(f, dh2, kappa);
    return type >= T_EEM ? b * mollifier(D, X0).val : b;
}

// Unmollified rows with their projected Hessian, for kappa > 0: the closed forms know the signs of the
// barrier's derivatives
FIPC_HD void barrier_row_closed(int type, const v3* X, double dh2, double kappa, double* E, double* g, double* Hb) {
    if (type == T_PP) barrier_row_pp(X, dh2, kappa, E, g, Hb);
    else if (type == T_PE) barrier_row_pe(X, dh2, kappa, E, g, Hb);
    else if (type == T_PT) barrier_row_plane<false>(X, dh2, kappa, E, g, Hb);
    else barrier_row_plane<true>(X, dh2, kappa, E, g, Hb);
}

// A row in reduced coordinates: any type and kappa, want = 1 or 2 (see barrier_row)
FIPC_HD int barrier_row_reduced(int type, const v3* X, const v3* X0, double dh2, double kappa, int want, double* E, double* g, double* Hb) {
    const RowMap m = row_map(type);
    v3 y[3];
    for (int k = 0; k < m.ny; ++k) {
        v3 s = mk(0, 0, 0);
        for (int v = 0; v < m.nv; ++v)
            if (m.C[k][v] != 0.0) s = s + m.C[k][v] * X[v];
        y[k] = s;
    }
    double fg[9] = {0}, fH[81] = {0};
    double Dv = 0.0, Dg[9] = {0}, DH[81] = {0};
    double f;
    // distance (f) and, for EE-type rows, the mollifier variable D = |e1 x e2|^2
    if (type == T_PP || type == T_PPM) {
        f = sq(y[0]);
        put3(fg, 0, y[0], 2.0);
        put_ident(fH, 0, 0, 2.0);
        if (type == T_PPM) Dv = cross_norm2(y[1], y[2], 1, 2, Dg, DH);
    } else if (type == T_PE) {
        f = line_dist(y[0], y[1], 0, 1, fg, fH);
    } else if (type == T_PEM) {
        f = line_dist(y[0], y[2], 0, 2, fg, fH);
        Dv = cross_norm2(y[1], y[2], 1, 2, Dg, DH);
    } else {
        f = triple_dist(y[0], y[1], y[2], fg, fH, &Dv, Dg, DH);
    }
    const double b = barrier_E(f, dh2, kappa);
    const Mollifier mo = type >= T_EEM ? mollifier(Dv, X0) : Mollifier{1.0, 0.0, 0.0};
    const double mval = mo.val, m1 = mo.d1, m2 = mo.d2;
    *E = b * mval;
    const double b1 = barrier_g(f, dh2, kappa), b2 = barrier_H(f, dh2, kappa);
    const int n = 3 * m.ny;
    double gy[9], Hy[81];
    for (int i = 0; i < n; ++i) gy[i] = mval * b1 * fg[i] + b * m1 * Dg[i];
    for (int i = 0; i < n; ++i)
        for (int j = 0; j < n; ++j)
            Hy[i * 9 + j] = mval * (b2 * fg[i] * fg[j] + b1 * fH[i * 9 + j])
                            + b1 * m1 * (fg[i] * Dg[j] + Dg[i] * fg[j])
                            + b * (m2 * Dg[i] * Dg[j] + m1 * DH[i * 9 + j]);
    // x-space gradient g = C^T gy
    for (int v = 0; v < m.nv; ++v)
        for (int c = 0; c < 3; ++c) {
            double s = 0.0;
            for (int k = 0; k < m.ny; ++k) s += m.C[k][v] * gy[3 * k + c];
            g[3 * v + c] = s;
        }
    // K = C Q (ny x ny coefficient matrix), M = K^T Hy K (blockwise, 3x3 identity factor)
    const int na = m.nv - 1;   // == ny
    const Helmert Q = helmert_basis();
    double K[3][3];
    for (int k = 0; k < m.ny; ++k)
        for (int a = 0; a < na; ++a) {
            double s = 0.0;
            for (int v = 0; v < m.nv; ++v) s += m.C[k][v] * Q.q[v][a];
            K[k][a] = s;
        }
    double M[81], HK[27];
    for (int bb = 0; bb < na; ++bb) {
        for (int r = 0; r < n; ++r)
            for (int j = 0; j < 3; ++j) {
                double s = 0.0;
                for (int l = 0; l < m.ny; ++l) s += K[l][bb] * Hy[r * 9 + 3 * l + j];
                HK[r * 3 + j] = s;
            }
        for (int a = 0; a < na; ++a)
            for (int ij = 0; ij < 9; ++ij) {
                double s = 0.0;
                for (int k = 0; k < m.ny; ++k) s += K[k][a] * HK[9 * k + ij];
                M[(3 * a + ij / 3) * 9 + 3 * bb + ij % 3] = s;
            }
    }
    int st = 0;
    if (want != 2) st = psd_project(n, M);
    // H = Q proj(M) Q^T in 3x3 vertex blocks
    for (int w = 0; w < m.nv; ++w) {
        for (int r = 0; r < n; ++r)
            for (int j = 0; j < 3; ++j) {
                double s = 0.0;
                for (int bb = 0; bb < na; ++bb) s += Q.q[w][bb] * M[r * 9 + 3 * bb + j];
                HK[r * 3 + j] = s;
            }
        for (int v = 0; v < m.nv; ++v)
            for (int ij = 0; ij < 9; ++ij) {
                double s = 0.0;
                for (int a = 0; a < na; ++a) s += Q.q[v][a] * HK[9 * a + ij];
                Hb[(v * 4 + w) * 9 + ij] = s;
            }
    }
    return st;
}

// the same out of line, for the rare callers
#if defined(__CUDACC__)
__host__ __device__ __noinline__ static
#else
static inline
#endif
int barrier_row_rare(int type, const v3* X, const v3* X0, double dh2, double kappa, int want, double* E, double* g, double* Hb) {
    return barrier_row_reduced(type, X, X0, dh2, kappa, want, E, g, Hb);
}

// Energy (E), gradient (g, 12 = 3*nv used) and projected Hessian in 3x3 vertex blocks
// (Hb[(v*4+w)*9 + i*3+j] for v,w < nv) of one constraint row.  X: the row's vertices
// (nv used), X0: rest positions of the four EE-type vertices (mollified types only).
// want: 0 energy only, 1 energy + gradient + projected Hessian, 2 energy + gradient + the
// Hessian without the projection.  Returns the eigen-solver status.
FIPC_HD int barrier_row(int type, const v3* X, const v3* X0, double dh2, double kappa, int want,
                        double* E, double* g, double* Hb) {
    if (!want) {
        *E = barrier_energy(type, X, X0, dh2, kappa);
        return 0;
    }
    if (want == 1 && type <= T_EE) {
        if (!(kappa > 0.0)) return barrier_row_rare(type, X, X0, dh2, kappa, want, E, g, Hb);
        barrier_row_closed(type, X, dh2, kappa, E, g, Hb);
        return 0;
    }
    return barrier_row_reduced(type, X, X0, dh2, kappa, want, E, g, Hb);
}

}  // namespace fipc
