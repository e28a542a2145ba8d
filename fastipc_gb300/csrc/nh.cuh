// Neo-Hookean tet element: energy, gradient and PSD-projected Hessian (host + device).
//
// Restates common/physics/neo_hookean.py (psi(sigma) 6-16, d psi/d sigma 20-34, its Hessian
// 38-58, P(F) 62-67, projected dP/dF 71-131) and the element assembly of
// projects/FastIPC/NEWTON_IPC.py:568-691 (F = Ds Dm^-1, scaled by dt^2 * vol0).
//
// dP/dF is never formed.  In the basis D_ab = u_a v_b^T (U, V from the SVD of F) it is the
// block matrix M of the reference: the projected 3x3 sigma-Hessian on {D_00, D_11, D_22} and
// one make_pd-ed 2x2 block per pair (a, b) on {D_ab, D_ba}.  With z_b = B^T-image of v_b
// (z_b[0] = -sum_m (Dm^-1 V)[m][b], z_b[m+1] = (Dm^-1 V)[m][b]) the 3x3 block (v, w) of the
// 12x12 element Hessian is U C(v,w) U^T with C_ac = sum_{b,d} M[ab][cd] z_b[v] z_d[w]; M has
// 21 nonzeros, so each block costs two 3x3 products.
#pragma once

#include "common.cuh"
#include "eig.cuh"

namespace fipc {

// make_pd of common/math/math_tools.py:40-64 on [[a, b], [c, d]] (row-major)
FIPC_HD void make_pd2(double* Mx) {
    const double a = Mx[0], b = (Mx[1] + Mx[2]) / 2.0, d = Mx[3];
    const double b2 = b * b, D = a * d - b2, T2 = (a + d) / 2.0;
    const double sq_ = sqrt(T2 * T2 - D);
    const double L2 = T2 - sq_;
    if (L2 < 0.0) {
        const double L1 = T2 + sq_;
        if (L1 <= 0.0) {
            Mx[0] = Mx[1] = Mx[2] = Mx[3] = 0.0;
        } else if (b2 == 0.0) {
            Mx[0] = L1;
            Mx[1] = Mx[2] = Mx[3] = 0.0;
        } else {
            const double L1md = L1 - d, r = L1md / L1;
            Mx[0] = r * L1md;
            Mx[1] = b * r;
            Mx[2] = b * r;
            Mx[3] = b2 / L1;
        }
    }
}

FIPC_HD double det3(const double* F) {
    return F[0] * (F[4] * F[8] - F[5] * F[7]) - F[1] * (F[3] * F[8] - F[5] * F[6]) + F[2] * (F[3] * F[7] - F[4] * F[6]);
}

// V (rows of 3, orthonormal to FP64 rounding, det +1) close to the right singular vectors of F: FP32 Jacobi
// rotations of F^T F, then Gram-Schmidt in FP64 (the norms are within a few 1e-7 of one, so three terms of
// the series of 1/sqrt do).  The identity when F is zero or not finite.
FIPC_HD void svd3_start(const double* F, double* V) {
    double m = 0.0;
#pragma unroll
    for (int i = 0; i < 9; ++i) m = fmax(m, fabs(F[i]));
    const float inv = (float)(1.0 / m);
    float f[9], a[6], v[9];   // a: 00 01 02 11 12 22
#pragma unroll
    for (int i = 0; i < 9; ++i) {
        f[i] = (float)F[i] * inv;
        v[i] = i % 4 == 0 ? 1.f : 0.f;
    }
    a[0] = f[0] * f[0] + f[3] * f[3] + f[6] * f[6];
    a[1] = f[0] * f[1] + f[3] * f[4] + f[6] * f[7];
    a[2] = f[0] * f[2] + f[3] * f[5] + f[6] * f[8];
    a[3] = f[1] * f[1] + f[4] * f[4] + f[7] * f[7];
    a[4] = f[1] * f[2] + f[4] * f[5] + f[7] * f[8];
    a[5] = f[2] * f[2] + f[5] * f[5] + f[8] * f[8];
#pragma unroll 1
    for (int sweep = 0; sweep < 5; ++sweep) {
        if (!(a[1] * a[1] + a[2] * a[2] + a[4] * a[4] > 1e-15f * (a[0] * a[0] + a[3] * a[3] + a[5] * a[5]))) break;
#pragma unroll
        for (int k = 0; k < 3; ++k) {
            // rotation of columns p, q; r the third
            const int p = k == 2 ? 1 : 0, q = k == 0 ? 1 : 2, r = 3 - p - q;
            float& app = a[p == 0 ? 0 : 3];
            float& aqq = a[q == 1 ? 3 : 5];
            float& apq = a[p == 0 ? (q == 1 ? 1 : 2) : 4];
            float& apr = a[p == 0 ? (r == 1 ? 1 : 2) : 1];          // (0,1), (0,2) or (1,0)
            float& aqr = a[q == 1 ? (r == 0 ? 1 : 4) : (r == 0 ? 2 : 4)];
            const float h = aqq - app, g = 2.f * apq, den = fabsf(h) + sqrtf(h * h + g * g);
            const float t = den > 0.f ? (h >= 0.f ? g : -g) / den : 0.f;
            const float c = 1.f / sqrtf(t * t + 1.f), sn = t * c;
            app -= t * apq;
            aqq += t * apq;
            apq = 0.f;
            const float x = apr, y = aqr;
            apr = c * x - sn * y;
            aqr = sn * x + c * y;
#pragma unroll
            for (int row = 0; row < 3; ++row) {
                const float vx = v[row * 3 + p], vy = v[row * 3 + q];
                v[row * 3 + p] = c * vx - sn * vy;
                v[row * 3 + q] = sn * vx + c * vy;
            }
        }
    }
    v3 a0 = mk(v[0], v[3], v[6]), a1 = mk(v[1], v[4], v[7]);
    double e = sq(a0) - 1.0;
    a0 = (1.0 + e * (0.375 * e - 0.5)) * a0;
    a1 = a1 - dot(a0, a1) * a0;
    e = sq(a1) - 1.0;
    a1 = (1.0 + e * (0.375 * e - 0.5)) * a1;
    v3 a2 = cross(a0, a1);
    if (!(fabs(e) < 1e-4)) {   // not finite
        a0 = mk(1, 0, 0);
        a1 = mk(0, 1, 0);
        a2 = mk(0, 0, 1);
    }
    V[0] = a0.x; V[3] = a0.y; V[6] = a0.z;
    V[1] = a1.x; V[4] = a1.y; V[7] = a1.z;
    V[2] = a2.x; V[5] = a2.y; V[8] = a2.z;
}

// Rotation-variant SVD by one-sided Jacobi (Hestenes) on the columns of F:
// F = U diag(s) V^T, det U = det V = +1, s descending in magnitude, s[2] < 0 iff det F < 0.
// The rotations are FP64, on F V with V from svd3_start: one sweep of small angles and one that finds nothing
// left, where starting from F takes four to six sweeps.  Element Hessians issue FP64 instructions
// back to back (88% of the pipe), so their count is the time: assembling the 960k-tet bar 4.5 -> 3.2 ms with
// the element Hessian's other savings below.
FIPC_HD void svd3(const double* F, double* U, double* s, double* V) {
    double B[9];
    svd3_start(F, V);
#pragma unroll
    for (int i = 0; i < 3; ++i)
#pragma unroll
        for (int j = 0; j < 3; ++j) B[i * 3 + j] = F[i * 3] * V[j] + F[i * 3 + 1] * V[3 + j] + F[i * 3 + 2] * V[6 + j];
    double n2[3];
#pragma unroll 1
    for (int sweep = 0; sweep < 10; ++sweep) {
        bool rotated = false;
#pragma unroll
        for (int c = 0; c < 3; ++c) n2[c] = B[c] * B[c] + B[3 + c] * B[3 + c] + B[6 + c] * B[6 + c];
#pragma unroll
        for (int k = 0; k < 3; ++k) {
            const int p = k == 2 ? 1 : 0, q = k == 0 ? 1 : 2;
            const double ga = B[p] * B[q] + B[3 + p] * B[3 + q] + B[6 + p] * B[6 + q];
            if (ga * ga <= 1e-30 * (n2[p] * n2[q]) || ga == 0.0) continue;
            rotated = true;
            const double h = n2[q] - n2[p];
            double t, c;
            if (fabs(ga) < 1e-3 * fabs(h)) {
                // tan 2a = 2 x, x = ga / h: series to x^5, of 1/sqrt(1 + t^2) to t^6
                const double x = ga / h, xx = x * x;
                t = x * (1.0 - xx * (1.0 - 2.0 * xx));
                const double tt = t * t;
                c = 1.0 - tt * (0.5 - 0.375 * tt);
            } else {
                const double zeta = h / (2.0 * ga);
                t = (zeta >= 0.0 ? 1.0 : -1.0) / (fabs(zeta) + sqrt(1.0 + zeta * zeta));
                c = 1.0 / sqrt(1.0 + t * t);
            }
            const double sn = c * t;
            n2[p] -= t * ga;
            n2[q] += t * ga;
#pragma unroll
            for (int r = 0; r < 3; ++r) {
                const double bp = B[r * 3 + p], bq = B[r * 3 + q];
                B[r * 3 + p] = c * bp - sn * bq;
                B[r * 3 + q] = sn * bp + c * bq;
                const double vp = V[r * 3 + p], vq = V[r * 3 + q];
                V[r * 3 + p] = c * vp - sn * vq;
                V[r * 3 + q] = sn * vp + c * vq;
            }
        }
        if (!rotated) break;
    }
#pragma unroll
    for (int c = 0; c < 3; ++c) n2[c] = B[c] * B[c] + B[3 + c] * B[3 + c] + B[6 + c] * B[6 + c];
    // descending order: each exchange negates one column, which keeps det V = +1
    double Bs[9];
#pragma unroll
    for (int i = 0; i < 9; ++i) Bs[i] = B[i];
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        const int p = k == 1 ? 1 : 0, q = p + 1;   // (0,1), (1,2), (0,1)
        const bool sw = n2[q] > n2[p];
        const double np = n2[p], nq = n2[q];
        n2[p] = sw ? nq : np;
        n2[q] = sw ? np : nq;
#pragma unroll
        for (int r = 0; r < 3; ++r) {
            const double bp = Bs[r * 3 + p], bq = Bs[r * 3 + q], vp = V[r * 3 + p], vq = V[r * 3 + q];
            Bs[r * 3 + p] = sw ? bq : bp;
            Bs[r * 3 + q] = sw ? -bp : bq;
            V[r * 3 + p] = sw ? vq : vp;
            V[r * 3 + q] = sw ? -vp : vq;
        }
    }
    // u0, u1 from the two largest columns, u2 = u0 x u1; s_i = u_i . b_i
    const v3 b0 = mk(Bs[0], Bs[3], Bs[6]), b1 = mk(Bs[1], Bs[4], Bs[7]), b2 = mk(Bs[2], Bs[5], Bs[8]);
    const double n0 = sqrt(sq(b0));
    const v3 u0 = (1.0 / n0) * b0;
    v3 u1 = b1 - dot(u0, b1) * u0;
    u1 = (1.0 / sqrt(sq(u1))) * u1;
    const v3 u2 = cross(u0, u1);
    U[0] = u0.x; U[3] = u0.y; U[6] = u0.z;
    U[1] = u1.x; U[4] = u1.y; U[7] = u1.z;
    U[2] = u2.x; U[5] = u2.y; U[8] = u2.z;
    s[0] = dot(u0, b0);
    s[1] = dot(u1, b1);
    s[2] = dot(u2, b2);
}

// psi from F directly: sum sigma^2 = |F|^2 and prod sigma = det F (energy-only paths)
FIPC_HD double nh_psi_F(const double* F, double la, double mu) {
    double s2 = 0.0;
    for (int i = 0; i < 9; ++i) s2 += F[i] * F[i];
    const double lp = log(det3(F));
    return mu / 2.0 * (s2 - 3) - (mu - la / 2.0 * lp) * lp;
}

// deformation gradient F = Ds Dm^-1 (row-major)
FIPC_HD void deformation_gradient(const v3* X, const double* IB, double* F) {
    const v3 d1 = X[1] - X[0], d2 = X[2] - X[0], d3 = X[3] - X[0];
    const double Ds[9] = {d1.x, d2.x, d3.x, d1.y, d2.y, d3.y, d1.z, d2.z, d3.z};
    for (int i = 0; i < 3; ++i)
        for (int j = 0; j < 3; ++j)
            F[i * 3 + j] = Ds[i * 3 + 0] * IB[0 * 3 + j] + Ds[i * 3 + 1] * IB[1 * 3 + j] + Ds[i * 3 + 2] * IB[2 * 3 + j];
}

// Element energy (returned), gradient g[12] and the 10 upper 3x3 blocks of the Hessian
// Hu[blk*9 + i*3 + j], blk enumerating (v, w) with v <= w in row order
// (0,0)(0,1)(0,2)(0,3)(1,1)(1,2)(1,3)(2,2)(2,3)(3,3).  w = dt^2 * vol0.
FIPC_HD double nh_element(const v3* X, const double* IB, double la, double mu, double wgt, double* g, double* Hu) {
    double F[9], U[9], s[3], V[9];
    deformation_gradient(X, IB, F);
    svd3(F, U, s, V);
    // one logarithm and one division of J = s0 s1 s2 serve the energy, the stress and the Hessian
    const double J = s[0] * s[1] * s[2], lp = log(J), rJ = 1.0 / J;
    // psi(sigma) (neo_hookean.py:6-16)
    const double psi = (mu / 2.0 * (s[0] * s[0] + s[1] * s[1] + s[2] * s[2] - 3) - (mu - la / 2.0 * lp) * lp) * wgt;
    // P(F) = mu F + (la ln J - mu) F^-T  (neo_hookean.py:62-67)
    {
        const double C[9] = {F[4] * F[8] - F[5] * F[7], F[5] * F[6] - F[3] * F[8], F[3] * F[7] - F[4] * F[6],
                             F[2] * F[7] - F[1] * F[8], F[0] * F[8] - F[2] * F[6], F[1] * F[6] - F[0] * F[7],
                             F[1] * F[5] - F[2] * F[4], F[2] * F[3] - F[0] * F[5], F[0] * F[4] - F[1] * F[3]};
        // det F itself, which the singular values' product misses by their rounding: its logarithm and
        // reciprocal from theirs and the relative difference r
        const double JF = F[0] * C[0] + F[1] * C[1] + F[2] * C[2], r = (JF - J) * rJ;
        const double sc = fabs(r) < 1e-6 ? (la * (lp + r * (1.0 - 0.5 * r)) - mu) * (rJ * (1.0 - r * (1.0 - r))) : (la * log(JF) - mu) / JF;
        double P[9];
        for (int i = 0; i < 9; ++i) P[i] = (mu * F[i] + sc * C[i]) * wgt;
        // g_{m+1, i} = sum_j IB[m][j] P[i][j], g_0 = -sum_m
        for (int i = 0; i < 3; ++i) {
            double acc = 0.0;
            for (int mm = 0; mm < 3; ++mm) {
                const double r = IB[mm * 3 + 0] * P[i * 3 + 0] + IB[mm * 3 + 1] * P[i * 3 + 1] + IB[mm * 3 + 2] * P[i * 3 + 2];
                g[(mm + 1) * 3 + i] = r;
                acc += r;
            }
            g[i] = -acc;
        }
    }
    // sigma-space gradient / projected Hessian and the three 2x2 blocks (neo_hookean.py:75-98)
    const double inv[3] = {s[1] * s[2] * rJ, s[0] * s[2] * rJ, s[0] * s[1] * rJ};
    double Hs[9];
    for (int i = 0; i < 3; ++i) {
        const double i2 = inv[i] * inv[i];
        Hs[i * 4] = mu * (1.0 + i2) - la * i2 * (lp - 1.0);
    }
    Hs[1] = Hs[3] = la * inv[0] * inv[1];
    Hs[5] = Hs[7] = la * inv[1] * inv[2];
    Hs[2] = Hs[6] = la * inv[0] * inv[2];
    psd_project3(Hs);
    const double middle = mu - la * lp;
    double Bk[3][4];
    const int pa[3] = {0, 1, 2}, pb[3] = {1, 2, 0};
    for (int k = 0; k < 3; ++k) {
        const int i = pa[k], j = pb[k];
        const double mid = middle * inv[i] * inv[j], left = (mu + mid) / 2.0;
        // (d psi/d s_i + d psi/d s_j) / (2 max(s_i + s_j, 1e-6)), whose numerator is (s_i + s_j)(mu - mid)
        const double ss = s[i] + s[j];
        double right = (mu - mid) / 2.0;
        if (ss < 0.000001) right *= ss / 0.000001;
        Bk[k][0] = left + right;
        Bk[k][1] = left - right;
        Bk[k][2] = left - right;
        Bk[k][3] = left + right;
        // its eigenvalues are 2 left and 2 right: with both clearly positive make_pd leaves the
        // block unchanged, so its square root is skipped
        if (!(left > 1e-8 * fabs(right) && right > 1e-8 * fabs(left))) make_pd2(Bk[k]);
    }
    // the weight dt^2 vol0 folded into the sigma-space coefficients once
    for (int i = 0; i < 9; ++i) Hs[i] *= wgt;
    for (int k = 0; k < 3; ++k)
        for (int i = 0; i < 4; ++i) Bk[k][i] *= wgt;
    // z_b over the 4 vertices
    double z[3][4];
    for (int b = 0; b < 3; ++b) {
        double acc = 0.0;
        for (int mm = 0; mm < 3; ++mm) {
            const double zz = IB[mm * 3 + 0] * V[0 * 3 + b] + IB[mm * 3 + 1] * V[1 * 3 + b] + IB[mm * 3 + 2] * V[2 * 3 + b];
            z[b][mm + 1] = zz;
            acc += zz;
        }
        z[b][0] = -acc;
    }
    // Blocks (v, w) with 1 <= v <= w <= 3 directly: U C U^T with C built from z_b[v] z_d[w].  The
    // Hessian is bilinear in (z[.][v], z[.][w]) and z[.][0] = -(z[.][1] + z[.][2] + z[.][3]), so
    // the blocks of vertex 0 follow by sums: H(0,w) = -sum_{v>=1} H(v,w) with H(v,w) = H(w,v)^T,
    // and H(0,0) = -sum_{w>=1} H(0,w)^T.
#pragma unroll
    for (int v = 1; v < 4; ++v)
#pragma unroll
        for (int w = v; w < 4; ++w) {
            // Hu block of (v, w), v <= w: (1,1) 4, (1,2) 5, (1,3) 6, (2,2) 7, (2,3) 8, (3,3) 9
            double* out = Hu + 9 * (v == 1 ? 3 + w : (v == 2 ? 5 + w : 9));
            double Z[3][3];  // Z[b][d] = z_b[v] z_d[w]
            for (int b = 0; b < 3; ++b)
                for (int d = 0; d < 3; ++d) Z[b][d] = v == w && d < b ? Z[d][b] : z[b][v] * z[d][w];
            double C[9];
            // Bk[0]: pair (0,1); Bk[1]: pair (1,2); Bk[2]: pair (2,0)   (row-major 2x2)
            C[0 * 3 + 0] = Hs[0] * Z[0][0] + Bk[0][0] * Z[1][1] + Bk[2][3] * Z[2][2];
            C[1 * 3 + 1] = Hs[4] * Z[1][1] + Bk[0][3] * Z[0][0] + Bk[1][0] * Z[2][2];
            C[2 * 3 + 2] = Hs[8] * Z[2][2] + Bk[1][3] * Z[1][1] + Bk[2][0] * Z[0][0];
            if (v == w) {   // Z, C and the block are symmetric
                C[0 * 3 + 1] = C[1 * 3 + 0] = (Hs[1] + Bk[0][1]) * Z[0][1];
                C[1 * 3 + 2] = C[2 * 3 + 1] = (Hs[5] + Bk[1][1]) * Z[1][2];
                C[0 * 3 + 2] = C[2 * 3 + 0] = (Hs[2] + Bk[2][2]) * Z[0][2];
            } else {
                C[0 * 3 + 1] = Hs[1] * Z[0][1] + Bk[0][1] * Z[1][0];
                C[1 * 3 + 0] = Hs[3] * Z[1][0] + Bk[0][2] * Z[0][1];
                C[1 * 3 + 2] = Hs[5] * Z[1][2] + Bk[1][1] * Z[2][1];
                C[2 * 3 + 1] = Hs[7] * Z[2][1] + Bk[1][2] * Z[1][2];
                C[0 * 3 + 2] = Hs[2] * Z[0][2] + Bk[2][2] * Z[2][0];
                C[2 * 3 + 0] = Hs[6] * Z[2][0] + Bk[2][1] * Z[0][2];
            }
            double T[9];
            for (int i = 0; i < 3; ++i)
                for (int c = 0; c < 3; ++c) T[i * 3 + c] = U[i * 3 + 0] * C[0 * 3 + c] + U[i * 3 + 1] * C[1 * 3 + c] + U[i * 3 + 2] * C[2 * 3 + c];
            for (int i = 0; i < 3; ++i)
                for (int j = 0; j < 3; ++j)
                    out[i * 3 + j] = v == w && j < i ? out[j * 3 + i] : T[i * 3 + 0] * U[j * 3 + 0] + T[i * 3 + 1] * U[j * 3 + 1] + T[i * 3 + 2] * U[j * 3 + 2];
        }
    // H(0,w), w = 1..3 (blocks 1..3) and H(0,0) (block 0)
    const double* H11 = Hu + 36;
    const double* H12 = Hu + 45;
    const double* H13 = Hu + 54;
    const double* H22 = Hu + 63;
    const double* H23 = Hu + 72;
    const double* H33 = Hu + 81;
    for (int i = 0; i < 3; ++i)
        for (int j = 0; j < 3; ++j) {
            const int ij = i * 3 + j, ji = j * 3 + i;
            Hu[9 + ij] = -(H11[ij] + H12[ji] + H13[ji]);
            Hu[18 + ij] = -(H12[ij] + H22[ij] + H23[ji]);
            Hu[27 + ij] = -(H13[ij] + H23[ij] + H33[ij]);
        }
    for (int i = 0; i < 3; ++i)
        for (int j = 0; j < 3; ++j) {
            const int ji = j * 3 + i;
            Hu[i * 3 + j] = -(Hu[9 + ji] + Hu[18 + ji] + Hu[27 + ji]);
        }
    return psi;
}

}  // namespace fipc
