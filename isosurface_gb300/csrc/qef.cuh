// Feature placement for DualContouring (and, through the row-bounded SVD
// steps, ExtendedMarchingCubes), on the device and on the host.
//
// * TangentPlanes::new over the 8 cell corners (src/feature/mod.rs:91-148)
//   and ParticleBasedMinimisation (src/feature/particle_minimisation.rs:25-72),
//   the f32 half, in qef_planes.cuh
// * MinimiseQEF (src/feature/qef.rs:36-68) with the 3-column f64 SVD of
//   src/math/svd.rs: Householder bidiagonalisation (factorize, :149-292),
//   accumulation of U and V (unpack, :295-410), implicit-shift QR with Givens
//   rotations (diagonalize/qrstep*, :413-847), sign and order normalisation
//   (singularize, :892-925) and the truncated solve (SVD::solve + solveSVD,
//   :55-84, :928-972: singular values below 0.1 are zeroed and then skipped,
//   which leaves their projection in the solution unscaled).
//
// The SVD steps are restated from swiftcoder/isosurface (src/math/svd.rs),
// Copyright 2021 Tristam MacDonald, licensed under the Apache License, Version
// 2.0 (http://www.apache.org/licenses/LICENSE-2.0).
//
// The steps and their operation order follow the reference so that vertex
// positions match it bit for bit (the translation unit is built with
// -fmad=false; f64 sqrt and division are IEEE).  The reference's QR loop has
// no iteration bound; here it stops after QR_SWEEP_LIMIT sweeps and reports it.
#pragma once
#include <cuda_runtime.h>

#include "qef_planes.cuh"

namespace iso {
namespace qef {

constexpr int QR_SWEEP_LIMIT = 10000;

// Every loop below has constant bounds (R rows, of which the first `rows`
// count) and every index is a constant once unrolled, so the matrices live in
// registers: indexed at run time they were in local memory, whose loads stood
// in every step of the chain (a 257 dual lattice's solves 138 us, now 121; a
// 128 solid's, with rows bounded by 6 where they can be, 140, now 92).
#define ISO_QEF_FN __host__ __device__ __forceinline__

// factorize_hh of column i of m from the diagonal down: n = rows - i entries
template <int R>
ISO_QEF_FN double householder_col(double (&m)[R][3], int i, int rows) {
    const int n = rows - i;
    double tau = 0.0;
    if (n > 1) {
        double xnorm;
        if (n == 2) {
            xnorm = fabs(m[i + 1][i]);
        } else {
            double scl = 0.0, ssq = 1.0;
#pragma unroll
            for (int y = 1; y < R; ++y) {
                if (y <= i || y >= rows) continue;
                const double v = fabs(m[y][i]);
                if (v != 0.0) {
                    // one division for either branch: a warp's lanes take both
                    const bool grow = scl < v;
                    const double r = (grow ? scl : v) / (grow ? v : scl);
                    ssq = grow ? 1.0 + ssq * r * r : ssq + r * r;
                    scl = grow ? v : scl;
                }
            }
            xnorm = scl * sqrt(ssq);
        }
        if (xnorm != 0.0) {
            const double alpha = m[i][i];
            double beta = sqrt(alpha * alpha + xnorm * xnorm);
            if (alpha >= 0.0) beta = -beta;
            tau = (beta - alpha) / beta;
            const double s = 1.0 / (alpha - beta);
            m[i][i] = beta;
#pragma unroll
            for (int y = 1; y < R; ++y)
                if (y > i && y < rows) m[y][i] *= s;
        }
    }
    return tau;
}

// factorize_hh over two entries
ISO_QEF_FN double householder_pair(double& x0, double& x1) {
    const double xnorm = fabs(x1);
    if (xnorm == 0.0) return 0.0;
    const double alpha = x0;
    double beta = sqrt(alpha * alpha + xnorm * xnorm);
    if (alpha >= 0.0) beta = -beta;
    const double tau = (beta - alpha) / beta;
    const double s = 1.0 / (alpha - beta);
    x0 = beta;
    x1 *= s;
    return tau;
}

// R bounds `rows` (8 for DualContouring's corners, 12 for the edge crossings
// of ExtendedMarchingCubes)
template <int R>
ISO_QEF_FN void bidiagonalise(double (&m)[R][3], double (&tau_u)[3], double (&tau_v)[2], int rows) {
#pragma unroll
    for (int i = 0; i < 3; ++i) {
        const double tau = householder_col(m, i, rows);
        tau_u[i] = tau;
        if (i == 2) break;
        if (tau != 0.0) {
#pragma unroll
            for (int x = 1; x < 3; ++x) {
                if (x <= i) continue;
                double wx = m[i][x];
#pragma unroll
                for (int y = 1; y < R; ++y)
                    if (y > i && y < rows) wx += m[y][x] * m[y][i];
                const double tau_wx = tau * wx;
                m[i][x] -= tau_wx;
#pragma unroll
                for (int y = 1; y < R; ++y)
                    if (y > i && y < rows) m[y][x] -= tau_wx * m[y][i];
            }
        }
        // the row right of the superdiagonal: two entries in row 0, one (nothing to do) in row 1
        tau_v[i] = 0.0;
        if (i == 0) {
            const double tv = householder_pair(m[0][1], m[0][2]);
            tau_v[0] = tv;
            if (tv != 0.0) {
#pragma unroll
                for (int y = 1; y < R; ++y) {
                    if (y >= rows) continue;
                    double wy = m[y][1];
                    wy += m[y][2] * m[0][2];
                    const double tau_wy = tv * wy;
                    m[y][1] -= tau_wy;
                    m[y][2] -= tau_wy * m[0][2];
                }
            }
        }
    }
}

template <int R>
ISO_QEF_FN void unpack(double (&u)[R][3], double (&v)[3][3], double (&tau_u)[3], double (&tau_v)[2], int rows) {
    v[0][0] = v[1][1] = v[2][2] = 1.0;
    v[0][1] = v[0][2] = v[1][0] = v[1][2] = v[2][0] = v[2][1] = 0.0;
#pragma unroll
    for (int i = 1; i >= 0; --i) {
        const double tau = tau_v[i];
        if (tau != 0.0) {
#pragma unroll
            for (int x = 1; x < 3; ++x) {
                if (x <= i) continue;
                double wx = v[i + 1][x];
#pragma unroll
                for (int y = 2; y < 3; ++y)
                    if (y >= i + 2) wx += v[y][x] * u[i][y];
                const double tau_wx = tau * wx;
                v[i + 1][x] -= tau_wx;
#pragma unroll
                for (int y = 2; y < 3; ++y)
                    if (y >= i + 2) v[y][x] -= tau_wx * u[i][y];
            }
        }
    }
#pragma unroll
    for (int i = 0; i < 2; ++i) tau_v[i] = u[i][i + 1];
#pragma unroll
    for (int i = 2; i >= 0; --i) {
        const double tau = tau_u[i];
        tau_u[i] = u[i][i];
        if (tau == 0.0) {
            u[i][i] = 1.0;
            if (i < 2) {
                u[i][2] = 0.0;
                if (i < 1) u[i][1] = 0.0;
            }
#pragma unroll
            for (int y = 1; y < R; ++y)
                if (y > i && y < rows) u[y][i] = 0.0;
        } else {
#pragma unroll
            for (int x = 1; x < 3; ++x) {
                if (x <= i) continue;
                double wx = 0.0;
#pragma unroll
                for (int y = 1; y < R; ++y)
                    if (y > i && y < rows) wx += u[y][x] * u[y][i];
                const double tau_wx = tau * wx;
                u[i][x] = -tau_wx;
#pragma unroll
                for (int y = 1; y < R; ++y)
                    if (y > i && y < rows) u[y][x] -= tau_wx * u[y][i];
            }
#pragma unroll
            for (int y = 1; y < R; ++y)
                if (y > i && y < rows) u[y][i] = u[y][i] * -tau;
            u[i][i] = 1.0 - tau;
        }
    }
}

// entries A..A+N-1 of the diagonal and those between them
template <int A, int N>
ISO_QEF_FN void chop(const double (&a)[3], double (&b)[2]) {
    double ai = a[A];
#pragma unroll
    for (int i = A; i < A + N - 1; ++i) {
        const double bi = b[i];
        const double ai1 = a[i + 1];
        if (fabs(bi) < 1e-5 * (fabs(ai) + fabs(ai1))) b[i] = 0.0;
        ai = ai1;
    }
}

ISO_QEF_FN void givens(double a, double b, double* c, double* s) {
    if (b == 0.0) {
        *c = 1.0;
        *s = 0.0;
    } else {
        // the larger of the two divides; the divisions and the root are
        // shared by both orders, as a warp's lanes take both
        const bool big_b = fabs(b) > fabs(a);
        const double t = (big_b ? -a : -b) / (big_b ? b : a);
        const double r = 1.0 / sqrt(1.0 + t * t);
        const double rt = r * t;
        *c = big_b ? rt : r;
        *s = big_b ? r : rt;
    }
}

ISO_QEF_FN void schur(double a1, double a2, double a3, double* c, double* s) {
    const double apq = a1 * a2 * 2.0;
    if (apq == 0.0) {
        *c = 1.0;
        *s = 0.0;
    } else {
        const double tau = (a2 * a2 + (a3 + a1) * (a3 - a1)) / apq;
        const double root = sqrt(1.0 + tau * tau);
        const bool up = tau >= 0.0;
        const double t = (up ? 1.0 : -1.0) / (up ? tau + root : root - tau);
        *c = 1.0 / sqrt(1.0 + t * t);
        *s = t * *c;
    }
}

// columns P and Q of the first `rows` rows rotated
template <int P, int Q, int R>
ISO_QEF_FN void rot_cols(double (&m)[R][3], int rows, double c, double s) {
#pragma unroll
    for (int i = 0; i < R; ++i) {
        if (i >= rows) continue;
        const double mp = m[i][P], mq = m[i][Q];
        m[i][P] = mp * c - mq * s;
        m[i][Q] = mp * s + mq * c;
    }
}

template <int P, int Q, int R>
ISO_QEF_FN void swap_cols(double (&m)[R][3], int rows) {
#pragma unroll
    for (int i = 0; i < R; ++i) {
        if (i >= rows) continue;
        const double t = m[i][P];
        m[i][P] = m[i][Q];
        m[i][Q] = t;
    }
}

// a zero on the diagonal at COL of the whole 3 x 3 bidiagonal
template <int COL, int R>
ISO_QEF_FN void qr_middle(double (&u)[R][3], double (&tau_u)[3], double (&tau_v)[2], int rows) {
    double x = tau_v[COL];
    double y = tau_u[COL + 1];
    double c, s;
    givens(y, -x, &c, &s);
    rot_cols<COL, COL + 1>(u, rows, c, s);
    tau_u[COL + 1] = x * s + y * c;
    tau_v[COL] = x * c - y * s;
    if (COL == 0) {
        const double z = tau_v[1];
        tau_v[1] *= c;
        x = z * -s;
        y = tau_u[2];
        givens(y, -x, &c, &s);
        rot_cols<0, 2>(u, rows, c, s);
        tau_u[2] = x * s + y * c;
    }
}

// a zero at the end of the diagonal
ISO_QEF_FN void qr_end(double (&v)[3][3], double (&tau_u)[3], double (&tau_v)[2]) {
    double x = tau_u[1];
    double y = tau_v[1];
    double c, s;
    givens(x, y, &c, &s);
    rot_cols<1, 2>(v, 3, c, s);
    tau_u[1] = x * c - y * s;
    tau_v[1] = x * s + y * c;
    const double z = tau_v[0];
    tau_v[0] *= c;
    x = tau_u[0];
    y = z * s;
    givens(x, y, &c, &s);
    rot_cols<0, 2>(v, 3, c, s);
    tau_u[0] = x * c - y * s;
}

ISO_QEF_FN double shift(const double (&tau_u)[3], const double (&tau_v)[2]) {
    const double ta = tau_u[1] * tau_u[1] + tau_v[0] * tau_v[0];
    const double tb = tau_u[2] * tau_u[2] + tau_v[1] * tau_v[1];
    const double tab = tau_u[1] * tau_v[1];
    const double dt = (ta - tb) / 2.0;
    const double root = sqrt(dt * dt + tab * tab);
    const bool up = dt >= 0.0;
    const double q = tab * tab / (up ? dt + root : root - dt);
    return up ? tb - q : tb + q;
}

// the 2 x 2 block of columns A and A + 1
template <int A, int R>
ISO_QEF_FN void qr_cols2(double (&u)[R][3], double (&v)[3][3], double (&tau_u)[3], double (&tau_v)[2], int rows) {
    double c, s;
    if (tau_u[A] == 0.0) {
        givens(tau_v[A], tau_u[A + 1], &c, &s);
        tau_u[A] = tau_v[A] * c - tau_u[A + 1] * s;
        tau_v[A] = tau_v[A] * s + tau_u[A + 1] * c;
        tau_u[A + 1] = 0.0;
        rot_cols<A, A + 1>(u, rows, c, s);
        swap_cols<A, A + 1>(v, 3);
    } else if (tau_u[A + 1] == 0.0) {
        givens(tau_u[A], tau_v[A], &c, &s);
        tau_u[A] = tau_u[A] * c - tau_v[A] * s;
        tau_v[A] = 0.0;
        rot_cols<A, A + 1>(v, 3, c, s);
    } else {
        schur(tau_u[A], tau_v[A], tau_u[A + 1], &c, &s);
        double a11 = tau_u[A] * c - tau_v[A] * s;
        double a21 = -tau_u[A + 1] * s;
        double a12 = tau_u[A] * s + tau_v[A] * c;
        double a22 = tau_u[A + 1] * c;
        rot_cols<A, A + 1>(v, 3, c, s);
        if (a11 * a11 + a21 * a21 < a12 * a12 + a22 * a22) {
            double t = a11;
            a11 = a12;
            a12 = t;
            t = a21;
            a21 = a22;
            a22 = t;
            swap_cols<A, A + 1>(v, 3);
        }
        givens(a11, a21, &c, &s);
        tau_u[A] = a11 * c - a21 * s;
        tau_v[A] = a12 * c - a22 * s;
        tau_u[A + 1] = a12 * s + a22 * c;
        rot_cols<A, A + 1>(u, rows, c, s);
    }
}

// one step on the whole 3 x 3 bidiagonal
template <int R>
ISO_QEF_FN void qr_cols3(double (&u)[R][3], double (&v)[3][3], double (&tau_u)[3], double (&tau_v)[2], int rows) {
    if (tau_u[0] == 0.0) {
        qr_middle<0>(u, tau_u, tau_v, rows);
        return;
    }
    if (tau_u[1] == 0.0) {
        qr_middle<1>(u, tau_u, tau_v, rows);
        return;
    }
    if (tau_u[2] == 0.0) {
        qr_end(v, tau_u, tau_v);
        return;
    }
    const double mu = shift(tau_u, tau_v);
    double y = tau_u[0] * tau_u[0] - mu;
    double z = tau_u[0] * tau_v[0];
    double ak = 0.0, bk = 0.0, zk;
    double ap = tau_u[0], bp = tau_v[0], aq = tau_u[1];
#pragma unroll
    for (int k = 0; k < 2; ++k) {
        double c, s;
        givens(y, z, &c, &s);
        if (k == 0) rot_cols<0, 1>(v, 3, c, s);
        else rot_cols<1, 2>(v, 3, c, s);
        double bk1 = bk * c - z * s;
        double ap1 = ap * c - bp * s;
        double bp1 = ap * s + bp * c;
        const double zp1 = aq * -s;
        const double aq1 = aq * c;
        if (k > 0) tau_v[0] = bk1;
        ak = ap1;
        bk = bp1;
        zk = zp1;
        ap = aq1;
        bp = (k < 1) ? tau_v[1] : 0.0;
        y = ak;
        z = zk;
        givens(y, z, &c, &s);
        if (k == 0) rot_cols<0, 1>(u, rows, c, s);
        else rot_cols<1, 2>(u, rows, c, s);
        const double ak1 = ak * c - zk * s;
        bk1 = bk * c - ap * s;
        const double zk1 = bp * -s;
        ap1 = bk * s + ap * c;
        bp1 = bp * c;
        tau_u[k] = ak1;
        ak = ak1;
        bk = bk1;
        zk = zk1;
        ap = ap1;
        bp = bp1;
        aq = (k < 1) ? tau_u[2] : 0.0;
        y = bk;
        z = zk;
    }
    tau_v[1] = bk;
    tau_u[2] = ap;
}

// returns false when the sweep bound was reached
template <int R>
ISO_QEF_FN bool diagonalise(double (&u)[R][3], double (&v)[3][3], double (&tau_u)[3], double (&tau_v)[2], int rows) {
    chop<0, 3>(tau_u, tau_v);
    int b = 2;
    int guard = 0;
    while (b > 0) {
        if (++guard > QR_SWEEP_LIMIT) return false;
        const double last = b == 2 ? tau_v[1] : tau_v[0];
        if (last == 0.0) {
            b -= 1;
        } else if (b == 2 && tau_v[0] != 0.0) {
            qr_cols3(u, v, tau_u, tau_v, rows);
            chop<0, 3>(tau_u, tau_v);
        } else if (b == 2) {
            qr_cols2<1>(u, v, tau_u, tau_v, rows);
            chop<1, 2>(tau_u, tau_v);
        } else {
            qr_cols2<0>(u, v, tau_u, tau_v, rows);
            chop<0, 2>(tau_u, tau_v);
        }
    }
    return true;
}

template <int R>
ISO_QEF_FN void singularise(double (&u)[R][3], double (&v)[3][3], double (&d)[3], int rows) {
#pragma unroll
    for (int j = 0; j < 3; ++j) {
        if (d[j] < 0.0) {
#pragma unroll
            for (int i = 0; i < 3; ++i) v[i][j] = -v[i][j];
            d[j] = -d[j];
        }
    }
    auto exchange = [&](double& a, double& b) {
        const double t = a;
        a = b;
        b = t;
    };
    // the largest of d[0..2] to the front, then of d[1..2] (the first of equals)
    if (d[1] > d[0] && !(d[2] > d[1])) {
        exchange(d[0], d[1]);
        swap_cols<0, 1>(u, rows);
        swap_cols<0, 1>(v, 3);
    } else if (d[1] > d[0] ? d[2] > d[1] : d[2] > d[0]) {
        exchange(d[0], d[2]);
        swap_cols<0, 2>(u, rows);
        swap_cols<0, 2>(v, 3);
    }
    if (d[2] > d[1]) {
        exchange(d[1], d[2]);
        swap_cols<1, 2>(u, rows);
        swap_cols<1, 2>(v, 3);
    }
}

// The least-squares step of MinimiseQEF over the planes (normal[i], d[i]),
// i < rows: SVD, truncated solve, the point relative to the centre of mass.
template <int R>
ISO_QEF_FN F3 solve_planes(const F3* normal, const float* dist, int rows, bool edge, bool* ok) {
    double u[R][3], v[3][3], d[3] = {0.0, 0.0, 0.0}, tau_v[2] = {0.0, 0.0};
#pragma unroll
    for (int i = 0; i < R; ++i) {
        const bool in = i < rows;
        u[i][0] = in ? (double)normal[i].x : 0.0;
        u[i][1] = in ? (double)normal[i].y : 0.0;
        u[i][2] = in ? (double)normal[i].z : 0.0;
    }
    bidiagonalise(u, d, tau_v, rows);
    unpack(u, v, d, tau_v, rows);
    *ok = diagonalise(u, v, d, tau_v, rows);
    singularise(u, v, d, rows);
    if (edge) {
        // the smallest singular value (the first of equals) goes
        double s_min = 1.7976931348623157e308;
        int id = 0;
#pragma unroll
        for (int i = 0; i < 3; ++i)
            if (d[i] < s_min) {
                s_min = d[i];
                id = i;
            }
#pragma unroll
        for (int i = 0; i < 3; ++i)
            if (i == id) d[i] = 0.0;
    }
#pragma unroll
    for (int i = 0; i < 3; ++i)
        if (d[i] < 0.1) d[i] = 0.0;
    double w[3] = {0.0, 0.0, 0.0};
#pragma unroll
    for (int i = 0; i < R; ++i) {
        if (i >= rows) continue;
        const double b = (double)dist[i];
        if (b != 0.0)
#pragma unroll
            for (int j = 0; j < 3; ++j) w[j] += b * u[i][j];
    }
#pragma unroll
    for (int i = 0; i < 3; ++i)
        if (d[i] != 0.0) w[i] /= d[i];
    double x[3];
#pragma unroll
    for (int i = 0; i < 3; ++i) {
        double s = 0.0;
#pragma unroll
        for (int j = 0; j < 3; ++j) s += w[j] * v[i][j];
        x[i] = s;
    }
    return f3((float)x[0], (float)x[1], (float)x[2]);
}

#undef ISO_QEF_FN

// MinimiseQEF::place_feature_with_tangents; *ok = false if the QR bound hit
__host__ __device__ inline F3 minimise_qef(const Planes& t, bool* ok) {
    *ok = true;
    if (t.feature == PLANAR) return t.com;
    return add(t.com, solve_planes<8>(t.normal, t.d, 8, t.feature == EDGE, ok));
}

}  // namespace qef
}  // namespace iso
