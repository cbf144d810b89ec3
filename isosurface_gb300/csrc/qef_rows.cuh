// MinimiseQEF's SVD (qef.cuh) by eight lanes, one row of U each (device only).
//
// A solve is one chain of f64 operations, a warp's f64 instruction holds its
// sub-partition's unit for 64 cycles whatever its active lanes, and a lattice
// has only a few thousand feature cells: a cell per lane leaves most
// sub-partitions idle while each busy one works through the rows one after
// the other.  Here an operation on all rows is one instruction; sums over the
// rows add the lanes' products in the rows' order, so every result has the
// bits of the one-lane solve.  The scalars are the same in all eight lanes,
// which therefore take every branch together.
#pragma once
#include <cuda_runtime.h>

#include "qef.cuh"

namespace iso {
namespace qef {

struct RowSolve {
    double u[3];    // row `y` of U
    double v[3];    // lanes 0 to 2: row `y` of V
    double d[3];    // tau_u, then the singular values
    double tv[2];   // tau_v, then the superdiagonal
    uint32_t mask;  // the group's lanes
    int y, rows;

    __device__ __forceinline__ double get(double x, int from) const { return __shfl_sync(mask, x, from, 8); }

    // s + the lanes' p of rows first .. rows - 1, in order
    __device__ __forceinline__ double add_rows(double s, double p, int first) const {
        for (int r = first; r < rows; ++r) s += get(p, r);
        return s;
    }

    // householder_col of column C
    template <int C>
    __device__ __forceinline__ double householder() {
        const int n = rows - C;
        double tau = 0.0;
        if (n <= 1) return tau;
        double xnorm;
        if (n == 2) {
            xnorm = fabs(get(u[C], C + 1));
        } else {
            // the running maximum before each row (magnitudes order as integers)
            const bool below = y > C && y < rows;
            const double v = below ? fabs(u[C]) : 0.0;
            double scl = 0.0, mine = 0.0;
            for (int r = C + 1; r < rows; ++r) {
                const double vr = get(v, r);
                if (r == y) mine = scl;
                if (__double_as_longlong(scl) < __double_as_longlong(vr)) scl = vr;
            }
            const bool some = v != 0.0, grow = __double_as_longlong(mine) < __double_as_longlong(v);
            const double ratio = some ? (grow ? mine : v) / (grow ? v : mine) : 0.0;
            const double term = grow ? ratio : ratio * ratio;
            const uint32_t base = (uint32_t)__ffs(mask) - 1;
            const uint32_t some_m = __ballot_sync(mask, some) >> base, grow_m = __ballot_sync(mask, grow) >> base;
            double ssq = 1.0;
            for (int r = C + 1; r < rows; ++r) {
                const double t = get(term, r);
                if (!(some_m >> r & 1u)) continue;
                ssq = grow_m >> r & 1u ? 1.0 + ssq * t * t : ssq + t;
            }
            xnorm = scl * sqrt(ssq);
        }
        if (xnorm != 0.0) {
            const double alpha = get(u[C], C);
            double beta = sqrt(alpha * alpha + xnorm * xnorm);
            if (alpha >= 0.0) beta = -beta;
            tau = (beta - alpha) / beta;
            const double s = 1.0 / (alpha - beta);
            if (y == C) u[C] = beta;
            else if (y > C && y < rows) u[C] *= s;
        }
        return tau;
    }

    // the reflection of column C, of factor tau, on column X
    template <int C, int X>
    __device__ __forceinline__ void reflect(double tau) {
        const double wx = add_rows(get(u[X], C), u[X] * u[C], C + 1), t = tau * wx;
        if (y == C) u[X] -= t;
        else if (y > C && y < rows) u[X] -= t * u[C];
    }

    __device__ __forceinline__ void bidiagonalise() {
        d[0] = householder<0>();
        if (d[0] != 0.0) {
            reflect<0, 1>(d[0]);
            reflect<0, 2>(d[0]);
        }
        double x0 = get(u[1], 0), x1 = get(u[2], 0);
        tv[0] = householder_pair(x0, x1);
        if (y == 0) {
            u[1] = x0;
            u[2] = x1;
        }
        if (tv[0] != 0.0 && y > 0 && y < rows) {
            double w = u[1];
            w += u[2] * x1;
            const double t = tv[0] * w;
            u[1] -= t;
            u[2] -= t * x1;
        }
        __syncwarp(mask);
        d[1] = householder<1>();
        if (d[1] != 0.0) reflect<1, 2>(d[1]);
        tv[1] = 0.0;
        d[2] = householder<2>();
    }

    template <int C>
    __device__ __forceinline__ void unpack_column() {
        const double tau = d[C];
        d[C] = get(u[C], C);
        const bool below = y > C && y < rows;
        if (tau == 0.0) {
            if (y == C) {
                u[C] = 1.0;
                if (C < 2) u[2] = 0.0;
                if (C < 1) u[1] = 0.0;
            }
            if (below) u[C] = 0.0;
            return;
        }
#pragma unroll
        for (int x = C + 1; x < 3; ++x) {
            const double wx = add_rows(0.0, u[x] * u[C], C + 1), t = tau * wx;
            if (y == C) u[x] = -t;
            else if (below) u[x] -= t * u[C];
        }
        if (below) u[C] = u[C] * -tau;
        if (y == C) u[C] = 1.0 - tau;
    }

    __device__ __forceinline__ void unpack() {
#pragma unroll
        for (int x = 0; x < 3; ++x) v[x] = y == x ? 1.0 : 0.0;
        const double tau = tv[0], u02 = get(u[2], 0);
        if (tau != 0.0) {
#pragma unroll
            for (int x = 1; x < 3; ++x) {
                double wx = get(v[x], 1);
                wx += get(v[x], 2) * u02;
                const double t = tau * wx;
                if (y == 1) v[x] -= t;
                if (y == 2) v[x] -= t * u02;
            }
        }
        tv[0] = get(u[1], 0);
        tv[1] = get(u[2], 1);
        unpack_column<2>();
        unpack_column<1>();
        unpack_column<0>();
    }

    template <int P, int Q>
    static __device__ __forceinline__ void rotate(double (&m)[3], double c, double s) {
        const double mp = m[P], mq = m[Q];
        m[P] = mp * c - mq * s;
        m[Q] = mp * s + mq * c;
    }
    template <int P, int Q>
    static __device__ __forceinline__ void swap(double (&m)[3]) {
        const double t = m[P];
        m[P] = m[Q];
        m[Q] = t;
    }

    // qr_middle, qr_end, qr_cols2 and qr_cols3 of qef.cuh
    template <int COL>
    __device__ __forceinline__ void middle() {
        double x = tv[COL], w = d[COL + 1], c, s;
        givens(w, -x, &c, &s);
        rotate<COL, COL + 1>(u, c, s);
        d[COL + 1] = x * s + w * c;
        tv[COL] = x * c - w * s;
        if (COL == 0) {
            const double z = tv[1];
            tv[1] *= c;
            x = z * -s;
            w = d[2];
            givens(w, -x, &c, &s);
            rotate<0, 2>(u, c, s);
            d[2] = x * s + w * c;
        }
    }
    __device__ __forceinline__ void end() {
        double x = d[1], w = tv[1], c, s;
        givens(x, w, &c, &s);
        rotate<1, 2>(v, c, s);
        d[1] = x * c - w * s;
        tv[1] = x * s + w * c;
        const double z = tv[0];
        tv[0] *= c;
        x = d[0];
        w = z * s;
        givens(x, w, &c, &s);
        rotate<0, 2>(v, c, s);
        d[0] = x * c - w * s;
    }
    template <int A>
    __device__ __forceinline__ void step2() {
        double c, s;
        if (d[A] == 0.0) {
            givens(tv[A], d[A + 1], &c, &s);
            d[A] = tv[A] * c - d[A + 1] * s;
            tv[A] = tv[A] * s + d[A + 1] * c;
            d[A + 1] = 0.0;
            rotate<A, A + 1>(u, c, s);
            swap<A, A + 1>(v);
        } else if (d[A + 1] == 0.0) {
            givens(d[A], tv[A], &c, &s);
            d[A] = d[A] * c - tv[A] * s;
            tv[A] = 0.0;
            rotate<A, A + 1>(v, c, s);
        } else {
            schur(d[A], tv[A], d[A + 1], &c, &s);
            double a11 = d[A] * c - tv[A] * s;
            double a21 = -d[A + 1] * s;
            double a12 = d[A] * s + tv[A] * c;
            double a22 = d[A + 1] * c;
            rotate<A, A + 1>(v, c, s);
            if (a11 * a11 + a21 * a21 < a12 * a12 + a22 * a22) {
                double t = a11;
                a11 = a12;
                a12 = t;
                t = a21;
                a21 = a22;
                a22 = t;
                swap<A, A + 1>(v);
            }
            givens(a11, a21, &c, &s);
            d[A] = a11 * c - a21 * s;
            tv[A] = a12 * c - a22 * s;
            d[A + 1] = a12 * s + a22 * c;
            rotate<A, A + 1>(u, c, s);
        }
    }
    __device__ __forceinline__ void step3() {
        if (d[0] == 0.0) return middle<0>();
        if (d[1] == 0.0) return middle<1>();
        if (d[2] == 0.0) return end();
        const double mu = shift(d, tv);
        double w = d[0] * d[0] - mu, z = d[0] * tv[0];
        double ak = 0.0, bk = 0.0, zk;
        double ap = d[0], bp = tv[0], aq = d[1];
#pragma unroll
        for (int k = 0; k < 2; ++k) {
            double c, s;
            givens(w, z, &c, &s);
            if (k == 0) rotate<0, 1>(v, c, s);
            else rotate<1, 2>(v, c, s);
            double bk1 = bk * c - z * s;
            double ap1 = ap * c - bp * s;
            double bp1 = ap * s + bp * c;
            const double zp1 = aq * -s;
            const double aq1 = aq * c;
            if (k > 0) tv[0] = bk1;
            ak = ap1;
            bk = bp1;
            zk = zp1;
            ap = aq1;
            bp = (k < 1) ? tv[1] : 0.0;
            w = ak;
            z = zk;
            givens(w, z, &c, &s);
            if (k == 0) rotate<0, 1>(u, c, s);
            else rotate<1, 2>(u, c, s);
            const double ak1 = ak * c - zk * s;
            bk1 = bk * c - ap * s;
            const double zk1 = bp * -s;
            ap1 = bk * s + ap * c;
            bp1 = bp * c;
            d[k] = ak1;
            ak = ak1;
            bk = bk1;
            zk = zk1;
            ap = ap1;
            bp = bp1;
            aq = (k < 1) ? d[2] : 0.0;
            w = bk;
            z = zk;
        }
        tv[1] = bk;
        d[2] = ap;
    }
    __device__ __forceinline__ bool diagonalise() {
        chop<0, 3>(d, tv);
        int b = 2, guard = 0;
        while (b > 0) {
            if (++guard > QR_SWEEP_LIMIT) return false;
            const double last = b == 2 ? tv[1] : tv[0];
            if (last == 0.0) {
                b -= 1;
            } else if (b == 2 && tv[0] != 0.0) {
                step3();
                chop<0, 3>(d, tv);
            } else if (b == 2) {
                step2<1>();
                chop<1, 2>(d, tv);
            } else {
                step2<0>();
                chop<0, 2>(d, tv);
            }
        }
        return true;
    }
    __device__ __forceinline__ void singularise() {
#pragma unroll
        for (int j = 0; j < 3; ++j)
            if (d[j] < 0.0) {
                v[j] = -v[j];
                d[j] = -d[j];
            }
        if (d[1] > d[0] && !(d[2] > d[1])) {
            swap<0, 1>(d);
            swap<0, 1>(u);
            swap<0, 1>(v);
        } else if (d[1] > d[0] ? d[2] > d[1] : d[2] > d[0]) {
            swap<0, 2>(d);
            swap<0, 2>(u);
            swap<0, 2>(v);
        }
        if (d[2] > d[1]) {
            swap<1, 2>(d);
            swap<1, 2>(u);
            swap<1, 2>(v);
        }
    }
};

// solve_planes of qef.cuh by the eight lanes of `mask` (an aligned group, all
// of which call it), lane y with plane y of `rows` (at most 8; lanes past
// them: anything): the point relative to the centre of mass, in every lane.
__device__ __forceinline__ F3 solve_planes_rows(uint32_t mask, F3 normal, float dist, int rows, bool edge, bool* ok) {
    RowSolve q;
    q.mask = mask;
    q.y = (int)(threadIdx.x & 7);
    q.rows = rows;
    const bool in = q.y < rows;
    q.u[0] = in ? (double)normal.x : 0.0;
    q.u[1] = in ? (double)normal.y : 0.0;
    q.u[2] = in ? (double)normal.z : 0.0;
    q.bidiagonalise();
    q.unpack();
    *ok = q.diagonalise();
    q.singularise();
    double (&d)[3] = q.d;
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
    const double b = in ? (double)dist : 0.0;
    const uint32_t some = __ballot_sync(mask, b != 0.0) >> (__ffs(mask) - 1);
    double w[3] = {0.0, 0.0, 0.0};
    const double p0 = b * q.u[0], p1 = b * q.u[1], p2 = b * q.u[2];
    for (int r = 0; r < rows; ++r) {
        const double a0 = q.get(p0, r), a1 = q.get(p1, r), a2 = q.get(p2, r);
        if (!(some >> r & 1u)) continue;
        w[0] += a0;
        w[1] += a1;
        w[2] += a2;
    }
    // lane j divides w[j]
    const double wj = q.y == 0 ? w[0] : q.y == 1 ? w[1] : w[2], dj = q.y == 0 ? d[0] : q.y == 1 ? d[1] : d[2];
    const double quot = dj != 0.0 ? wj / dj : wj;
#pragma unroll
    for (int j = 0; j < 3; ++j) w[j] = q.get(quot, j);
    double s = 0.0;
#pragma unroll
    for (int j = 0; j < 3; ++j) s += w[j] * q.v[j];
    const float x = (float)s;
    return f3(__shfl_sync(mask, x, 0, 8), __shfl_sync(mask, x, 1, 8), __shfl_sync(mask, x, 2, 8));
}

}  // namespace qef
}  // namespace iso
