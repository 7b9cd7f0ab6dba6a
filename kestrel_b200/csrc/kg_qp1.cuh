// kg_qp1.cuh — the simplex QP of the SQP step (src/sqp.rs:112-250) solved by
// one thread: min 1/2 y'Qy + c'y subject to y >= 0, sum y = 1, from y0, by the
// reference's active-set method.  Each iteration factors the free block of Q
// with the GMW81-modified LDL^T (src/cholesky.rs:6-65), solves it for the
// gradient and for the ones vector, and either releases the variable with the
// most negative multiplier or steps to the first blocking bound.
//
// It computes what the row-parallel form (qp_simplex_rows in kg_rowsolve.cuh)
// computes, operation for operation and in the same order (the same FMAs,
// quotients and sequential sums), so both give the same bits (FAST: to an ulp of
// each quotient); with a thread per slot a warp serves 32 pairs' QPs instead of two.
//
// The lanes' free sets differ, so the code has no branch on them: a fixed
// variable's rows and columns are zeros and its pivot 1, which adds exact
// zeros to every sum (branches on the free set ran each of its cases one after
// the other: 4,300 instructions an iteration, this form about 1,300).  A
// quotient by one divisor used several times (a pivot, the sum of y) is q = c r
// with r = 1 / d, corrected by the remainder: with r correctly rounded that is
// the correctly rounded quotient (Markstein, IBM J. Res. Dev. 34, 1990), in
// three instructions instead of a division.
#pragma once

#include <math_constants.h>

#include "kg_solver.cuh"

namespace kg {

__host__ __device__ __forceinline__ int popc9(unsigned v) {
    int n = 0;
#pragma unroll
    for (int i = 0; i < 9; i++) n += (v >> i) & 1u;
    return n;
}

// 1 / d: the correctly rounded quotient, or (FAST) the hardware's approximation r
// and one step of third order (1 / d = r / (1 - e) with e = 1 - d r, its series to
// e^2: the rest is e^3 = 2^-60), to an ulp, at a third of the latency (a division
// is a chain of 127 cycles, and an iteration has a pivot's in each of its nine
// columns one after the other).
template <bool FAST>
__host__ __device__ __forceinline__ double recip(double d) {
#ifdef __CUDA_ARCH__
    if (FAST) {
        double r;
        asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(r) : "d"(d));
        const double e = fma(-d, r, 1.0);
        return fma(fma(e, e, e), r, r);
    }
#endif
    return 1.0 / d;
}

// c / d, given r = 1 / d; correctly rounded when r is.
__host__ __device__ __forceinline__ double quot(double c, double d, double r) {
    const double q = c * r;
    return fma(fma(-q, d, c), r, q);
}

// Entry (i, j), i <= j, of the stored upper triangle of Q.
__host__ __device__ constexpr int upper_at(int i, int j) { return i * 9 - i * (i - 1) / 2 + (j - i); }
constexpr int QP_Q = 45;   // upper triangle of Q, then c
constexpr int QP_IN = 54;

// Column j of the factorisation and the ones after it.
template <int j, bool FAST, class QF>
__host__ __device__ __forceinline__ void ldl_columns(const QF& Q, unsigned F, double beta2, double rbeta2, double delta,
                                                     double (&L)[36], double (&d)[9], double (&rd)[9]) {
    const bool jf = (F >> j) & 1u;
    double p[9];
    double sjj = 0.0;
#pragma unroll
    for (int s = 0; s < j; s++) {
        const double ljs = L[j * (j - 1) / 2 + s];
        p[s] = d[s] * ljs;
        sjj = fma(p[s], ljs, sjj);
    }
    const double cjj = Q(j, j) - sjj;
    double theta = 0.0;
#pragma unroll
    for (int i = j + 1; i < 9; i++) {
        double sij = 0.0;
#pragma unroll
        for (int s = 0; s < j; s++) sij = fma(p[s], L[i * (i - 1) / 2 + s], sij);
        const double cij = jf && ((F >> i) & 1u) ? Q(j, i) - sij : 0.0;
        L[i * (i - 1) / 2 + j] = cij;
        theta = fmax(theta, fabs(cij));
    }
    const double dj = fmax(fmax(fabs(cjj), quot(theta * theta, beta2, rbeta2)), delta);
    d[j] = jf ? dj : 1.0;
    rd[j] = recip<FAST>(d[j]);
#pragma unroll
    for (int i = j + 1; i < 9; i++) L[i * (i - 1) / 2 + j] = quot(L[i * (i - 1) / 2 + j], d[j], rd[j]);
    if constexpr (j + 1 < 9) ldl_columns<j + 1, FAST>(Q, F, beta2, rbeta2, delta, L, d, rd);
}

// GMW81-modified LDL^T of the free block (mask F, nf free): L strictly lower
// (row i at i (i - 1) / 2), d the pivots, rd their reciprocals; fixed variables
// have zero rows and columns and pivot 1.  Q(i, j) reads the upper triangle.
template <bool FAST, class QF>
__host__ __device__ __forceinline__ void ldl_gmw_thread(const QF& Q, unsigned F, int nf, double (&L)[36],
                                                        double (&d)[9], double (&rd)[9]) {
    double gamma = 0.0, xi = 0.0;
#pragma unroll
    for (int r = 0; r < 9; r++) {
        const bool rf = (F >> r) & 1u;
        gamma = fmax(gamma, rf ? fabs(Q(r, r)) : 0.0);
#pragma unroll
        for (int j = r + 1; j < 9; j++) xi = fmax(xi, rf && ((F >> j) & 1u) ? fabs(Q(r, j)) : 0.0);
    }
    const double eps = 2.220446049250313e-16;
    const double delta = eps * fmax(1.0, gamma + xi);
    const double t = sqrt((double)nf * (double)nf - 1.0);
    const double ratio = (nf <= 1) ? 0.0 : xi / t;
    const double beta2 = fmax(fmax(gamma, ratio), eps);
    const double rbeta2 = recip<FAST>(beta2);
    ldl_columns<0, FAST>(Q, F, beta2, rbeta2, delta, L, d, rd);
}

// L D L^T z = b for two right-hand sides (zero at fixed variables), in the
// order of ldl_solve2_rows.
__host__ __device__ __forceinline__ void ldl_solve2_thread(const double (&L)[36], const double (&d)[9],
                                                           const double (&rd)[9], double (&b0)[9], double (&b1)[9]) {
#pragma unroll
    for (int i = 0; i < 9; i++) {
        double s0 = 0.0, s1 = 0.0;
#pragma unroll
        for (int j = 0; j < i; j++) {
            s0 = fma(b0[j], L[i * (i - 1) / 2 + j], s0);
            s1 = fma(b1[j], L[i * (i - 1) / 2 + j], s1);
        }
        b0[i] = b0[i] - s0;
        b1[i] = b1[i] - s1;
    }
#pragma unroll
    for (int i = 0; i < 9; i++) {
        b0[i] = quot(b0[i], d[i], rd[i]);
        b1[i] = quot(b1[i], d[i], rd[i]);
    }
#pragma unroll
    for (int i = 8; i >= 0; i--) {
        double t0 = 0.0, t1 = 0.0;
#pragma unroll
        for (int j = i + 1; j < 9; j++) {
            t0 = fma(b0[j], L[j * (j - 1) / 2 + i], t0);
            t1 = fma(b1[j], L[j * (j - 1) / 2 + i], t1);
        }
        b0[i] = b0[i] - t0;
        b1[i] = b1[i] - t1;
    }
}

// The QP from y (in) to y (out); in(k): the upper triangle of Q (row-major,
// k < 45), then c.  Returns the iteration count.
template <bool FAST, class In>
__host__ __device__ __forceinline__ int qp_simplex_thread(const In& in, const Tune& tu, double (&y)[9]) {
    auto Q = [&](int i, int j) { return in(i <= j ? upper_at(i, j) : upper_at(j, i)); };
    unsigned work = 0;
#pragma unroll
    for (int i = 0; i < 9; i++)
        if (y[i] == 0.0) work |= 1u << i;
    for (int it = 0; it < tu.qp_max_iter; it++) {
        {
            double s = 0.0;
#pragma unroll
            for (int i = 0; i < 9; i++) s += y[i];
            const double rs = recip<FAST>(s);
#pragma unroll
            for (int i = 0; i < 9; i++) y[i] = quot(y[i], s, rs);
        }
        const unsigned F = (~work) & 0x1FFu;
        const int nf = popc9(F);
        if (nf == 0) return it;
        // the gradient c + Q y (fixed variables' y are 0) and, on the free
        // block, the ones vector
        double gq[9], gf[9], on[9];
#pragma unroll
        for (int r = 0; r < 9; r++) {
            double s = 0.0;
#pragma unroll
            for (int j = 0; j < 9; j++) s = fma(Q(r, j), y[j], s);
            gq[r] = in(QP_Q + r) + s;
            const bool rf = (F >> r) & 1u;
            gf[r] = rf ? gq[r] : 0.0;
            on[r] = rf ? 1.0 : 0.0;
        }
        {
            double L[36], d[9], rd[9];
            ldl_gmw_thread<FAST>(Q, F, nf, L, d, rd);
            ldl_solve2_thread(L, d, rd, gf, on);
        }
        double sg = 0.0, so = 0.0;
#pragma unroll
        for (int i = 0; i < 9; i++) { sg += gf[i]; so += on[i]; }
        const double lambda = sg / so;
        double m = 0.0;
        bool m_nan = false;
#pragma unroll
        for (int i = 0; i < 9; i++) {
            gf[i] = lambda * on[i] - gf[i];
            const double a = fabs(gf[i]);
            m_nan = m_nan || isnan(a);
            m = fmax(m, a);
        }
        if (!m_nan && m <= tu.qp_zero_search_tol) {
            if (nf == 9) return it;
            int best = -1;
            double gb = 0.0;
#pragma unroll
            for (int i = 0; i < 9; i++)
                if (((work >> i) & 1u) && (best < 0 || gq[i] < gb)) { best = i; gb = gq[i]; }
            if (gb - lambda >= -tu.qp_conv_tol) return it;
            work &= ~(1u << best);
        } else {
            double alpha = 1.0;
            int block = -1;
#pragma unroll
            for (int i = 0; i < 9; i++) {
                const double pv = ((work >> i) & 1u) ? 0.0 : gf[i];
                gf[i] = pv;
                const double den = pv < 0.0 ? pv : -1.0;
                const double a = FAST ? -y[i] * recip<FAST>(den) : -y[i] / den;
                if (pv < 0.0 && a < alpha) { alpha = a; block = i; }
            }
#pragma unroll
            for (int i = 0; i < 9; i++) {
                y[i] = fmax(y[i] + alpha * gf[i], 0.0);
                if (i == block) y[i] = 0.0;
            }
            if (block >= 0) work |= 1u << block;
        }
    }
    return tu.qp_max_iter;
}

// Column j of the plain LDL^T of the block F (unit pivots and zero columns
// outside it) and the ones after it.
template <int j, class HF>
__device__ __forceinline__ void ldl_plain_columns(const HF& H, unsigned F, double (&L)[36], double (&D)[9],
                                                  bool& positive) {
    const bool jf = (F >> j) & 1u;
    double p[9], sjj = 0.0;
#pragma unroll
    for (int s = 0; s < j; s++) {
        const double l = L[j * (j - 1) / 2 + s];
        p[s] = D[s] * l;
        sjj = fma(p[s], l, sjj);
    }
    const double dj = H(upper_at(j, j)) - sjj;
    D[j] = jf ? dj : 1.0;
    positive = positive && D[j] > 0.0;
    const double rd = recip<true>(D[j]);
#pragma unroll
    for (int i = j + 1; i < 9; i++) {
        double sij = 0.0;
#pragma unroll
        for (int s = 0; s < j; s++) sij = fma(p[s], L[i * (i - 1) / 2 + s], sij);
        L[i * (i - 1) / 2 + j] = jf && ((F >> i) & 1u) ? quot(H(upper_at(j, i)) - sij, D[j], rd) : 0.0;
    }
    if constexpr (j + 1 < 9) ldl_plain_columns<j + 1>(H, F, L, D, positive);
}

// The reduced Hessian's condition estimate at a KKT point (condition_estimate
// of kg_solver.cuh, src/sqp.rs:313-391), with zero rows and unit pivots for the
// variables left out in place of a compacted matrix.  H(k): the upper triangle.
template <class HF>
__device__ __forceinline__ double condition_thread(const HF& H, const double (&x)[9], const double (&g)[9], double tol) {
    double lambda = 0.0;
#pragma unroll
    for (int i = 0; i < 9; i++) lambda = fma(x[i], g[i], lambda);
    unsigned F = 0;
#pragma unroll
    for (int i = 0; i < 9; i++)
        if (!(x[i] == 0.0 && g[i] >= lambda + tol)) F |= 1u << i;
    if (F == 0) return CUDART_INF;
    double L[36], D[9];
    bool positive = true;
    ldl_plain_columns<0>(H, F, L, D, positive);
    if (!positive) return CUDART_INF;
    int imax = -1, imin = -1;
    double dmax = 0.0, dmin = 0.0;
#pragma unroll
    for (int i = 0; i < 9; i++) {
        if (!((F >> i) & 1u)) continue;
        if (imax < 0 || D[i] >= dmax) { imax = i; dmax = D[i]; }
        if (imin < 0 || D[i] < dmin) { imin = i; dmin = D[i]; }
    }
    // |L e_max| and |L^-T e_min|
    double wmax = 0.0, wmin = 0.0, z[9];
#pragma unroll
    for (int i = 0; i < 9; i++) {
        double l = i == imax ? 1.0 : 0.0;
#pragma unroll
        for (int j = 0; j < i; j++)
            if (j == imax) l = L[i * (i - 1) / 2 + j];
        wmax = fma(l, l, wmax);
    }
#pragma unroll
    for (int i = 8; i >= 0; i--) {
        double s = 0.0;
#pragma unroll
        for (int j = i + 1; j < 9; j++) s = fma(z[j], L[j * (j - 1) / 2 + i], s);
        z[i] = (i == imin ? 1.0 : 0.0) - s;
        wmin = fma(z[i], z[i], wmin);
    }
    return sqrt(wmax) * sqrt(wmin) * (dmax / dmin);
}


}  // namespace kg
