// Small dense block operations of the exact-order sweeps, in the reference's order of operations.
#pragma once

#include "common.cuh"

namespace jxcpr {

// sum_j mat[i][j] v[j] of each row, Kahan-compensated (jxfpamg-0220/csrc/mat_vec_data/
// seq_bsr_matrix.c:841-872)
template <int BS>
__device__ __forceinline__ void blk_kahan(const double *mat, const double *v, double *out) {
#pragma unroll
    for (int i = 0; i < BS; ++i) {
        double sum = 0.0, c = 0.0;
#pragma unroll
        for (int j = 0; j < BS; ++j) {
            const double y = mat[i * BS + j] * v[j] - c;
            const double t = sum + y;
            c = (t - sum) - y;
            sum = t;
        }
        out[i] = sum;
    }
}

// ov += alpha mat v
template <int BS>
__device__ __forceinline__ void blk_matvec_stable(double alpha, const double *__restrict__ mat, const double *v,
                                                  double *ov) {
    double sum[BS];
    blk_kahan<BS>(mat, v, sum);
#pragma unroll
    for (int i = 0; i < BS; ++i) ov[i] += alpha * sum[i];
}

// x / d, correctly rounded, where r = 1 / d (correctly rounded) is at hand: two residual corrections of x r,
// each residual exact by the fused multiply-add; the last correction of a quotient within one unit in the
// last place rounds correctly when r does (P. Markstein, IBM J. Res. Dev. 34(1), 1990).  A third of the
// latency of a division, on the chain from one group of a sweep to the next.  Outside the exponents for which
// no step over- or underflows the division itself.
__device__ __forceinline__ double div_known(double x, double d, double r) {
    const unsigned hx = ((unsigned)__double2hiint(x) >> 20) & 0x7ffu, hd = ((unsigned)__double2hiint(d) >> 20) & 0x7ffu;
    if (hx - 623u < 801u && hd - 623u < 801u) {  // 2^-400 <= |x|, |d| < 2^401
        double q = x * r;
        q = fma(fma(-d, q, x), r, q);
        return fma(fma(-d, q, x), r, q);
    }
    return x / d;
}

// The parts of a 2x2 block's solve that do not depend on the right-hand side: 1 / det, or NaN where
// blk_inv_matvec takes its other branch (a determinant that cancels).
__device__ __forceinline__ double blk2_inv_det(const double *mat) {
    const double a11 = mat[0], a12 = mat[1], a21 = mat[2], a22 = mat[3];
    const double det = a11 * a22 - a12 * a21;
    if (fabs(det) < 1e-12 * (fabs(a11 * a22) + fabs(a12 * a21))) return __longlong_as_double(0x7ff8000000000000LL);
    return 1.0 / det;
}

// ov = mat^-1 v (seq_bsr_matrix.c:945-1100)
template <int BS>
__device__ __forceinline__ void blk_inv_matvec(const double *mat, const double *v, double *ov) {
    if (BS == 2) {
        const double a11 = mat[0], a12 = mat[1], a21 = mat[2], a22 = mat[3];
        const double det = a11 * a22 - a12 * a21;
        if (fabs(det) < 1e-12 * (fabs(a11 * a22) + fabs(a12 * a21))) {
            ov[0] = v[0] / (a11 + 1e-12);
            ov[1] = v[1] / (a22 + 1e-12);
            return;
        }
        const double inv_det = 1.0 / det;
        const double b1 = v[0], b2 = v[1];
        ov[0] = (a22 * b1 - a12 * b2) * inv_det;
        ov[1] = (-a21 * b1 + a11 * b2) * inv_det;
        return;
    }
    double m[9], x[3], o[3] = {0.0, 0.0, 0.0};
#pragma unroll
    for (int q = 0; q < 9; ++q) m[q] = mat[q];
#pragma unroll
    for (int q = 0; q < 3; ++q) x[q] = v[q];
    const int n = 3;
    for (int i = 0; i < n; ++i) {
        int mr = i;
        double mv = fabs(m[i * n + i]);
        for (int k = i + 1; k < n; ++k)
            if (fabs(m[k * n + i]) > mv) {
                mv = fabs(m[k * n + i]);
                mr = k;
            }
        if (mv < 1e-15) {
            for (int j = 0; j < n; ++j) {
                const double d = m[j * n + j];
                o[j] = (fabs(d) > 1e-12) ? x[j] / d : 0.0;
            }
            break;
        }
        if (mr != i) {
            for (int j = 0; j < n; ++j) {
                const double t = m[i * n + j];
                m[i * n + j] = m[mr * n + j];
                m[mr * n + j] = t;
            }
            const double t = x[i];
            x[i] = x[mr];
            x[mr] = t;
        }
        const double pivot = m[i * n + i];
        for (int k = i + 1; k < n; ++k) {
            const double fct = m[k * n + i] / pivot;
            m[k * n + i] = fct;
            for (int j = i + 1; j < n; ++j) m[k * n + j] -= fct * m[i * n + j];
        }
    }
    for (int i = 0; i < n; ++i) {
        o[i] = x[i];
        for (int j = 0; j < i; ++j) o[i] -= m[i * n + j] * o[j];
    }
    for (int i = n - 1; i >= 0; --i) {
        for (int j = i + 1; j < n; ++j) o[i] -= m[i * n + j] * o[j];
        const double d = m[i * n + i];
        if (fabs(d) > 1e-15) o[i] /= d; else o[i] = 0.0;
    }
#pragma unroll
    for (int q = 0; q < 3; ++q) ov[q] = o[q];
}

}  // namespace jxcpr
